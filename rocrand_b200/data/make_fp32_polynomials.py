"""Derives the single-precision polynomials of rocrand_b200/csrc/normal_math.cuh.

Weighted minimax fits by Lawson's iteration (C. L. Lawson, 1961): least squares on a dense
Chebyshev-spaced grid, the weights multiplied by the error until it levels out.  Run by hand;
prints the coefficients (rounded to float) and the largest weighted error.

  2 log(1 + f), f = z - 1, z in [2/3, 4/3), as g + g^2 Q(g) with g = 2f: relative to the
      logarithm for f < 0 (k = 0) and to 2 log(1 + f) - 2 ln 2 for f > 0 (k <= -1 there);
  sin r = r + r^3 S(r^2) and cos r = 1 - r^2/2 + r^4 C(r^2), |r| <= pi/4, relative.
"""

import numpy as np


def fit(x, target, weight, powers, rounds=1500):
    """Coefficients of x^p, p in powers, that level |weight (sum - target)|."""
    a = np.stack([x ** p for p in powers], 1)
    w = np.full(len(x), 1.0 / len(x))
    best = None
    for _ in range(rounds):
        s = np.sqrt(w) * weight
        m = (a * s[:, None]).astype(np.float64)
        scale = np.abs(m).max(0)
        c = np.linalg.lstsq(m / scale, (target * s).astype(np.float64), rcond=None)[0] / scale
        e = np.abs(weight * (a @ c - target)).astype(np.float64)
        if best is None or e.max() < best[0]:
            best = (e.max(), c)
        w = w * e / (w * e).sum()
    return best


def show(name, got):
    print("%s: 2^%.2f" % (name, np.log2(got[0])), [float(np.float32(v)) for v in got[1]])


def main():
    t = np.cos(np.linspace(0.0, np.pi, 8001))
    f = (t / 3.0).astype(np.longdouble)
    f = f[np.abs(f) > 1e-4]
    log = 2.0 * np.log1p(f)
    g = 2.0 * f
    size = np.where(f < 0, np.abs(log), np.abs(log - 2.0 * np.log(np.longdouble(2))))
    show("Q", fit(g, (log - g) / g ** 2, g ** 2 / size, range(9)))
    r = (np.cos(np.linspace(0.0, np.pi / 2, 6001))[:-1] * (np.pi / 4 * (1 + 2.0 ** -20))).astype(np.longdouble)
    r = r[r > 1e-3]
    show("S", fit(r, (np.sin(r) - r) / r ** 3, r ** 3 / np.sin(r), (0, 2, 4)))
    show("C", fit(r, (np.cos(r) - 1 + r * r / 2) / r ** 4, r ** 4 / np.cos(r), (0, 2, 4)))


if __name__ == "__main__":
    main()
