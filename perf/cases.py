"""Performance cases of the library's generate path, through its public entry points.

Three kinds of case:

* ``fill``  -- a program keeps a generator (``PRNG`` / ``QRNG``) and an output buffer and
  calls one of its methods again and again: the ordinary use of the library, from a thousand
  values to 2^28 (1 GiB of floats, the benchmark's size);
* ``reseed`` -- the same with a new seed before each call: a program that wants reproducible
  or independent streams per experiment, epoch or task;
* ``batch`` -- a plan of many small and large requests, laid out once and executed as one
  launch (``rocrand_b200_execute_batch_plan`` with its CUDA graph).

``exact`` restates the generators in plain torch / numpy and evaluates every transform in 64
bits.  MT19937 has no such restatement here: placing its 8192 generators 2^1000 values apart
takes minutes in Python.
"""

import ctypes
import functools
import math
import os

import numpy as np
import torch

import rocrand_b200 as rb

ENGINES = 512 * 256        # engines of XORWOW, MRG32k3a, MRG31k3p and LFSR113
REF_STRIDE = 1024 * 256    # vectors per round of the counter engines' output order
MASK32 = 0xFFFFFFFF

PSEUDO = {
    "xorwow": rb.PRNG.XORWOW, "mrg32k3a": rb.PRNG.MRG32K3A, "mtgp32": rb.PRNG.MTGP32,
    "philox4x32_10": rb.PRNG.PHILOX4_32_10, "mrg31k3p": rb.PRNG.MRG31K3P,
    "lfsr113": rb.PRNG.LFSR113, "mt19937": rb.PRNG.MT19937,
    "threefry2x32_20": rb.PRNG.THREEFRY2_32_20, "threefry2x64_20": rb.PRNG.THREEFRY2_64_20,
    "threefry4x32_20": rb.PRNG.THREEFRY4_32_20, "threefry4x64_20": rb.PRNG.THREEFRY4_64_20,
}
QUASI = {
    "sobol32": rb.QRNG.SOBOL32, "scrambled_sobol32": rb.QRNG.SCRAMBLED_SOBOL32,
    "sobol64": rb.QRNG.SOBOL64, "scrambled_sobol64": rb.QRNG.SCRAMBLED_SOBOL64,
}

# torch type of each distribution's output (unsigned words travel in the signed types)
TYPES = {
    "uint8": torch.int8, "uint16": torch.int16, "uint32": torch.int32, "uint64": torch.int64,
    "uniform_f16": torch.float16, "uniform_f32": torch.float32, "uniform_f64": torch.float64,
    "normal_f16": torch.float16, "normal_f32": torch.float32, "normal_f64": torch.float64,
    "log_normal_f16": torch.float16, "log_normal_f32": torch.float32,
    "log_normal_f64": torch.float64, "poisson": torch.int32,
}


def listed():
    return [
        # the default generator, a small array: a call's latency
        fill("xorwow_uniform_small", "xorwow", "uniform_f32", 1000),
        # noise for one layer or image: an ordinary size, odd, into the middle of a buffer
        fill("philox_normal_f32_odd", "philox4x32_10", "normal_f32", 1000003, misalign=1),
        # the headline: one GiB of uniform floats
        fill("philox_uniform_f32_2p28", "philox4x32_10", "uniform_f32", 1 << 28),
        # Monte Carlo in double precision
        fill("philox_normal_f64", "philox4x32_10", "normal_f64", 1 << 25),
        # the default generator's normals in bulk
        fill("xorwow_normal_f32", "xorwow", "normal_f32", 1 << 27),
        # event counts
        fill("mrg32k3a_poisson", "mrg32k3a", "poisson", (1 << 24) + 5, lam=10.0),
        # a new seed for each experiment, then one array of it
        dict(fill("mt19937_reseed", "mt19937", "uniform_f32", 1 << 20), kind="reseed"),
        # price paths: log-normal factors, not a round number
        fill("mt19937_log_normal_f32", "mt19937", "log_normal_f32", 10000001, mean=0.05, std=0.2),
        # raw bulk randomness from the block-parallel twister
        fill("mtgp32_uniform_f32", "mtgp32", "uniform_f32", 1 << 26),
        # 53-bit uniforms from a 64-bit counter engine
        fill("threefry4x64_uniform_f64", "threefry4x64_20", "uniform_f64", 1 << 25),
        # quasi-Monte Carlo integration: 64 dimensions of normals
        fill("sobol32_normal_f32_64d", "sobol32", "normal_f32", 1 << 20, dims=64),
        # many tasks' arrays in one launch
        batch("batch_512", 512, 10, 22, "philox4x32_10,xorwow"),
    ]


def fill(name, generator, dist, n, dims=1, misalign=0, mean=0.0, std=1.0, lam=0.0):
    """n values per dimension; the buffer starts `misalign` elements into an allocation."""
    return {"name": name, "kind": "fill", "generator": generator, "dist": dist, "n": n, "dims": dims,
            "misalign": misalign, "mean": mean, "std": std, "lambda": lam}


def batch(name, requests, lo, hi, generators):
    """Requests of log-uniform sizes in [2^lo, 2^hi]: half uniform, 30 % normal, 20 % Poisson."""
    return {"name": name, "kind": "batch", "requests": requests, "lo": lo, "hi": hi,
            "generators": generators}


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["fill", "reseed", "batch"], [0.75, 0.13, 0.12])[0]
    if kind == "batch":
        c = batch("", _log_int(rng, 16, 1024), 10, rng.choice([14, 18, 21]),
                  rng.choice(["philox4x32_10", "philox4x32_10,xorwow",
                              "philox4x32_10,xorwow,mrg32k3a,sobol32"]))
        del c["name"]
        return c
    quasi = kind == "fill" and rng.random() < 0.2
    generator = rng.choice(sorted(QUASI if quasi else PSEUDO))
    dists = [d for d in sorted(TYPES) if d != "uint64" or "64" in generator]
    # the types most in use come up more often than the narrow ones
    weight = {"uniform_f32": 4, "normal_f32": 4, "uniform_f64": 2, "normal_f64": 3, "uint32": 2, "poisson": 2}
    dist = rng.choices(dists, [weight.get(d, 1) for d in dists])[0]
    dims = _log_int(rng, 1, 1000) if quasi else 1
    n = max(1, _log_int(rng, 100, (1 << 27) if kind == "fill" else (1 << 24)) // dims)
    if rng.random() < 0.5:
        n |= 1
    lam = rng.choice([0.5, 4.0, 10.0, 500.0, 1000.0, 5000.0]) if dist == "poisson" else 0.0
    std = rng.choice([1.0, 0.25])
    c = fill("", generator, dist, n, dims, misalign=rng.choice([0, 0, 1, 2, 3]),
             mean=rng.choice([0.0, 0.5]), std=std, lam=lam)
    c["kind"] = kind
    del c["name"]
    return c


# ---- the calls ----

def _seed(seed):
    """A generator seed made from the case's seed."""
    return (seed * 2654435761 + 12345) & 0x7FFFFFFF


class Fill:
    def __init__(self, case, seed):
        self.case = case
        self.offset = 0
        self.seed = _seed(seed)
        g = case["generator"]
        if g in QUASI:
            self.offset = 1 + self.seed % 100000
            self.gen = rb.QRNG(QUASI[g], ndim=case["dims"], offset=self.offset)
        else:
            self.gen = rb.PRNG(PSEUDO[g], seed=self.seed)
        count = case["n"] * case["dims"]
        buf = torch.zeros(count + case["misalign"], dtype=TYPES[case["dist"]], device="cuda")
        self.out = buf[case["misalign"]:]

    def run(self):
        c, gen, out = self.case, self.gen, self.out
        if c["kind"] == "reseed":
            gen.seed = self.seed
        d = c["dist"]
        if d == "poisson":
            return gen.poisson(out, c["lambda"])
        if d.startswith("uint"):
            return gen.generate(out)
        if d.startswith("uniform"):
            return gen.uniform(out)
        if d.startswith("normal"):
            return gen.normal(out, c["mean"], c["std"])
        return gen.lognormal(out, c["mean"], c["std"])


BATCH_KINDS = [("uniform_f32", rb.B200_DIST_UNIFORM_FLOAT, torch.float32),
               ("normal_f32", rb.B200_DIST_NORMAL_FLOAT, torch.float32),
               ("poisson", rb.B200_DIST_POISSON, torch.int32)]


def _requests(case, seed):
    """The requests of a batch: (generator, kind, seed, n, first element in its kind's buffer)."""
    sizes = np.random.RandomState(42)  # the mix of sizes and kinds is the case's own
    seeds = np.random.RandomState(_seed(seed))
    gens = case["generators"].split(",")
    got, used = [], [0, 0, 0]
    for i in range(case["requests"]):
        n = int(round(2.0 ** sizes.uniform(case["lo"], case["hi"])))
        k = int(sizes.choice(3, p=[0.5, 0.3, 0.2]))
        got.append((gens[i % len(gens)], k, int(seeds.randint(1, (1 << 31) - 1)), n, used[k]))
        used[k] += (n + 127) // 128 * 128  # every request's output starts a 512-byte line
    return got, used


class Batch:
    def __init__(self, case, seed):
        self.lib = rb.load_library()
        requests, used = _requests(case, seed)
        self.out = {name: torch.zeros(max(1, used[k]), dtype=t, device="cuda")
                    for k, (name, _, t) in enumerate(BATCH_KINDS)}
        table = (rb.BatchRequest * len(requests))()
        for r, (g, k, s, n, at) in zip(table, requests):
            name, dist, _ = BATCH_KINDS[k]
            r.rng_type = PSEUDO.get(g) or QUASI[g]
            r.distribution = dist
            r.seed = s
            r.offset = 0
            r.param0, r.param1 = {"uniform_f32": (0.0, 0.0), "normal_f32": (0.0, 1.0), "poisson": (4.0, 0.0)}[name]
            r.output = self.out[name].data_ptr() + 4 * at
            r.n = n
        self.stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        self.plan = ctypes.c_void_p()
        rb.check_rocrand(self.lib.rocrand_b200_create_batch_plan(ctypes.byref(self.plan), table, len(requests),
                                                                 self.stream))

    def run(self):
        rb.check_rocrand(self.lib.rocrand_b200_execute_batch_plan(self.plan, 1, self.stream))
        return self.out

    def __del__(self):
        if getattr(self, "plan", None) is not None and self.plan.value:
            self.lib.rocrand_b200_destroy_batch_plan(self.plan)
            self.plan = None


def prepare(case, seed):
    return Batch(case, seed) if case["kind"] == "batch" else Fill(case, seed)


def run(state):
    return state.run()


def work(case):
    """Every output value written once; there is nothing to read.  The transforms' operations
    are not counted: they are not the tensor cores' kind of work."""
    if case["kind"] == "batch":
        mean = (2.0 ** case["hi"] - 2.0 ** case["lo"]) / ((case["hi"] - case["lo"]) * math.log(2.0))
        return {"bytes": case["requests"] * mean * 4, "flops": 0}
    return {"bytes": case["n"] * case["dims"] * TYPES[case["dist"]].itemsize, "flops": 0}


def tolerance(case):
    """Integers, uniforms and Poisson counts are defined bit for bit, and so are the quasi-random
    single- and half-precision normals.  The other transforms are rounded: about four times the
    error that the start shows against `exact`."""
    if case["kind"] == "batch":
        return {"rel": 2e-7, "max": 2e-6}
    d, g = case["dist"], case["generator"]
    if "normal" not in d or (g in QUASI and d in ("normal_f32", "normal_f16")):
        return "exact"
    if d.endswith("f64"):
        if g in QUASI or g == "threefry2x32_20":
            # the inverse error function's formula cancels: an ulp of its logarithm grows
            return {"rel": 4e-15, "max": 2e-13}
        return {"rel": 3e-16, "max": 4e-15}
    if d.endswith("f32"):
        return {"rel": 2e-7, "max": 2e-6}
    return {"rel": 1e-3, "max": 3e-3}


# ---- the same values in 64 bits, in plain torch and numpy ----

def _dev(a):
    return torch.as_tensor(a, dtype=torch.int64, device="cuda")


def _mulhilo(a, b):
    """High and low words of a 32 x 32-bit product in int64 (the wrapped sign is masked off)."""
    p = a * b
    return (p >> 32) & MASK32, p & MASK32


def _philox(seed, block):
    """Words of Philox4x32-10 blocks (counter < 2^64): [4, count]."""
    x = [block & MASK32, (block >> 32) & MASK32, torch.zeros_like(block), torch.zeros_like(block)]
    k0, k1 = seed & MASK32, seed >> 32
    for _ in range(10):
        h0, l0 = _mulhilo(x[0], 0xD2511F53)
        h1, l1 = _mulhilo(x[2], 0xCD9E8D57)
        x = [h1 ^ x[1] ^ k0, l1, h0 ^ x[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & MASK32, (k1 + 0xBB67AE85) & MASK32
    return torch.stack(x)


ROTATIONS = {
    (32, 4): [(10, 26), (11, 21), (13, 27), (23, 5), (6, 20), (17, 11), (25, 10), (18, 20)],
    (64, 4): [(14, 16), (52, 57), (23, 40), (5, 37), (25, 33), (46, 12), (58, 22), (32, 32)],
    (32, 2): [(13,), (15,), (26,), (6,), (17,), (29,), (16,), (24,)],
    (64, 2): [(16,), (42,), (12,), (31,), (16,), (32,), (24,), (21,)],
}


def _signed(v, bits):
    """A word as the int64 that holds it."""
    v &= (1 << bits) - 1
    return v - (1 << 64) if bits == 64 and v >> 63 else v


def _threefry(bits, width, seed, block):
    """Words of ThreeFry-20 blocks (counter < 2^32): [width, count]."""
    mask = MASK32 if bits == 32 else -1

    def rotl(v, r):
        return ((v << r) | ((v >> (bits - r)) & ((1 << r) - 1))) & mask

    full = (1 << bits) - 1
    keys = [(seed >> (16 * i)) & full for i in range(4)] if width == 4 else [seed & full, (seed >> 32) & full]
    keys.append(0x1BD11BDA if bits == 32 else 0x1BD11BDAA9FC1A22)
    for i in range(width):
        keys[width] ^= keys[i]
    x = [block] + [torch.zeros_like(block) for _ in range(width - 1)]
    x = [(v + _signed(keys[i], bits)) & mask for i, v in enumerate(x)]
    for r in range(20):
        rot = ROTATIONS[bits, width][r % 8]
        pairs = [(0, 1)] if width == 2 else [(0, 1), (2, 3)] if r % 4 < 2 else [(0, 3), (2, 1)]
        for (a, b), s in zip(pairs, rot):
            x[a] = (x[a] + x[b]) & mask
            x[b] = rotl(x[b], s) ^ x[a]
        if r % 4 == 3:
            i = r // 4 + 1
            for j in range(width):
                add = keys[(j + i) % (width + 1)] + (i if j == width - 1 else 0)
                x[j] = (x[j] + _signed(add, bits)) & mask
    return torch.stack(x)


def _xorwow_step(s):
    t = s[0] ^ (s[0] >> 2)
    v = (s[4] ^ (s[4] << 4)) ^ (t ^ (t << 1))
    return [s[1], s[2], s[3], s[4], v & MASK32]


def _lfsr113_step(s):
    out = []
    for v, a, b, keep, c in zip(s, (6, 2, 13, 3), (13, 27, 21, 12), (~1, ~7, ~15, ~127), (18, 2, 7, 13)):
        out.append((((v & keep & MASK32) << c) & MASK32) ^ ((((v << a) & MASK32) ^ v) >> b))
    return out


def _bits(words):
    """[.., w] words as [.., 32 w] bits."""
    return ((words.unsqueeze(-1) >> torch.arange(32, device="cuda")) & 1).flatten(-2).double()


@functools.lru_cache(None)
def _gf2_jumps(step, w, log2_jump):
    """Bit matrices of 2^log2_jump 2^b steps of a GF(2)-linear map on w words, b < 17."""
    basis = np.zeros((32 * w, w), dtype=np.int64)
    for i in range(32 * w):
        basis[i, i // 32] = 1 << (i % 32)
    m = _bits(torch.stack(step(list(_dev(basis).unbind(1))), 1))
    got = []
    for i in range(log2_jump + 17):
        if i >= log2_jump:
            got.append(m)
        m = (m @ m) % 2
    return got


def _gf2_engines(step, base, log2_jump, count):
    """States of engines e < count: `base` moved by e 2^log2_jump steps of a GF(2)-linear map."""
    w = len(base)
    x = _bits(_dev(base).unsqueeze(0).repeat(count, 1))
    e = torch.arange(count, device="cuda")
    for b, m in enumerate(_gf2_jumps(step, w, log2_jump)):
        x = torch.where(((e >> b) & 1).bool().unsqueeze(1), (x @ m) % 2, x)
    x = x.long().view(count, w, 32)
    return list((x << torch.arange(32, device="cuda")).sum(-1).unbind(1))


def _mod_engines(matrix, mod, base, log2_jump, count):
    """The same for a 3-word linear recurrence modulo `mod`."""
    m = [[v % mod for v in r] for r in matrix]

    def mul(a, b):
        return [[sum(a[i][k] * b[k][j] for k in range(3)) % mod for j in range(3)] for i in range(3)]

    for _ in range(log2_jump):
        m = mul(m, m)
    x = np.array([[v] * count for v in base], dtype=np.uint64)
    e = np.arange(count)
    for b in range(17):
        y = np.stack([sum((np.uint64(m[i][k]) * x[k]) % np.uint64(mod) for k in range(3)) % np.uint64(mod)
                      for i in range(3)])
        x = np.where((e >> b) & 1, y, x)
        m = mul(m, m)
    return [_dev(r.astype(np.int64)) for r in x]


def _stateful_words(gen, seed, steps, count):
    """Output words of engines e < count: [steps, count]."""
    out = torch.empty(steps, count, dtype=torch.int64, device="cuda")
    if gen == "xorwow":
        s = [123456789, 362436069, 521288629, 88675123, 5783321]
        t0 = 1228688033 * ((seed & MASK32) ^ 0x2C7F967F) & MASK32
        t1 = 2073658381 * ((seed >> 32) ^ 0xA03697CB) & MASK32
        base = [(s[0] + t0) & MASK32, s[1] ^ t0, (s[2] + t1) & MASK32, s[3] ^ t1, (s[4] + t0) & MASK32]
        d = (6615241 + t1 + t0) & MASK32
        s = _gf2_engines(_xorwow_step, base, 67, count)
        for i in range(steps):
            s = _xorwow_step(s)
            d = (d + 362437) & MASK32
            out[i] = (s[4] + d) & MASK32
    elif gen == "lfsr113":
        base = [(seed >> (16 * i)) & MASK32 for i in range(4)]
        base[0] += 2 if base[0] < 2 else 0
        base[1] += 8 if base[1] < 8 else 0
        s = _gf2_engines(_lfsr113_step, base, 55, count)
        for i in range(steps):
            s = _lfsr113_step(s)
            out[i] = s[0] ^ s[1] ^ s[2] ^ s[3]
    else:
        seed = seed or 12345
        k3a = gen == "mrg32k3a"
        m1, m2 = (4294967087, 4294944443) if k3a else (2147483647, 2147462579)
        x, y = (seed & MASK32) ^ 0x55555555, (seed >> 32) ^ 0xAAAAAAAA
        base1 = [x * seed % m1, y * seed % m1, x * seed % m1]
        base2 = [y * seed % m2, x * seed % m2, y * seed % m2]
        if k3a:  # words oldest first
            a1, a2 = [[0, 1, 0], [0, 0, 1], [-810728, 1403580, 0]], [[0, 1, 0], [0, 0, 1], [-1370589, 0, 527612]]
        else:    # words newest first
            a1, a2 = [[0, 1 << 22, 129], [1, 0, 0], [0, 1, 0]], [[1 << 15, 0, 32769], [1, 0, 0], [0, 1, 0]]
        jump = 76 if k3a else 72
        g = _mod_engines(a1, m1, base1, jump, count)
        h = _mod_engines(a2, m2, base2, jump, count)
        for i in range(steps):
            if k3a:
                g = [g[1], g[2], (1403580 * g[1] + 810728 * (m1 - g[0])) % m1]
                h = [h[1], h[2], (527612 * h[2] + 1370589 * (m2 - h[0])) % m2]
                p, q = g[2], h[2]
            else:
                g = [((g[1] << 22) + 129 * g[2]) % m1, g[0], g[1]]
                h = [((h[0] << 15) + 32769 * h[2]) % m2, h[0], h[1]]
                p, q = g[0], h[0]
            out[i] = p - q + torch.where(p <= q, m1, 0)
    return out


def _mtgp_words(seed, steps):
    """Output words of the 512 block generators, 256 a step: [steps, 512 * 256]."""
    path = os.path.join(os.path.dirname(os.path.abspath(rb.__file__)), "data", "mtgp32_params.bin")
    sets = np.fromfile(path, dtype="<u4", offset=12).reshape(512, 36).astype(np.int64)
    pos, sh1, sh2 = (_dev(sets[:, i]).unsqueeze(1) for i in range(3))
    tbl, tmp, mask = _dev(sets[:, 3:19]), _dev(sets[:, 19:35]), _dev(sets[:, 35:36])
    hidden = sets[:, 7] ^ ((sets[:, 11] << 16) & MASK32)
    b = (hidden + (hidden >> 16)) & MASK32
    b = (b + (b >> 8)) & 0xFF
    s = np.repeat((b * 0x01010101)[:, None], 351, 1)
    s[:, 0] = (seed ^ (seed >> 32)) + np.arange(512) + 1 & MASK32
    s[:, 1] = hidden
    for k in range(1, 351):
        s[:, k] ^= 1812433253 * (s[:, k - 1] ^ (s[:, k - 1] >> 30)) + k & MASK32
    # words[i] is state word i of the endless sequence, the last 351 kept
    state = _dev(s)
    out = torch.empty(steps, 512 * 256, dtype=torch.int64, device="cuda")
    t = torch.arange(256, device="cuda").unsqueeze(0)
    for i in range(steps):
        x = (state[:, 0:256] & mask) ^ state[:, 1:257]
        x = x ^ ((x << sh1) & MASK32)
        y = x ^ (state.gather(1, t + pos) >> sh2)
        r = y ^ tbl.gather(1, y & 15)
        v = state.gather(1, t + pos - 1)
        v = v ^ (v >> 16)
        v = v ^ (v >> 8)
        out[i] = (r ^ tmp.gather(1, v & 15)).flatten()
        state = torch.cat([state, r], 1)[:, 256:]
    return out


def _sobol_vectors(dims, bits):
    """Direction vectors of dimensions < dims from the Joe-Kuo parameters: [dims, bits]."""
    path = os.path.join(os.path.dirname(os.path.abspath(rb.__file__)), "data", "sobol_params.bin")
    raw = np.unpackbits(np.fromfile(path, dtype=np.uint8, offset=12), bitorder="little")
    at = 0

    def take(n):
        nonlocal at
        v = 0
        for i in range(n):
            v |= int(raw[at + i]) << i
        at += n
        return v

    got = [[1 << (bits - 1 - j) for j in range(bits)]]
    for _ in range(1, dims):
        s = take(5)
        a = take(s - 1)
        v = [take(j + 1) << (bits - 1 - j) for j in range(s)]
        for j in range(s, bits):
            x = v[j - s] ^ (v[j - s] >> s)
            for k in range(1, s):
                if (a >> (s - 1 - k)) & 1:
                    x ^= v[j - k]
            v.append(x)
        got.append(v)
    return got


def _f32(x):
    return x.to(torch.float32)


def _u_f32(v):
    """A word's single-precision uniform, rounded once to a float, in a double."""
    return _f32(_f32(v).double() * 2.0 ** -32 + 2.0 ** -32).double()


def _angle_f32(v, scale):
    c = torch.tensor(scale, dtype=torch.float32, device="cuda")
    return (_f32(v) * c + c).double()


def _box_muller(u, a):
    s = torch.sqrt(-2.0 * torch.log(u))
    return torch.stack([torch.sin(a) * s, torch.cos(a) * s], -1)


def _f64_of(x, y):
    return (x ^ (y << 21)).double() * 2.0 ** -53 + 2.0 ** -53


def _erfinv(x):
    """The reference's closed-form approximation of the inverse error function."""
    l = torch.log((1.0 - x) * (1.0 + x))
    t1 = 2.0 / (math.pi * 0.147) + 0.5 * l
    r = torch.sign(x) * torch.sqrt(torch.sqrt(t1 * t1 - l / 0.147) - t1)
    return torch.where(torch.isinf(l), torch.zeros_like(r), r)


def _apply(gen, dist, w, case):
    """The distribution's outputs [count, ow] for its input words w [iw, count], and nothing
    rounded but the uniforms that the transforms start from."""
    wide = gen in ("threefry2x64_20", "threefry4x64_20")
    base, kind = dist.rsplit("_", 1)
    mrg = {"mrg32k3a": 2.3283065498378288e-10, "mrg31k3p": 4.656612875245796923e-10}.get(gen)
    if mrg is not None and (dist == "uniform_f16" or kind == "f16"):
        w = ((w - 1).double() * {"mrg32k3a": 1.000000048661607, "mrg31k3p": 2.000000001396983862}[gen]).long()
    if base == "uniform":
        if kind == "f16":
            n = 4 if wide else 2
            return torch.stack([(((w[0] >> (16 * i)) & 0xFFFF) + 1).double() * 2.0 ** -16 for i in range(n)], -1)
        if mrg is not None:
            return (w[0].double() * mrg).unsqueeze(-1)
        if kind == "f32":
            return ((((w[0] >> 32) & MASK32) if wide else w[0]).double() * 2.0 ** -32 + 2.0 ** -32).unsqueeze(-1)
        v = (w[0] >> 11) & ((1 << 53) - 1) if wide else w[0] | ((w[1] >> 11) << 32)
        return (v.double() * 2.0 ** -53 + 2.0 ** -53).unsqueeze(-1)
    if kind == "f16":
        v = (w[0] & 0xFFFF) | (((w[0] >> 32) & 0xFFFF) << 16) if wide else w[0]
        z = _box_muller(((v & 0xFFFF) + 1).double() * 2.0 ** -16, _angle_f32(v >> 16, 9.58738e-05))
    elif mrg is not None:
        u, v = _f32(w[0].double() * mrg), _f32(w[1].double() * mrg)
        if kind == "f32":
            z = _box_muller(u.double(), (v * torch.tensor(6.2831855, dtype=torch.float32, device="cuda")).double())
        else:
            z = _box_muller(u.double(), v.double() * 2.0 * math.pi)
    elif kind == "f32":
        x, y = (w[0] & MASK32, (w[0] >> 32) & MASK32) if wide else (w[0], w[1])
        z = _box_muller(_u_f32(x), _angle_f32(y, 1.46291807e-09))
    elif gen == "threefry2x32_20":
        z = (_erfinv(2.0 * (w[0].double() * 2.0 ** -32 + 2.0 ** -32) - 1.0) * 1.41421353816986083984375).unsqueeze(-1)
    else:
        x = [w[0] & MASK32, (w[0] >> 32) & MASK32, w[1] & MASK32, (w[1] >> 32) & MASK32] if wide else list(w)
        z = _box_muller(_f64_of(x[0], x[1]), 2.0 * _f64_of(x[2], x[3]) * math.pi)
    z = case["mean"] + z * case["std"]
    return torch.exp(z) if base == "log_normal" else z


def _widths(gen, dist):
    """Input words and outputs of one application of a distribution."""
    wide = gen in ("threefry2x64_20", "threefry4x64_20")
    mrg = gen.startswith("mrg")
    base, kind = dist.rsplit("_", 1)
    if base == "uniform":
        if kind == "f16":
            return 1, 4 if wide else 2
        return (2 if kind == "f64" and not wide and not mrg else 1), 1
    if kind == "f16":
        return 1, 2
    if kind == "f32" or mrg:
        return (1 if wide else 2), 2
    if gen == "threefry2x32_20":
        return 1, 1
    return (2 if wide else 4), 2


def _fill_exact(case, seed, address):
    """One call's outputs on a fresh generator, for a buffer at `address`."""
    gen, dist, n = case["generator"], case["dist"], case["n"]
    iw, ow = _widths(gen, dist)
    size = TYPES[dist].itemsize
    if gen == "philox4x32_10" or gen.startswith("threefry"):
        width = 2 if "2x" in gen else 4
        per = width // iw * ow                       # elements of one output vector
        head = min(n, -(address // size) % per)
        vectors = (n - head) // per
        start0 = -(-head // ow) * iw                 # where the vectors of the first lane begin
        adj = head if gen == "philox4x32_10" and head else head // ow * iw
        out = torch.empty(n, dtype=torch.float64, device="cuda")

        def words(p):
            if gen == "philox4x32_10":
                b = _philox(seed, p // width)
            else:
                b = _threefry(64 if "x64" in gen else 32, width, seed, p // width)
            return b.gather(0, (p % width).unsqueeze(0))[0]

        def units(p):  # outputs of the units that begin at stream positions p
            return _apply(gen, dist, torch.stack([words(p + i) for i in range(iw)]), case)

        def at(j):
            return width * j + torch.where(j % REF_STRIDE == 0, start0, adj)

        def run_from(p, count):
            k = torch.arange(-(-count // ow), device="cuda")
            return units(p + k * iw).flatten()[:count]

        if head:
            out[:head] = run_from(0, head)
        for j0 in range(0, vectors, 1 << 21):
            j = torch.arange(j0, min(vectors, j0 + (1 << 21)), device="cuda")
            p = (at(j).unsqueeze(1) + torch.arange(width // iw, device="cuda") * iw).flatten()
            out[head + j0 * per:head + j0 * per + len(j) * per] = units(p).flatten()
        tail = n - head - vectors * per
        if tail:
            out[n - tail:] = run_from(int(at(_dev([vectors]))[0]), tail)
        return out
    mtgp = gen == "mtgp32"
    head = min(n, -(address // size) % ow)
    vectors = (n - head) // ow
    tail = n - head - vectors * ow
    rounds = -(-vectors // ENGINES)
    edge = 1 if mtgp else 2  # applications the head and tail may add
    steps = (rounds + edge) * iw
    w = _mtgp_words(seed, steps) if mtgp else _stateful_words(gen, seed, steps, min(ENGINES, vectors + 1))
    out = torch.empty(n, dtype=torch.float64, device="cuda")
    count = w.shape[1]
    for r in range(rounds):
        m = min(ENGINES, vectors - r * ENGINES)
        z = _apply(gen, dist, w[r * iw:(r + 1) * iw, :m], case)
        out[head + r * ENGINES * ow:head + (r * ENGINES + m) * ow] = z.flatten()
    if ow > 1 and (head or tail):
        # the slots after the last vector write them (MTGP32: the two threads after the last full
        # step, in the step that follows; the others: one engine, the head first)
        if mtgp:
            up = -(-vectors // 256) * 256
            spots = [(up // ENGINES, up % ENGINES), ((up + 1) // ENGINES, (up + 1) % ENGINES)]
        else:
            q, e = vectors // ENGINES, vectors % ENGINES
            spots = [(q, e), (q + (1 if head else 0), e)]
        z = [_apply(gen, dist, w[q * iw:(q + 1) * iw, e:e + 1], case).flatten() for q, e in spots]
        if head:
            out[:head] = z[0][:head]
        if tail:
            out[n - tail:] = z[1][:tail]
    return out


def _sobol_exact(case, offset):
    bits = 64 if "64" in case["generator"] else 32
    v = _sobol_vectors(case["dims"], bits)
    scrambled = case["generator"].startswith("scrambled")
    if scrambled:
        add = 640000 if bits == 32 else 1280000
        v = [[(x + add) & ((1 << bits) - 1) for x in r] for r in v]
    flat = [x for r in v for x in r]
    n, kind = case["n"], case["dist"].rsplit("_", 1)[1]
    k = (offset + torch.arange(n, device="cuda")) & MASK32
    gray = k ^ (k >> 1)
    rows = []
    for d in range(case["dims"]):
        x = torch.full_like(k, _signed(flat[d], bits) if scrambled else 0)
        for b in range(min(bits, 33)):
            x = torch.where((gray >> b) & 1 == 1, x ^ _signed(v[d][b], bits), x)
        top = (x >> 32) & MASK32 if bits == 64 else x
        if kind == "f16":
            u = ((top >> 16) + 1).double() * 2.0 ** -16 if case["dist"].startswith("uniform") else _u_f32(top)
        elif kind == "f32":
            u = top.double() * 2.0 ** -32 + 2.0 ** -32 if case["dist"].startswith("uniform") else _u_f32(top)
        elif bits == 64:
            u = ((x >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53 + 2.0 ** -53
        else:
            u = x.double() * 2.0 ** -32 + 2.0 ** -32
        if not case["dist"].startswith("uniform"):
            u = case["mean"] + _erfinv(2.0 * u - 1.0) * 1.41421353816986083984375 * case["std"]
            u = torch.exp(u) if case["dist"].startswith("log_normal") else u
        rows.append(u)
    return torch.stack(rows).flatten()


def exact(case, seed):
    if case["kind"] == "batch":
        requests, used = _requests(case, seed)
        if any(g not in PSEUDO for g, *_ in requests):
            return None
        out = {name: torch.zeros(max(1, used[k]), dtype=torch.float64, device="cuda") if k < 2 else None
               for k, (name, _, _) in enumerate(BATCH_KINDS)}
        for g, k, s, n, at in requests:
            if k < 2:
                c = fill("", g, BATCH_KINDS[k][0], n)
                out[BATCH_KINDS[k][0]][at:at + n] = _fill_exact(c, s, 0)
        return out
    if case["dist"].startswith("uint") or case["dist"] == "poisson" or case["generator"] == "mt19937":
        return None
    if case["generator"] in QUASI:
        return _sobol_exact(case, 1 + _seed(seed) % 100000)
    return _fill_exact(case, _seed(seed), case["misalign"] * TYPES[case["dist"]].itemsize)
