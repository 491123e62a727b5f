"""Philox calls whose vectors straddle two blocks: the shifted kernel's rows (sizes around a warp's
rows, its thresholds of 2^17 and 2^20 vectors, the vectors at multiples of 262144 that begin
elsewhere when the head is odd), a counter whose low word ends inside the call, and heads and
tails of every length, made by a block of their own."""

import numpy as np
import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

V17, V20 = 1 << 17, 1 << 20


def _run(lib, orc, seed, offset, calls):
    g = gu.create(lib, 404, seed, offset)
    ref = pyorc.run_sequence(orc, 404, seed, offset, calls)
    try:
        for k, ((d, n, p, mis), (ost, ovals)) in enumerate(zip(calls, ref)):
            st, vals = gu.device_generate(lib, g, d, n, p, mis)
            assert st == ost == 0
            if gu.bit_exact(404, d):
                assert np.array_equal(vals.view(np.uint8), np.asarray(ovals).view(np.uint8)), (k, d, n, mis)
            else:
                gu.compare_call(orc, 404, seed, offset, None, calls, k, vals, ovals)
    finally:
        lib.rocrand_destroy_generator(g)


@pytest.mark.parametrize("shift", [1, 2, 3])
def test_shifts_and_thresholds(lib, orc, shift):
    for vectors in (V17 - 1, V17, V17 + 31, V20 - 1, V20, V20 + 129):
        _run(lib, orc, 8, shift, [("uint", 4 * vectors + shift, (), 0)])


@pytest.mark.parametrize("dist,params", [("normal", [0.0, 1.0]), ("normal_double", [0.0, 1.0]),
                                         ("poisson", [3.0]), ("char", [])], ids=lambda x: str(x))
def test_odd_heads(lib, orc, dist, params):
    for mis in (1, 3):
        _run(lib, orc, 21, 0, [(dist, (1 << 21) + 777, params, mis)])


@pytest.mark.parametrize("before", [V17 + 1, V17 + 2, V17 + 40])
def test_low_word_ends(lib, orc, before):
    # the last counter used is the low word's last value, one behind it, or well inside
    _run(lib, orc, 5, 4 * ((1 << 32) - before) + 1, [("uint", 4 * (V17 + 1), (), 0), ("uint", 9, (), 0)])


@pytest.mark.parametrize("dist,params", [("char", []), ("normal_half", [0.0, 1.0]), ("uniform_double", []),
                                         ("normal", [0.0, 1.0])], ids=lambda x: str(x))
def test_heads_and_tails(lib, orc, dist, params):
    calls = [(dist, n, params, mis) for mis in range(0, 16, 3) for n in (1, 2, 7, 15, 16, 17, 31, 33, 300)]
    _run(lib, orc, 3, 0, calls)
