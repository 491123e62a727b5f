"""MTGP32's fill loop runs whole turns of four block steps at fixed ring offsets, then the rest
one step at a time: calls of every number of rounds around a turn, a part of a round, and a head
and tail, one after the other on one generator so that calls start at each of the four offsets."""

import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

ROUND = 512 * 256


@pytest.mark.parametrize("dist,params", [("uint", []), ("uniform_double", []), ("short", []), ("poisson", [4.0]),
                                         ("normal", [0.0, 1.0]), ("normal_half", [0.0, 1.0]),
                                         ("normal_double", [0.0, 1.0])], ids=lambda x: str(x))
def test_turns(lib, orc, dist, params):
    sizes = [1, 255, 256, 257, ROUND - 1, ROUND, ROUND + 1, 2 * ROUND + 300, 3 * ROUND, 5 * ROUND + 256,
             8 * ROUND, 3, 9 * ROUND + 777]
    calls = [(dist, n, params, k % 3) for k, n in enumerate(sizes)]
    g = gu.create(lib, 403, 31337, None)
    ref = pyorc.run_sequence(orc, 403, 31337, None, calls)
    try:
        for k, ((d, n, p, mis), (ost, ovals)) in enumerate(zip(calls, ref)):
            st, vals = gu.device_generate(lib, g, d, n, p, mis)
            assert st == ost == 0
            gu.compare_call(orc, 403, 31337, None, None, calls, k, vals, ovals)
    finally:
        lib.rocrand_destroy_generator(g)
