"""MT19937's staged rounds take a thread's units inside the call as runs: calls that begin and end
in the middle of a round, with runs of every length around a step of four and its remainders, a
head and tail served by a unit of its own, and calls inside one slot group."""

import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

S = 65536


@pytest.mark.parametrize("dist,params,ow", [("normal", [0.0, 1.0], 2), ("normal_double", [0.5, 2.0], 2),
                                            ("normal_half", [0.0, 1.0], 2), ("log_normal", [0.0, 0.5], 2)],
                         ids=lambda x: str(x))
def test_runs(lib, orc, dist, params, ow):
    units = [1, S - 1, 3 * S, 4 * S + 5, 5 * S + 1, 7 * S, 20, 2 * S + 3, 39 * S, S // 2]
    calls = [(dist, u * ow + k % 2, params, (0, 1, 0, 3)[k % 4]) for k, u in enumerate(units)]
    g = gu.create(lib, 407, 555, None)
    ref = pyorc.run_sequence(orc, 407, 555, None, calls)
    try:
        for k, ((d, n, p, mis), (ost, ovals)) in enumerate(zip(calls, ref)):
            st, vals = gu.device_generate(lib, g, d, n, p, mis)
            assert st == ost == 0
            gu.compare_call(orc, 407, 555, None, None, calls, k, vals, ovals)
    finally:
        lib.rocrand_destroy_generator(g)
