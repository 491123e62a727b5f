"""The packed fp32 / half Box-Muller in the fill kernels: call sizes around the pairs' loops (an
even and an odd number of rounds, a last round of one or a few units, a head and a tail that are
units alone), and the uniform 1, whose radius is 0."""

import numpy as np
import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

E = 512 * 256
GENS = {"xorwow": 401, "mrg32k3a": 402, "mtgp32": 403, "philox": 404, "mrg31k3p": 405, "lfsr113": 406,
        "threefry2x32": 408, "threefry2x64": 409, "threefry4x64": 411}


@pytest.mark.parametrize("name", sorted(GENS))
@pytest.mark.parametrize("dist,params", [("normal", [0.5, 2.0]), ("normal_half", [0.0, 1.0]),
                                         ("log_normal", [0.0, 0.5])], ids=lambda x: str(x))
def test_sizes_around_pairs(lib, orc, name, dist, params):
    offset = None if name == "mtgp32" else 0
    calls = [(dist, n, params, mis) for n, mis in
             ((2, 0), (2 * E, 0), (4 * E + 2, 0), (6 * E - 1, 1), (8 * E + 7, 1))]
    g = gu.create(lib, GENS[name], 99, offset)
    ref = pyorc.run_sequence(orc, GENS[name], 99, offset, calls)
    try:
        for k, ((d, n, p, mis), (ost, ovals)) in enumerate(zip(calls, ref)):
            st, vals = gu.device_generate(lib, g, d, n, p, mis)
            assert st == ost == 0
            gu.compare_call(orc, GENS[name], 99, offset, None, calls, k, vals, ovals)
    finally:
        lib.rocrand_destroy_generator(g)


def test_uniform_one(lib, orc):
    # word 0 of block 3895978 of seed 77 is 4294967185, which rounds up to u = 1
    offset = 4 * (3895978 - 2)
    for mis in (0, 2):  # one block per vector, and two
        calls = [("normal", 33, [0.0, 1.0], mis)]
        g = gu.create(lib, 404, 77, offset)
        st, vals = gu.device_generate(lib, g, *calls[0])
        assert st == 0
        lib.rocrand_destroy_generator(g)
        _, want = pyorc.run_sequence(orc, 404, 77, offset, calls)[0]
        assert np.count_nonzero(np.asarray(want) == 0) == 2
        assert np.array_equal(np.asarray(vals) == 0, np.asarray(want) == 0)
        gu.compare_call(orc, 404, 77, offset, None, calls, 0, vals, want)
