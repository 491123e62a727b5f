"""The stateful fill's wide blocks: misaligned outputs from 128 MiB on.  Calls one value below and at
that size, aligned and one element off, and the call after them, which shows every engine's state."""

import numpy as np
import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

LIMIT = 128 << 20


@pytest.mark.parametrize("rng,dist,params", [(401, "uint", []), (401, "char", []), (401, "uniform_double", []),
                                             (401, "poisson", [10.0]), (402, "uniform_double", []),
                                             (405, "uniform_double", []), (406, "short", [])],
                         ids=lambda x: str(x))
def test_around_the_limit(lib, orc, rng, dist, params):
    n = LIMIT // np.dtype(pyorc.DISTS[dist][1]).itemsize
    for calls in ([(dist, n, params, 1), (dist, 300001, params, 0)],
                  [(dist, n - 1, params, 1), (dist, n + 3, params, 0), (dist, 131073, params, 1)]):
        g = gu.create(lib, rng, 2024, 7)
        ref = pyorc.run_sequence(orc, rng, 2024, 7, calls)
        try:
            for (d, m, p, mis), (ost, want) in zip(calls, ref):
                st, got = gu.device_generate(lib, g, d, m, p, mis)
                assert st == ost == 0
                assert np.array_equal(got.view(np.uint8), np.asarray(want).view(np.uint8)), (m, mis)
        finally:
            lib.rocrand_destroy_generator(g)
