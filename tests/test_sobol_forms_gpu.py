"""Sobol's launch rule: the two forms of the 8-byte kinds and the block sizes, chosen by points,
dimensions and whether the rows are made of whole vectors, and the forms of Poisson and the fp32
normals.  Rows on both sides of each line of the rule, one element off, and one after the other on
one generator, whose launch shape must not outlive a change of buffer or size."""

import numpy as np
import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

# (dimensions, points): one wave of one-group blocks and a part (8 x 262144), more, fewer; many short
# and few long rows that split vectors; a row of one point less or more than a block's group
SHAPES = [(8, 262144), (8, 524288), (1, 1048576), (127, 32769), (128, 32769), (128, 32772), (200, 10487),
          (1000, 2099), (3, 1023), (3, 1025)]


@pytest.mark.parametrize("rng,dist,params", [(504, "ulonglong", []), (505, "uniform_double", []),
                                             (501, "uniform_double", []), (502, "poisson", [10.0]),
                                             (505, "poisson", [10.0]), (501, "normal", [0.0, 1.0]),
                                             (501, "poisson", [5000.0])], ids=lambda x: str(x))
def test_shapes(lib, orc, rng, dist, params):
    for dims, n in SHAPES:
        calls = [(dist, dims * n, params, mis) for mis in (0, 1, 4, 0)]
        calls.append((dist, dims * (n + 1), params, 0))
        g = gu.create(lib, rng, None, 11, dims)
        ref = pyorc.run_sequence(orc, rng, None, 11, calls, dims=dims)
        try:
            for k, ((d, m, p, mis), (ost, want)) in enumerate(zip(calls, ref)):
                st, got = gu.device_generate(lib, g, d, m, p, mis)
                assert st == ost == 0
                gu.compare_call(orc, rng, None, 11, dims, calls, k, np.asarray(got), want)
        finally:
            lib.rocrand_destroy_generator(g)
