"""MT19937's seeding kernels: the start states of all 8192 generators, word by word.

One round of raw words (78 slots of 65536 lanes) holds every word of every generator once, so
it shows each state word that the two jump digits made: both ends of the four 160-word slices
(the last one is ragged), of the 256 first-digit and the 32 second-digit values.  A generator
that has already run is reseeded, so the scratch of an earlier seeding is there."""

import numpy as np
import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu

ROUND = 78 * 65536


@pytest.mark.parametrize("seed", [0xfffffffffffffff5])
def test_every_start_state(lib, orc, seed):
    g = gu.create(lib, 407, 1234, None)
    try:
        st, _ = gu.device_generate(lib, g, "uint", 1000, [], 0)
        assert st == 0
        assert lib.rocrand_set_seed(g, seed) == 0
        st, vals = gu.device_generate(lib, g, "uint", ROUND, [], 0)
        assert st == 0
    finally:
        lib.rocrand_destroy_generator(g)
    ost, want = pyorc.run_sequence(orc, 407, seed, None, [("uint", ROUND, (), 0)])[0]
    assert ost == 0
    assert np.array_equal(np.asarray(vals).view(np.uint32), np.asarray(want).view(np.uint32))
