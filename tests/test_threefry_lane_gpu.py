"""The ThreeFry fast path folds the counter's fixed words into the launch: calls whose counters end
at the low word's last value, pass it by one block, and start just behind it (32-bit engines; an
offset cannot reach the 64-bit low word's end), and calls that start inside a block."""

import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rng,width", [(410, 4), (408, 2), (411, 4), (409, 2)])
@pytest.mark.parametrize("dist,params", [("uint", []), ("uniform_double", []), ("normal", [0.0, 1.0]),
                                         ("char", [])], ids=lambda x: str(x))
def test_counter_carry(lib, orc, rng, width, dist, params):
    # elements per 16-byte-or-so vector are at most 32: 40 blocks hold some vectors of any kind
    for blocks_before, shift in ((40, 0), (39, 0), (41, 0), (0, 0), (1, 0), (40, 1)):
        offset = width * ((1 << 32) - blocks_before) + shift
        for n, mis in ((40 * width, 0), (4096 + 5, 0), (1000, 1)):
            calls = [(dist, n, params, mis), (dist, 64, params, 0)]
            g = gu.create(lib, rng, 4711, offset)
            ref = pyorc.run_sequence(orc, rng, 4711, offset, calls)
            try:
                for k, ((d, m, p, s), (ost, ovals)) in enumerate(zip(calls, ref)):
                    st, vals = gu.device_generate(lib, g, d, m, p, s)
                    assert st == ost == 0
                    gu.compare_call(orc, rng, 4711, offset, None, calls, k, vals, ovals)
            finally:
                lib.rocrand_destroy_generator(g)
