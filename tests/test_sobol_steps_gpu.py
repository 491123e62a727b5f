"""Sobol points whose first index has each residue modulo 4 (the kernels keep three of the four
steps' direction vectors in registers), at the ends of a thread's group and a block's run.  (Calls
that pass the 32-bit counter's last point are left out: there the reference's device engine, which
the kernels follow, and its host engine, which the oracle restates, step differently.)"""

import pytest

from oracle import pyorc
from tests import gpu_util as gu

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rng", [501, 502, 504, 505])
@pytest.mark.parametrize("dist,params", [("uint", []), ("uniform_double", []), ("char", []), ("short", []),
                                         ("normal", [0.0, 1.0]), ("normal_half", [0.0, 1.0]),
                                         ("log_normal", [0.0, 0.5]), ("poisson", [7.0])], ids=lambda x: str(x))
def test_residues_and_ends(lib, orc, rng, dist, params):
    dims = 3
    for offset in (0, 1, 2, 3, 4093, 0x7ffffffd):
        calls = [(dist, n * dims, params, 0) for n in (1, 5, 1023, 1025, 4099)]
        g = gu.create(lib, rng, None, offset, dims)
        ref = pyorc.run_sequence(orc, rng, None, offset, calls, dims=dims)
        try:
            for k, ((d, n, p, mis), (ost, ovals)) in enumerate(zip(calls, ref)):
                st, vals = gu.device_generate(lib, g, d, n, p, mis)
                assert st == ost == 0
                gu.compare_call(orc, rng, None, offset, dims, calls, k, vals, ovals)
        finally:
            lib.rocrand_destroy_generator(g)
