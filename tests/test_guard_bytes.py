"""The guard bytes of the GPU tests' outputs (gpu_util.guarded_output) see a write next to an output."""

import pytest
import torch

from tests import gpu_util as gu


@pytest.mark.parametrize("dtype,mis", [(torch.uint8, 3), (torch.float16, 1), (torch.float32, 0),
                                       (torch.float64, 2)], ids=str)
def test_stray_writes_are_seen(dtype, mis):
    for n in (0, 1, 37):
        raw, out, address = gu.guarded_output(n, dtype, mis, device="cpu")
        at = address - raw.data_ptr()
        assert out.numel() == n and at == gu.GUARD + mis * out.element_size()
        assert raw.numel() >= at + n * out.element_size() + gu.GUARD
        out.zero_()
        gu.check_guards(raw, out)
        for stray in (at - 1, at + n * out.element_size(), 0, raw.numel() - 1):
            spoiled = raw.clone()
            spoiled[stray] = 0
            with pytest.raises(AssertionError):
                gu.check_guards(spoiled, spoiled[at:at + n * out.element_size()].view(dtype))
