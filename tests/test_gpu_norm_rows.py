"""``add_rms_norm`` in fp32, a CTA per row and (rows that are not whole 16-byte pieces) a warp per row, against the formula."""

import pytest
import torch

from atma_b200.inference_ops import add_rms_norm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,D", [(1, 8), (3, 264), (130, 1024), (2, 4096), (5, 1020), (4, 33)])
def test_fp32_rows(rows, D):
    torch.manual_seed(rows + D)
    x, y, w = (torch.randn(s, device="cuda") for s in ((rows, D), (rows, D), (D,)))
    total, h = add_rms_norm(x, y, w, 1e-6)
    assert torch.equal(total, x + y)
    s = (x + y).double()
    want = s * torch.rsqrt(s.square().mean(-1, keepdim=True) + 1e-6) * w.double()
    # the mean square of D values is off by D / 8 + 8 roundings at most, most of which cancel, its root by half of that
    assert (h.double() - want).abs().max() <= 2.0 ** -24 * 16 * want.abs().max()
    lead = torch.randn(rows * D + 1, device="cuda")[1:].view(rows, D)                # rows that are not 16-byte aligned
    assert torch.allclose(add_rms_norm(lead, None, w, 1e-6)[1], add_rms_norm(lead.clone(), None, w, 1e-6)[1], rtol=1e-6, atol=0)


@pytest.mark.parametrize("rows,D", [(2048, 504), (2049, 504), (2049, 512), (3000, 8)])
def test_many_fp32_rows(rows, D):
    """From 2049 rows on a row of fewer than 512 values has a warp."""
    test_fp32_rows(rows, D)
