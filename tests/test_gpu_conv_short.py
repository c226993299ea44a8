"""The packed gated convolution over sequences of a few tokens: the vector form against the channel-by-channel one, bit for bit."""

import pytest
import torch

import atma_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("K", [2, 3, 4])
@pytest.mark.parametrize("lengths", [[1] * 23, [2, 3, 1, 5, 4, 7, 6, 9, 8], [4] * 6 + [3], [17, 1, 30, 2]])
@pytest.mark.parametrize("form", ["fresh", "continued", "table and weights two bytes off"])
def test_runs_of_short_sequences(lengths, K, dtype, form):
    """Runs of four tokens with up to four sequences in them, ends and starts at every place; slots out of order, one sequence without."""
    D, total, n = 64, sum(lengths), len(lengths)
    g = torch.Generator().manual_seed(total + K)
    proj, w = torch.randn(total, 3 * D, generator=g).to(dtype).cuda(), torch.randn(D, K, generator=g).to(dtype).cuda()
    ends = torch.tensor(lengths).cumsum(0)
    rep = lambda t: t.repeat_interleave(torch.tensor(lengths)).int().cuda()               # noqa: E731
    slots = torch.randperm(n, generator=g)
    slots[n // 2] = -1
    maps = rep(ends - torch.tensor(lengths)), rep(ends), rep(slots)
    off = form.startswith("table")

    def table(seed):
        flat = torch.randn(n * D * (K - 1) + 1, generator=torch.Generator().manual_seed(seed)).to(dtype).cuda()
        return flat[off:off + n * D * (K - 1)].view(n, D, K - 1)

    if off:
        w = torch.cat([w.flatten()[:1], w.flatten()])[1:].view(D, K)
    init = table(5) if form == "continued" else None
    tables = table(6), table(6)
    out = atma_b200.lfm2_conv_packed(proj, w, tables[0], *maps, initial_state=init)
    strided = torch.zeros(total * 3 * D + 1, dtype=dtype, device="cuda")[1:].view(total, 3 * D)      # not on 16 bytes: channel by channel
    strided.copy_(proj)
    want = atma_b200.lfm2_conv_packed(strided, w, tables[1], *maps, initial_state=init)
    assert torch.equal(out, want) and torch.equal(*tables)
