"""16-bit prompt attention whose last key tile holds infinities or NaN behind the sequence's end - the next packed sequence's rows, or what
a cache page held before: the sequence keeps its bits."""

import pytest
import torch

import atma_b200
from atma_b200 import decoder_ops
from atma_b200.layer import PackedMaps
from tests.gpu_util import polar_params, rand
from tests.rizurax_util import group

pytestmark = pytest.mark.gpu
BAD = [float("nan"), float("inf")]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("H,Hkv", [(8, 2), (4, 4), (3, 1)])
@pytest.mark.parametrize("lens", [(300, 77, 200), (1, 1, 130), (128, 5, 256, 3), (127, 129)])
@pytest.mark.parametrize("window", [None, 50])
@pytest.mark.parametrize("bad", BAD)
def test_packed_polar(lens, H, Hkv, window, bad, dtype):
    n, T = len(lens), sum(lens)
    at = [sum(lens[:i]) for i in range(n + 1)]
    x = [rand((T, h, 128), i, dtype).cuda() for i, h in enumerate((H, Hkv, Hkv))]
    p, m = polar_params(H, 128)[1], PackedMaps(lens, range(n), "cuda")
    run = lambda x: atma_b200.polar_attention_packed_fwd(*x, m.tile_seq_starts, m.tile_q_starts, m.tile_seq_lens, window=window, **p)     # noqa: E731
    want = run(x)
    for first in (0, 1):
        y = [t.clone() for t in x]
        for i in range(first, n, 2):
            for t in y:
                t[at[i]:at[i + 1]] = bad
        got = run(y)
        for i in range(1 - first, n, 2):
            assert all(torch.equal(g[at[i]:at[i + 1]], w[at[i]:at[i + 1]]) for g, w in zip(got, want)), i
    assert atma_b200.device_status() == 0


@pytest.mark.parametrize("H,G,maps,dim,vdim", [(4, 2, 1, 128, 128), (3, 3, 1, 128, 128), (4, 2, 2, 64, 128), (4, 4, 1, 64, 64)])
@pytest.mark.parametrize("rows,start", [(1, 0), (200, 0), (127, 300), (256, 128), (130, 1)])
@pytest.mark.parametrize("window,keep", [(None, 0), (60, 4)])
@pytest.mark.parametrize("bad", BAD)
def test_pages_with_an_earlier_content(rows, start, window, keep, bad, H, G, maps, dim, vdim):
    n = rows + start
    pages = -(-n // 256)
    q, kc, vc = rand((rows, H, maps, dim), 1, torch.bfloat16).cuda(), rand((pages, 256, G, maps * dim), 2, torch.bfloat16).cuda(), rand((pages, 256, G, vdim), 3, torch.bfloat16).cuda()
    gate = rand((rows, H * vdim), 4, torch.bfloat16).cuda()
    kw = dict(scale=dim ** -0.5, lam=0.3, out_scale=0.7, eps=1e-6, window=window, keep_first=keep, sink=0.5, gate=gate)
    g = group([rows], [start], [0], [list(range(pages))])
    run = lambda k, v: decoder_ops.softmax_prefill(q, k, v, g, torch.zeros(rows, H * vdim, dtype=torch.bfloat16, device="cuda"), **kw)     # noqa: E731
    want = run(kc, vc)
    for c in (kc, vc):
        c.view(-1, *c.shape[2:])[n:] = bad
    assert torch.equal(run(kc, vc), want)
