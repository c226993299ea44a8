"""The global block with its projections side by side against the formulas one operation at a time."""

import pytest
import torch

from atma_b200 import block
from tests.conftest import max_rel
from tests.gpu_util import rand

pytestmark = pytest.mark.gpu


def weights(D, H, G, dk, bias, dtype, taps=4):
    w, i = {}, 0
    for name, rows, cols in (("attn.q", 2 * H * dk, D), ("attn.k", G * dk, D), ("attn.v", G * dk, D), ("attn.proj", D, H * dk), ("attn.mu_proj", D, H),
                             ("attn.mem.w_gamma", H, D), ("attn.mem.w_beta", H, D), ("attn.mem.gate", H * dk, D), ("attn.mem.proj", D, H * dk),
                             ("mlp.fc", 8 * D, D), ("mlp.proj", D, 4 * D)):
        i += 1
        w[name + ".weight"] = (rand((rows, cols), i) * cols ** -0.5).to(dtype).cuda()
        if bias:
            w[name + ".bias"] = (rand((rows,), i + 50) * 0.1).to(dtype).cuda()
    for n, c in (("q", H * dk), ("k", G * dk), ("v", G * dk)):
        w[f"attn.canon_{n}.weight"] = (rand((c, 1, taps), ord(n)) * 0.3).to(dtype).cuda()
    for n in ("null_base", "null_slope_raw", "len_gain_raw", "mag_beta_raw"):
        w["attn." + n] = rand((H,), len(n)).cuda()
    w["attn.v_null"] = rand((H, dk), 5).cuda()
    w["norm1.weight"], w["norm2.weight"] = (1 + 0.1 * rand((D,), 6)).to(dtype).cuda(), (1 + 0.1 * rand((D,), 7)).to(dtype).cuda()
    return w


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 3e-2)])      # sums in another order; roundings of 16-bit operands
@pytest.mark.parametrize("B,T,D,H,G,dk,bias,window", [(1, 300, 256, 4, 2, 64, True, None), (3, 65, 512, 4, 1, 128, False, None), (2, 1, 64, 4, 4, 32, True, None),
                                                      (1, 700, 1024, 8, 2, 128, True, 100)])
def test_side_by_side(monkeypatch, B, T, D, H, G, dk, bias, window, dtype, tol):
    w, x = weights(D, H, G, dk, bias, dtype), rand((B, T, D), 9, dtype).cuda()
    S0 = rand((B, H, dk, dk), 10).cuda() * 0.1
    kw = dict(head_dim=dk, num_kv_heads=G, window=window, initial_state=S0, mem_beta_bias=0.3, return_state=True)
    assert block._side_by_side(w, D, H, G, dk)
    got, S = block.global_block_forward(x, w, **kw)
    assert got.shape == x.shape and got.dtype == dtype
    monkeypatch.setattr(block, "_side_by_side", lambda *a: False)
    want, Sw = block.global_block_forward(x, w, **kw)
    assert max_rel(got, want) < tol and max_rel(S, Sw) < tol


def test_forms_that_go_one_by_one():
    w = weights(64, 2, 1, 32, True, torch.float32)
    assert not block._side_by_side(w, 64, 2, 1, 32)                           # rows that are not multiples of eight values
    w = weights(64, 4, 1, 32, True, torch.float32)
    del w["attn.mem.proj.weight"]
    x = rand((1, 20, 64), 9).cuda()
    assert not block._side_by_side(w, 64, 4, 1, 32) and block.global_block_forward(x, w, head_dim=32, num_kv_heads=1).shape == x.shape


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.bfloat16, 3e-2)])      # as above
@pytest.mark.parametrize("what", ["eps", "head biases", "row biases", "biases of one value", "taps"])
def test_arguments_of_every_kind(monkeypatch, what, dtype, tol):
    """No epsilon, biases of the memory's gates as tensors, convolutions of different lengths: as one operation at a time takes them."""
    B, T, D, H, G, dk = 2, 70, 256, 4, 2, 64
    w, x = weights(D, H, G, dk, True, dtype), rand((B, T, D), 9, dtype).cuda() * (1e-3 if what == "eps" else 1)
    kw = dict(head_dim=dk, num_kv_heads=G, return_state=True)
    if what == "eps":
        kw["eps"] = None
    elif what == "taps":
        w["attn.canon_k.weight"] = w["attn.canon_k.weight"][..., 1:].contiguous()
    else:
        shape = {"head biases": (H,), "row biases": (B, T, H), "biases of one value": (1,)}[what]
        kw.update(mem_gamma_bias=rand(shape, 3).cuda() + 3, mem_beta_bias=rand(shape, 4).cuda())
    assert block._side_by_side(w, D, H, G, dk) == (what != "taps")
    got, S = block.global_block_forward(x, w, **kw)
    monkeypatch.setattr(block, "_side_by_side", lambda *a: False)
    want, Sw = block.global_block_forward(x, w, **kw)
    assert max_rel(got, want) < tol and max_rel(S, Sw) < tol
