"""Host: which calls ``linear_act_if_faster`` takes from a library product with the activation behind it.  CPU tensors pass for CUDA
ones here and the kernel library is a stand-in that records calls, so nothing is launched."""

import types

import pytest
import torch

from atma_b200 import _lib, decoder_ops, inference_ops as io

M, K, N = 1024, 512, 8192


@pytest.fixture
def calls(monkeypatch):
    seen = []
    lib = types.SimpleNamespace(atma_linear_act=lambda *args: seen.append(args) or 0, atma_gelu_gate=lambda *args: seen.append("gate") or 0,
                                atma_bias_squared_relu=lambda *args: seen.append("relu") or 0)
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: None)            # the index of a CPU tensor's device
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(_lib, "load_decoder", lambda: lib)
    monkeypatch.setattr(_lib, "stream_ptr", lambda: None)
    return seen


def product(rows=M, k=K, n=N, dtype=torch.bfloat16):
    return torch.zeros(rows, k, dtype=dtype), torch.zeros(n, k, dtype=dtype), torch.zeros(n, dtype=dtype)


def served(calls, x, w, b=None, gated=True, out=None):
    before = len(calls)
    y = io.linear_act_if_faster(x, w, gated, b, out)
    assert (y is not None) == (len(calls) > before)
    return y is not None


@pytest.mark.parametrize("rows,k,n,yes", [(1024, 512, 8192, True), (799, 512, 8192, False), (1600, 256, 4096, True), (1600, 248, 4096, False), (614, 256, 16384, False),
                                          (615, 256, 16384, True), (820, 256, 8000, True), (2048, 260, 8192, False), (4096, 256, 8200, False)])
def test_sizes(calls, rows, k, n, yes):
    x, w, b = product(rows, k, n)
    assert served(calls, x, w, b) is yes and served(calls, x, w) is yes


def test_forms(calls):
    x, w, b = product()
    wide = torch.zeros(M, K + 16, dtype=torch.bfloat16)
    room = torch.zeros(M, N, dtype=torch.bfloat16)
    assert served(calls, x, w, b) and served(calls, wide[:, 8:8 + K], w, b) and served(calls, x, w, b, out=room[:, 64:64 + N // 2])
    assert served(calls, x, w, b, gated="plain_squared_relu") and served(calls, x, w, torch.zeros(N + 1, dtype=torch.bfloat16)[1:])
    assert all(served(calls, *product(dtype=torch.float16), gated=g) for g in ("squared_relu", "gelu_tanh", "plain_squared_relu"))


@pytest.mark.parametrize("bad", ["offset", "stride", "columns", "transposed", "weight", "dtype", "bias", "bias stride", "out", "out offset", "out on x", "grad", "subclass"])
def test_what_is_left_to_the_general_path(calls, bad):
    x, w, b = product()
    out, z = None, torch.zeros
    bf16 = dict(dtype=torch.bfloat16)
    if bad == "offset":
        x = z(M, K + 8, **bf16)[:, 4:4 + K]
    elif bad == "stride":
        x = z(M, K + 4, **bf16)[:, :K]
    elif bad == "columns":
        x = z(M, 2 * K, **bf16)[:, ::2]
    elif bad == "transposed":
        x = z(K, M, **bf16).t()
    elif bad == "weight":
        w = z(K, N, **bf16).t()
    elif bad == "dtype":
        x = x.float()
    elif bad == "bias":
        b = z(N, 1, **bf16)
    elif bad == "bias stride":
        b = z(2 * N, **bf16)[::2]
    elif bad == "out":
        out = z(M, N, **bf16)
    elif bad == "out offset":
        out = z(M, N, **bf16)[:, 4:4 + N // 2]
    elif bad == "out on x":
        room = z(M, K + N // 2, **bf16)
        x, out = room[:, :K], room[:, K:]
    elif bad == "grad":
        w.requires_grad_()
    elif bad == "subclass":
        x = x.as_subclass(type("Marked", (torch.Tensor,), {}))
    assert not served(calls, x, w, b, out=out) and not calls


def test_what_surrounds_the_call(calls):
    x, w, b = product()
    with pytest.MonkeyPatch.context() as m:
        m.setattr(torch, "is_autocast_enabled", lambda: True)
        assert not served(calls, x, w, b)
    seen = []
    torch.func.vmap(lambda v: (seen.append(io.linear_act_if_faster(v, w, True, b)), v)[1])(x[None])
    assert seen == [None]
    with torch.no_grad():
        assert served(calls, x, w.requires_grad_(), b)


def test_half_precision_of_the_decoders(calls):
    """Their activations are bf16: an fp16 product of many rows goes where it went, and is refused there."""
    x, w, b = product(dtype=torch.float16)
    decoder_ops.squared_relu_linear(x, w, b)
    decoder_ops.gelu_gated_linear(x, w, torch.zeros(M, N // 2, dtype=torch.float16))
    assert calls == ["relu", "gate"]


@pytest.mark.parametrize("rows,k,n,yes", [(8399, 5568, 1792, False), (14080, 7808, 2432, False), (1635, 7744, 9472, False), (1281, 3200, 5568, False),
                                          (24320, 5376, 4160, True), (5628, 5120, 3264, True), (6955, 3392, 4480, True), (2816, 256, 3776, True),
                                          (12000, 1024, 8192, True), (3000, 1024, 8192, True), (4096, 2048, 16384, True)])
def test_sizes_whose_last_turn_is_nearly_empty(rows, k, n, yes):
    """Measured on both sides of the line."""
    assert io._linear_act_pays(rows, n, k) is yes
