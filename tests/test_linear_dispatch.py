"""Host: which products ``inference_ops.linear`` takes from the library, and what the entries refuse before a launch.  CPU
tensors pass for CUDA ones here and the kernel library is a stand-in that records calls, so nothing is launched."""

import contextlib
import types

import pytest
import torch
import torch.nn.functional as F

from atma_b200 import _lib, inference_ops as io

M, K, N = 512, 1024, 1024                     # the smallest product that is worth it


@pytest.fixture
def calls(monkeypatch):
    """The calls that would have been launched."""
    seen = []

    def entry(name):
        return lambda *args: seen.append((name, args)) or 0

    lib = types.SimpleNamespace(atma_linear_f32=entry("linear_f32"), atma_linear_f32_scratch_bytes=lambda *a: 16,
                                atma_decode_linear=entry("decode_linear"), atma_decode_linear_k8=entry("decode_linear_k8"))
    monkeypatch.setattr(torch.Tensor, "is_cuda", property(lambda t: True))
    monkeypatch.setattr(torch.cuda, "current_device", lambda: None)            # the index of a CPU tensor's device
    monkeypatch.setattr(_lib, "load", lambda: lib)
    monkeypatch.setattr(_lib, "load_decoder", lambda: lib)
    monkeypatch.setattr(_lib, "stream_ptr", lambda: None)
    return seen


def product(rows=M, k=K, n=N, dtype=torch.float32):
    g = torch.Generator().manual_seed(1)
    return torch.randn(rows, k, generator=g).to(dtype), torch.randn(n, k, generator=g).to(dtype), torch.randn(n, generator=g).to(dtype)


def served(calls, x, w, b=None):
    """Whether the kernel was asked; the library's product has to be right where it was not."""
    before = len(calls)
    y = io.linear(x, w, b)
    asked = len(calls) > before
    if not asked:
        assert torch.equal(y, F.linear(x, w, b))
    return asked


@pytest.mark.parametrize("rows,k,n,yes", [(512, 1024, 1024, True), (511, 1024, 1024, False), (128, 4096, 1024, True), (127, 8192, 1024, False),
                                          (4096, 128, 4096, True), (8192, 127, 4096, False), (4096, 4096, 128, True), (8192, 4096, 127, False),
                                          (1 << 17, 64, 64, False), (16384, 256, 128, False), (16384, 513, 131, True), (256, 8192, 256, True),
                                          (256, 8224, 256, False), (512, 8224, 512, True), (128, 32768, 128, False)])
def test_thresholds(calls, rows, k, n, yes):
    x, w, _ = product(rows, k, n)
    assert served(calls, x, w) is yes


def test_forms_of_x(calls):
    x, w, b = product()
    assert served(calls, x.view(2, M // 2, K), w, b) and served(calls, x.t().contiguous().t(), w, b)
    assert calls[-1][1][1] == K                                                 # transposed rows were made contiguous
    assert served(calls, x.requires_grad_(False), torch.nn.Parameter(w, requires_grad=False), b)
    assert not served(calls, x, w.t().contiguous().t(), b) and not served(calls, x.double(), w.double(), b.double())
    assert not served(calls, torch._neg_view(x), w, b)


@pytest.mark.parametrize("shape", [(), (1,), (1, N), (M, N)])
def test_a_bias_that_is_broadcast_stays_with_the_library(calls, shape):
    x, w, _ = product()
    assert not served(calls, x, w, torch.randn(shape))


@pytest.mark.parametrize("n", [2, N - 1, N + 1])
def test_a_bias_of_the_wrong_length_is_refused(calls, n):
    x, w, _ = product()
    with pytest.raises(RuntimeError):
        io.linear(x, w, torch.zeros(n))
    with pytest.raises(ValueError):
        io.linear_f32(x, w, torch.zeros(n))
    x, w, _ = product(4, 64, 64, torch.bfloat16)
    with pytest.raises(ValueError):
        io.decode_linear(x, w, torch.zeros(63, dtype=x.dtype))
    assert not calls


def test_other_devices_are_refused(calls, monkeypatch):
    x, w, b = product()
    for a in ((x.to("meta"), w, b), (x, w.to("meta"), b), (x, w, b.to("meta"))):
        assert not io.linear_f32_supported(*a)
        with pytest.raises(ValueError):
            io.linear_f32(*a)
    x16, w16, b16 = product(4, 64, 64, torch.bfloat16)
    for a in ((x16, w16.to("meta"), b16), (x16, w16, b16.to("meta"))):
        assert not io.decode_linear_supported(*a[:2], bias=a[2])
        with pytest.raises(ValueError):
            io.decode_linear(*a)
    monkeypatch.setattr(torch.cuda, "current_device", lambda: 1)
    assert not served(calls, x, w, b) and not io.decode_linear_supported(x16, w16)
    assert not calls


def test_what_is_around_the_call(calls):
    x, w, b = product()
    assert served(calls, x, w, b)
    for i in range(3):                                                          # each of the three may ask for its gradient
        t = [x, w, b]
        t[i] = t[i].clone().requires_grad_()
        assert not served(calls, *t)
        with torch.no_grad():
            assert served(calls, *t)
    with torch.autocast("cuda", enabled=False):
        assert served(calls, x, w, b)
    with contextlib.ExitStack() as s:
        s.enter_context(pytest.MonkeyPatch.context()).setattr(torch, "is_autocast_enabled", lambda: True)
        assert not served(calls, x, w, b)
    n = len(calls)
    torch.func.vmap(lambda t: io.linear(t, w, b))(x.view(2, M // 2, K))
    torch.func.jvp(lambda t: io.linear(t, w, b), (x,), (x,))
    with torch.autograd.forward_ad.dual_level():
        io.linear(x, w, b)

    class Counts(torch.utils._python_dispatch.TorchDispatchMode):
        seen = 0

        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            Counts.seen += 1
            return func(*args, **(kwargs or {}))

    with Counts():
        io.linear(x, w, b)
    assert len(calls) == n and Counts.seen > 0
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        assert not served(calls, x, w, b)
    finally:
        torch.backends.cuda.matmul.allow_tf32 = False
    assert served(calls, x, w, b)


def test_small_batches_of_a_model(calls):
    """K a multiple of 8: the weight-streaming kernel with its own entry, unless bias or alignment do not fit."""
    from atma_b200.model import AtmaModel
    m = AtmaModel.__new__(AtmaModel)
    m.small_batch_linear = True
    x, w, b = product(3, 1032, 64, torch.bfloat16)
    m._linear(x, w, b)
    assert [c[0] for c in calls] == ["decode_linear_k8"]
    shifted = torch.empty(64 * 1032 + 1, dtype=torch.bfloat16)[1:].view(64, 1032).copy_(w)
    for a in ((x, w, b[:1]), (x, w, b.sum()), (x, shifted, b)):
        assert torch.equal(m._linear(*a), F.linear(*a))
    assert len(calls) == 1
