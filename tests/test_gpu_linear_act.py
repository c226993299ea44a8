"""``linear_act`` against 64 bits and against a product with the activation behind it, at the edges of its tiles (256 rows, 128 or
256 results, 64 columns) and of the persistent schedule."""

import pytest
import torch
import torch.nn.functional as F

from atma_b200 import device_status
from atma_b200.inference_ops import linear_act, linear_act_supported

pytestmark = pytest.mark.gpu


def act(y, form):
    """The activation of 64-bit products, rounded nowhere."""
    if form == "plain_squared_relu":
        return y.relu().square()
    first, second = y.chunk(2, -1)
    return second * first.relu().square() if form == "squared_relu" else F.gelu(first, approximate="tanh") * second


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("form", ["squared_relu", "gelu_tanh", "plain_squared_relu"])
@pytest.mark.parametrize("M,N,K,bias,strided", [(256, 256, 64, True, False), (1, 16, 8, False, True), (257, 272, 72, True, True), (127, 528, 200, False, False),
                                                (3001, 2064, 1032, True, True), (511, 8192, 1024, True, False), (20000, 1040, 320, True, True)])
def test_against_64_bits(M, N, K, bias, strided, form, dtype):
    torch.manual_seed(M + N + K)
    width = N if form == "plain_squared_relu" else N // 2
    x = torch.randn(M, K + 8, device="cuda").to(dtype)[:, :K] if strided else torch.randn(M, K, device="cuda").to(dtype)
    w = (torch.randn(N, K, device="cuda") * K ** -0.5).to(dtype)
    b = (0.5 * torch.randn(N, device="cuda")).to(dtype) if bias else None
    room = torch.full((M, width + 24), 7.0, device="cuda", dtype=dtype)
    out = room[:, 8:8 + width] if strided else None
    assert linear_act_supported(x, w, form, b, out)
    got = linear_act(x, w, form, b, out)
    assert device_status() == 0
    y = x.double() @ w.double().T + (0 if b is None else b.double())
    want = act(y, form)
    # half a unit in the last place, u, for each product (twice where relu squares it; gelu's slope is below 1.13), the square and
    # the result: 5 u of |first|^2 |second|, |first| |second| or |y|^2 at most.  fp32 sums are off by less than 2^-20 of a row's size.
    u = 2.0 ** (-8 if dtype == torch.bfloat16 else -11)
    size = y.square() if form == "plain_squared_relu" else y.abs().chunk(2, -1)[0] ** (2 if form == "squared_relu" else 1) * y.abs().chunk(2, -1)[1]
    assert ((got.double() - want).abs() <= 5 * u * size + 2.0 ** -20 * size.max() + 2.0 ** -24).all()
    if strided:
        assert (room[:, :8] == 7).all() and (room[:, 8 + width:] == 7).all()


def test_rows_keep_to_themselves():
    """An infinity or a NaN reaches its own row (of x) or feature (of w) only."""
    torch.manual_seed(0)
    x, w = torch.randn(700, 128, device="cuda").bfloat16(), (torch.randn(608, 128, device="cuda") / 11).bfloat16()
    clean = linear_act(x, w, "gelu_tanh")
    x[300, 5], w[10, 7], w[333, 3] = float("nan"), float("inf"), float("nan")
    got = linear_act(x, w, "gelu_tanh")
    rows, cols = torch.arange(700, device="cuda") != 300, ~torch.isin(torch.arange(304, device="cuda"), torch.tensor([10, 29], device="cuda"))
    assert torch.equal(got[rows][:, cols], clean[rows][:, cols]) and got[300].isnan().all()
    assert got[rows][:, 29].isnan().all()


def test_capture_and_streams():
    torch.manual_seed(1)
    x, w = torch.randn(900, 512, device="cuda").half(), (torch.randn(1024, 512, device="cuda") / 22).half()
    want = linear_act(x, w, "squared_relu")
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        got = linear_act(x, w, "squared_relu")
    g.replay()
    sides = [torch.cuda.Stream() for _ in range(3)]
    outs = []
    for s in sides:
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            outs.append(linear_act(x, w, "squared_relu"))
    torch.cuda.synchronize()
    assert torch.equal(got, want) and all(torch.equal(o, want) for o in outs)


def test_what_it_does_not_take():
    x, w = torch.zeros(600, 64, device="cuda", dtype=torch.bfloat16), torch.zeros(64, 64, device="cuda", dtype=torch.bfloat16)
    assert linear_act_supported(x, w, True)
    for bad in ((x.float(), w.float()), (x[:, 4:60], w[:, :56].contiguous()), (x[:, :60], w[:, :60].contiguous()), (x.t(), w), (x, w[:40]), (x.cpu(), w.cpu()),
                (x.clone().requires_grad_(), w)):
        assert not linear_act_supported(*bad, True)
