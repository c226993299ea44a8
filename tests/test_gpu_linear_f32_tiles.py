"""The fp32 product where a CTA takes several tiles in turn: figures of columns that differ from tile to tile, last tiles of rows that
are nearly empty, results that are summed again between two tiles' products."""

import pytest
import torch

import atma_b200
from atma_b200.inference_ops import linear_f32
from tests.test_gpu_conv_elementwise import _product_bound

pytestmark = pytest.mark.gpu


# (4628, 128, 2560): 370 tiles of 148 CTAs, of which four have nothing but tiles of 20 rows; with one or two stages of 64 columns a
# tile's products are over before a warp that still writes the tile in front is asked for anything.  The others: one stage, a part
# of one, three stages (odd: buffers change sides from tile to tile), many; three tiles a CTA and more
@pytest.mark.parametrize("M,K,N", [(4628, 128, 2560), (4640, 64, 5120), (4624, 40, 8192), (4624, 192, 8192), (1056, 128, 16384), (4624, 1024, 8192),
                                   (20000, 100, 520)])
@pytest.mark.parametrize("again", [False, True])
def test_tiles_in_turn(M, K, N, again):
    g = torch.Generator(device="cuda").manual_seed(M + K)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")        # noqa: E731
    size = torch.exp2(torch.randint(-30, 31, (N, 1), generator=g, device="cuda").float())
    x, w = rand(M, K), rand(N, K) * size                                  # a column's power of two in another tile's place shows
    b = rand(N) * size[:, 0].flip(0)
    x[torch.rand(M, generator=g, device="cuda") < 0.2] = 0                # those rows are the bias, to the bit
    if again:                                                             # small values decide results of some tiles of rows
        rows = (torch.arange(M, device="cuda") // 128 % 3 == 1) & (torch.arange(M, device="cuda") % 8 == 0)
        x[rows, 1:] *= 2.0 ** -29
        w[::5, 0] = 0
    zero = (x == 0).all(1)
    for _ in range(3):
        y = linear_f32(x, w, b)
        assert torch.equal(y[zero], b.expand(int(zero.sum()), N))
        for r in range(0, M, 2048):
            part = slice(r, r + 2048)
            off = (y[part] - (x[part].double() @ w.double().t() + b)).abs()
            assert (off <= _product_bound(x[part], w) + b.abs() * 2 ** -23).all()
    assert atma_b200.device_status() == 0


@pytest.mark.parametrize("K", [2 ** 15 - 64, 2 ** 15 - 63, 2 ** 15])       # tiles in turn, and from 2^15 on (padded to 64) a CTA per tile
def test_long_sums_that_are_all_taken_again(K):
    """176 tiles; every other tile of rows is summed again from one end to the other, while other warps wait for it."""
    M, N = 2000, 2600
    g = torch.Generator(device="cuda").manual_seed(K)
    x, w = torch.randn(M, K, generator=g, device="cuda"), torch.randn(N, K, generator=g, device="cuda")
    x[(torch.arange(M, device="cuda") // 128) % 2 == 0, 1:] *= 2.0 ** -29
    w[:, 0] = 0
    y = linear_f32(x, w)
    for r in range(0, M, 500):
        part = slice(r, r + 500)
        assert ((y[part] - x[part].double() @ w.double().t()).abs() <= _product_bound(x[part], w)).all()
    assert atma_b200.device_status() == 0
