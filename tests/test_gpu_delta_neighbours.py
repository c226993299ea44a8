"""The decoders' delta rule over packed sequences some of which hold infinities or NaN: the others keep their bits."""

import pytest
import torch

from tests.rizurax_util import group
from tests.test_gpu_rizurax import DELTA_SHAPES, _delta_case, _delta_tables, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shape", DELTA_SHAPES[:3])
@pytest.mark.parametrize("lens", [(65, 70), (3, 5, 200, 1, 17), (127, 2, 64, 61), (1500, 1, 33, 2000)])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_others_keep_their_bits(lens, bad, shape, dtype):
    """A chunk holds rows of the next sequence behind a sequence's last ones, with factors of zero."""
    n, T = len(lens), sum(lens)
    z, w, _, _, eps = _delta_case(shape, dtype, T, 3)
    at = [sum(lens[:i]) for i in range(n + 1)]

    def run(z):
        conv, state = _delta_tables(w, n, dtype)
        out = torch.empty(T, w.heads * w.vdim, dtype=dtype, device="cuda")
        ops().delta_prefill(z, w, conv, state, group(list(lens), [0] * n, list(range(n)), [[0]] * n), out, eps)
        return [(out[at[i]:at[i + 1]], state[i], conv[i]) for i in range(n)]

    want = run(z)
    for first in (0, 1):
        y = z.clone()
        for i in range(first, n, 2):
            y[at[i]:at[i + 1]][::2] = bad
        for i, got in enumerate(run(y)):
            if i % 2 != first:
                assert all(torch.equal(a, b) for a, b in zip(got, want[i])), i
