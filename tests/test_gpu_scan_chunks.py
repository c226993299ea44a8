"""The tensor-core scan where its chunks, halves and rings begin and end, and the forms of its two stages."""

import ctypes

import pytest
import torch
import torch.nn.functional as F

import atma_b200
import oracle
from atma_b200 import _lib
from atma_b200.gated_delta import scan_factors, scan_recur
from conftest import max_rel

pytestmark = pytest.mark.gpu


def inputs(B, T, H, Hkv, dtype, seed, spread=0.0):
    """``spread``: rows of k and q are scaled by powers of two up to 2^+-spread, which the normalisation takes out again."""
    g = torch.Generator().manual_seed(seed)
    q, k, v = (torch.randn(B, T, n, 128, generator=g) for n in (H, Hkv, Hkv))
    if spread:
        q, k = (x * 2.0 ** torch.empty(B, T, x.shape[2], 1).uniform_(-spread, spread, generator=g).round() for x in (q, k))
    glog = F.logsigmoid(torch.randn(B, T, H, generator=g) + 2.0)
    beta = torch.sigmoid(torch.randn(B, T, H, generator=g))
    return [x.to(dtype) for x in (q, k, v)] + [glog, beta, torch.randn(B, H, 128, 128, generator=g) * 0.3]


@pytest.mark.parametrize("spread", [0.0, 5.0])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H,Hkv", [(1, 1, 1, 1), (2, 63, 2, 1), (1, 64, 4, 2), (3, 65, 2, 2), (1, 127, 8, 2), (1, 193, 4, 1), (2, 449, 3, 3)])
def test_chunk_edges(B, T, H, Hkv, dtype, spread):
    q, k, v, glog, beta, S0 = inputs(B, T, H, Hkv, dtype, T + H, spread)
    rep = lambda x: x.repeat_interleave(H // Hkv, 2)  # noqa: E731
    o_ref, S_ref = oracle.chunk_gated_delta_rule_oracle(q, rep(k), rep(v), glog, beta, initial_state=S0)
    o, S = atma_b200.chunk_gated_delta_rule(q=q.cuda(), k=k.cuda(), v=v.cuda(), g=glog.cuda(), beta=beta.cuda(), scale=1.0,
                                            initial_state=S0.cuda(), output_final_state=True, use_qk_l2norm_in_kernel=True)
    assert max_rel(o, o_ref) < 2e-2 and max_rel(S, S_ref) < 2e-2          # 16-bit operands, as for the other sizes of this scan


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("T", [40, 64, 200])
def test_key_rows_without_a_length(T, dtype):
    """1 / |k| of rows of zeros and of rows of the type's smallest numbers is beyond fp16; the normalisation makes nothing of the
    ones and unit vectors of the others."""
    q, k, v, glog, beta, S0 = inputs(2, T, 2, 1, dtype, T)
    k[:, 3::7] = 0
    k[:, 5::11] = torch.randn(k[:, 5::11].shape, generator=torch.Generator().manual_seed(1)).sign().to(dtype) * 2.0 ** -24
    k[:, 8::13] *= 1000
    v[:, 1::9] *= 2000                                                    # U of the size of what fp16 holds
    o_ref, S_ref = oracle.chunk_gated_delta_rule_oracle(q, k, v, glog, beta, initial_state=S0)
    o, S = atma_b200.chunk_gated_delta_rule(q=q.cuda(), k=k.cuda(), v=v.cuda(), g=glog.cuda(), beta=beta.cuda(), scale=1.0,
                                            initial_state=S0.cuda(), output_final_state=True, use_qk_l2norm_in_kernel=True)
    assert max_rel(o, o_ref) < 2e-2 and max_rel(S, S_ref) < 2e-2          # as above


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), -float("inf")])
@pytest.mark.parametrize("lengths", [(65, 70), (1, 1, 200), (127, 5), (64, 64), (17, 300, 30), (193, 2, 61)])
def test_a_sequence_keeps_its_bits_whatever_its_neighbours_hold(lengths, bad, dtype):
    """A chunk holds rows of the next sequence behind a sequence's last ones.  Every other sequence's rows go bad, the others' outputs
    and states stay as they were; packed, and as rows of a batch."""
    n, total, H, Hkv = len(lengths), sum(lengths), 3, 1
    at = [sum(lengths[:i]) for i in range(n + 1)]

    def packed(x, S0):
        table = S0.clone()
        o = atma_b200.packed_gated_delta_prefill(*(t[0].cuda() for t in x), torch.tensor(at), table, torch.arange(n).cuda())
        return [(o[at[i]:at[i + 1]], table[i]) for i in range(n)]

    def dense(x, S0):
        o, S = atma_b200.chunk_gated_delta_rule(**dict(zip(("q", "k", "v", "g", "beta"), (t.cuda() for t in x))), scale=1.0, initial_state=S0,
                                                output_final_state=True, use_qk_l2norm_in_kernel=True)
        return list(zip(o, S))

    x = inputs(1, total, H, Hkv, dtype, total)[:5]
    S0 = torch.randn(n, H, 128, 128, generator=torch.Generator().manual_seed(3)).cuda() * 0.3
    cases = [(packed, x, lambda t, i: t[:, at[i]:at[i + 1]], S0)]
    cases += [(dense, inputs(3, T, H, Hkv, dtype, T)[:5], lambda t, i: t[i:i + 1], S0[:1].expand(3, -1, -1, -1)) for T in set(lengths)]
    for call, x, part, S in cases:
        want = call(x, S)
        for first in (0, 1):
            y = [t.clone() for t in x]
            for i in range(first, len(want), 2):
                for t in y[:3]:
                    part(t, i)[:, ::2] = bad
            for i, (g, w) in enumerate(zip(call(y, S), want)):
                if i % 2 != first:
                    assert torch.equal(g[0], w[0]) and torch.equal(g[1], w[1])
    assert atma_b200.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H,Hkv", [(2, 320, 4, 2), (1, 1000, 2, 1)])
def test_two_calls_equal_one(B, T, H, Hkv, dtype):
    """scan_factors keeps the rows that scan_recur needs, so the inputs may change in between."""
    q, k, v, glog, beta, S0 = (x.cuda() for x in inputs(B, T, H, Hkv, dtype, 5))
    o, S = atma_b200.chunk_gated_delta_rule(q=q, k=k, v=v, g=glog, beta=beta, scale=1.0, initial_state=S0, output_final_state=True,
                                            use_qk_l2norm_in_kernel=True, segments=1)
    f = scan_factors(q, k, v, glog, beta)
    for x in (q, k, v):
        x.zero_()
    o2, S2 = scan_recur(f, list(range(B)), initial_state=S0)
    assert torch.equal(o, o2) and torch.equal(S, S2)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("B,T,H,Hkv", [(2, 320, 4, 2), (1, 1000, 2, 1)])
def test_two_calls_over_the_rows_themselves(B, T, H, Hkv, dtype):
    """Without a copy the recurrences give what they give with one: outputs, states, and states with v = 0."""
    q, k, v, glog, beta, S0 = (x.cuda() for x in inputs(B, T, H, Hkv, dtype, 6))
    fs = [scan_factors(q, k, v, glog, beta, keep_rows=keep) for keep in (True, False)]
    for want_output in (True, False):
        for zero in (None, [True] * B):
            (o, S), (o2, S2) = (scan_recur(f, list(range(B)), S0, zero, want_output) for f in fs)
            assert torch.equal(S, S2) and (not want_output or torch.equal(o, o2))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_outputs_two_bytes_off(dtype):
    """o may start at any 16-bit value: from an odd one its values are stored one by one."""
    B, T, H, Hkv = 2, 150, 3, 1
    q, k, v, glog, beta, S0 = (x.cuda() for x in inputs(B, T, H, Hkv, dtype, 9))
    lib = _lib.load()
    scratch = torch.empty(lib.atma_gated_delta_scan_scratch_bytes(B, T, H, 128, 128), dtype=torch.uint8, device="cuda")
    out = []
    for off in (0, 1):
        buf = torch.full((B * T * H * 128 + 2,), 7.0, dtype=dtype, device="cuda")
        _lib.check(lib.atma_gated_delta_scan(_lib.ptr(q), _lib.ptr(k), _lib.ptr(v), _lib.dtype_code(q), _lib.ptr(glog), _lib.ptr(beta),
                                             _lib.ptr(S0), ctypes.c_void_p(buf.data_ptr() + 2 * off), None, _lib.ptr(scratch), B, T, H, Hkv,
                                             128, 128, 1, 1.0, _lib.stream_ptr()))
        assert (buf[:off] == 7).all() and (buf[off + B * T * H * 128:] == 7).all()
        out.append(buf[off:off + B * T * H * 128])
    assert torch.equal(*out)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("place", ["q", "k", "v", "behind k"])
@pytest.mark.parametrize("T,segments", [(150, 1), (4096, 4)])
def test_outputs_in_the_place_of_inputs(T, segments, place, dtype):
    """o over q, k or v, or over the end of one and what follows: the rows are read before o is written, in both passes over segments
    and in packed batches."""
    B, H = 2, 2
    x = [t.cuda() for t in inputs(B, T, H, H, dtype, 11)]
    lib, n = _lib.load(), B * T * H * 128
    scratch = torch.empty(max(lib.atma_gated_delta_scan_scratch_bytes(B, T, H, 128, 128),
                              lib.atma_gated_delta_scan_varlen_scratch_bytes(B * T, 2, H, 128, 128)), dtype=torch.uint8, device="cuda")
    cu = torch.tensor([0, T - 3, B * T], dtype=torch.int32, device="cuda")
    for packed in (False, True):
        out = []
        for over in (False, True):
            buf = torch.zeros(4 * n, dtype=dtype, device="cuda")
            for i in range(3):
                buf[i * n:(i + 1) * n] = x[i].flatten()
            q, k, v = (buf.data_ptr() + 2 * i * n for i in range(3))
            at = (3 * n if not over else n + n // 2 + 128 if place == "behind k" else "qkv".index(place) * n)
            o = ctypes.c_void_p(buf.data_ptr() + 2 * at)
            if packed:
                _lib.check(lib.atma_gated_delta_scan_varlen(q, k, v, _lib.dtype_code(x[0]), _lib.ptr(x[3]), _lib.ptr(x[4]), _lib.ptr(cu), 2, B * T,
                                                            _lib.ptr(x[5]), None, None, 0, None, None, o, _lib.ptr(scratch), H, H, 128, 128, 1, 1.0,
                                                            _lib.stream_ptr()))
            else:
                _lib.check(lib.atma_gated_delta_scan_segmented(q, k, v, _lib.dtype_code(x[0]), _lib.ptr(x[3]), _lib.ptr(x[4]), _lib.ptr(x[5]), o, None,
                                                               _lib.ptr(scratch), B, T, H, H, 128, 128, 1, 1.0, segments, _lib.stream_ptr()))
            out.append(buf[at:at + n].clone())
        assert torch.equal(*out)
