"""One ATMA global block forward on the GPU, composed from this package's kernels.

Host-side mirror of the reference's ``Block.forward`` with a Polar attention core and the
gated-delta memory branch (model/reference.py:127-195,230-233; model/blocks.py:463-490;
model/layers.py:19-31): pre-norm RMSNorm, q/k/v projections, per-head RMSNorm of q and k,
the three Canon depthwise convs (residual form), Polar attention, the additive memory channel,
then the squared-ReLU gated MLP.  Every mixing step goes through the C ABI:

    norms, residual    -> add_rms_norm
    projections        -> one product of the weights side by side (``linear_f32`` for fp32 rows in numbers, else the library)
    q, k, v            -> qkv_prep_prefill (head norms and Canon convs)
    Polar core         -> polar_attention_fwd (un-expanded KV heads, (B,T,H,dk) storage viewed as (B,H,T,dk))
    memory scan        -> chunk_gated_delta_rule (in-kernel L2 norm, [K,V] fp32 state)
    gates              -> sigmoid_gate_mul, rms_sigmoid_gate, squared_relu_gate
    output             -> one product: W_o, mem.proj and W_mu side by side, their inputs likewise

With a launch per operation of the formulas (55 of them; blocks without a memory or with other head sizes still run so) the host
was as long as the kernels, and the input rows were split into their terms six times: 1 x 2048 rows of 1024 in fp32 1137 us, 848 so.

It takes the reference block's ``state_dict`` as is, so a parity test can load the oracle's
weights and compare outputs.
"""

import torch
import torch.nn.functional as F

from .causal_conv1d import causal_conv1d_fn
from .gated_delta import chunk_gated_delta_rule
from .inference_ops import add_rms_norm, linear, qkv_prep_prefill, rms_sigmoid_gate, sigmoid_gate_mul, squared_relu_gate
from .polar import polar_attention_fwd


def _linear(x, sd, name):
    w = sd[name + ".weight"].to(x.dtype)
    b = sd.get(name + ".bias")
    return linear(x, w, None if b is None else b.to(x.dtype))


def _canon(x_btc, weight):
    """x + depthwise causal conv(x); x (B, T, C), weight (C, 1, K) as nn.Conv1d stores it."""
    out = causal_conv1d_fn(x_btc.transpose(1, 2), weight.squeeze(1).to(x_btc.dtype))
    return x_btc + out.transpose(1, 2)


IN = ("attn.q", "attn.k", "attn.v", "attn.mem.gate", "attn.mem.w_gamma", "attn.mem.w_beta")
OUT = ("attn.proj", "attn.mem.proj", "attn.mu_proj")


def _side_by_side(sd, D, H, Hkv, dk):
    """Whether the projections can go as one product and their parts be read in place."""
    if any(n + ".weight" not in sd for n in IN + OUT) or len({n + ".bias" in sd for n in IN}) != 1:
        return False
    taps = {sd[f"attn.canon_{i}.weight"].shape[-1] for i in "qkv"}
    return dk % 8 == 0 and dk <= 128 and D <= 4096 and (2 * H) % 8 == 0 and len(taps) == 1 and 2 <= min(taps) <= 4


def _mixed(x, h, sd, H, Hkv, dk, window, mem_gamma_bias, mem_beta_bias, initial_state):
    """The mixing of rows h (B*T, D), projections side by side: (its output (B*T, D), the memory's final state)."""
    B, T, D = x.shape
    n, Hd, dt, dev = B * T, H * dk, x.dtype, x.device
    both = lambda names, kind, dim: torch.cat([sd[i + kind].to(dt) for i in names], dim)  # noqa: E731
    z = linear(h, both(IN, ".weight", 0), both(IN, ".bias", 0) if "attn.q.bias" in sd else None)
    q_gate, k, v, mem_gate, g, beta = z.split([2 * Hd, Hkv * dk, Hkv * dk, Hd, H, H], 1)
    q_gate = q_gate.view(n, H, 2 * dk)
    start = torch.zeros(n, dtype=torch.int32, device=dev) if B == 1 else torch.arange(0, n, T, dtype=torch.int32, device=dev).repeat_interleave(T)
    taps = [sd[f"attn.canon_{i}.weight"].squeeze(1) for i in "qkv"]
    q, k, v = qkv_prep_prefill(q_gate, k.reshape(n, Hkv, dk), v.reshape(n, Hkv, dk), *taps, None, None, None, start, start + T, start)
    q, k, v = (t.view(B, T, -1, dk) for t in (q, k, v))
    n_keys = torch.arange(1, T + 1, device=dev, dtype=torch.float32)
    c, mag = polar_attention_fwd(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), n_keys, v_null=sd["attn.v_null"],
                                 null_base=sd["attn.null_base"], null_slope_raw=sd["attn.null_slope_raw"],
                                 len_gain_raw=sd["attn.len_gain_raw"], mag_beta_raw=sd["attn.mag_beta_raw"], window=window)
    c = c[0].transpose(0, 1) if B == 1 else c.transpose(1, 2).reshape(n, H, dk)
    logits = [t.float().view(B, T, H) for t in (g, beta)]
    g, beta = (t if isinstance(bias, (int, float)) and bias == 0 else t + bias for t, bias in zip(logits, (mem_gamma_bias, mem_beta_bias)))
    r, S = chunk_gated_delta_rule(q=q, k=k, v=v, g=F.logsigmoid(g), beta=torch.sigmoid(beta), scale=1.0,
                                  initial_state=initial_state, output_final_state=True, use_qk_l2norm_in_kernel=True)
    act = torch.cat([sigmoid_gate_mul(c, q_gate[..., dk:]).view(n, Hd), rms_sigmoid_gate(r.view(n, H, dk), mem_gate),
                     mag.transpose(1, 2).reshape(n, H)], 1)
    biases = [sd[i + ".bias"].to(dt) for i in OUT if i + ".bias" in sd]
    return linear(act, both(OUT, ".weight", 1), sum(biases[1:], biases[0]) if biases else None), S


@torch.no_grad()
def global_block_forward(x, sd, *, head_dim, num_kv_heads, window=None, mem_chunk=64, mem_gamma_bias=3.9,
                         mem_beta_bias=0.0, eps=1e-6, initial_state=None, return_state=False):
    """x (B, T, D) on the GPU; ``sd`` the reference block's state_dict (tensors on the same
    device).  Returns the block output (B, T, D) (and the memory's final [K,V] state)."""
    if mem_chunk != 64:
        raise ValueError("the scan kernels use 64-token chunks (the result does not depend on the chunk size)")
    B, T, D = x.shape
    dk = head_dim
    H = sd["attn.null_base"].shape[0]
    Hkv = num_kv_heads
    if B * T > 0 and _side_by_side(sd, D, H, Hkv, dk):
        rows = x.reshape(B * T, D)
        eps = torch.finfo(torch.float32).eps if eps is None else eps          # as F.rms_norm's None, 16-bit inputs included
        _, h = add_rms_norm(rows, None, sd["norm1.weight"], eps)
        out, S = _mixed(x, h, sd, H, Hkv, dk, window, mem_gamma_bias, mem_beta_bias, initial_state)
        rows, h = add_rms_norm(rows, out, sd["norm2.weight"], eps)
        fc = _linear(h, sd, "mlp.fc")
        half = fc.shape[-1] // 2
        x = (rows + _linear(squared_relu_gate(fc[:, :half], fc[:, half:]), sd, "mlp.proj")).view(B, T, D)
        return (x, S) if return_state else x
    h = F.rms_norm(x, (D,), weight=sd["norm1.weight"].to(x.dtype), eps=eps)

    q_gate = _linear(h, sd, "attn.q").view(B, T, H, 2 * dk)
    q, gate = q_gate[..., :dk], q_gate[..., dk:]
    k = _linear(h, sd, "attn.k").view(B, T, Hkv, dk)
    v = _linear(h, sd, "attn.v").view(B, T, Hkv, dk)
    q = F.rms_norm(q, (dk,))
    k = F.rms_norm(k, (dk,))
    q = _canon(q.reshape(B, T, H * dk), sd["attn.canon_q.weight"]).view(B, T, H, dk)
    k = _canon(k.reshape(B, T, Hkv * dk), sd["attn.canon_k.weight"]).view(B, T, Hkv, dk)
    v = _canon(v.reshape(B, T, Hkv * dk), sd["attn.canon_v.weight"]).view(B, T, Hkv, dk)

    n_keys = torch.arange(1, T + 1, device=x.device, dtype=torch.float32)
    c, mag = polar_attention_fwd(q.transpose(1, 2), k.transpose(1, 2), v.transpose(1, 2), n_keys,
                                 v_null=sd["attn.v_null"], null_base=sd["attn.null_base"],
                                 null_slope_raw=sd["attn.null_slope_raw"], len_gain_raw=sd["attn.len_gain_raw"],
                                 mag_beta_raw=sd["attn.mag_beta_raw"], window=window)
    c_flat = c.transpose(1, 2).reshape(B, T, H * dk)
    out = _linear(c_flat * torch.sigmoid(gate.reshape(B, T, H * dk)), sd, "attn.proj")
    out = out + _linear(mag.transpose(1, 2), sd, "attn.mu_proj")

    S = None
    if "attn.mem.proj.weight" in sd:
        g_logit = _linear(h, sd, "attn.mem.w_gamma").float() + mem_gamma_bias
        b_logit = _linear(h, sd, "attn.mem.w_beta").float() + mem_beta_bias
        r, S = chunk_gated_delta_rule(q=q.contiguous(), k=k.contiguous(), v=v.contiguous(), g=F.logsigmoid(g_logit),
                                      beta=torch.sigmoid(b_logit), scale=1.0, initial_state=initial_state,
                                      output_final_state=True, use_qk_l2norm_in_kernel=True)
        r = F.rms_norm(r.float(), (dk,)).reshape(B, T, H * dk).to(x.dtype)
        out = out + _linear(r * torch.sigmoid(_linear(h, sd, "attn.mem.gate")), sd, "attn.mem.proj")
    x = x + out

    h2 = F.rms_norm(x, (D,), weight=sd["norm2.weight"].to(x.dtype), eps=eps)
    fc = _linear(h2, sd, "mlp.fc")
    half = fc.shape[-1] // 2
    act = squared_relu_gate(fc[..., :half].reshape(B * T, half), fc[..., half:].reshape(B * T, half)).view(B, T, half)
    x = x + _linear(act, sd, "mlp.proj")
    return (x, S) if return_state else x
