"""Gated delta rule (linear attention): the per-token state update of Qwen3-Next style layers.

`GatedDelta` is a whole layer between its projections on CUDA (csrc/kernels/gdn_layer.cu).  `decode_step` advances a batch of per-request states by one token.  On CUDA it is one kernel
(csrc/kernels/gdn.cu: the state crosses HBM once in each direction); elsewhere the same arithmetic in
tensor ops, which is also the reference the GPU test compares against."""
from __future__ import annotations

from dataclasses import dataclass

import torch

from . import _lib
from ._lib import F, I, L, P, check, ptr, stream

_lib.register_signature("xllm_gdn_decode_step", [P, P, P, P, P, P, P, P, I, I, I, I, P])
_lib.register_signature("xllm_gdn_prefill", [P, L, I, P, P, P, P, P, P, I, I, I, I, P])
_lib.register_signature("xllm_gdn_layer", [P] * 9 + [L, L, I, I, I, P, P, L, I] + [P] * 13 + [I] * 9 + [F, F, P])
_lib.register_signature("xllm_gdn_blob_bytes", [I, I, I], L)
_lib.register_signature("xllm_sigmoid_gate", [P, P, L, I, L, I, I, P])


def layer_supported(dtype, device, nk, nv, dk, dv, taps):
    """Whether `GatedDelta` takes layers of these sizes."""
    return (torch.device(device).type == "cuda" and dtype == torch.bfloat16 and nv % nk == 0 and 0 < dk <= 128 and 0 < dv <= 128
            and dk % 4 == 0 and dv % 4 == 0 and 2 <= taps <= 4)


@dataclass
class GatedDelta:
    """Sizes and small weights (bf16) of one layer: convolution, decays and betas, recurrence, gated norm."""
    nk: int
    nv: int
    dk: int
    dv: int
    taps: int
    eps: float
    conv_w: torch.Tensor         # [2 nk dk + nv dv, taps], q | k | v channels
    dt_bias: torch.Tensor        # [nv]
    a_log: torch.Tensor          # [nv]
    norm_w: torch.Tensor         # [dv]

    def __call__(self, rec, tail, slots, cu_q, kv_lens, n_decode, q, k, v, z, b, a, qk_stride, v_stride, z_stride, ba_stride,
                 max_q_len=None):
        """rec [slots, nv, dk, dv] fp32 and tail [slots, channels, taps - 1] are advanced over the rows of the sequences
        (the first `n_decode` have one each, none more than max_q_len, default: all); returns the rows of the output projection [T, nv dv].  q, k, v, z, b, a: views
        that start at head 0's place in the projection rows, rows by stride(0); `qk_stride`: between heads of q and k;
        `v_stride`, `z_stride`, `ba_stride`: between the blocks of the nv / nk value heads that share a key head."""
        T, dev, bf, f32 = q.shape[0], q.device, torch.bfloat16, torch.float32
        nk, nv, dk, dv, n = self.nk, self.nv, self.dk, self.dv, slots.shape[0]
        assert q.stride(0) == k.stride(0) == v.stride(0) and a.stride(0) == b.stride(0)
        for t in (q, k, v, z, b, a, tail, self.conv_w, self.dt_bias, self.a_log, self.norm_w):
            assert t.dtype == bf and t.stride(-1) == 1
        for t in (slots, cu_q, kv_lens):
            assert t.dtype == torch.int32 and t.is_contiguous()
        assert cu_q.shape[0] == n + 1 and kv_lens.shape[0] == n
        assert rec.dtype == f32 and rec.is_contiguous() and rec.shape[1:] == (nv, dk, dv)
        assert tail.is_contiguous() and tail.shape[1:] == (2 * nk * dk + nv * dv, self.taps - 1)
        assert self.conv_w.is_contiguous()
        dkp, dvp = 64 if dk <= 64 else 128, (dv + 7) // 8 * 8
        yq, yk = torch.empty(T, nk, dkp, dtype=bf, device=dev), torch.empty(T, nk, dkp, dtype=bf, device=dev)
        yv, out = torch.empty(T, nv, dvp, dtype=bf, device=dev), torch.empty(T, nv * dv, dtype=bf, device=dev)
        factors = torch.empty(2 * T * (nk + nv), dtype=f32, device=dev)            # decays and betas first: pairs
        fq, fk = factors[2 * T * nv:], factors[T * (2 * nv + nk):]
        o = blobs = None
        if n > n_decode:
            o = torch.empty(T, nv, dv, dtype=f32, device=dev)
            blobs = torch.empty(_lib.load().xllm_gdn_blob_bytes(T, n - n_decode, nv), dtype=torch.uint8, device=dev)
        check(_lib.load().xllm_gdn_layer(
            ptr(rec), ptr(tail), ptr(slots), ptr(cu_q), ptr(kv_lens), ptr(q), ptr(k), ptr(v), ptr(z), q.stride(0), z.stride(0),
            qk_stride, v_stride, z_stride, ptr(b), ptr(a), a.stride(0), ba_stride, ptr(self.conv_w), ptr(self.dt_bias),
            ptr(self.a_log), ptr(self.norm_w), ptr(yq), ptr(yk), ptr(yv), ptr(fq), ptr(fk), ptr(factors), ptr(o), ptr(blobs), ptr(out),
            n_decode, n, T, min(T, max_q_len or T), nv, nk, dk, dv, self.taps, dk ** -0.5, self.eps, stream()), "gdn_layer")
        from . import _count
        _count(1 + int(n_decode > 0) + 3 * int(n > n_decode))
        return out


def sigmoid_gate_(out, gate, gate_head_stride):
    """out [T, heads, d] bf16 times sigmoid(gate), in place; `gate`: a view that starts at head 0's gate, rows by stride(0)."""
    T, heads, d = out.shape
    assert out.dtype == gate.dtype == torch.bfloat16 and out.is_contiguous() and gate.stride(-1) == 1
    check(_lib.load().xllm_sigmoid_gate(ptr(out), ptr(gate), gate.stride(0), gate_head_stride, T, heads, d, stream()),
          "sigmoid_gate")
    from . import _count
    _count()
    return out


def decode_step_reference(S, q, k, v, g, beta):
    """S [B, nv, dk, dv]; q, k [B, nv, dk]; v [B, nv, dv]; g, beta [B, nv] (fp32).  Returns (S', o [B, nv, dv])."""
    S = S * g.exp()[:, :, None, None]
    delta = (v - (S * k[..., None]).sum(-2)) * beta[..., None]
    S = S + k[..., None] * delta[:, :, None, :]
    return S, (S * q[..., None]).sum(-2)


def decode_step(state, slots, q, k, v, g, beta, out=None):
    """Updates `state[slots]` ([n_slots, nv, dk, dv] fp32) in place and returns o [B, nv, dv] (fp32)."""
    B, nv, dk = q.shape
    dv = v.shape[-1]
    if not state.is_cuda:
        S, o = decode_step_reference(state[slots], q.float(), k.float(), v.float(), g.float(), beta.float())
        state[slots] = S
        if out is not None:
            out.copy_(o)
            return out
        return o
    assert state.dtype == torch.float32 and state.is_contiguous() and slots.dtype == torch.int64
    q, k, v = q.float().contiguous(), k.float().contiguous(), v.float().contiguous()
    g, beta = g.float().contiguous(), beta.float().contiguous()
    if out is None or not out.is_contiguous() or out.dtype != torch.float32:
        res = torch.empty(B, nv, dv, dtype=torch.float32, device=q.device)
    else:
        res = out
    check(_lib.load().xllm_gdn_decode_step(ptr(state), ptr(slots.contiguous()), ptr(q), ptr(k), ptr(v), ptr(g), ptr(beta),
                                           ptr(res), B, nv, dk, dv, stream()), "gdn_decode_step")
    if out is not None and res is not out:
        out.copy_(res)
        return out
    return res


def prefill_reference(S, q, k, v, g, beta):
    """The recurrence over the n tokens of one sequence: S [nv, dk, dv]; q, k [n, nv, dk]; v [n, nv, dv];
    g, beta [n, nv].  Returns (S', o [n, nv, dv])."""
    out = []
    S = S[None]
    for t in range(q.shape[0]):
        S, o = decode_step_reference(S, q[t:t + 1], k[t:t + 1], v[t:t + 1], g[t:t + 1], beta[t:t + 1])
        out.append(o[0])
    return S[0], torch.stack(out) if out else v.new_zeros(0, *v.shape[1:])


def prefill(state, slot: int, fresh: bool, q, k, v, g, beta, out=None):
    """Advances `state[slot]` over the n tokens of a prompt chunk in place (from zero when `fresh`) and
    returns o [n, nv, dv] fp32.  One kernel on CUDA for dk in {32, 64, 128, 256}."""
    n, nv, dk = q.shape
    dv = v.shape[-1]
    if not state.is_cuda or dk not in (32, 64, 128, 256):
        S0 = torch.zeros_like(state[slot]) if fresh else state[slot]
        S, o = prefill_reference(S0, q.float(), k.float(), v.float(), g.float(), beta.float())
        state[slot] = S
        if out is not None:
            out.copy_(o)
            return out
        return o
    assert state.dtype == torch.float32 and state.is_contiguous()
    q, k, v = q.float().contiguous(), k.float().contiguous(), v.float().contiguous()
    g, beta = g.float().contiguous(), beta.float().contiguous()
    res = out if (out is not None and out.is_contiguous() and out.dtype == torch.float32) else \
        torch.empty(n, nv, dv, dtype=torch.float32, device=q.device)
    check(_lib.load().xllm_gdn_prefill(ptr(state), int(slot), int(bool(fresh)), ptr(q), ptr(k), ptr(v), ptr(g), ptr(beta),
                                       ptr(res), n, nv, dk, dv, stream()), "gdn_prefill")
    from . import _count
    _count()
    if out is not None and res is not out:
        out.copy_(res)
        return out
    return res
