"""Gated-delta-net (GDN) linear attention for B200: chunked prefill, fused recurrent decode, gated RMSNorm.

Entry points follow the calling convention of the reference's kernel library
(python/avelang_kernels/amdgpu_gemm.py:458-494): plain module-level functions that take torch tensors,
raise ValueError on dtype/shape/device problems, allocate the result unless ``out=`` is given, enqueue on
torch's current stream of the tensors' device and return without synchronising.  The reference itself has
no GDN kernels; the numerical contract is the recurrence

    M <- exp(g_t) M;  r = M^T k_t;  u = beta_t (v_t - r);  M <- M + k_t u^T;  o_t = scale M^T q_t

with M the fp32 key-major state [dk, dv] of one (sequence, value head).

Layouts: q, k ``[B, T, Hk, dk]``; v, z, o ``[B, T, Hv, dv]``; g (log decay) and beta ``[B, T, Hv]`` fp32; value head
h reads key head ``h // (Hv // Hk)``.  Varlen: ``B == 1`` and int32 ``cu_seqlens [N+1]`` on the device.  States:
fp32 ``[N or num_slots, Hv, dk, dv]``.  The innermost dimension must be contiguous; head/token/batch strides
are free as long as rows stay 16-byte aligned, so head-sharded slices of a packed tensor are accepted as is.
"""
from __future__ import annotations

import ctypes

import torch

from . import _lib, torch_ops  # noqa: F401  (torch_ops declares the operators the native functions call)

__all__ = ["chunk_gated_delta_rule", "fused_recurrent_gated_delta_rule", "mixed_prefill_decode_step", "gated_rmsnorm",
           "causal_conv1d_silu", "causal_conv1d_update", "gate_beta", "decode_layer_step", "gated_delta_rule_backward", "GatedDeltaRuleFunction", "prefill_launch_count", "read_status"]

_native = _lib.host  # checks and allocation of every public function, and the operators behind them (csrc/host.cpp)
_lib.register_operators()


def _status_word(device: torch.device) -> torch.Tensor:
    return _native.status_word(device.index if device.index is not None else torch.cuda.current_device())


def read_status(device=None, reset: bool = True) -> int:
    """Device status word accumulated by earlier calls (synchronises).  Bits: 1 = a state index beyond the
    pool, 2 = malformed cu_seqlens, 4 = a bounded device wait gave up.  The affected sequences were skipped (with a
    malformed cu_seqlens the whole batch of a prefill or backward call)."""
    device = torch.device("cuda", torch.cuda.current_device()) if device is None else torch.device(device)
    w = _status_word(device)
    val = int(w.item())
    if reset and val:
        w.zero_()
    return val


def chunk_gated_delta_rule(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=False,
                           use_qk_l2norm_in_kernel=False, cu_seqlens=None, *, z=None, norm_weight=None,
                           norm_eps=1e-6, state_indices=None, inplace_state=True, chunk_size=64, out=None, out_peers=None,
                           max_seqlen=None):
    """Chunked (chunk 64) gated delta rule over whole sequences.  Returns ``(o, final_state or None)``.

    With ``z`` the gated RMSNorm ``rmsnorm(o) * silu(z)`` (weight ``norm_weight``, eps ``norm_eps``) is fused and
    ``o`` is the normalised output.  With ``state_indices`` the initial states are read from, and the final
    states written to, slots of the ``initial_state`` pool (in place unless ``inplace_state=False``).

    ``out_peers`` (needs ``z``): int64 device tensor of base addresses of buffers laid out exactly like ``out``, one per
    GPU of the node (peer-mapped, this GPU's included).  The normalised rows are then stored into all of them by the
    norm kernel itself (a fused all-gather over NVLink) instead of into ``out``; the caller must put a barrier between
    this call and any reader of those buffers.

    ``max_seqlen`` (with ``cu_seqlens``): an upper bound of the longest sequence, known to the host.  With it the
    parallel parts that a batch of few long sequences is cut into are sized from the real chain length
    instead of the packed total; results agree to rounding with and without it.  A sequence longer than the bound is skipped and flagged in the status word, like a
    malformed ``cu_seqlens`` entry."""
    return _native.prefill(q, k, v, g, beta, scale, initial_state, output_final_state, use_qk_l2norm_in_kernel, cu_seqlens, z,
                           norm_weight, norm_eps, state_indices, inplace_state, chunk_size, out, out_peers, max_seqlen)


def prefill_launch_count(q, k, v, *, z=None, cu_seqlens=None, max_seqlen=None, push=False) -> int:
    """Number of kernels one ``chunk_gated_delta_rule`` call on tensors of these shapes enqueues (``push``: with the
    fused all-gather).  Asked from the library, which derives it from the same schedule it launches."""
    B, T, Hk, dk = q.shape
    Hv, dv = v.shape[2], v.shape[3]
    n_seqs = B if cu_seqlens is None else cu_seqlens.numel() - 1
    a = _lib.GdnArgs()
    a.struct_size = ctypes.sizeof(_lib.GdnArgs)
    # only shapes, strides and the presence of optional tensors enter the count: nothing is read through the pointers
    a.q, a.k, a.v, a.o = q.data_ptr(), k.data_ptr(), v.data_ptr(), v.data_ptr()
    a.g = a.beta = v.data_ptr()
    a.z = z.data_ptr() if z is not None else None
    a.cu_seqlens = cu_seqlens.data_ptr() if cu_seqlens is not None else None
    a.B, a.T, a.Hk, a.Hv, a.dk, a.dv, a.n_seqs, a.num_slots, a.chunk = B, T, Hk, Hv, dk, dv, n_seqs, n_seqs, 64
    for name, t in (("q", q), ("k", k), ("v", v), ("z", z), ("o", v)):
        if t is not None:
            setattr(a, f"{name}_stride_b", t.stride(0)); setattr(a, f"{name}_stride_t", t.stride(1)); setattr(a, f"{name}_stride_h", t.stride(2))
    a.g_stride_b, a.g_stride_t = T * Hv, Hv
    if max_seqlen is not None and cu_seqlens is not None:
        a.max_seqlen = min(int(max_seqlen), T)
    if push:
        a.o_peers, a.n_peers = v.data_ptr(), 2  # only their presence matters for the count
    return int(_lib.load().ave_gdn_prefill_launch_count(ctypes.byref(a)))


def fused_recurrent_gated_delta_rule(q, k, v, g, beta, scale=None, initial_state=None, output_final_state=True,
                                     use_qk_l2norm_in_kernel=False, cu_seqlens=None, *, state_indices=None,
                                     inplace_state=True, z=None, norm_weight=None, norm_eps=1e-6, out=None):
    """Token-by-token gated delta rule with the state tile held on chip; ``T == 1`` with ``state_indices`` is the
    continuous-batching decode step: each sequence's state is streamed once in and once out of its slot of the
    ``initial_state`` pool (updated in place unless ``inplace_state=False``).  A negative slot index skips the
    sequence (no state access, zero output).  Returns ``(o, state)``."""
    return _native.decode(q, k, v, g, beta, scale, initial_state, output_final_state, use_qk_l2norm_in_kernel, cu_seqlens,
                          state_indices, inplace_state, z, norm_weight, norm_eps, out)


def mixed_prefill_decode_step(q, k, v, g, beta, cu_seqlens, n_decode, state_pool, state_indices, scale=None,
                              use_qk_l2norm_in_kernel=False, *, z=None, norm_weight=None, norm_eps=1e-6, out=None):
    """One continuous-batching step over a packed batch (``B == 1``) ordered decode-first: sequences ``[0, n_decode)``
    have exactly one token each and take the bandwidth-streaming decode kernel, the remaining sequences are prefill
    (or chunked-prefill continuation) sequences of any length and take the chunked kernel.  Every sequence reads its
    state from, and writes it back to, slot ``state_indices[n]`` of ``state_pool`` in place (a fresh sequence starts
    from a zeroed slot).  ``cu_seqlens`` describes the whole packed batch; its first ``n_decode + 1`` entries must be
    ``0, 1, ..., n_decode`` (not checked: that would need a device synchronisation).  Everything goes to the current stream
    (the two parts run beside one another on the GPU).  Where a prompt names the slot of a single-token sequence, the single token comes
    first; single-token sequences, and prompts, that share a slot among themselves have no order.  Returns ``o`` ``[1, T, Hv, dv]``."""
    return _native.mixed(q, k, v, g, beta, cu_seqlens, n_decode, state_pool, state_indices, scale, use_qk_l2norm_in_kernel, z,
                         norm_weight, norm_eps, out)


def gated_delta_rule_backward(q, k, v, g, beta, d_o, scale=None, initial_state=None, d_final_state=None, cu_seqlens=None):
    """Gradients of ``chunk_gated_delta_rule`` / ``fused_recurrent_gated_delta_rule`` (without the in-kernel L2 norm and
    without the fused gated norm) for d = 128.  ``d_o``: bf16, shaped like ``v``; ``d_final_state``: optional fp32 gradient
    of the final states.  Returns ``(dq, dk, dv, dg, dbeta, d_initial_state)``: dq, dk in the dtype and shape of q, k (the
    value heads sharing a key head are summed), dv in the dtype of v, dg, dbeta fp32, ``d_initial_state`` fp32 or None
    when no initial state was given.  Chunked like the forward pass (64 tokens), every fp32 operand carried to 24 bits."""
    return _native.backward(q, k, v, g, beta, d_o, scale, initial_state, d_final_state, cu_seqlens)


class GatedDeltaRuleFunction(torch.autograd.Function):
    """``o, final_state = GatedDeltaRuleFunction.apply(q, k, v, g, beta, scale, initial_state)``: the chunked forward pass
    with the chunked backward pass attached (d = 128, dense batches, no in-kernel L2 norm, no fused gated norm)."""

    @staticmethod
    def forward(ctx, q, k, v, g, beta, scale, initial_state):
        o, final = chunk_gated_delta_rule(q, k, v, g, beta, scale, initial_state, output_final_state=True)
        ctx.save_for_backward(q, k, v, g, beta, initial_state if initial_state is not None else torch.empty(0, device=q.device))
        ctx.scale, ctx.has_state = scale, initial_state is not None
        return o, final

    @staticmethod
    def backward(ctx, d_o, d_final):
        q, k, v, g, beta, s0 = ctx.saved_tensors
        d_o = torch.zeros_like(v) if d_o is None else d_o.to(torch.bfloat16).contiguous()
        d_final = None if d_final is None else d_final.float().contiguous()
        dq, dk, dv, dg, dbeta, ds0 = gated_delta_rule_backward(q, k, v, g, beta, d_o, ctx.scale, s0 if ctx.has_state else None, d_final)
        return dq, dk, dv, dg, dbeta, None, ds0


def decode_layer_step(proj, conv_weight, conv_state, A_log, dt_bias, state_pool, state_indices=None, *, Hk, Hv, conv_bias=None,
                      norm_weight=None, norm_eps=1e-6, scale=None, gate_first=False, out=None):
    """One decode step of a whole GDN layer behind its in-projection, in one kernel.  ``proj``: bf16 ``[N, >= 2*Hk*128 +
    2*Hv*128 + 2*Hv]``, each row the new token's projection ``[q | k | v | z | b | a]`` (a column slice of a wider matrix
    is accepted); ``conv_weight`` bf16 ``[2*Hk*128 + Hv*128, W]`` (W in 2..4, rows in q | k | v order), ``conv_state`` bf16
    ``[slots, W-1, C]`` and ``state_pool`` fp32 ``[slots, Hv, 128, 128]`` share the slot index ``state_indices[n]`` (or n)
    and are updated in place; ``A_log``, ``dt_bias`` ``[Hv]``.  Computes conv update + SiLU, q/k L2 norm, gate and beta,
    the delta-rule update and the gated RMSNorm with z; the results are those of ``causal_conv1d_update`` + ``gate_beta`` +
    ``fused_recurrent_gated_delta_rule`` run one after the other.  Returns ``o [N, Hv, 128]``."""
    return _native.decode_layer(proj, conv_weight, conv_state, A_log, dt_bias, state_pool, state_indices, Hk, Hv, conv_bias, norm_weight,
                                norm_eps, scale, gate_first, out)


def gated_rmsnorm(x, z, weight=None, eps=1e-6, *, gate_first=False, out=None):
    """``y = weight * x * rsqrt(mean(x^2) + eps) * silu(z)`` over the last dimension (64 or 128), bf16 in/out,
    fp32 math.  ``x``/``z``/``out``: ``[..., H, d]`` with a contiguous last dimension."""
    return _native.rmsnorm(x, z, weight, eps, gate_first, out)


def causal_conv1d_silu(x, weight, bias=None, cu_seqlens=None, *, out=None):
    """Depthwise causal convolution over time followed by SiLU: ``y[t, c] = silu(bias[c] + sum_j weight[c, j] *
    x[t - (W-1) + j, c])`` with zero history at the start of every sequence.  ``x``: bf16 ``[B, T, C]`` (channel
    stride 1, row stride free, so a column slice of a wider projection output is accepted), ``weight``: bf16
    ``[C, W]`` with W in 2..4, optional ``bias`` bf16 ``[C]``, optional int32 ``cu_seqlens`` (``B == 1``)."""
    return _native.conv(x, weight, bias, cu_seqlens, out)


def causal_conv1d_update(x, conv_state, weight, bias=None, state_indices=None, *, out=None):
    """Decode-time step of ``causal_conv1d_silu``: ``x`` bf16 ``[N, C]`` (one new token per sequence), ``conv_state`` bf16
    ``[slots, W-1, C]`` holding each sequence's last W-1 inputs (oldest first), updated in place; optional int32
    ``state_indices [N]`` selects the slots (negative: skip that sequence; beyond the pool: skip it and raise bit 1 of
    the status word).  Returns ``y [N, C]``."""
    return _native.conv_update(x, conv_state, weight, bias, state_indices, out)


def gate_beta(a_in, b_in, A_log, dt_bias):
    """``g = -exp(A_log) * softplus(a + dt_bias)`` and ``beta = sigmoid(b)`` in fp32.  ``a_in``, ``b_in``: bf16
    ``[..., Hv]`` (last dimension contiguous, one common row stride); ``A_log``, ``dt_bias``: ``[Hv]``."""
    return _native.gate(a_in, b_in, A_log, dt_bias)
