"""Operator layer: the CASTLE attention core as torch-facing functions.  The work between a call and
the C-ABI library's launches (descriptors, scratch, the passes around the kernels, the autograd node)
is native, in csrc/host.cpp; this file holds the operators' contracts and limits.

`castle_attention` mirrors the reference operator
`castle_attention_triton(qc, kc, vc, qu, ku, vu, scale, return_U_for_cache)`
(lookahead_keys_attention/lookahead_keys_attention_triton.py:416-605): same
argument order (causal triple first), unscaled inputs, returns `out` or
`(out, U)`, six input gradients, no gradient through U.
`castle_decode_step` replaces the single-token branch of the reference module
(lookahead_keys_attention/lookahead_keys_attention.py:166-203).
"""
from __future__ import annotations

import torch

from . import _lib
from ._lib import CastleTensor


def _device_index(device) -> int:
    device = torch.device(device)
    return torch.cuda.current_device() if device.index is None else device.index


def status_word(device) -> torch.Tensor:
    """Per-device int32 the kernels OR error bits into (0 = fine)."""
    return _lib.host().status_word(_device_index(device))


def check_status(device=None):
    """Synchronising check of the device status word; raises on a kernel-side failure."""
    devs = [_device_index(device)] if device is not None else _lib.host().status_devices()
    for d in devs:
        w = status_word(torch.device("cuda", d))
        v = int(w.item())
        if v != 0:
            w.zero_()
            raise RuntimeError(f"castle kernels reported status {v} on cuda:{d} (1 = a bounded wait ran out)")


def release_workspaces():
    """Free every cached scratch buffer (one per device and stream, grown on demand and kept between
    calls; they are re-created on the next call)."""
    _lib.host().release_workspaces()


def _desc(t: torch.Tensor) -> CastleTensor:
    """(B, H, N, d) tensor or view with a contiguous last dim -> castle_tensor_t, for callers of the C ABI."""
    assert t.dim() == 4 and (t.stride(3) == 1 or t.shape[3] == 1)
    return CastleTensor(t.data_ptr(), t.stride(0), t.stride(1), t.stride(2))


# Bound on the forward's scratch per launch.  The soft-max partials take N^2/128 * (8 + 2*d) bytes
# per (batch, head) pair (O(N^2), where the reference kernel needs O(N*d)), so a call is cut into
# launches over whole batch rows, or over head ranges of one batch row, that each stay below it.
MAX_WORKSPACE_BYTES = 16 << 30


def forward_chunks(B: int, H: int, per_pair: int, limit: int | None = None):
    """Rectangles (b0, b1, h0, h1) of the (batch, head) grid that a forward is launched over, each needing at most
    `limit` bytes of scratch at `per_pair` bytes per pair.  A rectangle spans several batch rows only with all heads,
    so that the per-pair fp32 buffers (lse, state) of a rectangle stay contiguous.  (csrc/host.cpp, for_chunks.)"""
    return _lib.host().forward_chunks(B, H, per_pair, MAX_WORKSPACE_BYTES if limit is None else limit)


# From this sequence length on, bf16 callers are computed with fp16 operands.  The lookahead state W grows
# like sqrt(N) (|W| ~ 100 at N = 8192) and the gate's and the state's 16-bit copies are what the long-range
# gradients are made of: with 8 significant bits dqc misses |a-b| <= 2e-2 + 1e-2|b| from N ~ 8192 on, with
# fp16's 11 bits it holds at N = 16384.  (The tensor cores cannot mix an fp16 operand with a bf16 one in a
# single product, so the inputs are converted once instead; at these lengths that pass is < 1 % of the work.)
# fp32 callers run with fp16 operands at every length (as the reference operator does,
# lookahead_keys_attention_triton.py:437-442).
# Costs: values beyond +-65504 in q/k/v saturate, and the upstream gradient is rescaled by a power of two
# (exactly) so that small gradients do not underflow.
LONG_SEQ_FP16 = 6144


class _Traced(torch.autograd.Function):
    """An operator while torch.jit.trace is recording: a Python autograd function becomes a node of the traced graph,
    which calls it again when the graph runs; of the native operator the tracer would only see the allocations."""

    @staticmethod
    def forward(ctx, packed_op, scale, return_U, *inputs):
        with torch.enable_grad():
            leaves = [t.detach().requires_grad_(t.requires_grad) for t in inputs]
            limits = (scale, return_U, None, MAX_WORKSPACE_BYTES, LONG_SEQ_FP16)
            host = _lib.host()
            result = host.attention_packed(*leaves, *limits, None, True) if packed_op else host.attention(*leaves, *limits)
        out, *U = result if return_U else (result,)
        ctx.graph = leaves, out
        if return_U:
            ctx.mark_non_differentiable(*U)
        return (out.detach(), *U) if return_U else out.detach()

    @staticmethod
    def backward(ctx, grad, *_):
        leaves, out = ctx.graph
        wanted = [t for t in leaves if t.requires_grad]
        grads = iter(torch.autograd.grad(out, wanted, grad, retain_graph=True))
        return (None, None, None, *(next(grads) if t.requires_grad else None for t in leaves))


def castle_attention_packed(packed, scale, return_U_for_cache=False, cache_out=None):
    """Parallel CASTLE attention on the packed projection output (B, N, 6, H, d), order
    qu,ku,vu,qc,kc,vc (the layout `to_all_qkv` produces).  Returns out (B, H, N, d) [, U].
    With `cache_out` = four (B, H, N, d) views (U, qu, kc, vc) of decode-cache buffers, the
    kernels write the cache rows themselves and the returned U is cache_out[0].
    Its gradient is the packed buffer the backward kernels write, so autograd has nothing to
    scatter or sum (six separate view-gradients cost ~10 extra passes)."""
    if torch._C._is_tracing() and cache_out is None:
        return _Traced.apply(True, float(scale), bool(return_U_for_cache), packed)
    return _lib.host().attention_packed(packed, scale, return_U_for_cache, cache_out, MAX_WORKSPACE_BYTES, LONG_SEQ_FP16,
                                        None, True)


def castle_attention(qc, kc, vc, qu, ku, vu, scale, return_U_for_cache=False, cache_out=None):
    """Parallel CASTLE attention on (B, H, N, d) tensors (views are fine).
    Returns `out`, or `(out, U)` when `return_U_for_cache`; `cache_out` as in `castle_attention_packed`."""
    if torch._C._is_tracing() and cache_out is None:
        return _Traced.apply(False, float(scale), bool(return_U_for_cache), qc, kc, vc, qu, ku, vu)
    return _lib.host().attention(qc, kc, vc, qu, ku, vu, scale, return_U_for_cache, cache_out, MAX_WORKSPACE_BYTES,
                                 LONG_SEQ_FP16)


def castle_decode_step(qc, kc, vc, qu, ku, vu, U, qu_cache, kc_cache, vc_cache, cache_len: int, scale: float):
    """One cached token.  The four caches are (B, H, capacity, d) buffers with `cache_len`
    valid rows; they are updated IN PLACE (row `cache_len` appended, U[0:cache_len] rewritten).
    The six new-token tensors are (B, H, 1, d).  Returns out (B, H, 1, d)."""
    return _lib.host().decode_step(qc, kc, vc, qu, ku, vu, U, qu_cache, kc_cache, vc_cache, cache_len, scale)
