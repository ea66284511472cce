"""`Castle` - drop-in for the reference module of the same name
(lookahead_keys_attention/lookahead_keys_attention.py:41-214): same constructor
arguments, state-dict keys (`to_all_qkv.weight`, `combine_heads.weight`,
`norm.weight`), `forward(x, cache=None, return_next_cache=None)` conventions
and `Cache` tuple.  The attention cores run as sm_100a kernels through the
C-ABI library, rotary embedding included.  A plain layer is one native call
(csrc/host.cpp): RMSNorm and the projections of a few tokens are kernels of this
package, the other projections library products, and the gradient one autograd
node.  Where a submodule was replaced, wrapped or hooked, or something records or
replaces torch functions, the submodules are called as modules instead.

Difference from the reference, by design: the decode step appends to
pre-allocated cache buffers and rewrites the lookahead keys `U` IN PLACE
instead of concatenating new tensors every token (:185-203), so a cache
returned by step t shares memory with the cache returned by step t-1, and
only the LATEST cache of a chain may be decoded from (an older one raises).
Pass `inplace_cache=False` to get the reference's functional behaviour (each
step then copies the caches first, and any cache can be decoded from again).
Only caches this module returned (or took over through `cache_from_buffers`)
are ever written; a cache made of the caller's own tensors is copied first.
"""
from __future__ import annotations

from collections import namedtuple

import torch
from torch import nn
from torch.nn.modules.module import _has_any_global_hook

from . import _lib, ops

Cache = namedtuple("Cache", ("U", "qu_cache", "kc_cache", "vc_cache"))


class _CacheBuffers:
    """Four (B, H, capacity, d) buffers the module allocated, and how many of their rows are valid
    NOW.  Decode steps append to them and rewrite U in place, so only the cache returned by the
    latest step still describes their contents."""

    __slots__ = ("bufs", "length", "capacity")

    def __init__(self, bufs, length):
        self.bufs, self.length = list(bufs), int(length)
        self.capacity = self.bufs[0].shape[2]

    def views(self, n):
        return _lib.host().first_rows(self.bufs, n)


class ModuleCache(Cache):
    """The `Cache` tuple as this module returns it: the same four fields, each a `[:, :, :t]` view,
    plus a record of the capacity buffers behind them.  Ownership is explicit: the in-place decode
    path is taken only for a `ModuleCache` that is the latest one of its buffers.  Any other cache
    (a plain tuple of the caller's tensors, slices, a re-wrapped copy) is treated as read-only
    input and copied into fresh buffers first, so the caller's memory is never written."""

    def __new__(cls, state: _CacheBuffers, length: int, views=None):
        self = tuple.__new__(cls, state.views(length) if views is None else views)
        self._state, self._length = state, int(length)
        return self

    def is_current(self) -> bool:
        return self._state.length == self._length


def cache_from_buffers(U, qu_cache, kc_cache, vc_cache, length: int) -> ModuleCache:
    """Hand four caller-allocated (B, H, capacity, d) buffers with `length` valid rows over to the
    module: from now on decode steps append to them and rewrite U IN PLACE (no copy is made)."""
    bufs = [U, qu_cache, kc_cache, vc_cache]
    shape = tuple(U.shape)
    for b in bufs:
        if b.dim() != 4 or tuple(b.shape) != shape or b.dtype != U.dtype or not b.is_contiguous():
            raise ValueError("cache_from_buffers: four contiguous (B, H, capacity, d) buffers of one dtype expected")
    if not 0 <= length <= shape[2]:
        raise ValueError("cache_from_buffers: length out of range")
    return ModuleCache(_CacheBuffers(bufs, length), length)


class _Rotary(nn.Module):
    """This package's own rotary embedding (pairs of adjacent channels rotated by
    position * theta^(-2i/d)).  The module's passes apply it inside their kernels (csrc/rotary.cuh),
    with the rounding points of `rotate`, which states it in torch operations.  The reference delegates to the third-party
    `rotary_embedding_torch` package, which is not available to compare against;
    numerical agreement with that package is not claimed."""

    def __init__(self, dim, theta=10000.0):
        super().__init__()
        self.register_buffer("freqs", theta ** (-torch.arange(0, dim, 2).float() / dim), persistent=False)

    def rotate(self, t, offset=0):
        n = t.shape[-2]
        ang = (torch.arange(n, device=t.device, dtype=torch.float32) + offset)[:, None] * self.freqs.to(t.device)
        cos, sin = ang.cos().to(t.dtype), ang.sin().to(t.dtype)
        a, b = t[..., 0::2], t[..., 1::2]
        return torch.stack((a * cos - b * sin, a * sin + b * cos), dim=-1).flatten(-2)


class Castle(nn.Module):
    def __init__(self, dim, heads=8, dim_head=64, use_triton=None, rotary_emb=False, prenorm=False,
                 inplace_cache=True, cache_headroom=256):
        super().__init__()
        dim_inner = dim_head * heads
        self.dim, self.dim_head, self.heads = dim, dim_head, heads
        # Attribute kept for callers that read it; the value follows the reference's default rule
        # (lookahead_keys_attention.py:58, "CUDA available and the kernel backend importable") with this
        # package's kernels in the place of Triton.  It selects nothing: there is one code path.
        self.use_triton = bool(use_triton) if use_triton is not None else torch.cuda.is_available()
        self.scale = dim_head ** -0.5
        self.norm = nn.RMSNorm(dim) if prenorm else nn.Identity()
        self.rotary_emb = _Rotary(dim_head) if rotary_emb else None
        self.to_all_qkv = nn.Linear(dim, dim_inner * 6, bias=False)
        self.combine_heads = nn.Linear(dim_inner, dim, bias=False)
        self.inplace_cache = inplace_cache
        self.cache_headroom = cache_headroom

    def _split(self, qkvs):
        b, n, _ = qkvs.shape
        # 'b n (qkv h d) -> qkv b h n d', order qu, ku, vu, qc, kc, vc (reference :77,104); views, no copies
        return qkvs.view(b, n, 6, self.heads, self.dim_head).permute(2, 0, 3, 1, 4).unbind(0)

    def _new_buffers(self, b, h, d, rows, like) -> _CacheBuffers:
        cap = rows + max(self.cache_headroom, rows // 4)
        return _CacheBuffers(_lib.host().new_caches(like, b, h, cap, d), 0)

    def _new_cache(self, like) -> _CacheBuffers:
        """The cache of a prompt of `like`'s batch size, length and type lives in buffers with spare rows so that decode
        steps can append in place.  The forward's kernels fill it themselves: from their operand tiles where those are
        the caller's values, otherwise in the pass that makes the operands."""
        return self._new_buffers(like.shape[0], self.heads, self.dim_head, like.shape[1], like)

    def _state_in_place(self, cache, t):
        """The capacity buffers behind `cache` if row t can be appended to them as they are, else None."""
        if not isinstance(cache, ModuleCache) or cache._length != t:
            return None
        state = cache._state
        if state.length != t and self.inplace_cache:
            raise RuntimeError(
                "this cache was advanced in place by a later decode step and no longer holds its rows; "
                "construct Castle(..., inplace_cache=False) to decode from one cache more than once")
        return state if self.inplace_cache and t < state.capacity else None

    def _buffers_for_step(self, cache, t, like) -> _CacheBuffers:
        """Capacity buffers holding rows [0, t) of `cache` with room for row t."""
        state = self._state_in_place(cache, t)
        if state is not None:
            return state
        # a foreign cache, a full buffer, or functional semantics asked for: copy into fresh buffers
        b, h, _, d = like.shape
        fresh = self._new_buffers(b, h, d, t + 1, like)
        if t > 0:
            with torch.no_grad():
                for buf, src in zip(fresh.bufs, cache):
                    buf[:, :, :t].copy_(src)
        fresh.length = t
        return fresh

    def _plain_layer(self):
        """What the native path takes of this layer: norm weight and eps, the two projection weights and the head
        sizes; or None where a submodule was replaced, has a bias, hooks or a forward of its own (how offloading wraps
        it), so that it must be called as a module."""
        mods = self._modules
        norm, qkv, combine = mods["norm"], mods["to_all_qkv"], mods["combine_heads"]
        if type(qkv) is not nn.Linear or type(combine) is not nn.Linear or _has_any_global_hook():
            return None
        for m in (norm, qkv, combine):
            own = m.__dict__
            if ("forward" in own or own["_forward_hooks"] or own["_forward_pre_hooks"] or own["_backward_hooks"]
                    or own["_backward_pre_hooks"]):
                return None
        wq, wc = qkv._parameters, combine._parameters
        try:
            if wq["bias"] is not None or wc["bias"] is not None:
                return None
            if type(norm) is nn.Identity:
                return None, None, wq["weight"], wc["weight"], self.heads, self.dim_head
            if type(norm) is nn.RMSNorm and norm._parameters["weight"] is not None and len(norm.normalized_shape) == 1:
                return norm._parameters["weight"], norm.eps, wq["weight"], wc["weight"], self.heads, self.dim_head
        except KeyError:   # a data-parallel replica holds its weights as plain attributes
            pass
        return None

    def _project(self, x):
        """The packed projection (b, n, 6, heads, dim_head) with the submodules called as modules."""
        return self.to_all_qkv(self.norm(x)).view(x.shape[0], x.shape[1], 6, self.heads, self.dim_head)

    def _merge(self, out):
        return self.combine_heads(out.permute(0, 2, 1, 3).flatten(2))   # 'b h n d -> b n (h d)'

    def _forward_operators(self, x, cache, return_next_cache):
        """Submodules and operators called from here: under torch.jit.trace, which has to see them, and with a rotary
        embedding of the caller's own (a subclass, or another object with `rotate(t, offset)`) in the place of `_Rotary`."""
        seq_len = x.shape[1]
        qu, ku, vu, qc, kc, vc = self._split(self.to_all_qkv(self.norm(x)))
        t = cache[0].shape[-2] if cache is not None else 0
        if self.rotary_emb is not None:
            qc, kc, qu, ku, vu = (self.rotary_emb.rotate(v, t) for v in (qc, kc, qu, ku, vu))
        if seq_len == 1:
            with torch.no_grad():
                state = self._buffers_for_step(cache, t, qu)
                out = ops.castle_decode_step(qc, kc, vc, qu, ku, vu, *state.bufs, t, self.scale)
            state.length = t + 1
            return (self._merge(out), ModuleCache(state, t + 1)) if return_next_cache else self._merge(out)
        assert cache is None, "must be inferencing single tokens if receiving cache"
        if not return_next_cache:
            return self._merge(ops.castle_attention(qc, kc, vc, qu, ku, vu, self.scale))
        out, U = ops.castle_attention(qc, kc, vc, qu, ku, vu, self.scale, True)
        state = self._buffers_for_step((U, qu, kc, vc), seq_len, qu)
        return self._merge(out), ModuleCache(state, seq_len)

    def forward(self, x, cache: Cache | None = None, return_next_cache=None):
        host = _lib.host()
        seq_len = x.shape[1]
        is_inference = seq_len == 1
        if return_next_cache is None:
            return_next_cache = is_inference
        layer = self._plain_layer()
        rotary, freqs = self.rotary_emb, None
        if rotary is not None:
            if type(rotary) is not _Rotary or "rotate" in rotary.__dict__:
                return self._forward_operators(x, cache, return_next_cache)
            freqs = rotary._buffers["freqs"]

        # The native calls return None where their torch functions have to be seen (a tracer, a torch function mode).
        if is_inference:
            t = 0 if cache is None else cache._length if isinstance(cache, ModuleCache) else cache[0].shape[-2]
            state = self._state_in_place(cache, t)
            out = host.layer_decode(x, *layer, self.scale, freqs, state.bufs, t) if layer is not None and state is not None else None
            if out is None:
                if torch._C._is_tracing():
                    return self._forward_operators(x, cache, return_next_cache)
                packed = self._project(x)
                if state is None:
                    state = self._buffers_for_step(cache, t, packed[:, :, 0].transpose(1, 2))
                out = self.combine_heads(host.decode_packed(packed, self.scale, freqs, state.bufs, t))
            state.length = t + 1
            return (out, ModuleCache(state, t + 1)) if return_next_cache else out

        assert cache is None, "must be inferencing single tokens if receiving cache"
        limits = (ops.MAX_WORKSPACE_BYTES, ops.LONG_SEQ_FP16)
        out = state = views = None

        if layer is not None and not torch.is_autocast_enabled("cuda"):   # under autocast only the projection knows the type
            if return_next_cache:
                state = self._new_cache(x)
                views = state.views(seq_len)
            out = host.layer_forward(x, *layer, self.scale, freqs, views, *limits)
        if out is None:
            if torch._C._is_tracing():
                return self._forward_operators(x, cache, return_next_cache)
            packed = self._project(x)
            if return_next_cache:
                state = self._new_cache(packed)
                views = state.views(seq_len)
            out = self._merge(host.attention_packed(packed, self.scale, False, views, *limits, freqs, False))
        if not return_next_cache:
            return out
        state.length = seq_len
        return out, ModuleCache(state, seq_len, views)
