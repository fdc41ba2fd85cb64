"""A recurrent mixer with a matrix state per head, a decay per key channel that depends on the token,
and a bonus for the present token (time mixing in the manner of RWKV).

With h' the token before h in the request (zeros before the first), each of the five branches reads its own blend
   m_s = h + (h' - h) * mu_s,   s in (r, k, v, g, w)
   r, k, v = W_r m_r, W_k m_k, W_v m_v   (heads x head_dim each);   gate = silu(W_g m_g)
   decay w = exp(-exp(W_w2 tanh(W_w1 m_w) + w0))                     per head and key channel
   o_t = (S_(t-1) + diag(u) k_t v_t^T)^T r_t;    S_t = diag(w_t) S_(t-1) + k_t v_t^T      per head
   y = W_o (concat_heads(o / rms(o)) * norm * gate)
The state (S in 32-bit, and the last h of the step in the activation type) lives in the request's state slot;
the recurrence, the decay and the unit norm are 32-bit in both precisions.
"""
from __future__ import annotations

from typing import Dict

import torch

from .. import native
from .base import Mixer
from .linear import linear, streams
from .registry import register
from .spec import CacheEntry, CacheNeed, ParamSpec

_BRANCHES = ("r", "k", "v", "g", "w")


@register("mixer", "decayed_state_mixing")
class DecayedStateMixing(Mixer):
    graph_safe = True
    _rkvg = None

    def __init__(self, hidden_size: int, num_heads: int, head_dim: int, decay_rank: int, norm_eps: float):
        if not native.wkv_supports(head_dim, head_dim):
            raise ValueError(f"decayed_state_mixing: head_dim {head_dim} is beyond what the kernel takes (128)")
        self.hidden_size, self.nh, self.hd, self.rank, self.norm_eps = hidden_size, num_heads, head_dim, decay_rank, norm_eps

    def params(self) -> Dict[str, ParamSpec]:
        W, D = self.hidden_size, self.nh * self.hd
        return {
            "mu": ParamSpec((len(_BRANCHES), W), role="vector", init="half", rows=(1,) * len(_BRANCHES),
                            members_lack_axis=True),
            "r.weight": ParamSpec((D, W)), "k.weight": ParamSpec((D, W)), "v.weight": ParamSpec((D, W)),
            "g.weight": ParamSpec((D, W)),
            "w1.weight": ParamSpec((self.rank, W)), "w2.weight": ParamSpec((D, self.rank)),
            "w0": ParamSpec((D,), role="vector", init="zeros"),
            "u": ParamSpec((self.nh, self.hd), role="vector", init="normal"),
            "norm": ParamSpec((D,), role="vector", init="norm"),
            "o.weight": ParamSpec((W, D)),
        }

    def cache_need(self) -> CacheNeed:
        return CacheNeed("state", states=(
            CacheEntry("wkv", (self.nh, self.hd, self.hd), "float32"),
            CacheEntry("shift", (self.hidden_size,), "compute")))

    def after_load(self) -> None:
        # the four maps of equal sizes as one array, of which they are views: one product of four in a step of many rows
        # (once: captured steps read them where they lie)
        maps = [self.w_r_weight, self.w_k_weight, self.w_v_weight, self.w_g_weight]
        if self._rkvg is not None and all(a.data_ptr() == b.data_ptr() for a, b in zip(maps, self._rkvg)):
            return
        self._rkvg = None
        if self.rt.dtype == torch.bfloat16:
            self._rkvg = torch.stack(maps)
            self.w_r_weight, self.w_k_weight, self.w_v_weight, self.w_g_weight = self._rkvg

    def reserve(self, tokens, seqs, longest) -> None:
        n = sum(native.linear_tc_most(tokens, seqs, self.nh, self.hd, self.hd, True)) if self.rt.dtype == torch.bfloat16 and self.hd <= 64 else 0
        if n:
            self.rt.workspace.get("dsm.chunks", (n,), torch.float32)

    def forward(self, x, step, cache, writes_cache):
        T, W = x.shape
        D = self.nh * self.hd
        ws, dt = self.rt.workspace, self.rt.dtype
        mixes = ws.get("dsm.mixes", (len(_BRANCHES), T, W), dt)
        native.token_shift_mix(mixes, x, self.w_mu, cache.states["shift"], step.seq_of_token, step.cu_q,
                               step.state_slots, writes_cache)
        four = ws.get("dsm.rkvg", (4, T, D), dt)
        r, k, v, g = four.unbind(0)
        if self._rkvg is not None and not streams(T, D, W, W):
            # (one launch: 2,048 rows of 2,048 numbers 51 us, 62 and the gaps between them in four)
            native.gemm_batched(four.transpose(0, 1), mixes[:4].transpose(0, 1), self._rkvg)
        else:
            for m, w, out in zip(mixes, (self.w_r_weight, self.w_k_weight, self.w_v_weight, self.w_g_weight), (r, k, v, g)):
                linear(m, w, None, out)
        a = linear(mixes[4], self.w_w1_weight, None, ws.get("dsm.a", (T, self.rank), dt))
        native.tanh_(a)
        d = linear(a, self.w_w2_weight, None, ws.get("dsm.d", (T, D), torch.float32))
        y = ws.get("dsm.y", (T, D), dt)
        n = native.wkv_scratch_elems(T, step.num_seqs, self.nh, self.hd, self.hd, step.max_q_len) if dt == torch.bfloat16 else 0
        native.wkv(y, r, k, v, d, g, self.w_w0, self.w_u, self.w_norm, cache.states["wkv"], step.cu_q,
                   step.state_slots, step.num_seqs, self.nh, self.hd, self.hd, self.norm_eps, writes_cache,
                   ws.get("dsm.chunks", (n,), torch.float32) if n else None)
        return linear(y, self.w_o_weight, None, ws.get("dsm.out", (T, W), dt))
