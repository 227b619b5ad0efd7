"""Latent attention: keys and values are up-projections of one low-rank row per token, plus one rotated key part that all
heads share; only that row is cached.

With h the mixer's input, per token
    [q | g | d] = W_in h            q: heads x [nope_dim | rot_dim];  g: one gate logit per head;  d: [kv_rank | rot_dim]
    c = rmsnorm(d[:kv_rank]) * w    k_rot = rope(d[kv_rank:])          -> the cache row [c | k_rot]
    score(i, j, head) = (q_nope . (W_uk c_j) + rope(q_rot) . k_rot_j) * scale,   j in the sliding window of i
    out = W_o concat_heads( sigmoid(g) * sum_j softmax_j(score) (W_uv c_j) )
The kernels work in latent space: W_uk is absorbed into the query (q_lat = W_uk^T q_nope, a batched GEMM over heads) and
W_uv is applied to the weighted sum of the c_j, so every head reads the same cache row once.  Prompts in bf16 whose queries
fill the device by themselves (``splits`` 1) have the visible rows expanded per head instead (``_takes_expanded``).  A layer built with ``kv_from`` has no down-projection: it reads another layer's rows with its own W_uk, W_uv,
queries and window.

Variations, all parameters of the spec:
* ``q_rank``: the queries pass a latent of their own, ``q = W_uq (rmsnorm(W_dq h) * w_q)``; the input projection is then
  ``[dq | g | d]``.
* ``gate``: "head" (one logit per head, as above), "element" (``sigmoid(W_g h)`` holds heads * v_dim numbers, one for every
  number the heads put out; applied after W_uv) or "none".
* ``rot_layout``: "interleaved" pairs dimension 2i with 2i+1; "half" pairs i with i + rot_dims/2.  The kernels turn
  interleaved pairs; a "half" checkpoint has the rows of its rotated query and key parts reordered once at load time (the
  same reordering on both sides of the dot product leaves the scores as they are).
* ``exact_weights``: in bf16 the softmax weights enter the weighted sum as two bf16 terms (16 bits) instead of one.
* ``rotary``: a ``rotary.RotarySpec`` whose ``table()`` (rescaled frequencies, magnitude) replaces the plain table.
"""
from __future__ import annotations

import functools
from dataclasses import dataclass
from typing import Optional

import torch
import torch.nn as nn
from torch.nn import functional as F

from . import _native as N
from .rotary import RotarySpec

EXPAND_MIN_TOKENS = 16               # tokens a step appends from which its rows are expanded per head
EXPAND_MAX_SLOTS_PER_TOKEN = 64      # expanded rows per such token
EXPAND_MAX_BYTES = 512 << 20         # of the expanded rows of a step


# Sequences of a step that takes the layer's one call.  us a call, separate calls / one: one token of width 2048 over 1024 of 2048 rows 88 / 45, of
# 4096 over 300 104 / 58, two sequences 102 / 61; replayed as a graph 40.5 / 33.2, 53.9 / 51.2 and 60.4 / 55.4.  Graphed, every layer's weights
# and rows from memory, over 300 and 2000 rows: width 1024 48 / 42 and 47 / 41, 2048 50 / 46 and 50 / 45, 4096 63 / 59 and 63 / 58; two sequences
# 48 / 43 and 50 / 44, 52 / 48 and 52 / 48, 66 / 63 and 66 / 62.
STEP_MAX_ROWS = 2
# More rows: rows times weights of a layer that runs in one call, and its weights (_native.layer_rows).  us a call, separate / one, keys and values expanded
# per head: width 1024, 17, 400 and 2048 rows 92 / 40, 95 / 56, 95 / 76; 2048, 17, 400, 1024 and 2048 rows 93 / 43, 92 / 66, 92 / 76, 110 / 108; 4096 (44M
# weights), 17, 120, 300 and 700 rows 99 / 76, 98 / 70, 95 / 83, 101 / 114; 69M, 17, 120 and 300 rows 96 / 88, 101 / 83, 97 / 93; 98M, 17, 120 and 200
# rows 101 / 97, 95 / 92, 99 / 104; 173M, 17, 60 and 200 rows 120 / 126, 106 / 109, 121 / 126.  A few rows, replayed as a graph: one token of four
# sequences over 1500 rows, widths 1024 and 2048: 37 / 34, 43 / 39 (4096: 55 / 59, so not there).
LAYER_MAX_PRODUCTS, LAYER_MAX_WEIGHTS = 12 << 30, 100 << 20
# Rows times heads of a step in one call whose queries stay in latent space (every four rows read the heads' weights again, and long walks leave no host
# time to save), and its weights.  us, separate / one: 24 heads, 3, 8 and 16 tokens over 300 rows 89 / 66, 89 / 71, 87 / 83, over 2000 rows 4, 8 and 16
# tokens 203 / 197, 202 / 200, 203 / 214; 32 heads (44M weights) 92 / 82, 90 / 85, 92 / 104, 219 / 213, 220 / 216, 219 / 236, one sequence's 8 and 12
# tokens 100 / 100, 100 / 109; 40 heads (69M) 3 and 8 tokens 97 / 97, 98 / 102, over 2000 rows 223 / 227, 224 / 232.
LATENT_MAX_ROW_HEADS, LATENT_MAX_WEIGHTS = 256, 3 << 24


@functools.lru_cache(maxsize=1024)
def _layer_scratch_bytes(*sizes: int) -> int:
    return N.call_ret("ll_latent_layer_scratch_bytes", *sizes)


@functools.lru_cache(maxsize=1024)
def _expanded_supported(*sizes: int) -> bool:
    return N.has("ll_latent_layer") and bool(N.call_ret("ll_latent_prompt_supported", *sizes))


@dataclass
class LatentAttentionSpec:
    width: int
    heads: int
    nope_dim: int                 # un-rotated query / key dimensions per head
    rot_dim: int                  # rotated dimensions per head (one key part for all heads)
    v_dim: int
    kv_rank: int
    window: Optional[int]         # position i sees i - window + 1 .. i; None: everything before it
    scale: float
    rot_base: float = 10000.0
    rot_dims: Optional[int] = None   # the first rot_dims of the rotated part turn, the rest pass; default all
    eps: float = 1e-5
    kv_from: Optional[int] = None    # index of the layer whose cache rows this layer reads
    q_rank: Optional[int] = None     # queries through a normed latent of this size; None: q = W_q h
    gate: str = "head"               # "head" | "element" | "none"
    rot_layout: str = "interleaved"  # "interleaved" | "half"
    exact_weights: bool = False      # softmax weights as two bf16 terms in the tensor-core form
    rotary: Optional[RotarySpec] = None   # rescaled frequencies and magnitude; None: base^(-2i/rot_dims)

    def __post_init__(self):
        if self.rotary is not None:
            self.rot_dims, self.rot_base = self.rotary.dims, self.rotary.base
        if self.gate not in ("head", "element", "none") or self.rot_layout not in ("interleaved", "half"):
            raise ValueError(f"latent attention: gate {self.gate!r}, rotary layout {self.rot_layout!r}")
        if self.rot_dims is None:
            self.rot_dims = self.rot_dim
        if self.rot_dims % 2 or not 0 <= self.rot_dims <= self.rot_dim:
            raise ValueError(f"rot_dims {self.rot_dims} must be even and at most rot_dim {self.rot_dim}")

    @property
    def row(self) -> int:
        return self.kv_rank + self.rot_dim

    @property
    def q_head(self) -> int:
        return self.nope_dim + self.rot_dim

    @property
    def gate_cols(self) -> int:
        return {"head": self.heads, "element": self.heads * self.v_dim, "none": 0}[self.gate]

    def rope_table(self, n_pos: int, device) -> torch.Tensor:
        if self.rotary is not None:
            return self.rotary.table(n_pos, device)
        return build_rope_table(n_pos, self.rot_dims, self.rot_base, device)

    def rot_order(self) -> torch.Tensor:
        """Where every dimension of the stored rotated part sits in the checkpoint's: the identity, or for the "half" layout
        (i paired with i + rot_dims/2) the order that puts the two of a pair side by side."""
        order = list(range(self.rot_dim))
        if self.rot_layout == "half":
            half = self.rot_dims // 2
            for i in range(half):
                order[2 * i], order[2 * i + 1] = i, i + half
        return torch.tensor(order, dtype=torch.long)


def build_rope_table(n_pos: int, rot_dims: int, base: float, device) -> torch.Tensor:
    """``[n_pos, rot_dims / 2, 2]`` fp32 (cos, sin) of ``pos * base^(-2i / rot_dims)``; angles formed in float64 so that the
    table is exact to fp32 rounding at any position."""
    i = torch.arange(rot_dims // 2, dtype=torch.float64)
    freq = torch.pow(torch.tensor(float(base), dtype=torch.float64), -2.0 * i / max(rot_dims, 1))
    ang = torch.arange(n_pos, dtype=torch.float64)[:, None] * freq[None]
    if rot_dims == 0:                       # nothing turns: a table the kernels never index, but a valid address
        return torch.zeros((n_pos, 1, 2), dtype=torch.float32, device=device)
    return torch.stack((ang.cos(), ang.sin()), dim=-1).float().contiguous().to(device)


class LatentAttention(nn.Module):
    def __init__(self, spec: LatentAttentionSpec, dtype: torch.dtype, device, project: bool = True) -> None:
        super().__init__()
        s = self.spec = spec
        self.owns_cache = s.kv_from is None
        self.q_cols = s.heads * s.q_head
        self.q_in = s.q_rank if s.q_rank is not None else self.q_cols       # what the input projection holds for the queries
        self.gate_col0 = self.q_in
        self.kv_col0 = self.q_in + s.gate_cols
        n_in = self.kv_col0 + (s.row if self.owns_cache else 0)
        self.n_in = n_in
        n_in = (n_in + 7) // 8 * 8          # rows of zeros up to a multiple of 8: the library's fast GEMMs want aligned outputs
        kw = dict(dtype=dtype, device=device)
        # [W_q | W_dq; W_g; W_dkv]; project False: the layer keeps the input and output projections, stacked with others
        self.w_in = nn.Parameter(torch.empty((n_in, s.width), **kw), requires_grad=False) if project else None
        self.q_norm = nn.Parameter(torch.ones(s.q_rank, dtype=torch.float32, device=device), requires_grad=False) \
            if s.q_rank is not None else None
        self.w_uq = nn.Parameter(torch.empty((self.q_cols, s.q_rank), **kw), requires_grad=False) if s.q_rank is not None else None
        self.w_uk = nn.Parameter(torch.empty((s.heads, s.nope_dim, s.kv_rank), **kw), requires_grad=False)
        self.w_uv_t = nn.Parameter(torch.empty((s.heads, s.kv_rank, s.v_dim), **kw), requires_grad=False)
        self.w_o = nn.Parameter(torch.empty((s.width, s.heads * s.v_dim), **kw), requires_grad=False) if project else None
        self.kv_norm = nn.Parameter(torch.ones(s.kv_rank, dtype=torch.float32, device=device), requires_grad=False) \
            if self.owns_cache else None

    @property
    def out_cols(self) -> int:
        """What ``attend`` puts out per token."""
        return self.spec.heads * self.spec.v_dim

    def state_shapes(self, B: int):
        return []

    def cache_shapes(self, B: int, ring: int):
        return [(B, ring, self.spec.row)] if self.owns_cache else []

    def _q_rows(self, w: torch.Tensor) -> torch.Tensor:
        """The rotated part of every head's query rows in the stored order."""
        s = self.spec
        w = w.reshape(s.heads, s.q_head, -1)
        return torch.cat([w[:, : s.nope_dim], w[:, s.nope_dim:][:, s.rot_order()]], dim=1).reshape(self.q_cols, -1)

    def in_rows(self, get) -> torch.Tensor:
        """The rows of the input projection."""
        s = self.spec
        parts = [get("dq")] if s.q_rank is not None else [self._q_rows(get("q"))]
        if s.gate != "none":
            parts.append(get("g"))
        if self.owns_cache:
            dkv = get("dkv")
            parts.append(torch.cat([dkv[: s.kv_rank], dkv[s.kv_rank:][s.rot_order()]], dim=0))
        return torch.cat(parts, dim=0)

    def load(self, get) -> None:
        """``get(suffix)`` returns the tensor '<layer>.mix.<suffix>' ([out, in] for the Linears)."""
        s = self.spec
        if self.w_in is not None:
            self.w_in.zero_()
            self.w_in[: self.n_in].copy_(self.in_rows(get))
            self.w_o.copy_(get("o"))
        if s.q_rank is not None:
            self.q_norm.copy_(get("dq.norm").float())
            self.w_uq.copy_(self._q_rows(get("uq")))
        self.w_uk.copy_(get("uk").reshape(s.heads, s.nope_dim, s.kv_rank))
        self.w_uv_t.copy_(get("uv").reshape(s.heads, s.v_dim, s.kv_rank).transpose(1, 2))
        if self.owns_cache:
            self.kv_norm.copy_(get("dkv.norm").float())

    def forward(self, x_act: torch.Tensor, B: int, T: int, pos_ids: torch.Tensor, rope: torch.Tensor, cache: torch.Tensor,
                splits: int = 1, end: Optional[int] = None) -> torch.Tensor:
        """x_act ``[B*T, width]`` -> ``[B*T, width]``; ``cache`` ``[B, S, row]`` is this layer's or its source's (already
        appended to by the source in this step).  ``end``: as in ``attend``."""
        at, rows = (self._takes_step(x_act, B, cache), 0) if T == 1 else (None, 0)
        if not at and (T > 1 or B > STEP_MAX_ROWS) and self.w_in is not None:
            rows = self._layer_form(B, T, cache, splits, end)
            if rows is not None and N.layer_rows(B * T, self.w_in.numel() + self.w_o.numel(), LAYER_MAX_PRODUCTS, LAYER_MAX_WEIGHTS):
                at = self._takes_layer(x_act, B * T, cache, "ll_latent_layer")
        if at:
            return self._one_call(at, x_act, B, T, pos_ids, rope, cache, rows, splits)
        return F.linear(self.attend(F.linear(x_act, self.w_in), B, T, pos_ids, rope, cache, splits, end=end), self.w_o)

    def _takes_step(self, x_act: torch.Tensor, B: int, cache: torch.Tensor):
        """One token of one or two sequences."""
        return self._takes_layer(x_act, B, cache, "ll_latent_layer") if 1 <= B <= STEP_MAX_ROWS else None

    def _layer_form(self, B: int, T: int, cache: torch.Tensor, splits: int, end: Optional[int]) -> Optional[int]:
        """Cache rows per sequence that a call of several rows expands per head, 0: queries stay in latent space; ``None``: not in one call.  The form is
        the one that the separate calls would take."""
        s, S = self.spec, cache.shape[1]
        if T >= EXPAND_MIN_TOKENS and splits == 1:
            first, rows = self._visible(T, S, end)
            if s.v_dim % 64 or not (first is None or (first == 0 and (B == 1 or rows == S))):
                return None
            if s.scale > 0 and self._expand_pays(B, T, rows) and cache.data_ptr() % 16 == 0 and _expanded_supported(
                    s.nope_dim, s.rot_dim, s.v_dim, s.kv_rank, self.w_in.shape[0], s.q_head, s.heads * s.v_dim):
                return rows
        return 0 if B * T * s.heads <= LATENT_MAX_ROW_HEADS and self.w_in.numel() + self.w_o.numel() <= LATENT_MAX_WEIGHTS else None

    def _expand_pays(self, B: int, T: int, rows: int) -> bool:
        s = self.spec
        return rows <= EXPAND_MAX_SLOTS_PER_TOKEN * T and 2 * B * rows * s.heads * (s.nope_dim + s.v_dim) <= EXPAND_MAX_BYTES

    def _takes_layer(self, x_act: torch.Tensor, M: int, cache: torch.Tensor, entry: str):
        """``M`` bf16 rows, plain queries, at most a gate per head: the whole layer in one call, if its weights are
        what the layer was built with.  Their addresses, or ``None``."""
        s, p = self.spec, self._parameters
        w = p.get("w_in")
        if not (w is not None and s.q_rank is None and s.gate != "element" and x_act.is_cuda
                and x_act.dtype is torch.bfloat16 and cache.dtype is torch.bfloat16 and cache.is_contiguous()
                and cache.get_device() == x_act.get_device() and x_act.shape == (M, s.width) and s.kv_rank <= 1024 and s.nope_dim <= 1024
                and N.has(entry)):
            return None
        n_in = w.shape[0]
        if n_in < self.n_in or (s.width | s.kv_rank | s.v_dim | n_in) % 8:
            return None
        return N.step_rows(x_act, (w, p.get("w_uk"), p.get("w_uv_t"), p.get("w_o")),
                           ((n_in, s.width), (s.heads, s.nope_dim, s.kv_rank), (s.heads, s.kv_rank, s.v_dim), (s.width, s.heads * s.v_dim)))

    def _one_call(self, at, x_act: torch.Tensor, B: int, T: int, pos_ids: torch.Tensor, rope: torch.Tensor, cache: torch.Tensor, rows: int,
                  splits: int) -> torch.Tensor:
        s, p = self.spec, self._parameters
        x, w_in, w_uk, w_uv_t, w_o = at
        n_in = p["w_in"].shape[0]
        norm = None if not self.owns_cache else p["kv_norm"] if "kv_norm" in p else self.kv_norm
        out = torch.empty_like(x_act)
        scratch = x_act.new_empty(_layer_scratch_bytes(B, T, n_in, s.heads, s.nope_dim, s.rot_dim, s.kv_rank, s.v_dim, rows, splits) // 2)  # (whole pieces)
        N.call("ll_latent_layer", x, w_in, n_in, w_uk, w_uv_t, w_o, N.ptr(norm), float(s.eps), N.ptr(rope), N.ptr(pos_ids), N.ptr(cache), B, T, s.width,
               s.heads, s.nope_dim, s.rot_dim, s.rot_dims, s.v_dim, s.kv_rank, cache.shape[1], rows, self.gate_col0 if s.gate == "head" else -1,
               self.kv_col0, s.window if s.window is not None else 0, float(s.scale), splits, 2 if s.exact_weights else 1, N.ptr(out),
               N.ptr(scratch), N.stream())
        return out

    def attend(self, proj: torch.Tensor, B: int, T: int, pos_ids: torch.Tensor, rope: torch.Tensor, cache: torch.Tensor,
               splits: int = 1, out: Optional[torch.Tensor] = None, end: Optional[int] = None) -> torch.Tensor:
        """``proj``: the input projection's output (this mixer's columns first).  Returns the gated heads
        ``[B*T, heads * v_dim]`` before the output projection, in ``out`` (a column slice) when given.  ``end``: the position after
        the step's last, when the host knows it (positions are consecutive); then only rows that some query sees are expanded,
        else every slot of the cache."""
        s = self.spec
        M = B * T
        dt = N.dtype_code(proj.dtype)
        st = N.stream()
        dev = proj.device
        S = cache.shape[1]
        if self.owns_cache:
            N.call("ll_latent_kv_append", N.ptr(proj), dt, proj.stride(0), self.kv_col0, N.ptr(self.kv_norm), float(s.eps),
                   N.ptr(rope), N.ptr(pos_ids), N.ptr(cache), B, T, s.kv_rank, s.rot_dim, s.rot_dims, S, st)
        if s.q_rank is not None:
            cq = torch.empty((M, s.q_rank), dtype=proj.dtype, device=dev)
            N.call("ll_row_norm", N.ptr(proj), proj.stride(0), N.ptr(self.q_norm), float(s.eps), N.ptr(cq), s.q_rank, dt, M, s.q_rank, st)
            q = F.linear(cq, self.w_uq)                                       # [M, heads * q_head]
        else:
            q = proj
        first, rows = self._visible(T, S, end)
        if T >= EXPAND_MIN_TOKENS and splits == 1 and self._takes_expanded(q, out, cache, B, T, rows):
            o = self._attend_expanded(proj, q, B, T, pos_ids, rope, cache, out, first, rows)
        else:
            o = self._attend_latent(proj, q, B, T, pos_ids, rope, cache, splits, out)
        if s.gate == "element":
            N.call("ll_sigmoid_gate_mul", N.ptr(o), o.stride(0), N.ptr_at(proj, self.gate_col0), proj.stride(0), N.ptr(o), o.stride(0), dt,
                   M, s.heads * s.v_dim, st)
        elif s.gate == "head" and s.q_rank is not None:
            raise NotImplementedError("a gate per head beside latent queries")
        return o

    def _visible(self, T: int, S: int, end: Optional[int]):
        """(first position, rows) that the queries of a step of ``T`` tokens up to position ``end`` see; (None, S) when that is not known."""
        if end is None:
            return None, S
        first = 0 if self.spec.window is None else max(0, end - T - self.spec.window + 1)
        return (first, end - first) if end - first <= S else (None, S)

    def _takes_expanded(self, q, out, cache, B: int, T: int, rows: int) -> bool:
        """Whether a step of several tokens expands ``rows`` cache rows per head (one up-projection of each) and attends over plain keys and
        values on the tcgen05 kernel: bf16, sizes that kernel takes, not too many rows for the queries.  Both sides measured (128 + 64
        dimensions, rank 512, graphed ``attend``, us): 16 heads, 16 tokens after 0 / 1000 positions 29 / 101 -> 21 / 39, 200 after 0 / 7000
        48 / 574 -> 27 / 192, 2048 after 0 734 -> 68; 64 heads, 16 after 1000 102 -> 50, 200 after 7000 1679 -> 267.  Rows that no query
        sees are not worth forming: with all of 8192 slots expanded, 150 tokens at position 0 took 41 -> 60 (16 heads) and 76 -> 146 (64)."""
        s = self.spec
        return (q.dtype == torch.bfloat16 and cache.dtype == torch.bfloat16 and s.scale > 0 and self._expand_pays(B, T, rows)
                and N.has("ll_latent_prompt_attn") and cache.is_contiguous() and (out is None or (out.stride(1) == 1 and out.data_ptr() % 16 == 0))
                and bool(N.call_ret("ll_latent_prompt_supported", s.nope_dim, s.rot_dim, s.v_dim, s.kv_rank, q.stride(0), s.q_head,
                                    s.heads * s.v_dim if out is None else out.stride(0)))
                and (q.data_ptr() | cache.data_ptr()) % 16 == 0)

    def _attend_expanded(self, proj, q, B: int, T: int, pos_ids, rope, cache, out, first: Optional[int], n: int) -> torch.Tensor:
        """``n`` rows per sequence from position ``first`` on, in the order of their positions; ``first`` None: the ring as it lies."""
        s = self.spec
        S = cache.shape[1]
        if out is None:
            out = torch.empty((B * T, s.heads * s.v_dim), dtype=proj.dtype, device=proj.device)
        rope_at = N.ptr(rope)
        if first is not None:
            a = first % S
            cache = cache[:, a: a + n] if a + n <= S else torch.cat([cache[:, a:], cache[:, : a + n - S]], dim=1)
            cache = cache.contiguous()                            # (one sequence whose rows do not wrap: a view)
            if first > 0:                                         # the kernel's positions count from the first row
                pos_ids, rope_at = pos_ids - first, N.ptr_at(rope, first * s.rot_dims)
        c = cache.view(B * n, s.row)[:, : s.kv_rank]
        k = F.linear(c, self.w_uk.view(s.heads * s.nope_dim, s.kv_rank))                # [B * n, heads * nope]
        v = torch.bmm(c.expand(s.heads, B * n, s.kv_rank), self.w_uv_t)                 # [heads, B * n, v_dim]
        q_rot = torch.empty((B * T, s.heads, s.rot_dim), dtype=q.dtype, device=q.device)
        gate = N.ptr_at(proj, self.gate_col0) if s.gate == "head" and s.q_rank is None else None
        N.call("ll_latent_prompt_attn", N.ptr(q), q.stride(0), s.nope_dim, s.q_head, gate, proj.stride(0), rope_at, N.ptr(pos_ids),
               N.ptr(k), k.stride(0), s.nope_dim, N.ptr(v), s.v_dim, B * n * s.v_dim, N.ptr(cache), N.ptr(q_rot), N.ptr(out), out.stride(0),
               B, T, s.heads, s.kv_rank, s.rot_dim, s.rot_dims, s.v_dim, n, s.window if s.window is not None else 0, float(s.scale),
               2 if s.exact_weights else 1, N.stream())
        return out

    def _attend_latent(self, proj, q, B: int, T: int, pos_ids, rope, cache, splits: int, out) -> torch.Tensor:
        s = self.spec
        M, S, dev = B * T, cache.shape[1], proj.device
        q_nope = q[:, : self.q_cols].view(M, s.heads, s.q_head)[:, :, : s.nope_dim].transpose(0, 1)   # [H, M, nope] view
        q_lat = torch.bmm(q_nope, self.w_uk)                                  # [H, M, kv_rank]
        o_lat = torch.empty_like(q_lat)
        scratch = None
        if splits > 1:
            scratch = torch.empty(N.call_ret("ll_latent_attn_scratch_bytes", M, s.heads, s.kv_rank, splits) // 4,
                                  dtype=torch.float32, device=dev)
        head_gate = self.gate_col0 if (s.gate == "head" and s.q_rank is None) else -1
        N.call("ll_latent_attn_terms", N.ptr(q_lat), M * s.kv_rank, s.kv_rank, N.ptr(q), q.stride(0), s.nope_dim, s.q_head,
               head_gate, N.ptr(rope), N.ptr(pos_ids), N.ptr(cache), N.ptr(o_lat), M * s.kv_rank, s.kv_rank, N.dtype_code(proj.dtype), B, T,
               s.heads, s.kv_rank, s.rot_dim, s.rot_dims, S, s.window if s.window is not None else 0, float(s.scale), splits,
               2 if s.exact_weights else 1, N.ptr(scratch), N.stream())
        if out is None:
            return torch.bmm(o_lat, self.w_uv_t).transpose(0, 1).reshape(M, s.heads * s.v_dim)
        torch.bmm(o_lat, self.w_uv_t, out=out.view(M, s.heads, s.v_dim).transpose(0, 1))   # the heads' products land in the rows
        return out
