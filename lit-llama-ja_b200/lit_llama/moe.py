"""Mixture-of-experts feed-forward with an optional always-on shared expert; the experts are gated linear units or plain
squared-relu layers.

    z = W_r h + b  (fp32)      the ``top`` largest logits choose the experts
    weights: softmax over the chosen logits (``score`` "chosen"), or the chosen entries of the softmax over ALL experts
             divided by their sum + 1e-20 (``score`` "all"), or, with scores sigmoid(z), the chosen scores divided by
             their sum + 1e-20 (``score`` "sigmoid"), where score + ``correction`` (a learned number per expert) makes the
             choice and the score alone the weight; in every case times ``weight_scale``
    groups:  the experts form ``groups`` equal groups of neighbours; only experts of the ``keep_groups`` groups with the
             largest group score can be chosen (its best expert, or the sum of its two best: ``group_top``)
    expert(h) = W_down( g * sigmoid(alpha * g) * (u + up_shift) ),  g = min(W_gate h, limit),  u = clamp(W_up h, -limit, limit)
                (limit inf, alpha 1, up_shift 0: the plain silu-gated unit), or W_down relu(W_up h)^2 (``unit`` "relu2")
    y = sum_k w_k expert_k(h)  +  [sigmoid(w_sg . h) *] shared(h)

The experts' weights are stacked ([X, 2 ff, width] for [gate; up] or [X, ff, width] for up alone, [X, width, ff] for down) and run as two grouped GEMMs
over the (token, choice) pairs sorted by expert; counts, offsets and the permutation never leave the device, so a step
is one fixed launch sequence.  More than a few bfloat16 tokens go through ``ll_moe_prompt``: the router, the sort, the gathered rows, both
projections on the tcgen05 tensor cores with the shared expert's tiles among the experts' (the activation is the first one's epilogue), and the
combination, six kernels under programmatic launches.  A few tokens go through ``ll_moe_step``.  What neither takes (fp32, other layouts, weights
that want a gradient) runs as separate calls: grouped GEMMs that take rows in place or, with rows that TMA can tile, the tcgen05 ones, and
the shared expert as dense library GEMMs with its gate logit as one more output row.
"""
from __future__ import annotations

import functools
import os
from dataclasses import dataclass
from typing import Optional

import torch
import torch.nn as nn
from torch.nn import functional as F

from . import _native as N
from .feed_forward import glu_unit, relu_squared_

# the tcgen05 path: at least this many (token, choice) rows in the step, and on average per expert.  Graphed, us, mma.sync / tcgen05: 32 experts of
# 2048 x 1024, four chosen, a shared one, 9 tokens 109 / 88, 64 119 / 104, 300 164 / 112, 2048 527 / 185; 16 of 1024 x 768, two chosen 49 / 39,
# 51 / 42, 74 / 48, 165 / 77; 16 of 1024 x 1024, four chosen, none shared, 9 tokens 43 / 45, 64 69 / 44.  Fewer rows are the steps of a few tokens.
TC_MIN_ROWS = int(os.environ.get("LLB200_MOE_TC_MIN_ROWS", "8"))
TC_MIN_ROWS_PER_EXPERT = float(os.environ.get("LLB200_MOE_TC_MIN_ROWS_PER_EXPERT", "0.25"))


def tc_least_rows(size: int, experts: int, shared: bool) -> int:
    """Rows per expert from which the tcgen05 kernels take experts of ``size`` = width x ff numbers.  A tile is 256 weight rows whatever the tokens, so
    many small experts with a few rows each are the mma.sync kernels' (16-row tiles, a CTA each) unless a shared expert's products come with them.
    Graphed, us, mma.sync / tcgen05 at 2, 8, 16 and 64 rows an expert, four chosen, none shared: 32 experts of 512 x 256 25 / 28, 28 / 28, 37 / 28, 44 / 31,
    of 1024 x 512 40 / 46, 42 / 46, 64 / 47, 83 / 53, of 1024 x 768 56 / 57, 59 / 58, 79 / 58, 91 / 64; 128 of 512 x 256 48 / 48, 58 / 68, 72 / 68,
    105 / 82, of 1024 x 256 73 / 76, 87 / 95, 106 / 96, 165 / 114, of 1024 x 768 135 / 128, 163 / 155, 203 / 157, 292 / 180; with a shared one of 256,
    128 of 1024 x 256 85 / 81, 98 / 95, 116 / 97, 174 / 120.  Smaller still, 256 of 256 x 64: 39 / 52, 48 / 68, 59 / 73, 114 / 132 (through the separate
    calls 156 from 48 rows on), with a shared one 47 / 53, 57 / 69, 69 / 74, 125 / 136.  Eight experts: 23 / 24 to 29 / 27 at 8 rows."""
    if experts > 64 and size <= 1 << 16:
        return 48
    return 16 if experts >= 16 and size < 3 << 18 and not shared else 0


STEP_MAX_TOKENS, STEP_SMALL_EXPERT = 8, 1 << 22       # tokens of a step; ff * width
STEP_REPEAT_BYTES = 300 << 20                         # of weights that a step reads for one token after another


@functools.lru_cache(maxsize=1024)
def step_pays(M: int, width: int, ff: int, shared_ff: int, experts: int, top: int, branches: int) -> bool:
    """Whether ``M`` tokens go through ``ll_moe_step``: sizes that it takes, and no fewer microseconds in the grouped kernels.

    A step reads a choice's weights for its token alone, the grouped kernels read an expert's once for all of its tokens and take 40 to 60 us
    more around that.  So what counts is what is read again: the choices less the distinct experts they can be expected to name, times an
    expert's bytes; 300 MB of it are those 40 us.  Graphed, us, grouped / step (repeated MB): experts of 4096 x 1024, 16 of them and four
    chosen, 6 tokens 106 / 99 (273), 8 tokens 107 / 127 (443); 32 and four, 8 tokens 158 / 139 (277); 64 and eight, 5 tokens 197 / 180 (222),
    6 tokens 205 / 211 (320); of 2048 x 2048 the same to 5 us; of 2048 x 1024, 64 and eight, 8 tokens 160 / 143 (277); of 4096 x 2048, 16 and
    four, 4 tokens 173 / 136 (255).  More than four tokens of larger experts keep the grouped kernels: 16 and four at 6 tokens 179 / 198, 32
    and four at 8 tokens 247 / 263."""
    most = STEP_MAX_TOKENS if ff * width <= STEP_SMALL_EXPERT else STEP_MAX_TOKENS // 2
    if not 1 <= M <= most or not N.has("ll_moe_step") or not N.call_ret("ll_moe_step_supported", M, width, ff, shared_ff):
        return False
    distinct = experts * (1.0 - (1.0 - top / experts) ** M)
    return (M * top - distinct) * (branches + 1) * ff * width * 2 <= STEP_REPEAT_BYTES


@functools.lru_cache(maxsize=1024)
def _step_scratch_bytes(M: int, experts: int, top: int, ff: int, shared_ff: int) -> int:
    return N.call_ret("ll_moe_step_scratch_bytes", M, experts, top, ff, shared_ff)


@dataclass
class MoESpec:
    width: int
    experts: int
    top: int
    ff: int
    limit: float
    shared_ff: Optional[int] = None      # None: no shared expert
    shared_limit: Optional[float] = None
    shared_gate: bool = True             # the shared expert is scaled by sigmoid(w_sg . h)
    router_bias: bool = True
    alpha: float = 1.702                 # slope inside the sigmoid of the gated unit
    up_shift: float = 1.0                # the up branch enters as (u + up_shift): 1 or 0
    score: str = "chosen"                # "chosen": softmax over the chosen logits; "all": over all experts, renormalised;
                                         # "sigmoid": sigmoid of every logit, renormalised over the chosen
    groups: int = 1                      # equal groups of neighbouring experts
    keep_groups: int = 1                 # groups whose experts can be chosen (groups == 1: all)
    group_top: int = 1                   # a group's score: its largest choice score (1) or the sum of its two largest (2)
    correction: bool = False             # a learned number per expert added to the score for the choice alone ("sigmoid")
    weight_scale: float = 1.0            # the experts' weights are multiplied by this
    unit: str = "glu"                    # "glu", or "relu2": experts without a gate branch, the square of relu


def glu_clamp(gu: torch.Tensor, ff: int, limit: float, alpha: float) -> torch.Tensor:
    """The clamped gated unit with the up branch shifted by 1."""
    return glu_unit(gu, ff, limit, alpha, 1.0)


_SCORES = {"chosen": 0, "all": 1, "sigmoid": 2}


class MoE(nn.Module):
    def __init__(self, spec: MoESpec, dtype: torch.dtype, device) -> None:
        super().__init__()
        s = self.spec = spec
        if not 0 < s.top <= s.experts:
            raise ValueError(f"top {s.top} of {s.experts} experts")
        if s.up_shift not in (0.0, 1.0) or s.score not in _SCORES or s.unit not in ("glu", "relu2") or s.group_top not in (1, 2):
            raise ValueError(f"up_shift {s.up_shift} (0 or 1), score {s.score!r} ({sorted(_SCORES)}), unit {s.unit!r} ('glu' or 'relu2'), "
                             f"group_top {s.group_top} (1 or 2)")
        if s.correction and s.score != "sigmoid":
            raise ValueError("a correction of the choice goes with sigmoid scores")
        if s.groups < 1 or s.experts % s.groups or not 1 <= s.keep_groups <= s.groups \
                or s.top > s.keep_groups * (s.experts // s.groups):
            raise ValueError(f"{s.experts} experts in {s.groups} groups, {s.keep_groups} kept, cannot give {s.top} choices")
        self.up_mode = 3 if s.unit == "relu2" else 1 if s.up_shift == 1.0 else 2      # of the first grouped GEMM
        branches = 1 if s.unit == "relu2" else 2
        kw = dict(dtype=dtype, device=device)
        f32 = dict(dtype=torch.float32, device=device)
        self.w_router = nn.Parameter(torch.empty((s.experts, s.width), **f32), requires_grad=False)
        self.b_router = nn.Parameter(torch.zeros(s.experts, **f32), requires_grad=False) if s.router_bias else None
        self.correction = nn.Parameter(torch.zeros(s.experts, **f32), requires_grad=False) if s.correction else None
        self.w_gu = nn.Parameter(torch.empty((s.experts, branches * s.ff, s.width), **kw), requires_grad=False)
        self.w_down = nn.Parameter(torch.empty((s.experts, s.width, s.ff), **kw), requires_grad=False)
        if s.shared_ff:
            # [gate; up; sg] (no gate rows for relu2), zero rows up to a multiple of 8
            rows = (branches * s.shared_ff + (1 if s.shared_gate else 0) + 7) // 8 * 8
            self.shared_cols = branches * s.shared_ff
            self.w_shared_in = nn.Parameter(torch.empty((rows, s.width), **kw), requires_grad=False)
            self.w_shared_down = nn.Parameter(torch.empty((s.width, s.shared_ff), **kw), requires_grad=False)

    def load(self, get) -> None:
        """``get(suffix)`` returns the tensor '<layer>.mlp.<suffix>'."""
        s = self.spec
        self.w_router.copy_(get("router").float())
        if self.b_router is not None:
            self.b_router.copy_(get("router.b").float())
        if self.correction is not None:
            self.correction.copy_(get("correction").float())
        gated = s.unit == "glu"
        for e in range(s.experts):
            if gated:
                self.w_gu[e, : s.ff].copy_(get(f"e{e}.gate"))
            self.w_gu[e, self.w_gu.shape[1] - s.ff:].copy_(get(f"e{e}.up"))
            self.w_down[e].copy_(get(f"e{e}.down"))
        if s.shared_ff:
            f = s.shared_ff
            self.w_shared_in.zero_()
            n = self.shared_cols
            if gated:
                self.w_shared_in[:f].copy_(get("shared.gate"))
            self.w_shared_in[n - f:n].copy_(get("shared.up"))
            if s.shared_gate:
                self.w_shared_in[n:n + 1].copy_(get("shared.sg").reshape(1, s.width))
            self.w_shared_down.copy_(get("shared.down"))

    def route(self, x_act: torch.Tensor):
        """(expert_idx [M, top] int32, expert_w [M, top] fp32, offsets [X + 1], perm [M * top])."""
        s = self.spec
        M, dev = x_act.shape[0], x_act.device
        i32 = dict(dtype=torch.int32, device=dev)
        idx = torch.empty((M, s.top), **i32)
        w = torch.empty((M, s.top), dtype=torch.float32, device=dev)
        counts, rank = torch.empty(s.experts, **i32), torch.empty(M * s.top, **i32)
        offsets, perm = torch.empty(s.experts + 1, **i32), torch.empty(M * s.top, **i32)
        N.call("ll_moe_route_choice", N.ptr(x_act), N.dtype_code(x_act.dtype), N.ptr(self.w_router), N.ptr(self.b_router), M, s.width,
               s.experts, s.top, _SCORES[s.score], N.ptr(self.correction), float(s.weight_scale), s.groups,
               s.keep_groups if s.groups > 1 else 1, s.group_top, N.ptr(idx), N.ptr(w), N.ptr(counts), N.ptr(rank), N.ptr(offsets),
               N.ptr(perm), N.stream())
        return idx, w, offsets, perm

    def takes_tensor_cores(self, n_rows: int, x_act: torch.Tensor) -> bool:
        """Whether a step of ``n_rows`` (token, choice) rows runs its expert GEMMs on the tcgen05 kernels: bfloat16, rows
        that TMA can tile (16-byte multiples on 16-byte boundaries, the other kernels read any), and enough of them (``tc_least_rows``)."""
        s = self.spec
        return (x_act.dtype == torch.bfloat16 and s.width % 8 == 0 and s.ff % 8 == 0 and x_act.stride(0) % 8 == 0
                and n_rows >= TC_MIN_ROWS and n_rows >= max(TC_MIN_ROWS_PER_EXPERT, tc_least_rows(s.width * s.ff, s.experts, bool(s.shared_ff))) * s.experts
                and (x_act.data_ptr() | self.w_gu.data_ptr() | self.w_down.data_ptr()) % 16 == 0 and N.has("ll_moe_grouped_gemm_tc"))

    def _one_call(self, entry: str, at, x_act: torch.Tensor, M: int, scratch_bytes: int) -> torch.Tensor:
        """The whole layer through ``ll_moe_step`` or ``ll_moe_prompt``."""
        s, p = self.spec, self._parameters
        sff = s.shared_ff or 0
        x, w_gu, w_down, ws_in, ws_down = at if sff else (*at, None, None)
        router = p["w_router"] if "w_router" in p else self.w_router
        bias = p["b_router"] if "b_router" in p else self.b_router
        correction = p["correction"] if "correction" in p else self.correction
        out = torch.empty_like(x_act)
        scratch = x_act.new_empty(scratch_bytes // 2)          # (whole pieces of 128 bytes)
        N.call(entry, x, N.ptr(router), N.ptr(bias), N.ptr(correction), _SCORES[s.score], float(s.weight_scale), s.groups,
               s.keep_groups if s.groups > 1 else 1, s.group_top, w_gu, w_down, ws_in, ws_down, M, s.width, s.experts, s.top, s.ff, sff,
               1 if s.shared_gate else 0, self.up_mode, float(s.limit), float(s.alpha), float(s.shared_limit if s.shared_limit is not None else s.limit),
               N.ptr(out), N.ptr(scratch), N.stream())
        return out

    def _rows(self, x_act: torch.Tensor, M: int):
        """The addresses of dense bf16 rows and of weights that are what the module was built with, or ``None``."""
        s = self.spec
        branches = 1 if s.unit == "relu2" else 2
        if not (x_act.dtype is torch.bfloat16 and x_act.is_cuda and x_act.shape == (M, s.width)):
            return None
        p = self._parameters
        up, down = (s.experts, branches * s.ff, s.width), (s.experts, s.width, s.ff)
        if not s.shared_ff:
            return N.step_rows(x_act, (p.get("w_gu"), p.get("w_down")), (up, down))
        w = p.get("w_shared_in")
        if w is None or w.shape[0] < branches * s.shared_ff + (1 if s.shared_gate else 0):
            return None
        return N.step_rows(x_act, (p.get("w_gu"), p.get("w_down"), w, p.get("w_shared_down")),
                           (up, down, (w.shape[0], s.width), (s.width, s.shared_ff)))

    def _takes_step(self, x_act: torch.Tensor, M: int):
        """A few bf16 tokens (``step_pays``) in three launches: the rows' addresses, or ``None``."""
        s = self.spec
        if not step_pays(M, s.width, s.ff, s.shared_ff or 0, s.experts, s.top, 1 if s.unit == "relu2" else 2):
            return None
        return self._rows(x_act, M)

    def _takes_prompt(self, x_act: torch.Tensor, M: int):
        """More of them, that take the tcgen05 kernels, in one call: the rows' addresses, or ``None``."""
        s = self.spec
        if not (N.has("ll_moe_prompt") and N.call_ret("ll_moe_prompt_supported", M, s.width, s.experts, s.ff, s.shared_ff or 0)):
            return None
        return self._rows(x_act, M)

    def forward(self, x_act: torch.Tensor) -> torch.Tensor:
        s, M = self.spec, x_act.shape[0]
        at = self._takes_step(x_act, M) if M <= STEP_MAX_TOKENS else None
        if at:
            return self._one_call("ll_moe_step", at, x_act, M, _step_scratch_bytes(M, s.experts, s.top, s.ff, s.shared_ff or 0))
        tensor_cores = self.takes_tensor_cores(M * s.top, x_act)
        at = self._takes_prompt(x_act, M) if tensor_cores else None
        if at:
            return self._one_call("ll_moe_prompt", at, x_act, M, N.call_ret("ll_moe_prompt_scratch_bytes", M, s.width, s.experts, s.top, s.ff,
                                                                             s.shared_ff or 0))
        dev, dtype = x_act.device, x_act.dtype
        dt, st = N.dtype_code(dtype), N.stream()
        _, w, offsets, perm = self.route(x_act)
        n = M * s.top
        h = torch.empty((n, s.ff), dtype=dtype, device=dev)
        y = torch.empty((n, s.width), dtype=dtype, device=dev)
        if tensor_cores:
            xs = torch.empty((n, s.width), dtype=dtype, device=dev)
            N.call("ll_moe_gather_rows", N.ptr(x_act), x_act.stride(0), N.ptr(perm), s.top, n, s.width, N.ptr(xs), st)
            N.call("ll_moe_grouped_gemm_tc", N.ptr(xs), N.ptr(self.w_gu), N.ptr(offsets), N.ptr(perm), self.up_mode, n, s.experts, s.ff,
                   s.width, float(s.limit), float(s.alpha), N.ptr(h), s.ff, st)
            N.call("ll_moe_grouped_gemm_tc", N.ptr(h), N.ptr(self.w_down), N.ptr(offsets), N.ptr(perm), 0, n, s.experts, s.width, s.ff,
                   0.0, 0.0, N.ptr(y), s.width, st)
        else:
            N.call("ll_moe_grouped_gemm", N.ptr(x_act), x_act.stride(0), N.ptr(self.w_gu), N.ptr(offsets), N.ptr(perm), self.up_mode,
                   dt, n, s.top, s.experts, s.ff, s.width, float(s.limit), float(s.alpha), N.ptr(h), s.ff, st)
            N.call("ll_moe_grouped_gemm", N.ptr(h), s.ff, N.ptr(self.w_down), N.ptr(offsets), N.ptr(perm), 0, dt, n, s.top, s.experts,
                   s.width, s.ff, 0.0, 0.0, N.ptr(y), s.width, st)
        ys = gate = None
        gate_ld = 0
        if s.shared_ff:
            gu = F.linear(x_act, self.w_shared_in)
            if s.unit == "relu2":
                hs = relu_squared_(gu)[:, :s.shared_ff] if not s.shared_gate else relu_squared_(gu[:, :s.shared_ff].contiguous())
            else:
                hs = glu_unit(gu, s.shared_ff, s.shared_limit if s.shared_limit is not None else s.limit, s.alpha, s.up_shift)
            ys = F.linear(hs, self.w_shared_down)
            if s.shared_gate:
                gate, gate_ld = gu[:, self.shared_cols:], gu.stride(0)
        out = torch.empty((M, s.width), dtype=dtype, device=dev)
        N.call("ll_moe_combine", N.ptr(y), N.ptr(w), s.top, N.ptr(ys), s.width, N.ptr(gate), gate_ld, N.ptr(out), dt, M, s.width, st)
        return out
