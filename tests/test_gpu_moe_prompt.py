"""A mixture-of-experts layer for more than a few tokens: the one call and the separate calls beside it against float64 sums of the same bf16 numbers, at
the edges of the sort and of the tiles, and which of the two a module takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@torch.no_grad()
def _module(width, X, top, ff, shared=0, unit="glu", up_shift=1.0, gate=True, score="chosen", seed=0):
    from lit_llama.moe import MoE, MoESpec

    spec = MoESpec(width, X, top, ff, 1.5, shared or None, 1.1, shared_gate=gate, alpha=1.7, up_shift=up_shift, score=score, unit=unit, router_bias=score == "chosen")
    mix = MoE(spec, torch.bfloat16, "cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)
    for p in mix.parameters():
        p.copy_(torch.randn(p.shape, generator=g, device="cuda") * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.1))
    return mix


def _rows(M, width, seed=1):
    return torch.randn((M, width), generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(torch.bfloat16)


def _exact(mix, x):
    """(the layer in 64 bits for the choices that the router makes, a bound of its error).  The unit's result is rounded to bf16 (2^-9), so is a second
    projection's, and where the separate calls round the unit's inputs as well these may be 2^-8 off; the unit's slope is at most 1.1 in the gate
    and the gate itself in the other branch."""
    s = mix.spec
    idx, w, _, _ = mix.route(x)
    xd = x.double()

    def expert(w_in, w_out, n, rows, limit):
        z, mag = rows @ w_in.double().T, (rows.abs() @ w_in.double().abs().T) * (2.0 ** -24 * rows.shape[1])
        g, u, eg, eu = z[:, :n], z[:, -n:], mag[:, :n], mag[:, -n:]
        if s.unit == "relu2":
            h = u.clamp(min=0) ** 2
            e = 2 * u.abs() * (u.abs() * 2.0 ** -8 + eu)
        else:
            g, u = g.clamp(max=limit), u.clamp(-limit, limit) + s.up_shift
            h = g * torch.sigmoid(s.alpha * g) * u
            e = 1.1 * u.abs() * (g.abs() * 2.0 ** -8 + eg) + g.abs() * (u.abs() * 2.0 ** -8 + eu)
        e = e + h.abs() * 2.0 ** -8
        y = h @ w_out.double().T
        return y, e @ w_out.double().abs().T + y.abs() * 2.0 ** -8

    want, bound = torch.zeros_like(xd), torch.zeros_like(xd)
    for e in range(s.experts):
        m, c = (idx == e).nonzero(as_tuple=True)
        if m.numel():
            y, err = expert(mix.w_gu[e], mix.w_down[e], s.ff, xd[m], s.limit)
            want.index_add_(0, m, w[m, c].double()[:, None] * y)
            bound.index_add_(0, m, w[m, c].double().abs()[:, None] * err)
    if s.shared_ff:
        n = mix.shared_cols
        y, err = expert(mix.w_shared_in[:n], mix.w_shared_down, s.shared_ff, xd, s.shared_limit)
        z = xd @ mix.w_shared_in[n].double() if s.shared_gate else torch.full((len(x),), 1e9, dtype=torch.float64, device="cuda")
        sg = torch.sigmoid(z)[:, None]
        want, bound = want + sg * y, bound + sg * err + (z.abs() * 2.0 ** -8 * 0.25)[:, None] * y.abs() * bool(s.shared_gate)
    return want, 1.1 * bound + want.abs() * 2.0 ** -8 + 1e-6


def _check(mix, x, monkeypatch):
    """Both ways; how many rows an expert has."""
    from lit_llama import _native as N
    from lit_llama import moe as MOE

    entries = []
    one = MOE.MoE._one_call
    monkeypatch.setattr(MOE.MoE, "_one_call", lambda self, entry, *a: entries.append(entry) or one(self, entry, *a))
    want, bound = _exact(mix, x)
    got = mix(x)
    assert entries == ["ll_moe_prompt"] and N.call_ret("ll_moe_tc_error") == 0
    assert bool(((got.double() - want).abs() <= bound).all())
    assert torch.equal(got, mix(x))                         # the pairs of an expert come in no fixed order: no result depends on it
    monkeypatch.setattr(mix, "_takes_prompt", lambda *a: None)
    assert mix.takes_tensor_cores(x.shape[0] * mix.spec.top, x)
    other = mix(x)
    assert len(entries) == 2 and N.call_ret("ll_moe_tc_error") == 0
    assert bool(((other.double() - want).abs() <= bound).all())
    return torch.bincount(mix.route(x)[0].flatten(), minlength=mix.spec.experts)


# no shared expert, one with and without a gate; every unit; widths that are no whole tile
@pytest.mark.parametrize("M", [9, 70, 300])
@pytest.mark.parametrize("width,X,top,ff,shared", [(72, 5, 2, 40, 24), (264, 4, 3, 520, 0), (512, 32, 4, 256, 384)])
@pytest.mark.parametrize("unit,up_shift,gate,score", [("glu", 1.0, True, "chosen"), ("glu", 0.0, False, "sigmoid"), ("relu2", 1.0, True, "all")])
@torch.no_grad()
def test_layer(M, width, X, top, ff, shared, unit, up_shift, gate, score, monkeypatch):
    _check(_module(width, X, top, ff, shared, unit, up_shift, gate, score, M), _rows(M, width), monkeypatch)


@torch.no_grad()
def test_experts_that_no_token_chooses(monkeypatch):
    mix = _module(128, 6, 2, 64, 64)
    for e in (0, 3, 5):
        mix.b_router[e] = -50.0
    counts = _check(mix, _rows(200, 128), monkeypatch)
    assert counts[[0, 3, 5]].sum() == 0 and int(counts.min()) == 0


# up to 16384 pairs are sorted by one block, more are placed by a grid; one expert has most of them, or there are more experts than threads
@pytest.mark.parametrize("pairs,top,X", [(16383, 3, 7), (16384, 2, 32), (16385, 5, 40), (40000, 4, 6), (40000, 2, 1500), (16388, 4, 4), (16000, 2, 2600), (16000, 4, 4096)])
@torch.no_grad()
def test_sort_of_many_pairs(pairs, top, X, monkeypatch):
    from lit_llama import moe as MOE

    monkeypatch.setattr(MOE, "tc_least_rows", lambda *a: 0)
    mix = _module(32, X, top, 24, 16, seed=pairs)
    if X == 40:
        mix.b_router[7] = 9.0                               # an expert of nearly every token
    counts = _check(mix, _rows(pairs // top, 32), monkeypatch)
    assert int(counts.sum()) == pairs


@pytest.mark.parametrize("what", ["x", "w_gu", "w_down"])
@pytest.mark.parametrize("M", [9, 64])
@torch.no_grad()
def test_operands_off_16_byte_boundaries(M, what):
    """They take the kernels that read any address, and give the same numbers up to rounding."""
    mix, x = _module(64, 8, 2, 48, 32), _rows(M, 64)
    want = mix(x).double()

    def shifted(t):
        buf = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")
        return buf[1: 1 + t.numel()].view(t.shape).copy_(t)

    if what == "x":
        x = shifted(x)
    else:
        setattr(mix, what, torch.nn.Parameter(shifted(getattr(mix, what)), requires_grad=False))
    got = mix(x).double()
    assert float((got - want).norm()) <= 2.0 ** -6 * float(want.norm())


@pytest.mark.parametrize("X", [1, 319, 2048, 2049, 4097])
@pytest.mark.parametrize("mode,n", [(0, 264), (1, 72)])
def test_tiles_of_many_experts(X, mode, n):
    """The grouped products by the table that every CTA makes: less than an entry a thread, several, and entries of several experts."""
    from lit_llama import _native as N

    g, k = torch.Generator(device="cuda").manual_seed(X), 64
    counts = torch.randint(0, 4, (X,), generator=g, device="cuda")
    counts[X // 2], counts[X - 1] = 300, 1
    offsets = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), counts.cumsum(0)]).int()
    rows = int(offsets[-1])
    perm = torch.randperm(rows, generator=g, device="cuda").int()
    a, w = _rows(rows, k, X), torch.randn((X, (2 if mode else 1) * n, k), generator=g, device="cuda").mul_(k ** -0.5).to(torch.bfloat16)
    c = torch.full((rows, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    N.call("ll_moe_grouped_gemm_tc", N.ptr(a), N.ptr(w), N.ptr(offsets), N.ptr(perm), mode, rows, X, n, k, 1.5, 1.7, N.ptr(c), n, N.stream())
    assert N.call_ret("ll_moe_tc_error") == 0
    of = torch.repeat_interleave(torch.arange(X, device="cuda"), counts)
    z, mag = [torch.cat([torch.bmm(f(wd[of[i:i + 512]]), f(ad[i:i + 512])[..., None])[..., 0] for i in range(0, rows, 512)])
              for f in (lambda t: t, torch.abs) for ad, wd in [(a.double(), w.double())]]
    mag = mag * (k * 2.0 ** -24)
    if mode:                                               # the unit's slope is at most 1.1 in the gate and the gate itself in the other branch
        gate, up = z[:, :n].clamp(max=1.5), z[:, n:].clamp(-1.5, 1.5) + 1.0
        want = gate * torch.sigmoid(1.7 * gate) * up
        mag = 1.1 * up.abs() * mag[:, :n] + gate.abs() * mag[:, n:] + want.abs() * 2.0 ** -20
    else:
        want = z
    got = (c if mode else c[perm.long()]).double()
    assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + mag + 1e-30).all())
