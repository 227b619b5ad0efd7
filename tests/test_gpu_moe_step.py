"""Steps of a few tokens (one kernel for the first projections, one for the second with the combination) against float64 sums of the same bf16
numbers: every unit, shared experts with and without a gate, widths at the edges of the loads, and the route a module takes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@torch.no_grad()
def _module(width, X, top, ff, shared, unit, up_shift, gate, score, seed):
    from lit_llama.moe import MoE, MoESpec

    spec = MoESpec(width, X, top, ff, 1.5, shared or None, 1.1, shared_gate=gate, alpha=1.7, up_shift=up_shift, score=score, unit=unit, router_bias=score == "chosen")
    mix = MoE(spec, torch.bfloat16, "cuda")
    g = torch.Generator(device="cuda").manual_seed(seed)
    for p in mix.parameters():
        p.copy_(torch.randn(p.shape, generator=g, device="cuda") * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.1))
    return mix


def _unit(s, g, u, limit):
    if s.unit == "relu2":
        return u.clamp(min=0) ** 2
    g, u = g.clamp(max=limit), u.clamp(-limit, limit)
    return g * torch.sigmoid(s.alpha * g) * (u + s.up_shift)


@pytest.mark.parametrize("M", [1, 2, 3, 8])
@pytest.mark.parametrize("width,X,top,ff,shared", [(8, 3, 1, 8, 0), (72, 5, 2, 40, 24), (264, 4, 3, 1032, 16), (2048, 32, 4, 1024, 1536), (1024, 16, 2, 768, 1280),
                                                  (512, 12, 7, 64, 0)])
@pytest.mark.parametrize("unit,up_shift,gate,score", [("glu", 1.0, True, "chosen"), ("glu", 0.0, False, "sigmoid"), ("relu2", 1.0, True, "all")])
def test_step(M, width, X, top, ff, shared, unit, up_shift, gate, score):
    mix = _module(width, X, top, ff, shared, unit, up_shift, gate, score, M + width)
    s = mix.spec
    x = torch.empty((M, width), dtype=torch.bfloat16, device="cuda")
    x.copy_(torch.randn((M, width), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda"))
    assert mix._takes_step(x, M)
    got = mix(x).double()
    idx, w, _, _ = mix.route(x.contiguous())
    xd, want = x.double(), torch.zeros((M, width), dtype=torch.float64, device="cuda")
    bound = torch.zeros((M, width), dtype=torch.float64, device="cuda")

    def expert(w_in, w_out, n, m, limit, rounded):
        """(output, its error bound): h is rounded to bf16 (2^-9 of it), so is the output; ``rounded``: so are the unit's inputs, which may
        besides end on the other neighbour (2^-8 of each), and the unit's slope is at most 1.1 in the gate and the gate in the other branch"""
        gu = w_in.double() @ xd[m]
        g, u = gu[:n], gu[gu.shape[0] - n:]
        h = _unit(s, g, u, limit)
        err = h.abs() * 2.0 ** -9 + (xd[m].abs().sum() * 2.0 ** -22)
        if rounded:
            err = err + (2 * u.clamp(min=0) * u.abs() if s.unit == "relu2" else 1.1 * (u.clamp(-limit, limit) + s.up_shift).abs() * g.abs() + g.abs().clamp(max=limit) * u.abs()) * 2.0 ** -8
        y = w_out.double() @ h
        return y, w_out.double().abs() @ err + y.abs() * 2.0 ** -9

    for m in range(M):
        for c in range(top):
            y, e = expert(mix.w_gu[idx[m, c]], mix.w_down[idx[m, c]], ff, m, s.limit, False)
            want[m] += w[m, c].double() * y
            bound[m] += w[m, c].double().abs() * e
        if shared:
            n = mix.shared_cols
            y, e = expert(mix.w_shared_in[:n], mix.w_shared_down, shared, m, s.shared_limit, True)
            z = float(mix.w_shared_in[n].double() @ xd[m]) if gate else 0.0
            sg = 1.0 / (1.0 + 2.718281828459045 ** -z) if gate else 1.0
            want[m] += sg * y
            bound[m] += sg * e + (abs(z) * 2.0 ** -8 * 0.25 * y.abs() if gate else 0.0)
    bad = ~((got - want).abs() <= 1.1 * bound + want.abs() * 2.0 ** -8 + 1e-5)
    assert not bad.any(), (bad.nonzero()[:5], got[bad][:5], want[bad][:5], bound[bad][:5])


def test_route_of_a_module():
    """Nine tokens, odd widths, strided rows and rows off 16-byte boundaries take the grouped kernels, as before; the same numbers up to rounding."""
    mix = _module(256, 8, 2, 64, 32, "glu", 1.0, True, "chosen", 1)
    x = torch.randn((9, 256), generator=torch.Generator(device="cuda").manual_seed(0), device="cuda").to(torch.bfloat16)
    assert not mix._takes_step(x, 9) and mix._takes_step(x[:8], 8)
    a, b = mix(x)[:8].double(), mix(x[:8]).double()
    assert (a - b).norm() <= 0.01 * a.norm()
    shifted = torch.zeros(8 * 256 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(8, 256)
    assert not mix._takes_step(shifted, 8) and not mix._takes_step(torch.zeros((2, 512), dtype=torch.bfloat16, device="cuda")[:, :256], 2)
    wide = _module(4096, 2, 1, 2048, 0, "glu", 1.0, True, "chosen", 3)
    x = torch.zeros((5, 4096), dtype=torch.bfloat16, device="cuda")
    assert wide._takes_step(x[:4], 4) and not wide._takes_step(x, 5)
    assert not _module(36, 4, 2, 64, 0, "glu", 1.0, True, "chosen", 2)._takes_step(torch.zeros((2, 36), dtype=torch.bfloat16, device="cuda"), 2)


@pytest.mark.parametrize("name,how", [("w_gu", "shifted"), ("w_down", "shifted"), ("w_shared_in", "shifted"), ("w_shared_down", "shifted"),
                                      ("w_shared_in", "strided"), ("w_shared_down", "strided"), ("w_down", "plain"), ("w_shared_in", "plain")])
def test_weights_that_the_step_cannot_read(name, how):
    """Weights off 16-byte boundaries, a shared expert's in strided rows and tensors that are no parameters take the grouped kernels and dense
    layers: the same numbers up to rounding."""
    mix = _module(256, 8, 2, 64, 32, "glu", 1.0, True, "chosen", 5)
    x = torch.randn((3, 256), generator=torch.Generator(device="cuda").manual_seed(5), device="cuda").to(torch.bfloat16)
    assert mix._takes_step(x, 3)
    want = mix(x).double()
    w = getattr(mix, name).detach()
    if how == "shifted":
        new = torch.empty(w.numel() + 1, dtype=w.dtype, device="cuda")[1:].view(w.shape).copy_(w)
    elif how == "strided":
        new = torch.empty(w.shape[:-1] + (2 * w.shape[-1],), dtype=w.dtype, device="cuda")[..., : w.shape[-1]].copy_(w)
    else:
        new = w.clone()
    if how == "plain":
        delattr(mix, name)
        object.__setattr__(mix, name, new)
    else:
        setattr(mix, name, torch.nn.Parameter(new, requires_grad=False))
    assert not mix._takes_step(x, 3)
    assert (mix(x).double() - want).norm() <= 0.01 * want.norm()


@pytest.mark.parametrize("name", ["w_shared_in", "w_shared_down"])
@pytest.mark.parametrize("other", ["fp32", "cpu", "narrow"])
def test_shared_weights_of_another_kind_are_refused(name, other):
    """The dense layers refuse a shared expert of another dtype, on another device or of other widths, and so does the module."""
    mix = _module(256, 8, 2, 64, 32, "glu", 1.0, True, "chosen", 6)
    x = torch.ones((2, 256), dtype=torch.bfloat16, device="cuda")
    w = getattr(mix, name).detach()
    setattr(mix, name, torch.nn.Parameter(w.float() if other == "fp32" else w.cpu() if other == "cpu" else w[:, :-8].clone(), requires_grad=False))
    assert not mix._takes_step(x, 2)
    with pytest.raises(RuntimeError):
        mix(x)


@pytest.mark.parametrize("width,ff,shared", [(72, 40, 24), (264, 1032, 16), (2048, 1024, 1536)])
def test_infinite_weights_at_the_end_of_a_row(width, ff, shared):
    """A row's last weights are infinite: outputs are infinite where the grouped kernels' are, and no numbers nowhere else either."""
    mix = _module(width, 4, 2, ff, shared, "glu", 1.0, True, "chosen", 7)
    with torch.no_grad():
        mix.w_down[:, 1, -1], mix.w_down[:, 6, -2] = float("inf"), -float("inf")
        mix.w_shared_down[3, -1] = float("inf")
        mix.w_shared_in[mix.shared_cols, -1] = float("inf")
    x = torch.randn((2, width), generator=torch.Generator(device="cuda").manual_seed(7), device="cuda").to(torch.bfloat16)
    assert mix._takes_step(x, 2)
    got = mix(x).double()
    mix._takes_step = lambda *a: False
    want = mix(x).double()
    assert want.isinf().any() and torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()].sign(), want[want.isinf()].sign())
    ok = want.isfinite()
    assert (got[ok] - want[ok]).norm() <= 0.01 * want[ok].norm()
