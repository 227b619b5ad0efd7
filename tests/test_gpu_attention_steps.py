"""One token of one or two sequences through a whole attention layer in one call, against the layer's separate calls with library products (the same
kernels between the projections, the same roundings; projections in another order of sums), for every kind of layer that takes it; the calls that
do not; and the projections' kernels at the edges of their loads, through their layers' sizes."""
import pytest
import torch
from torch.nn import functional as F

pytestmark = pytest.mark.gpu


@torch.no_grad()
def _fill(mix, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    for p in mix.parameters():
        p.copy_(torch.randn(p.shape, generator=g, device="cuda") * (p.shape[-1] ** -0.5) if p.dim() > 1 else 1.0 + 0.1 * torch.randn(p.shape, generator=g, device="cuda"))
    return mix


def _close(a, b, caches_a, caches_b):
    """The projections' sums differ in order: their bf16 outputs may end on the other neighbour, which travels through scores and products."""
    assert (a.double() - b.double()).norm() <= 0.01 * b.double().norm()
    for x, y in zip(caches_a, caches_b):
        assert (x.double() - y.double()).norm() <= 0.005 * y.double().norm()


@pytest.mark.parametrize("B", [1, 2])
@pytest.mark.parametrize("width,heads,nope,rot,v,rank,window,past", [(64, 2, 16, 8, 24, 40, None, 5), (2048, 16, 128, 64, 128, 512, 1024, 1500), (1024, 8, 64, 32, 64, 256, None, 70),
                                                                     (264, 3, 24, 16, 40, 72, 3, 9)])
@pytest.mark.parametrize("gate,splits,own", [("head", 1, True), ("none", 4, True), ("head", 3, False)])
def test_latent_step(B, width, heads, nope, rot, v, rank, window, past, gate, splits, own):
    from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec

    spec = LatentAttentionSpec(width=width, heads=heads, nope_dim=nope, rot_dim=rot, v_dim=v, kv_rank=rank, window=window, scale=(nope + rot) ** -0.5,
                               gate=gate, kv_from=None if own else 0)
    mix = _fill(LatentAttention(spec, torch.bfloat16, "cuda"), B + width)
    g = torch.Generator(device="cuda").manual_seed(past)
    x = torch.randn((B, width), generator=g, device="cuda").to(torch.bfloat16)
    cache = torch.randn((B, past + 1, rank + rot), generator=g, device="cuda").to(torch.bfloat16)
    pos = torch.tensor([past], dtype=torch.int32, device="cuda")
    rope = spec.rope_table(past + 1, "cuda")
    other = cache.clone()
    assert mix._takes_step(x, B, cache)
    got = mix(x, B, 1, pos, rope, cache, splits)
    want = F.linear(mix.attend(F.linear(x, mix.w_in), B, 1, pos, rope, other, splits), mix.w_o)
    _close(got, want, [cache], [other])
    assert not mix._takes_step(x[:, :-8].contiguous(), B, cache) and not mix._takes_step(x.unsqueeze(1), B, cache)
    assert not mix._takes_step(x.float(), B, cache) and not mix._takes_step(x.repeat(3, 1), 3, cache)
    assert not mix._takes_step(torch.empty((B, 2 * width), dtype=torch.bfloat16, device="cuda")[:, :width], B, cache) or B == 1


@pytest.mark.parametrize("B", [1, 2])
@pytest.mark.parametrize("width,heads,kv_heads,dim,window,chunk,past", [(64, 4, 2, 16, None, None, 6), (2048, 16, 4, 128, None, None, 900), (1024, 8, 8, 64, 100, None, 300),
                                                                        (520, 5, 5, 96, None, 64, 130)])
@pytest.mark.parametrize("cap,gate,norm,sink,splits", [(50.0, True, False, False, 1), (0.0, False, True, True, 4), (0.0, True, False, True, 2)])
def test_softmax_step(B, width, heads, kv_heads, dim, window, chunk, past, cap, gate, norm, sink, splits):
    from lit_llama.rotary import RotarySpec
    from lit_llama.softmax_attention import SoftmaxAttention, SoftmaxAttentionSpec

    spec = SoftmaxAttentionSpec(width=width, heads=heads, kv_heads=kv_heads, dim=dim, vdim=dim, scale=dim ** -0.5, eps=1e-5, rotary=RotarySpec(dim // 2),
                                softcap=cap, window=window, chunk=chunk, gate=gate, qk_norm=norm, sink=sink)
    mix = _fill(SoftmaxAttention(spec, torch.bfloat16, "cuda"), B + width)
    g = torch.Generator(device="cuda").manual_seed(past)
    u = torch.randn((B, width), generator=g, device="cuda").to(torch.bfloat16)
    caches = [torch.randn((B, past + 1, kv_heads * dim), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]
    others = [c.clone() for c in caches]
    pos = torch.tensor([past], dtype=torch.int32, device="cuda")
    assert mix._takes_step(u, B, caches)
    got = mix(u, B, 1, pos, caches, None, splits)
    want = F.linear(mix.attend(F.linear(u, mix.w_in), B, 1, pos, others, None, splits), mix.w_o)
    _close(got, want, caches, others)
    assert not mix._takes_step(u[:, :-8].contiguous(), B, caches) and not mix._takes_step(u.unsqueeze(1), B, caches)
    assert not mix._takes_step(u.float(), B, caches) and not mix._takes_step(u.repeat(3, 1), 3, caches)


@pytest.mark.parametrize("M", [1, 2])
@pytest.mark.parametrize("width,heads,v", [(8, 1, 8), (264, 2, 16), (2056, 3, 24), (4096, 32, 128)])
def test_projections_against_64_bits(M, width, heads, v):
    """A layer whose one key is its own row: weights are 1, so the layer is its projections alone."""
    from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec

    spec = LatentAttentionSpec(width=width, heads=heads, nope_dim=8, rot_dim=8, v_dim=v, kv_rank=16, window=1, scale=0.25, gate="none", kv_from=0)
    mix = _fill(LatentAttention(spec, torch.bfloat16, "cuda"), M + width)
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, width), generator=g, device="cuda").to(torch.bfloat16)
    cache = torch.randn((M, 1, 24), generator=g, device="cuda").to(torch.bfloat16)
    got = mix(x, M, 1, torch.zeros(1, dtype=torch.int32, device="cuda"), spec.rope_table(1, "cuda"), cache, 1).double()
    o = torch.einsum("mr,hrv->mhv", cache[:, 0, :16].double(), mix.w_uv_t.double()).reshape(M, -1)
    want, size = o @ mix.w_o.double().t(), o.abs() @ mix.w_o.double().abs().t()
    # o is rounded to bf16 (2^-9 of each term, 2^-8 beside the other neighbour), the output once more
    assert ((got - want).abs() <= size * 2.0 ** -8 + want.abs() * 2.0 ** -8 + 1e-6).all()


def _latent(width=64, heads=2, nope=16, rot=8, v=24, rank=40):
    from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec

    spec = LatentAttentionSpec(width=width, heads=heads, nope_dim=nope, rot_dim=rot, v_dim=v, kv_rank=rank, window=None, scale=(nope + rot) ** -0.5)
    mix = _fill(LatentAttention(spec, torch.bfloat16, "cuda"), 3)
    args = dict(B=1, T=1, pos_ids=torch.tensor([4], dtype=torch.int32, device="cuda"), rope=spec.rope_table(8, "cuda"))
    return mix, args, lambda: torch.zeros((1, 8, rank + rot), dtype=torch.bfloat16, device="cuda")


def _softmax(width=64, heads=4, kv_heads=2, dim=16):
    from lit_llama.rotary import RotarySpec
    from lit_llama.softmax_attention import SoftmaxAttention, SoftmaxAttentionSpec

    spec = SoftmaxAttentionSpec(width=width, heads=heads, kv_heads=kv_heads, dim=dim, vdim=dim, scale=dim ** -0.5, eps=1e-5, rotary=RotarySpec(dim // 2))
    mix = _fill(SoftmaxAttention(spec, torch.bfloat16, "cuda"), 4)
    args = dict(B=1, T=1, pos_ids=torch.tensor([4], dtype=torch.int32, device="cuda"))
    return mix, args, lambda: [torch.zeros((1, 8, kv_heads * dim), dtype=torch.bfloat16, device="cuda") for _ in range(2)]


def _call(mix, x, args, held):
    return mix(x, args["B"], args["T"], args["pos_ids"], args["rope"], held, 1) if "rope" in args else mix(x, args["B"], args["T"], args["pos_ids"], held, None, 1)


LAYERS = [(_latent, ("w_in", "w_uk", "w_uv_t", "w_o")), (_softmax, ("w_in", "w_o"))]


@pytest.mark.parametrize("make,name", [(m, n) for m, names in LAYERS for n in names])
@pytest.mark.parametrize("other", ["fp32", "fp16", "cpu"])
def test_weights_of_another_kind_are_refused(make, name, other):
    """The dense layers refuse weights of another dtype or on another device than the step's rows, and so does the layer."""
    mix, args, held = make()
    x = torch.ones((1, 64), dtype=torch.bfloat16, device="cuda")
    assert mix._takes_step(x, 1, held())
    w = getattr(mix, name)
    new = w.detach().float() if other == "fp32" else w.detach().half() if other == "fp16" else w.detach().cpu()
    setattr(mix, name, torch.nn.Parameter(new, requires_grad=False))
    assert not mix._takes_step(x, 1, held())
    with pytest.raises(RuntimeError):
        _call(mix, x, args, held())


@pytest.mark.parametrize("make,names", LAYERS)
def test_weights_of_another_shape(make, names):
    """A narrower output projection is refused where its rows do not fit, and serves where they do, as a dense layer of its own."""
    mix, args, held = make()
    x = torch.randn((1, 64), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").to(torch.bfloat16)
    whole = _call(mix, x, args, held())
    w_o = mix.w_o.detach()
    mix.w_o = torch.nn.Parameter(w_o[:40].clone(), requires_grad=False)
    assert not mix._takes_step(x, 1, held())
    part = _call(mix, x, args, held())
    assert part.shape == (1, 40) and (part.double() - whole[:, :40].double()).norm() <= 0.01 * whole[:, :40].double().norm()
    mix.w_o = torch.nn.Parameter(w_o[:, :-8].clone(), requires_grad=False)
    assert not mix._takes_step(x, 1, held())
    with pytest.raises(RuntimeError):
        _call(mix, x, args, held())


@pytest.mark.parametrize("make,name", [(m, n) for m, names in LAYERS for n in names])
@pytest.mark.parametrize("how", ["shifted", "strided", "plain", "grad"])
def test_weights_that_the_step_cannot_read(make, name, how):
    """Weights off 16-byte boundaries or in strided rows, and tensors that are no parameters, go through the dense layers: the same numbers up to
    the order of sums.  So does a weight that a gradient is wanted for."""
    mix, args, held = make()
    x = torch.randn((1, 64), generator=torch.Generator(device="cuda").manual_seed(2), device="cuda").to(torch.bfloat16)
    want = _call(mix, x, args, held()).double()
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
        setattr(mix, name, torch.nn.Parameter(new, requires_grad=how == "grad"))
    assert not mix._takes_step(x, 1, held())
    got = _call(mix, x, args, held())
    assert got.requires_grad == (how == "grad" and name in ("w_uv_t", "w_o"))
    assert (got.detach().double() - want).norm() <= 0.01 * want.norm()


def _same_kinds(a, b):
    """Infinities of the same sign and no numbers in the same places, and numbers close to each other."""
    return torch.equal(a.isnan(), b.isnan()) and torch.equal(a.isinf(), b.isinf()) and torch.equal(a[a.isinf()].sign(), b[b.isinf()].sign()) \
        and bool(((a - b).abs()[a.isfinite()] <= 0.02 * b[b.isfinite()].abs().amax()).all())


@pytest.mark.parametrize("width", [64, 264, 2056])
@pytest.mark.parametrize("make,gate_row", [(_latent, lambda m: m.gate_col0 + 1), (_softmax, lambda m: m.cols["g"] + 3)])
def test_infinite_weights_at_the_end_of_a_row(make, gate_row, width):
    """A row's last weights are infinite and its length fills no whole round of the warp's loads: sums are infinite, or no numbers, exactly where the
    dense layers' are."""
    mix, args, held = make(width=width)
    x = torch.randn((1, width), generator=torch.Generator(device="cuda").manual_seed(width), device="cuda").to(torch.bfloat16)
    with torch.no_grad():
        mix.w_o[1, -1], mix.w_o[5, -3] = float("inf"), -float("inf")
        mix.w_in[gate_row(mix), -2] = float("inf")
        x[0, -2] = 1.0                       # (that gate is open)
    assert mix._takes_step(x, 1, held())
    got = _call(mix, x, args, held()).double()
    attend = (args["B"], args["T"], args["pos_ids"]) + ((args["rope"], held()) if "rope" in args else (held(),))
    want = F.linear(mix.attend(F.linear(x, mix.w_in), *attend), mix.w_o).double()
    assert want.isinf().any() and _same_kinds(got, want)
