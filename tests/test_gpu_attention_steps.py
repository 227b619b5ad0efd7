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
