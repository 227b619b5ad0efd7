"""The kernels around a LLaMA prompt's Linears in their 16-byte forms: rotation and cache append, residual with the norm after it, causal attention over
cache slots, positions.  References are float64 on the same bf16 numbers, rounded where the kernels round."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from lit_llama import _native as N


def _rand(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("B,T,nh,hs,S", [(1, 1, 1, 8, 4), (2, 7, 3, 40, 5), (1, 33, 4, 128, 64), (3, 3, 32, 64, 3), (1, 5, 3, 20, 8)])
def test_rotation_and_append(B, T, nh, hs, S):
    """Heads of whole 16-byte pieces, and (20) the general form; more tokens than slots leave the rest of the cache alone."""
    g = torch.Generator(device="cuda").manual_seed(hs)
    E, T = nh * hs, min(T, S)
    qkv, rope = _rand(g, B * T, 3 * E), torch.randn(50, hs // 2, 2, generator=g, device="cuda")
    pos = torch.randperm(50, generator=g, device="cuda")[:T].int()
    slots = torch.randperm(S, generator=g, device="cuda")[:T].int()
    q = torch.empty(B, nh, T, hs, dtype=torch.bfloat16, device="cuda")
    k, v = (torch.full((B, nh, S, hs), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    N.call("ll_rope_kv_append", N.ptr(qkv), N.ptr(rope), N.ptr(pos), N.ptr(slots), N.ptr(q), N.ptr(k), N.ptr(v), N.LL_BF16, B, T, nh, hs, S, N.stream())
    x = qkv.view(B, T, 3, nh, hs).permute(2, 0, 3, 1, 4).double()
    c = rope[pos.long()].double()
    a, b, co, si = x[..., 0::2], x[..., 1::2], c[..., 0], c[..., 1]
    turned = torch.stack((a * co - b * si, b * co + a * si), -1).flatten(-2)
    mag = torch.stack((a.abs() * co.abs() + b.abs() * si.abs(), b.abs() * co.abs() + a.abs() * si.abs()), -1).flatten(-2)
    near = lambda got, i: ((got.double() - turned[i]).abs() <= turned[i].abs() * 2.0 ** -8 + mag[i] * 2.0 ** -22).all()      # noqa: E731
    assert bool(near(q, 0)) and bool(near(k[:, :, slots.long()], 1)) and torch.equal(v[:, :, slots.long()].double(), x[2])
    rest = torch.ones(S, dtype=torch.bool, device="cuda")
    rest[slots.long()] = False
    assert bool((k[:, :, rest] == 7).all()) and bool((v[:, :, rest] == 7).all())


@pytest.mark.parametrize("rows,dim", [(1, 8), (3, 264), (63, 4096), (64, 4096), (65, 4104), (64, 8200), (2, 32768)])
def test_residual_and_norm(rows, dim):
    """The same numbers as the residual and the norm on their own, which round x + h, its square, the mean and every product."""
    g = torch.Generator(device="cuda").manual_seed(dim)
    x, h, w = _rand(g, rows, dim), _rand(g, rows, dim), _rand(g, dim)
    s, y, z = torch.empty_like(x), torch.empty_like(x), torch.empty_like(x)
    N.call("ll_add_rmsnorm", N.ptr(x), N.ptr(h), N.ptr(s), N.ptr(w), N.ptr(y), rows, dim, 1e-5, N.stream())
    assert torch.equal(s, x + h)
    N.call("ll_rmsnorm", N.ptr(s), N.ptr(w), N.ptr(z), N.LL_BF16, rows, dim, 1e-5, N.stream())
    assert torch.equal(y, z)


@pytest.mark.parametrize("B,T,H,hs,S,first", [(1, 2, 2, 64, 40, 0), (2, 130, 3, 128, 300, 17), (1, 300, 2, 40, 300, 0), (1, 20, 2, 64, 32, 25)])
def test_causal_attention_over_slots(B, T, H, hs, S, first):
    """As masked attention over the cache's slots; positions past the cache (the last case) see all of it.  The weights carry 16 bits, the result is
    rounded to bf16 once: half a unit of it (2^-9) and 2^-14 of the largest value."""
    g = torch.Generator(device="cuda").manual_seed(T)
    q, k, v = _rand(g, B, H, T, hs), _rand(g, B, H, S, hs), _rand(g, B, H, S, hs)
    pos64 = torch.arange(first, first + T, device="cuda")
    pos, slots, seen = torch.empty((3, T), dtype=torch.int32, device="cuda").unbind(0)
    N.call("ll_prompt_pos", N.ptr(pos), N.ptr(slots), N.ptr(seen), N.ptr(pos64), T, S, 2048, N.stream())
    assert torch.equal(pos.long(), pos64) and torch.equal(slots.long(), pos64 % S) and torch.equal(seen.long(), pos64.clamp(max=S - 1))
    y = torch.empty(B, T, H * hs, dtype=torch.bfloat16, device="cuda")
    N.call("ll_causal_attn", N.ptr(q), N.ptr(k), N.ptr(v), N.ptr(seen), N.ptr(y), B, T, H, hs, S, hs ** -0.5, N.stream())
    assert N.call_ret("ll_softmax_attn_tc_error") == 0
    mask = torch.arange(S, device="cuda")[None] <= pos64[:, None]
    sc = (q.double() @ k.double().transpose(2, 3) * hs ** -0.5).masked_fill(~mask, -math.inf)
    want = (torch.softmax(sc, -1) @ v.double()).transpose(1, 2).reshape(B, T, H * hs)
    assert bool(((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + float(v.abs().max()) * 2.0 ** -14).all())


@pytest.mark.parametrize("bad", [-1, 16])
def test_a_position_outside_the_table_is_reported(bad):
    pos64 = torch.tensor([3, bad, 5], device="cuda")
    out = torch.empty((3, 3), dtype=torch.int32, device="cuda")
    N.call("ll_prompt_pos", N.ptr(out[0]), N.ptr(out[1]), N.ptr(out[2]), N.ptr(pos64), 3, 8, 16, N.stream())
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="rotary table"):
        N.check_waits()
    assert int(out[0].min()) >= 0 and int(out[0].max()) < 16 and int(out[1].max()) < 8
    N.check_waits()                                        # reported once
