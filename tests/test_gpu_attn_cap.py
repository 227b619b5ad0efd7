"""Prompt attention under a cap at the ends of what its weights can be: scores that a cap bounds have no running maximum, so weights lie between 2^-72 and 2^72
(a cap of 50) instead of being at most 2^8, and the sums they enter are fp32."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


# all scores at the cap, all at its negative, keys at either; values as large and as small as the sums hold with 300 keys (2^(127 - 72 - 9), 2^(-126 + 72 + 8)
# with the second terms of weights 2^-8 below the first), and beside a cap past the bound (56) what a maximum leaves room for
@pytest.mark.parametrize("cap,power", [(50.0, 44), (50.0, 0), (50.0, -44), (20.0, 80), (56.0, 100), (56.0, -60)])
@pytest.mark.parametrize("keys", ["top", "bottom", "mixed"])
@pytest.mark.parametrize("T,H,dim", [(300, 2, 64), (130, 3, 128)])
@torch.no_grad()
def test_scores_at_the_ends(cap, power, keys, T, H, dim):
    from lit_llama import _native as N

    g = torch.Generator(device="cuda").manual_seed(T)
    q = torch.full((T, H * dim), 16.0, dtype=torch.bfloat16, device="cuda")
    sign = torch.ones(T, device="cuda") if keys == "top" else -torch.ones(T, device="cuda") if keys == "bottom" else \
        torch.where(torch.rand(T, generator=g, device="cuda") < 0.5, -1.0, 1.0)
    k = (16.0 * sign[None, :, None]).expand(1, T, H * dim).to(torch.bfloat16).contiguous()          # products of 16384 and more: tanh is 1
    v = (torch.randn((1, T, H * dim), generator=g, device="cuda") * 2.0 ** power).to(torch.bfloat16)
    pos, y = torch.arange(T, dtype=torch.int32, device="cuda"), torch.empty((T, H * dim), dtype=torch.bfloat16, device="cuda")
    N.call("ll_softmax_attn_rows", N.ptr(q), H * dim, None, 0, N.ptr(k), N.ptr(v), N.LL_BF16, N.ptr(pos), None, None, dim ** -0.5, cap, 1, T, H, H, dim, dim, 0, 0,
           T, 1, 0, 1, 0.0, 1.0, 0.0, None, N.ptr(y), y.stride(0), N.stream())
    assert N.call_ret("ll_softmax_attn_tc_error") == 0
    s = (cap * sign.double())[None].expand(T, T).masked_fill(~torch.ones((T, T), dtype=torch.bool, device="cuda").tril(), -math.inf)
    want = torch.softmax(s, -1) @ v[0].double()
    # a rounding to bf16, and weights of 16 bits: 2^-16 of the largest value
    assert bool(((y.double() - want).abs() <= want.abs() * 2.0 ** -8 + float(v.abs().max()) * 2.0 ** -14).all())
