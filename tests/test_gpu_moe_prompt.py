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
