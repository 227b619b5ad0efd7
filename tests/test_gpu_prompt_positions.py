"""Positions of a LLaMA prompt that are no whole numbers, or that lie outside the rotary table, and caches of another shape than the call's."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@torch.no_grad()
def _model(layers=2, **more):
    from lit_llama.model import LLaMA, LLaMAConfig

    m = LLaMA(LLaMAConfig(block_size=64, vocab_size=100, n_layer=layers, n_head=4, n_embd=256, **more)).to("cuda", torch.bfloat16).eval()
    g = torch.Generator(device="cuda").manual_seed(0)
    for p in m.parameters():
        p.copy_(torch.randn(p.shape, generator=g, device="cuda") * (p.shape[-1] ** -0.5) if p.dim() > 1 else torch.ones_like(p))
    return m


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16, torch.bool, torch.uint8, torch.int16])
@torch.no_grad()
def test_positions_are_whole_numbers_of_32_or_64_bits(dtype):
    m, idx = _model(1), torch.arange(5, device="cuda")[None]
    want = m(idx, 16, torch.arange(5, device="cuda"))
    m.reset_cache()
    assert torch.equal(m(idx, 16, torch.arange(5, device="cuda", dtype=torch.int32)), want)
    m.reset_cache()
    with pytest.raises(RuntimeError):
        m(idx, 16, torch.arange(5, device="cuda").to(dtype))


@torch.no_grad()
def test_caches_of_another_shape_are_refused():
    """Caches made for another length, batch or dtype than a prompt's, before anything is written to them."""
    m, idx, pos = _model(), torch.arange(6, device="cuda")[None], torch.arange(6, device="cuda")
    m(idx, 16, pos)
    held = [[t.clone() for t in kv] for kv in m.kv_caches]
    for args in ((idx, 32, pos), (idx, 12, pos), (idx.repeat(2, 1), 16, pos)):
        with pytest.raises(RuntimeError, match="cache"):
            m(*args)
    assert all(torch.equal(a, b) for kv, kv0 in zip(m.kv_caches, held) for a, b in zip(kv, kv0))
    m.kv_caches = [tuple(t.float() for t in kv) for kv in m.kv_caches]
    with pytest.raises(RuntimeError, match="cache"):
        m(idx, 16, pos)
    m.reset_cache()
    m(idx, 32, pos)
