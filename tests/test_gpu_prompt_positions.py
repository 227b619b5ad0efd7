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


@pytest.mark.parametrize("bad", [64, -1, 1 << 40])
@torch.no_grad()
def test_a_bad_position_takes_no_other_row(bad):
    """A token outside the rotary table: the call is reported, and no row of the caches but those of the other tokens is written."""
    from lit_llama import _native as N

    m, idx = _model(), torch.arange(4, device="cuda")[None]
    m(idx[:, :1].repeat(1, 2), 64, torch.tensor([0, 63], device="cuda"))
    torch.cuda.synchronize()
    first = [[t[:, :, [0, 63]].clone() for t in kv] for kv in m.kv_caches]
    with pytest.raises(RuntimeError, match="rotary table"):
        m(idx, 64, torch.tensor([4, bad, 5, 6], device="cuda"))
        torch.cuda.synchronize()
        N.check_waits()
    torch.cuda.synchronize()
    rest = [s for s in range(64) if s not in (0, 4, 5, 6, 63)]
    for kv, kv0 in zip(m.kv_caches, first):
        for t, t0 in zip(kv, kv0):
            assert torch.equal(t[:, :, [0, 63]], t0) and bool((t[:, :, rest] == 0).all())
    N.check_waits()


@pytest.mark.parametrize("hs", [40, 20])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@torch.no_grad()
def test_a_token_without_a_slot(hs, dtype):
    """Slot -1: no key and no value is stored, and the token's queries are no numbers, so that its logits are none either."""
    from lit_llama import _native as N

    T, nh, S = 5, 3, 8
    qkv, rope = torch.randn((T, 3 * nh * hs), device="cuda").to(dtype), torch.randn((S, hs // 2, 2), device="cuda")
    pos, slots = torch.tensor([0, 1, 0, 3, 4], dtype=torch.int32, device="cuda"), torch.tensor([0, 1, -1, 3, 4], dtype=torch.int32, device="cuda")
    q = torch.zeros((1, nh, T, hs), dtype=dtype, device="cuda")
    held = torch.full((2, 3, nh, S, hs), 7.0, dtype=dtype, device="cuda")            # a cache and its neighbours on both sides
    N.call("ll_rope_kv_append", N.ptr(qkv), N.ptr(rope), N.ptr(pos), N.ptr(slots), N.ptr(q), N.ptr(held[0, 1]), N.ptr(held[1, 1]), N.dtype_code(dtype), 1, T, nh,
           hs, S, N.stream())
    assert bool(q[0, :, 2].isnan().all()) and bool(q[0, :, [0, 1, 3, 4]].isfinite().all())
    assert bool((held[:, [0, 2]] == 7.0).all()) and bool((held[:, 1, :, [2, 5, 6, 7]] == 7.0).all()) and bool((held[:, 1, :, [0, 1, 3, 4]] != 7.0).any())


@torch.no_grad()
def test_the_reported_row_of_a_prompt():
    """What a bad position becomes: a valid rotary row, no slot, the first slot to look at."""
    from lit_llama import _native as N

    out = torch.empty((3, 4), dtype=torch.int32, device="cuda")
    N.call("ll_prompt_pos", *(N.ptr(o) for o in out), N.ptr(torch.tensor([3, 16, -5, 9], device="cuda")), 4, 8, 16, N.stream())
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="rotary table"):
        N.check_waits()
    assert out.tolist() == [[3, 0, 0, 9], [3, -1, -1, 1], [3, 0, 0, 7]]
