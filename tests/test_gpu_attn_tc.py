"""The tcgen05 form of prompts' softmax attention (csrc/attn_tc.cuh) at the edges of its tiles (64 keys, 128 and 256 queries), against the
fp32 form of the same call, and latent attention over expanded rows against attention in latent space."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def _softmax(T, past, ring, H=4, G=2, dim=64, vdim=64, B=1, window=0, chunk=0, cap=0.0, sink=False, slopes=False, gate=False, y_pad=0, form=0,
             spoil=False, seed=0):
    from lit_llama import _native as N

    g = torch.Generator(device="cuda").manual_seed(seed)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    q, kc, vc, gt = rnd(B * T, H * dim), rnd(B, ring, G * dim), rnd(B, ring, G * vdim), rnd(B * T, H * vdim)
    if spoil:                                  # slots without a position of the sequence hold whatever they hold
        used = torch.zeros(ring, dtype=torch.bool, device="cuda")
        lo = past if window == 0 else min(past, window - 1)
        used[[(p % ring) for p in range(past - lo, past + T)]] = True
        kc[:, ~used] = math.nan
        vc[:, ~used] = math.inf
    pos = torch.arange(past, past + T, dtype=torch.int32, device="cuda")
    sk = torch.randn(H, generator=g, device="cuda") if sink else None
    sl = torch.rand(H, generator=g, device="cuda") * 0.1 if slopes else None
    y = torch.zeros((B * T, H * vdim + y_pad), dtype=torch.bfloat16, device="cuda")
    N.call("ll_softmax_attn_rows", N.ptr(q), H * dim, N.ptr(gt) if gate else None, H * vdim if gate else 0, N.ptr(kc), N.ptr(vc), N.LL_BF16,
           N.ptr(pos), N.ptr(sk), N.ptr(sl), dim ** -0.5, cap, B, T, H, G, dim, vdim, window, chunk, ring, 1, form, 1, 0.0, 1.0, 0.0, None,
           N.ptr(y), y.stride(0), N.stream())
    torch.cuda.synchronize()
    assert N.call_ret("ll_softmax_attn_tc_error") == 0
    return y, float(vc[torch.isfinite(vc)].abs().max())


CASES = [dict(T=t, past=0, ring=512) for t in (16, 63, 64, 65, 127, 128, 129, 255, 256, 257, 300)] + [
    dict(T=130, past=41, ring=152, chunk=23), dict(T=40, past=250, ring=256, window=20),      # two key blocks reach past the last key
    dict(T=70, past=900, ring=256, window=100),                       # the ring wraps inside a key block
    dict(T=200, past=77, ring=300, window=64, spoil=True),
    dict(T=130, past=0, ring=130, spoil=True), dict(T=40, past=5, ring=400, spoil=True),
    dict(T=300, past=33, ring=512, chunk=50), dict(T=129, past=0, ring=129, chunk=128),
    dict(T=257, past=3, ring=260, cap=50.0), dict(T=200, past=0, ring=200, cap=1.5), dict(T=150, past=0, ring=150, sink=True, gate=True),
    dict(T=200, past=9, ring=209, slopes=True), dict(T=100, past=9, ring=109, slopes=True, cap=20.0),
    dict(T=129, past=0, ring=129, dim=128, vdim=128, gate=True, B=3), dict(T=129, past=0, ring=129, dim=128, vdim=40, H=3, G=3),
    dict(T=64, past=0, ring=64, dim=40, vdim=128, H=8, G=1), dict(T=90, past=0, ring=90, dim=8, vdim=8), dict(T=33, past=0, ring=33, y_pad=8),
    dict(T=33, past=0, ring=33, y_pad=2),                              # rows of the output off 16-byte boundaries: the form before it
]


# a block's tiles from both ends: an even and an odd number of them, positions before the step, a window of most queries; caps with and without a bound
APART = [dict(T=513, past=70, ring=583, cap=50.0, sink=True, gate=True), dict(T=640, past=0, ring=640), dict(T=385, past=0, ring=385, cap=100.0, sink=True),
         dict(T=700, past=20, ring=720, window=400), dict(T=640, past=3, ring=700, cap=1.5, slopes=True, spoil=True)]
CASES += APART
# with no more tiles than SMs a block takes one of them; the same walks with more: two tiles a block, from both ends or neighbours
CASES += [dict(c, B=149 // (-(-c["T"] // 128) * 4) + 1) for c in APART + [
    dict(T=300, past=33, ring=512, chunk=50), dict(T=513, past=77, ring=650, window=64, spoil=True), dict(T=257, past=3, ring=260, cap=50.0),
    dict(T=129, past=0, ring=129, dim=128, vdim=128, gate=True), dict(T=40, past=250, ring=256, window=20)]]


@pytest.mark.parametrize("case", CASES, ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_softmax_prompt_against_fp32_form(case):
    got, top = _softmax(**case)
    want, _ = _softmax(**case, form=1)
    got, want = got.float(), want.float()
    assert torch.isfinite(got).all()
    # both round the same sum to bf16 (2^-9 each, two neighbours at a tie); the weights carry 16 bits, so the sums before the gate are
    # 2^-16 of the largest value apart; exponentials and the sigmoid 1e-6
    assert ((got - want).abs() <= want.abs() * 2.0 ** -7 + top * 2.0 ** -14).all()


@pytest.mark.parametrize("T,past,S,window,terms", [(16, 0, 16, None, False), (64, 30, 128, None, True), (129, 0, 200, 50, False), (257, 100, 400, None, True),
                                                   (100, 300, 256, 64, False)])
@pytest.mark.parametrize("nope,rot,v,rank,gate", [(128, 64, 128, 64, "head"), (24, 8, 40, 48, "none"), (64, 32, 64, 256, "head")])
def test_latent_prompt_expanded_against_latent_space(T, past, S, window, terms, nope, rot, v, rank, gate):
    from lit_llama import _native as N
    from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec

    B, H = 2, 3
    spec = LatentAttentionSpec(width=64, heads=H, nope_dim=nope, rot_dim=rot, v_dim=v, kv_rank=rank, window=window, scale=(nope + rot) ** -0.5,
                               gate=gate, exact_weights=terms)
    m = LatentAttention(spec, torch.bfloat16, "cuda")
    g = torch.Generator(device="cuda").manual_seed(T)
    for p in m.parameters():
        if p.dim() > 1:
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") / math.sqrt(p.shape[-1]))
    proj = torch.randn((B * T, m.w_in.shape[0]), generator=g, device="cuda").to(torch.bfloat16)
    pos = torch.arange(past, past + T, dtype=torch.int32, device="cuda")
    rope = spec.rope_table(past + T, "cuda")
    cache = torch.randn((B, S, spec.row), generator=g, device="cuda").to(torch.bfloat16)
    used = torch.zeros(S, dtype=torch.bool, device="cuda")
    used[[p % S for p in range(max(0, past - (window or past + 1) + 1), past + T)]] = True
    cache[:, ~used] = math.nan                 # never read, though the up-projection of every slot is formed
    outs = []
    for expanded in (True, False):
        c, out = cache.clone(), torch.zeros((B * T, H * v + 8), dtype=torch.bfloat16, device="cuda")[:, : H * v]
        m._takes_expanded = lambda *a, e=expanded: e
        outs.append(m.attend(proj, B, T, pos, rope, c, 1, out).double())
    assert N.call_ret("ll_latent_prompt_error") == 0
    # operands rounded to bf16 once more on either side (the query in latent space; the keys and values per head): 2^-9 a number, which
    # over a row's sum leaves about 2^-8 of it, twice
    assert torch.isfinite(outs[0]).all()
    assert (outs[0] - outs[1]).norm() <= 2.0 ** -6.5 * outs[1].norm()


@pytest.mark.parametrize("T,S,window", [(16, 16, 0), (129, 129, 0), (300, 512, 100)])
@pytest.mark.parametrize("terms", [1, 2])
@pytest.mark.parametrize("scale", [0.02, 0.2])
def test_weights_add_up_to_what_they_are_divided_by(T, S, window, terms, scale):
    """Values that are all 1 come back as 1: the sum a row is divided by is that of the weights the product saw.  The fp32 sums on both sides
    are off by a few 2^-24 of T numbers, two terms by 2^-17: well inside the half step of bf16 below 1 (2^-9)."""
    from lit_llama import _native as N

    B, H, nope, rot, v, rank = 2, 3, 64, 32, 64, 64
    g = torch.Generator(device="cuda").manual_seed(T)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    q, k, cache = rnd(B * T, H * (nope + rot)), rnd(B * S, H * nope), rnd(B, S, rank + rot)
    ones = torch.ones((H, B * S, v), dtype=torch.bfloat16, device="cuda")
    pos = torch.arange(T, dtype=torch.int32, device="cuda")
    rope = torch.tensor([1.0, 0.0], device="cuda").repeat(T, rot // 2).contiguous()
    q_rot, y = torch.empty((B * T, H, rot), dtype=torch.bfloat16, device="cuda"), torch.zeros((B * T, H * v), dtype=torch.bfloat16, device="cuda")
    N.call("ll_latent_prompt_attn", N.ptr(q), q.stride(0), nope, nope + rot, None, 0, N.ptr(rope), N.ptr(pos), N.ptr(k), k.stride(0), nope,
           N.ptr(ones), v, B * S * v, N.ptr(cache), N.ptr(q_rot), N.ptr(y), y.stride(0), B, T, H, rank, rot, rot, v, S, window, scale, terms,
           N.stream())
    torch.cuda.synchronize()
    assert N.call_ret("ll_latent_prompt_error") == 0
    assert bool((y == 1.0).all())


def test_positions_that_do_not_rise():
    """Queries in any order of their positions see the keys up to their own: the same rows as in rising order.  (Nothing is written outside
    a key block's rows in shared memory, whatever the last query's position is.)"""
    from lit_llama import _native as N

    T, H, G, dim = 300, 4, 2, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)  # noqa: E731
    q, kc, vc = rnd(T, H * dim), rnd(1, T, G * dim), rnd(1, T, G * dim)
    outs = []
    for order in (torch.arange(T, device="cuda"), torch.arange(T - 1, -1, -1, device="cuda"), torch.randperm(T, generator=g, device="cuda")):
        pos, qs = order.to(torch.int32), q[order].contiguous()
        y = torch.zeros((T, H * dim), dtype=torch.bfloat16, device="cuda")
        N.call("ll_softmax_attn_rows", N.ptr(qs), H * dim, None, 0, N.ptr(kc), N.ptr(vc), N.LL_BF16, N.ptr(pos), None, None, dim ** -0.5, 0.0, 1, T, H,
               G, dim, dim, 0, 0, T, 1, 0, 1, 0.0, 1.0, 0.0, None, N.ptr(y), y.stride(0), N.stream())
        torch.cuda.synchronize()
        assert N.call_ret("ll_softmax_attn_tc_error") == 0
        back = torch.empty_like(y)
        back[order] = y
        outs.append(back.float())
    for other in outs[1:]:           # a row's maximum moves elsewhere: the weights' scale differs by a power that is not exact, 2^-16, and bf16 rounds
        assert ((outs[0] - other).abs() <= outs[0].abs() * 2.0 ** -7 + 2.0 ** -12).all()


@pytest.mark.parametrize("T,past,S,window,rows", [(64, 0, 1024, None, 64), (130, 70, 512, None, 200), (257, 100, 400, 50, 306), (100, 300, 256, 64, 163),
                                                  (129, 500, 200, 50, 178), (33, 8, 41, None, 41)])
@pytest.mark.parametrize("B", [1, 2])
def test_only_visible_rows_are_expanded(monkeypatch, T, past, S, window, rows, B):
    """With the end of the step known, the rows its queries see are formed and no others: rings that are nearly empty, rings that wrap,
    windows that begin after position 0.  The result is that of the form in latent space."""
    from lit_llama import _native as N
    from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec

    H, nope, rot, v, rank = 3, 64, 32, 64, 64
    spec = LatentAttentionSpec(width=64, heads=H, nope_dim=nope, rot_dim=rot, v_dim=v, kv_rank=rank, window=window, scale=(nope + rot) ** -0.5)
    m = LatentAttention(spec, torch.bfloat16, "cuda")
    g = torch.Generator(device="cuda").manual_seed(T)
    for p in m.parameters():
        if p.dim() > 1:
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") / math.sqrt(p.shape[-1]))
    proj = torch.randn((B * T, m.w_in.shape[0]), generator=g, device="cuda").to(torch.bfloat16)
    pos = torch.arange(past, past + T, dtype=torch.int32, device="cuda")
    rope = spec.rope_table(past + T, "cuda")
    cache = torch.randn((B, S, spec.row), generator=g, device="cuda").to(torch.bfloat16)
    used = torch.zeros(S, dtype=torch.bool, device="cuda")
    used[[p % S for p in range(max(0, past - (window or past + 1) + 1), past + T)]] = True
    cache[:, ~used] = math.nan
    formed, call = [], N.call
    monkeypatch.setattr(N, "call", lambda name, *a: (formed.append(a[25]) if name == "ll_latent_prompt_attn" else None, call(name, *a))[1])
    got = m.attend(proj, B, T, pos, rope, cache.clone(), 1, end=past + T).double()
    m._takes_expanded = lambda *a: False
    want = m.attend(proj, B, T, pos, rope, cache.clone(), 1, end=past + T).double()
    assert formed == [rows] and N.call_ret("ll_latent_prompt_error") == 0
    assert torch.isfinite(got).all()
    assert (got - want).norm() <= 2.0 ** -6.5 * want.norm()      # as above


@pytest.mark.parametrize("family", ["lepalorn", "bumulix", "zekonex"])
def test_models_say_where_a_step_ends(family, monkeypatch, tmp_path):
    import importlib

    from lit_llama.latent_attention import LatentAttention

    util = importlib.import_module(f"tests.util_{family}")
    cfg, W = util.case_mixed()
    m = util.load(util.write_model(tmp_path, cfg, W), torch.bfloat16)
    ends, attend = [], LatentAttention.attend
    monkeypatch.setattr(LatentAttention, "attend", lambda self, *a, end=None, **kw: (ends.append((a[2], end)), attend(self, *a, end=end, **kw))[1])
    util.run_schedule(m, list(range(9)), [5, 3, 1], 64)
    assert {e for t, e in ends if t == 5} == {5} and {e for t, e in ends if t == 3} == {8}
    assert {e for t, e in ends if t == 1} <= {None}              # a captured step's position is known to the device alone


@pytest.mark.parametrize("T,past,S,window,terms", [(129, 0, 200, 50, False), (257, 100, 400, None, True), (385, 20, 420, None, False)])
def test_latent_tiles_of_many_sequences(T, past, S, window, terms):
    """More tiles than SMs (two a block, neighbours or from both ends) against the same sequences two at a time (a tile a block): a row meets the same
    keys in the same order, in blocks that may start elsewhere (its weights round apart by 2^-9 at most, and the row once more)."""
    from lit_llama import _native as N
    from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec

    B, H, nope, rot, v = 28, 3, 64, 32, 64
    spec = LatentAttentionSpec(width=64, heads=H, nope_dim=nope, rot_dim=rot, v_dim=v, kv_rank=256, window=window, scale=(nope + rot) ** -0.5,
                               gate="head", exact_weights=terms)
    m = LatentAttention(spec, torch.bfloat16, "cuda")
    g = torch.Generator(device="cuda").manual_seed(T)
    for p in m.parameters():
        if p.dim() > 1:
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") / math.sqrt(p.shape[-1]))
    proj = torch.randn((B * T, m.w_in.shape[0]), generator=g, device="cuda").to(torch.bfloat16)
    pos = torch.arange(past, past + T, dtype=torch.int32, device="cuda")
    rope = spec.rope_table(past + T, "cuda")
    cache = torch.randn((B, S, spec.row), generator=g, device="cuda").to(torch.bfloat16)
    m._takes_expanded = lambda *a: True
    both = []
    for n in (B, 2):
        outs = []
        for b in range(0, B, n):
            out = torch.zeros((n * T, H * v), dtype=torch.bfloat16, device="cuda")
            outs.append(m.attend(proj[b * T:(b + n) * T], n, T, pos, rope, cache[b:b + n].clone(), 1, out).double())
        both.append(torch.cat(outs))
    assert N.call_ret("ll_latent_prompt_error") == 0
    assert torch.isfinite(both[0]).all() and (both[0] - both[1]).norm() <= 2.0 ** -7.5 * both[1].norm()
