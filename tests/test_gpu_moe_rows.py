"""Expert rows at the edges of their tiles, routing at the edges of its forms, and the 16-byte forms beside the general ones.

References: float64 sums over the same bf16 numbers; bf16 results are within half a unit in the last place (2^-9) of the value
they round, plus the fp32 error of their sums (2^-24 a term, of the sum of magnitudes).
"""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from lit_llama import _native as N


def _rand(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, dtype=torch.float32) * scale).cuda()


# counts: one expert empty, whole tiles, one row, tiles of more CTAs than the chip has (each takes three tiles or more)
@pytest.mark.parametrize("counts,n", [((0, 128, 1, 129, 0), 136), ((700, 0, 1300, 256, 750), 4104), ((5, 0, 0, 3, 1), 72)])
@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("k", [64, 328])
def test_expert_tiles(counts, n, mode, k):
    g = torch.Generator().manual_seed(n + k + mode)
    X, rows, top = len(counts), sum(counts), 1
    offsets = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32).cuda()
    perm = torch.randperm(rows, generator=g).int().cuda()
    a = _rand(g, rows, k).bfloat16()
    w = _rand(g, X, (2 if mode in (1, 2) else 1) * n, k, scale=k ** -0.5).bfloat16()
    limit, alpha = 1.5, 1.7
    c = torch.full((rows, n), float("nan"), dtype=torch.bfloat16, device="cuda")
    N.call("ll_moe_grouped_gemm_tc", N.ptr(a), N.ptr(w), N.ptr(offsets), N.ptr(perm), mode, rows, X, n, k, limit, alpha, N.ptr(c), n, N.stream())
    assert N.call_ret("ll_moe_tc_error") == 0
    ad, wd = a.double(), w.double()
    for e in range(X):
        lo, hi = int(offsets[e]), int(offsets[e + 1])
        z = ad[lo:hi] @ wd[e].T
        err = (ad[lo:hi].abs() @ wd[e].abs().T) * (k * 2.0 ** -24)
        if mode in (1, 2):
            gate, up = z[:, :n].clamp(max=limit), z[:, n:].clamp(-limit, limit) + (1.0 if mode == 1 else 0.0)
            want = gate * torch.sigmoid(alpha * gate) * up
            # the unit's slope is at most 1.1 in the gate and the gate itself in the other branch; 8 rounded steps of its own
            err = 1.1 * up.abs() * err[:, :n] + gate.abs() * err[:, n:] + want.abs() * 2.0 ** -20
        elif mode == 3:
            want, err = z.clamp(min=0) ** 2, 2 * z.abs() * err + z ** 2 * 2.0 ** -23
        else:
            want = z
        got = (c[perm[lo:hi].long()] if mode == 0 else c[lo:hi]).double()
        assert bool(((got - want).abs() <= want.abs() * 2.0 ** -8 + err + 1e-30).all()), e


@pytest.mark.parametrize("M", [1, 148, 149, 1183, 1184, 1191])
@pytest.mark.parametrize("dim,X,shift", [(64, 5, 0), (2048, 32, 0), (72, 9, 1), (30, 4, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_routing_forms(M, dim, X, shift, dtype):
    """One, four and eight tokens to a block, aligned rows and shifted ones, widths that are no multiple of 4."""
    g = torch.Generator().manual_seed(M + dim)
    top = 2
    x = _rand(g, M * dim + shift)[shift:].to(dtype) if not shift else _rand(g, M * dim + shift).to(dtype)[shift:]
    w, bias = _rand(g, X, dim, scale=dim ** -0.5), _rand(g, X, scale=0.1)
    idx, ew = torch.empty(M, top, dtype=torch.int32, device="cuda"), torch.empty(M, top, device="cuda")
    counts, rank = torch.empty(X, dtype=torch.int32, device="cuda"), torch.empty(M * top, dtype=torch.int32, device="cuda")
    offsets, perm = torch.empty(X + 1, dtype=torch.int32, device="cuda"), torch.empty(M * top, dtype=torch.int32, device="cuda")
    N.call("ll_moe_route", N.ptr(x), N.dtype_code(dtype), N.ptr(w), N.ptr(bias), M, dim, X, top, N.ptr(idx), N.ptr(ew), N.ptr(counts),
           N.ptr(rank), N.ptr(offsets), N.ptr(perm), N.stream())
    xd = x.view(M, dim).double()
    z = xd @ w.double().T + bias.double()
    err = (dim * 2.0 ** -24) * (xd.abs() @ w.double().abs().T + 1).max()
    best = z.topk(top, 1).values
    chosen = z.gather(1, idx.long())
    assert float((chosen - best).abs().max()) <= 2 * err                    # near ties may fall either way
    assert float((ew.double() - torch.softmax(chosen, 1)).abs().max()) <= 2 * err + 2.0 ** -20
    assert bool((idx[:, 0] != idx[:, 1]).all())
    flat = idx.flatten().long()
    assert torch.equal(counts.long(), torch.bincount(flat, minlength=X))
    assert torch.equal(offsets.long().cpu(), torch.cat([torch.zeros(1, dtype=torch.long), counts.long().cpu().cumsum(0)]))
    assert torch.equal(perm.long().sort().values.cpu(), torch.arange(M * top))
    assert torch.equal(flat[perm.long()].cpu(), torch.repeat_interleave(torch.arange(X), counts.long().cpu()))


@pytest.mark.parametrize("dim,ld,shift", [(64, 64, 0), (72, 80, 0), (72, 75, 0), (70, 70, 0), (64, 64, 1), (1032, 1032, 0)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("shared", [0, 1, 2])
def test_combined_rows(dim, ld, shift, dtype, shared):
    g = torch.Generator().manual_seed(dim)
    M, top = 37, 3
    y, w = _rand(g, M * top * dim + shift).to(dtype)[shift:], _rand(g, M, top)
    sy, sg = _rand(g, M, ld).to(dtype), _rand(g, M, 1).to(dtype)
    out = torch.empty(M, dim, dtype=dtype, device="cuda")
    N.call("ll_moe_combine", N.ptr(y), N.ptr(w), top, N.ptr(sy) if shared else 0, ld, N.ptr(sg) if shared == 2 else 0, 1, N.ptr(out),
           N.dtype_code(dtype), M, dim, N.stream())
    yd = y.view(M, top, dim).double()
    want, mag = (w.double()[..., None] * yd).sum(1), (w.double()[..., None] * yd).abs().sum(1)
    if shared:
        s = (torch.sigmoid(sg.double()) if shared == 2 else 1.0) * sy.double()[:, :dim]
        want, mag = want + s, mag + s.abs()
    tol = mag * 2.0 ** -20 + (want.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0)
    assert bool(((out.double() - want).abs() <= tol).all())


@pytest.mark.parametrize("dim,rot", [(64, 64), (128, 64), (128, 0), (96, 48), (80, 48), (72, 72)])
@pytest.mark.parametrize("norm", [False, True])
@pytest.mark.parametrize("values", ["own", "keys", "none"])
@pytest.mark.parametrize("shift", [0, 8, 1])
def test_rotated_rows(dim, rot, norm, values, shift):
    """Aligned rows (16-byte pieces) and shifted ones or rotations of other sizes (the general form), a ring shorter than the positions."""
    g = torch.Generator().manual_seed(dim + rot)
    B, T, H, G, ring = 2, 5, 6, 2, 16
    q, k, v = (_rand(g, B * T, h * dim + shift).bfloat16() for h in (H, G, G))
    qn, kn = (1 + _rand(g, H * dim, scale=0.1), 1 + _rand(g, G * dim, scale=0.1)) if norm else (None, None)
    freq = torch.tensor(1e4 ** (-np.arange(max(rot // 2, 1)) / max(rot // 2, 1)), dtype=torch.float32).cuda()
    pos = torch.arange(13, 13 + T, dtype=torch.int32).cuda()
    qo = torch.empty(B * T, H * dim, dtype=torch.bfloat16, device="cuda")
    kc, vc = (torch.zeros(B, ring, G * dim, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    eps = 1e-5
    has_k = values != "none"
    N.call("ll_qk_rotary_append", N.ptr(q), H * dim + shift, N.ptr(k) if has_k else 0, G * dim + shift, N.ptr(v) if values == "own" else 0,
           G * dim + shift, N.LL_BF16, N.ptr(qn) if norm else 0, N.ptr(kn) if norm else 0, eps, N.ptr(freq), rot, N.ptr(pos), N.ptr(qo),
           N.ptr(kc), N.ptr(vc), B, T, H, G, dim, dim, ring, N.stream())

    def row(x, w, heads):
        x = x[:, :heads * dim].double()
        if w is not None:
            x = x / torch.sqrt((x * x).mean(1, keepdim=True) + eps) * w.double()
        plain, x, h2 = x, x.view(B, T, heads, dim).clone(), rot // 2
        # angles in fp32, as both forms compute them
        ang = (pos.float()[:, None] * freq[None, :h2]).double().view(1, T, 1, h2)
        a, b = x[..., :h2].clone(), x[..., h2:rot].clone()
        x[..., :h2], x[..., h2:rot] = a * ang.cos() - b * ang.sin(), b * ang.cos() + a * ang.sin()
        mag = x.abs()
        mag[..., :h2] = mag[..., h2:rot] = a.abs() + b.abs()
        return plain.view(B, T, -1), x.reshape(B, T, -1), mag.reshape(B, T, -1)

    def near(got, want, mag):       # half a bf16 step, and fp32 steps of the norm, the angle's sine and the rotation
        assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + mag * 2.0 ** -19).all())

    _, want, mag = row(q, qn, H)
    near(qo.view(B, T, -1), want, mag)
    if has_k:
        plain, want, mag = row(k, kn, G)
        at = (pos.long() % ring)
        near(kc[:, at], want, mag)
        near(vc[:, at], v[:, :G * dim].double().view(B, T, -1) if values == "own" else plain, plain.abs())
        rest = torch.ones(ring, dtype=torch.bool)
        rest[at.cpu()] = False
        assert not kc[:, rest.cuda()].any() and not vc[:, rest.cuda()].any()


@pytest.mark.parametrize("M", [1, 3, 9, 300, 1400])
@pytest.mark.parametrize("score", ["chosen", "all", "sigmoid"])
def test_a_row_of_no_numbers(M, score):
    """A token of NaNs has no expert to choose: it is routed to a valid one, comes out as NaNs, and the other tokens as without it."""
    from lit_llama.moe import MoE, MoESpec

    mix = MoE(MoESpec(64, 8, 2, 32, 7.0, 16, 7.0, score=score, router_bias=False), torch.bfloat16, "cuda")
    g = torch.Generator(device="cuda").manual_seed(M)
    with torch.no_grad():
        for p in mix.parameters():
            p.copy_(torch.randn(p.shape, generator=g, device="cuda") * p.shape[-1] ** -0.5)
    x = torch.randn((M, 64), generator=g, device="cuda").to(torch.bfloat16)
    want = mix(x)
    x[M // 2] = float("nan")
    idx, w, offsets, perm = mix.route(x)
    assert bool(((idx >= 0) & (idx < 8)).all()) and int(offsets[-1]) == 2 * M and torch.equal(perm.sort().values, torch.arange(2 * M, device="cuda", dtype=perm.dtype))
    assert bool(w[M // 2].isnan().all())
    got = mix(x)
    keep = torch.arange(M, device="cuda") != M // 2
    assert bool(got[M // 2].isnan().all()) and torch.equal(got[keep], want[keep])
