"""The recurrence whose last column is the constant 1 (matrix memory with its normaliser), in chunks on tensor cores, against 64 bits beside
the walk token by token: edges of chunks and of column tiles, heads narrower than the padded tiles, a state to start from."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [64, 65, 127, 128, 321])
@pytest.mark.parametrize("n,vdim,H,qk", [(8, 8, 3, 3), (64, 64, 2, 2), (40, 120, 2, 1), (128, 256, 4, 4)])
@pytest.mark.parametrize("first", [0, 7])
def test_unit_chunks_against_64_bits(T, n, vdim, H, qk, first):
    from lit_llama import recurrence as R

    B, p = 2, vdim + 1
    g = torch.Generator(device="cuda").manual_seed(T + n + vdim)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    q, k, v = (rnd(B * T, c).to(torch.bfloat16) for c in (qk * n, qk * n, H * vdim))
    keep, take = torch.sigmoid(3.0 + 2.0 * rnd(B * T, H)), torch.exp(-rnd(B * T, H).abs())
    keep[B * T // 2] = 0.0                                   # a memory that is wiped
    state = rnd(B, H, n, p)
    pos = torch.arange(first, first + T, dtype=torch.int32, device="cuda")
    got = {}
    for chunks in (True, False):
        R.USE_CHUNKS, was = chunks, R.USE_CHUNKS
        try:
            s = state.clone()
            y = R.decay_scan(q, 0, k, 0, v, 0, keep, False, take, None, n ** -0.5, s, pos, B, T, H, qk, n, p, unit_col=True)
        finally:
            R.USE_CHUNKS = was
        got[chunks] = (y.double(), s.double())
    S = state.double() if first else torch.zeros_like(state, dtype=torch.float64)
    heads = torch.arange(H, device="cuda") // (H // qk)
    qd, kd = (t.double().view(B, T, qk, n)[:, :, heads] for t in (q, k))
    vd = torch.cat([v.double().view(B, T, H, vdim), torch.ones((B, T, H, 1), dtype=torch.float64, device="cuda")], dim=-1)
    want = torch.empty((B, T, H, p), dtype=torch.float64, device="cuda")
    for t in range(T):
        S = keep.double().view(B, T, H)[:, t, :, None, None] * S + (take.double().view(B, T, H)[:, t, :, None] * kd[:, t])[..., None] * vd[:, t, :, None]
        want[:, t] = (S * qd[:, t, :, :, None]).sum(2) * n ** -0.5
    want = want.view(B * T, H * p)
    for i, (name, ref) in enumerate((("y", want), ("state", S))):
        err = [float((got[c][i] - ref).norm() / ref.norm()) for c in (True, False)]
        # 24-bit terms and fp32 sums on both sides: the chunks' error is of the walk's size (a few fp32 roundings)
        assert err[0] <= 2.0 * err[1] + 2.0 ** -22, (name, err)
