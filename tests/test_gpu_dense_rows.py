"""Products with any number of rows (csrc/dense_rows.cu, csrc/small_rows.cuh) at the edges of their forms, and layers that run in one call against
the same layers by separate calls.

References: float64 sums over the same bf16 numbers; results are within half a unit in the last place (2^-9) of the value they round, plus the fp32
error of their sums (2^-24 a term, of the sum of magnitudes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

if torch.cuda.is_available():
    from lit_llama import _native as N


def _rand(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(torch.bfloat16)


def _check(got, x, w):
    want, mag = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    assert bool(((got.double() - want).abs() <= want.abs() * 2.0 ** -8 + mag * (x.shape[1] * 2.0 ** -24)).all())


# rows: of each form, the first and last of its tiles of 8, 16, 32 and 256 rows; weights: less than a tile, ragged ones, k that is no whole stage
@pytest.mark.parametrize("M", [1, 2, 3, 8, 9, 16, 17, 32, 33, 64, 65, 257, 700])
@pytest.mark.parametrize("n,k", [(8, 8), (136, 72), (1000, 264), (264, 1032), (4808, 512), (2048, 2048)])
def test_rows(M, n, k):
    g = torch.Generator(device="cuda").manual_seed(M + n)
    x, w = _rand(g, M, k + 8)[:, :k], _rand(g, n, k, scale=k ** -0.5)
    y = torch.full((M, n + 8), float("nan"), dtype=torch.bfloat16, device="cuda")
    N.call("ll_rows_linear", N.ptr(x), x.stride(0), N.ptr(w), N.ptr(y), y.stride(0), M, n, k, N.stream())
    assert N.call_ret("ll_dense_rows_error") == 0
    _check(y[:, :n], x, w)
    assert bool(y[:, n:].isnan().all())                    # nothing past a row's end


@pytest.mark.parametrize("M", [1, 33, 300, 1500])
@pytest.mark.parametrize("heads,cols,k", [(1, 64, 256), (3, 128, 512), (16, 64, 200), (16, 128, 512)])
def test_weights_with_columns_side_by_side(M, heads, cols, k):
    g = torch.Generator(device="cuda").manual_seed(M + heads)
    x, w = _rand(g, M, k + 32)[:, :k], _rand(g, heads, k, cols, scale=k ** -0.5)
    y = torch.empty((M, heads * cols), dtype=torch.bfloat16, device="cuda")
    N.call("ll_dense_rows", N.ptr(x), x.stride(0), N.ptr(w), cols, N.ptr(y), heads * cols, M, heads * cols, k, N.stream())
    assert N.call_ret("ll_dense_rows_error") == 0
    _check(y, x, w.transpose(1, 2).reshape(heads * cols, k))


def _layers(kind, B, T, past, g):
    if kind == "softmax":
        from lit_llama.rotary import RotarySpec
        from lit_llama.softmax_attention import SoftmaxAttention, SoftmaxAttentionSpec

        m = SoftmaxAttention(SoftmaxAttentionSpec(width=256, heads=4, kv_heads=2, dim=64, vdim=64, scale=0.125, eps=1e-5, rotary=RotarySpec(32), qk_norm=True),
                             torch.bfloat16, "cuda")
        held = [_rand(g, B, past + T + 3, 128) for _ in range(2)]
        args = lambda x, pos, h: (x, B, T, pos, h)                                                   # noqa: E731
    elif kind == "latent":
        from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec

        spec = LatentAttentionSpec(width=256, heads=4, nope_dim=64, rot_dim=32, v_dim=64, kv_rank=128, window=100, scale=96 ** -0.5)
        m, rope = LatentAttention(spec, torch.bfloat16, "cuda"), spec.rope_table(past + T + 3, "cuda")
        held = [_rand(g, B, past + T + 3, spec.row)]
        args = lambda x, pos, h: (x, B, T, pos, rope, h[0])                                          # noqa: E731
    else:
        from lit_llama.recurrence import MatrixMemoryMixer, MatrixMemorySpec

        m = MatrixMemoryMixer(MatrixMemorySpec(256, 4, 64, 64, 15.0, 1e-5), torch.bfloat16, "cuda")
        held = [torch.zeros(n, dtype=torch.float32, device="cuda") for n in m.state_shapes(B)]
        args = lambda x, pos, h: (x, B, T, pos, h)                                                   # noqa: E731
    for p in m.parameters():
        p.copy_(torch.randn(p.shape, generator=g, device="cuda") * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.1) + (0.0 if p.dim() > 1 else 1.0))
    return m, held, args


@pytest.mark.parametrize("kind", ["softmax", "latent", "matrix"])
@pytest.mark.parametrize("B,T,past", [(3, 1, 5), (8, 1, 40), (1, 2, 0), (2, 9, 30), (1, 16, 0), (1, 17, 200), (2, 70, 3), (1, 300, 0)])
@torch.no_grad()
def test_layer_in_one_call(kind, B, T, past, monkeypatch):
    """The same kernels between products that round the same sums: a bf16 step of a projection here and there, which the softmax, norms and sums of
    a layer pass on at about its size (2^-8 of the result's norm, over two projections and the kernels between them 2^-6)."""
    g = torch.Generator(device="cuda").manual_seed(B * T)
    m, held, args = _layers(kind, B, T, past, g)
    x, pos = _rand(g, B * T, 256), torch.arange(past, past + T, dtype=torch.int32, device="cuda")
    took, outs, states = [], [], []
    one = type(m)._one_call
    monkeypatch.setattr(type(m), "_one_call", lambda self, *a: took.append(1) or one(self, *a))
    for go in (True, False):
        monkeypatch.setattr(N, "layer_rows", lambda *a, go=go: go)
        h = [t.clone() for t in held]
        outs.append(m(*args(x, pos, h)).double())
        states.append(h)
    assert len(took) == 1 and N.call_ret("ll_dense_rows_error") == 0
    assert bool(torch.isfinite(outs[0]).all())
    assert float((outs[0] - outs[1]).norm()) <= 2.0 ** -6 * float(outs[1].norm())
    for a, b in zip(*states):
        assert float((a.double() - b.double()).norm()) <= 2.0 ** -6 * float(b.double().norm())


@pytest.mark.parametrize("kind", ["softmax", "latent", "matrix"])
@torch.no_grad()
def test_a_captured_prompt_keeps_the_separate_calls(kind):
    g = torch.Generator(device="cuda").manual_seed(5)
    m, held, args = _layers(kind, 1, 40, 0, g)
    x, pos = _rand(g, 40, 256), torch.arange(40, dtype=torch.int32, device="cuda")
    want = m(*args(x, pos, [t.clone() for t in held])).double()
    h = [t.clone() for t in held]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = m(*args(x, pos, h))
    for a, b in zip(h, held):
        a.copy_(b)
    graph.replay()
    assert float((y.double() - want).norm()) <= 2.0 ** -6 * float(want.norm())


@torch.no_grad()
def test_weights_written_just_before(monkeypatch):
    """A layer whose weights a kernel of the same stream has just written reads the new ones."""
    g = torch.Generator(device="cuda").manual_seed(9)
    m, held, args = _layers("softmax", 3, 1, 5, g)
    x, pos = _rand(g, 3, 256), torch.tensor([5], dtype=torch.int32, device="cuda")
    w = [p.clone() for p in (m.w_in, m.w_o)]
    want = m(*args(x, pos, [t.clone() for t in held]))
    for _ in range(50):
        m.w_in.zero_(), m.w_o.zero_()
        m(*args(x, pos, [t.clone() for t in held]))
        h = [t.clone() for t in held]
        m.w_o.copy_(w[1]), m.w_in.copy_(w[0])
        assert torch.equal(m(*args(x, pos, h)), want)
