"""A gated feed-forward of int4 layers through its module, at 1 to 128 rows: the values, which kernels run, when the single-token streams are made,
and what a captured step finds."""
import pytest
import torch

from tests.test_gpu_int4_gated import _layer

pytestmark = pytest.mark.gpu


def _mlp(K=256, H=512, zero="whole"):
    from lit_llama.model import MLP

    mlp = MLP.__new__(MLP)
    torch.nn.Module.__init__(mlp)
    mlp.c_fc1, mlp.c_fc2, mlp.c_proj = _layer(H, K, 128, zero, False, 1), _layer(H, K, 128, "whole", False, 2), _layer(K, H, 128, "whole", False, 3)
    return mlp


def _x(M, K=256):
    return torch.randn((M, K), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)


def _calls(monkeypatch):
    from lit_llama import _native as NV

    names, call, gemv = [], NV.call, NV.gemv
    monkeypatch.setattr(NV, "call", lambda name, *a: (names.append(name), call(name, *a))[1])
    monkeypatch.setattr(NV, "gemv", lambda a: (names.append("gemv2" if a.epilogue == NV.EPI_SWIGLU else "gemv"), gemv(a))[1])
    return names


def _check(h, x, l1, l2):
    """h = bf16(bf16(silu(a)) * b): a and b are sums of weights that are rounded to bf16 or not (2^-9 of each term), rounded to bf16 themselves
    (2^-8); silu's slope is at most 1.1; two more roundings follow."""
    a, b, ea, eb = [], [], [], []
    for lin, v, e in ((l1, a, ea), (l2, b, eb)):
        w = lin.get_weight(torch.bfloat16).double()
        v.append(x.double() @ w.t())
        e.append(x.double().abs() @ w.abs().t() * 2.0 ** -9 + v[0].abs() * 2.0 ** -8)
    a, b, ea, eb = a[0], b[0], ea[0], eb[0]
    s = a * torch.sigmoid(a)
    assert ((h.double() - s * b).abs() <= 1.05 * (1.1 * ea * (b.abs() + eb) + s.abs() * eb) + (s * b).abs() * 2.0 ** -7 + 1e-5).all()


@pytest.mark.parametrize("M", [1, 2, 5, 8, 9, 16, 17, 64, 127, 128])
@pytest.mark.parametrize("zero", ["whole", "mixed"])
def test_values(M, zero, monkeypatch):
    from lit_llama.quantization import gated_pair

    mlp, x = _mlp(zero=zero), _x(M)
    names = _calls(monkeypatch)
    h = gated_pair(mlp.c_fc1, mlp.c_fc2, x)
    assert names[-1] == ("gemv2" if M <= 8 else "ll_int4_batch_gated")
    _check(h, x, mlp.c_fc1, mlp.c_fc2)


@pytest.mark.parametrize("M", [1, 8, 16, 128])
def test_layers_of_different_parameter_dtypes(M, monkeypatch):
    """fp32 scales beside bf16 ones of the same numbers: the streams hold both, the byte kernels take neither layer of the pair."""
    from lit_llama.quantization import gated_pair

    mlp, x = _mlp(), _x(M)
    mlp.c_fc2.scales, mlp.c_fc2.zeros = mlp.c_fc2.scales.float(), mlp.c_fc2.zeros.float()
    names = _calls(monkeypatch)
    h = gated_pair(mlp.c_fc1, mlp.c_fc2, x)
    assert (h is None) == (M > 8)
    if h is not None:
        _check(h, x, mlp.c_fc1, mlp.c_fc2)
    y = mlp(x)
    assert "ll_int4_batch_gated" not in names
    mlp.c_fc2.scales, mlp.c_fc2.zeros = mlp.c_fc2.scales.to(torch.bfloat16), mlp.c_fc2.zeros.to(torch.bfloat16)
    mlp.c_fc2._streams = {}
    want = mlp(x)
    assert (y.double() - want.double()).norm() <= 0.01 * want.double().norm()


@pytest.mark.parametrize("M", [9, 128])
def test_a_batch_makes_the_streams_of_the_tokens_after_it(M, monkeypatch):
    """Once, for all three layers: the next token prepares nothing, and a step captured right after the batch runs the GEMV."""
    mlp = _mlp()
    names = _calls(monkeypatch)
    mlp(_x(M))
    assert names.count("ll_int4_prepare") == 3
    mlp(_x(M))
    assert names.count("ll_int4_prepare") == 3
    del names[:]
    x, graph = _x(1), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = mlp(x)
    assert names == ["gemv2", "gemv"]
    graph.replay()
    assert torch.equal(y, mlp(x))
    assert "ll_int4_prepare" not in names


def test_a_captured_step_without_streams(monkeypatch):
    """Nothing is prepared under capture: the byte kernels serve single tokens then, with the same weights."""
    mlp, x = _mlp(), _x(1)
    names = _calls(monkeypatch)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = mlp(x)
    assert "ll_int4_prepare" not in names and "gemv" not in names and "gemv2" not in names
    graph.replay()
    want = mlp(x)
    assert names[-1] == "gemv" and (y.double() - want.double()).norm() <= 0.01 * want.double().norm()
