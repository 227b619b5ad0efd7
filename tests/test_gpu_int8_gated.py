"""The gated pair of two llm.int8 layers (x prepared once, both products and their finish in one kernel per step) against the layers one after
the other: the same integer sums, roundings and order of outliers, so the same numbers up to 64 outliers a block."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(N, K, bias, seed):
    from lit_llama.quantization import Linear8bitLt

    g = torch.Generator(device="cuda").manual_seed(seed)
    lin = Linear8bitLt(K, N, bias=bias, device="cuda", dtype=torch.bfloat16)
    state = {"weight": torch.randn((N, K), generator=g, device="cuda") * K ** -0.5}
    if bias:
        state["bias"] = torch.randn(N, generator=g, device="cuda")
    lin.load_state_dict(state)
    return lin


@pytest.mark.parametrize("M", [1, 16, 17, 33, 64, 65, 128, 191, 256, 257, 600])
@pytest.mark.parametrize("N,K", [(33, 128), (64, 256), (200, 640), (1000, 384), (9600, 128)])
@pytest.mark.parametrize("outliers,bias,transposed", [(0, False, True), (3, True, True), (64, True, False), (100, False, True)])
def test_gated_pair_is_the_two_layers(M, N, K, outliers, bias, transposed):
    from lit_llama import _native as NV
    from lit_llama.quantization import gated_pair

    l1, l2 = _layer(N, K, bias, N + K), _layer(N, K, bias, N + K + 1)
    if not transposed:
        l1._cbt = l2._cbt = None
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, K), generator=g, device="cuda") * 0.5
    cols = torch.randperm(K, generator=g, device="cuda")[:outliers]
    rows = torch.rand(M, generator=g, device="cuda") < 0.5             # a feature stands out in some blocks of 64 rows and not in others
    x[:, cols] = torch.where(rows[:, None], torch.sign(x[:, cols]) * (8.0 + x[:, cols].abs()), x[:, cols])
    x = x.to(torch.bfloat16)
    h = gated_pair(l1, l2, x.view(1, M, K))
    a, b = l1(x), l2(x)
    want = torch.empty_like(a)
    NV.call("ll_silu_mul", NV.ptr(a), NV.ptr(b), NV.ptr(want), NV.dtype_code(a.dtype), a.numel(), NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int8_tc_error") == 0 and h.shape == (1, M, N)
    # silu from a fast exponential and division may end on the other bf16 neighbour: a rounding each of it and of the product
    assert ((h[0].double() - want.double()).abs() <= want.double().abs() * 2.0 ** -7).all()
    if outliers <= 64:
        same = torch.empty_like(a)                                     # the layers' outputs themselves are the same: silu of the same numbers
        same.copy_((a.float() / (1.0 + torch.exp(-a.float()))).to(torch.bfloat16) * b)
        assert (h[0] == want).float().mean() >= 0.99 and (same == want).float().mean() >= 0.99


def test_hooks_keep_the_layers():
    from lit_llama.quantization import gated_pair

    l1, l2 = _layer(64, 128, False, 1), _layer(64, 128, False, 2)
    x = torch.randn((4, 128), device="cuda", dtype=torch.bfloat16)
    assert gated_pair(l1, l2, x) is not None and gated_pair(l1, l2, x.float()) is None
    handle = l2.register_forward_hook(lambda *_: None)
    assert gated_pair(l1, l2, x) is None
    handle.remove()
    assert gated_pair(l1, l2, x) is not None
