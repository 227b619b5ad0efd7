"""Batches of up to 128 rows through int4 layers (one range of steps per SM, partial sums added in the order of k) against 64-bit products of the
unpacked weights: each size of the row tile and its edges, ranges that begin and end inside a tile, cross several, or hold less than one, last
columns that fill no tile, several groups a row, fractional zeros, a bias; the same for the gated pair."""
import pytest
import torch

from tests.test_gpu_int4_gated import _close, _layer

pytestmark = pytest.mark.gpu

SIZES = [(16, 128, 128), (144, 640, 128), (272, 1280, 256), (528, 768, 768), (1040, 2048, 128), (2560, 256, 128)]


def _scratch(NV, M, N, K, layers, grid):
    n = NV.call_ret("ll_int4_batch_scratch_bytes", M, N, K, layers, grid)
    return torch.full((n // 4 + 4,), float("nan"), dtype=torch.float32, device="cuda"), n // 4


@pytest.mark.parametrize("M", [1, 9, 16, 17, 32, 33, 64, 65, 127, 128])
@pytest.mark.parametrize("N,K,group", SIZES)
@pytest.mark.parametrize("grid,zero,bias", [(0, "whole", False), (1, "mixed", True), (3, "mixed", False), (7, "whole", True), (29, "mixed", True)])
def test_int4_batch(M, N, K, group, grid, zero, bias):
    from lit_llama import _native as NV

    lin = _layer(N, K, group, zero, bias, M + N + K)
    x = torch.randn((M, K), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    y = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    ws, used = _scratch(NV, M, N, K, 1, grid)
    NV.call("ll_int4_batch", NV.ptr(lin.quant_weight), NV.ptr(lin.scales), NV.ptr(lin.zeros), NV.ptr(x), NV.ptr(lin.bias), NV.ptr(y), NV.ptr(ws), M, N, K,
            group, grid, NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int4_batch_error") == 0 and bool((y[M] == 7.0).all()) and bool(ws[used:].isnan().all())
    w = lin.get_weight(torch.bfloat16).double()
    want, size = x.double() @ w.t() + (lin.bias.double() if bias else 0.0), x.double().abs() @ w.abs().t() + 4.0
    # the same bf16 weights; fp32 sums (K roundings of 2^-24 of the terms' sizes) and one rounding to bf16
    assert ((y[:M].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * K * 2.0 ** -24).all()


@pytest.mark.parametrize("M", [1, 16, 33, 128])
@pytest.mark.parametrize("N,K,group", SIZES)
@pytest.mark.parametrize("grid,zero,bias", [(0, "whole", False), (5, "mixed", True), (31, "mixed", False)])
def test_int4_batch_gated(M, N, K, group, grid, zero, bias):
    from lit_llama import _native as NV

    l1, l2 = _layer(N, K, group, zero, bias, M + N), _layer(N, K, group, "whole", bias, M + K)
    x = torch.randn((M, K), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    h = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    ws, used = _scratch(NV, M, N, K, 2, grid)
    NV.call("ll_int4_batch_gated", NV.ptr(l1.quant_weight), NV.ptr(l1.scales), NV.ptr(l1.zeros), NV.ptr(l1.bias), NV.ptr(l2.quant_weight),
            NV.ptr(l2.scales), NV.ptr(l2.zeros), NV.ptr(l2.bias), NV.ptr(x), NV.ptr(h), NV.ptr(ws), M, N, K, group, grid, NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int4_batch_error") == 0 and bool((h[M] == 7.0).all()) and bool(ws[used:].isnan().all())
    _close(h[:M], x, l1, l2)
