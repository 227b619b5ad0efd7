"""Dense products by pairs of CTAs against 64-bit products of the same bf16 operands: edges of the 256-row and 256- or 128-column tiles, k that
is no multiple of a stage, fewer and more tiles than pairs, several bands of row tiles, rows of y that TMA cannot store, a bias; the gated form
against the separate steps' roundings."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _operands(M, N, K, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((M, K), generator=g, device="cuda").bfloat16()
    w = [(torch.randn((N, K), generator=g, device="cuda") * K ** -0.5).bfloat16() for _ in range(2)]
    b = [torch.randn(N, generator=g, device="cuda").bfloat16() for _ in range(2)]
    return x, w, b


@pytest.mark.parametrize("columns", [128, 256])
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (128, 256, 64), (129, 264, 72), (256, 128, 512), (257, 1000, 328), (300, 257, 200), (2049, 520, 136),
                                   (2500, 2304, 64), (600, 19200, 128)])
@pytest.mark.parametrize("bias", [False, True])
def test_pair_product(columns, M, N, K, bias):
    from lit_llama import _native as NV

    x, w, b = _operands(M, N, K, M + N + K)
    y = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    NV.call("ll_gemm_bf16_tc_form", NV.ptr(x), NV.ptr(w[0]), NV.ptr(b[0] if bias else None), NV.ptr(y), M, N, K, columns, NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_gemm_bf16_tc_error") == 0 and bool((y[M] == 7.0).all())
    want = x.double() @ w[0].double().t() + (b[0].double() if bias else 0.0)
    size = x.double().abs() @ w[0].double().abs().t() + 4.0
    # fp32 sums (K roundings of 2^-24 of the terms' sizes) and one rounding to bf16
    assert ((y[:M].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * K * 2.0 ** -24).all()


@pytest.mark.parametrize("M,N,K", [(1, 8, 64), (256, 128, 128), (257, 136, 200), (2049, 1000, 72), (300, 9600, 64)])
@pytest.mark.parametrize("bias", [False, True])
def test_gated_pair_product(M, N, K, bias):
    """h = bf16(bf16(silu(a)) * b) of a, b rounded to bf16: a and b may be a rounding off where their fp32 sums differ in order (2^-8 each),
    silu's slope is at most 1.1, and two more roundings follow."""
    from lit_llama import _native as NV

    x, w, b = _operands(M, N, K, M + N + K)
    h = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    b1, b2 = (b if bias else (None, None))
    NV.call("ll_gemm_bf16_gated", NV.ptr(x), NV.ptr(w[0]), NV.ptr(b1), NV.ptr(w[1]), NV.ptr(b2), NV.ptr(h), M, N, K, NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_gemm_bf16_tc_error") == 0 and bool((h[M] == 7.0).all())
    a, c = [x.double() @ w[i].double().t() + (b[i].double() if bias else 0.0) for i in range(2)]
    want = a * torch.sigmoid(a) * c
    tol = 1.1 * a.abs() * 2.0 ** -8 * c.abs() + want.abs() * 3 * 2.0 ** -8 + 1e-5
    assert ((h[:M].double() - want).abs() <= tol).all()
