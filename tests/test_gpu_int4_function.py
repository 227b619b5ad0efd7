"""The reference's function for one packed weight (no module, no bias) against 64-bit sums of the de-quantised weights, at the rows where its kernel changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,dtype", [(1, torch.bfloat16), (9, torch.bfloat16), (16, torch.bfloat16), (128, torch.bfloat16), (129, torch.bfloat16), (300, torch.bfloat16),
                                     (6145, torch.bfloat16), (3, torch.float32), (40, torch.float32)])
@pytest.mark.parametrize("N,K", [(256, 512), (48, 384)])
def test_function(M, dtype, N, K):
    from lit_llama.quantization import qlinear_4bit_weight

    g = torch.Generator(device="cuda").manual_seed(M + N)
    packed = torch.randint(0, 256, (K // 2, N), generator=g, device="cuda", dtype=torch.uint8)
    scales = (torch.rand((N, 1), generator=g, device="cuda") * 0.05 + 0.01).to(torch.bfloat16)
    zeros = torch.randint(0, 16, (N, 1), generator=g, device="cuda").to(torch.bfloat16)
    x = torch.randn((M, K), generator=g, device="cuda").to(dtype)
    got = qlinear_4bit_weight(x, packed.t(), scales, zeros).double()
    q = torch.stack([packed & 15, packed >> 4], dim=1).reshape(K, N).t().double()
    w = (q - zeros.double()) * scales.double()
    want, size = x.double() @ w.t(), x.double().abs() @ w.abs().t()
    # bf16: weights rounded to bf16 (2^-9 of each term), the output too (2^-8 beside the other neighbour); fp32: sums of K terms
    bound = size * 2.0 ** -9 + want.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else size * (K * 2.0 ** -24)
    assert got.shape == (M, N) and ((got - want).abs() <= 1.01 * bound + 1e-5).all()
