"""The many-row int4 kernel (weights de-quantised into tensor memory) against the unpacked weights through 64-bit products: edges of row
tiles (128, 192, 256) and several tiles a block, a last column tile that is not full, one and many steps of 128 k, several groups a row, fractional zeros, a bias."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [1, 64, 65, 129, 192, 193, 256, 257, 600])
@pytest.mark.parametrize("N,K,group", [(16, 128, 128), (144, 384, 128), (1000 // 16 * 16, 512, 512), (272, 1280, 256), (2560, 640, 640)])
@pytest.mark.parametrize("zero,bias", [("whole", False), ("fraction", True), ("beyond", False)])
def test_int4_rows(M, N, K, group, zero, bias):
    from lit_llama import _native as NV
    from lit_llama.quantization import ColBlockQuantizedLinear

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    prev = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        lin = ColBlockQuantizedLinear(K, N, bias, bits=4, tile_cols=group).to("cuda")
    finally:
        torch.set_default_dtype(prev)
    lin.quant_weight.copy_(torch.randint(0, 256, lin.quant_weight.shape, generator=g, device="cuda", dtype=torch.uint8))
    lin.scales.copy_(torch.rand(lin.scales.shape, generator=g, device="cuda") * 0.02 + 0.005)
    z = torch.randint(0, 16, lin.zeros.shape, generator=g, device="cuda").float()
    lin.zeros.copy_(z + 0.37 if zero == "fraction" else z * 20.0 - 100.0 if zero == "beyond" else z)
    if bias:
        lin.bias.copy_(torch.randn(N, generator=g, device="cuda"))
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    y = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")            # a guard row behind the output
    NV.call("ll_int4_rows", NV.ptr(lin.quant_weight), NV.ptr(lin.scales), NV.ptr(lin.zeros), NV.ptr(x), NV.ptr(lin.bias), NV.ptr(y), M, N, K, group,
            NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int4_rows_error") == 0 and bool((y[M] == 7.0).all())
    w = lin.get_weight(dtype=torch.bfloat16).double()
    want = x.double() @ w.t() + (lin.bias.double() if bias else 0.0)
    size = x.double().abs() @ w.abs().t()
    # the same bf16 weights; fp32 sums (K roundings of 2^-24 of the terms' sizes) and one rounding to bf16
    assert ((y[:M].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * K * 2.0 ** -24 + 1e-30).all()


def test_module_route_and_refusals():
    from lit_llama import _native as NV
    from lit_llama.quantization import ColBlockQuantizedLinear

    assert NV.call_ret("ll_int4_rows_supported", 4096, 4096, 128) == 1
    for n, k, group in ((4097, 4096, 128), (4096, 4096, 64), (4096, 4096, 96), (4096, 200, 200)):
        assert NV.call_ret("ll_int4_rows_supported", n, k, group) == 0
    g = torch.Generator(device="cuda").manual_seed(0)
    lin = ColBlockQuantizedLinear(256, 48, False, bits=4, tile_cols=64).to("cuda", torch.bfloat16)      # groups of 64: the unpacked route
    lin.quant_weight.copy_(torch.randint(0, 256, lin.quant_weight.shape, generator=g, device="cuda", dtype=torch.uint8))
    lin.scales.fill_(0.01)
    lin.zeros.fill_(8.0)
    x = torch.randn((300, 256), generator=g, device="cuda").to(torch.bfloat16)
    want = x.float() @ lin.get_weight(torch.float32).t()
    assert (lin(x).float() - want).abs().max() <= 2.0 ** -7 * want.abs().max()


@pytest.mark.parametrize("M", [8192, 8193])
def test_longest_steps(M):
    """The last step of the kernel and the first one of the unpacked copy."""
    from lit_llama.quantization import ColBlockQuantizedLinear

    g = torch.Generator(device="cuda").manual_seed(M)
    lin = ColBlockQuantizedLinear(256, 144, False, bits=4, tile_cols=128).to("cuda", torch.bfloat16)
    lin.quant_weight.copy_(torch.randint(0, 256, lin.quant_weight.shape, generator=g, device="cuda", dtype=torch.uint8))
    lin.scales.fill_(0.01)
    lin.zeros.fill_(8.0)
    x = torch.randn((M, 256), generator=g, device="cuda").to(torch.bfloat16)
    w = lin.get_weight(torch.bfloat16).double()
    want, size = x.double() @ w.t(), x.double().abs() @ w.abs().t()
    assert ((lin(x).double() - want).abs() <= want.abs() * 2.0 ** -8 + size * 256 * 2.0 ** -24 + 1e-30).all()


@pytest.mark.parametrize("tile_rows", [128, 192, 256])
@pytest.mark.parametrize("grid", [1, 2, 5])
@pytest.mark.parametrize("M,N,K,group", [(513, 400, 128, 128), (700, 272, 384, 128), (260, 1040, 640, 640), (513, 528, 1280, 256)])
def test_blocks_that_walk_several_tiles(tile_rows, grid, M, N, K, group):
    """Every tile size with few blocks, so that each walks three tiles and more: one, three, five and ten steps a tile (the four groups take
    every fourth step, across tiles), partial last tiles of rows and columns, fractional zeros, a bias."""
    from lit_llama import _native as NV
    from lit_llama.quantization import ColBlockQuantizedLinear

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    lin = ColBlockQuantizedLinear(K, N, True, bits=4, tile_cols=group).to("cuda", torch.bfloat16)
    lin.quant_weight.copy_(torch.randint(0, 256, lin.quant_weight.shape, generator=g, device="cuda", dtype=torch.uint8))
    lin.scales.copy_(torch.rand(lin.scales.shape, generator=g, device="cuda") * 0.02 + 0.005)
    z = torch.randint(0, 16, lin.zeros.shape, generator=g, device="cuda").float()
    z[::3] += 0.37                                                     # whole zeros beside fractional ones
    lin.zeros.copy_(z)
    lin.bias.copy_(torch.randn(N, generator=g, device="cuda"))
    x = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    y = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    assert ((M + tile_rows - 1) // tile_rows) * ((N + 127) // 128) >= 3 * grid or grid == 5
    NV.call("ll_int4_rows_form", NV.ptr(lin.quant_weight), NV.ptr(lin.scales), NV.ptr(lin.zeros), NV.ptr(x), NV.ptr(lin.bias), NV.ptr(y), M, N, K,
            group, tile_rows, grid, NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int4_rows_error") == 0 and bool((y[M] == 7.0).all())
    w = lin.get_weight(dtype=torch.bfloat16).double()
    want, size = x.double() @ w.t() + lin.bias.double(), x.double().abs() @ w.abs().t()
    assert ((y[:M].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * K * 2.0 ** -24 + 1e-30).all()
