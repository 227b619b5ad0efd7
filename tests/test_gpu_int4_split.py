"""Many rows through int4 layers whose last wave of tiles is cut along k for all pairs of CTAs, against 64-bit products of the unpacked weights:
one part, many, of one step, of unequal steps, two a pair; whole waves before them and none; partial tiles; and the same sums from call to call."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# rows, columns, k, group, rows of a tile, blocks, parts (0: the rule's)
FORMS = [(1, 16, 128, 128, 128, 4, 1), (129, 144, 384, 128, 128, 6, 3), (300, 528, 1280, 256, 128, 8, 2), (300, 528, 1152, 128, 160, 16, 2),
         (513, 272, 640, 640, 224, 14, 2), (700, 784, 1280, 128, 256, 16, 3), (700, 784, 1152, 128, 192, 148, 4), (129, 1040, 2944, 128, 0, 0, 0),
         (520, 1040, 4096, 128, 0, 0, 0), (512, 4096, 11008, 128, 0, 0, 0), (1100, 4096, 4096, 128, 0, 0, 0)]


def _layer(N, K, group, bias, seed):
    from lit_llama.quantization import ColBlockQuantizedLinear

    g = torch.Generator(device="cuda").manual_seed(seed)
    lin = ColBlockQuantizedLinear(K, N, bias, bits=4, tile_cols=group).to("cuda", torch.bfloat16)
    lin.quant_weight.copy_(torch.randint(0, 256, lin.quant_weight.shape, generator=g, device="cuda", dtype=torch.uint8))
    lin.scales.copy_((torch.rand(lin.scales.shape, generator=g, device="cuda") + 0.5) * 0.2 * K ** -0.5)
    z = torch.randint(4, 12, lin.zeros.shape, generator=g, device="cuda").float()
    z[::3] += 0.37                                             # whole zeros beside fractional ones
    lin.zeros.copy_(z)
    if bias:
        lin.bias.copy_(torch.randn(N, generator=g, device="cuda"))
    return lin


def _scratch(M, N, K, layers, tile_rows, grid, parts):
    from lit_llama import _native as NV

    nbytes = NV.call_ret("ll_int4_rows_scratch_bytes", M, N, K, layers, tile_rows, grid, parts)
    return torch.full((nbytes + 16,), 255, dtype=torch.uint8, device="cuda"), nbytes       # (any contents: NaN as floats, -1 as counters)


@pytest.mark.parametrize("M,N,K,group,tile_rows,grid,parts", FORMS)
def test_split_rows(M, N, K, group, tile_rows, grid, parts):
    from lit_llama import _native as NV

    lin = _layer(N, K, group, True, M + N + K)
    x = torch.randn((M, K), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    y = torch.full((2, M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    scratch, nbytes = _scratch(M, N, K, 1, tile_rows, grid, parts)
    assert nbytes > 0 or parts == 0
    for out in y:
        NV.call("ll_int4_rows_split", NV.ptr(lin.quant_weight), NV.ptr(lin.scales), NV.ptr(lin.zeros), NV.ptr(x), NV.ptr(lin.bias), NV.ptr(out),
                NV.ptr(scratch) if nbytes else None, M, N, K, group, tile_rows, grid, parts, NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int4_rows_error") == 0 and bool((y[:, M] == 7.0).all()) and bool((scratch[nbytes:] == 255).all())
    w = lin.get_weight(dtype=torch.bfloat16).double()
    want, size = x.double() @ w.t() + lin.bias.double(), x.double().abs() @ w.abs().t()
    # one rounding to bf16 of an fp32 sum of K terms
    assert ((y[0, :M].double() - want).abs() <= want.abs() * 2.0 ** -8 + size * K * 2.0 ** -24 + 1e-30).all()
    assert torch.equal(y[0], y[1])


@pytest.mark.parametrize("M,N,K,group,tile_rows,grid,parts", FORMS)
def test_split_gated_rows(M, N, K, group, tile_rows, grid, parts):
    from lit_llama import _native as NV

    l1, l2 = _layer(N, K, group, True, M + N), _layer(N, K, group, False, M + K)
    x = torch.randn((M, K), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    h = torch.full((2, M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    scratch, nbytes = _scratch(M, N, K, 2, tile_rows, grid, parts)
    assert nbytes > 0 or parts == 0
    for out in h:
        NV.call("ll_int4_rows_gated_split", NV.ptr(l1.quant_weight), NV.ptr(l1.scales), NV.ptr(l1.zeros), NV.ptr(l1.bias), NV.ptr(l2.quant_weight),
                NV.ptr(l2.scales), NV.ptr(l2.zeros), None, NV.ptr(x), NV.ptr(out), NV.ptr(scratch) if nbytes else None, M, N, K, group, tile_rows,
                grid, parts, NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int4_rows_error") == 0 and bool((h[:, M] == 7.0).all()) and bool((scratch[nbytes:] == 255).all())
    ws = [lin.get_weight(torch.bfloat16).double() for lin in (l1, l2)]
    a, b = [x.double() @ w.t() + (0.0 if lin.bias is None else lin.bias.double()) for w, lin in zip(ws, (l1, l2))]
    # a and b are fp32 sums, 16 products to a step of the tensor cores, and rounded to bf16; silu's slope is at most 1.1; silu(a) and the product are
    # rounded again (one more for silu's own error)
    da, db = [v.abs() * 2.0 ** -8 + (x.double().abs() @ w.abs().t()) * (K / 16) * 2.0 ** -23 for v, w in zip((a, b), ws)]
    want = a * torch.sigmoid(a) * b
    err = (h[0, :M].double() - want).abs()
    assert (err <= 1.1 * da * (b.abs() + db) + (a * torch.sigmoid(a)).abs() * db + want.abs() * 3 * 2.0 ** -8 + 1e-30).all()
    assert torch.equal(h[0], h[1])
