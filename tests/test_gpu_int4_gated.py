"""Two int4 layers and their gated product in one kernel (weights de-quantised into tensor memory; past 6144 rows a bf16 copy of each) against
64-bit products of the unpacked weights, and the module's choice between the one kernel and the separate layers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _layer(N, K, group, zero, bias, seed):
    from lit_llama.quantization import ColBlockQuantizedLinear

    g = torch.Generator(device="cuda").manual_seed(seed)
    prev = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        lin = ColBlockQuantizedLinear(K, N, bias, bits=4, tile_cols=group).to("cuda")
    finally:
        torch.set_default_dtype(prev)
    lin.quant_weight.copy_(torch.randint(0, 256, lin.quant_weight.shape, generator=g, device="cuda", dtype=torch.uint8))
    lin.scales.copy_((torch.rand(lin.scales.shape, generator=g, device="cuda") + 0.5) * 0.2 * K ** -0.5)
    z = torch.randint(4, 12, lin.zeros.shape, generator=g, device="cuda").float()
    if zero == "mixed":                                        # whole zeros beside fractional ones
        z[::3] += 0.37
    lin.zeros.copy_(z)
    if bias:
        lin.bias.copy_(torch.randn(N, generator=g, device="cuda"))
    return lin


def _close(h, x, l1, l2):
    """h = bf16(bf16(silu(a)) * b) of a, b rounded to bf16: a and b may be a rounding off where their fp32 sums differ in order (2^-8 each),
    silu's slope is at most 1.1, and two more roundings follow."""
    a, b = [x.double() @ lin.get_weight(torch.bfloat16).double().t() + (0.0 if lin.bias is None else lin.bias.double()) for lin in (l1, l2)]
    want = a * torch.sigmoid(a) * b
    assert ((h.double() - want).abs() <= 1.1 * a.abs() * 2.0 ** -8 * b.abs() + want.abs() * 3 * 2.0 ** -8 + 1e-5).all()


@pytest.mark.parametrize("tile_rows,grid", [(0, 0), (128, 2), (160, 4), (192, 2), (224, 4), (256, 2)])
@pytest.mark.parametrize("M,N,K,group", [(1, 16, 128, 128), (129, 144, 384, 128), (513, 272, 640, 640), (300, 400, 1280, 256), (700, 528, 768, 128)])
@pytest.mark.parametrize("zero,bias", [("whole", False), ("mixed", True)])
def test_gated_rows(tile_rows, grid, M, N, K, group, zero, bias):
    from lit_llama import _native as NV

    l1, l2 = _layer(N, K, group, zero, bias, M + N), _layer(N, K, group, "whole", bias, M + K)
    x = torch.randn((M, K), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    h = torch.full((M + 1, N), 7.0, dtype=torch.bfloat16, device="cuda")
    NV.call("ll_int4_rows_gated", NV.ptr(l1.quant_weight), NV.ptr(l1.scales), NV.ptr(l1.zeros), NV.ptr(l1.bias), NV.ptr(l2.quant_weight),
            NV.ptr(l2.scales), NV.ptr(l2.zeros), NV.ptr(l2.bias), NV.ptr(x), NV.ptr(h), M, N, K, group, tile_rows, grid, NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int4_rows_error") == 0 and bool((h[M] == 7.0).all())
    _close(h[:M], x, l1, l2)


@pytest.mark.parametrize("M", [129, 6144, 6145])
def test_module_takes_the_one_kernel_and_hooks_keep_the_layers(M):
    from lit_llama.model import MLP, LLaMAConfig
    from lit_llama.quantization import gated_pair
    from lit_llama.utils import EmptyInitOnDevice, quantization

    with EmptyInitOnDevice(device="cuda", dtype=torch.bfloat16), quantization("gptq.int4", groupsize=128):
        mlp = MLP(LLaMAConfig(n_embd=256, n_head=2)).eval()
    H = mlp.c_fc1.out_features
    mlp.c_fc1, mlp.c_fc2, mlp.c_proj = _layer(H, 256, 128, "mixed", False, 1), _layer(H, 256, 128, "whole", False, 2), _layer(256, H, 128, "whole", False, 3)
    x = torch.randn((1, M, 256), generator=torch.Generator(device="cuda").manual_seed(M), device="cuda").to(torch.bfloat16)
    h = gated_pair(mlp.c_fc1, mlp.c_fc2, x)
    assert h is not None and h.shape == (1, M, H)
    _close(h[0], x[0], mlp.c_fc1, mlp.c_fc2)
    y = mlp(x)
    seen = []
    handle = mlp.c_fc1.register_forward_hook(lambda _m, inp, _out: seen.append(inp[0].shape))
    assert gated_pair(mlp.c_fc1, mlp.c_fc2, x) is None
    y_hooked = mlp(x)
    handle.remove()
    assert seen == [x.shape]                                   # a calibration hook sees the layer's input as before
    size = y.double().abs().mean()
    assert (y.double() - y_hooked.double()).abs().max() <= 0.05 * size + 0.05 * y.double().abs().max()
    mlp.c_fc2.forward = lambda inp: inp                        # a forward set on the instance is called
    assert gated_pair(mlp.c_fc1, mlp.c_fc2, x) is None
