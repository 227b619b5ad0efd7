"""Layers whose first launch is a kernel with tensor maps, as the first thing that a new thread does: the same numbers as in the thread before."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(*shape, seed=0):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(torch.bfloat16)


def _int4(N, K, seed):
    from lit_llama.quantization import ColBlockQuantizedLinear

    lin = ColBlockQuantizedLinear(K, N, False, bits=4, tile_cols=128).to("cuda", torch.bfloat16)
    lin.quant_weight.copy_(torch.randint(0, 256, lin.quant_weight.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed), dtype=torch.uint8))
    lin.scales.fill_(0.2 * K ** -0.5), lin.zeros.fill_(7.0)
    return lin


def _layer(kind):
    """(a call that makes its maps first, the output)"""
    if kind in ("int4 batch", "int4 rows", "int4 gated rows"):
        from lit_llama.quantization import gated_pair

        x, lin = _rand(32 if kind == "int4 batch" else 200, 512), [_int4(256, 512, i) for i in range(2)]
        return (lambda: gated_pair(*lin, x)) if "gated" in kind else lambda: lin[0](x)
    if kind == "bf16 product":
        from lit_llama import _native as N

        w, x, y = _rand(256, 512, seed=1), _rand(300, 512), torch.empty((300, 256), dtype=torch.bfloat16, device="cuda")
        return lambda: N.call("ll_gemm_bf16_tc", N.ptr(x), N.ptr(w), None, N.ptr(y), 300, 256, 512, N.stream()) or y.clone()
    from lit_llama.rotary import RotarySpec
    from lit_llama.softmax_attention import SoftmaxAttention, SoftmaxAttentionSpec

    m = SoftmaxAttention(SoftmaxAttentionSpec(width=256, heads=4, kv_heads=2, dim=64, vdim=64, scale=0.125, eps=1e-5, rotary=RotarySpec(32), qk_norm=True),
                         torch.bfloat16, "cuda")
    for i, p in enumerate(m.parameters()):
        p.copy_(_rand(*p.shape, seed=i) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 1.0))
    x, pos, kv = _rand(60, 256), torch.arange(60, dtype=torch.int32, device="cuda"), [torch.zeros((1, 64, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2)]
    return lambda: m(x, 1, 60, pos, kv)


@pytest.mark.parametrize("kind", ["int4 batch", "int4 rows", "int4 gated rows", "bf16 product", "softmax layer"])
@torch.no_grad()
def test_first_call_of_a_thread(kind):
    call = _layer(kind)
    want = call()
    call()                                                 # (memory for the thread's call is in the pool)
    torch.cuda.synchronize()
    got = []

    def work():
        with torch.no_grad():
            try:
                got.append(call())
            except RuntimeError as e:
                got.append(e)

    t = threading.Thread(target=work)
    t.start()
    t.join()
    assert isinstance(got[0], torch.Tensor), got[0]
    assert torch.equal(got[0], want)
