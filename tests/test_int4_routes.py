"""Which kernel a call of an int4 layer goes to, on the host: the library's launches are recorded instead of made."""
import pytest
import torch


@pytest.fixture
def launches(monkeypatch):
    from lit_llama import quantization as q

    names = []
    monkeypatch.setattr(q.N, "require_cuda", lambda *t: None)
    monkeypatch.setattr(q.N, "stream", lambda: 0)
    monkeypatch.setattr(q.N, "call", lambda name, *a: names.append(name))
    monkeypatch.setattr(q, "_INT8_WS", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return names


@pytest.mark.parametrize("M,dtype,last", [(4, torch.float32, "ll_qlinear_simt"), (16, torch.bfloat16, "ll_int4_batch"), (128, torch.bfloat16, "ll_int4_batch"),
                                          (300, torch.bfloat16, "ll_int4_rows"), (6145, torch.bfloat16, "ll_gemm_bf16_tc")])
def test_function_on_plain_tensors(launches, M, dtype, last):
    """The reference's function has no module: its layer's tensors are no buffers."""
    from lit_llama.quantization import qlinear_4bit_weight

    N, K = 256, 512
    weight = torch.zeros((K // 2, N), dtype=torch.uint8).t()
    scales = torch.ones((N, 1), dtype=torch.bfloat16)
    y = qlinear_4bit_weight(torch.zeros((M, K), dtype=dtype), weight, scales, torch.zeros_like(scales))
    assert y.shape == (M, N) and y.dtype == dtype and launches[-1] == last
