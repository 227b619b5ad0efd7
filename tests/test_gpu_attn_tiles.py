"""Which tiles a block of the prompt attention takes, at the edges of the rule: three tiles, more blocks than SMs, a second round of blocks that is nearly full
and one that is not, and caps with and without a bound of their own, against the fp32 form of the same call."""
import pytest
import torch

from tests.test_gpu_attn_tc import _softmax

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case", [dict(T=300, B=30), dict(T=385, B=13), dict(T=513, B=20), dict(T=513, B=30), dict(T=640, B=20, window=400), dict(T=520, B=10, window=200),
                                  dict(T=513, B=20, cap=50.0, sink=True), dict(T=513, B=13, cap=80.0, slopes=True, gate=True), dict(T=300, B=30, cap=80.0)],
                         ids=lambda c: "-".join(f"{k}{v}" for k, v in c.items()))
def test_tiles_of_blocks(case):
    case = dict(case, past=3, ring=case["T"] + 5)
    got, top = _softmax(**case)
    want, _ = _softmax(**case, form=1)
    got, want = got.float(), want.float()
    # as in test_gpu_attn_tc: both round the same sum to bf16, the weights carry 16 bits
    assert torch.isfinite(got).all() and ((got - want).abs() <= want.abs() * 2.0 ** -7 + top * 2.0 ** -14).all()
