"""A layer of several rows called once and then captured, in a process that has made no library product before: the captured step takes the library's."""
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

SCRIPT = """
import sys, torch
sys.path.insert(0, sys.argv[1])
torch.set_grad_enabled(False)
g = torch.Generator(device="cuda").manual_seed(0)
rand = lambda *s: torch.randn(s, generator=g, device="cuda").to(torch.bfloat16)
T = 40
if sys.argv[2] == "softmax":
    from lit_llama.rotary import RotarySpec
    from lit_llama.softmax_attention import SoftmaxAttention, SoftmaxAttentionSpec
    m = SoftmaxAttention(SoftmaxAttentionSpec(width=256, heads=4, kv_heads=2, dim=64, vdim=64, scale=0.125, eps=1e-5, rotary=RotarySpec(32), qk_norm=True),
                         torch.bfloat16, "cuda")
    held = [rand(1, T, 128) for _ in range(2)]
    call = lambda x, pos, h: m(x, 1, T, pos, h)
elif sys.argv[2] == "latent":
    from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec
    spec = LatentAttentionSpec(width=256, heads=4, nope_dim=64, rot_dim=32, v_dim=64, kv_rank=128, window=100, scale=96 ** -0.5)
    m, rope = LatentAttention(spec, torch.bfloat16, "cuda"), spec.rope_table(T, "cuda")
    held = [rand(1, T, spec.row)]
    call = lambda x, pos, h: m(x, 1, T, pos, rope, h[0])
else:
    from lit_llama.recurrence import MatrixMemoryMixer, MatrixMemorySpec
    m = MatrixMemoryMixer(MatrixMemorySpec(256, 4, 64, 64, 15.0, 1e-5), torch.bfloat16, "cuda")
    held = [torch.zeros(n, dtype=torch.float32, device="cuda") for n in m.state_shapes(1)]
    call = lambda x, pos, h: m(x, 1, T, pos, h)
for p in m.parameters():
    p.copy_(rand(*p.shape) * (p.shape[-1] ** -0.5 if p.dim() > 1 else 0.1) + (0.0 if p.dim() > 1 else 1.0))
x, pos = rand(T, 256), torch.arange(T, dtype=torch.int32, device="cuda")
want = call(x, pos, [t.clone() for t in held]).double()
h = [t.clone() for t in held]
graph = torch.cuda.CUDAGraph()
with torch.cuda.graph(graph):
    y = call(x, pos, h)
graph.replay()
assert float((y.double() - want).norm()) <= 2.0 ** -6 * float(want.norm())
"""


@pytest.mark.parametrize("kind", ["softmax", "latent", "matrix"])
def test_captured_after_one_call(kind):
    import lit_llama

    r = subprocess.run([sys.executable, "-c", SCRIPT, str(Path(lit_llama.__file__).parent.parent), kind], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stderr[-2000:]
