"""Quantized layers called by two threads on one stream, and captured graphs replayed on two streams: every result as that of the call alone."""
import threading

import pytest
import torch

pytestmark = pytest.mark.gpu

KINDS = ["rows", "gated_rows", "batch", "gated_batch", "int8", "gated_int8", "int8_prompt"]


def _int4(N, K, seed):
    from lit_llama.quantization import ColBlockQuantizedLinear

    g = torch.Generator(device="cuda").manual_seed(seed)
    lin = ColBlockQuantizedLinear(K, N, False, bits=4, tile_cols=128).to("cuda", torch.bfloat16)
    lin.quant_weight.copy_(torch.randint(0, 256, lin.quant_weight.shape, generator=g, device="cuda", dtype=torch.uint8))
    lin.scales.copy_((torch.rand(lin.scales.shape, generator=g, device="cuda") + 0.5) * 0.2 * K ** -0.5)
    lin.zeros.copy_(torch.randint(4, 12, lin.zeros.shape, generator=g, device="cuda").float())
    return lin


def _int8(N, K, seed):
    from lit_llama.quantization import Linear8bitLt

    lin = Linear8bitLt(K, N, bias=False, device="cuda", dtype=torch.bfloat16)
    lin.load_state_dict({"weight": torch.randn((N, K), generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda") * 0.05})
    return lin


def _calls(kind):
    """Two calls of the same sizes on different rows."""
    from lit_llama.quantization import gated_pair

    g = torch.Generator(device="cuda").manual_seed(1)
    M, N, K = {"rows": (300, 1024, 11008), "gated_rows": (300, 11008, 4096), "int8_prompt": (130, 1024, 2048)}.get(kind, (32, 1024, 2048))
    layers = [(_int8 if "int8" in kind else _int4)(N, K, i) for i in range(2 if "gated" in kind else 1)]
    xs = [torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16) for _ in range(2)]
    for i, x in enumerate(xs):
        x[:, 7 * i: 7 * i + 3] *= 30.0                    # outlier features, others in either call
    run = (lambda x: gated_pair(*layers, x)) if "gated" in kind else layers[0]
    return [lambda x=x: run(x) for x in xs]


@pytest.mark.parametrize("kind", KINDS)
@torch.no_grad()
def test_two_threads_on_one_stream(kind):
    calls = _calls(kind)
    want = [c() for c in calls]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        with torch.no_grad():
            try:
                for _ in range(200):
                    if not torch.equal(calls[i](), want[i]):
                        wrong.append(i)
            except RuntimeError as e:
                wrong.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("kind", KINDS)
@torch.no_grad()
def test_two_graphs_on_two_streams(kind):
    calls = _calls(kind)
    want = [c() for c in calls]
    torch.cuda.synchronize()
    graphs, outs, streams = [], [], [torch.cuda.Stream() for _ in range(2)]
    for c in calls:
        graphs.append(torch.cuda.CUDAGraph())
        with torch.cuda.graph(graphs[-1]):
            outs.append(c())
    for _ in range(200):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(o, w) for o, w in zip(outs, want))
