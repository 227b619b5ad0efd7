"""Scratch of quantized layers, on the host: the library's launches are recorded instead of made.  A call that begins while another one is still in the
library (two threads: the interpreter is let go there) must not be given the other's scratch."""
import gc
import threading
import weakref
from types import SimpleNamespace

import pytest
import torch

# entry -> where its scratch stands among the arguments
SCRATCH = {"ll_int4_rows_sized": 6, "ll_int4_rows_gated_sized": 10, "ll_int4_batch": 6, "ll_int4_batch_gated": 10}


@pytest.fixture
def library(monkeypatch):
    from lit_llama import quantization as q

    class Library:
        depth, inner, seen = 0, None, []

        def call(self, name, *a):
            if name not in SCRATCH:
                return
            self.seen.append((name, a[SCRATCH[name]]))
            if self.depth == 0 and self.inner is not None:
                self.depth = 1
                other = threading.Thread(target=self.inner)
                other.start()
                other.join()
                self.depth = 0

    lib = Library()
    lib.seen = []
    monkeypatch.setattr(q.N, "require_cuda", lambda *t: None)
    monkeypatch.setattr(q.N, "stream", lambda: 0)
    monkeypatch.setattr(q.N, "call", lib.call)
    monkeypatch.setattr(q, "_INT8_WS", {})
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return lib


def _int4(N, K):
    from lit_llama.quantization import ColBlockQuantizedLinear

    lin = ColBlockQuantizedLinear(K, N, False, bits=4, tile_cols=128).to(torch.bfloat16)
    lin.quant_weight.zero_(), lin.scales.fill_(1.0), lin.zeros.zero_()
    return lin


def _two_at_once(library, call):
    library.inner = call
    call()
    assert len(library.seen) == 2 and all(at for _, at in library.seen)
    return library.seen[0][1] != library.seen[1][1]


@pytest.mark.parametrize("M,N,K", [(300, 1024, 11008), (32, 256, 512)])
def test_one_layer(library, M, N, K):
    """Prompts with cut tiles, and batches."""
    lin, x = _int4(N, K), torch.zeros((M, K), dtype=torch.bfloat16)
    lin._make_step_stream = lambda x: None
    assert _two_at_once(library, lambda: lin(x))


@pytest.mark.parametrize("M,N,K", [(300, 11008, 4096), (32, 256, 512)])
def test_gated_layers(library, M, N, K):
    from lit_llama.quantization import gated_pair

    l1, l2, x = _int4(N, K), _int4(N, K), torch.zeros((M, K), dtype=torch.bfloat16)
    l1._make_step_stream = l2._make_step_stream = lambda x: None
    rows = SimpleNamespace(shape=x.shape, device=SimpleNamespace(type="cuda"), reshape=x.reshape)
    assert _two_at_once(library, lambda: gated_pair(l1, l2, rows))


def test_a_captured_call_has_its_own(library, monkeypatch):
    """Two captures of one thread on one stream, and the calls between them."""
    from lit_llama import quantization as q

    held = [q._int8_workspace(torch.device("cpu"), 1000)]
    assert q._int8_workspace(torch.device("cpu"), 1000) is held[0]
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: True)
    held += [q._int8_workspace(torch.device("cpu"), 1000) for _ in range(2)]
    assert len({t.data_ptr() for t in held}) == 3


def test_buffers_of_a_thread_go_with_it(monkeypatch):
    from lit_llama import quantization as q

    monkeypatch.setattr(q.N, "stream", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    before, made = len(q._INT8_WS), []
    t = threading.Thread(target=lambda: made.append(weakref.ref(q._int8_workspace(torch.device("cpu"), 5000))))
    t.start()
    t.join()
    del t
    gc.collect()
    assert len(q._INT8_WS) == before and made[0]() is None


@pytest.mark.parametrize("layers", [1, 2])
def test_a_scratch_that_is_too_small_is_refused(layers):
    """One byte less than the launch needs: nothing is launched (the addresses are never used)."""
    from lit_llama import _native as N

    M, Nout, K = 300, 11008 if layers == 2 else 1024, 4096 if layers == 2 else 11008
    need = N.call_ret("ll_int4_rows_scratch_bytes", M, Nout, K, layers, 0, 0, 0)
    assert need > 0
    entry, pointers = ("ll_int4_rows_gated_sized", 11) if layers == 2 else ("ll_int4_rows_sized", 7)
    with pytest.raises(RuntimeError, match=f"scratch of {need - 1} bytes"):
        N.call(entry, *([1 << 20] * pointers), need - 1, M, Nout, K, 128, 0, 0, 0, None)
