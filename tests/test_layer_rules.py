"""Which rows and sizes a layer takes in one call, on the host."""
import pytest
import torch


@pytest.fixture
def native(monkeypatch):
    from lit_llama import _native as N

    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: N.capturing)
    monkeypatch.setattr(N, "capturing", False, raising=False)
    monkeypatch.setattr(N, "_ready_library", lambda: None)
    return N


def test_rows_of_a_layer_in_one_call(native, monkeypatch):
    """Rows times weights and the weights themselves bound it; a capture keeps a few rows of a layer that is not large, and no more."""
    N, most, largest = native, 6 << 30, 1 << 26
    assert N.layer_rows(17, 1 << 25, most, largest) and N.layer_rows(96, 1 << 26, most, largest)
    assert not N.layer_rows(97, 1 << 26, most, largest) and not N.layer_rows(3, (1 << 26) + 1, most, largest)
    assert N.layer_rows(8, 1 << 25, 0, 0) and not N.layer_rows(8, (1 << 25) + 1, most, N.LARGE_WEIGHTS)
    monkeypatch.setattr(N, "capturing", True)
    assert N.layer_rows(8, 1 << 25, most, largest) and not N.layer_rows(9, 1 << 10, most, largest)


@pytest.mark.parametrize("B,T,S,end,v,width,want", [(3, 1, 100, None, 64, 1024, 0), (16, 1, 100, None, 64, 2048, 0), (17, 1, 100, None, 64, 2048, None), (4, 1, 100, 5, 64, 8192, None),
                                                    (1, 20, 100, 20, 64, 1024, 20), (2, 20, 100, 20, 64, 1024, None), (2, 20, 20, 20, 64, 1024, 20),
                                                    (2, 20, 50, None, 64, 1024, 50), (1, 20, 100, 60, 40, 1024, None), (1, 20, 3000, 2900, 64, 1024, 0)])
def test_form_of_a_latent_layer_in_one_call(native, B, T, S, end, v, width, want):
    """Expanded rows where the separate calls would expand all rows from the first on; else queries in latent space, while their heads are few and the
    weights not large."""
    from lit_llama.latent_attention import LatentAttention, LatentAttentionSpec

    with torch.device("meta"):
        m = LatentAttention(LatentAttentionSpec(width=width, heads=width // 128, nope_dim=64, rot_dim=32, v_dim=v, kv_rank=256, window=None, scale=0.1), torch.bfloat16, "meta")
    cache = torch.zeros((B, S, m.spec.row), dtype=torch.bfloat16)
    assert m._layer_form(B, T, cache, 1, end) == want


def test_rows_from_which_experts_take_the_tensor_cores():
    from lit_llama.moe import tc_least_rows

    assert tc_least_rows(2048 * 1024, 32, False) == 0 == tc_least_rows(1024 * 768, 256, False) == tc_least_rows(512 * 256, 128, True)
    assert tc_least_rows(1024 * 512, 32, False) == 16 and tc_least_rows(64 * 24, 8, False) == 0
    assert tc_least_rows(256 * 256, 128, True) == 48 == tc_least_rows(256 * 64, 256, False)
