"""The wide rounds of the matrix memory's gates at their edges (the same numbers as in rounds of 256 tokens), and the read-out norm of parts that stay
in registers (up to 256 numbers) beside the first that does not, against 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gates(raw, bias, cap, state, pos, T, H):
    from lit_llama import _native as N

    out = [torch.empty((2, T, H), device="cuda") for _ in range(3)]
    N.call("ll_matrix_memory_gates", N.ptr(raw), N.ptr_at(raw, H), N.dtype_code(raw.dtype), 2 * H, N.ptr(bias[0]), N.ptr(bias[1]), cap, N.ptr(state),
           N.ptr(pos), *[N.ptr(o) for o in out], 2, T, H, N.stream())
    return out


@pytest.mark.parametrize("T", [257, 1023, 1024, 1025, 2081])
@pytest.mark.parametrize("dtype,cap", [(torch.bfloat16, 15.0), (torch.float32, 0.0)])
def test_gates_in_wide_rounds(T, dtype, cap):
    H = 3
    g = torch.Generator(device="cuda").manual_seed(T)
    raw = (4 * torch.randn((2, T, 2 * H), generator=g, device="cuda")).to(dtype)
    bias = torch.randn((2, H), generator=g, device="cuda")
    whole, parts = torch.randn((2, H), generator=g, device="cuda"), None
    parts = whole.clone()
    pos = torch.arange(5, 5 + T, dtype=torch.int32, device="cuda")
    got = _gates(raw.contiguous(), bias, cap, whole, pos, T, H)
    for t in range(0, T, 256):                         # narrow rounds, the stabiliser carried by the state: whole warps of tokens in the same order
        n = min(256, T - t)
        want = _gates(raw[:, t:t + n].contiguous(), bias, cap, parts, pos[t:t + n].contiguous(), n, H)
        for a, b in zip(got, want):
            assert torch.equal(a[:, t:t + n], b)
    assert torch.equal(whole, parts)


@pytest.mark.parametrize("size", [1, 31, 33, 255, 256, 257])
@pytest.mark.parametrize("gate_first,sigmoid,shared,unit", [(False, True, False, True), (True, False, True, False), (False, False, True, True)])
def test_read_out_norm(size, gate_first, sigmoid, shared, unit):
    from lit_llama.recurrence import gated_group_norm

    rows, groups, part = 5, 9, size + 1                # parts start on odd addresses
    g = torch.Generator(device="cuda").manual_seed(size)
    y = torch.randn((rows, groups * part), generator=g, device="cuda")
    gate = torch.randn((rows, groups * size + 1), generator=g, device="cuda")
    w = torch.randn(size if shared else groups * size, generator=g, device="cuda")
    stab = torch.randn((rows, groups), generator=g, device="cuda") if unit else None
    got = gated_group_norm(y, gate, 1, w, shared, 1e-5, groups, gate_first, torch.float32, sigmoid=sigmoid, part=size, stab=stab)
    yd, z = y.double().view(rows, groups, part), gate[:, 1:].double().reshape(rows, groups, size)
    v = yd[..., :size]
    if unit:
        v = v / (torch.maximum(yd[..., size].abs(), (-stab.double()).exp()) + 1e-6)[..., None]
    s = torch.sigmoid(z) * (1.0 if sigmoid else z)
    t = v * s if gate_first else v
    k = (t.square().mean(-1, keepdim=True) + 1e-5).rsqrt()
    want = t * k * (w.double() if shared else w.double().view(groups, size)) * (1.0 if gate_first else s)
    # a lane's nine terms, five shuffles, and some thirty roundings of the divider, the gate, the root and the products
    assert ((got.double().view_as(want) - want).abs() <= 48 * 2.0 ** -24 * want.abs() + 1e-30).all()
