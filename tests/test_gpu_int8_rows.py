"""llm.int8 prompts (M > 64, one product on the tensor cores) against the passes of 64 rows that the same call makes with a workspace for 64
rows: the same integer sums and roundings, so the same numbers."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(65, 64, 128), (127, 130, 256), (128, 128, 128), (129, 257, 384), (200, 1000, 512), (1023, 96, 256), (1025, 33, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("outliers,bias,transposed", [(0, False, True), (5, True, True), (40, True, False)])
def test_rows_against_passes(M, N, K, dtype, outliers, bias, transposed):
    from lit_llama import _native as NV

    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    x = torch.randn((M, K), generator=g, device="cuda")
    cols = torch.randperm(K, generator=g, device="cuda")[:outliers]
    rows = torch.rand(M, generator=g, device="cuda") < 0.3            # a feature stands out in some blocks of 64 rows and not in others
    rows[64:] &= torch.arange(64, M, device="cuda") < 2 * M // 3
    x[:, cols] = torch.where(rows[:, None], x[:, cols] * 30.0, x[:, cols])
    x[M // 2] = 0.0                                                    # a row without a scale
    x = x.to(dtype)
    w = (torch.randn((N, K), generator=g, device="cuda") * 0.05).to(dtype)
    cb, scb = torch.empty((N, K), dtype=torch.int8, device="cuda"), torch.empty(N, device="cuda")
    NV.call("ll_int8_quantize_weight", NV.ptr(w), NV.dtype_code(dtype), NV.ptr(cb), NV.ptr(scb), N, K, NV.stream())
    cbt = cb.t().contiguous() if transposed else None
    b = torch.randn(N, generator=g, device="cuda").to(dtype) if bias else None
    outs = []
    for m in (M, 64):
        ws = torch.full((NV.call_ret("ll_int8_workspace_bytes", m, N, K),), 0x5A, dtype=torch.uint8, device="cuda")
        y = torch.empty((M, N), dtype=dtype, device="cuda")
        NV.call("ll_int8_linear", NV.ptr(x), NV.dtype_code(dtype), NV.ptr(cb), NV.ptr(cbt), NV.ptr(scb), NV.ptr(b), NV.ptr(y), M, N, K, 6.0, NV.ptr(ws),
                ws.numel(), NV.stream())
        outs.append(y)
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int8_tc_error") == 0
    # up to 64 outliers a block are summed in the same order on both sides
    assert torch.equal(outs[0], outs[1])


@pytest.mark.parametrize("M", [1, 15, 16, 17, 32, 33, 48, 49, 64])
@pytest.mark.parametrize("N,K", [(33, 128), (128, 384), (1000, 1024), (256, 4096 * 10)])
@pytest.mark.parametrize("offset", [0, 1])
def test_small_batches_against_64_bits(M, N, K, offset):
    """Up to 64 rows: every padded row count, a last column tile that is not full, one and many ranges of k, a K whose preparation does not
    fit a resident grid, activations off 16-byte boundaries."""
    from lit_llama import _native as NV

    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.empty(M * K + 8, dtype=torch.float16, device="cuda")[offset: offset + M * K].view(M, K)
    x.copy_(torch.randn((M, K), generator=g, device="cuda"))
    x[:, 5::97] *= 9.0
    cb = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    scb = torch.rand(N, generator=g, device="cuda") + 0.5
    ws = torch.full((NV.call_ret("ll_int8_workspace_bytes", M, N, K),), 0x5A, dtype=torch.uint8, device="cuda")
    y = torch.empty((M, N), dtype=torch.float32, device="cuda")
    xf = x.float()
    ya, yf = torch.empty((M, N), dtype=torch.float16, device="cuda"), y
    NV.call("ll_int8_linear", NV.ptr(x), NV.LL_F16, NV.ptr(cb), None, NV.ptr(scb), None, NV.ptr(ya), M, N, K, 6.0, NV.ptr(ws), ws.numel(), NV.stream())
    NV.call("ll_int8_linear", NV.ptr(xf), NV.LL_F32, NV.ptr(cb), None, NV.ptr(scb), None, NV.ptr(yf), M, N, K, 6.0, NV.ptr(ws), ws.numel(), NV.stream())
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int8_tc_error") == 0
    assert torch.equal(ya.float(), yf)                                 # x.half() either way
    a = x.double()
    big = a.abs() >= 6.0
    cols = big.any(0)
    rest = a.masked_fill(big, 0.0)
    sca = rest.abs().amax(1)
    # (a tensor over a tensor: a number over a tensor is a product with its reciprocal, which may end on another code)
    ca = torch.round((rest.float() * (torch.full_like(sca, 127.0).float() / sca.float())[:, None]).double()).masked_fill(cols[None], 0.0)
    want = (ca @ cb.double().t()) * sca[:, None] * scb.double()[None] / 127.0 ** 2
    wo = (cb.double()[:, cols] * scb.double()[:, None] / 127.0).half().double()
    odd, size = a[:, cols] @ wo.t(), a[:, cols].abs() @ wo.abs().t()
    # both parts and their sum rounded to fp16 (2^-11 of each); an outlier's weight may round to the other fp16 neighbour, where its fp32
    # product (one rounding of SCB / 127, one of the product) sits on the other side of the middle: 2^-10 of the term
    assert ((yf.double() - want - odd).abs() <= 2.0 ** -11 * (want.abs() + odd.abs() + (want + odd).abs()) * 1.01 + 2.0 ** -10 * size + 1e-4).all()


def test_more_outliers_than_one_stage():
    from lit_llama.quantization import Linear8bitLt

    g = torch.Generator(device="cuda").manual_seed(3)
    M, N, K = 150, 200, 1024
    lin = Linear8bitLt(K, N, bias=False, device="cuda", dtype=torch.float32)
    lin.load_state_dict({"weight": torch.randn((N, K), generator=g, device="cuda") * 0.05})
    x = torch.randn((M, K), generator=g, device="cuda") * 0.5
    x[:, ::3] = torch.sign(x[:, ::3]) * (7.0 + x[:, ::3].abs())        # 342 outlier features: several stages of the finishing kernel
    y = lin(x).double()
    a, cb, scb = x.half().double(), lin.weight.CB.double(), lin.weight.SCB.double()
    cols = torch.zeros(K, dtype=torch.bool, device="cuda")
    cols[::3] = True
    rest = a.masked_fill(cols[None], 0.0)
    sca = rest.abs().amax(1)
    ca = torch.round((rest.float() * (torch.full_like(sca, 127.0).float() / sca.float())[:, None]).double())
    want = (ca @ cb.t()) * sca[:, None] * scb[None] / 127.0 ** 2 + a[:, cols] @ (cb[:, cols] * scb[:, None] / 127.0).half().double().t()
    # fp16 roundings of the two parts and of their sum (2^-11 each of the largest value)
    assert (y - want).abs().max() <= 4 * 2.0 ** -11 * want.abs().max()


def test_small_batches_on_many_streams():
    """A call's kernels wait for no block that may not be running: rows of 35840 features on twelve streams at once, more blocks than the
    device holds together, give what one stream after the other gives."""
    from lit_llama import _native as NV

    g = torch.Generator(device="cuda").manual_seed(11)
    M, N, K, S = 5, 40, 35840, 12
    x = torch.randn((S, M, K), generator=g, device="cuda").to(torch.bfloat16)
    x[:, 1::2, 7::501] *= 20.0                                         # outliers in some rows
    cb = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    scb = torch.rand(N, generator=g, device="cuda") + 0.5
    need = NV.call_ret("ll_int8_workspace_bytes", M, N, K)
    ws = torch.full((S, (need + 255) // 256 * 256), 0x5A, dtype=torch.uint8, device="cuda")
    outs = []
    for streams in ([torch.cuda.Stream() for _ in range(S)], [torch.cuda.current_stream()] * S):
        y = torch.zeros((S, M, N), dtype=torch.bfloat16, device="cuda")
        torch.cuda.synchronize()
        for _ in range(5):
            for i, st in enumerate(streams):
                NV.call("ll_int8_linear", NV.ptr(x[i]), NV.LL_BF16, NV.ptr(cb), None, NV.ptr(scb), None, NV.ptr(y[i]), M, N, K, 6.0, NV.ptr(ws[i]),
                        ws.shape[1], st.cuda_stream)
        torch.cuda.synchronize()
        outs.append(y)
    assert NV.call_ret("ll_int8_tc_error") == 0
    assert torch.equal(outs[0], outs[1]) and bool(outs[0].any())


@pytest.mark.parametrize("M", [1, 16, 33, 64, 70])
@pytest.mark.parametrize("outliers", [1, 32, 64, 65, 96, 128, 129, 300])
@pytest.mark.parametrize("N,transposed", [(70, True), (64, False)])
def test_long_outlier_lists(M, outliers, N, transposed):
    """Lists that end inside a share, at its end, inside a stage and after several stages."""
    from lit_llama import _native as NV

    g = torch.Generator(device="cuda").manual_seed(M + outliers)
    K = 384
    cols = torch.randperm(K, generator=g, device="cuda")[:outliers]
    x = torch.randn((M, K), generator=g, device="cuda").clamp(-4, 4)
    x[:, cols] = torch.sign(x[:, cols]) * (6.0 + 3.0 * x[:, cols].abs())
    x = x.half()
    cb = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    cbt = cb.t().contiguous() if transposed else None
    scb = torch.rand(N, generator=g, device="cuda") + 0.5
    ws = torch.full((NV.call_ret("ll_int8_workspace_bytes", M, N, K),), 0x5A, dtype=torch.uint8, device="cuda")
    y = torch.empty((M, N), dtype=torch.float32, device="cuda")
    xf = x.float()
    NV.call("ll_int8_linear", NV.ptr(xf), NV.LL_F32, NV.ptr(cb), NV.ptr(cbt), NV.ptr(scb), None, NV.ptr(y), M, N, K, 6.0, NV.ptr(ws),
            ws.numel(), NV.stream())
    torch.cuda.synchronize()
    a, out = x.double(), torch.zeros(K, dtype=torch.bool, device="cuda")
    out[cols] = True
    rest = a.masked_fill(out[None], 0.0)
    sca = rest.abs().amax(1)
    ca = torch.round((rest.float() * (torch.full_like(sca, 127.0).float() / sca.clamp_min(1e-30).float())[:, None]).double())
    want = (ca @ cb.double().t()) * sca[:, None] * scb.double()[None] / 127.0 ** 2
    wo = (cb.double()[:, out] * scb.double()[:, None] / 127.0).half().double()
    odd, size = a[:, out] @ wo.t(), a[:, out].abs() @ wo.abs().t()
    # as above: both parts and their sum rounded to fp16, an outlier's weight possibly on its other fp16 neighbour
    assert ((y.double() - want - odd).abs() <= 2.0 ** -11 * (want.abs() + odd.abs() + (want + odd).abs()) * 1.01 + 2.0 ** -10 * size + 1e-4).all()


def test_a_wait_that_ran_out_fails_the_next_launch():
    from lit_llama import _native as NV

    x = torch.ones(64, device="cuda")
    y = torch.empty_like(x)
    args = (NV.ptr(x), NV.ptr(x), NV.ptr(y), NV.LL_F32, 64, NV.stream())
    w = torch.zeros((128, 128), dtype=torch.int8, device="cuda")       # (a launch that shares the word with its kernel)
    ws = torch.empty(NV.call_ret("ll_int8_workspace_bytes", 1, 128, 128), dtype=torch.uint8, device="cuda")
    a, o, s = torch.zeros((1, 128), device="cuda"), torch.empty((1, 128), device="cuda"), torch.ones(128, device="cuda")
    NV.call("ll_int8_linear", NV.ptr(a), NV.LL_F32, NV.ptr(w), None, NV.ptr(s), None, NV.ptr(o), 1, 128, 128, 6.0, NV.ptr(ws), ws.numel(), NV.stream())
    NV.call("ll_add", *args)
    NV.call_ret("ll_wait_report", 203)                                 # as a kernel leaves it
    with pytest.raises(RuntimeError, match="int4 rows, code 203"):
        NV.call("ll_add", *args)
    NV.call("ll_add", *args)
    torch.cuda.synchronize()
    assert bool((y == 2).all())


def test_a_captured_call_keeps_its_workspace():
    """A step captured with a small workspace is replayed after a longer prompt on its stream needed a larger one: it still writes to its own."""
    from lit_llama.quantization import Linear8bitLt

    g = torch.Generator(device="cuda").manual_seed(5)
    K, Nout, st = 1024, 2048, torch.cuda.Stream()
    lin = Linear8bitLt(K, Nout, bias=False, device="cuda", dtype=torch.float32)
    lin.load_state_dict({"weight": torch.randn((Nout, K), generator=g, device="cuda") * 0.05})
    x, long = torch.randn((8, K), generator=g, device="cuda"), torch.randn((900, K), generator=g, device="cuda")
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(st):
        want = lin(x)
        st.synchronize()
        with torch.cuda.graph(graph, stream=st):
            y = lin(x)
        lin(long)
        st.synchronize()
        others = [torch.full((n,), 0x33, dtype=torch.uint8, device="cuda") for n in (1 << 17, 1 << 18, 1 << 19, 1 << 20, 1 << 21, 3 << 20) for _ in range(8)]
        for _ in range(3):
            graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)
    assert all(bool((o == 0x33).all()) for o in others)


@pytest.mark.parametrize("M,N", [(65, 70), (200, 64), (385, 300), (640, 260), (2100, 5000)])
@pytest.mark.parametrize("transposed", [True, False])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_prompts_with_long_and_short_lists(M, N, transposed, dtype):
    """Every block of 64 rows has a list of its own length: none, what the finishing warps add themselves, one more, several stages, half of all
    features; few tiles (one a CTA) and more than the CTAs that take them one by one.  Against 64 bits, and both gated layers against each alone."""
    from lit_llama import _native as NV

    K = 384
    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn((M, K), generator=g, device="cuda").clamp(-4, 4)
    lists = [0, 5, 16, 17, 28, 29, 32, 33, 64, 65, 190]
    for b in range((M + 63) // 64):
        cols = torch.randperm(K, generator=g, device="cuda")[: lists[(7 * b + M) % len(lists)]]
        rows = slice(64 * b, min(64 * b + 64, M))
        x[rows, cols] = torch.sign(x[rows, cols]) * (6.5 + 3.0 * x[rows, cols].abs())
    x = x.to(dtype).half().to(dtype)
    layers = []
    for i in range(2):
        cb = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
        layers.append((cb, cb.t().contiguous() if transposed else None, (torch.rand(N, generator=g, device="cuda") + 0.5) * 0.05,
                       torch.randn(N, generator=g, device="cuda").to(torch.bfloat16).to(dtype)))      # (a number of every dtype)
    ws = torch.full((NV.call_ret("ll_int8_gated_workspace_bytes", M, N, K),), 0x5A, dtype=torch.uint8, device="cuda")
    outs = []
    for cb, cbt, scb, bias in layers:
        y = torch.empty((M, N), dtype=dtype, device="cuda")
        NV.call("ll_int8_linear", NV.ptr(x), NV.dtype_code(dtype), NV.ptr(cb), NV.ptr(cbt), NV.ptr(scb), NV.ptr(bias), NV.ptr(y), M, N, K, 6.0, NV.ptr(ws),
                ws.numel(), NV.stream())
        outs.append(y)
    if dtype == torch.bfloat16:
        h, want_h = torch.empty_like(outs[0]), torch.empty_like(outs[0])
        ws.fill_(0x5A)
        NV.call("ll_int8_gated", NV.ptr(x), *(NV.ptr(t) for layer in layers for t in layer), NV.ptr(h), M, N, K, 6.0, NV.ptr(ws), ws.numel(), NV.stream())
        NV.call("ll_silu_mul", NV.ptr(outs[0]), NV.ptr(outs[1]), NV.ptr(want_h), NV.LL_BF16, M * N, NV.stream())
        # (silu comes from a fast exponential and division: now and then on the other bf16 neighbour, a rounding each of it and of the product)
        assert ((h.double() - want_h.double()).abs() <= want_h.double().abs() * 2.0 ** -7).all() and (h == want_h).float().mean() >= 0.99
    for y, (cb, cbt, scb, bias) in zip(outs, layers):
        for b in range((M + 63) // 64):
            rows = slice(64 * b, min(64 * b + 64, M))
            a = x[rows].double()
            out = (a.abs() >= 6.0).any(0)
            rest = a.masked_fill(out[None], 0.0)
            sca = rest.abs().amax(1)
            ca = torch.round((rest.float() * (torch.full_like(sca, 127.0).float() / sca.float())[:, None]).double())
            want = (ca @ cb.double().t()) * sca[:, None] * scb.double()[None] / 127.0 ** 2 + bias.double()[None]
            wo = (cb.double()[:, out] * scb.double()[:, None] / 127.0).half().double()
            odd, size = a[:, out] @ wo.t(), a[:, out].abs() @ wo.abs().t()
            # both parts and their sum rounded to fp16, an outlier's weight possibly on its other fp16 neighbour, the result to the dtype (bf16:
            # eight significant bits, half a unit in the last place is up to 2^-8 of the number)
            bound = 2.0 ** -11 * (want.abs() + odd.abs() + (want + odd).abs()) * 1.01 + 2.0 ** -10 * size + 1e-4
            bound = bound + ((want + odd).abs() * 2.0 ** -8 * 1.01 if dtype == torch.bfloat16 else 0.0)
            assert ((y[rows].double() - want - odd).abs() <= bound).all()
    assert NV.call_ret("ll_int8_tc_error") == 0


@pytest.mark.parametrize("M,N,K", [(2, 64, 128), (7, 64, 256), (8, 33, 16384), (8, 33, 16512), (9, 64, 8192), (9, 64, 8320), (24, 64, 1152), (40, 64, 256),
                                   (63, 130, 512), (64, 64, 2048), (64, 64, 2176)])
def test_rows_of_a_cluster(M, N, K):
    """Few rows are prepared by a cluster of eight CTAs: every number of rows a CTA can have, and both sides of the line to a CTA per row."""
    test_small_batches_against_64_bits(M, N, K, 0)


@pytest.mark.parametrize("M", [5, 12, 64, 130])
def test_columns_that_stand_out_once(M):
    """Column 97 m stands out in row m alone; infinities stand out, NaN does not and counts as nothing; the rows around keep their own scales."""
    from lit_llama import _native as NV

    N, K = 16, 16384
    g = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn((M, K), generator=g, device="cuda").clamp(-4, 4).half()
    r = torch.arange(M, device="cuda")
    x[r, 97 * r] = 8.0
    x[M - 1, 5] = float("nan")
    cb = torch.randint(-127, 128, (N, K), generator=g, device="cuda", dtype=torch.int8)
    scb = torch.rand(N, generator=g, device="cuda") + 0.5
    ys = []
    for v in (x, torch.where(x.isnan(), torch.zeros_like(x), x)):
        ws = torch.full((NV.call_ret("ll_int8_workspace_bytes", M, N, K),), 0x5A, dtype=torch.uint8, device="cuda")
        y = torch.empty((M, N), dtype=torch.float16, device="cuda")
        NV.call("ll_int8_linear", NV.ptr(v), NV.LL_F16, NV.ptr(cb), None, NV.ptr(scb), None, NV.ptr(y), M, N, K, 6.0, NV.ptr(ws), ws.numel(), NV.stream())
        ys.append(y)
    torch.cuda.synchronize()
    assert NV.call_ret("ll_int8_tc_error") == 0
    assert torch.equal(ys[0], ys[1])
    a = torch.where(x.isnan(), torch.zeros_like(x), x).double()
    for b0 in range(0, M, 64):                                 # a column is taken out for a block of 64 rows
        v = a[b0:b0 + 64]
        big = v >= 6.0
        cols, sca = big.any(0), v.masked_fill(big, 0.0).abs().amax(1)
        ca = torch.round(v.masked_fill(big, 0.0).float() * (torch.full_like(sca, 127.0).float() / sca.float())[:, None]).double().masked_fill(cols[None], 0.0)
        wo = (cb.double()[:, cols] * scb.double()[:, None] / 127.0).half().double()
        main, odd, size = (ca @ cb.double().t()) * sca[:, None] * scb.double()[None] / 127.0 ** 2, v[:, cols] @ wo.t(), v[:, cols].abs() @ wo.abs().t()
        # both parts and their sum rounded to fp16 (2^-11 of each); an outlier's weight may round to the other fp16 neighbour (2^-10 of the term)
        err = (ys[0][b0:b0 + 64].double() - (main + odd)).abs()
        assert (err <= 2.0 ** -11 * (main.abs() + odd.abs() + (main + odd).abs()) + 2.0 ** -10 * size + 1e-6).all()
