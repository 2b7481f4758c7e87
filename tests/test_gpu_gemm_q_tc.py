"""GPU: the tcgen05 kernel that dequantises Q4_0 / Q8_0 weights on their way to the tensor cores, at the
edges of its tiles: every accumulator layout (16, 32, 64, 128 and 256 columns, several column tiles),
row counts around the 128-row tile, one group of K and uneven splits of K, unaligned activations.

Bar against a 64-bit dequantise-and-dot: a dequantised weight is rounded to fp16 once (relative error at
most 2^-11, 2^-11 / sqrt(3) rms, independent between products, so the same relative to the result) and an
fp16 result once more: sqrt(2) * 2^-11 / sqrt(3) = 4.0e-4, and 2.82e-4 without the second; the margin
of a tenth is for small samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUND = 2.0 ** -11 / np.sqrt(3.0)


def data(oracle, fmt, M, N, K):
    rng = np.random.default_rng(M * 31 + N * 7 + K + fmt)
    W = (rng.standard_normal((N, K)) * 0.02).astype(np.float32).astype(np.float16)
    X = rng.standard_normal((M, K)).astype(np.float16)
    return X, oracle.quantize_weights(W, fmt)


@pytest.mark.parametrize("fmt,M,N,K", [
    (0, 5, 128, 256), (0, 16, 129, 512), (0, 17, 127, 768), (0, 32, 1000, 2304), (0, 33, 260, 1024), (0, 48, 128, 1280),
    (0, 64, 640, 2816), (0, 65, 130, 512), (0, 128, 257, 1536), (0, 129, 384, 768), (0, 256, 128, 2048),
    (0, 257, 200, 512), (0, 300, 19000, 256), (0, 520, 136, 1024),
    (1, 13, 128, 256), (1, 16, 1000, 4096), (1, 32, 129, 768), (1, 64, 260, 2560), (1, 80, 127, 1024),
    (1, 128, 512, 1536), (1, 200, 130, 512), (1, 256, 300, 2304), (1, 513, 128, 768)])
def test_tile_edges_against_64_bit(tc, ctx, oracle, fmt, M, N, K):
    X, Wq = data(oracle, fmt, M, N, K)
    want = oracle.dequant_dot_f64(X.astype(np.float64), Wq, fmt, N)
    with ctx.buffer_from_array(X) as bx, ctx.buffer_from_array(Wq) as bw, ctx.buffer(M * N * 4) as by:
        ctx.gemv_quantized(bx, bw, by, fmt, M, N, K)
        assert "tcgen05" in tc.cuda_last_kernel_name()
        got = by.to_numpy((M, N), np.float16).astype(np.float64)
        assert oracle.scaled_rms(got, want) <= 1.1 * np.sqrt(2.0) * ROUND
        if fmt == 0:                                          # fp32 results
            tc.gemv_quantized_ex(ctx, bx, bw, by, fmt, M, N, K, "f16", "f32", None)
            got32 = by.to_numpy((M, N), np.float32).astype(np.float64)
            assert oracle.scaled_rms(got32, want) <= 1.1 * ROUND
            assert np.array_equal(got32.astype(np.float32).astype(np.float16), got.astype(np.float16))
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("fmt,M", [(0, 8), (0, 40), (1, 20)])
def test_activations_at_any_even_address(tc, ctx, oracle, fmt, M):
    """Rows that start 2, 8 or 14 bytes past a 16-byte boundary give the same bits as aligned ones."""
    N, K = 300, 1024
    X, Wq = data(oracle, fmt, M, N, K)
    outs = []
    for off in (0, 2, 8, 14):
        with ctx.buffer(X.nbytes + 16) as bx, ctx.buffer_from_array(Wq) as bw, ctx.buffer(M * N * 2) as by:
            bx.upload(X, off)
            tc.raw_gemv_quantized(ctx, bx.device_ptr() + off, bw.device_ptr(), by.device_ptr(), fmt, M, N, K)
            import torch
            torch.cuda.synchronize()
            assert "tcgen05" in tc.cuda_last_kernel_name()
            outs.append(by.to_numpy((M, N), np.float16))
    assert all(np.array_equal(outs[0], o) for o in outs[1:])


def test_non_finite_weights_scales_and_activations(tc, ctx, oracle):
    """An infinite activation makes the results of its row non-finite, an infinite scale those of its
    weight row; nothing else changes."""
    M, N, K = 16, 256, 512
    X, Wq = data(oracle, 0, M, N, K)
    with ctx.buffer(M * K * 2) as bx, ctx.buffer(Wq.nbytes) as bw, ctx.buffer(M * N * 2) as by:
        def call(x, w):
            bx.upload(x)
            bw.upload(w)
            ctx.gemv_quantized(bx, bw, by, 0, M, N, K)
            return by.to_numpy((M, N), np.float16)
        base = call(X, Wq)
        X2 = X.copy()
        X2[3, 77] = np.inf
        got = call(X2, Wq)
        assert not np.isfinite(got[3]).any()
        keep = np.arange(M) != 3
        assert np.array_equal(got[keep], base[keep])
        W2 = Wq.copy().reshape(N, K // 32, 18)
        W2[5, 2, :2] = np.array([np.inf], np.float16).view(np.uint8)
        got = call(X, W2.reshape(Wq.shape))
        assert not np.isfinite(got[:, 5]).any()
        keep = np.arange(N) != 5
        assert np.array_equal(got[:, keep], base[:, keep])


@pytest.mark.parametrize("fmt,M", [(0, 5), (0, 33), (1, 16), (0, 130)])
def test_products_that_share_their_activations_run_as_one_launch(tc, ctx, oracle, fmt, M):
    """q, k and v of a layer (different row counts), recorded with the norm fused: one pass over the rows and
    one product launch a submission, whether launched directly or replayed from a graph."""
    K, Ns = 512, (384, 130, 127)
    X, _ = data(oracle, fmt, M, 64, K)
    g = (1 + 0.1 * np.random.default_rng(3).standard_normal(K)).astype(np.float16)
    ws = [data(oracle, fmt, M + i, n, K)[1] for i, n in enumerate(Ns)]
    want = [oracle.fused_rmsnorm_gemv_quantized_f32(X.astype(np.float32), g.astype(np.float32), w, fmt, n) for w, n in zip(ws, Ns)]
    bx, bg = ctx.buffer_from_array(X), ctx.buffer_from_array(g)
    bw, by = [ctx.buffer_from_array(w) for w in ws], [ctx.buffer(M * n * 2) for n in Ns]
    s = ctx.stream()
    for _ in range(4):
        before = tc.launch_count()
        for w, y, n in zip(bw, by, Ns):
            tc.fused_rmsnorm_gemv_quantized_ex(ctx, bx, bg, w, y, fmt, M, n, K, 1e-5, "f16", "f16", s)
        s.sync()
        assert tc.launch_count() - before == 2
        for y, n, v in zip(by, Ns, want):
            # three roundings to fp16: weights, normalised rows, result
            assert oracle.scaled_rms(y.to_numpy((M, n), np.float16), v) <= 1.1 * np.sqrt(3.0) * ROUND
    s.close()
    for b in [bx, bg] + bw + by:
        b.close()


def test_dependent_products_do_not_share_a_launch(tc, ctx, oracle):
    """A recorded product that writes what a neighbour reads or writes keeps its place: the second product
    overwrites the activations of both, the third overwrites the first one's result."""
    M, K = 8, 512
    X, w1 = data(oracle, 0, M, K, K)
    _, w2 = data(oracle, 0, M + 1, K, K)
    bx, b1, b2, by = ctx.buffer_from_array(X), ctx.buffer_from_array(w1), ctx.buffer_from_array(w2), ctx.buffer(M * K * 2)
    s = ctx.stream()
    ctx.gemv_quantized_async(bx, b1, by, 0, M, K, K, s)      # y = W1 x
    ctx.gemv_quantized_async(bx, b2, bx, 0, M, K, K, s)      # x is overwritten after that (its value is not looked at: in place)
    s.sync()
    y1 = by.to_numpy((M, K), np.float16)
    assert oracle.scaled_rms(y1.astype(np.float64), oracle.dequant_dot_f64(X.astype(np.float64), w1, 0, K)) <= 5e-4
    bx.upload(X)
    ctx.gemv_quantized_async(bx, b1, by, 0, M, K, K, s)
    ctx.gemv_quantized_async(bx, b2, by, 0, M, K, K, s)      # the same result buffer: the later product's values stay
    s.sync()
    y2 = by.to_numpy((M, K), np.float16)
    assert oracle.scaled_rms(y2.astype(np.float64), oracle.dequant_dot_f64(X.astype(np.float64), w2, 0, K)) <= 5e-4
    s.close()
    for b in (bx, b1, b2, by):
        b.close()


def test_captured_call_outlives_a_larger_one(tc, ctx, oracle):
    """A fused call captured in a CUDA graph with more rows than the stream's room for normalised rows holds goes
    through it in slabs, and the graph stays valid when a later, larger call makes a bigger room."""
    import torch
    N, K, M, big = 256, 4096, 300, 700
    X, Wq = data(oracle, 0, big, N, K)
    g = (1 + 0.1 * np.random.default_rng(5).standard_normal(K)).astype(np.float16)
    want = oracle.fused_rmsnorm_gemv_quantized_f32(X[:M].astype(np.float32), g.astype(np.float32), Wq, 0, N)
    x, w, gam = (torch.from_numpy(t.view(np.uint8) if t.dtype == np.uint8 else t).cuda() for t in (X, Wq, g))
    y, y2 = torch.zeros(M, N, dtype=torch.float16, device="cuda"), torch.zeros(big, N, dtype=torch.float16, device="cuda")
    st = torch.cuda.Stream()

    def call(m, out):
        tc.raw_fused_rmsnorm_gemv_quantized(ctx, x.data_ptr(), gam.data_ptr(), w.data_ptr(), out.data_ptr(), "q4_0", m, N, K,
                                            1e-5, "f16", "f16", st.cuda_stream)
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        call(8, y2)                                   # the first room: 1 MB, 127 rows
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=st):
            call(M, y)
        call(big, y2)                                 # a larger room
        torch.cuda.synchronize()
        y.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert oracle.scaled_rms(y.cpu().numpy(), want) <= 1.1 * np.sqrt(3.0) * ROUND
    assert tc.take_device_error(ctx) == 0
    del graph


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("w_off,M,K", [(2, 128, 1024), (8, 128, 1024), (2, 16, 1024), (8, 512, 512)])
def test_prefill_block_with_weights_at_any_even_address(tc, ctx, oracle, fmt, w_off, M, K):
    """Weights that no tiled copy can describe although K is a multiple of 256: prefill-sized calls dequantise them once
    and multiply them as a GEMM - two launches, three with the norm -, smaller ones stream them."""
    import torch
    N = 130
    X, Wq = data(oracle, fmt, M, N, K)
    g = (1 + 0.1 * np.random.default_rng(8).standard_normal(K)).astype(np.float16)
    want = oracle.dequant_dot_f64(X.astype(np.float64), Wq, fmt, N)
    x64 = X.astype(np.float64)
    wantf = oracle.dequant_dot_f64(x64 / np.sqrt((x64 * x64).mean(axis=1, keepdims=True) + 1e-5) * g, Wq, fmt, N)
    once = M >= (96 if fmt == 0 else 13)
    with ctx.buffer_from_array(X) as bx, ctx.buffer_from_array(g) as bg, ctx.buffer(Wq.nbytes + 16) as bw, ctx.buffer(M * N * 2) as by:
        bw.upload(Wq, w_off)
        for fused in (False, True):
            before = tc.launch_count()
            if fused:
                tc.raw_fused_rmsnorm_gemv_quantized(ctx, bx.device_ptr(), bg.device_ptr(), bw.device_ptr() + w_off, by.device_ptr(),
                                                    fmt, M, N, K, 1e-5)
            else:
                tc.raw_gemv_quantized(ctx, bx.device_ptr(), bw.device_ptr() + w_off, by.device_ptr(), fmt, M, N, K)
            torch.cuda.synchronize()
            assert ("dequant_gemm" if once else "generic_rows") in tc.cuda_last_kernel_name()
            assert tc.launch_count() - before == (2 + fused if once else (M + 3) // 4)
            got = by.to_numpy((M, N), np.float16).astype(np.float64)
            assert oracle.scaled_rms(got, wantf if fused else want) <= 1.1 * np.sqrt(3.0 if fused else 2.0) * ROUND
    assert tc.take_device_error(ctx) == 0


def test_large_fused_call_does_not_depend_on_the_room_of_earlier_ones(tc, ctx, oracle):
    """4700 rows with fp32 results go through the room for normalised rows in slabs of the call's own, whatever
    size the room has grown to: the same bits."""
    import torch
    M, N, K = 4700, 1280, 2048
    X, Wq = data(oracle, 0, 64, N, K)
    x = torch.from_numpy(X).cuda().repeat(128, 1)
    g, w = torch.ones(4 * K, dtype=torch.float16, device="cuda"), torch.from_numpy(Wq).cuda()
    big_w = torch.zeros(128 * 4 * K // 32 * 18, dtype=torch.uint8, device="cuda")
    outs = [torch.zeros(M, N, dtype=torch.float32, device="cuda") for _ in range(2)]
    y = torch.zeros(2048, 128, dtype=torch.float32, device="cuda")
    with ctx.stream() as s:
        st = s.cuda_handle()
        torch.cuda.synchronize()

        def call(rows, weights, out, n, k):
            tc.raw_fused_rmsnorm_gemv_quantized(ctx, x.data_ptr(), g.data_ptr(), weights.data_ptr(), out.data_ptr(), 0, rows, n, k,
                                                1e-5, "f16", "f32", st)
        call(M, w, outs[0], N, K)
        call(2048, big_w, y, 128, 4 * K)         # a room more than three times as large
        call(M, w, outs[1], N, K)
        torch.cuda.synchronize()
    assert torch.equal(outs[0], outs[1])
    want = oracle.fused_rmsnorm_gemv_quantized_f32(X[:8].astype(np.float32), np.ones(K, np.float32), Wq, 0, N)
    assert oracle.scaled_rms(outs[0][:8].cpu().numpy(), want) <= 1.1 * np.sqrt(2.0) * ROUND
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("fmt,M,N,K", [(0, 8, 19200, 2048), (0, 5, 22016, 2304), (1, 16, 19000, 4096), (0, 33, 19073, 3072), (0, 260, 9600, 2048),
                                       (1, 130, 20000, 2048)])
def test_tiles_left_over_after_whole_rounds(tc, ctx, oracle, fmt, M, N, K):
    """More tiles than SMs and a few left over, whose K is split in a launch of their own (two launches): the first
    rows of W, and the last ones, which are in it."""
    X, Wq = data(oracle, fmt, M, N, K)
    blocks = np.asarray(Wq).reshape(N, -1)
    some = np.r_[0:64, N - 700:N]
    want = oracle.dequant_dot_f64(X.astype(np.float64), np.ascontiguousarray(blocks[some]), fmt, len(some))
    with ctx.buffer_from_array(X) as bx, ctx.buffer_from_array(Wq) as bw, ctx.buffer(M * N * 2) as by:
        outs = []
        for _ in range(3):
            before = tc.launch_count()
            ctx.gemv_quantized(bx, bw, by, fmt, M, N, K)
            assert "tcgen05" in tc.cuda_last_kernel_name() and tc.launch_count() - before == 2
            outs.append(by.to_numpy((M, N), np.float16))
    assert np.array_equal(outs[0], outs[1]) and np.array_equal(outs[0], outs[2])
    assert oracle.scaled_rms(outs[0][:, some].astype(np.float64), want) <= 1.1 * np.sqrt(2.0) * ROUND
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("fmt,M,N,K,once", [(0, 4096, 2048, 4096, True), (0, 4095, 2048, 4096, False), (1, 4096, 2048, 4096, True),
                                            (0, 4100, 1024, 8448, True), (1, 4095, 1024, 8448, False), (1, 4096, 1024, 4096, False)])
def test_very_many_rows_dequantise_once(tc, ctx, oracle, fused, fmt, M, N, K, once):
    """From some thousands of rows on the weights are dequantised once and multiplied as a GEMM (two launches, three
    with the norm); below, the tcgen05 kernel dequantises on the way (one or two, and the norm pass)."""
    import torch
    X, Wq = data(oracle, fmt, 64, N, K)
    g = (1 + 0.1 * np.random.default_rng(8).standard_normal(K)).astype(np.float16)
    x, w, gam = torch.from_numpy(X).cuda().repeat((M + 63) // 64, 1)[:M].contiguous(), torch.from_numpy(Wq).cuda(), torch.from_numpy(g).cuda()
    x64 = X.astype(np.float64)
    if fused:
        x64 = x64 / np.sqrt((x64 * x64).mean(axis=1, keepdims=True) + 1e-5) * g
    want = oracle.dequant_dot_f64(x64[:8], Wq, fmt, N)
    y = torch.zeros(M, N, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    before = tc.launch_count()
    if fused:
        tc.raw_fused_rmsnorm_gemv_quantized(ctx, x.data_ptr(), gam.data_ptr(), w.data_ptr(), y.data_ptr(), fmt, M, N, K, 1e-5)
    else:
        tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), fmt, M, N, K)
    torch.cuda.synchronize()
    launches = tc.launch_count() - before
    assert launches == (3 if fused else 2) if once else launches - fused in (1, 2)
    got = y.cpu().numpy()
    bar = 1.1 * np.sqrt(3.0 if fused else 2.0) * ROUND
    for at in (0, 64 * ((M - 8) // 64)):                      # the first copy of the rows and the last
        assert oracle.scaled_rms(got[at:at + 8].astype(np.float64), want) <= bar
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("fmt,M,N,K", [
    (0, 5, 3841, 4096), (0, 16, 3900, 4352), (0, 32, 4096, 14336), (0, 17, 8192, 8192), (1, 16, 3800, 4096), (1, 13, 11008, 4096),
    (0, 8, 19200, 2048), (0, 16, 38000, 768), (0, 32, 57000, 256), (0, 33, 19073, 3072), (0, 64, 38100, 2048), (0, 100, 20000, 2048),
    (0, 130, 20000, 2048), (0, 300, 9700, 2304), (0, 256, 19100, 2048), (1, 48, 20000, 2048), (1, 128, 28672, 2304), (1, 520, 7000, 4096)])
def test_shares_of_the_unit_list(tc, ctx, oracle, fmt, M, N, K):
    """Every CTA has the same number of units, wherever tiles end: shares shorter than a tile (a tile of two to six
    CTAs), longer, of one unit more or less, in every accumulator layout.  One launch; the same bits each time."""
    import torch
    X, Wq = data(oracle, fmt, M, 128, K)
    reps = (N + 127) // 128                                   # every tile the same 128 rows: one oracle call for all of them
    want = oracle.dequant_dot_f64(X.astype(np.float64), Wq, fmt, 128)
    x, w = torch.from_numpy(X).cuda(), torch.from_numpy(np.asarray(Wq)).cuda().reshape(128, -1).repeat(reps, 1)[:N].contiguous()
    want = torch.from_numpy(want).cuda().repeat(1, reps)[:, :N]
    y = torch.empty(M, N, dtype=torch.float16, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    outs = []
    for _ in range(3):
        y.fill_(float("nan"))
        before = tc.launch_count()
        tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), fmt, M, N, K, "f16", "f16", st)
        assert "tcgen05" in tc.cuda_last_kernel_name() and tc.launch_count() - before == 1
        outs.append(y.clone())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    err = ((outs[0].double() - want) / want.square().mean().sqrt()).square()
    bar = 1.1 * np.sqrt(2.0) * ROUND
    assert err.mean().sqrt().item() <= bar
    # a tile's share of the error: one wrong tile would vanish in the mean of all
    assert err.mean(0).sqrt().max().item() <= 4 * bar
    assert tc.take_device_error(ctx) == 0


def distinct_tiles(oracle, fmt, M, N, K, seed=0):
    """Weights whose tiles of 128 rows differ, for the price of one: the same rows, further on in every tile, times a power
    of two of its own.  Returns activations, weights, the 64-bit results without those factors, and the factors."""
    import torch
    X, Wq = data(oracle, fmt, M, 128, K)
    if seed:
        _, Wq = data(oracle, fmt, M + seed, 128, K)
    rows = torch.arange(N, device="cuda")
    tile = rows // 128
    at, power = (rows + tile) % 128, tile % 5 - 2
    w = torch.from_numpy(np.asarray(Wq)).cuda().reshape(128, K // 32, -1)[at].contiguous()
    d = w[:, :, :2].contiguous().view(torch.float16)
    w[:, :, :2] = (d * torch.pow(2.0, power.half()).view(-1, 1, 1)).view(torch.uint8)
    want = torch.from_numpy(oracle.dequant_dot_f64(X.astype(np.float64), Wq, fmt, 128)).cuda()[:, at]
    return torch.from_numpy(X).cuda(), w, want, torch.pow(2.0, power.double())


def check_tiles(got, want, factors, bar):
    """All results against `bar`, and each column: one wrong tile would vanish in the mean of all."""
    err = ((got.double() / factors - want) / want.square().mean().sqrt()).square()
    assert err.mean().sqrt().item() <= bar
    assert err.mean(0).sqrt().max().item() <= 4 * bar


@pytest.mark.parametrize("fmt,M,N,K", [
    (0, 5, 3841, 4096), (0, 16, 3900, 4352), (0, 32, 4096, 14336), (0, 17, 8192, 8192), (1, 16, 3800, 4096), (1, 13, 11008, 4096),
    (0, 8, 19200, 2048), (0, 16, 38000, 768), (0, 32, 57000, 256), (0, 33, 19073, 3072), (0, 64, 38100, 2048), (0, 100, 20000, 2048),
    (0, 130, 20000, 2048), (0, 300, 9700, 2304), (0, 256, 19100, 2048), (1, 48, 20000, 2048), (1, 128, 28672, 2304), (1, 520, 7000, 4096)])
def test_shares_over_tiles_that_differ(tc, ctx, oracle, fmt, M, N, K):
    """The shapes of the test above over tiles that can be told apart: a unit of the wrong tile, or a neighbour's sums at
    the wrong place, shows."""
    import torch
    x, w, want, factors = distinct_tiles(oracle, fmt, M, N, K)
    y = torch.empty(M, N, dtype=torch.float16, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    outs = []
    for _ in range(3):
        y.fill_(float("nan"))
        before = tc.launch_count()
        tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), fmt, M, N, K, "f16", "f16", st)
        assert "tcgen05" in tc.cuda_last_kernel_name() and tc.launch_count() - before == 1
        outs.append(y.clone())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    check_tiles(outs[0], want, factors, 1.1 * np.sqrt(2.0) * ROUND)
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("fmt,M,K,Ns", [(0, 8, 2048, (9000, 5000, 5100)), (0, 5, 4096, (130, 11009, 127, 7700)), (1, 16, 2304, (10010, 9001)),
                                        (0, 40, 3072, (6400, 6500, 6337)), (0, 130, 2048, (10011, 9990)), (0, 300, 2304, (4993, 4700))])
def test_shares_that_go_on_in_the_next_matrix(tc, ctx, oracle, fmt, M, K, Ns):
    """Products that share their activations, recorded: one launch whose runs of units cross from one matrix to the next
    (another tensor map, row count and result), with row counts that are no whole tiles.  Launched directly, captured and
    replayed, always the same bits."""
    import torch
    cases = [distinct_tiles(oracle, fmt, M, n, K, seed=i) for i, n in enumerate(Ns)]
    x = cases[0][0]                             # the same activations in each
    ys = [torch.empty(M, n, dtype=torch.float16, device="cuda") for n in Ns]
    torch.cuda.synchronize()
    wrap = lambda t: ctx.buffer_from_ptr(t.data_ptr(), t.numel() * t.element_size())
    bx, bws, bys = wrap(x), [wrap(w) for _, w, _, _ in cases], [wrap(y) for y in ys]
    first = None
    with ctx.stream() as s:
        for _ in range(4):
            for y in ys:
                y.fill_(float("nan"))
            torch.cuda.synchronize()
            before = tc.launch_count()
            for bw, by, n in zip(bws, bys, Ns):
                ctx.gemv_quantized_async(bx, bw, by, fmt, M, n, K, s)
            s.sync()
            assert tc.launch_count() - before == 1 and "tcgen05" in tc.cuda_last_kernel_name()
            got = [y.clone() for y in ys]
            first = first or got
            assert all(torch.equal(a, b) for a, b in zip(got, first))
    for got, (_, _, want, factors) in zip(first, cases):
        check_tiles(got, want, factors, 1.1 * np.sqrt(2.0) * ROUND)
    for b in [bx] + bws + bys:
        b.close()
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("fmt,M,N,K", [(0, 8, 19200, 2048), (0, 5, 22016, 2304), (1, 16, 19000, 4096), (0, 33, 19073, 3072), (0, 260, 9600, 2048),
                                       (1, 130, 20000, 2048)])
def test_tiles_left_over_in_a_captured_call(tc, ctx, oracle, fmt, M, N, K):
    """A captured call has no scratch for shares: whole rounds of tiles, and the rest in a launch of its own in which their K
    is split."""
    import torch
    x, w, want, factors = distinct_tiles(oracle, fmt, M, N, K)
    y = torch.empty(M, N, dtype=torch.float16, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    before = tc.launch_count()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=st):
        tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), fmt, M, N, K, "f16", "f16", st.cuda_stream)
    assert tc.launch_count() - before == 2 and "tcgen05" in tc.cuda_last_kernel_name()
    outs = []
    for _ in range(3):
        y.fill_(float("nan"))
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            graph.replay()
        torch.cuda.synchronize()
        outs.append(y.clone())
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    check_tiles(outs[0], want, factors, 1.1 * np.sqrt(2.0) * ROUND)
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("fmt,M,N,K", [(0, 32, 768, 28672), (0, 16, 1024, 20480), (0, 8, 1400, 10240), (1, 16, 2048, 28672), (0, 16, 2048, 28672),
                                       (1, 14, 2400, 14336), (0, 32, 2560, 11008), (1, 32, 2560, 14336), (0, 8, 2800, 8192)])
def test_few_tiles_of_long_rows(tc, ctx, oracle, fmt, M, N, K):
    """Fewer tiles than SMs by far: split over clusters, or shares with up to ten CTAs a tile; one launch, the same bits."""
    import torch
    x, w, want, factors = distinct_tiles(oracle, fmt, M, N, K)
    st = torch.cuda.current_stream().cuda_stream
    outs = []
    for _ in range(3):
        y = torch.full((M, N), float("nan"), device="cuda").half()
        before = tc.launch_count()
        tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), fmt, M, N, K, "f16", "f16", st)
        assert "tcgen05" in tc.cuda_last_kernel_name() and tc.launch_count() - before == 1
        outs.append(y)
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    check_tiles(outs[0], want, factors, 1.1 * np.sqrt(2.0) * ROUND)
    assert tc.take_device_error(ctx) == 0
