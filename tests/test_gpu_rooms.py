"""GPU: scratch that belongs to a stream, when the caller captures the stream in a CUDA graph: a captured call
takes the room there is, and the graph stays valid whatever later calls need - more rows on the same stream,
attention, more streams than the library keeps rooms for.

Bars: fp16 results, 2^-11 / sqrt(3) rms for each rounding (weights, normalised rows, result), a tenth on top."""
import ctypes
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROUND = 2.0 ** -11 / np.sqrt(3.0)


def on_device(*arrays):
    import torch
    return [torch.from_numpy(a).cuda() for a in arrays]


def capture(stream, call):
    import torch
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        call()
    return graph


def disturb(tc, ctx, oracle):
    """Grows every room there is: attention with more and more key chunks, and dense and batched calls on more streams
    than the library keeps rooms for."""
    import torch
    rng = np.random.default_rng(1)
    for Sk in (4096, 16384):
        q, k = np.zeros((1, 32, 1, 128), np.float16), np.zeros((1, 8, Sk, 128), np.float16)
        bufs = [ctx.buffer_from_array(t) for t in (q, k, k, q)]
        tc.attention_forward(ctx, *bufs, 1, 32, 1, Sk, 128, causal=False, kv_heads=8)
        for b in bufs:
            b.close()
    M, N, K = 3, 264, 512
    x, g, w = on_device(rng.standard_normal((16, K)).astype(np.float16), np.ones(K, np.float16),
                        (rng.standard_normal((K, N)) * 0.02).astype(np.float16))
    y = torch.zeros(16, N, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream(priority=p) for p in (0, -1) for _ in range(20)]
    assert len({s.cuda_stream for s in streams}) > 33
    for s in streams:
        for m in (M, 16):
            tc.raw_fused_norm_gemv_f16(ctx, x.data_ptr(), g.data_ptr(), 0, w.data_ptr(), y.data_ptr(), m, N, K, 1e-5, s.cuda_stream)
        torch.cuda.synchronize()


@pytest.mark.parametrize("K,M,big", [(4096, 300, 700), (1056, 300, 700)])
def test_captured_quantized_call(tc, ctx, oracle, K, M, big):
    """K a multiple of 256: normalised rows in slabs of the room there is.  Else: normalised rows and the weights as
    fp16, or the kernel that needs neither."""
    import torch
    N = 256
    rng = np.random.default_rng(K)
    X = rng.standard_normal((big, K)).astype(np.float16)
    g = (1 + 0.1 * rng.standard_normal(K)).astype(np.float16)
    Wq = oracle.quantize_weights((rng.standard_normal((N, K)) * 0.02).astype(np.float16), 0)
    want = oracle.fused_rmsnorm_gemv_quantized_f32(X[:M].astype(np.float32), g.astype(np.float32), Wq, 0, N)
    x, gam, w = on_device(X, g, Wq)
    y, y2 = (torch.zeros(m, N, dtype=torch.float16, device="cuda") for m in (M, big))
    st = torch.cuda.Stream()
    torch.cuda.synchronize()

    def call(m, out):
        tc.raw_fused_rmsnorm_gemv_quantized(ctx, x.data_ptr(), gam.data_ptr(), w.data_ptr(), out.data_ptr(), "q4_0", m, N, K,
                                            1e-5, "f16", "f16", st.cuda_stream)
    call(100, y2)
    torch.cuda.synchronize()
    graph = capture(st, lambda: call(M, y))
    call(big, y2)
    torch.cuda.synchronize()
    disturb(tc, ctx, oracle)
    call(big, y2)
    torch.cuda.synchronize()
    y.zero_()
    with torch.cuda.stream(st):
        graph.replay()
    torch.cuda.synchronize()
    assert oracle.scaled_rms(y.cpu().numpy(), want) <= 1.1 * np.sqrt(3.0) * ROUND
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("M,warm", [(2, 0), (2, 2), (4, 1), (16, 0), (16, 5), (40, 16)])
def test_captured_dense_call(tc, ctx, oracle, M, warm):
    """The dense fused call: partial sums in a room of the graph's up to four rows, normalised rows in the stream's above; on
    a stream that has no rooms yet (warm = 0), and on one whose rooms are for fewer rows."""
    import torch
    N, K, big = 520, 1536, 64
    rng = np.random.default_rng(M + warm)
    X = rng.standard_normal((big, K)).astype(np.float16)
    g = (1 + 0.1 * rng.standard_normal(K)).astype(np.float16)
    W = (rng.standard_normal((K, N)) * 0.02).astype(np.float16)
    x64 = X[:M].astype(np.float64)
    want = (x64 / np.sqrt((x64 * x64).mean(axis=1, keepdims=True) + 1e-5) * g) @ W.astype(np.float64)
    x, gam, w = on_device(X, g, W)
    y, y2 = (torch.zeros(m, N, dtype=torch.float16, device="cuda") for m in (M, big))
    st = torch.cuda.Stream()
    torch.cuda.synchronize()

    def call(m, out, n=N):
        tc.raw_fused_norm_gemv_f16(ctx, x.data_ptr(), gam.data_ptr(), 0, w.data_ptr(), out.data_ptr(), m, n, K, 1e-5, st.cuda_stream)
    if warm:
        call(warm, y2)
        torch.cuda.synchronize()
    graph = capture(st, lambda: call(M, y))
    for m in (4, big):
        call(m, y2)
    torch.cuda.synchronize()
    disturb(tc, ctx, oracle)
    for _ in range(2):                        # the second replay finds the room as the first left it
        y.zero_()
        with torch.cuda.stream(st):
            graph.replay()
        torch.cuda.synchronize()
        assert oracle.scaled_rms(y.cpu().numpy(), want) <= 1.1 * np.sqrt(2.0) * ROUND
    assert tc.take_device_error(ctx) == 0


def test_captured_attention_without_room_for_its_chunks(tc, ctx):
    """A raw attention call captured on a context whose scratch is too small takes a row's keys in one piece; one that
    is captured after an eager call of its size gives the eager call's bits, also after the scratch has grown."""
    import torch
    B, H, Sq, Sk, D = 1, 1, 8192, 2048, 128
    st = torch.cuda.Stream()
    q, k, v = (torch.randn(B, H, s, D, device="cuda").half() for s in (Sq, Sk, Sk))
    o, o2, ref = (torch.zeros_like(q) for _ in range(3))
    torch.cuda.synchronize()

    def call(out, sk=Sk):
        d = tc.TCAttentionDesc(B, H, Sq, sk, D, tc.TC_DTYPE_F16, tc.TC_DTYPE_F32, 0.0, False, False, H, 0, None)
        rc = tc.lib().tcx_raw_attention_forward(ctx.handle, ctypes.byref(d), *(ctypes.c_void_p(t.data_ptr()) for t in (q, k, v, out)),
                                                None, ctypes.c_void_p(st.cuda_stream))
        assert rc == 0
    first = capture(st, lambda: call(o))
    call(ref)
    torch.cuda.synchronize()
    second = capture(st, lambda: call(o2))
    qq, kk = np.zeros((1, 64, 64, 128), np.float16), np.zeros((1, 8, 16384, 128), np.float16)
    bufs = [ctx.buffer_from_array(t) for t in (qq, kk, kk, qq)]
    tc.attention_forward(ctx, *bufs, 1, 64, 64, 16384, 128, causal=False, kv_heads=8)
    for b in bufs:
        b.close()
    for graph, out in ((first, o), (second, o2)):
        out.zero_()
        with torch.cuda.stream(st):
            graph.replay()
        torch.cuda.synchronize()
    assert torch.equal(o2, ref)
    assert (o.double() - ref.double()).abs().max() <= 2.0 ** -10 * ref.double().abs().max()
    assert tc.take_device_error(ctx) == 0


def dense_case(seed, M, N=520, K=1536):
    """Inputs of a dense fused call, and that call on a stream."""
    rng = np.random.default_rng(seed)
    x, g, w = on_device(rng.standard_normal((M, K)).astype(np.float16), (1 + 0.1 * rng.standard_normal(K)).astype(np.float16),
                        (rng.standard_normal((K, N)) * 0.02).astype(np.float16))
    import torch
    x64 = x.double()
    want = (x64 * torch.rsqrt((x64 * x64).mean(dim=1, keepdim=True) + 1e-5) * g.double()) @ w.double()

    def call(tc, ctx, out, handle):
        tc.raw_fused_norm_gemv_f16(ctx, x.data_ptr(), g.data_ptr(), 0, w.data_ptr(), out.data_ptr(), M, N, K, 1e-5, handle)
    return call, want.cpu().numpy()


def test_captured_dense_calls_beside_others(tc, ctx, oracle):
    """Graphs captured on one stream, replayed on two others at a time beside eager calls on the first: no launch takes
    another's sums."""
    import torch
    cases = [dense_case(i, 2) for i in range(3)]
    outs = [torch.zeros(2, 520, dtype=torch.float16, device="cuda") for _ in cases]
    streams = [torch.cuda.Stream() for _ in cases]
    torch.cuda.synchronize()
    first = streams[0]
    cases[0][0](tc, ctx, outs[0], first.cuda_stream)
    torch.cuda.synchronize()
    graphs = [capture(first, lambda i=i: cases[i][0](tc, ctx, outs[i], first.cuda_stream)) for i in (1, 2)]
    for _ in range(20):
        for o in outs:
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        for _ in range(10):
            for graph, st in zip(graphs, streams[1:]):
                with torch.cuda.stream(st):
                    graph.replay()
            cases[0][0](tc, ctx, outs[0], first.cuda_stream)
        torch.cuda.synchronize()
        for o, (_, want) in zip(outs, cases):
            assert oracle.scaled_rms(o.cpu().numpy(), want) <= 1.1 * np.sqrt(2.0) * ROUND
    assert tc.take_device_error(ctx) == 0


def test_captured_decode_attention_beside_others(tc, ctx):
    """Two captures of a decode step's attention have their chunks' states in rooms of their own: one launch each, the
    eager call's bits, also when they run at a time, beside eager calls on the stream they were captured on."""
    import torch
    B, H, Hkv, Sk, D = 8, 32, 8, 2048, 128
    gen = torch.Generator(device="cuda")
    gen.manual_seed(11)
    half = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).half()
    cases = [[half(B, h, s, D) for h, s in ((H, 1), (Hkv, Sk), (Hkv, Sk))] for _ in range(3)]
    outs = [torch.zeros(B, H, 1, D, device="cuda").half() for _ in cases]
    streams = [torch.cuda.Stream() for _ in cases]
    d = tc.TCAttentionDesc(B, H, 1, Sk, D, tc.TC_DTYPE_F16, tc.TC_DTYPE_F32, 0.0, False, False, Hkv, 0, None)
    torch.cuda.synchronize()

    def call(i):
        rc = tc.lib().tcx_raw_attention_forward(ctx.handle, ctypes.byref(d), *(ctypes.c_void_p(t.data_ptr()) for t in cases[i] + [outs[i]]),
                                                None, ctypes.c_void_p(streams[0].cuda_stream))
        assert rc == 0
    before = tc.launch_count()
    graphs = [capture(streams[0], lambda i=i: call(i)) for i in (1, 2)]
    assert tc.launch_count() - before == 2
    refs = []
    for i in range(3):
        call(i)
        torch.cuda.synchronize()
        refs.append(outs[i].clone())
        s = torch.softmax(cases[i][0].double().view(B, Hkv, 4, D) @ cases[i][1].double().transpose(2, 3) / D ** 0.5, 3) @ cases[i][2].double()
        assert ((refs[i].double().view(s.shape) - s).square().mean() / s.square().mean()).sqrt().item() <= 1.05 * ROUND
    for _ in range(20):
        for o in outs:
            o.fill_(float("nan"))
        torch.cuda.synchronize()
        for _ in range(10):
            for graph, st in zip(graphs, streams[1:]):
                with torch.cuda.stream(st):
                    graph.replay()
            call(0)
        torch.cuda.synchronize()
        assert all(torch.equal(o, r) for o, r in zip(outs, refs))
    assert tc.take_device_error(ctx) == 0


def test_rooms_of_graphs_that_are_gone_are_used_again(tc, ctx, oracle):
    """48 graphs captured and dropped, a room of 1.6 MB each: what is held at the end is a few of them."""
    import gc
    import time
    import torch
    call, want = dense_case(7, 4, 11008, 4096)
    out = torch.zeros(4, 11008, dtype=torch.float16, device="cuda")
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    free = None
    for i in range(48):
        graph = capture(st, lambda: call(tc, ctx, out, st.cuda_stream))
        out.zero_()
        torch.cuda.synchronize()
        with torch.cuda.stream(st):
            graph.replay()
        torch.cuda.synchronize()
        assert i % 16 or oracle.scaled_rms(out.cpu().numpy(), want) <= 1.1 * np.sqrt(2.0) * ROUND
        del graph
        gc.collect()
        time.sleep(0.01)                      # the driver tells of it from a thread of its own
        if i == 7:
            free = torch.cuda.mem_get_info()[0]
    assert free - torch.cuda.mem_get_info()[0] <= 16 << 20
    assert tc.take_device_error(ctx) == 0


def test_no_room_for_shares_that_are_not_dealt_out(tc, ctx):
    """Calls whose tiles stay whole leave memory as it is: scratch for the shares of 256 columns is 19 MB a stream."""
    import torch
    M, N, K = 256, 4096, 1024
    x, y = torch.randn(M, K, device="cuda").half(), torch.zeros(M, N, device="cuda").half()
    w = torch.zeros(tc.quantized_size("q4_0", N, K), dtype=torch.uint8, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(8)]

    def call(st):
        tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), "q4_0", M, N, K, "f16", "f16", st.cuda_stream)
        torch.cuda.synchronize()
    torch.cuda.synchronize()
    call(streams[0])
    free = torch.cuda.mem_get_info()[0]
    for st in streams:
        call(st)
    assert "tcgen05" in tc.cuda_last_kernel_name()
    assert free - torch.cuda.mem_get_info()[0] <= 16 << 20
    assert (y == 0).all() and tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("per_thread", [True, False])
def test_threads_that_hand_sums_over(tc, ctx, oracle, per_thread):
    """Dense, batched and attention calls of four threads at a time, none in another's room: on streams of their own, and on
    cudaStreamPerThread, which is one handle and a stream for each thread."""
    import torch
    N, K, M, S, B = 19968, 2048, 8, 1300, 20
    Wq = oracle.quantize_weights((np.random.default_rng(4).standard_normal((128, K)) * 0.02).astype(np.float16), 0)
    w = on_device(np.asarray(Wq))[0].reshape(128, -1).repeat(N // 128, 1).contiguous()
    d = tc.TCAttentionDesc(B, 8, 1, S, 128, tc.TC_DTYPE_F16, tc.TC_DTYPE_F32, 0.0, False, False, 2, 0, None)
    wrong = []

    def work(i):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(i)
        half = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).half()
        dense, want = dense_case(20 + i, 3)
        own = torch.cuda.Stream()
        st = 2 if per_thread else own.cuda_stream
        x, q, k, v = half(M, K), half(B, 8, 1, 128), half(B, 2, S, 128), half(B, 2, S, 128)
        y, o, z = torch.zeros(M, N, device="cuda").half(), torch.zeros_like(q), torch.zeros(3, 520, device="cuda").half()
        torch.cuda.synchronize()
        first = None
        for _ in range(10):
            for _ in range(5):
                dense(tc, ctx, z, st)
                tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), 0, M, N, K, "f16", "f16", st)
                rc = tc.lib().tcx_raw_attention_forward(ctx.handle, ctypes.byref(d), *(ctypes.c_void_p(t.data_ptr()) for t in (q, k, v, o)),
                                                        None, ctypes.c_void_p(st))
                assert rc == 0
            torch.cuda.synchronize()
            got = [t.clone() for t in (z, y, o)]
            torch.cuda.synchronize()
            first = first or got
            if not all(torch.equal(a, b) for a, b in zip(got, first)):
                wrong.append((i, "bits"))
        if oracle.scaled_rms(first[0].cpu().numpy(), want) > 1.1 * np.sqrt(2.0) * ROUND:
            wrong.append((i, "dense"))
        rows = oracle.dequant_dot_f64(x.cpu().numpy().astype(np.float64), Wq, 0, 128)
        if oracle.scaled_rms(first[1][:, N - 128:].cpu().numpy(), rows) > 1.1 * np.sqrt(2.0) * ROUND:
            wrong.append((i, "batched"))
        s = torch.softmax(q.double().view(B, 2, 4, 128) @ k.double().transpose(2, 3) / 128 ** 0.5, 3) @ v.double()
        if oracle.scaled_rms(first[2].cpu().numpy().reshape(B, 2, 4, 128), s.cpu().numpy()) > 1.1 * ROUND:
            wrong.append((i, "attention"))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
    assert tc.take_device_error(ctx) == 0


def test_streams_in_the_rooms_of_closed_ones(tc, ctx, oracle):
    """A stream that is opened after another was closed takes its rooms: the sums handed over in them are the new
    stream's, smaller calls and larger ones."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    half = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).half()
    S, B, N, K = 1300, 20, 19200, 2048
    w = torch.zeros(tc.quantized_size("q4_0", N, K), dtype=torch.uint8, device="cuda")
    tc.raw_quantize_weights(ctx, (half(N, K) * 0.02).data_ptr(), w.data_ptr(), "q4_0", N, K)
    q, k, v, x = half(B, 8, 1, 128), half(B, 2, S, 128), half(B, 2, S, 128), half(32, K)
    dense = [dense_case(30 + m, m) for m in (1, 4)]
    torch.cuda.synchronize()

    def work(s, m, b):
        st = s.cuda_handle()
        z, y, o = torch.zeros(m, 520, device="cuda").half(), torch.zeros(8 * m, N, device="cuda").half(), torch.zeros(b, 8, 1, 128, device="cuda").half()
        torch.cuda.synchronize()
        d = tc.TCAttentionDesc(b, 8, 1, S, 128, tc.TC_DTYPE_F16, tc.TC_DTYPE_F32, 0.0, False, False, 2, 0, None)
        before = tc.launch_count()
        dense[m > 1][0](tc, ctx, z, st)
        tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), 0, 8 * m, N, K, "f16", "f16", st)
        rc = tc.lib().tcx_raw_attention_forward(ctx.handle, ctypes.byref(d), *(ctypes.c_void_p(t.data_ptr()) for t in (q, k, v, o)), None,
                                                ctypes.c_void_p(st))
        assert rc == 0 and tc.launch_count() - before == 3
        torch.cuda.synchronize()
        assert oracle.scaled_rms(z.cpu().numpy(), dense[m > 1][1]) <= 1.1 * np.sqrt(2.0) * ROUND
        return z, y, o
    sizes = [(1, 16), (4, 20), (1, 16), (4, 20), (4, 20), (1, 16)]
    with ctx.stream() as s:
        refs = {size: work(s, *size) for size in sizes}
    for size in sizes:
        with ctx.stream() as s, ctx.stream() as s2:
            for st in (s, s2, s):
                assert all(torch.equal(a, b) for a, b in zip(work(st, *size), refs[size]))
    assert tc.take_device_error(ctx) == 0


def test_threads_on_streams_of_their_own(tc, ctx, oracle):
    """Fused batched calls of growing size from four threads: no call's rows are normalised into another's room."""
    import torch
    N, K = 256, 1024
    rng = np.random.default_rng(9)
    X = rng.standard_normal((256, K)).astype(np.float16)
    g = (1 + 0.1 * rng.standard_normal(K)).astype(np.float16)
    Wq = oracle.quantize_weights((rng.standard_normal((N, K)) * 0.02).astype(np.float16), 0)
    x, gam, w = on_device(X, g, Wq)
    torch.cuda.synchronize()
    rows = (8, 16, 40, 100, 256)

    def call(m, at, out, st):
        tc.raw_fused_rmsnorm_gemv_quantized(ctx, x[at:].data_ptr(), gam.data_ptr(), w.data_ptr(), out.data_ptr(), "q4_0", m, N, K,
                                            1e-5, "f16", "f16", st.cuda_stream)
    wrong = []

    def work(i):
        st = torch.cuda.Stream()
        for m in rows:
            at = (37 * i) % (257 - m)
            out, ref = (torch.zeros(m, N, dtype=torch.float16, device="cuda") for _ in range(2))
            torch.cuda.synchronize()
            for _ in range(20):
                call(m, at, out, st)
            st.synchronize()
            call(m, at, ref, st)
            st.synchronize()
            if not torch.equal(out, ref):
                wrong.append((i, m))
            full = oracle.fused_rmsnorm_gemv_quantized_f32(X[at:at + m].astype(np.float32), g.astype(np.float32), Wq, 0, N)
            if oracle.scaled_rms(out.cpu().numpy(), full) > 1.1 * np.sqrt(3.0) * ROUND:
                wrong.append((i, m, "values"))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
