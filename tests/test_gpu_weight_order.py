"""GPU: weights written by the work just before a product on the same stream, without a synchronisation: the
product reads what was written.  Raw calls behind the quantiser or a copy, and recorded lists in which an
operation's result is a later one's weights."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("fmt,M,N,K", [
    (0, 1, 2048, 4096), (1, 1, 2048, 4096), (1, 1, 11008, 4096), (0, 3, 1000, 1056), (1, 1, 1000, 1056), (1, 8, 4096, 1024),
    (0, 8, 4096, 4096), (0, 40, 22016, 2048), (0, 200, 2048, 1024), (1, 16, 4096, 4096), (1, 100, 2048, 1056), (0, 3, 400, 20512)])
def test_raw_call_reads_the_weights_written_before_it(tc, ctx, fused, fmt, M, N, K):
    import torch
    name = ("q4_0", "q8_0")[fmt]
    size = tc.quantized_size(fmt, N, K)
    st = torch.cuda.Stream()
    with torch.cuda.stream(st):
        ws = [(torch.randn(N, K, device="cuda") * 0.02).half() for _ in range(2)]
        x, g = torch.randn(M, K, device="cuda").half(), torch.ones(K, device="cuda").half()
        q = torch.zeros(size, dtype=torch.uint8, device="cuda")
        blocks = [torch.zeros_like(q) for _ in range(2)]
        outs = [torch.zeros(M, N, dtype=torch.float16, device="cuda") for _ in range(8)]

        def product(w, y):
            if fused:
                tc.raw_fused_rmsnorm_gemv_quantized(ctx, x.data_ptr(), g.data_ptr(), w.data_ptr(), y.data_ptr(), name, M, N, K,
                                                    1e-5, "f16", "f16", st.cuda_stream)
            else:
                tc.raw_gemv_quantized(ctx, x.data_ptr(), w.data_ptr(), y.data_ptr(), name, M, N, K, "f16", "f16", st.cuda_stream)
        want = [torch.zeros_like(outs[0]) for _ in range(2)]
        for w, b, y in zip(ws, blocks, want):
            tc.raw_quantize_weights(ctx, w.data_ptr(), b.data_ptr(), name, N, K, st.cuda_stream)
            st.synchronize()
            product(b, y)
            st.synchronize()
        for i, y in enumerate(outs):
            if i < 4:
                tc.raw_quantize_weights(ctx, ws[i & 1].data_ptr(), q.data_ptr(), name, N, K, st.cuda_stream)
            else:
                q.copy_(blocks[i & 1])
            product(q, y)
        st.synchronize()
    for i, y in enumerate(outs):
        # the few-row kernels add partial sums in any order: a last place of fp16 beside cancelled sums
        d = (y.double() - want[i & 1].double()).abs().max().item()
        assert d <= 2.0 ** -10 * want[i & 1].double().abs().max().item(), i
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("fmt,M,N1,K1,N2,K2", [(0, 8, 2304, 2048, 128, 512), (1, 1, 8704, 4096, 64, 256), (1, 16, 2176, 1024, 256, 256)])
def test_recorded_result_that_is_a_later_operations_weights(tc, ctx, oracle, fmt, M, N1, K1, N2, K2):
    """Operation 0 is in front, operation 1 writes the buffer that operation 3 takes as weights; the same list with a
    wait after each operation gives the same results."""
    bb = (18, 34)[fmt]
    assert M * N1 * 2 == N2 * (K2 // 32) * bb
    rng = np.random.default_rng(N1 + M)
    X1, X2 = rng.standard_normal((M, K1)).astype(np.float16), rng.standard_normal((M, K2)).astype(np.float16)
    w1 = oracle.quantize_weights((rng.standard_normal((N1, K1)) * 0.02).astype(np.float16), fmt)
    b1, b2, bw, bt = (ctx.buffer_from_array(t) for t in (X1, X2, w1, np.zeros(M * N1 * 2, np.uint8)))
    y0, y2, y3 = (ctx.buffer(M * n * 2) for n in (N1, N1, N2))
    s = ctx.stream()
    results = []
    for wait in (True, False, False, False):
        bt.upload(np.zeros(M * N1 * 2, np.uint8))
        for x, w, y, n, k in ((b1, bw, y0, N1, K1), (b1, bw, bt, N1, K1), (b1, bw, y2, N1, K1), (b2, bt, y3, N2, K2)):
            ctx.gemv_quantized_async(x, w, y, fmt, M, n, k, s)
            if wait:
                s.sync()
        s.sync()
        results.append(y3.to_numpy((M, N2), np.float16).astype(np.float64))
    s.close()
    for b in (b1, b2, bw, bt, y0, y2, y3):
        b.close()
    fine = np.isfinite(results[0])
    for r in results[1:]:
        assert np.array_equal(np.isfinite(r), fine)
        scale = np.abs(results[0][fine]).max()
        assert np.abs(r[fine] - results[0][fine]).max() <= 2.0 ** -9 * scale
    assert tc.take_device_error(ctx) == 0
