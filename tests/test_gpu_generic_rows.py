"""GPU: the kernel for quantized rows that no tiled copy can describe (K not a multiple of 256, weights at
any even address), at the edges of its blocks-per-lane and rows-per-warp split.

fp32 activations and results stay fp32 arithmetic: a sum of K products in fp32 differs from the 64-bit one
by about sqrt(K) * 2^-24 relative to its terms, below 2e-6 scaled RMS for K up to 9000."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 1, 32), (2, 3, 96), (3, 5, 1056), (4, 37, 992), (1, 601, 4128), (3, 1187, 2080),
                                   (4, 150, 8352), (6, 40, 544), (4, 20, 20512)])
def test_fp32_rows_against_64_bit(tc, ctx, oracle, fmt, M, N, K):
    rng = np.random.default_rng(M * 31 + N * 7 + K + fmt)
    Wq = oracle.quantize_weights((rng.standard_normal((N, K)) * 0.02).astype(np.float16), fmt)
    X = rng.standard_normal((M, K)).astype(np.float32)
    g = (1 + 0.1 * rng.standard_normal(K)).astype(np.float32)
    want = oracle.dequant_dot_f64(X.astype(np.float64), Wq, fmt, N)
    x64 = X.astype(np.float64)
    xn = x64 / np.sqrt((x64 * x64).mean(axis=1, keepdims=True) + 1e-5) * g
    wantf = oracle.dequant_dot_f64(xn, Wq, fmt, N)
    with ctx.buffer_from_array(X) as bx, ctx.buffer_from_array(Wq) as bw, ctx.buffer_from_array(g) as bg, \
            ctx.buffer(M * N * 4) as by:
        tc.gemv_quantized_ex(ctx, bx, bw, by, fmt, M, N, K, "f32", "f32", None)
        assert "generic" in tc.cuda_last_kernel_name()
        assert oracle.scaled_rms(by.to_numpy((M, N), np.float32).astype(np.float64), want) <= 2e-6
        tc.fused_rmsnorm_gemv_quantized_ex(ctx, bx, bg, bw, by, fmt, M, N, K, 1e-5, "f32", "f32", None)
        assert oracle.scaled_rms(by.to_numpy((M, N), np.float32).astype(np.float64), wantf) <= 2e-6


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("w_off,x_off", [(2, 0), (4, 2), (6, 6), (8, 10), (1, 0), (14, 14)])
def test_any_weight_and_activation_address(tc, ctx, oracle, fmt, w_off, x_off):
    """Same bits wherever the operands lie, up to fp32 summation order."""
    import torch
    M, N, K = 3, 70, 1120
    rng = np.random.default_rng(w_off + 100 * x_off + fmt)
    Wq = oracle.quantize_weights((rng.standard_normal((N, K)) * 0.02).astype(np.float16), fmt)
    X = rng.standard_normal((M, K)).astype(np.float16)
    want = oracle.dequant_dot_f64(X.astype(np.float64), Wq, fmt, N)
    with ctx.buffer(X.nbytes + 16) as bx, ctx.buffer(Wq.nbytes + 16) as bw, ctx.buffer(M * N * 4) as by:
        bx.upload(X, x_off)
        bw.upload(Wq, w_off)
        tc.raw_gemv_quantized(ctx, bx.device_ptr() + x_off, bw.device_ptr() + w_off, by.device_ptr(), fmt, M, N, K, "f16", "f32")
        torch.cuda.synchronize()
        assert oracle.scaled_rms(by.to_numpy((M, N), np.float32).astype(np.float64), want) <= 2e-6


@pytest.mark.parametrize("M,launches", [(1, 1), (4, 1), (7, 2)])
def test_weights_at_an_odd_address_take_four_rows_a_launch(tc, ctx, oracle, M, launches):
    import torch
    N, K = 70, 1120
    rng = np.random.default_rng(M)
    Wq = oracle.quantize_weights((rng.standard_normal((N, K)) * 0.02).astype(np.float16), 0)
    X = rng.standard_normal((M, K)).astype(np.float16)
    want = oracle.dequant_dot_f64(X.astype(np.float64), Wq, 0, N)
    with ctx.buffer_from_array(X) as bx, ctx.buffer(Wq.nbytes + 16) as bw, ctx.buffer(M * N * 4) as by:
        bw.upload(Wq, 1)
        before = tc.launch_count()
        tc.raw_gemv_quantized(ctx, bx.device_ptr(), bw.device_ptr() + 1, by.device_ptr(), 0, M, N, K, "f16", "f32")
        torch.cuda.synchronize()
        assert tc.launch_count() - before == launches
        assert tc.cuda_last_kernel_name() == "q4_0_gemv_generic_sm100"
        assert oracle.scaled_rms(by.to_numpy((M, N), np.float32).astype(np.float64), want) <= 2e-6


@pytest.mark.parametrize("fmt", [0, 1])
def test_fp32_sums_are_closer_than_one_chain_per_block(tc, ctx, oracle, fmt):
    """The order of additions: against 64 bits the kernel is closer than 32 fused multiply-adds in a row per block,
    then the scale, added over 32 lanes' blocks in a tree (restated here in numpy; a few thousand results, so that
    the two errors stand apart by many times their scatter)."""
    M, N, K = 3, 1500, 4128
    rng = np.random.default_rng(4128 + fmt)
    Wq = oracle.quantize_weights((rng.standard_normal((N, K)) * 0.02).astype(np.float16), fmt)
    X = rng.standard_normal((M, K)).astype(np.float32)
    want = oracle.dequant_dot_f64(X.astype(np.float64), Wq, fmt, N)
    with ctx.buffer_from_array(X) as bx, ctx.buffer_from_array(Wq) as bw, ctx.buffer(M * N * 4) as by:
        tc.gemv_quantized_ex(ctx, bx, bw, by, fmt, M, N, K, "f32", "f32", None)
        assert "generic_rows" in tc.cuda_last_kernel_name()
        got = by.to_numpy((M, N), np.float32).astype(np.float64)
    blocks = Wq.reshape(N, K // 32, -1)
    d = blocks[:, :, :2].copy().view(np.float16)[:, :, 0].astype(np.float32)
    qs = blocks[:, :, 2:]
    q = np.concatenate([qs & 15, qs >> 4], axis=2).astype(np.float32) - 8 if fmt == 0 else qs.copy().view(np.int8).astype(np.float32)
    chain = np.zeros((M, N), np.float32)
    for m in range(M):
        x = X[m].reshape(-1, 32).astype(np.float64)
        acc = np.zeros(d.shape, np.float32)
        for i in range(32):
            acc = (x[None, :, i] * q[:, :, i] + acc).astype(np.float32)
        lanes = np.zeros((N, 160), np.float32)
        lanes[:, :d.shape[1]] = acc * d
        for c in range(0, 160, 32):
            v = lanes[:, c:c + 32]
            while v.shape[1] > 1:
                v = v[:, :v.shape[1] // 2] + v[:, v.shape[1] // 2:]
            chain[m] += v[:, 0]
    assert oracle.scaled_rms(got, want) <= 0.92 * oracle.scaled_rms(chain.astype(np.float64), want)


@pytest.mark.parametrize("fmt", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 3, 50016), (1, 200, 40032), (2, 1190, 16416), (1, 9571, 2080), (3, 9472, 1056), (4, 9546, 1056), (1, 2300, 28704)])
def test_units_of_a_warp_over_groups_and_chunks(tc, ctx, oracle, fmt, M, N, K):
    """A warp goes from unit to unit by a step of so many chunks and row groups: one group a CTA to more than there are warps,
    CTAs with a row more that have a group more, rows of up to the length that fits shared memory, each unit once.
    Bar as above: 32 products in two chains, 32 blocks in a tree and up to 49 chunks in order round less often than
    a chain of 9000."""
    rng = np.random.default_rng(N + K + fmt)
    rows = min(N, 97)                                    # the weights repeat, N / 97 no whole number: the oracle's share of the time
    Wq = np.asarray(oracle.quantize_weights((rng.standard_normal((rows, K)) * 0.02).astype(np.float16), fmt)).reshape(rows, -1)
    X = rng.standard_normal((M, K)).astype(np.float32)
    at = np.arange(N) % rows
    want = oracle.dequant_dot_f64(X.astype(np.float64), Wq, fmt, rows)[:, at]
    with ctx.buffer_from_array(X) as bx, ctx.buffer_from_array(np.ascontiguousarray(Wq[at])) as bw, ctx.buffer(M * N * 4) as by:
        tc.gemv_quantized_ex(ctx, bx, bw, by, fmt, M, N, K, "f32", "f32", None)
        assert "generic" in tc.cuda_last_kernel_name()
        got = by.to_numpy((M, N), np.float32).astype(np.float64)
    assert oracle.scaled_rms(got, want) <= 2e-6
    assert np.abs(got - want).max() <= 2e-5 * np.sqrt((want * want).mean())      # ten times the bar: a wrong unit would be 1e4 times it
