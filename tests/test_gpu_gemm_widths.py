"""GPU: tc_gemm on the tensor cores over tile widths: shapes that take narrow, odd and 256-wide tiles, both
forms of both operands.  One rounding of the result: fp16 2^-11 / sqrt(3) = 2.82e-4 scaled RMS, bf16
2^-8 / sqrt(3) = 2.26e-3; a twentieth on top for the fp32 sums and small samples."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(8, 72, 64), (5, 4096, 136), (128, 2368, 192), (130, 9480, 72), (512, 11008, 128), (300, 1000, 520),
                                   (1024, 4800, 64)])
@pytest.mark.parametrize("ta,tb", [(False, True), (False, False), (True, True)])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_widths_against_64_bit(tc, ctx, M, N, K, ta, tb, dtype):
    import torch
    if ta and M % 8:
        pytest.skip("a transposed A has rows of M elements, which the tiled copies need in multiples of 8")
    dt = torch.float16 if dtype == "f16" else torch.bfloat16
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N + K)
    A = torch.randn((K, M) if ta else (M, K), generator=g, device="cuda").to(dt)
    B = torch.randn((N, K) if tb else (K, N), generator=g, device="cuda").to(dt)
    C = torch.full((M, N), float("nan"), device="cuda", dtype=dt)
    bufs = [ctx.buffer_from_ptr(t.data_ptr(), t.numel() * 2) for t in (A, B, C)]
    torch.cuda.synchronize()
    tc.gemm(ctx, *bufs, M, N, K, dtype=dtype, transpose_a=ta, transpose_b=tb)
    assert tc.cuda_last_kernel_name() == "gemm_f16_tcgen05_sm100"
    want = (A.double().t() if ta else A.double()) @ (B.double().t() if tb else B.double())
    err = ((C.double() - want).square().mean() / want.square().mean()).sqrt().item()
    for b in bufs:
        b.close()
    assert err <= 1.05 * (2.0 ** -11 if dtype == "f16" else 2.0 ** -8) / np.sqrt(3.0)
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("M,N,K", [(16, 4096, 328), (40, 2000, 1032), (300, 1000, 520)])
def test_padded_rows_against_64_bit(tc, ctx, M, N, K):
    # leading dimensions larger than K, K no multiple of 64: what lies behind a row's K elements does not count
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N + K)
    A = torch.randn((M, K + 72), generator=g, device="cuda").half()
    B = torch.randn((N, K + 200), generator=g, device="cuda").half()
    C = torch.full((M, N), float("nan"), device="cuda", dtype=torch.float16)
    bufs = [ctx.buffer_from_ptr(t.data_ptr(), t.numel() * 2) for t in (A, B, C)]
    torch.cuda.synchronize()
    tc.gemm(ctx, *bufs, M, N, K, transpose_b=True, lda=K + 72, ldb=K + 200)
    assert tc.cuda_last_kernel_name() == "gemm_f16_tcgen05_sm100"
    want = A[:, :K].double() @ B[:, :K].double().t()
    err = ((C.double() - want).square().mean() / want.square().mean()).sqrt().item()
    for b in bufs:
        b.close()
    assert err <= 1.05 * 2.0 ** -11 / np.sqrt(3.0)
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("M,N,ldc", [(1021, 160, 160), (130, 96, 104), (131, 40, 48), (257, 248, 248), (66, 32, 40), (5, 304, 304)])
@pytest.mark.parametrize("dtype", ["f16", "bf16"])
def test_rows_and_columns_past_the_result_stay(tc, ctx, M, N, ldc, dtype):
    """Rows and columns that are no multiples of the groups of four rows and 32 columns a store covers, rows of C further
    apart than its columns: results within one rounding, everything around them untouched."""
    import torch
    dt, K = torch.float16 if dtype == "f16" else torch.bfloat16, 192
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N)
    A, B = torch.randn(M, K, generator=g, device="cuda").to(dt), torch.randn(N, K, generator=g, device="cuda").to(dt)
    C = torch.full((M + 8, ldc), 7.0, device="cuda", dtype=dt)
    bufs = [ctx.buffer_from_ptr(t.data_ptr(), t.numel() * 2) for t in (A, B, C)]
    torch.cuda.synchronize()
    tc.gemm(ctx, *bufs, M, N, K, dtype=dtype, transpose_b=True, ldc=ldc)
    assert tc.cuda_last_kernel_name() == "gemm_f16_tcgen05_sm100"
    for b in bufs:
        b.close()
    want = A.double() @ B.double().t()
    err = ((C[:M, :N].double() - want).square().mean() / want.square().mean()).sqrt().item()
    assert err <= 1.05 * (2.0 ** -11 if dtype == "f16" else 2.0 ** -8) / np.sqrt(3.0)
    assert (C[M:] == 7.0).all() and (C[:, N:] == 7.0).all()
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("M", [1, 33, 63, 64, 65, 96, 128])
@pytest.mark.parametrize("N,K", [(40, 64), (264, 128), (1000, 1024)])
@pytest.mark.parametrize("tb", [True, False])
def test_both_forms_of_the_read_out(tc, ctx, M, N, K, tb):
    """Around the number of rows from which results leave by pieces of rows, one to four slices of K a stage; rows of the result
    before and behind it stay.  (One row takes the row kernel: the bar is the same.)"""
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(M + N + K)
    A, B = torch.randn(M, K, generator=g, device="cuda").half(), torch.randn((N, K) if tb else (K, N), generator=g, device="cuda").half()
    room = torch.full((M + 16, N), 7.0, device="cuda").half()
    C = room[8:8 + M]
    bufs = [ctx.buffer_from_ptr(t.data_ptr(), t.numel() * 2) for t in (A, B, C)]
    torch.cuda.synchronize()
    tc.gemm(ctx, *bufs, M, N, K, transpose_b=tb)
    for b in bufs:
        b.close()
    want = A.double() @ (B.double().t() if tb else B.double())
    # of few results the rms scatters: three times 1 / sqrt(2 n)
    bar = 1.05 * 2.0 ** -11 / np.sqrt(3.0) * (1 + 3 / np.sqrt(2 * M * N))
    assert ((C.double() - want).square().mean() / want.square().mean()).sqrt().item() <= bar
    assert (room[:8] == 7.0).all() and (room[8 + M:] == 7.0).all()
    assert tc.take_device_error(ctx) == 0
