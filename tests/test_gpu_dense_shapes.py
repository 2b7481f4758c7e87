"""GPU: the dense fused norm + GEMV where its K ranges have to follow shared memory: few strips of very long
columns, several rows at a time.

Bar: normalised rows and results are fp16, 2^-11 / sqrt(3) rms each, a tenth on top."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BAR = 1.1 * np.sqrt(2.0) * 2.0 ** -11 / np.sqrt(3.0)


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(57088, 21504), (8192, 28672), (264, 40008), (1000, 1)])
def test_long_columns(tc, ctx, M, N, K):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(N + K + M)
    x, g = torch.randn(M, K, device="cuda", generator=gen).half(), (1 + 0.1 * torch.randn(K, device="cuda", generator=gen)).half()
    w = torch.empty(K, N, dtype=torch.float16, device="cuda").normal_(0, 0.02, generator=gen)
    y = torch.zeros(M, N, dtype=torch.float16, device="cuda")
    torch.cuda.synchronize()
    tc.raw_fused_norm_gemv_f16(ctx, x.data_ptr(), g.data_ptr(), 0, w.data_ptr(), y.data_ptr(), M, N, K, 1e-5)
    torch.cuda.synchronize()
    assert "split" in tc.cuda_last_kernel_name()
    xn = x.double()
    xn = xn * torch.rsqrt((xn * xn).mean(dim=1, keepdim=True) + 1e-5) * g.double()
    want = torch.cat([xn @ w[:, c:c + 4096].double() for c in range(0, N, 4096)], dim=1)
    err = (((y.double() - want) ** 2).mean() / (want ** 2).mean()).sqrt().item()
    assert err <= BAR
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("M", [1, 2, 3, 4])
@pytest.mark.parametrize("N,K", [(8, 30016), (200, 16000), (264, 4000), (1400, 8082), (2600, 9114), (520, 63), (256, 129)])
def test_many_ranges_per_strip(tc, ctx, M, N, K):
    """One to about a hundred K ranges a strip, whose sums the last one takes several at a time: a whole number of times and
    with some left over, full strips and narrow ones; the same bits each time."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(N + K + M)
    x, g = torch.randn(M, K, device="cuda", generator=gen).half(), (1 + 0.1 * torch.randn(K, device="cuda", generator=gen)).half()
    w = torch.empty(K, N, dtype=torch.float16, device="cuda").normal_(0, 0.02, generator=gen)
    outs = []
    for _ in range(3):
        y = torch.full((M, N), float("nan"), device="cuda").half()
        torch.cuda.synchronize()
        tc.raw_fused_norm_gemv_f16(ctx, x.data_ptr(), g.data_ptr(), 0, w.data_ptr(), y.data_ptr(), M, N, K, 1e-5)
        torch.cuda.synchronize()
        outs.append(y)
    assert "split" in tc.cuda_last_kernel_name()
    assert torch.equal(outs[0], outs[1]) and torch.equal(outs[0], outs[2])
    xn = x.double()
    xn = xn * torch.rsqrt((xn * xn).mean(dim=1, keepdim=True) + 1e-5) * g.double()
    want = xn @ w.double()
    # of few results the rms scatters: 1 / sqrt(2 n), three of them, and the odd one near a power of two
    bar = BAR * (1 + 3 / np.sqrt(2 * M * N))
    assert ((outs[0].double() - want).square().mean() / want.square().mean()).sqrt().item() <= bar
    assert tc.take_device_error(ctx) == 0
