"""GPU: the device error word.  A kernel that gives up on a bounded wait sets it and leaves a wrong result; every
synchronous operation reports it until it is taken.  No kernel gives up here: the word is set from the host."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def calls(tc, ctx):
    """(name, buffers, call) of every kind of synchronous operation."""
    rng = np.random.default_rng(3)
    half = lambda *shape: ctx.buffer_from_array((rng.standard_normal(shape) * 0.1).astype(np.float16))
    K, N = 512, 520
    x, g, b, w, y = half(1, K), half(K), half(K), half(K, N), ctx.buffer(N * 2)
    stats = [ctx.buffer(4) for _ in range(2)]
    wf, wq, yq = half(N, K), ctx.buffer(tc.quantized_size("q4_0", N, K)), ctx.buffer(8 * N * 2)
    x8 = half(8, K)
    q, kv, o = half(4, 8, 1, 128), half(4, 2, 640, 128), ctx.buffer(4 * 8 * 128 * 2)
    qp, kp, op = half(1, 8, 256, 64), half(1, 8, 256, 64), ctx.buffer(8 * 256 * 64 * 2)
    cos = ctx.buffer_from_array(np.ones((1, 32), np.float32))
    out = [
        ("quantize", lambda: tc.quantize_weights(ctx, wf, wq, "q4_0", N, K)),
        ("gemv", lambda: tc.gemv_quantized(ctx, x, wq, y, "q4_0", 1, N, K)),
        ("batched gemv", lambda: tc.gemv_quantized(ctx, x8, wq, yq, "q4_0", 8, N, K)),
        ("dense rmsnorm gemv", lambda: tc.fused_rmsnorm_gemv(ctx, x, g, w, y, 1, N, K, 1e-5)),
        ("dense layernorm gemv", lambda: tc.fused_layernorm_gemv(ctx, x, g, b, w, y, 1, N, K, 1e-5)),
        ("attention, decode", lambda: tc.attention_forward(ctx, q, kv, kv, o, 4, 8, 1, 640, 128, causal=False, kv_heads=2)),
        ("attention, prefill", lambda: tc.attention_forward(ctx, qp, kp, kp, op, 1, 8, 256, 256, 64, causal=True, kv_heads=8)),
        ("gemm", lambda: tc.gemm(ctx, x8, w, yq, 8, N, K)),
        ("rmsnorm", lambda: tc.rmsnorm_forward(ctx, x, g, y, stats[0], 1, K, 1e-5)),
        ("layernorm", lambda: tc.layernorm_forward(ctx, x, g, b, y, stats[0], stats[1], 1, K, 1e-5)),
        ("swiglu", lambda: tc.swiglu_forward(ctx, x, x, y, K)),
        ("rope", lambda: tc.rope_forward(ctx, x, cos, cos, 1, 1, 1, 64)),
    ]
    return out, [x, g, b, w, y, wf, wq, yq, x8, q, kv, o, qp, kp, op, cos] + stats


def test_synchronous_operations_report_a_device_error(tc, ctx):
    ops, bufs = calls(tc, ctx)
    for _, call in ops:
        call()
    assert tc.take_device_error(ctx) == 0
    tc.set_device_error(ctx, 1)
    try:
        for name, call in ops:
            with pytest.raises(tc.TensorcoreError) as e:
                call()
                pytest.fail(name + " reported success")
            assert e.value.status == tc.TC_ERR_INTERNAL, name
        with ctx.stream() as s:
            tc.gemv_quantized_ex(ctx, bufs[0], bufs[6], bufs[4], "q4_0", 1, 520, 512, "f16", "f16", s)
            with pytest.raises(tc.TensorcoreError):
                s.sync()
    finally:
        assert tc.take_device_error(ctx) == 1
    for _, call in ops:
        call()
    assert tc.take_device_error(ctx) == 0
    for b in bufs:
        b.close()


def test_raw_calls_do_without_hand_over_scratch_until_the_error_is_taken(tc, ctx):
    """Once a kernel has given up, words of its launch may lie in the scratch that sums are handed over in.  Raw calls
    then take kernels that need none (merged chunks: the same bits), and the first ones after the error was taken have
    empty scratch again."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(5)
    half = lambda *shape: torch.randn(*shape, device="cuda", generator=gen).half()
    st = torch.cuda.Stream()
    x, g, w, y = half(2, 1536), half(1536), half(1536, 520) * 0.02, torch.zeros(2, 520, device="cuda").half()
    q, k, v, o = half(20, 8, 1, 128), half(20, 2, 1300, 128), half(20, 2, 1300, 128), torch.zeros(20, 8, 1, 128, device="cuda").half()
    N, K = 19200, 2048
    wf = half(N, K) * 0.02
    wq, xb, yb = torch.zeros(tc.quantized_size("q4_0", N, K), dtype=torch.uint8, device="cuda"), half(8, K), torch.zeros(8, N, device="cuda").half()
    torch.cuda.synchronize()
    tc.raw_quantize_weights(ctx, wf.data_ptr(), wq.data_ptr(), "q4_0", N, K, st.cuda_stream)
    d = tc.TCAttentionDesc(20, 8, 1, 1300, 128, tc.TC_DTYPE_F16, tc.TC_DTYPE_F32, 0.0, False, False, 2, 0, None)

    def run():
        """Results, and how many launches each call took."""
        outs = []
        for call, out in ((lambda: tc.raw_fused_norm_gemv_f16(ctx, x.data_ptr(), g.data_ptr(), 0, w.data_ptr(), y.data_ptr(), 2, 520, 1536, 1e-5,
                                                              st.cuda_stream), y),
                          (lambda: tc.lib().tcx_raw_attention_forward(ctx.handle, ctypes.byref(d), *(ctypes.c_void_p(t.data_ptr()) for t in (q, k, v, o)),
                                                                      None, ctypes.c_void_p(st.cuda_stream)), o),
                          (lambda: tc.raw_gemv_quantized(ctx, xb.data_ptr(), wq.data_ptr(), yb.data_ptr(), "q4_0", 8, N, K, "f16", "f16", st.cuda_stream), yb)):
            before = tc.launch_count()
            assert not call()
            outs.append((tc.cuda_last_kernel_name(), tc.launch_count() - before))
            st.synchronize()
            outs[-1] += (out.clone(),)
        torch.cuda.synchronize()
        return outs
    usual = run()
    assert [u[1] for u in usual] == [1, 1, 1] and "split" in usual[0][0]
    tc.set_device_error(ctx, 1)
    without = run()
    assert [u[1] for u in without] == [1, 2, 2] and "split" not in without[0][0]
    assert torch.equal(without[1][2], usual[1][2])
    for i, bar in ((0, 2.0 ** -11), (2, 2.0 ** -11)):       # sums in another order: a few roundings of the results differ
        a, b = usual[i][2].double(), without[i][2].double()
        assert ((a - b).square().mean() / a.square().mean()).sqrt().item() <= bar
    assert tc.take_device_error(ctx) == 1 and tc.take_device_error(ctx) == 0
    for a, b in zip(run(), usual):
        assert a[:2] == b[:2] and torch.equal(a[2], b[2])
