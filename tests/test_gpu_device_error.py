"""GPU: the device error word.  A kernel that gives up on a bounded wait sets it and leaves a wrong result; every
synchronous operation reports it until it is taken.  No kernel gives up here: the word is set from the host."""
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
