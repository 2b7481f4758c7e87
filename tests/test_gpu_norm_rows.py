"""GPU: the row normalisation over row lengths that take each register count and the scalar kernel, against
64-bit arithmetic: one fp16 rounding of the result (2^-11 relative, half a unit in the last place) after
fp32 arithmetic of a few roundings (4 * 2^-24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("D", [8, 100, 2048, 2056, 4096, 8192, 14336, 16384, 16392])
@pytest.mark.parametrize("layer", [False, True])
def test_rows_against_64_bit(tc, ctx, D, layer):
    N = 5
    rng = np.random.default_rng(D)
    X = (rng.standard_normal((N, D)) * 3 + 0.5).astype(np.float16)
    g = (1 + 0.1 * rng.standard_normal(D)).astype(np.float16)
    b = (0.1 * rng.standard_normal(D)).astype(np.float16)
    x = X.astype(np.float64)
    mean = x.mean(axis=1, keepdims=True) if layer else 0.0
    rstd = 1.0 / np.sqrt(((x - mean) ** 2).mean(axis=1, keepdims=True) + 1e-5)
    want = (x - mean) * rstd * g + (b.astype(np.float64) if layer else 0.0)
    with ctx.buffer_from_array(X) as bx, ctx.buffer_from_array(g) as bg, ctx.buffer_from_array(b) as bb, \
            ctx.buffer(X.nbytes) as by, ctx.buffer(N * 4) as bm, ctx.buffer(N * 4) as br:
        if layer:
            tc.layernorm_forward(ctx, bx, bg, bb, by, bm, br, N, D, 1e-5)
        else:
            tc.rmsnorm_forward(ctx, bx, bg, by, br, N, D, 1e-5)
        got = by.to_numpy((N, D), np.float16).astype(np.float64)
        assert np.allclose(br.to_numpy((N,), np.float32), rstd[:, 0], rtol=1e-6)
    # the sum with beta can cancel: fp32 error relative to its terms
    terms = np.abs((x - mean) * rstd * g) + np.abs(b.astype(np.float64))
    assert (np.abs(got - want) <= 2.0 ** -11 * np.abs(want) + 2.0 ** -21 * terms + 2.0 ** -25).all()
