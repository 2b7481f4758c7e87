"""GPU: the matrix attention kernel (head_dim 64 and 128) at the edges of its row tiles (16 and 64 rows of
(query, head) pairs), key steps (64) and key chunks, with every mask.

Bar against 64-bit softmax attention: the one rounding is the fp16 result, 2^-11 relative at most
(2^-11 / sqrt(3) = 2.82e-4 scaled RMS; a twentieth on top for the fp32 sums and small samples); the
log-sum-exp is an fp32 number: half a unit in the last place of its scores (up to 500 with ALiBi), 2^-23
relative with the sum's own rounding, and 1e-5."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def exact(Q, K, V, causal, window, slopes):
    B, H, Sq, D = Q.shape
    Hkv, Sk = K.shape[1], K.shape[2]
    q, k, v = (t.astype(np.float64) for t in (Q, K, V))
    k, v = np.repeat(k, H // Hkv, axis=1), np.repeat(v, H // Hkv, axis=1)
    s = q @ k.transpose(0, 1, 3, 2) / np.sqrt(D)
    i, j = np.arange(Sq)[:, None], np.arange(Sk)[None, :]
    if slopes is not None:
        s = s - np.asarray(slopes, np.float64)[None, :, None, None] * (i - j)
    hide = np.zeros((Sq, Sk), bool)
    if causal:
        hide |= j > i
    if window > 0:
        hide |= i - j > window
    s = np.where(hide, -np.inf, s)
    m = s.max(axis=-1, keepdims=True)
    p = np.exp(s - np.where(np.isfinite(m), m, 0.0))
    l = p.sum(axis=-1, keepdims=True)
    o = np.where(l > 0, p / np.where(l > 0, l, 1.0), 0.0) @ v
    with np.errstate(divide="ignore"):
        return o, (m + np.log(l))[..., 0]


def tcgen05(B, H, Hkv, Sq, Sk):
    """Which kernel a call takes on 148 SMs (prefill_block in attention.cu)."""
    R = Sq * (H // Hkv)
    tiles = B * Hkv * ((R + 63) // 64)
    if R <= 64 or Sk <= 128:
        return False
    return tiles > 296 if Sk <= 256 else 4 * tiles > 148 or tiles * ((Sk + 63) // 64) > 640


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D,causal,window,alibi", [
    (1, 1, 1, 1, 1, 128, False, 0, False), (2, 8, 1, 1, 63, 64, False, 0, False), (1, 16, 2, 2, 65, 128, False, 0, False),
    (1, 17, 1, 1, 200, 64, False, 0, True), (3, 4, 4, 16, 16, 64, True, 0, False), (1, 4, 4, 17, 17, 128, True, 0, False),
    (1, 8, 2, 64, 64, 128, True, 0, False), (2, 6, 2, 43, 129, 64, True, 0, True), (1, 8, 4, 200, 200, 128, True, 50, False),
    (1, 2, 2, 130, 70, 128, True, 0, False), (1, 2, 2, 300, 300, 64, False, 20, False), (1, 4, 1, 96, 1000, 128, False, 0, True),
    (1, 2, 2, 150, 40, 64, False, 30, False), (1, 8, 8, 300, 300, 128, True, 50, False), (2, 6, 6, 400, 400, 64, True, 0, True),
    (1, 8, 8, 310, 257, 128, False, 20, False), (1, 8, 8, 1, 16, 128, False, 0, False), (2, 15, 1, 1, 130, 64, False, 0, True),
    (1, 8, 8, 130, 300, 128, True, 0, False), (1, 5, 1, 13, 700, 128, True, 40, False), (1, 16, 8, 330, 258, 64, True, 33, True),
    (1, 40, 40, 600, 250, 64, False, 0, False)])
def test_against_64_bit(tc, ctx, B, H, Hkv, Sq, Sk, D, causal, window, alibi):
    rng = np.random.default_rng(Sq * 31 + Sk + D)
    Q = rng.standard_normal((B, H, Sq, D)).astype(np.float16)
    K = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    V = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    slopes = [2.0 ** -(1 + h % 8) for h in range(H)] if alibi else None
    want, lse = exact(Q, K, V, causal, window, slopes)
    bufs = [ctx.buffer_from_array(t) for t in (Q, K, V)] + [ctx.buffer(Q.nbytes), ctx.buffer(B * H * Sq * 4)]
    tc.attention_forward(ctx, *bufs[:4], B, H, Sq, Sk, D, LSE=bufs[4], causal=causal, kv_heads=Hkv, window_size=window,
                         alibi_slopes=slopes)
    assert tc.cuda_last_kernel_name() == ("attention_prefill_tcgen05_sm100" if tcgen05(B, H, Hkv, Sq, Sk) else "attention_mma_sm100")
    got = bufs[3].to_numpy(Q.shape, np.float16).astype(np.float64)
    got_lse = bufs[4].to_numpy((B, H, Sq), np.float32).astype(np.float64)
    for b in bufs:
        b.close()
    rms = np.sqrt(((got - want) ** 2).mean() / (want ** 2).mean())
    assert rms <= 1.05 * 2.0 ** -11 / np.sqrt(3.0)
    assert np.abs(got - want).max() <= 2.0 ** -11 * np.abs(want).max() + 1e-5
    seen = np.isfinite(lse)
    assert np.array_equal(seen, np.isfinite(got_lse)) and (np.abs(got_lse[seen] - lse[seen]) <= 1e-5 + 2.0 ** -23 * np.abs(lse[seen])).all()
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("off,Sq", [(2, 3), (4, 3), (8, 3), (8, 50)])
def test_unaligned_cache_takes_the_vector_kernel(tc, ctx, D, off, Sq):
    """A cache 2, 4 or 8 bytes past a 16-byte boundary gives the same results."""
    B, H, Hkv, Sk = 1, 4, 2, 150
    rng = np.random.default_rng(D)
    Q = rng.standard_normal((B, H, Sq, D)).astype(np.float16)
    K = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    V = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    want, _ = exact(Q, K, V, True, 0, None)
    bq, bo = ctx.buffer_from_array(Q), ctx.buffer(Q.nbytes)
    hold = [ctx.buffer(K.nbytes + 16) for _ in range(2)]
    views = []
    for h, t in zip(hold, (K, V)):
        h.upload(t, off)
        views.append(ctx.buffer_from_ptr(h.device_ptr() + off, t.nbytes))
    tc.attention_forward(ctx, bq, views[0], views[1], bo, B, H, Sq, Sk, D, causal=True, kv_heads=Hkv)
    assert tc.cuda_last_kernel_name() == "attention_decode_sm100"
    got = bo.to_numpy(Q.shape, np.float16).astype(np.float64)
    for b in [bq, bo] + views + hold:
        b.close()
    assert np.abs(got - want).max() <= 2.0 ** -11 * np.abs(want).max() + 1e-5


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("Sq,Sk", [(1, 300), (1, 3000), (100, 300), (40, 700)])
@pytest.mark.parametrize("window", [2 ** 31 - 1, 2 ** 31 - 200, 5000])
def test_a_window_wider_than_the_queries_hides_nothing(tc, ctx, D, Sq, Sk, window):
    """INT_MAX as "no limit", without the causal mask: keys far ahead of the query stay visible."""
    B, H, Hkv = 1, 4, 2
    rng = np.random.default_rng(Sq + Sk + D)
    Q = rng.standard_normal((B, H, Sq, D)).astype(np.float16)
    K = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    V = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    want, _ = exact(Q, K, V, False, 0, None)
    bufs = [ctx.buffer_from_array(t) for t in (Q, K, V)] + [ctx.buffer(Q.nbytes)]
    tc.attention_forward(ctx, *bufs, B, H, Sq, Sk, D, causal=False, kv_heads=Hkv, window_size=window)
    got = bufs[3].to_numpy(Q.shape, np.float16).astype(np.float64)
    for b in bufs:
        b.close()
    assert np.abs(got - want).max() <= 2.0 ** -11 * np.abs(want).max() + 1e-5


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk,gap", [(1, 8192, 18.0), (1, 4096, 22.0), (20, 1024, 18.0), (100, 8192, 18.0), (130, 2048, 22.0)])
def test_many_small_probabilities_beside_a_large_one(tc, ctx, D, Sq, Sk, gap):
    """Key 0 scores `gap` above all others (probabilities of e^-gap, down to 2^-32) and has values of zero: the
    result is made of the small probabilities alone.  Bar: the result's rounding, 2^-11 relative, the exponential's
    and the sum's, less than 1e-5, and what the two fp16 numbers of a probability leave out, 2^-40 of the largest
    probability for each key."""
    B, H, Hkv = 1, 4, 2
    Q, K, V = (np.zeros((B, h, s, D), np.float16) for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
    Q[..., 0] = 1.0
    K[:, :, 0, 0] = gap
    V[:, :, 1:, :] = 1000.0 * (1.0 + np.arange(D) / D)
    bufs = [ctx.buffer_from_array(t) for t in (Q, K, V)] + [ctx.buffer(Q.nbytes)]
    tc.attention_forward(ctx, *bufs, B, H, Sq, Sk, D, causal=False, kv_heads=Hkv, softmax_scale=1.0)
    got = bufs[3].to_numpy(Q.shape, np.float16).astype(np.float64)
    for b in bufs:
        b.close()
    p = np.exp(-gap)
    want = (Sk - 1) * p / (1.0 + (Sk - 1) * p) * V[0, 0, 1].astype(np.float64)
    assert want.min() > 2.0 ** -14
    assert (np.abs(got - want) <= (2.0 ** -11 + 1e-5) * want + Sk * 2.0 ** -40 * float(V.max())).all()


@pytest.mark.parametrize("D", [64, 96, 128])
@pytest.mark.parametrize("Sq,Sk,causal,window", [(1, 200, False, 0), (1, 3000, False, 0), (20, 70, True, 0), (150, 300, True, 0)])
def test_an_infinite_value_makes_its_element_infinite(tc, ctx, D, Sq, Sk, causal, window):
    """V[key, d] = inf: element d of every row that sees the key is inf, as p * inf is, and not NaN; nothing
    else changes.  The key's score is the row's average, far from underflow."""
    B, H, Hkv, key, d = 1, 4, 2, 0, 37
    rng = np.random.default_rng(Sq + Sk + D)
    Q = rng.standard_normal((B, H, Sq, D)).astype(np.float16)
    K = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    V = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    K[:, :, key] = 0
    bufs = [ctx.buffer_from_array(t) for t in (Q, K, V)] + [ctx.buffer(Q.nbytes)]
    outs = []
    for value in (V[0, 0, key, d], np.inf, -np.inf):
        V[:, :, key, d] = value
        bufs[2].upload(V)
        tc.attention_forward(ctx, *bufs, B, H, Sq, Sk, D, causal=causal, kv_heads=Hkv, window_size=window)
        outs.append(bufs[3].to_numpy(Q.shape, np.float16))
    for b in bufs:
        b.close()
    rest = np.arange(D) != d
    for got, value in zip(outs[1:], (np.inf, -np.inf)):
        assert (got[..., d] == value).all()
        assert np.array_equal(got[..., rest], outs[0][..., rest])


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("Sq,Sk", [(1, 3000), (5, 40), (20, 70), (150, 200), (70, 3000)])
@pytest.mark.parametrize("off", [2, 8])
def test_results_at_any_even_address(tc, ctx, D, Sq, Sk, off):
    """O past a 16-byte boundary: the same kernel and the same bits, nothing written beside them."""
    B, H, Hkv = 1, 4, 2
    rng = np.random.default_rng(Sq + Sk + D)
    Q = rng.standard_normal((B, H, Sq, D)).astype(np.float16)
    K = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    V = rng.standard_normal((B, Hkv, Sk, D)).astype(np.float16)
    bufs = [ctx.buffer_from_array(t) for t in (Q, K, V)] + [ctx.buffer(Q.nbytes)]
    hold = ctx.buffer(Q.nbytes + 32)
    hold.upload(np.full(Q.nbytes + 32, 0x5A, np.uint8))
    view = ctx.buffer_from_ptr(hold.device_ptr() + off, Q.nbytes)
    tc.attention_forward(ctx, *bufs, B, H, Sq, Sk, D, causal=False, kv_heads=Hkv)
    name = tc.cuda_last_kernel_name()
    tc.attention_forward(ctx, *bufs[:3], view, B, H, Sq, Sk, D, causal=False, kv_heads=Hkv)
    assert tc.cuda_last_kernel_name() == name and name != "attention_decode_sm100"
    got = hold.to_numpy((Q.nbytes + 32,), np.uint8)
    assert np.array_equal(got[off:off + Q.nbytes].view(np.uint16).reshape(Q.shape), bufs[3].to_numpy(Q.shape, np.uint16))
    assert (got[:off] == 0x5A).all() and (got[off + Q.nbytes:] == 0x5A).all()
    for b in [view, hold] + bufs:
        b.close()


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D,causal", [(5, 8, 8, 512, 1000, 64, False), (5, 8, 8, 512, 1300, 128, False), (2, 8, 8, 1300, 1300, 128, True), (40, 8, 8, 1, 3000, 128, False),
                                                    (40, 8, 8, 20, 1500, 64, False)])
def test_many_key_steps_in_one_block(tc, ctx, B, H, Hkv, Sq, Sk, D, causal):
    """So many row tiles that a block takes eight key steps or more: the ring of K and V is used several times over."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(Sk)
    q, k, v = (torch.randn(B, h, s, D, device="cuda", generator=gen).half() for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
    o = torch.zeros_like(q)
    torch.cuda.synchronize()
    bufs = [ctx.buffer_from_ptr(t.data_ptr(), t.numel() * 2) for t in (q, k, v, o)]
    before = tc.launch_count()
    tc.attention_forward(ctx, *bufs, B, H, Sq, Sk, D, causal=causal, kv_heads=Hkv)
    assert tc.launch_count() - before <= 2
    for b in bufs:
        b.close()
    s = torch.matmul(q.double(), k.double().transpose(2, 3)) / D ** 0.5
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    want = torch.matmul(torch.softmax(s, dim=3), v.double())
    err = (((o.double() - want) ** 2).mean() / (want ** 2).mean()).sqrt().item()
    assert err <= 1.05 * 2.0 ** -11 / np.sqrt(3.0)
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D,bar", [(64, 8, 8, 1, 1, 128, 1.6e-7), (64, 8, 8, 1, 1, 64, 1.2e-7), (4, 8, 8, 512, 512, 128, 2.2e-7),
                                                 (4, 8, 8, 512, 512, 64, 2.2e-7), (64, 8, 8, 1, 4096, 128, 3.8e-7)])
def test_scores_have_no_bias(tc, ctx, B, H, Hkv, Sq, Sk, D, bar):
    """The log-sum-exp against 64 bits over normal data.  Mean: fp32 multiply-adds have it below 6e-8; the scale of the
    scores is an fp32 number, which leaves up to 6e-8 of the scores (about one on average).  Root mean square: an fp32
    result's own rounding (2.7e-8 around 0.8, 1.4e-7 around 6, 2.8e-7 around 9) and about 1.5e-7 of the scores'."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(Sk)
    q, k, v = (torch.randn(B, h, s, D, device="cuda", generator=gen).half() for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
    o, lse = torch.zeros_like(q), torch.zeros(B, H, Sq, device="cuda")
    torch.cuda.synchronize()
    bufs = [ctx.buffer_from_ptr(t.data_ptr(), t.numel() * t.element_size()) for t in (q, k, v, o, lse)]
    tc.attention_forward(ctx, *bufs[:4], B, H, Sq, Sk, D, LSE=bufs[4], causal=False, kv_heads=Hkv)
    for b in bufs:
        b.close()
    want = torch.logsumexp(q.double() @ k.double().transpose(2, 3) / D ** 0.5, 3)
    err = lse.double() - want
    assert abs((err * want.sign()).mean().item()) <= 1.2e-7
    assert (err ** 2).mean().sqrt().item() <= bar


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D,causal,window", [
    (64, 8, 8, 1, 640, 128, False, 0), (37, 8, 2, 2, 1023, 128, True, 0), (20, 14, 2, 1, 2100, 64, False, 0), (20, 6, 3, 4, 1300, 128, False, 700),
    (70, 5, 1, 1, 4096, 64, False, 0), (10, 16, 8, 3, 257, 64, True, 0), (20, 48, 3, 1, 1500, 128, False, 0), (50, 8, 4, 1, 1, 128, False, 0)])
def test_chunks_merged_in_the_kernel(tc, ctx, B, H, Hkv, Sq, Sk, D, causal, window):
    """Up to 16 rows per K/V head: the chunks of a row's keys are merged by the kernel that has them, in one launch,
    to the same bits when captured.  Bars: one rounding of O, 2^-11 / sqrt(3) rms (a
    twentieth for small samples); the log-sum-exp as in test_scores_have_no_bias."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(Sk + H * Sq)
    q, k, v = (torch.randn(B, h, s, D, device="cuda", generator=gen).half() for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
    # another call's chunks, so that the captured one finds room for its own
    room = [ctx.buffer(64 * 64 * 64 * 256), ctx.buffer(8 * 16384 * 256)]
    tc.attention_forward(ctx, room[0], room[1], room[1], room[0], 1, 64, 64, 16384, 128, causal=False, kv_heads=8)
    for b in room:
        b.close()
    st = torch.cuda.Stream()
    torch.cuda.synchronize()
    outs = []
    for captured in (False, False, True):
        o, lse = torch.full_like(q, float("nan")), torch.full((B, H, Sq), float("nan"), device="cuda")
        torch.cuda.synchronize()
        d = tc.TCAttentionDesc(B, H, Sq, Sk, D, tc.TC_DTYPE_F16, tc.TC_DTYPE_F32, 0.0, causal, True, Hkv, window, None)

        def call():
            rc = tc.lib().tcx_raw_attention_forward(ctx.handle, ctypes.byref(d), *(ctypes.c_void_p(t.data_ptr()) for t in (q, k, v, o, lse)),
                                                    ctypes.c_void_p(st.cuda_stream))
            assert rc == 0
        if captured:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=st):
                call()
            with torch.cuda.stream(st):
                graph.replay()
        else:
            before = tc.launch_count()
            call()
            assert tc.launch_count() - before == 1 and tc.cuda_last_kernel_name() == "attention_mma_sm100"
        torch.cuda.synchronize()
        outs.append((o, lse))
    for o, lse in outs[1:]:
        assert torch.equal(o, outs[0][0]) and torch.equal(lse, outs[0][1])
    s = torch.matmul(q.double().view(B, Hkv, H // Hkv, Sq, D), k.double().unsqueeze(2).transpose(3, 4)) / D ** 0.5
    i, j = torch.arange(Sq, device="cuda")[:, None], torch.arange(Sk, device="cuda")[None, :]
    hidden = ((j > i) if causal else torch.zeros_like(j > i)) | ((i - j > window) if window else torch.zeros_like(j > i))
    s = s.masked_fill(hidden, float("-inf"))
    want = torch.matmul(torch.softmax(s, dim=4), v.double().unsqueeze(2)).reshape(B, H, Sq, D)
    o, lse = outs[0]
    assert ((o.double() - want).square().mean() / want.square().mean()).sqrt().item() <= 1.05 * 2.0 ** -11 / np.sqrt(3.0)
    assert (lse.double() - torch.logsumexp(s, 4).reshape(B, H, Sq)).square().mean().sqrt().item() <= 3.8e-7
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D,causal,off", [
    (5, 21, 3, 130, 300, 128, True, 0), (9, 15, 5, 77, 700, 64, False, 0), (2, 22, 2, 65, 2000, 128, False, 1), (37, 8, 8, 129, 260, 64, True, 3),
    (3, 39, 13, 200, 450, 128, True, 0), (40, 8, 8, 65, 300, 128, False, 0)])
def test_prefill_rows_of_odd_groups(tc, ctx, B, H, Hkv, Sq, Sk, D, causal, off):
    """The prefill kernel's rows - queries of 3 to 11 heads per K/V head, tiles that are not full, results `off` elements past a
    16-byte boundary, key chunks - against 64 bits; bars as in test_chunks_merged_in_the_kernel."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(Sk)
    q, k, v = (torch.randn(B, h, s, D, device="cuda", generator=gen).half() for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
    room = torch.full((q.numel() + 16,), float("nan"), device="cuda").half()
    o, lse = room[off:off + q.numel()].view(q.shape), torch.full((B, H, Sq), float("nan"), device="cuda")
    torch.cuda.synchronize()
    bufs = [ctx.buffer_from_ptr(t.data_ptr(), t.numel() * t.element_size()) for t in (q, k, v, o, lse)]
    tc.attention_forward(ctx, *bufs[:4], B, H, Sq, Sk, D, LSE=bufs[4], causal=causal, kv_heads=Hkv)
    assert tc.cuda_last_kernel_name() == "attention_prefill_tcgen05_sm100"
    for b in bufs:
        b.close()
    s = torch.matmul(q.double().view(B, Hkv, H // Hkv, Sq, D), k.double().unsqueeze(2).transpose(3, 4)) / D ** 0.5
    if causal:
        s = s.masked_fill(~torch.ones(Sq, Sk, dtype=torch.bool, device="cuda").tril(), float("-inf"))
    want = torch.matmul(torch.softmax(s, dim=4), v.double().unsqueeze(2)).reshape(B, H, Sq, D)
    assert ((o.double() - want).square().mean() / want.square().mean()).sqrt().item() <= 1.05 * 2.0 ** -11 / np.sqrt(3.0)
    assert (lse.double() - torch.logsumexp(s, 4).reshape(B, H, Sq)).square().mean().sqrt().item() <= 3.8e-7
    assert torch.isnan(room[off + q.numel():]).all() and torch.isnan(room[:off]).all()
    assert tc.take_device_error(ctx) == 0


@pytest.mark.parametrize("B,H,Hkv,Sq,Sk,D,causal,window,chunked", [
    (64, 8, 8, 1, 640, 128, False, 0, False), (37, 8, 2, 2, 1023, 128, True, 0, True), (20, 14, 2, 1, 2100, 64, False, 0, True),
    (20, 6, 3, 4, 1300, 128, False, 700, True), (70, 5, 1, 1, 4096, 64, False, 0, True), (20, 48, 3, 1, 1500, 128, False, 0, True),
    (1, 160, 16, 1, 456, 128, False, 0, True), (4, 72, 8, 1, 274, 128, False, 0, True), (22, 30, 2, 1, 700, 64, False, 0, True),
    (40, 1, 1, 1, 500, 128, False, 0, True), (13, 39, 3, 1, 1100, 128, False, 0, True), (2, 16, 8, 8, 377, 64, False, 0, True)])
def test_chunks_merged_in_the_kernel_in_other_forms(tc, ctx, B, H, Hkv, Sq, Sk, D, causal, window, chunked):
    """A captured call has room of its graph's and is the same one launch, whatever ran before; a call without scratch to hand
    chunks over in (an error is set) merges them in a launch of its own.  Both to the eager call's bits."""
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(Sk + H * Sq)
    q, k, v = (torch.randn(B, h, s, D, device="cuda", generator=gen).half() for h, s in ((H, Sq), (Hkv, Sk), (Hkv, Sk)))
    st = torch.cuda.Stream()
    d = tc.TCAttentionDesc(B, H, Sq, Sk, D, tc.TC_DTYPE_F16, tc.TC_DTYPE_F32, 0.0, causal, True, Hkv, window, None)
    outs = []
    for form in ("captured", "eager", "without"):
        o, lse = torch.full_like(q, float("nan")), torch.full((B, H, Sq), float("nan"), device="cuda")
        torch.cuda.synchronize()

        def call():
            rc = tc.lib().tcx_raw_attention_forward(ctx.handle, ctypes.byref(d), *(ctypes.c_void_p(t.data_ptr()) for t in (q, k, v, o, lse)),
                                                    ctypes.c_void_p(st.cuda_stream))
            assert rc == 0
        before = tc.launch_count()
        if form == "captured":
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=st):
                call()
            with torch.cuda.stream(st):
                graph.replay()
        elif form == "without":
            tc.set_device_error(ctx, 1)
            call()
            assert tc.take_device_error(ctx) == 1
        else:
            call()
        assert tc.launch_count() - before == (2 if form == "without" and chunked else 1) and tc.cuda_last_kernel_name() == "attention_mma_sm100"
        torch.cuda.synchronize()
        outs.append((o, lse))
    for o, lse in outs[1:]:
        assert torch.equal(o, outs[0][0]) and torch.equal(lse, outs[0][1])
    assert not torch.isnan(outs[0][0]).any() and tc.take_device_error(ctx) == 0
