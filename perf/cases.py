"""The work a user of this library has it do, as measurable cases.

Every case goes through the public entry points of the `tensorcore_b200` binding: the reference's
synchronous calls on buffers, the raw-pointer calls on a CUDA stream, and the decode session of
`tensorcore_b200.decode`.  Weights are N(0, 0.02^2) in Q4_0 / Q8_0 blocks (or fp16 for the dense
operations), activations N(0, 1), norm weights 1 + N(0, 0.1^2).

listed()          the cases; draw(rng) one more of the same ranges
prepare / run     what a program has in hand before a call, and one pass
work / tolerance  bytes and operations a pass cannot do without; agreed accuracy
exact             the same results in 64-bit torch, without this library
"""
import math

import torch

import tensorcore_b200 as tc
from tensorcore_b200 import decode

BLOCK = {"q4_0": 18, "q8_0": 34}
EPS = 1e-5


# ---- the cases -----------------------------------------------------------------------------------
def listed():
    return [
        # One key projection of a grouped-query model, as the reference's synchronous call: the smallest
        # call a decode loop makes, where launch and wait count.
        dict(name="gemv_q4_kv_proj_m1", op="gemv", api="sync", fmt="q4_0", M=1, N=1024, K=8192, x="f16", y="f16", fused=False),
        # Norm and gate projection of a 7B layer in Q8_0, one row (single-sequence decode).
        dict(name="rmsnorm_gemv_q8_ffn_m1", op="gemv", api="sync", fmt="q8_0", M=1, N=11008, K=4096, x="f16", y="f16", fused=True),
        # fp32 activations and results over a matrix whose sizes are no multiples of anything but a block.
        dict(name="gemv_q8_f32_ragged_m3", op="gemv", api="raw", fmt="q8_0", M=3, N=5003, K=4128, x="f32", y="f32", fused=False),
        # A whole decode step of one sequence: every projection of a 7B model in Q4_0 (32 layers + head).
        dict(name="decode_token_q4_7b", op="session", fmt="q4_0", M=1, layers=32, d=4096, ff=11008, kv=4096, vocab=32000),
        # The same for eight sequences together, four layers and the head of the 7B shape.
        dict(name="decode_step_q4_b8", op="session", fmt="q4_0", M=8, layers=4, d=4096, ff=11008, kv=4096, vocab=32000),
        # One large projection for 32 sequences (a server's decode batch).
        dict(name="gemv_q4_batch_m32", op="gemv", api="raw", fmt="q4_0", M=32, N=28672, K=4096, x="f16", y="f16", fused=False),
        # The same in Q8_0 with the norm in front, 16 sequences.
        dict(name="rmsnorm_gemv_q8_batch_m16", op="gemv", api="raw", fmt="q8_0", M=16, N=11008, K=4096, x="f16", y="f16", fused=True),
        # A prefill block of 512 rows through norm + gate projection of an 8B-sized layer.
        dict(name="prefill_rmsnorm_q4_m512", op="gemv", api="raw", fmt="q4_0", M=512, N=14336, K=4096, x="f16", y="f16", fused=True),
        # Norm + dense fp16 projection, one row.
        dict(name="dense_rmsnorm_gemv_m1", op="dense", norm="rms", M=1, N=11008, K=4096),
        # Attention of a decode step: eight sequences, grouped-query heads, 4096 cached keys.
        dict(name="attention_decode_b8_gqa", op="attn", B=8, H=32, Hkv=8, Sq=1, Sk=4096, D=128, causal=False, lse=False),
        # Attention of the 512-row prefill block (causal), with the log-sum-exp.
        dict(name="attention_prefill_512", op="attn", B=1, H=32, Hkv=8, Sq=512, Sk=512, D=128, causal=True, lse=True),
        # Dense fp16 product of a prefill block with a transposed weight matrix.
        dict(name="gemm_f16_prefill", op="gemm", dtype="f16", M=512, N=11008, K=4096, ta=False, tb=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _mult(v, m):
    return max(m, int(round(v / m)) * m)


def draw(rng):
    kind = rng.choice(["one", "one", "ragged", "token", "step", "batch", "batch", "prefill", "dense", "decode_attn",
                       "prefill_attn", "gemm"])
    fmt = rng.choice(["q4_0", "q8_0"])
    if kind == "one":
        return dict(op="gemv", api=rng.choice(["sync", "raw"]), fmt=fmt, M=rng.choice([1, 1, 1, 2, 3, 4]), N=_log(rng, 256, 32000),
                    K=_mult(_log(rng, 512, 14336), 256), x="f16", y="f16", fused=rng.random() < 0.5)
    if kind == "ragged":
        f32 = rng.random() < 0.5
        return dict(op="gemv", api="raw", fmt=fmt, M=rng.randint(1, 4), N=_log(rng, 100, 8000), K=32 * _log(rng, 9, 260),
                    x="f32" if f32 else "f16", y="f32" if f32 else "f16", fused=rng.random() < 0.5)
    if kind in ("token", "step"):
        d = _mult(_log(rng, 1024, 8192), 256)
        ff = _mult(d * rng.uniform(2.5, 3.5), 256)
        kv = _mult(d // rng.choice([1, 2, 4, 8]), 128)
        vocab = _log(rng, 4000, 128256)
        per_layer = (2 * d * d + 2 * d * kv + 3 * d * ff) * 18 / 32
        top = 32 if kind == "token" else 6
        M = 1 if kind == "token" else _log(rng, 2, 16)
        layers = max(1, min(top, int(2.4e9 / per_layer / math.sqrt(M))))
        return dict(op="session", fmt="q4_0", M=M, layers=rng.randint(1, layers), d=d,
                    ff=ff, kv=kv, vocab=vocab)
    if kind == "batch":
        return dict(op="gemv", api=rng.choice(["sync", "raw"]), fmt=fmt, M=_log(rng, 5, 64), N=_log(rng, 1024, 28672),
                    K=_mult(_log(rng, 2048, 14336), 256), x="f16", y="f16", fused=rng.random() < 0.5)
    if kind == "prefill":
        N, K = _log(rng, 1024, 14336), _mult(_log(rng, 2048, 8192), 256)
        return dict(op="gemv", api="raw", fmt=fmt, M=_log(rng, 65, min(1024, 512 * 14336 * 4096 // (N * K))), N=N, K=K, x="f16", y="f16",
                    fused=rng.random() < 0.5)
    if kind == "dense":
        return dict(op="dense", norm=rng.choice(["rms", "layer"]), M=rng.choice([1, 1, 2, 4, _log(rng, 5, 32)]),
                    N=_mult(_log(rng, 1024, 16384), 8), K=_mult(_log(rng, 1024, 8192), 8))
    if kind == "decode_attn":
        hkv = rng.choice([1, 2, 4, 8])
        return dict(op="attn", B=_log(rng, 1, 16), H=hkv * rng.choice([1, 2, 4, 8]), Hkv=hkv, Sq=1, Sk=_log(rng, 64, 8192),
                    D=rng.choice([64, 128, 128]), causal=False, lse=rng.random() < 0.5)
    if kind == "prefill_attn":
        hkv, rep, b = rng.choice([2, 4, 8]), rng.choice([1, 2, 4]), rng.choice([1, 2])
        s = _log(rng, 48, min(1024, int(512 * math.sqrt(32 / (b * hkv * rep)))))
        return dict(op="attn", B=b, H=hkv * rep, Hkv=hkv, Sq=s, Sk=s, D=rng.choice([64, 128, 128]),
                    causal=rng.random() < 0.8, lse=rng.random() < 0.5)
    N, K = _mult(_log(rng, 512, 12288), 8), _mult(_log(rng, 512, 8192), 8)
    return dict(op="gemm", dtype=rng.choice(["f16", "f16", "bf16"]), M=_mult(_log(rng, 8, min(2048, 512 * 11008 * 4096 // (N * K))), 8), N=N,
                K=K, ta=rng.random() < 0.2, tb=rng.random() < 0.6)


# ---- data ----------------------------------------------------------------------------------------
_ctx = None


def _context():
    global _ctx
    if _ctx is None:
        _ctx = tc.Context()
    return _ctx


def _gen(seed, what):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 1000003 + what)
    return g


def _normal(shape, g, scale=1.0, mean=0.0, dtype=torch.float32):
    t = torch.empty(shape, dtype=torch.float32, device="cuda")
    t.normal_(mean, scale, generator=g)
    return t.to(dtype)


def _quant_rows(w, fmt):
    """fp32 [rows, K] to GGUF blocks, uint8 [rows, K / 32, block bytes]."""
    b = w.view(w.shape[0], -1, 32)
    if fmt == "q4_0":
        hi, lo = b.amax(dim=2), b.amin(dim=2)
        d = (torch.where(hi > -lo, hi, lo) / -8.0).to(torch.float16)
        df = d.float().unsqueeze(2)
        q = torch.where(df != 0, b / df, torch.zeros_like(b)).add_(8.5).floor_().clamp_(0, 15).to(torch.uint8)
        qs = q[:, :, :16] | (q[:, :, 16:] << 4)
    else:
        d = (b.abs().amax(dim=2) / 127.0).to(torch.float16)
        df = d.float().unsqueeze(2)
        qs = torch.where(df != 0, b / df, torch.zeros_like(b)).round_().clamp_(-127, 127).to(torch.int8).view(torch.uint8)
    return torch.cat([d.unsqueeze(2).view(torch.uint8), qs], dim=2)


def _weights(N, K, fmt, g):
    out = torch.empty((N, K // 32, BLOCK[fmt]), dtype=torch.uint8, device="cuda")
    step = max(1, (1 << 25) // K)
    for r in range(0, N, step):
        n = min(step, N - r)
        out[r:r + n] = _quant_rows(_normal((n, K), g, 0.02), fmt)
    return out


def _dequant64(w, fmt):
    N, nb, _ = w.shape
    d = w[:, :, :2].contiguous().view(torch.float16).double()
    qs = w[:, :, 2:]
    if fmt == "q4_0":
        q = torch.cat([qs & 15, qs >> 4], dim=2).double() - 8.0
    else:
        q = qs.contiguous().view(torch.int8).double()
    return (q * d).reshape(N, nb * 32)


def _times64(x, w, fmt):
    """x [M, K] double times dequantised w, in row pieces."""
    N, K = w.shape[0], w.shape[1] * 32
    step = max(1, (1 << 27) // K)
    return torch.cat([x @ _dequant64(w[r:r + step], fmt).t() for r in range(0, N, step)], dim=1)


def _rms64(x, gamma):
    return x * torch.rsqrt((x * x).mean(dim=1, keepdim=True) + EPS) * gamma


def _gemv_data(c, seed):
    dt = torch.float32 if c["x"] == "f32" else torch.float16
    return (_normal((c["M"], c["K"]), _gen(seed, 1), dtype=dt), _normal((c["K"],), _gen(seed, 2), 0.1, 1.0, dt),
            _weights(c["N"], c["K"], c["fmt"], _gen(seed, 3)))


def _session_data(c, seed):
    """Input rows, norm weights and projections of a whole model, named as decode.Model asks for them."""
    s = decode.LlamaShape("case", c["layers"], c["d"], c["ff"], c["d"] // 128, c["kv"] // 128, c["vocab"])
    t, g = {}, _gen(seed, 5)
    for l in range(s.n_layers):
        for p in decode.PROJ:
            if p in ("attn_k", "attn_v"):
                n, k = c["kv"], c["d"]
            else:
                n, k = s.proj_shape(p)
            t["blk.%d.%s.weight" % (l, p)] = _weights(n, k, c["fmt"], g)
        t["blk.%d.attn_norm.weight" % l] = _normal((c["d"],), g, 0.1, 1.0, torch.float16)
        t["blk.%d.ffn_norm.weight" % l] = _normal((c["d"],), g, 0.1, 1.0, torch.float16)
    t["output_norm.weight"] = _normal((c["d"],), g, 0.1, 1.0, torch.float16)
    t["output.weight"] = _weights(c["vocab"], c["d"], c["fmt"], g)
    return s, t, _normal((c["M"], c["d"]), _gen(seed, 6), dtype=torch.float16)


def _dense_data(c, seed):
    h = torch.float16
    return (_normal((c["M"], c["K"]), _gen(seed, 1), dtype=h), _normal((c["K"],), _gen(seed, 2), 0.1, 1.0, h),
            _normal((c["K"],), _gen(seed, 4), 0.1, 0.0, h), _normal((c["K"], c["N"]), _gen(seed, 3), 0.02, dtype=h))


def _attn_data(c, seed):
    h = torch.float16
    return (_normal((c["B"], c["H"], c["Sq"], c["D"]), _gen(seed, 1), dtype=h),
            _normal((c["B"], c["Hkv"], c["Sk"], c["D"]), _gen(seed, 2), dtype=h),
            _normal((c["B"], c["Hkv"], c["Sk"], c["D"]), _gen(seed, 3), dtype=h))


def _gemm_data(c, seed):
    dt = torch.float16 if c["dtype"] == "f16" else torch.bfloat16
    sa = (c["K"], c["M"]) if c["ta"] else (c["M"], c["K"])
    sb = (c["N"], c["K"]) if c["tb"] else (c["K"], c["N"])
    return _normal(sa, _gen(seed, 1), dtype=dt), _normal(sb, _gen(seed, 2), 0.02, dtype=dt)


# ---- what a program holds, and a pass ---------------------------------------------------------------
def _wrap(t):
    """A tc_buffer over a torch tensor's memory (used in place)."""
    return _context().buffer_from_ptr(t.data_ptr(), t.numel() * t.element_size())


class _Owner:
    """A decode session and what its buffers lie in; closed when nothing refers to it any more."""

    def __init__(self, c, seed):
        ctx = _context()
        shape, self.tensors, x = _session_data(c, seed)
        self.bufs = {k: _wrap(v) for k, v in self.tensors.items()}
        self.model = decode.Model(shape, tc.TC_QUANT_Q4_0, lambda n: self.bufs[n].handle.value)
        torch.cuda.synchronize()
        self.session = decode.DecodeSession(ctx, self.model, c["M"])
        self.session.x.upload(x.cpu().numpy())

    def __del__(self):
        if getattr(self, "session", None) is not None:
            torch.cuda.synchronize()     # nothing reads the session's buffers any more
            self.session.close()
            for b in self.bufs.values():
                b.close()


class _View:
    """A session's fp16 buffer as torch sees it; keeps the session."""

    def __init__(self, owner, buf, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (buf.device_ptr(), False), "shape": shape, "typestr": "<f2", "version": 3}


class _Session:
    """A decode session and its results (logits, last hidden rows) as torch tensors."""

    def __init__(self, c, seed):
        self.owner = _Owner(c, seed)
        self.session = self.owner.session
        last = self.session.hidden((c["layers"] - 1) & 1)
        self.out = [torch.as_tensor(_View(self.owner, b, s), device="cuda") for b, s in
                    ((self.session.logits, (c["M"], c["vocab"])), (last, (c["M"], c["d"])))]


class _Plain:
    """Tensors of a single call and the buffers that wrap them."""

    def __init__(self, **tensors):
        self.t = tensors
        self.b = {k: _wrap(v) for k, v in tensors.items()}

    def __del__(self):
        for b in getattr(self, "b", {}).values():
            b.close()


def prepare(case, seed):
    c = case
    if c["op"] == "session":
        return dict(c=c, s=_Session(c, seed))
    if c["op"] == "gemv":
        x, gamma, w = _gemv_data(c, seed)
        y = torch.zeros((c["M"], c["N"]), dtype=x.dtype if c["y"] == c["x"] else torch.float32, device="cuda")
        return dict(c=c, s=_Plain(x=x, gamma=gamma, w=w, y=y))
    if c["op"] == "dense":
        x, gamma, beta, w = _dense_data(c, seed)
        return dict(c=c, s=_Plain(x=x, gamma=gamma, beta=beta, w=w, y=torch.zeros((c["M"], c["N"]), dtype=torch.float16, device="cuda")))
    if c["op"] == "attn":
        q, k, v = _attn_data(c, seed)
        return dict(c=c, s=_Plain(q=q, k=k, v=v, o=torch.zeros_like(q),
                                  lse=torch.zeros((c["B"], c["H"], c["Sq"]), dtype=torch.float32, device="cuda")))
    a, b = _gemm_data(c, seed)
    return dict(c=c, s=_Plain(a=a, b=b, y=torch.zeros((c["M"], c["N"]), dtype=a.dtype, device="cuda")))


def run(state):
    c, s, ctx = state["c"], state["s"], _ctx
    if c["op"] == "session":
        s.session.run(1)
        return s.out
    if c["op"] == "gemv":
        if c["api"] == "raw":
            t, st = s.t, torch.cuda.current_stream().cuda_stream
            if c["fused"]:
                tc.raw_fused_rmsnorm_gemv_quantized(ctx, t["x"].data_ptr(), t["gamma"].data_ptr(), t["w"].data_ptr(), t["y"].data_ptr(),
                                                    c["fmt"], c["M"], c["N"], c["K"], EPS, c["x"], c["y"], st)
            else:
                tc.raw_gemv_quantized(ctx, t["x"].data_ptr(), t["w"].data_ptr(), t["y"].data_ptr(), c["fmt"], c["M"], c["N"], c["K"],
                                      c["x"], c["y"], st)
        elif c["fused"]:
            tc.fused_rmsnorm_gemv_quantized(ctx, s.b["x"], s.b["gamma"], s.b["w"], s.b["y"], c["fmt"], c["M"], c["N"], c["K"], EPS)
        else:
            tc.gemv_quantized(ctx, s.b["x"], s.b["w"], s.b["y"], c["fmt"], c["M"], c["N"], c["K"])
        return s.t["y"]
    if c["op"] == "dense":
        if c["norm"] == "rms":
            tc.fused_rmsnorm_gemv(ctx, s.b["x"], s.b["gamma"], s.b["w"], s.b["y"], c["M"], c["N"], c["K"], EPS)
        else:
            tc.fused_layernorm_gemv(ctx, s.b["x"], s.b["gamma"], s.b["beta"], s.b["w"], s.b["y"], c["M"], c["N"], c["K"], EPS)
        return s.t["y"]
    if c["op"] == "attn":
        tc.attention_forward(ctx, s.b["q"], s.b["k"], s.b["v"], s.b["o"], c["B"], c["H"], c["Sq"], c["Sk"], c["D"],
                             LSE=s.b["lse"] if c["lse"] else None, causal=c["causal"], kv_heads=c["Hkv"])
        return [s.t["o"], s.t["lse"]] if c["lse"] else s.t["o"]
    tc.gemm(ctx, s.b["a"], s.b["b"], s.b["y"], c["M"], c["N"], c["K"], dtype=c["dtype"], transpose_a=c["ta"], transpose_b=c["tb"])
    return s.t["y"]


# ---- what it costs at least, and how close results agree ---------------------------------------------
def work(case):
    c = case
    if c["op"] == "gemv":
        xs, ys = (4 if c["x"] == "f32" else 2), (4 if c["y"] == "f32" else 2)
        return {"bytes": c["N"] * (c["K"] // 32) * BLOCK[c["fmt"]] + c["M"] * (c["K"] * xs + c["N"] * ys) + (c["K"] * xs if c["fused"] else 0),
                "flops": 2 * c["M"] * c["N"] * c["K"]}
    if c["op"] == "session":
        d, ff, kv, L = c["d"], c["ff"], c["kv"], c["layers"]
        w = L * (2 * d * d + 2 * d * kv + 3 * d * ff) + c["vocab"] * d
        return {"bytes": w // 32 * BLOCK[c["fmt"]] + c["M"] * (d + c["vocab"]) * 2 + (2 * L + 1) * d * 2, "flops": 2 * c["M"] * w}
    if c["op"] == "dense":
        return {"bytes": 2 * (c["K"] * c["N"] + c["M"] * (c["K"] + c["N"]) + c["K"] * (1 if c["norm"] == "rms" else 2)),
                "flops": 2 * c["M"] * c["N"] * c["K"]}
    if c["op"] == "attn":
        pairs = sum(min(i + 1, c["Sk"]) for i in range(c["Sq"])) if c["causal"] else c["Sq"] * c["Sk"]
        return {"bytes": 2 * c["D"] * (2 * c["B"] * c["H"] * c["Sq"] + 2 * c["B"] * c["Hkv"] * c["Sk"]) + (4 * c["B"] * c["H"] * c["Sq"] if c["lse"] else 0),
                "flops": 4 * c["B"] * c["H"] * pairs * c["D"]}
    return {"bytes": 2 * (c["M"] * c["K"] + c["K"] * c["N"] + c["M"] * c["N"]), "flops": 2 * c["M"] * c["N"] * c["K"]}


def tolerance(case):
    c = case
    if c["op"] == "session":
        return {"rel": 1.5e-2}       # several hundred dependent fp16 results
    if c["op"] == "gemv" and c["x"] == "f32":
        return {"rel": 2e-4}
    if c["op"] == "gemm" and c["dtype"] == "bf16":
        return {"rel": 7e-3}
    return {"rel": 1.2e-3}           # fp16 results, weights or normalised rows rounded to fp16


def exact(case, seed):
    c = case
    if c["op"] == "gemv":
        x, gamma, w = _gemv_data(c, seed)
        x = x.double()
        return _times64(_rms64(x, gamma.double()) if c["fused"] else x, w, c["fmt"])
    if c["op"] == "session":
        _, t, h = _session_data(c, seed)
        h = h.double()
        f = c["fmt"]
        for l in range(c["layers"]):
            p = "blk.%d." % l
            q = _times64(_rms64(h, t[p + "attn_norm.weight"].double()), t[p + "attn_q.weight"], f)
            o = _times64(q, t[p + "attn_output.weight"], f)
            gate = _times64(_rms64(o, t[p + "ffn_norm.weight"].double()), t[p + "ffn_gate.weight"], f)
            h = _times64(gate, t[p + "ffn_down.weight"], f)
        return [_times64(_rms64(h, t["output_norm.weight"].double()), t["output.weight"], f), h]
    if c["op"] == "dense":
        x, gamma, beta, w = (v.double() for v in _dense_data(c, seed))
        if c["norm"] == "rms":
            return _rms64(x, gamma) @ w
        x = x - x.mean(dim=1, keepdim=True)
        return (x * torch.rsqrt((x * x).mean(dim=1, keepdim=True) + EPS) * gamma + beta) @ w
    if c["op"] == "attn":
        q, k, v = (t.double() for t in _attn_data(c, seed))
        rep = c["H"] // c["Hkv"]
        o, lse = [], []
        for b in range(c["B"]):
            s = torch.matmul(q[b].view(c["Hkv"], rep, c["Sq"], c["D"]), k[b].unsqueeze(1).transpose(2, 3)) / math.sqrt(c["D"])
            if c["causal"]:
                keep = torch.ones((c["Sq"], c["Sk"]), dtype=torch.bool, device=s.device).tril()
                s = s.masked_fill(~keep, float("-inf"))
            m = torch.logsumexp(s, dim=3, keepdim=True)
            o.append(torch.matmul(torch.exp(s - m), v[b].unsqueeze(1)).reshape(c["H"], c["Sq"], c["D"]))
            lse.append(m.reshape(c["H"], c["Sq"]))
        return [torch.stack(o), torch.stack(lse)] if c["lse"] else torch.stack(o)
    a, b = (t.double() for t in _gemm_data(c, seed))
    return (a.t() if c["ta"] else a) @ (b.t() if c["tb"] else b)
