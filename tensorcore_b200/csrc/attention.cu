// Scaled-dot-product attention forward.
//
// Interface replaced: tc_attention_forward (include/tensorcore/attention.h:24-60; arithmetic of
// lib/ops/attention_cpu.cpp:131-277): fp16 Q [B,H,Sq,D], K/V [B,Hkv,Sk,D], O [B,H,Sq,D], optional
// fp32 LSE [B,H,Sq]; softmax in fp32; causal mask (key index > query index), sliding window
// (query - key > window), ALiBi (score -= slope * (query - key)), grouped-query heads.
//
//   * head_dim 64 and 128, Q, K and V 16-byte aligned: tensor cores, attention_mma_kernel below for a decode
//     step or a small block and attention_tc.cu for a prefill block (prefill_block below).
//   * Other head_dims and addresses: attention_decode_kernel, a streaming pass per query row on the CUDA
//     cores.  A lane takes a key for the scores (the query rows in shared memory), then the lanes
//     switch to a slice of D each and walk the step's 32 value rows, eight row loads in flight at a
//     time, the probabilities broadcast by shuffle; two query heads that share a K/V head go together.
//   * A row's keys are cut into chunks when there are too few CTAs otherwise.  A CTA keeps an
//     online-softmax state (running maximum m, denominator l, unnormalised output o[D]) for its chunk;
//     with one chunk it writes O (and LSE) itself, else it leaves (m, l, o) in scratch and a second
//     small kernel merges the chunks.
#include "attention_math.cuh"
#include "handover.cuh"
#include "kernels.h"

#include <cuda_fp16.h>
#include <cstdint>

namespace tcb {
namespace {

using namespace attn;

constexpr int kAttnWarps = 4;
constexpr int kAttnMaxD = 128;

__device__ __forceinline__ float warp_max(float v) {
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sum(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Any head_dim up to 128.  G: query heads per CTA.
template <int G>
__global__ void __launch_bounds__(kAttnWarps * 32) attention_decode_kernel(const AttnParams p) {
    // the merge kernel that follows may be set up now; it waits for this grid before it reads anything
    asm volatile("griddepcontrol.launch_dependents;");
    constexpr int kPer = kAttnMaxD / 32;                     // output elements per lane
    __shared__ float q_s[G][kAttnMaxD];
    __shared__ float o_s[kAttnWarps][G][kAttnMaxD];
    __shared__ float m_s[kAttnWarps][G], l_s[kAttnWarps][G];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int D = p.D;
    // blockIdx.x = ((b * heads_per_grid) + hg) * Sq + i, where hg counts groups of G query heads
    const int groups = p.Hq / G;
    const int i = blockIdx.x % p.Sq, bg = blockIdx.x / p.Sq, hg = bg % groups, b = bg / groups;
    const int h0 = hg * G;                                   // first query head of the group
    const int hkv = h0 / (p.Hq / p.Hkv);
    const int chunk = blockIdx.y;
    const __half* Kh = p.K + (static_cast<size_t>(b) * p.Hkv + hkv) * p.Sk * D;
    const __half* Vh = p.V + (static_cast<size_t>(b) * p.Hkv + hkv) * p.Sk * D;
    for (int t = tid; t < G * D; t += blockDim.x) {
        const int g = t / D, d = t - g * D;
        q_s[g][d] = __half2float(p.Q[((static_cast<size_t>(b) * p.Hq + h0 + g) * p.Sq + i) * D + d]);
    }
    __syncthreads();
    float slope[G];
#pragma unroll
    for (int g = 0; g < G; ++g) slope[g] = p.slopes ? p.slopes[h0 + g] : 0.f;
    const int k0 = chunk * p.keys_per_chunk, k1 = min(p.Sk, k0 + p.keys_per_chunk);

    // this lane's slice of the output: `per` consecutive elements when D is a multiple of 32 (one
    // vector load per value row), else elements lane, lane + 32, ...
    const int per = (D & 31) == 0 && p.v_vec ? D >> 5 : 0;
    auto elem = [&](int t) { return per ? lane * per + t : lane + 32 * t; };
    float o[G][kPer];
    float m[G], l[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        m[g] = -INFINITY;
        l[g] = 0.f;
#pragma unroll
        for (int t = 0; t < kPer; ++t) o[g][t] = 0.f;
    }
    for (int j0 = k0 + warp * 32; j0 < k1; j0 += kAttnWarps * 32) {
        const int j = j0 + lane;
        float s[G];
#pragma unroll
        for (int g = 0; g < G; ++g) s[g] = -INFINITY;
        if (j < k1) {
            const __half* kr = Kh + static_cast<size_t>(j) * D;
            float acc[G];
#pragma unroll
            for (int g = 0; g < G; ++g) acc[g] = 0.f;
            {
                for (int d = 0; d < D; ++d) {
                    const float kv = __half2float(kr[d]);
#pragma unroll
                    for (int g = 0; g < G; ++g) acc[g] = fmaf(q_s[g][d], kv, acc[g]);
                }
            }
#pragma unroll
            for (int g = 0; g < G; ++g) {
                float sc = acc[g] * p.scale;
                if (p.causal && j > i) sc = -INFINITY;
                if (p.window > 0 && i - j > p.window) sc = -INFINITY;
                if (p.slopes) sc -= slope[g] * static_cast<float>(i - j);
                s[g] = sc;
            }
        }
        float pj[G];
        bool any = false;
#pragma unroll
        for (int g = 0; g < G; ++g) {
            const float m_new = fmaxf(m[g], warp_max(s[g]));
            pj[g] = 0.f;
            if (m_new > -INFINITY) {                          // else everything so far is masked
                const float keep = m[g] > -INFINITY ? __expf(m[g] - m_new) : 0.f;
                if (s[g] > -INFINITY) pj[g] = __expf(s[g] - m_new);
                l[g] = l[g] * keep + warp_sum(pj[g]);
#pragma unroll
                for (int t = 0; t < kPer; ++t) o[g][t] *= keep;
                m[g] = m_new;
                any = true;
            }
        }
        if (!any) continue;                                   // warp-uniform
        const int n = min(32, k1 - j0);
        constexpr int kRows = 8;                              // value rows in flight
        for (int c0 = 0; c0 < n; c0 += kRows) {
            float v[kRows][kPer];
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                const int c = c0 + r;
                const __half* vr = Vh + static_cast<size_t>(j0 + (c < n ? c : n - 1)) * D;
                if (per == 4) {
                    const uint2 raw = __ldg(reinterpret_cast<const uint2*>(vr + 4 * lane));
                    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&raw.x));
                    const float2 bq = __half22float2(*reinterpret_cast<const __half2*>(&raw.y));
                    v[r][0] = a.x; v[r][1] = a.y; v[r][2] = bq.x; v[r][3] = bq.y;
                } else if (per == 2) {
                    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(vr + 2 * lane));
                    v[r][0] = a.x; v[r][1] = a.y;
                } else {
#pragma unroll
                    for (int t = 0; t < kPer; ++t) {
                        const int d = elem(t);
                        v[r][t] = (d < D && (per == 0 || t < per)) ? __half2float(vr[d]) : 0.f;
                    }
                }
            }
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                const int c = c0 + r;
                if (c >= n) break;
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const float pc = __shfl_sync(0xffffffffu, pj[g], c);
#pragma unroll
                    for (int t = 0; t < kPer; ++t) o[g][t] = fmaf(pc, v[r][t], o[g][t]);
                }
            }
        }
    }
    // merge the CTA's warps
#pragma unroll
    for (int g = 0; g < G; ++g) {
        if (lane == 0) { m_s[warp][g] = m[g]; l_s[warp][g] = l[g]; }
#pragma unroll
        for (int t = 0; t < kPer; ++t) {
            const int d = elem(t);
            if (d < D && (per == 0 || t < per)) o_s[warp][g][d] = o[g][t];
        }
    }
    __syncthreads();
    for (int t = tid; t < G * D; t += blockDim.x) {
        const int g = t / D, d = t - g * D;
        float mm = -INFINITY;
        for (int w = 0; w < kAttnWarps; ++w) mm = fmaxf(mm, m_s[w][g]);
        float ll = 0.f, acc = 0.f;
        for (int w = 0; w < kAttnWarps; ++w) {
            if (m_s[w][g] > -INFINITY) {
                const float e = __expf(m_s[w][g] - mm);
                ll += l_s[w][g] * e;
                acc += o_s[w][g][d] * e;
            }
        }
        const size_t row = (static_cast<size_t>(b) * p.Hq + h0 + g) * p.Sq + i;
        if (p.chunks == 1) {
            p.O[row * D + d] = __float2half_rn(ll != 0.f ? acc / ll : 0.f);
            if (d == 0 && p.LSE) p.LSE[row] = mm + logf(fmaxf(ll, 1e-30f));
        } else {
            float* dst = p.part + (row * p.chunks + chunk) * (D + 2);
            dst[2 + d] = acc;
            if (d == 0) { dst[0] = mm; dst[1] = ll; }
        }
    }
}

// ---------------------------------------------------------------------------------------
// Matrix kernel, head_dim 64 and 128: scores and outputs on the tensor cores (mma.sync m16n8k16).
//
// For decode steps and small blocks: up to 64 (query, head) pairs that share a K/V head, head fastest, are one
// tile, so the heads of a grouped-query decode step read the cache once.  K and V arrive in steps of 64 keys through a ring in shared memory
// (cp.async, 16-byte pieces, piece index XORed with the row so that ldmatrix is conflict-free).
//   SPLIT_KEYS (9 to 16 rows; attention_mma8_kernel below for up to 8): all four warps hold the same rows and take 16 keys of a step each,
//     with softmax states of their own that are merged at the end (a thread per row for the weights, then four
//     elements a thread at a time: 16 x 16, 8 heads 19.1 us a call with a division and a branch per element).
//   else: a warp owns 16 of the 64 rows and takes all 64 keys.
// The scores' products are exact and summed in fp32.  The probabilities are fp32 numbers; for the product with V
// each is split into two fp16 numbers (attention_math.cuh says to how many bits), which costs a third
// more MMAs and keeps the result as close to a 64-bit one as fp32 multiply-adds had it.
// A decode step is bound by the cache stream; two CTAs per SM overlap the chains of their steps (scores,
// maximum, exponentials, outputs).
// ---------------------------------------------------------------------------------------
constexpr int kStepKeys = 64;
constexpr int kMergeMaxChunks = 128;
constexpr int kMergeHere = 8;          // chunks that the attention kernel can merge itself
constexpr int kMmaRows = 64;           // rows (query, head) of a tile

// Words of a chunk's states for R rows that another CTA merges: sums, then maximum and sum of each row; in 16 bytes.
__host__ __device__ constexpr int attention_state_words(int R, int D) { return R * D + ((2 * R + 3) & ~3); }

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Partial softmax states that a CTA leaves for the one that merges its row (handover.cuh).
__device__ __forceinline__ void state_store4(uint32_t* dst, float4 v) {
    using handover::word_of;
    handover::store4(dst, make_uint4(word_of(v.x), word_of(v.y), word_of(v.z), word_of(v.w)));
}
// An 8 x 8 matrix of 16-bit elements, a thread's two those of row lane / 4, transposed.
__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
    uint32_t r;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
    return r;
}
template <int D> struct MmaShape {
    static constexpr int kStages = D == 128 ? 3 : 4;
    static constexpr int kStageBytes = 2 * kStepKeys * D * 2;
    static constexpr int kSmem = kStages * kStageBytes;
};

// The end of the kernels whose warps split the keys of a step (ROWS rows): o_s has each warp's outputs, rows STRIDE
// elements apart, ml_s its maximum and sum per row, both in the ring, which everybody has finished reading.
// HERE: the chunks' states - sums, then maximum and sum per row - go to the CTA of the last chunk, which started last, and
// it merges them: all words it needs are asked for at a time, however many elements a thread has, and the weights are
// worked out once per row.  (With a trip for every four elements of a thread, and maximum and sum beside them, 16 rows
// of head_dim 128 took up to 4 us longer than with a merge launch.  Raw calls back to back, merge launch / that / this: 18
// sequences, 64 heads on 4 x 527 keys 14.5 / 16.6 / 14.4 us, 6 sequences, 256 on 16 x 2338 27.9 / 30.0 / 27.2, head_dim 64,
// 39 sequences, 24 on 8, four queries x 1624 35.0 / 33.0 / 31.1, 160 on 16 x 456, eight chunks of a step, 8.4 / 12.5 / 10.4.)
// Calls whose chunks are not merged here run an instance without that code, which cost them up to 1 us.
template <int D, int ROWS, int STRIDE, bool HERE>
__device__ __forceinline__ void merge_warps(const AttnParams& p, float* o_s, float* ml_s, int R, int G, int b, int hkv, int bk, int chunk) {
    const int tid = threadIdx.x;
    float* w_s = ml_s + kAttnWarps * ROWS * 2;                       // [ROWS][warp]
    __syncthreads();
    auto row_of = [&](int r) {
        const int i = p.by_per_kv(r);
        return (static_cast<size_t>(b) * p.Hq + hkv * G + (r - i * G)) * p.Sq + i;
    };
    const int n = p.chunks - 1;                                      // HERE: chunks that others have
    const bool merges = HERE && chunk == n;
    const int state_words = attention_state_words(R, D);
    uint32_t* const states = HERE ? p.states + static_cast<size_t>(bk) * n * state_words : nullptr;
    float* m_s = w_s + ROWS * kAttnWarps;                            // [ROWS]: the CTA's maxima and sums
    float* l_s = m_s + ROWS;
    if (tid < R) {                                                   // at most 16 rows
        float mm = -INFINITY, ll = 0.f, f[kAttnWarps];
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) mm = fmaxf(mm, ml_s[(w * ROWS + tid) * 2]);
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) {
            const float mw = ml_s[(w * ROWS + tid) * 2];
            f[w] = mw > -INFINITY ? __expf(mw - mm) : 0.f;
            ll += ml_s[(w * ROWS + tid) * 2 + 1] * f[w];
        }
        const float inv = p.chunks > 1 ? 1.f : ll != 0.f ? 1.0f / ll : 0.f;
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) w_s[tid * kAttnWarps + w] = f[w] * inv;
        if (merges) {
            m_s[tid] = mm;
            l_s[tid] = ll;
        } else if (HERE) {
            uint32_t* dst = states + static_cast<size_t>(chunk) * state_words + R * D + 2 * tid;
            handover::store(dst, handover::word_of(mm));
            handover::store(dst + 1, handover::word_of(ll));
        } else if (p.chunks > 1) {
            float* dst = p.part + (row_of(tid) * p.chunks + chunk) * (D + 2);
            dst[0] = mm;
            dst[1] = ll;
        } else if (p.LSE) {
            p.LSE[row_of(tid)] = mm + logf(fmaxf(ll, 1e-30f));
        }
    }
    __syncthreads();
    auto sum_of = [&](int r, int c) {                                // four elements of the CTA's own
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < kAttnWarps; ++w) {
            const float4 v = *reinterpret_cast<const float4*>(o_s + (w * ROWS + r) * STRIDE + c);
            const float f = w_s[r * kAttnWarps + w];
            acc.x = fmaf(f, v.x, acc.x); acc.y = fmaf(f, v.y, acc.y);
            acc.z = fmaf(f, v.z, acc.z); acc.w = fmaf(f, v.w, acc.w);
        }
        return acc;
    };
    auto write = [&](int r, int c, float4 acc) {
        __half* dst = p.O + row_of(r) * D + c;
        const uint2 v = make_uint2(pack_h2(acc.x, acc.y), pack_h2(acc.z, acc.w));
        if (p.o_vec) {
            *reinterpret_cast<uint2*>(dst) = v;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                reinterpret_cast<uint16_t*>(dst)[e] = static_cast<uint16_t>((e < 2 ? v.x : v.y) >> (16 * (e & 1)));
        }
    };
    constexpr int kThreads = kAttnWarps * 32;
    if (!merges) {
        for (int t = tid; t < R * (D / 4); t += kThreads) {
            const int r = t / (D / 4), c = 4 * (t % (D / 4));
            const float4 acc = sum_of(r, c);
            if (HERE) {
                state_store4(states + static_cast<size_t>(chunk) * state_words + 4 * t, acc);
            } else if (p.chunks > 1) {
                float2* dst = reinterpret_cast<float2*>(p.part + (row_of(r) * p.chunks + chunk) * (D + 2) + 2 + c);
                dst[0] = make_float2(acc.x, acc.y);
                dst[1] = make_float2(acc.z, acc.w);
            } else {
                write(r, c, acc);
            }
        }
        return;
    }
    if constexpr (HERE) {
        constexpr int kOthers = kMergeHere - 1, kTurns = ROWS * (D / 4) / kThreads;
        static_assert(ROWS * kMergeHere <= kThreads && ROWS * (D / 4) % kThreads == 0, "");
        constexpr uint32_t kNone = handover::kNothing;
        const long long t0 = clock64();
        uint4 o[kTurns][kOthers];
        auto ask = [&]() {
#pragma unroll
            for (int u = 0; u < kTurns; ++u)
#pragma unroll
                for (int i = 0; i < kOthers; ++i)
                    if (i < n && u * kThreads + tid < R * (D / 4)) o[u][i] = handover::load4(states + static_cast<size_t>(i) * state_words + 4 * (u * kThreads + tid));
        };
        ask();
        // Weights: eight threads per row, one per chunk (the last is this CTA's), sums of them as in the merge kernel below.
        float* e_s = l_s + ROWS;                                     // [ROWS][chunk]
        float* ll_s = e_s + ROWS * kMergeHere;
        bool ok = true;
        if (tid < ROWS * kMergeHere) {
            const int r = tid / kMergeHere, c = tid % kMergeHere;
            float m = -INFINITY, l = 0.f;
            if (r < R && c == n) {
                m = m_s[r];
                l = l_s[r];
            } else if (r < R && c < n) {
                uint32_t* src = states + static_cast<size_t>(c) * state_words + R * D + 2 * r;
                uint32_t mw, lw;
                for (;;) {
                    mw = handover::load(src);
                    lw = handover::load(src + 1);
                    ok = handover::there(mw) && handover::there(lw);
                    if (ok || clock64() - t0 > 2000000000LL) break;
                }
                handover::store(src, kNone);
                handover::store(src + 1, kNone);
                m = __uint_as_float(mw);
                l = __uint_as_float(lw);
            }
            __syncwarp();
            float mm = m;
#pragma unroll
            for (int x = 4; x > 0; x >>= 1) mm = fmaxf(mm, __shfl_xor_sync(0xffffffffu, mm, x));
            const float e = m > -INFINITY ? __expf(m - mm) : 0.f;
            float ll = l * e;
#pragma unroll
            for (int x = 4; x > 0; x >>= 1) ll += __shfl_xor_sync(0xffffffffu, ll, x);
            e_s[tid] = e;
            if (c == 0 && r < R) {
                ll_s[r] = ll;
                if (p.LSE) p.LSE[row_of(r)] = mm + logf(fmaxf(ll, 1e-30f));
            }
        }
        __syncthreads();
        while (ok) {
            bool all = true;
#pragma unroll
            for (int u = 0; u < kTurns; ++u)
#pragma unroll
                for (int i = 0; i < kOthers; ++i)
                    if (i < n && u * kThreads + tid < R * (D / 4)) all = all && handover::there(o[u][i]);
            if (all) break;
            ok = clock64() - t0 <= 2000000000LL;
            ask();
        }
        if (!ok) {                               // a thread waits once; what it has not taken is emptied with the error
            if (p.err) atomicOr(p.err, ERR_WAIT_TIMEOUT);
            return;
        }
#pragma unroll
        for (int u = 0; u < kTurns; ++u) {
            const int t = u * kThreads + tid, r = t / (D / 4), c = 4 * (t % (D / 4));
            if (t >= R * (D / 4)) break;
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
            auto add = [&](float e, float4 v) {
                sum.x = fmaf(v.x, e, sum.x); sum.y = fmaf(v.y, e, sum.y);
                sum.z = fmaf(v.z, e, sum.z); sum.w = fmaf(v.w, e, sum.w);
            };
#pragma unroll
            for (int i = 0; i < kOthers; ++i) {
                if (i >= n) continue;
                handover::store4(states + static_cast<size_t>(i) * state_words + 4 * t, make_uint4(kNone, kNone, kNone, kNone));
                add(e_s[r * kMergeHere + i], make_float4(__uint_as_float(o[u][i].x), __uint_as_float(o[u][i].y),
                                                         __uint_as_float(o[u][i].z), __uint_as_float(o[u][i].w)));
            }
            add(e_s[r * kMergeHere + n], sum_of(r, c));
            const float ll = ll_s[r];
            write(r, c, ll != 0.f ? make_float4(sum.x / ll, sum.y / ll, sum.z / ll, sum.w / ll) : make_float4(0.f, 0.f, 0.f, 0.f));
        }
    }
}

template <int D, bool SPLIT_KEYS, bool HERE>
__global__ void __launch_bounds__(kAttnWarps * 32, 2) attention_mma_kernel(const AttnParams p) {
    asm volatile("griddepcontrol.launch_dependents;");
    using S = MmaShape<D>;
    constexpr int kKeys = SPLIT_KEYS ? 16 : 64;           // keys of a step this warp takes
    constexpr int kNT = kKeys / 8, kPieces = D / 8;
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
    const int G = p.per_kv, R = p.Sq * G;
    const int tile_no = SPLIT_KEYS ? 0 : p.by_heads(static_cast<int>(blockIdx.x)), bk = static_cast<int>(blockIdx.x) - tile_no * p.B * p.Hkv;
    const int row_tiles = SPLIT_KEYS ? 1 : (R + kMmaRows - 1) / kMmaRows;
    const int tile0 = SPLIT_KEYS ? 0 : (row_tiles - 1 - tile_no) * kMmaRows;    // long causal tiles first
    const int b = p.by_Hkv(bk), hkv = bk - b * p.Hkv;
    const int chunk = blockIdx.y;
    const __half* Kh = p.K + static_cast<size_t>(bk) * p.Sk * D;
    const __half* Vh = p.V + static_cast<size_t>(bk) * p.Sk * D;

    // this thread's two rows, their queries, and the fragments of the query matrix
    const int r_lo = tile0 + (SPLIT_KEYS ? 0 : warp * 16) + gq;
    int qi[2];
    float slope[2];
    size_t row_at[2];
    bool live[2];
    uint32_t qf[D / 16][4];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int r = r_lo + 8 * e;
        live[e] = r < R;
        const int rr = live[e] ? r : R - 1;
        qi[e] = p.by_per_kv(rr);
        const int h = hkv * G + (rr - qi[e] * G);
        row_at[e] = (static_cast<size_t>(b) * p.Hq + h) * p.Sq + qi[e];
        slope[e] = p.slopes ? p.slopes[h] : 0.f;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(p.Q + row_at[e] * D) + tq;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            qf[k][e] = src[8 * k];
            qf[k][2 + e] = src[8 * k + 4];
        }
    }
    // keys any row of the tile can see, in whole steps from the chunk's start
    const int i_min = p.by_per_kv(tile0), i_max = p.by_per_kv(min(R, tile0 + kMmaRows) - 1);
    int k0 = chunk * p.keys_per_chunk, k1 = min(p.Sk, k0 + p.keys_per_chunk);
    if (p.causal) k1 = min(k1, i_max + 1);
    if (p.window > 0 && i_min - p.window > k0) k0 += (i_min - p.window - k0) / kStepKeys * kStepKeys;
    const int steps = k1 > k0 ? (k1 - k0 + kStepKeys - 1) / kStepKeys : 0;

    auto fetch = [&](int st) {
        if (st < steps) {
            const int base = k0 + st * kStepKeys;
            const uint32_t dst = ring + (st % S::kStages) * S::kStageBytes;
#pragma unroll
            for (int u = 0; u < kStepKeys * kPieces / (kAttnWarps * 32); ++u) {
                const int e = tid + u * kAttnWarps * 32, key = e / kPieces, piece = e % kPieces;
                const bool in = base + key < k1;
                const size_t at = static_cast<size_t>(in ? base + key : k0) * D + piece * 8;
                const uint32_t off = static_cast<uint32_t>(key * D * 2 + ((piece ^ (key & 7)) * 16));
                cp_async16(dst + off, Kh + at, in);
                cp_async16(dst + kStepKeys * D * 2 + off, Vh + at, in);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int st = 0; st < S::kStages - 1; ++st) fetch(st);

    float o[D / 8][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < D / 8; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
    const int mi = lane >> 3, ml = lane & 7;               // ldmatrix: which 8x8 matrix, which of its rows

    for (int st = 0; st < steps; ++st) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S::kStages - 2) : "memory");
        __syncthreads();                                   // the step has landed; everyone is done with the one before
        fetch(st + S::kStages - 1);
        const uint32_t ks = ring + (st % S::kStages) * S::kStageBytes, vs = ks + kStepKeys * D * 2;
        const int kw = SPLIT_KEYS ? warp * 16 : 0, jb = k0 + st * kStepKeys + kw;   // this warp's first key

        float s[kNT][4];
#pragma unroll
        for (int n = 0; n < kNT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
#pragma unroll
        for (int k = 0; k < D / 16; ++k)
#pragma unroll
            for (int n = 0; n < kNT; n += 2) {
                const int key = kw + n * 8 + (mi >> 1) * 8 + ml, piece = 2 * k + (mi & 1);
                uint32_t bf[4];
                ldmatrix4(bf, ks + static_cast<uint32_t>(key * D * 2 + ((piece ^ ml) * 16)));
                mma_16816(s[n], qf[k], bf[0], bf[1]);
                mma_16816(s[n + 1], qf[k], bf[2], bf[3]);
            }
        const bool masked = jb + kKeys > k1 || (p.causal && jb + kKeys - 1 > i_min) || p.window > 0;
        // straight-line selects: a branch per element costs more than the arithmetic; a NaN score counts as masked
        float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
        for (int n = 0; n < kNT; ++n) { scale2(s[n][0], s[n][1], p.scale); scale2(s[n][2], s[n][3], p.scale); }
        if (p.slopes) {
#pragma unroll
            for (int n = 0; n < kNT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) s[n][e] -= slope[e >> 1] * static_cast<float>(qi[e >> 1] - (jb + n * 8 + 2 * tq + (e & 1)));
        }
        if (masked) {
#pragma unroll
            for (int n = 0; n < kNT; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int i = qi[e >> 1], j = n * 8 + 2 * tq + (e & 1);
                    const int hi = (p.causal ? min(k1, i + 1) : k1) - jb, lo = p.window > 0 ? i - p.window - jb : 0;
                    s[n][e] = j < hi && j >= lo ? s[n][e] : -INFINITY;
                }
        }
#pragma unroll
        for (int n = 0; n < kNT; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                s[n][e] = fmaxf(s[n][e], -INFINITY);
                mx[e >> 1] = fmaxf(mx[e >> 1], s[n][e]);
            }
        float ref[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 1));
            mx[e] = fmaxf(mx[e], __shfl_xor_sync(0xffffffffu, mx[e], 2));
            const float m_new = fmaxf(m[e], mx[e]);
            ref[e] = m_new > -INFINITY ? m_new : 0.f;      // a row that sees no key so far keeps zero sums
            const float keep = exp_of(m[e] - ref[e]);
            m[e] = m_new;
            l[e] *= keep;
#pragma unroll
            for (int n = 0; n < D / 8; ++n) { o[n][2 * e] *= keep; o[n][2 * e + 1] *= keep; }
        }
#pragma unroll
        for (int n = 0; n < kNT; ++n)
#pragma unroll
            for (int e = 0; e < 4; e += 2) {
                s[n][e] = exp_of(s[n][e] - ref[e >> 1]);       // now the probability ...
                s[n][e + 1] = exp_of(s[n][e + 1] - ref[e >> 1]);
                scale2(s[n][e], s[n][e + 1], kProbScale);      // ... 2^15 times
                l[e >> 1] += s[n][e];
                l[e >> 1] += s[n][e + 1];
            }
#pragma unroll
        for (int k = 0; k < kKeys / 16; ++k) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {                  // (rows lo, hi) x (keys 0-7, 8-15)
                const float a = s[2 * k + (q >> 1)][2 * (q & 1)], c = s[2 * k + (q >> 1)][2 * (q & 1) + 1];
                split_h2(a, c, hi[q], lo[q]);
            }
#pragma unroll
            for (int n = 0; n < D / 8; n += 2) {
                const int key = kw + k * 16 + (mi & 1) * 8 + ml, piece = n + (mi >> 1);
                uint32_t bf[4];
                ldmatrix4_trans(bf, vs + static_cast<uint32_t>(key * D * 2 + ((piece ^ ml) * 16)));
                mma_16816(o[n], hi, bf[0], bf[1]);
                mma_16816(o[n + 1], hi, bf[2], bf[3]);
                mma_16816(o[n], lo, bf[0], bf[1]);
                mma_16816(o[n + 1], lo, bf[2], bf[3]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 1);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 2);
        l[e] *= kProbUnscale;
#pragma unroll
        for (int n = 0; n < D / 8; ++n) { o[n][2 * e] *= kProbUnscale * kUngrow; o[n][2 * e + 1] *= kProbUnscale * kUngrow; }
    }

    if constexpr (!SPLIT_KEYS) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (!live[e]) continue;
            if (p.chunks == 1) {
                const float inv = l[e] != 0.f ? 1.0f / l[e] : 0.f;
                __half* dst = p.O + row_at[e] * D + 2 * tq;
#pragma unroll
                for (int n = 0; n < D / 8; ++n) {
                    const __half2 v = __floats2half2_rn(o[n][2 * e] * inv, o[n][2 * e + 1] * inv);
                    if (p.o_vec) *reinterpret_cast<__half2*>(dst + 8 * n) = v;
                    else { dst[8 * n] = __low2half(v); dst[8 * n + 1] = __high2half(v); }
                }
                if (tq == 0 && p.LSE) p.LSE[row_at[e]] = m[e] + logf(fmaxf(l[e], 1e-30f));
            } else {
                float* dst = p.part + (row_at[e] * p.chunks + chunk) * (D + 2);
#pragma unroll
                for (int n = 0; n < D / 8; ++n)
                    *reinterpret_cast<float2*>(dst + 2 + 8 * n + 2 * tq) = make_float2(o[n][2 * e], o[n][2 * e + 1]);
                if (tq == 0) { dst[0] = m[e]; dst[1] = l[e]; }
            }
        }
    } else {
        // Merge the warps' states through the ring, which everybody has finished reading.
        float* o_s = reinterpret_cast<float*>(smem);                     // [warp][16][D]
        float* ml_s = o_s + kAttnWarps * 16 * D;                         // [warp][16][2]
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int r = gq + 8 * e;
#pragma unroll
            for (int n = 0; n < D / 8; ++n)
                *reinterpret_cast<float2*>(o_s + (warp * 16 + r) * D + 8 * n + 2 * tq) = make_float2(o[n][2 * e], o[n][2 * e + 1]);
            if (tq == 0) { ml_s[(warp * 16 + r) * 2] = m[e]; ml_s[(warp * 16 + r) * 2 + 1] = l[e]; }
        }
        merge_warps<D, 16, D, HERE>(p, o_s, ml_s, R, G, b, hkv, bk, chunk);
    }
}

// The same for up to eight rows per K/V head (a decode step): keys are the rows of the matrices, queries their columns
// (m16n8k16: S^T = K Q^T, O^T = V^T P^T), so that no half of them is padding.  Half as many MMAs, exponentials
// and rescalings; P goes from the result's layout to the operand's by movmatrix.  Eight sequences, 32 heads on 8 K/V
// heads x 4096 keys, whole calls: 40.6 us as rows of 16 with a merge launch, 39.5 merged in the kernel, 38.0 so (of
// which 12 are launch and wait); 16 sequences, 64 heads x 8192 keys 96.6 -> 93.4 (6.7 TB/s); 8 heads on 2 x 4096 keys
// 20.1 -> 19.2.
template <int D, bool HERE>
__global__ void __launch_bounds__(kAttnWarps * 32, 2) attention_mma8_kernel(const AttnParams p) {
    asm volatile("griddepcontrol.launch_dependents;");
    using S = MmaShape<D>;
    constexpr int kPieces = D / 8, kStride = D + 4;       // kStride: four rows' stores of a warp on banks of their own
    extern __shared__ __align__(128) uint8_t smem[];
    const uint32_t ring = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, tq = lane & 3;
    const int G = p.per_kv, R = p.Sq * G;                 // at most 8
    const int bk = blockIdx.x, b = p.by_Hkv(bk), hkv = bk - b * p.Hkv, chunk = blockIdx.y;
    const __half* Kh = p.K + static_cast<size_t>(bk) * p.Sk * D;
    const __half* Vh = p.V + static_cast<size_t>(bk) * p.Sk * D;
    auto row_at = [&](int r) {
        const int i = p.by_per_kv(r);
        return (static_cast<size_t>(b) * p.Hq + hkv * G + (r - i * G)) * p.Sq + i;
    };

    const int k0 = chunk * p.keys_per_chunk;
    int k1 = min(p.Sk, k0 + p.keys_per_chunk);
    if (p.causal) k1 = min(k1, p.Sq);
    const int steps = k1 > k0 ? (k1 - k0 + kStepKeys - 1) / kStepKeys : 0;

    // this thread's pieces of a step: piece tid % kPieces of keys tid / kPieces + u * kKeysAtOnce
    constexpr int kKeysAtOnce = kAttnWarps * 32 / kPieces, kCopies = kStepKeys / kKeysAtOnce;
    const int my_key = tid / kPieces, my_piece = tid % kPieces;
    const size_t my_at = static_cast<size_t>(my_key) * D + my_piece * 8;
    static_assert(kKeysAtOnce % 8 == 0, "the swizzle of a thread's pieces is the same for all of them");
    const uint32_t my_off = static_cast<uint32_t>(my_key * D * 2 + ((my_piece ^ (my_key & 7)) * 16));
    auto fetch = [&](int st) {
        if (st < steps) {
            const int base = k0 + st * kStepKeys;
            const uint32_t dst = ring + (st % S::kStages) * S::kStageBytes + my_off;
            const __half* ks = Kh + static_cast<size_t>(base) * D + my_at;
            const __half* vs = Vh + static_cast<size_t>(base) * D + my_at;
            if (base + kStepKeys <= k1) {
#pragma unroll
                for (int u = 0; u < kCopies; ++u) {
                    cp_async16(dst + u * kKeysAtOnce * D * 2, ks + u * kKeysAtOnce * D, true);
                    cp_async16(dst + kStepKeys * D * 2 + u * kKeysAtOnce * D * 2, vs + u * kKeysAtOnce * D, true);
                }
            } else {
#pragma unroll
                for (int u = 0; u < kCopies; ++u) {
                    const bool in = base + my_key + u * kKeysAtOnce < k1;
                    const size_t at = in ? static_cast<size_t>(u) * kKeysAtOnce * D : 0;
                    cp_async16(dst + u * kKeysAtOnce * D * 2, in ? ks + at : Kh, in);
                    cp_async16(dst + kStepKeys * D * 2 + u * kKeysAtOnce * D * 2, in ? vs + at : Vh, in);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int st = 0; st < S::kStages - 1; ++st) fetch(st);

    // the queries as the second operand, and this thread's two rows of the scores
    uint32_t qf[D / 16][2];
    {
        const uint32_t* src = reinterpret_cast<const uint32_t*>(p.Q + row_at(min(gq, R - 1)) * D) + tq;
#pragma unroll
        for (int k = 0; k < D / 16; ++k) { qf[k][0] = src[8 * k]; qf[k][1] = src[8 * k + 4]; }
    }
    int qi[2];
    float slope[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int r = min(2 * tq + e, R - 1);
        qi[e] = p.by_per_kv(r);
        slope[e] = p.slopes ? p.slopes[hkv * G + (r - qi[e] * G)] : 0.f;
    }

    float o[D / 16][4], m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
#pragma unroll
    for (int n = 0; n < D / 16; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[n][e] = 0.f;
    const int mi = lane >> 3, ml = lane & 7;               // ldmatrix: which 8x8 matrix, which of its rows

    for (int st = 0; st < steps; ++st) {
        asm volatile("cp.async.wait_group %0;" ::"n"(S::kStages - 2) : "memory");
        __syncthreads();                                   // the step has landed; everyone is done with the one before
        fetch(st + S::kStages - 1);
        const uint32_t ks = ring + (st % S::kStages) * S::kStageBytes, vs = ks + kStepKeys * D * 2;
        const int kw = warp * 16, jb = k0 + st * kStepKeys + kw;   // this warp's 16 keys

        // element e: key gq + 8 (e / 2), row 2 tq + e % 2
        float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            const int key = kw + (mi & 1) * 8 + ml, piece = 2 * k + (mi >> 1);
            uint32_t af[4];
            ldmatrix4(af, ks + static_cast<uint32_t>(key * D * 2 + ((piece ^ ml) * 16)));
            mma_16816(s, af, qf[k][0], qf[k][1]);
        }
        scale2(s[0], s[1], p.scale);
        scale2(s[2], s[3], p.scale);
        if (p.slopes) {
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] -= slope[e & 1] * static_cast<float>(qi[e & 1] - (jb + gq + 8 * (e >> 1)));
        }
        if (jb + 16 > k1 || (p.causal && jb + 15 > 0) || p.window > 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = qi[e & 1], j = gq + 8 * (e >> 1);
                const int hi = (p.causal ? min(k1, i + 1) : k1) - jb, lo = p.window > 0 ? i - p.window - jb : 0;
                s[e] = j < hi && j >= lo ? s[e] : -INFINITY;
            }
        }
        float ref[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            s[e] = fmaxf(s[e], -INFINITY);                 // a NaN score counts as masked
            s[2 + e] = fmaxf(s[2 + e], -INFINITY);
            float mx = fmaxf(s[e], s[2 + e]);
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
            const float m_new = fmaxf(m[e], mx);
            ref[e] = m_new > -INFINITY ? m_new : 0.f;      // a row that sees no key so far keeps zero sums
            const float keep = exp_of(m[e] - ref[e]);
            m[e] = m_new;
            l[e] *= keep;
#pragma unroll
            for (int n = 0; n < D / 16; ++n) { o[n][e] *= keep; o[n][2 + e] *= keep; }
        }
        uint32_t hi[2], lo[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            float a = exp_of(s[2 * h] - ref[0]), c = exp_of(s[2 * h + 1] - ref[1]);      // the probability ...
            scale2(a, c, kProbScale);                                                   // ... 2^15 times
            l[0] += a;
            l[1] += c;
            split_h2(a, c, hi[h], lo[h]);
            hi[h] = transpose_8x8(hi[h]);
            lo[h] = transpose_8x8(lo[h]);
        }
#pragma unroll
        for (int n = 0; n < D / 16; ++n) {
            const int key = kw + (mi >> 1) * 8 + ml, piece = 2 * n + (mi & 1);
            uint32_t af[4];
            ldmatrix4_trans(af, vs + static_cast<uint32_t>(key * D * 2 + ((piece ^ ml) * 16)));
            mma_16816(o[n], af, hi[0], hi[1]);
            mma_16816(o[n], af, lo[0], lo[1]);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    float* o_s = reinterpret_cast<float*>(smem);                     // [warp][8][kStride]
    float* ml_s = o_s + kAttnWarps * 8 * kStride;                    // [warp][8][2]
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 4);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 8);
        l[e] += __shfl_xor_sync(0xffffffffu, l[e], 16);
        l[e] *= kProbUnscale;
        float* dst = o_s + (warp * 8 + 2 * tq + e) * kStride + gq;
#pragma unroll
        for (int n = 0; n < D / 16; ++n) {
            dst[16 * n] = o[n][e] * (kProbUnscale * kUngrow);
            dst[16 * n + 8] = o[n][2 + e] * (kProbUnscale * kUngrow);
        }
        if (gq == 0) { ml_s[(warp * 8 + 2 * tq + e) * 2] = m[e]; ml_s[(warp * 8 + 2 * tq + e) * 2 + 1] = l[e]; }
    }
    merge_warps<D, 8, kStride, HERE>(p, o_s, ml_s, R, G, b, hkv, bk, chunk);
}
// Merges the chunks of a row: one CTA per row, a thread per chunk for the weights exp(m_c - m), then
// a thread per output element with the chunks' partial outputs as independent loads.
__global__ void __launch_bounds__(128) attention_merge_kernel(const AttnParams p) {
    __shared__ float e_s[kMergeMaxChunks];
    __shared__ float red_s[4];
    const int row = blockIdx.x, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int D = p.D, chunks = p.chunks;
    // launched with programmatic stream serialisation: the grid that wrote the chunks is complete,
    // and its writes visible, once this returns (without that launch attribute it returns at once)
    asm volatile("griddepcontrol.wait;" ::: "memory");
    const float* base = p.part + static_cast<size_t>(row) * chunks * (D + 2);
    float mc = -INFINITY, lc = 0.f;
    if (tid < chunks) {
        mc = base[static_cast<size_t>(tid) * (D + 2)];
        lc = base[static_cast<size_t>(tid) * (D + 2) + 1];
    }
    float mm = warp_max(mc);
    if (lane == 0) red_s[warp] = mm;
    __syncthreads();
    mm = fmaxf(fmaxf(red_s[0], red_s[1]), fmaxf(red_s[2], red_s[3]));
    const float e = mc > -INFINITY ? __expf(mc - mm) : 0.f;
    if (tid < chunks) e_s[tid] = e;
    float ll = warp_sum(lc * e);
    __syncthreads();                    // red_s has been read by everyone
    if (lane == 0) red_s[warp] = ll;
    __syncthreads();
    ll = (red_s[0] + red_s[1]) + (red_s[2] + red_s[3]);
    for (int d = tid; d < D; d += 128) {
        float acc = 0.f;
#pragma unroll 8
        for (int c = 0; c < chunks; ++c) acc = fmaf(base[static_cast<size_t>(c) * (D + 2) + 2 + d], e_s[c], acc);
        p.O[static_cast<size_t>(row) * D + d] = __float2half_rn(ll != 0.f ? acc / ll : 0.f);
    }
    if (tid == 0 && p.LSE) p.LSE[row] = mm + logf(fmaxf(ll, 1e-30f));
}

// Up to 16 rows per K/V head: the warps of a CTA split the keys of a step.
bool attention_split_keys(int Hq, int Hkv, int Sq) { return static_cast<long long>(Sq) * (Hq / Hkv) <= 16; }

// Query heads one CTA of the vector kernel takes together: two of those that share a K/V head (the
// other pairs of the same K/V head run in other CTAs and find the cache in L2).
int attention_group(int Hq, int Hkv) {
    const int per = Hq / Hkv;
    return per % 2 == 0 ? 2 : 1;
}

// Whether the tcgen05 kernel takes a call of `heads` K/V heads with R (query, head) pairs each.  It needs about
// 4 us before its first scores and then takes a step of 128 keys for 128 rows in the time of one step of 64 keys for
// 64 rows here, so it wins where a block has several steps and there are tiles for more than one wave of this
// kernel (two CTAs per SM), or so much work that few tiles have to share it.  Whole calls, head_dim 128, tcgen05 /
// mma.sync kernel, microseconds (8 or 32 heads on 8 K/V heads unless given):
//   100 x 100, 8 heads 20.3 / 17.9     256 x 256, 32 heads 22.8 / 20.8       512 x 512, 32 heads 27.8 / 37.4
//   1000 x 128, 32 heads 30.2 / 28.3   4 x 256 x 256, 32 heads 34.2 / 38.8   20 x 1000, 8 heads on 1 27.9 / 19.8
//   100 x 512, 8 heads 25.6 / 19.2     100 x 512, 32 heads 21.6 / 25.2 (causal)
bool prefill_block(long long heads, long long R, int Sk, int sms) {
    if (R <= kMmaRows || Sk <= 128) return false;
    const long long tiles = heads * ((R + kMmaRows - 1) / kMmaRows);
    if (Sk <= 256) return tiles > 2LL * sms;
    return 4 * tiles > sms || tiles * ((Sk + kStepKeys - 1) / kStepKeys) > 640;
}

// How a row's keys are cut: chunks of keys_per_chunk keys.
void attention_chunks(int B, int Hq, int Hkv, int Sq, int Sk, bool matrix, int sm_count, int* chunks, int* keys_per_chunk) {
    const int sms = sm_count > 0 ? sm_count : 148;
    if (!matrix) {
        // Enough CTAs for eight per SM, chunks of at least 128 keys (one step of 32 keys per warp): a
        // step is a few dependent round trips to memory, so the bandwidth comes from many warps in
        // flight, not from long chunks.
        const long long ctas = static_cast<long long>(B) * (Hq / attention_group(Hq, Hkv)) * Sq;
        int c = static_cast<int>((8LL * sms + ctas - 1) / ctas);
        const int most = (Sk + 127) / 128;
        if (c > most) c = most;
        if (c > kMergeMaxChunks) c = kMergeMaxChunks;
        if (c < 1) c = 1;
        *chunks = c;
        *keys_per_chunk = (Sk + c - 1) / c;
        return;
    }
    // Matrix kernels: the number of chunks whose waves of CTAs (two per SM; one of the prefill kernel) take the
    // fewest key steps, a CTA's start and end counted as two steps and the merge as three.  Against each of 1 to 16 chunks
    // (23 decode shapes, whole calls): within 1.3 us of the best; 64 heads x 4096 keys in 3 / 4 / 5 / 8 / 9 chunks 39.0 /
    // 37.4 / 43.3 / 40.3 / 40.2 us.
    const long long R = static_cast<long long>(Sq) * (Hq / Hkv);
    const bool prefill = prefill_block(static_cast<long long>(B) * Hkv, R, Sk, sms);    // 128-row tiles, one CTA per SM, steps of 128 keys
    const long long tiles = prefill ? (R + 127) / 128 : (R + kMmaRows - 1) / kMmaRows;
    const long long ctas = static_cast<long long>(B) * Hkv * tiles, slots = prefill ? sms : 2LL * sms;
    const int step_keys = prefill ? 128 : kStepKeys, steps = (Sk + step_keys - 1) / step_keys;
    int best = 1;
    double best_cost = 0.0;
    for (int c = 1; c <= steps && c <= kMergeMaxChunks; ++c) {
        const int per = (steps + c - 1) / c;
        const double cost = static_cast<double>((ctas * c + slots - 1) / slots) * (per + 2.0) + (c > 1 ? 3.0 + 0.05 * c : 0.0);
        if (c == 1 || cost < best_cost) { best = c; best_cost = cost; }
    }
    const int per = (steps + best - 1) / best;
    *keys_per_chunk = per * step_keys;
    *chunks = (steps + per - 1) / per;
}

template <int D>
cudaError_t launch_matrix(const AttnParams& p, bool prefill, cudaStream_t stream) {
    const long long R = static_cast<long long>(p.Sq) * (p.Hq / p.Hkv);
    if (prefill) return launch_attention_prefill(p, stream);
    const bool split = attention_split_keys(p.Hq, p.Hkv, p.Sq);
    const long long x = static_cast<long long>(p.B) * p.Hkv * ((R + kMmaRows - 1) / kMmaRows);
    if (x > 0x7fffffffLL) return cudaErrorNotSupported;
    const dim3 grid(static_cast<unsigned>(x), static_cast<unsigned>(p.chunks));
    auto* kernel = R <= 8 ? (p.states ? attention_mma8_kernel<D, true> : attention_mma8_kernel<D, false>)
                 : !split ? attention_mma_kernel<D, false, false>
                          : p.states ? attention_mma_kernel<D, true, true> : attention_mma_kernel<D, true, false>;
    kernel<<<grid, kAttnWarps * 32, MmaShape<D>::kSmem, stream>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_vector(dim3 grid, cudaStream_t stream, const AttnParams& p) {
    if (p.group == 2) attention_decode_kernel<2><<<grid, kAttnWarps * 32, 0, stream>>>(p);
    else attention_decode_kernel<1><<<grid, kAttnWarps * 32, 0, stream>>>(p);
    return cudaGetLastError();
}

}  // namespace

cudaError_t init_attention_kernels() {
    auto allow = [](auto* kernel, int bytes) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes); };
    cudaError_t e = cudaSuccess;
    for (auto* k : {attention_mma_kernel<128, true, true>, attention_mma_kernel<128, true, false>, attention_mma_kernel<128, false, false>,
                    attention_mma8_kernel<128, true>, attention_mma8_kernel<128, false>})
        if (e == cudaSuccess) e = allow(k, MmaShape<128>::kSmem);
    for (auto* k : {attention_mma_kernel<64, true, true>, attention_mma_kernel<64, true, false>, attention_mma_kernel<64, false, false>,
                    attention_mma8_kernel<64, true>, attention_mma8_kernel<64, false>})
        if (e == cudaSuccess) e = allow(k, MmaShape<64>::kSmem);
    return e == cudaSuccess ? init_attention_prefill_kernels() : e;
}

bool attention_on_matrix_kernels(int D, const void* Q, const void* K, const void* V) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(Q) | reinterpret_cast<uintptr_t>(K) | reinterpret_cast<uintptr_t>(V);
    return (D == 64 || D == 128) && (at & 15u) == 0;
}

size_t attention_scratch_floats(int B, int Hq, int Hkv, int Sq, int Sk, int D, bool matrix, int sm_count, int* chunks_out) {
    int chunks = 1, per = Sk;
    attention_chunks(B, Hq, Hkv, Sq, Sk, matrix, sm_count, &chunks, &per);
    if (chunks_out) *chunks_out = chunks;
    const size_t rows = static_cast<size_t>(B) * Hq * Sq;
    return chunks > 1 ? rows * chunks * (D + 2) : 0;
}

size_t attention_state_bytes(int B, int Hq, int Hkv, int Sq, int D, bool matrix, int chunks) {
    if (!matrix || chunks < 2 || chunks > kMergeHere || !attention_split_keys(Hq, Hkv, Sq)) return 0;
    return static_cast<size_t>(B) * Hkv * (chunks - 1) * attention_state_words(Sq * (Hq / Hkv), D) * sizeof(uint32_t);
}

cudaError_t launch_attention_forward(const void* Q, const void* K, const void* V, void* O, float* LSE,
                                     float* scratch, uint32_t* states, const float* slopes_dev, int B, int Hq, int Hkv, int Sq,
                                     int Sk, int D, float scale, bool causal, int window, int sm_count,
                                     cudaStream_t stream, int* launches, uint32_t* err_word, const char** name) {
    if (D <= 0 || D > kAttnMaxD) return cudaErrorNotSupported;
    const long long rows_ll = static_cast<long long>(B) * Hq * Sq;
    if (rows_ll <= 0 || rows_ll > 0x7fffffffLL) return cudaErrorNotSupported;
    const int rows = static_cast<int>(rows_ll);
    AttnParams p;
    p.Q = static_cast<const __half*>(Q); p.K = static_cast<const __half*>(K); p.V = static_cast<const __half*>(V);
    p.O = static_cast<__half*>(O); p.LSE = LSE; p.part = scratch; p.slopes = slopes_dev;
    p.B = B; p.per_kv = Hq / Hkv; p.Hq = Hq; p.Hkv = Hkv; p.Sq = Sq; p.Sk = Sk; p.D = D;
    p.by_per_kv.set(p.per_kv); p.by_Hkv.set(Hkv); p.by_heads.set(B * Hkv);
    p.group = attention_group(Hq, Hkv);
    const bool matrix = attention_on_matrix_kernels(D, Q, K, V);
    attention_chunks(B, Hq, Hkv, Sq, Sk, matrix, sm_count, &p.chunks, &p.keys_per_chunk);
    p.states = matrix && attention_split_keys(Hq, Hkv, Sq) && p.chunks > 1 && p.chunks <= kMergeHere ? states : nullptr;
    if (p.chunks > 1 && !scratch && !p.states) { p.chunks = 1; p.keys_per_chunk = Sk; }
    // The tensor core truncates its running sums: a score of D / 16 steps comes out smaller by 2.2e-8 of itself per step
    // on average (mean over 150,000 scores of normal data, mma.sync and tcgen05 alike: 1.8e-7 at head_dim 128, 0.9e-7
    // at 64, always towards zero), where fp32 multiply-adds round without a bias.  The scale makes up for it, as far as an
    // fp32 number can.  LSE of 512 x 512, head_dim 128: 2.8e-7 rms from 64 bits without, 2.0e-7 with multiply-adds.
    const float matrix_scale = static_cast<float>(static_cast<double>(scale) * (1.0 + 2.2e-8 * (D / 16)));
    // A window that no query can look back beyond hides nothing; so the kernels' `i - window` stays within int.
    p.scale = matrix ? matrix_scale : scale; p.causal = causal ? 1 : 0; p.window = window < Sq - 1 ? window : 0;
    p.o_vec = (reinterpret_cast<uintptr_t>(O) & 15u) == 0;
    // the vector kernel's lanes load D / 32 elements of a value row at a time
    p.v_vec = (reinterpret_cast<uintptr_t>(V) & (D == 128 ? 7u : 3u)) == 0;
    p.err = err_word;
    cudaError_t e = cudaErrorNotSupported;
    if (matrix) {
        const bool prefill = prefill_block(static_cast<long long>(B) * Hkv, static_cast<long long>(Sq) * (Hq / Hkv), Sk,
                                           sm_count > 0 ? sm_count : 148);
        e = D == 128 ? launch_matrix<128>(p, prefill, stream) : launch_matrix<64>(p, prefill, stream);
        if (name) *name = prefill ? "attention_prefill_tcgen05_sm100" : "attention_mma_sm100";
    }
    if (e == cudaErrorNotSupported) {
        e = launch_vector(dim3(static_cast<unsigned>(rows / p.group), static_cast<unsigned>(p.chunks)), stream, p);
        if (name) *name = "attention_decode_sm100";
    }
    if (e != cudaSuccess) return e;
    if (launches) *launches += 1;
    if (p.chunks > 1 && !p.states) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(rows));
        cfg.blockDim = dim3(128);
        cfg.stream = stream;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaLaunchKernelEx(&cfg, attention_merge_kernel, p);
        if (e == cudaSuccess && launches) *launches += 1;
    }
    return e;
}

}  // namespace tcb
