// Attention of a prefill block on the sm_100a tensor cores (tcgen05), head_dim 64 and 128.
//
// Same operation and data as attention.cu (include/tensorcore/attention.h:24-60; arithmetic of
// lib/ops/attention_cpu.cpp:131-277); this kernel takes it when more than 64 (query, head) pairs share a K/V
// head.
//
//   * A CTA owns 128 of those pairs (head fastest, so a tile's rows see about the same keys) and walks the
//     keys 128 at a time; a long cache is cut into chunks like in the other kernels.
//   * A loader warp brings K and V through a three-stage ring (TMA boxes of 128 keys x 64 elements, 128-byte
//     swizzle; keys past the cache's end are zeros).
//   * One issuing warp: S = Q K^T (M128 x N128, operands in shared memory) into one of two score buffers
//     in tensor memory, the next step's while this step's softmax runs; then O += P V with P in tensor
//     memory (the A operand) and V as it lies (MN-major).
//   * Eight softmax warps, two threads per row with 64 scores each in registers: running maximum (exchanged
//     between the two), exponentials; O is rescaled in tensor memory only when a row's maximum has grown.  The probabilities are fp32
//     numbers; each goes to the tensor core as two fp16 numbers (attention_math.cuh says to how many bits), two MMAs.
//
// What bounds it: latency.  Causal 512 x 512, 32 heads on 8 K/V heads, head_dim 128 is 128 CTAs of up to four
// steps; clock stamps of the longest: about 8000 clocks until the first scores (barriers, tensor memory, Q, cold
// code), then 3500 a step - exponentials and masks 2100 to 2500, rescaling 600, storing P 500 - in which 1060
// clocks of P V and 530 of Q K^T hide, and 1900 to store O.  28.3 us through the synchronous call (10 us of it
// launch and wait; 31 with three warps of cp.async as loaders, which a step then waited 1700 clocks for),
// 38 us on the mma.sync kernel, whose tensor instructions run at an eighth of the rate, 388 us as a
// streaming pass per query row.
#include "attention_math.cuh"
#include "kernels.h"
#include "sm100_prims.cuh"
#include "tensor_map.h"

#include <cuda_fp16.h>

namespace tcb {
namespace {

using namespace sm100;
using namespace attn;

constexpr int kRows = 128, kKeys = 128, kStages = 3;
constexpr int kSoftWarps = 8, kLoadWarp = kSoftWarps, kIssueWarp = kSoftWarps + 1;
constexpr int kThreads = (kIssueWarp + 1) * 32;
constexpr int kBarBytes = 3072;
constexpr uint32_t kSwizzle128 = 2;
// tensor memory columns
constexpr uint32_t kColS = 0, kColPHi = 256, kColPLo = 320, kColO = 384, kTmemCols = 512;

struct PrefillBars {
    uint64_t q_full, k_full[kStages], v_full[kStages], kv_empty[kStages], s_full[2], s_empty[2], p_full, pv_done, drain, both[4];
    uint32_t tmem_base;
    int abort_flag;
    float pair[2][2][kRows];      // what the two threads of a row tell each other, two buffers
};
static_assert(sizeof(PrefillBars) <= kBarBytes, "barrier block too large");

__device__ __forceinline__ uint64_t desc128(uint32_t addr, uint32_t lbo) {
    return smem_desc_kmajor(addr, lbo, 1024u) | (static_cast<uint64_t>(kSwizzle128) << 61);
}

template <int D>
__global__ void __launch_bounds__(kThreads, 1) attention_prefill_kernel(const AttnParams p, const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap) {
    constexpr int kSlabs = D / 64;                         // 64-element (128-byte) pieces of a row
    constexpr uint32_t kSlab = kKeys * 128;                // bytes of one piece of 128 rows
    constexpr uint32_t kTile = kSlabs * kSlab;             // Q, or one stage's K or V
    extern __shared__ __align__(1024) uint8_t smem[];
    PrefillBars* bars = reinterpret_cast<PrefillBars*>(smem);
    volatile int* abort_flag = &bars->abort_flag;
    const uint32_t q_s = s_u32(smem + kBarBytes), ring = q_s + kTile;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    const int G = p.Hq / p.Hkv, R = p.Sq * G;
    const int heads = p.B * p.Hkv, bk = blockIdx.x % heads;
    const int row_tiles = (R + kRows - 1) / kRows;
    const int tile0 = (row_tiles - 1 - static_cast<int>(blockIdx.x / heads)) * kRows;    // long causal tiles first
    const int b = bk / p.Hkv, hkv = bk % p.Hkv, chunk = blockIdx.y;
    // keys any row of the tile can see, in whole steps from the chunk's start
    const int i_min = tile0 / G, i_max = (min(R, tile0 + kRows) - 1) / G;
    int k0 = chunk * p.keys_per_chunk, k1 = min(p.Sk, k0 + p.keys_per_chunk);
    if (p.causal) k1 = min(k1, i_max + 1);
    if (p.window > 0 && i_min - p.window > k0) k0 += (i_min - p.window - k0) / kKeys * kKeys;
    const int steps = k1 > k0 ? (k1 - k0 + kKeys - 1) / kKeys : 0;

    if (tid == 0) {
        bar_init(&bars->q_full, kSoftWarps);
        for (int i = 0; i < kStages; ++i) {
            bar_init(&bars->k_full[i], 1);
            bar_init(&bars->v_full[i], 1);
            bar_init(&bars->kv_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            bar_init(&bars->s_full[i], 1);
            bar_init(&bars->s_empty[i], kSoftWarps);
        }
        bar_init(&bars->p_full, kSoftWarps);
        bar_init(&bars->pv_done, 1);
        bar_init(&bars->drain, 1);
        for (int i = 0; i < 4; ++i) bar_init(&bars->both[i], 2);
        bars->abort_flag = 0;
        fence_barrier_init();
    }
    if (tid == kLoadWarp * 32) { prefetch_tensormap(&kmap); prefetch_tensormap(&vmap); }
    __syncthreads();
    // The first K and V are on their way while tensor memory is allocated.
    auto fetch = [&](const CUtensorMap* map, uint64_t* bar, uint32_t offset, int key) {
        bar_expect_tx(bar, kTile);
#pragma unroll
        for (int sl = 0; sl < kSlabs; ++sl)
            tensor_load_3d(smem + kBarBytes + kTile + offset + sl * kSlab, map, 64 * sl, key, bk, bar);
    };
    if (warp == kLoadWarp && steps > 0) {
        if (elect_one()) {
            fetch(&kmap, &bars->k_full[0], 0, k0);
            fetch(&vmap, &bars->v_full[0], kTile, k0);
        }
        __syncwarp();
    }
    if (warp == kIssueWarp) tmem_alloc(&bars->tmem_base, kTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = bars->tmem_base;
    bool failed = false;

    if (warp < kSoftWarps) {
        // ---------------- softmax: two threads per row = TMEM lane, half of the keys (or columns of O) each ------
        constexpr int kHalf = kKeys / 2;
        const int quad = warp & 3, hf = warp >> 2, lr = quad * 32 + lane, r = tile0 + lr;
        const bool live = r < R;
        const int rr = live ? r : R - 1, i = rr / G, h = hkv * G + (rr - i * G);
        const size_t row_at = (static_cast<size_t>(b) * p.Hq + h) * p.Sq + i;
        const float slope = p.slopes ? p.slopes[h] : 0.f;
        const uint32_t lanes = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        {
            const uint4* src = reinterpret_cast<const uint4*>(p.Q + row_at * D);
#pragma unroll
            for (int u = 0; u < D / 16; ++u) {
                const int c = hf * (D / 16) + u;
                sts128(q_s + (c / 8) * kSlab + lr * 128 + (((c & 7) ^ (lr & 7)) * 16), src[c]);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->q_full);
        }
        // the row's other thread is in warp +-4: a value each through shared memory
        uint32_t turn = 0;
        auto exchange = [&](float v) {
            bars->pair[turn][hf][lr] = v;
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->both[quad]);
            if (!wait_all(&bars->both[quad], turn, abort_flag)) failed = true;
            const float other = bars->pair[turn][hf ^ 1][lr];
            turn ^= 1u;
            return other;
        };
        float m = -INFINITY, l = 0.f;
        for (int t = 0; t < steps; ++t) {
            const int buf = t & 1, jb = k0 + t * kKeys + hf * kHalf;      // this thread's first key
            if (!wait_all(&bars->s_full[buf], static_cast<uint32_t>(t >> 1) & 1u, abort_flag)) { failed = true; break; }
            tc_fence_after_sync();
            uint32_t raw[kHalf / 16][16];
#pragma unroll
            for (int c = 0; c < kHalf / 16; ++c)
                tmem_ld16(lanes + kColS + static_cast<uint32_t>(buf * kKeys + hf * kHalf + 16 * c), raw[c]);
            tmem_wait_ld();
            float s[kHalf];
#pragma unroll
            for (int e = 0; e < kHalf; ++e) {
                asm volatile("" : "+r"(raw[e / 16][e % 16]));                    // read behind the wait
                s[e] = __uint_as_float(raw[e / 16][e % 16]);
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->s_empty[buf]);
            const bool masked = jb + kHalf > k1 || (p.causal && jb + kHalf - 1 > i_min) || p.window > 0;
            // Straight-line selects throughout: a branch per element made this part four times as long.  A NaN
            // score counts as masked, as in the other kernels.
#pragma unroll
            for (int e = 0; e < kHalf; e += 2) scale2(s[e], s[e + 1], p.scale);
            if (p.slopes) {
#pragma unroll
                for (int e = 0; e < kHalf; ++e) s[e] -= slope * static_cast<float>(i - jb - e);
            }
            if (masked) {
                const int hi_e = (p.causal ? min(k1, i + 1) : k1) - jb, lo_e = p.window > 0 ? i - p.window - jb : 0;
#pragma unroll
                for (int e = 0; e < kHalf; ++e) s[e] = e < hi_e && e >= lo_e ? s[e] : -INFINITY;
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < kHalf; ++e) {
                s[e] = fmaxf(s[e], -INFINITY);
                mx[e & 3] = fmaxf(mx[e & 3], s[e]);
            }
            const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            const float m_new = fmaxf(m, fmaxf(mine, exchange(mine)));
            if (failed) break;
            const float ref = m_new > -INFINITY ? m_new : 0.f;          // a row that sees no key so far keeps zero sums
            const float keep = exp_of(m - ref);
            m = m_new;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < kHalf; e += 2) {
                s[e] = exp_of(s[e] - ref);                               // now the probability ...
                s[e + 1] = exp_of(s[e + 1] - ref);
                scale2(s[e], s[e + 1], kProbScale);                      // ... 2^15 times
                sum[e & 3] += s[e];
                sum[(e + 1) & 3] += s[e + 1];
            }
            l = l * keep + ((sum[0] + sum[1]) + (sum[2] + sum[3]));      // over this thread's keys
            if (t > 0) {
                // P and O are free once the product of the step before is done
                if (!wait_all(&bars->pv_done, static_cast<uint32_t>(t - 1) & 1u, abort_flag)) { failed = true; break; }
                tc_fence_after_sync();
                if (__any_sync(0xffffffffu, keep != 1.f)) {
#pragma unroll
                    for (int c = 0; c < D / 2; c += 32) {
                        const uint32_t at = lanes + kColO + static_cast<uint32_t>(hf * (D / 2) + c);
                        uint32_t v[16], w[16];
                        tmem_ld16(at, v);
                        tmem_ld16(at + 16u, w);
                        tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            asm volatile("" : "+r"(v[e]), "+r"(w[e]));
                            v[e] = __float_as_uint(__uint_as_float(v[e]) * keep);
                            w[e] = __float_as_uint(__uint_as_float(w[e]) * keep);
                        }
                        tmem_st16(at, v);
                        tmem_st16(at + 16u, w);
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < kHalf / 32; ++c) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) split_h2(s[32 * c + 2 * e], s[32 * c + 2 * e + 1], hi[e], lo[e]);
                tmem_st16(lanes + kColPHi + static_cast<uint32_t>(hf * (kHalf / 2) + 16 * c), hi);
                tmem_st16(lanes + kColPLo + static_cast<uint32_t>(hf * (kHalf / 2) + 16 * c), lo);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->p_full);
        }
        if (!failed && steps > 0) {
            if (!wait_all(&bars->pv_done, static_cast<uint32_t>(steps - 1) & 1u, abort_flag)) failed = true;
            tc_fence_after_sync();
        }
        if (!failed) l += exchange(l);
        if (!failed) {
            const float inv = l != 0.f ? kUngrow / l : 0.f;              // l and O are both 2^15 times as large here
            float* part = p.part + (row_at * p.chunks + chunk) * (D + 2);
            {
                constexpr int kQ = D / 32;                 // pieces of 16 columns of this thread's half
                uint32_t v[kQ][16];
#pragma unroll
                for (int q = 0; q < kQ; ++q) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) v[q][e] = 0u;
                    if (steps > 0) tmem_ld16(lanes + kColO + static_cast<uint32_t>(hf * (D / 2) + 16 * q), v[q]);
                }
                tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < kQ; ++q) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) asm volatile("" : "+r"(v[q][e]));
                    const int c = hf * (D / 2) + 16 * q;
                    if (!live) continue;
                    if (p.chunks == 1) {
                        uint32_t o[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            o[e] = pack_h2(__uint_as_float(v[q][2 * e]) * inv, __uint_as_float(v[q][2 * e + 1]) * inv);
                        if (p.o_vec) {
                            uint4* dst = reinterpret_cast<uint4*>(p.O + row_at * D + c);
                            dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
                            dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
                        } else {
                            uint16_t* dst = reinterpret_cast<uint16_t*>(p.O + row_at * D + c);
#pragma unroll
                            for (int e = 0; e < 16; ++e) dst[e] = static_cast<uint16_t>(o[e / 2] >> (16 * (e & 1)));
                        }
                    } else {
#pragma unroll
                        for (int e = 0; e < 16; e += 2)
                            *reinterpret_cast<float2*>(part + 2 + c + e) = make_float2(__uint_as_float(v[q][e]) * (kProbUnscale * kUngrow), __uint_as_float(v[q][e + 1]) * (kProbUnscale * kUngrow));
                    }
                }
            }
            if (live && hf == 0) {
                if (p.chunks > 1) { part[0] = m; part[1] = l * kProbUnscale; }
                else if (p.LSE) p.LSE[row_at] = m + logf(fmaxf(l * kProbUnscale, 1e-30f));
            }
        }
        tc_fence_before_sync();
    } else if (warp == kLoadWarp) {
        // ---------------- loader ------------------------------------------------------------------------------
        int sent = steps > 0 ? 1 : 0;
        for (int t = 1; t < steps; ++t, ++sent) {
            const int st = t % kStages;
            if (!wait_all(&bars->kv_empty[st], (static_cast<uint32_t>(t / kStages) & 1u) ^ 1u, abort_flag)) { failed = true; break; }
            if (elect_one()) {
                fetch(&kmap, &bars->k_full[st], static_cast<uint32_t>(st) * 2u * kTile, k0 + t * kKeys);
                fetch(&vmap, &bars->v_full[st], static_cast<uint32_t>(st) * 2u * kTile + kTile, k0 + t * kKeys);
            }
            __syncwarp();
        }
        if (failed || *abort_flag) {                       // copies in flight land before the shared memory is released
            for (int t = sent > kStages ? sent - kStages : 0; t < sent; ++t) {
                bar_wait(&bars->k_full[t % kStages], static_cast<uint32_t>(t / kStages) & 1u, nullptr, 100000000LL);
                bar_wait(&bars->v_full[t % kStages], static_cast<uint32_t>(t / kStages) & 1u, nullptr, 100000000LL);
            }
        }
    } else {
        // ---------------- MMA issue -----------------------------------------------------------------------------
        const uint32_t id_s = idesc_f16_f32(kRows, kKeys), id_o = idesc_f16_f32(kRows, D) | (1u << 16);     // V is MN-major
        auto scores = [&](int t) {
            const int st = t % kStages, buf = t & 1;
            if (!wait_all(&bars->k_full[st], static_cast<uint32_t>(t / kStages) & 1u, abort_flag)) { failed = true; return; }
            if (!wait_all(&bars->s_empty[buf], (static_cast<uint32_t>(t >> 1) & 1u) ^ 1u, abort_flag)) { failed = true; return; }
            tc_fence_after_sync();
            const uint32_t k_s = ring + static_cast<uint32_t>(st) * 2u * kTile;
            if (elect_one()) {
#pragma unroll
                for (int j = 0; j < D / 16; ++j) {
                    const uint32_t off = (j / 4) * kSlab + (j % 4) * 32;
                    mma_f16_ss(tmem + kColS + static_cast<uint32_t>(buf * kKeys), desc128(q_s + off, 16u), desc128(k_s + off, 16u), id_s,
                               j > 0 ? 1u : 0u);
                }
                mma_commit(&bars->s_full[buf]);
            }
            __syncwarp();
        };
        if (steps > 0 && wait_all(&bars->q_full, 0, abort_flag)) {
            scores(0);
            for (int t = 0; t < steps && !failed; ++t) {
                if (t + 1 < steps) scores(t + 1);
                if (failed) break;
                const int st = t % kStages;
                if (!wait_all(&bars->v_full[st], static_cast<uint32_t>(t / kStages) & 1u, abort_flag)) { failed = true; break; }
                if (!wait_all(&bars->p_full, static_cast<uint32_t>(t) & 1u, abort_flag)) { failed = true; break; }
                tc_fence_after_sync();
                const uint32_t v_s = ring + static_cast<uint32_t>(st) * 2u * kTile + kTile;
                if (elect_one()) {
#pragma unroll
                    for (int j = 0; j < kKeys / 16; ++j) {
                        const uint64_t vd = desc128(v_s + j * 2048, kSlab);
                        mma_f16_ts(tmem + kColO, tmem + kColPHi + 8u * j, vd, id_o, t > 0 || j > 0 ? 1u : 0u);
                        mma_f16_ts(tmem + kColO, tmem + kColPLo + 8u * j, vd, id_o, 1u);
                    }
                    mma_commit(&bars->pv_done);
                    mma_commit(&bars->kv_empty[st]);
                }
                __syncwarp();
            }
        } else if (steps > 0) {
            failed = true;
        }
        if (failed || *abort_flag) {
            // every MMA issued has completed before tensor and shared memory are released
            if (elect_one()) mma_commit(&bars->drain);
            __syncwarp();
            bar_wait(&bars->drain, 0, nullptr, 100000000LL);
        }
    }
    if (failed) {
        *abort_flag = 1;
        if (p.err) atomicOr(p.err, ERR_WAIT_TIMEOUT);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == kIssueWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem, kTmemCols);
    }
}

template <int D> constexpr int kSmem = kBarBytes + kRows * D * 2 + kStages * 2 * kKeys * D * 2;

}  // namespace

cudaError_t init_attention_prefill_kernels() {
    const cudaFuncAttribute a = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const cudaError_t e = cudaFuncSetAttribute(attention_prefill_kernel<128>, a, kSmem<128>);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(attention_prefill_kernel<64>, a, kSmem<64>);
}

cudaError_t launch_attention_prefill(const AttnParams& p, cudaStream_t stream) {
    const long long R = static_cast<long long>(p.Sq) * (p.Hq / p.Hkv);
    const long long x = static_cast<long long>(p.B) * p.Hkv * ((R + kRows - 1) / kRows);
    if (R > 0x7fffff00LL || x > 0x7fffffffLL) return cudaErrorNotSupported;
    const dim3 grid(static_cast<unsigned>(x), static_cast<unsigned>(p.chunks));
    CUtensorMap kmap, vmap;
    const uint64_t heads = static_cast<uint64_t>(p.B) * p.Hkv;
    if (!encode_heads_sw128(&kmap, p.K, heads, p.Sk, p.D, kKeys) || !encode_heads_sw128(&vmap, p.V, heads, p.Sk, p.D, kKeys))
        return cudaErrorNotSupported;
    if (p.D == 128) attention_prefill_kernel<128><<<grid, kThreads, kSmem<128>, stream>>>(p, kmap, vmap);
    else attention_prefill_kernel<64><<<grid, kThreads, kSmem<64>, stream>>>(p, kmap, vmap);
    return cudaGetLastError();
}

}  // namespace tcb
