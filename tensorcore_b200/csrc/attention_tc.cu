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
//   * Sixteen softmax warps, four threads per row with 32 scores each in registers (two with 64: 3500 clocks a step
//     where four take 2900): running maximum (an atomic on the row's word in shared memory), exponentials; O is rescaled
//     in tensor memory only when a row's maximum has grown.  The probabilities are fp32
//     numbers; each goes to the tensor core as two fp16 numbers (attention_math.cuh says to how many bits), two MMAs.
//   * Q and O cross global memory by whole rows, O through shared memory (a thread per row takes a clock for each lane
//     and 16 bytes: O 2650 clocks instead of 2400).  Rows' queries and heads by multiplication (FastDiv): the device's
//     divisions were 700 clocks of the way to the first load.
//
// What bounds it: latency.  Causal 512 x 512, 32 heads on 8 K/V heads, head_dim 128 is 128 CTAs of up to four
// steps; clock stamps of the longest, inputs in HBM: barriers and tensor memory ready at 3500, Q in shared memory 5400,
// first scores 6800; 3100 a step - scores and maximum 1000 to 1250, exponentials 1000, the wait for P V, rescaling and
// storing P 850, the wait for the next scores 270 - in which 1060 clocks of P V and 530 of Q K^T hide; 1500 for the last
// P V, 2400 for O (1500 of them through shared memory); 23,100 in all.  Whole calls: 28.2 us with two
// threads per row, 25.8 now (10 us of it launch and wait), 2048 x 2048 97.5 -> 88.3, 4 x 2048 x 2048 without a mask
// 500 -> 467; 38 us on the mma.sync kernel, whose tensor instructions run at an eighth of the rate, 388 us as a
// streaming pass per query row.  The instance of head_dim 128 spills 40 bytes (96 registers, what 18 warps leave).
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
constexpr int kParts = 4;                      // softmax threads per row
constexpr int kSoftWarps = 4 * kParts, kLoadWarp = kSoftWarps, kIssueWarp = kSoftWarps + 1;
constexpr int kThreads = (kIssueWarp + 1) * 32;
constexpr int kBarBytes = 3072;
constexpr uint32_t kSwizzle128 = 2;
// tensor memory columns
constexpr uint32_t kColS = 0, kColPHi = 256, kColPLo = 320, kColO = 384, kTmemCols = 512;

struct PrefillBars {
    uint64_t q_full, k_full[kStages], v_full[kStages], kv_empty[kStages], s_full[2], s_empty[2], p_full, pv_done, drain, both[4];
    uint32_t tmem_base;
    int abort_flag;
    int best[3][kRows];           // the threads of a row work out its maximum here (order_of), in turn in three buffers
};
static_assert(sizeof(PrefillBars) <= kBarBytes, "barrier block too large");

__device__ __forceinline__ uint64_t desc128(uint32_t addr, uint32_t lbo) {
    return smem_desc_kmajor(addr, lbo, 1024u) | (static_cast<uint64_t>(kSwizzle128) << 61);
}

// Floats (no NaN) as integers of the same order, and back.
__device__ __forceinline__ int order_of(float v) {
    const int b = __float_as_int(v);
    return b >= 0 ? b : b ^ 0x7fffffff;
}
__device__ __forceinline__ float value_of(int b) { return __int_as_float(b >= 0 ? b : b ^ 0x7fffffff); }

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

    const int G = p.per_kv, R = p.Sq * G;
    const int heads = p.B * p.Hkv, tile_no = p.by_heads(static_cast<int>(blockIdx.x)), bk = static_cast<int>(blockIdx.x) - tile_no * heads;
    const int row_tiles = (R + kRows - 1) / kRows;
    const int tile0 = (row_tiles - 1 - tile_no) * kRows;    // long causal tiles first
    const int b = p.by_Hkv(bk), hkv = bk - b * p.Hkv, chunk = blockIdx.y;
    // keys any row of the tile can see, in whole steps from the chunk's start
    const int i_min = p.by_per_kv(tile0);
    auto query_of = [&](int lrow) { return p.by_per_kv(tile0 + lrow); };
    const int i_max = query_of(min(R - tile0, kRows) - 1);
    int k0 = chunk * p.keys_per_chunk, k1 = min(p.Sk, k0 + p.keys_per_chunk);
    if (p.causal) k1 = min(k1, i_max + 1);
    if (p.window > 0 && i_min - p.window > k0) k0 += (i_min - p.window - k0) / kKeys * kKeys;
    const int steps = k1 > k0 ? (k1 - k0 + kKeys - 1) / kKeys : 0;

    // Rows of Q and O are read and written whole, D / 8 lanes of a warp to a row (a thread per row took a clock per lane
    // and 16 bytes: 2600 for O, as much for Q); a softmax warp has the eight rows from my_row0.
    auto row_of = [&](int lrow, bool* there) {
        *there = tile0 + lrow < R;
        if (!*there) lrow = R - 1 - tile0;
        const int i = query_of(lrow);
        return (b * p.Hq + hkv * G + (tile0 + lrow - i * G)) * p.Sq + i;      // below 2^31 (launch_attention_forward)
    };
    constexpr int kLanes = D / 8, kRowsAtOnce = 32 / kLanes, kTurns = 8 / kRowsAtOnce;      // of 16 bytes; rows a load; loads
    const int quad = warp & 3, part_no = warp >> 2, piece = lane % kLanes;
    const int my_row0 = quad * 32 + part_no * 8 + lane / kLanes;
    int rows_at[kTurns];
    bool rows_live[kTurns];
    uint4 q_piece[kTurns];
    if (warp < kSoftWarps) {                 // on its way while barriers and tensor memory are set up
#pragma unroll
        for (int u = 0; u < kTurns; ++u) {
            rows_at[u] = row_of(my_row0 + u * kRowsAtOnce, &rows_live[u]);
            asm volatile("" : "+r"(rows_at[u]));          // not to be worked out again for O
            // (volatile: the compiler would move the load down to its use)
            asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(q_piece[u].x), "=r"(q_piece[u].y), "=r"(q_piece[u].z), "=r"(q_piece[u].w) : "l"(p.Q + static_cast<size_t>(rows_at[u]) * D + piece * 8));
        }
    }
    // The loader's own barriers, and the first K and V on their way; tensor memory and the other barriers beside it.
    auto fetch = [&](const CUtensorMap* map, uint64_t* bar, uint32_t offset, int key) {
        bar_expect_tx(bar, kTile);
#pragma unroll
        for (int sl = 0; sl < kSlabs; ++sl)
            tensor_load_3d(smem + kBarBytes + kTile + offset + sl * kSlab, map, 64 * sl, key, bk, bar);
    };
    if (warp == kLoadWarp) {
        if (lane == 0) { prefetch_tensormap(&kmap); prefetch_tensormap(&vmap); }
        if (lane < kStages) {
            bar_init(&bars->k_full[lane], 1);
            bar_init(&bars->v_full[lane], 1);
            bar_init(&bars->kv_empty[lane], 1);
        }
        fence_barrier_init();
        fence_proxy_async();
        __syncwarp();
        if (steps > 0 && elect_one()) {
            fetch(&kmap, &bars->k_full[0], 0, k0);
            fetch(&vmap, &bars->v_full[0], kTile, k0);
        }
        __syncwarp();
    } else if (warp == kIssueWarp) {
        if (lane < 4) {
            bar_init(&bars->both[lane], kParts);
        } else if (lane < 6) {
            bar_init(&bars->s_full[lane - 4], 1);
            bar_init(&bars->s_empty[lane - 4], kSoftWarps);
        } else if (lane == 6) {
            bar_init(&bars->q_full, kSoftWarps);
            bar_init(&bars->p_full, kSoftWarps);
            bar_init(&bars->pv_done, 1);
            bar_init(&bars->drain, 1);
            bars->abort_flag = 0;
        }
        fence_barrier_init();
        __syncwarp();
        tmem_alloc(&bars->tmem_base, kTmemCols);
    }
    for (int e = tid; e < 3 * kRows; e += kThreads) (&bars->best[0][0])[e] = order_of(-INFINITY);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem = bars->tmem_base;
    bool failed = false;

    if (warp < kSoftWarps) {
        // ---------------- softmax: kParts threads per row = TMEM lane, a part of the keys (or columns of O) each ------
        constexpr int kMine = kKeys / kParts, kCols = D / kParts;
        const int lr = quad * 32 + lane, r = tile0 + lr, i = query_of(r < R ? lr : R - 1 - tile0);      // this thread's row
        const float slope = p.slopes ? p.slopes[hkv * G + ((r < R ? r : R - 1) - i * G)] : 0.f;
        const uint32_t lanes = tmem + (static_cast<uint32_t>(quad * 32) << 16);
        {
#pragma unroll
            for (int u = 0; u < kTurns; ++u) {
                const int lrow = my_row0 + u * kRowsAtOnce;
                sts128(q_s + (piece / 8) * kSlab + lrow * 128 + (((piece & 7) ^ (lrow & 7)) * 16), q_piece[u]);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->q_full);
        }
        // The row's other threads are four warps apart.  A buffer is cleared once the barrier after its use has shown
        // that all of them have read it, and used again behind the next.
        auto row_wait = [&](uint32_t parity) {
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->both[quad]);
            if (!wait_all(&bars->both[quad], parity, abort_flag)) failed = true;
        };
        auto row_max = [&](float v, int t) {
            atomicMax(&bars->best[t % 3][lr], order_of(v));
            row_wait(static_cast<uint32_t>(t) & 1u);
            const float all = value_of(bars->best[t % 3][lr]);
            if (part_no == 0) bars->best[(t + 2) % 3][lr] = order_of(-INFINITY);
            return all;
        };
        float m = -INFINITY, l = 0.f;
        for (int t = 0; t < steps; ++t) {
            const int buf = t & 1, jb = k0 + t * kKeys + part_no * kMine;      // this thread's first key
            if (!wait_all(&bars->s_full[buf], static_cast<uint32_t>(t >> 1) & 1u, abort_flag)) { failed = true; break; }
            tc_fence_after_sync();
            uint32_t raw[kMine / 16][16];
#pragma unroll
            for (int c = 0; c < kMine / 16; ++c)
                tmem_ld16(lanes + kColS + static_cast<uint32_t>(buf * kKeys + part_no * kMine + 16 * c), raw[c]);
            tmem_wait_ld();
            float s[kMine];
#pragma unroll
            for (int e = 0; e < kMine; ++e) {
                asm volatile("" : "+r"(raw[e / 16][e % 16]));                    // read behind the wait
                s[e] = __uint_as_float(raw[e / 16][e % 16]);
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->s_empty[buf]);
            const bool masked = jb + kMine > k1 || (p.causal && jb + kMine - 1 > i_min) || p.window > 0;
            // Straight-line selects throughout: a branch per element made this part four times as long.  A NaN
            // score counts as masked, as in the other kernels.
#pragma unroll
            for (int e = 0; e < kMine; e += 2) scale2(s[e], s[e + 1], p.scale);
            if (p.slopes) {
#pragma unroll
                for (int e = 0; e < kMine; ++e) s[e] -= slope * static_cast<float>(i - jb - e);
            }
            if (masked) {
                const int hi_e = (p.causal ? min(k1, i + 1) : k1) - jb, lo_e = p.window > 0 ? i - p.window - jb : 0;
#pragma unroll
                for (int e = 0; e < kMine; ++e) s[e] = e < hi_e && e >= lo_e ? s[e] : -INFINITY;
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int e = 0; e < kMine; ++e) {
                s[e] = fmaxf(s[e], -INFINITY);
                mx[e & 3] = fmaxf(mx[e & 3], s[e]);
            }
            const float mine = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            const float m_new = fmaxf(m, row_max(mine, t));
            if (failed) break;
            const float ref = m_new > -INFINITY ? m_new : 0.f;          // a row that sees no key so far keeps zero sums
            const float keep = exp_of(m - ref);
            m = m_new;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int e = 0; e < kMine; e += 2) {
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
                    uint32_t v[kCols / 16][16];
                    const uint32_t at = lanes + kColO + static_cast<uint32_t>(part_no * kCols);
#pragma unroll
                    for (int c = 0; c < kCols / 16; ++c) tmem_ld16(at + 16u * c, v[c]);
                    tmem_wait_ld();
#pragma unroll
                    for (int c = 0; c < kCols / 16; ++c) {
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            asm volatile("" : "+r"(v[c][e]));
                            v[c][e] = __float_as_uint(__uint_as_float(v[c][e]) * keep);
                        }
                        tmem_st16(at + 16u * c, v[c]);
                    }
                }
            }
#pragma unroll
            for (int c = 0; c < kMine / 32; ++c) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) split_h2(s[32 * c + 2 * e], s[32 * c + 2 * e + 1], hi[e], lo[e]);
                tmem_st16(lanes + kColPHi + static_cast<uint32_t>(part_no * (kMine / 2) + 16 * c), hi);
                tmem_st16(lanes + kColPLo + static_cast<uint32_t>(part_no * (kMine / 2) + 16 * c), lo);
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
        if (!failed) {                                       // the row's sum, through the ring: every copy and MMA is done
            float* sums = reinterpret_cast<float*>(smem + kBarBytes + kTile);
            sums[part_no * kRows + lr] = l;
            row_wait(static_cast<uint32_t>(steps) & 1u);
            l = sums[lr];
#pragma unroll
            for (int k = 1; k < kParts; ++k) l += sums[k * kRows + lr];
        }
        if (!failed) {
            // Through shared memory, so that rows leave whole: results as they go to O, or fp32 as they go to scratch.
            const float scale = p.chunks > 1 ? kProbUnscale * kUngrow : l != 0.f ? kUngrow / l : 0.f;      // l and O are both 2^15 times as large here
            constexpr int kStrideH = D * 2 + 16, kStrideF = D * 4 + 16;                  // bytes; odd multiples of 16
            const uint32_t rows_s = ring + kRows * 4 * kParts;                           // behind the sums
            uint32_t v[kCols / 16][16];
#pragma unroll
            for (int q = 0; q < kCols / 16; ++q) {
#pragma unroll
                for (int e = 0; e < 16; ++e) v[q][e] = 0u;
                if (steps > 0) tmem_ld16(lanes + kColO + static_cast<uint32_t>(part_no * kCols + 16 * q), v[q]);
            }
            tmem_wait_ld();
#pragma unroll
            for (int q = 0; q < kCols / 16; ++q) {
                float f[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    asm volatile("" : "+r"(v[q][e]));
                    f[e] = __uint_as_float(v[q][e]) * scale;
                }
                const int c = part_no * kCols + 16 * q;
                if (p.chunks == 1) {
#pragma unroll
                    for (int e = 0; e < 16; e += 8)
                        sts128(rows_s + lr * kStrideH + (c + e) * 2,
                               make_uint4(pack_h2(f[e], f[e + 1]), pack_h2(f[e + 2], f[e + 3]), pack_h2(f[e + 4], f[e + 5]), pack_h2(f[e + 6], f[e + 7])));
                } else {
#pragma unroll
                    for (int e = 0; e < 16; e += 4)
                        sts128(rows_s + lr * kStrideF + (c + e) * 4,
                               make_uint4(__float_as_uint(f[e]), __float_as_uint(f[e + 1]), __float_as_uint(f[e + 2]), __float_as_uint(f[e + 3])));
                }
            }
            if (r < R && part_no == 0) {
                bool there;
                const size_t at = row_of(lr, &there);
                if (p.chunks > 1) {
                    float* part = p.part + (at * p.chunks + chunk) * (D + 2);
                    part[0] = m;
                    part[1] = l * kProbUnscale;
                } else if (p.LSE) {
                    p.LSE[at] = m + logf(fmaxf(l * kProbUnscale, 1e-30f));
                }
            }
            row_wait(static_cast<uint32_t>(steps + 1) & 1u);
            if (!failed) {
#pragma unroll
                for (int u = 0; u < kTurns; ++u) {
                    const int lrow = my_row0 + u * kRowsAtOnce;
                    if (!rows_live[u]) continue;
                    if (p.chunks > 1) {
                        float* part = p.part + (static_cast<size_t>(rows_at[u]) * p.chunks + chunk) * (D + 2) + 2;
#pragma unroll
                        for (int x = 0; x < 2; ++x) {
                            const int c = (x * kLanes + piece) * 4;
                            const uint4 w = lds128(rows_s + lrow * kStrideF + c * 4);
                            reinterpret_cast<uint2*>(part + c)[0] = make_uint2(w.x, w.y);
                            reinterpret_cast<uint2*>(part + c)[1] = make_uint2(w.z, w.w);
                        }
                        continue;
                    }
                    const uint4 w = lds128(rows_s + lrow * kStrideH + piece * 16);
                    __half* dst = p.O + static_cast<size_t>(rows_at[u]) * D + piece * 8;
                    if (p.o_vec) {
                        *reinterpret_cast<uint4*>(dst) = w;
                    } else {
                        const uint32_t o[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                        for (int e = 0; e < 8; ++e) reinterpret_cast<uint16_t*>(dst)[e] = static_cast<uint16_t>(o[e / 2] >> (16 * (e & 1)));
                    }
                }
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
