// Dense fp16 / bf16 GEMM on the sm_100a tensor cores: C[M,N] = alpha * A[M,K] . op(B) + beta * C, 16-bit
// storage, fp32 accumulation - the case of tc_gemm that the fused-norm callers and a prefill of
// dequantised weights use (include/tensorcore/gemm.h:16-58; arithmetic lib/ops/gemm_cpu.cpp:544-568,
// which adds the products in k order; here the tensor core's order, same fp32 accumulation).
//
//   * One CTA per SM walks the tiles of C (128 or 256 rows x 64 to 256 columns), each over the whole K, 64
//     at a time, through a ring of stages that keeps running across tiles; two sets of accumulators in
//     tensor memory where they fit, so that one tile is read out and stored while the next one's MMAs
//     run.  What bounds the K loop is what an SM takes in from L2, 64 bytes a clock.  Clock stamps of a CTA, clocks per
//     64 of K (bytes it copies / tensor work): 256 x 160 860 (53 KB, 832 clocks / 640), 128 x 64 382 (24.6 KB, 384 / 216),
//     256 x 256 1023 (65.5 KB, 1024 / 1024).  With few rows of A the waits and the issue of a K step are the bound, so a
//     stage then holds several.  512 x 11008 x 4096 (256 x 160), inputs in HBM: 5500 clocks to the first operands, 54,800
//     for 64 steps, 3700 for the last MMAs and the read-out, which nothing hides.
//   * The issuing lane runs its loop alone, and the rows of a tile are a constant of the instance: a wait of the
//     whole warp at each stage and a branch between MMAs cost 70 clocks a stage and more (whole calls,
//     512 x 4096 x 11008 78.4 -> 55.8 us, 1024 x 4096 x 4096 47.9 -> 37.6, 512 x 11008 x 4096 51.5 -> 48.9).
//   * Operands reach shared memory by tiled TMA copies of 128-byte rows written with the 128-byte
//     swizzle, the layout the MMA's shared-memory descriptors read directly:
//       - A ([M][K]) and a transposed B ([N][K]) are K-major: a box of 64 k x 128 (or BN) rows;
//         8-row groups 1024 bytes apart, a K step of 16 elements 32 bytes further along the row.
//       - B as given ([K][N], N contiguous) is MN-major: boxes of 64 n x 64 k, one per 64 columns,
//         8192 bytes apart; 8 k are 1024 bytes, a K step of 16 is 2048 bytes.  A transposed
//         ([K][M]) is loaded the same way.
//     (Which of the descriptor's two strides is which was settled on the device: for the swizzled
//     MN-major form the first is the stride along N, the second the one along K; for the K-major
//     form the second is the stride between 8-row groups and the first is not used.)
//   * That lane issues tcgen05.mma (M128 x N64..256 x K16, kind::f16, both operands from shared
//     memory) into BN columns of tensor memory per 128 rows; tcgen05.commit hands the stage back to the producer.
//   * Four warps per 128 rows read the accumulators (one TMEM lane = one row of the tile per thread), apply
//     alpha and beta and store 16-bit results, 64 bytes of eight rows a store: threads exchange pieces by shuffles.
//     (16 bytes of 32 rows took the load/store unit a clock a row: whole calls, 512 x 11008 x 4096 54.1 -> 49.8 us,
//     512 x 12288 x 512 23.8 -> 20.9, 4096^3 109.4 -> 105.8, 512 x 11008 x 4096 with B as given 53.0 -> 47.4.)
// Rows and columns past M, N and K are zero-filled by TMA and masked at the store.  Every wait is
// bounded: it sets the error word and lets the kernel end.
#include "kernels.h"
#include "sm100_prims.cuh"
#include "tensor_map.h"

#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace tcb {
namespace {

using namespace sm100;

constexpr int kBM = 128, kBK = 64;
constexpr int kMaxStages = 12;   // the ring is as deep as shared memory allows, up to this
constexpr int kGemmThreads = 10 * 32;         // producer, MMA issuer, four epilogue warps per 128 rows of the tile
constexpr int kGemmBarBytes = 1024;
constexpr uint32_t kGemmTmemCols = 512;      // two accumulators of up to 256 columns
constexpr uint32_t kSwizzle128 = 2;           // layout type of the shared-memory descriptor

struct GemmParams {
    __half* C;
    uint32_t* err;
    int M, N, K, ldc;
    int mt;            // rows of a tile in units of 128: 1 or 2
    int accs;          // accumulator sets: 2 where tensor memory has room
    int bn;            // columns of a tile: multiple of 16 (of 64 when B is MN-major), at most 256
    float alpha, beta;
    int b_kmajor;      // B was given transposed ([N][K])
    int a_mnmajor;     // A was given transposed ([K][M])
    int bf16;          // operands and result are bfloat16 (else binary16)
    // Bytes one stage's copy of A delivers.  With fewer than 128 rows of A (given row-major) the box
    // holds only the rows there are, rounded up to the 8-row swizzle atom: the tile's other rows stay
    // whatever shared memory held, and feed accumulator rows that the epilogue never stores.
    uint32_t a_tx;
    uint32_t a_stage;  // bytes between the stages of the A ring (a_tx rounded to the 1024-byte swizzle atom)
    int stages;        // ring depth: a stage's copy takes about 1.4 us to land, so a call that streams B
                       // with few rows of A needs many stages in flight to use the memory system
};

struct GemmBars {
    uint64_t full[kMaxStages];
    uint64_t empty[kMaxStages];
    uint64_t acc_full[2];     // MMA issuer -> epilogue warps, per accumulator
    uint64_t acc_empty[2];    // epilogue warps -> MMA issuer
    uint64_t drain;
    uint32_t tmem_base;
    int abort_flag;
};
static_assert(sizeof(GemmBars) <= kGemmBarBytes, "barrier block too large");

// Shared-memory operand descriptor with a layout type; strides in bytes.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
    return smem_desc_kmajor(saddr, lbo, sbo) | (static_cast<uint64_t>(layout) << 61);
}

__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}
// Four neighbouring threads' four pieces of 16 bytes, transposed: piece k of a thread becomes the one at its place
// among the four of thread k.
__device__ __forceinline__ void transpose_pieces(uint32_t (&h)[4][4], int lane) {
#pragma unroll
    for (int bit = 1; bit <= 2; bit <<= 1) {
        const bool upper = (lane & bit) != 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (k & bit) continue;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const uint32_t give = upper ? h[k][e] : h[k | bit][e];
                const uint32_t got = __shfl_xor_sync(0xffffffffu, give, bit);
                if (upper) h[k][e] = got;
                else h[k | bit][e] = got;
            }
        }
    }
}

// KS: 64-wide K slices per stage.  MT: rows of a tile in units of 128; fixed for each instance, because a branch
// between two MMAs costs the issuing thread more than the MMA (4096^3 in 128 x 256 tiles 134 us with MT a run-time
// value, 121 with a constant).
// WIDE: results leave by 64-byte pieces of rows.  Up to kNarrowRows rows most lanes of a store have no row anyway, and an
// instance without that code (36 to 62 registers, not 63) is faster: raw norm + GEMM calls back to back, wide / narrow, 8 x
// 4592 x 4000 20.2 / 18.7 us, 27 x 8096 x 640 26.7 / 24.7; on average narrow takes 0.980 / 0.993 / 0.985 / 0.990 / 0.998 of
// the time up to 8 / 16 / 32 / 48 / 64 rows (200 shapes), 0.998 from 65 to 128.
constexpr int kNarrowRows = 64;
template <int KS, int MT, bool WIDE>
__global__ void __launch_bounds__(kGemmThreads, 1)
gemm_f16_tc_kernel(const GemmParams p, const __grid_constant__ CUtensorMap amap, const __grid_constant__ CUtensorMap bmap) {
    const int BN = p.bn;
    constexpr int tile_rows = kBM * MT;
    const int kBSlice = BN * kBK * 2, kBStage = KS * kBSlice;
    const uint32_t a_slice = p.a_stage / KS;
    extern __shared__ __align__(1024) uint8_t smem[];
    GemmBars* bars = reinterpret_cast<GemmBars*>(smem);
    volatile int* abort_flag = &bars->abort_flag;
    uint8_t* a_ring = smem + kGemmBarBytes;
    const int stages = p.stages;
    const uint32_t a_stage = p.a_stage;
    uint8_t* b_ring = a_ring + stages * a_stage;
    // The warp number by shuffle and an elected lane for copies, MMAs and commits, so that the compiler has their
    // operands as uniform values: under `lane == 0` an MMA took 70 to 112 clocks to issue, as long as the tensor
    // core works on a 256-wide one.
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int ksteps = (p.K + kBK * KS - 1) / (kBK * KS);
    // Tiles of C, numbered column-block-major (the CTAs running at the same time share a block of B's
    // columns and walk down A); CTA c takes tiles c, c + gridDim.x, ...
    const int tiles_m = (p.M + tile_rows - 1) / tile_rows, tiles_n = (p.N + BN - 1) / BN;
    const int n_tiles = tiles_m * tiles_n;

    if (tid == 0) {
        for (int i = 0; i < stages; ++i) { bar_init(&bars->full[i], 1); bar_init(&bars->empty[i], 1); }
        for (int i = 0; i < 2; ++i) { bar_init(&bars->acc_full[i], 1); bar_init(&bars->acc_empty[i], 4 * MT); }
        bar_init(&bars->drain, 1);
        bars->abort_flag = 0;
        fence_barrier_init();
        prefetch_tensormap(&amap);
        prefetch_tensormap(&bmap);
    }
    if (warp == 1) tmem_alloc(&bars->tmem_base, kGemmTmemCols);     // two accumulators: a tile's epilogue overlaps the next tile's MMAs
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = bars->tmem_base;
    bool failed = false;

    if (warp == 0) {
        int issued = 0, s = 0;
        uint32_t par = 0;
        for (int t = blockIdx.x; t < n_tiles && !failed; t += gridDim.x) {
            const int m0 = (t % tiles_m) * tile_rows, n0 = (t / tiles_m) * BN;
            for (int ks = 0; ks < ksteps; ++ks) {
                if (!wait_all(&bars->empty[s], par ^ 1u, abort_flag)) { failed = true; break; }
                if (elect_one()) {
                    bar_expect_tx(&bars->full[s], p.a_tx + kBStage);
                    // K-major operands: a box per slice of 64 k; MN-major ones ([K][M], B as given): boxes of 64 m (n) x
                    // KS * 64 k.  What lies past K reads as zeros.
                    if (p.a_mnmajor) {
                        for (int c = 0; c < 2 * MT; ++c)
                            tensor_load_2d(a_ring + s * a_stage + c * KS * 8192, &amap, m0 + 64 * c, ks * KS * kBK, &bars->full[s]);
                    } else {
#pragma unroll
                        for (int sl = 0; sl < KS; ++sl)
                            tensor_load_2d(a_ring + s * a_stage + sl * a_slice, &amap, (ks * KS + sl) * kBK, m0, &bars->full[s]);
                    }
                    if (!p.b_kmajor) {
                        for (int c = 0; c < BN / 64; ++c)
                            tensor_load_2d(b_ring + s * kBStage + c * KS * 8192, &bmap, n0 + 64 * c, ks * KS * kBK, &bars->full[s]);
                    } else {
#pragma unroll
                        for (int sl = 0; sl < KS; ++sl)
                            tensor_load_2d(b_ring + s * kBStage + sl * kBSlice, &bmap, (ks * KS + sl) * kBK, n0, &bars->full[s]);
                    }
                }
                __syncwarp();
                ++issued;
                if (++s == stages) { s = 0; par ^= 1u; }
            }
        }
        if (failed || *abort_flag) {
            // Let copies already in flight land before the CTA's shared memory is released.
            const int first = issued > stages ? issued - stages : 0;
            for (int c = first; c < issued; ++c)
                bar_wait(&bars->full[c % stages], static_cast<uint32_t>(c / stages) & 1u, nullptr, 100000000LL);
        }
    } else if (warp == 1) {
        // bit 16: B is MN-major; bits 7-9 and 10-12: operand formats (0 binary16, 1 bfloat16)
        const uint32_t idesc = idesc_f16_f32(kBM, BN) | (p.b_kmajor ? 0u : (1u << 16)) | (p.a_mnmajor ? (1u << 15) : 0u) |
                               (p.bf16 ? ((1u << 7) | (1u << 10)) : 0u);
        // descriptor strides, and how far a K step of 16 moves along (in the descriptor's 16-byte units)
        const uint64_t a_form = p.a_mnmajor ? smem_desc(0, 8192u * KS, 1024u, kSwizzle128) : smem_desc(0, 16u, 1024u, kSwizzle128);
        const uint64_t b_form = p.b_kmajor ? smem_desc(0, 16u, 1024u, kSwizzle128) : smem_desc(0, 8192u * KS, 1024u, kSwizzle128);
        const uint32_t a_step = p.a_mnmajor ? 128u : 2u, b_step = p.b_kmajor ? 2u : 128u;
        // ... and a slice of 64; the second 128 rows lie 128 rows of a slice, or two boxes, further on
        const uint32_t a_next = p.a_mnmajor ? 512u : a_slice >> 4, b_next = p.b_kmajor ? static_cast<uint32_t>(kBSlice) >> 4 : 512u;
        const uint32_t a_half = p.a_mnmajor ? 1024u * KS : 1024u;
        if (elect_one()) {
            int s = 0;
            uint32_t par = 0;
            uint32_t acc_par = 0;
            for (int t = blockIdx.x, acc = 0; t < n_tiles && !failed; t += gridDim.x) {
                // the accumulator's previous tile has been read out
                if (!bar_wait(&bars->acc_empty[acc], acc_par ^ 1u, abort_flag)) { failed = true; break; }
                tc_fence_after_sync();
                const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(acc * MT * BN);
                for (int ks = 0; ks < ksteps; ++ks) {
                    if (!bar_wait(&bars->full[s], par, abort_flag)) { failed = true; break; }
                    tc_fence_after_sync();
                    const uint64_t adesc = a_form | ((s_u32(a_ring + s * a_stage) >> 4) & 0x3FFFu);
                    const uint64_t bdesc = b_form | ((s_u32(b_ring + s * kBStage) >> 4) & 0x3FFFu);
#pragma unroll
                    for (int sl = 0; sl < KS; ++sl) {
#pragma unroll
                        for (int j = 0; j < kBK / 16; ++j) {
                            const uint64_t ad = adesc + static_cast<uint64_t>(sl * a_next + j * a_step);
                            const uint64_t bd = bdesc + static_cast<uint64_t>(sl * b_next + j * b_step);
                            const uint32_t add = (ks > 0 || sl > 0 || j > 0) ? 1u : 0u;
                            mma_f16_ss(d_tmem, ad, bd, idesc, add);
                            if (MT == 2) mma_f16_ss(d_tmem + BN, ad + a_half, bd, idesc, add);
                        }
                    }
                    mma_commit(&bars->empty[s]);
                    if (ks + 1 == ksteps) mma_commit(&bars->acc_full[acc]);
                    if (++s == stages) { s = 0; par ^= 1u; }
                }
                if (++acc == p.accs) { acc = 0; acc_par ^= 1u; }
            }
            if (failed || *abort_flag) {
                // every MMA issued so far has completed before the tensor memory is released
                mma_commit(&bars->drain);
                bar_wait(&bars->drain, 0, nullptr, 100000000LL);
            }
        }
    }
    if (failed) {
        *abort_flag = 1;
        if (p.err) atomicOr(p.err, ERR_WAIT_TIMEOUT);
    }
    __syncwarp();

    if (warp >= 2 && warp < 2 + 4 * MT) {
        const int quad = warp & 3;                          // the TMEM lanes this warp may read
        const int half = warp >= 6 ? 1 : 0;                 // which 128 rows of the tile
        const bool vec = (p.ldc % 8 == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15u) == 0) && p.beta == 0.f;
        uint32_t acc_par = 0;
        for (int t = blockIdx.x, acc = 0; t < n_tiles; t += gridDim.x) {
            const int m0 = (t % tiles_m) * tile_rows + half * kBM, n0 = (t / tiles_m) * BN;
            const int row = m0 + quad * 32 + lane;
            const bool ok = bar_wait_warp(&bars->acc_full[acc], acc_par, abort_flag) &&
                            __all_sync(0xffffffffu, !*abort_flag);
            if (!ok) {
                if (lane == 0 && !*abort_flag) {
                    *abort_flag = 1;
                    if (p.err) atomicOr(p.err, ERR_WAIT_TIMEOUT);
                }
                break;
            }
            tc_fence_after_sync();
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16) + static_cast<uint32_t>((acc * MT + half) * BN);
            int c0 = 0;
            if (WIDE && vec) {
                // 32 columns at a time: a thread has 64 bytes of its row, and groups of four threads exchange 16-byte pieces
                // so that each store writes 64 bytes of eight rows, not 16 of 32.
                const int group_row = row - (lane & 3), piece = lane & 3;
#pragma unroll 1
                for (; c0 + 32 <= BN && n0 + c0 + 32 <= p.N; c0 += 32) {
                    uint32_t v[16], w[16], h[4][4];
                    tmem_ld16(taddr + c0, v);
                    tmem_ld16(taddr + c0 + 16, w);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        asm volatile("" : "+r"(v[e]), "+r"(w[e]));
                        const float f0 = p.alpha * __uint_as_float(e < 8 ? v[2 * (e & 7)] : w[2 * (e & 7)]);
                        const float f1 = p.alpha * __uint_as_float(e < 8 ? v[2 * (e & 7) + 1] : w[2 * (e & 7) + 1]);
                        h[e / 4][e % 4] = p.bf16 ? pack_bf16(f0, f1) : pack_f16(f0, f1);
                    }
                    transpose_pieces(h, lane);
                    __half* out = p.C + static_cast<size_t>(group_row) * p.ldc + n0 + c0 + 8 * piece;
#pragma unroll
                    for (int k = 0; k < 4; ++k, out += p.ldc)
                        if (group_row + k < p.M) *reinterpret_cast<uint4*>(out) = make_uint4(h[k][0], h[k][1], h[k][2], h[k][3]);
                }
            }
#pragma unroll 1
            for (; c0 < BN; c0 += 16) {
                uint32_t v[16];
                tmem_ld16(taddr + c0, v);
                tmem_wait_ld();
                if (row < p.M && n0 + c0 < p.N) {
                    __half* crow = p.C + static_cast<size_t>(row) * p.ldc + n0 + c0;
                    if (vec && n0 + c0 + 16 <= p.N) {
                        uint32_t h[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) {
                            const float f0 = p.alpha * __uint_as_float(v[2 * e]), f1 = p.alpha * __uint_as_float(v[2 * e + 1]);
                            h[e] = p.bf16 ? pack_bf16(f0, f1) : pack_f16(f0, f1);
                        }
                        reinterpret_cast<uint4*>(crow)[0] = make_uint4(h[0], h[1], h[2], h[3]);
                        reinterpret_cast<uint4*>(crow)[1] = make_uint4(h[4], h[5], h[6], h[7]);
                    } else {
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            if (n0 + c0 + e >= p.N) break;
                            float f = p.alpha * __uint_as_float(v[e]);
                            if (p.bf16) {
                                __nv_bfloat16* cb = reinterpret_cast<__nv_bfloat16*>(crow);
                                if (p.beta != 0.f) f += p.beta * __bfloat162float(cb[e]);
                                cb[e] = __float2bfloat16_rn(f);
                            } else {
                                if (p.beta != 0.f) f += p.beta * __half2float(crow[e]);
                                crow[e] = __float2half_rn(f);
                            }
                        }
                    }
                }
            }
            // the accumulator may take the tile after next
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->acc_empty[acc]);
            if (++acc == p.accs) { acc = 0; acc_par ^= 1u; }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kGemmTmemCols);
    }
}

cudaError_t launch_tile(const GemmParams& p, const void* A, const void* B, int lda, int ldb, bool transpose_b,
                        const LaunchEnv& env, cudaStream_t stream) {
    const bool transpose_a = p.a_mnmajor != 0;
    const int BN = p.bn;
    CUtensorMap amap, bmap;
    // A decode batch or a short prefill block has far fewer than 128 rows: copying only those (2 KB
    // instead of 16 KB a stage at 16 rows) leaves the SM's copy bandwidth to B, which is what such a
    // call streams.
    const int tile_rows = kBM * p.mt;
    const int a_rows = (!transpose_a && p.M < tile_rows) ? ((p.M + 7) & ~7) : tile_rows;
    GemmParams q = p;
    q.a_tx = static_cast<uint32_t>(a_rows) * kBK * 2u;
    // Several 64-wide slices per stage while four stages still fit: a stage's barriers and waits cost more than the
    // MMAs of a slice when the tile is small (16 x 4096 x 4096: 590 clocks a slice with one per stage, 420
    // with four; the kernel 27.7 -> 21.1 us).  Any K and leading dimension: what a last stage holds past K is zeros
    // (16 x 9672 x 5136, K not of whole slices: a call 43.7 us with one slice per stage, 39.2 with four).
    int ks = 1;
    const int slice_bytes = static_cast<int>(q.a_tx) + BN * kBK * 2;
    while (ks < 4 && p.K >= 2 * ks * kBK && 4 * 2 * ks * slice_bytes <= env.smem_optin - kGemmBarBytes)
        ks *= 2;
    q.a_tx *= static_cast<uint32_t>(ks);
    q.a_stage = q.a_tx;     // a multiple of 1024: a_rows is a multiple of 8 rows of 128 bytes
    const int stage_bytes = ks * slice_bytes;
    q.stages = (env.smem_optin - kGemmBarBytes) / stage_bytes;
    if (q.stages > kMaxStages) q.stages = kMaxStages;
    if (q.stages < 2) return cudaErrorNotSupported;
    const int smem = kGemmBarBytes + q.stages * stage_bytes;
    const bool oka = transpose_a
        ? encode_rows_sw128(&amap, A, static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.M), static_cast<uint64_t>(lda), kBK * ks)
        : encode_rows_sw128(&amap, A, static_cast<uint64_t>(p.M), static_cast<uint64_t>(p.K), static_cast<uint64_t>(lda), a_rows);
    if (!oka) return cudaErrorNotSupported;
    const bool okb = !transpose_b
        ? encode_rows_sw128(&bmap, B, static_cast<uint64_t>(p.K), static_cast<uint64_t>(p.N), static_cast<uint64_t>(ldb), kBK * ks)
        : encode_rows_sw128(&bmap, B, static_cast<uint64_t>(p.N), static_cast<uint64_t>(p.K), static_cast<uint64_t>(ldb), BN);
    if (!okb) return cudaErrorNotSupported;
    const long tiles = static_cast<long>((p.N + BN - 1) / BN) * ((p.M + tile_rows - 1) / tile_rows);
    const long sms = env.sm_count > 0 ? env.sm_count : 148;
    const dim3 grid(static_cast<unsigned>(tiles < sms ? tiles : sms));     // one CTA per SM walks the tiles
    const bool wide = p.mt == 2 || p.M > kNarrowRows;
    auto* kernel = p.mt == 2 ? (ks == 4 ? gemm_f16_tc_kernel<4, 2, true> : ks == 2 ? gemm_f16_tc_kernel<2, 2, true> : gemm_f16_tc_kernel<1, 2, true>)
                   : wide    ? (ks == 4 ? gemm_f16_tc_kernel<4, 1, true> : ks == 2 ? gemm_f16_tc_kernel<2, 1, true> : gemm_f16_tc_kernel<1, 1, true>)
                             : (ks == 4 ? gemm_f16_tc_kernel<4, 1, false> : ks == 2 ? gemm_f16_tc_kernel<2, 1, false> : gemm_f16_tc_kernel<1, 1, false>);
    kernel<<<grid, (2 + 4 * p.mt) * 32, smem, stream>>>(q, amap, bmap);
    return cudaGetLastError();
}

}  // namespace

cudaError_t init_gemm_tc_kernel(int smem_optin) {
    for (auto* k : {gemm_f16_tc_kernel<1, 1, true>, gemm_f16_tc_kernel<2, 1, true>, gemm_f16_tc_kernel<4, 1, true>, gemm_f16_tc_kernel<1, 1, false>,
                    gemm_f16_tc_kernel<2, 1, false>, gemm_f16_tc_kernel<4, 1, false>, gemm_f16_tc_kernel<1, 2, true>, gemm_f16_tc_kernel<2, 2, true>,
                    gemm_f16_tc_kernel<4, 2, true>}) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// cudaErrorNotSupported when the operands are outside what the tiled copies can describe: the leading
// dimensions must be multiples of 8 elements and the bases 16-byte aligned.
cudaError_t launch_gemm_f16_tc(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                               bool transpose_b, float alpha, float beta, const LaunchEnv& env, cudaStream_t stream,
                               bool bf16, bool transpose_a) {
    if (M <= 0 || N <= 0 || K <= 0 || lda % 8 || ldb % 8) return cudaErrorNotSupported;
    if ((reinterpret_cast<uintptr_t>(A) & 15u) || (reinterpret_cast<uintptr_t>(B) & 15u)) return cudaErrorNotSupported;
    GemmParams p{};
    p.C = static_cast<__half*>(C);
    p.err = env.err_word;
    p.M = M; p.N = N; p.K = K; p.ldc = ldc;
    p.alpha = alpha; p.beta = beta;
    p.b_kmajor = transpose_b ? 1 : 0;
    p.bf16 = bf16 ? 1 : 0;
    p.a_mnmajor = transpose_a ? 1 : 0;
    // Tile: the one whose rounds over the SMs take least, by a model of a 64-wide K step and of what a tile costs
    // beside its steps.  A step is four MMAs of N / 2 clocks per 128 rows, each at least 54 (the measured floor with
    // both operands in shared memory), or its traffic, counted as the stage's bytes written once, A read
    // once and B once per 128 rows, at 120 bytes per clock (a form that was fitted; the header says what the traffic is).  256 rows need less traffic per flop; their two
    // accumulators leave room for a second set only up to 128 columns, so a wider tile's read-out is not hidden:
    // 10000 clocks a round, against 1500 per 128 rows where it is (3000 to 7000 choose worse tiles: 256 x 14336 x 4096
    // 47 us instead of 44.5, 2048^3 30 instead of 28.7).  Fitted to whole calls of 144 shapes (M 64 to
    // 8192, K 1024 to 11008) in eight tiles each: a step of 128 rows x 64 / 128 / 192 / 256 columns takes 180 / 270 /
    // 300 / 373 ns, of 256 rows x 128 / 192 / 256 365 / 460 / 635 ns; the tile chosen is 0.3 % slower than the
    // best of the eight on average, 9 % at most.  B as given is laid out in pieces of 64 columns.
    const long sms = env.sm_count > 0 ? env.sm_count : 148;
    const long ksteps = (K + kBK - 1) / kBK;
    double best = 0.0;
    for (int mt = 1; mt <= (M > kBM ? 2 : 1); ++mt) {
        const long rows = kBM * mt, tiles_m = (M + rows - 1) / rows;
        const long a_bytes = (transpose_a || M >= rows ? rows : ((M + 7) & ~7)) * kBK * 2L;
        for (int bn = 256; bn >= 64; bn -= transpose_b ? 16 : 64) {
            const long tiles = tiles_m * ((N + bn - 1) / bn), rounds = (tiles + sms - 1) / sms;
            const int accs = 2 * mt * bn <= static_cast<int>(kGemmTmemCols) ? 2 : 1;
            const double mma = 4.0 * mt * (bn > 108 ? bn / 2.0 : 54.0), traffic = (a_bytes + bn * kBK * 2L + mt * (kBM + bn) * kBK * 2L) / 120.0;
            const double cost = static_cast<double>(rounds) * (ksteps * (mma > traffic ? mma : traffic) + (accs == 1 ? 10000.0 : 1500.0 * mt));
            if (best == 0.0 || cost < best) { best = cost; p.bn = bn; p.mt = mt; p.accs = accs; }
        }
    }
    return launch_tile(p, A, B, lda, ldb, transpose_b, env, stream);
}

}  // namespace tcb
