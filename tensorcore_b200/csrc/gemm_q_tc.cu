// Quantized GEMV / GEMM for five activation rows or more on the sm_100a tensor cores (tcgen05):
//
//   Y[m][n] = sum_k X[m][k] * dequant(W)[n][k],   Q4_0 or Q8_0 blocks, fp16 X, any number of rows.
//
// The reference computes this as independent dequant-dots per output element, re-reading the weights
// for every activation row (lib/ops/quantized_cpu.cpp:193-228).  Here the packed weights are read
// once per tile of up to 256 activation rows and never exist as fp16 in memory:
//
//   * Up to four matrices that share their activations (q, k and v; gate and up) are one launch.
//   * A CTA owns 128 weight rows x NB activation rows (NB = 16 .. 256, the MMA's N) and a K range; a
//     cluster of up to 8 CTAs shares a tile along K when there are fewer tiles than SMs.  The unit of
//     work is one group of 8 blocks (256 weights) of the 128 rows: a single tiled TMA copy of 128 rows
//     x 144 (Q4_0) or 272 (Q8_0) raw bytes into a ring.
//   * Four dequantising warpgroups (two with more than 64 columns) take the units in turn, one thread per
//     weight row.  A thread turns 64 weights (two blocks) at a time into fp16 q * d - the zero point
//     subtracted exactly, one rounding, the same value a dequantised copy would hold - in natural K order,
//     and stores them with tcgen05.st into its own TMEM lane: the MMA's A operand (128 lanes = 128
//     weight rows) lives in tensor memory, in slots of 32 columns (two to four per warpgroup), so that
//     a warpgroup fills one slot while the MMAs read the other.
//   * Activations arrive as plain 128-byte-swizzled K-major tiles by TMA (natural K order needs no
//     shuffling by threads); rows past M read as zeros.
//   * One issuing warp per accumulator: tcgen05.mma M128 x NB x K16, fp32 accumulate.  With up to 64 columns four
//     warps issue, each for one warpgroup into an accumulator of its own, with 128 columns two, with 256
//     columns (128 clocks of tensor work per MMA) one; the accumulators are added in the epilogue in a
//     fixed order.  An MMA takes 39 clocks to issue (N up to 64; 66 and 130 at 128 and 256), so the 16 of a
//     unit are 624 of the 970 clocks a unit takes at 8 rows: two issuers might do.  Four date from an MMA that
//     took 112 clocks, and fewer have not been measured.
//   * Epilogue: tcgen05.ld, then a direct store, or with a K split a fixed-order sum over the cluster
//     through distributed shared memory.  Results do not depend on timing.
//
// What bounds it: up to about 64 rows the weight stream and the dequantising instructions (14 per
// eight Q4_0 weights, issued by 16 warps; the zero point and the scale cannot be one fused
// multiply-add because 1032 d does not fit fp16), from 128 rows on the tensor pipe.
// Back to back on a stream, weights from HBM, against the kernel of 256-row tiles with separate
// activation staging (Q4_0 up to 95 rows) and the dequantised copy plus GEMM (the others) before it:
//   Q4_0 14336 x 4096   32 rows  22.0 -> 11.8 us (2.8 TB/s)    512 rows  95 -> 53 us (1130 TFLOP/s)
//   Q8_0 11008 x 4096   16 rows  51 -> 15.3 us (3.1 TB/s)
// Per 128-row unit of 256 weights in steady state: Q4_0 0.51 us at 8 rows, 1.9 us at 256 rows (1.08 us
// of tensor work at the clock's peak); Q8_0 0.82 us at 16 rows, which is the weight stream at 6.3 TB/s.
#include "kernels.h"
#include "sm100_prims.cuh"
#include "tensor_map.h"

#include <cuda.h>
#include <cuda_fp16.h>

#include <atomic>
#include <cstdlib>
#include <type_traits>

namespace tcb {
namespace {

using namespace sm100;

constexpr int kRows = 128;                 // weight rows per CTA = TMEM lanes
constexpr int kWgs = 4;                    // dequantising warpgroups
constexpr int kDqWarps = 4 * kWgs;
constexpr int kRawWarp = kDqWarps;         // raw weight copies, TMEM allocation
constexpr int kXWarp = kDqWarps + 1;       // activation copies
constexpr int kMmaWarp = kDqWarps + 2;     // four issuers
constexpr int kThreads = (kDqWarps + 2 + 4) * 32;
constexpr int kMaxRing = 12;
constexpr int kMaxSlots = 4;
constexpr int kMaxMats = 4;                // matrices that share their activations in one launch
constexpr int kSub = 64;                   // weights per row and A slot
constexpr uint32_t kTmemCols = 512;
constexpr int kBarBytes = 1024;
constexpr uint32_t kSwizzle128 = 2;        // descriptor layout type

struct QtcParams {
    void* Y[kMaxMats];
    int N[kMaxMats];
    int tile0[kMaxMats];   // first row tile of each matrix (INT_MAX past the last)
    uint32_t* err;
    int M;
    int y_f32;
    int nb;            // MMA N extent: multiple of 16, <= 256
    int groups;        // K / 256
    int split;         // CTAs per tile = cluster size
    int col_tiles;     // tiles of nb activation rows
    int tile_base;     // first tile of this launch
    int wait_first;    // the kernel before may write the weights
    int raw_stages;    // per warpgroup (a ring that several groups shared would let one wait on a
                       // barrier phase while an earlier one, which it never observes, is still open)
    int x_stages;      // per issuer
    int off_raw, off_x;
};

struct QtcMaps { CUtensorMap w[kMaxMats], x; };

struct Bars {
    uint64_t raw_full[kMaxRing], raw_empty[kMaxRing];
    uint64_t x_full[kMaxRing], x_empty[kMaxRing];
    uint64_t a_full[kWgs][kMaxSlots], a_empty[kWgs][kMaxSlots];
    uint64_t d_full;
    uint32_t tmem_base;
    int abort_flag;
    int sent[2 * kMaxRing];      // copies issued per stage, for the producers' own clean-up
};
static_assert(sizeof(Bars) <= kBarBytes, "barrier block too large");

template <int FMT> struct QFmt;
template <> struct QFmt<FMT_Q4_0> { static constexpr int kBlock = 18, kGroup = 144, kVec = 3, kElem = 1; };
template <> struct QFmt<FMT_Q8_0> { static constexpr int kBlock = 34, kGroup = 272, kVec = 5, kElem = 4; };

__device__ __forceinline__ uint32_t h2_bits(__half2 v) { return *reinterpret_cast<uint32_t*>(&v); }
__device__ __forceinline__ __half2 bits_h2(uint32_t v) { return *reinterpret_cast<__half2*>(&v); }
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t mask, uint32_t bits) {
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(r) : "r"(a), "r"(mask), "r"(bits));
    return r;
}

// A block whose first byte is byte O of the held words: 16 fp16 pairs in K order.  Blocks start at
// even bytes, so a pair of neighbouring quants never straddles a word.
// A nibble ORed into the mantissa of 1024.0 (bits 0-3) or of 64.0 (bits 4-7), or a biased byte ORed
// into 1024.0, is that constant plus the value exactly; the subtraction leaves q exactly.
template <int FMT, int O, int NW>
__device__ __forceinline__ void dequant_block(const uint32_t (&g)[NW], uint32_t (&out)[16]) {
    const __half2 d2 = bits_h2(__byte_perm(g[O / 4], 0, (O & 2) ? 0x3232 : 0x1010));
    if constexpr (FMT == FMT_Q4_0) {
        const __half2 c_lo = bits_h2(0x64086408u);   // 1032
        const __half2 c_hi = bits_h2(0x54805480u);   // 72
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int at = O + 2 + 2 * i;
            const uint32_t v = __byte_perm(g[at / 4], 0, (at & 2) ? 0x4342 : 0x4140);
            out[i] = h2_bits(__hmul2(__hsub2(bits_h2(and_or(v, 0x000F000Fu, 0x64006400u)), c_lo), d2));
            out[8 + i] = h2_bits(__hmul2(__hsub2(bits_h2(and_or(v, 0x00F000F0u, 0x54005400u)), c_hi), d2));
        }
    } else {
        const __half2 c = bits_h2(0x64806480u);      // 1152 = 1024 + 128
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int at = O + 2 + 2 * i;
            const uint32_t u = g[at / 4] ^ 0x80808080u;
            const uint32_t v = __byte_perm(u, 0x64646464u, (at & 2) ? 0x4342 : 0x4140);
            out[i] = h2_bits(__hmul2(__hsub2(bits_h2(v), c), d2));
        }
    }
}

// Two blocks (64 weights) of quarter S of a group, from the 16-byte pieces that cover them.
template <int FMT, int S>
__device__ __forceinline__ void dequant_quarter(const uint32_t (&g)[4 * QFmt<FMT>::kVec], uint32_t taddr) {
    using F = QFmt<FMT>;
    constexpr int first = 2 * S * F::kBlock - 16 * ((2 * S * F::kBlock) / 16);   // first byte inside the pieces
    uint32_t out[16];
    dequant_block<FMT, first>(g, out);
    tmem_st16(taddr, out);
    dequant_block<FMT, first + F::kBlock>(g, out);
    tmem_st16(taddr + 16, out);
}
template <int FMT, int S>
__device__ __forceinline__ void load_quarter(uint32_t row, uint32_t (&g)[4 * QFmt<FMT>::kVec]) {
    using F = QFmt<FMT>;
    constexpr int at = 16 * ((2 * S * F::kBlock) / 16);
#pragma unroll
    for (int v = 0; v < F::kVec; ++v) {
        const uint4 t = lds128(row + at + 16 * v);
        g[4 * v] = t.x; g[4 * v + 1] = t.y; g[4 * v + 2] = t.z; g[4 * v + 3] = t.w;
    }
}

struct Pos {                                // position in a ring
    int i = 0;
    uint32_t ph = 0;
    __device__ __forceinline__ void next(int size) { if (++i == size) { i = 0; ph ^= 1u; } }
};

// I: accumulators and issuers; unit u is issued by warp u % I.  SLOTS: A slots per warpgroup.  XK: 64-wide
// K slices per activation stage.  With one or two issuers two warpgroups keep up with the MMAs.
template <int FMT, int I, int SLOTS, int XK>
__global__ void __launch_bounds__(kThreads, 1)
gemm_q_tc_kernel(const QtcParams p, const __grid_constant__ QtcMaps maps) {
    using F = QFmt<FMT>;
    constexpr int kRawBytes = kRows * F::kGroup;
    constexpr int kActive = I == 4 ? 4 : 2;          // warpgroups that dequantise
    static_assert(I == kActive || SLOTS == 4, "a slot's position follows from the unit when an issuer serves two groups");
    extern __shared__ __align__(1024) uint8_t smem[];
    Bars* bars = reinterpret_cast<Bars*>(smem);
    volatile int* abort_flag = &bars->abort_flag;
    int* sent = bars->sent;
    // The warp number by shuffle, and one elected lane inside warp-uniform control flow around every copy, MMA
    // and commit: operands then are uniform values for the compiler.  An MMA issued from under `lane == 0`
    // took 70 to 112 clocks instead of 39 (M128 x N16..64 x K16, one issuing warp).
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int split = p.split, nb = p.nb;
    const int tile = p.tile_base + blockIdx.x / split;
    const int crank = split > 1 ? static_cast<int>(cluster_ctarank()) : 0;
    const int g0 = p.groups * crank / split;
    const int n_units = p.groups * (crank + 1) / split - g0;
    const int rt = tile / p.col_tiles;
    int mat = 0, N = p.N[0], first_tile = 0;
    void* Y = p.Y[0];
#pragma unroll
    for (int i = 1; i < kMaxMats; ++i)
        if (rt >= p.tile0[i]) { mat = i; N = p.N[i]; Y = p.Y[i]; first_tile = p.tile0[i]; }
    const CUtensorMap* wmap = &maps.w[mat];
    const int row0 = (rt - first_tile) * kRows;
    const int m0 = (tile % p.col_tiles) * nb;
    uint8_t* raw_ring = smem + p.off_raw;
    uint8_t* x_ring = smem + p.off_x;
    const int x_bytes = nb * 128 * XK;

    if (!p.wait_first) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == kRawWarp * 32) prefetch_tensormap(wmap);
    if (tid == kXWarp * 32) prefetch_tensormap(&maps.x);
    if (tid == 0) {
        for (int i = 0; i < kMaxRing; ++i) {
            bar_init(&bars->raw_full[i], 1);
            bar_init(&bars->raw_empty[i], 4);        // the four warps of the warpgroup that reads it
            bar_init(&bars->x_full[i], 1);
            bar_init(&bars->x_empty[i], 1);          // commit of the issuer that read it
            sent[i] = sent[kMaxRing + i] = 0;
        }
        for (int j = 0; j < kWgs; ++j)
            for (int s = 0; s < kMaxSlots; ++s) {
                bar_init(&bars->a_full[j][s], 4);
                bar_init(&bars->a_empty[j][s], 1);
            }
        bar_init(&bars->d_full, I);
        bars->abort_flag = 0;
        fence_barrier_init();
    }
    if (warp == kRawWarp) tmem_alloc(&bars->tmem_base, kTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = bars->tmem_base;
    const uint32_t a_col0 = static_cast<uint32_t>(I * nb);      // accumulators first, then the A slots
    bool failed = false;

    if (warp < kDqWarps) {
        // ---------------- dequantisers: one thread per weight row --------------------------------------
        const int wg = warp >> 2, q = warp & 3;
        const uint32_t a_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + a_col0 + static_cast<uint32_t>(wg * SLOTS * 32);
        const uint32_t row_off = static_cast<uint32_t>(q * 32 + lane) * F::kGroup;
        Pos slot;
        Pos ring;
        for (int u = wg; u < n_units && wg < kActive && !failed; u += kActive) {
            const int st = wg + kActive * ring.i;
            if (!wait_all(&bars->raw_full[st], ring.ph, abort_flag)) { failed = true; break; }
            ring.next(p.raw_stages);
            const uint32_t row = s_u32(raw_ring + st * kRawBytes) + row_off;
            uint32_t g[4 * F::kVec];
            auto quarter = [&](auto sc) {
                constexpr int S = decltype(sc)::value;
                if (failed) return;
                load_quarter<FMT, S>(row, g);
                if (!wait_all(&bars->a_empty[wg][slot.i], slot.ph ^ 1u, abort_flag)) { failed = true; return; }
                tc_fence_after_sync();
                dequant_quarter<FMT, S>(g, a_base + static_cast<uint32_t>(slot.i * 32));
                tmem_wait_st();
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    bar_arrive(&bars->a_full[wg][slot.i]);
                    // the raw stage goes back only after every value loaded from it has been consumed by a
                    // tcgen05.st that has completed
                    if (S == 3) { fence_proxy_async(); bar_arrive(&bars->raw_empty[st]); }
                }
                slot.next(SLOTS);
            };
            quarter(std::integral_constant<int, 0>{});
            quarter(std::integral_constant<int, 1>{});
            quarter(std::integral_constant<int, 2>{});
            quarter(std::integral_constant<int, 3>{});
        }
    } else if (warp == kRawWarp) {
        // ---------------- weight producer: 128 rows x one group per unit; rows past N read as zeros -----
        if (p.wait_first) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        }
        Pos ring;
        for (int r = 0; r < n_units && !failed; r += kActive) {
#pragma unroll
            for (int j = 0; j < kActive; ++j) {
                if (r + j >= n_units) break;
                const int st = j + kActive * ring.i;
                if (!wait_all(&bars->raw_empty[st], ring.ph ^ 1u, abort_flag)) { failed = true; break; }
                if (elect_one()) {
                    bar_expect_tx(&bars->raw_full[st], kRawBytes);
                    tensor_load_2d(raw_ring + st * kRawBytes, wmap, (g0 + r + j) * (F::kGroup / F::kElem), row0, &bars->raw_full[st]);
                    sent[st] += 1;
                }
                __syncwarp();
            }
            ring.next(p.raw_stages);
        }
        if (failed || *abort_flag) {             // copies in flight land before the shared memory is released
            for (int st = 0; st < kActive * p.raw_stages; ++st)
                if (sent[st] > 0) bar_wait(&bars->raw_full[st], static_cast<uint32_t>(sent[st] - 1) & 1u, nullptr, 100000000LL);
        }
    } else if (warp == kXWarp) {
        // ---------------- activation producer, in the order the issuers consume ---------------------------
        // Activations belong to the stream's order: wait for the kernel before this one here, with
        // the weight copies already in flight where nothing that may still run writes them.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        Pos ring;
        for (int r = 0; r < n_units && !failed; r += I)
            for (int s = 0; s < 4 && !failed; s += XK) {
#pragma unroll
                for (int j = 0; j < I; ++j) {
                    if (r + j >= n_units) break;
                    const int st = j * p.x_stages + ring.i;
                    if (!wait_all(&bars->x_empty[st], ring.ph ^ 1u, abort_flag)) { failed = true; break; }
                    if (elect_one()) {
                        bar_expect_tx(&bars->x_full[st], x_bytes);
                        tensor_load_3d(x_ring + st * x_bytes, &maps.x, 0, m0, (g0 + r + j) * 4 + s, &bars->x_full[st]);
                        sent[kMaxRing + st] += 1;
                    }
                    __syncwarp();
                }
                ring.next(p.x_stages);
            }
        if (failed || *abort_flag) {
            for (int st = 0; st < I * p.x_stages; ++st)
                if (sent[kMaxRing + st] > 0)
                    bar_wait(&bars->x_full[st], static_cast<uint32_t>(sent[kMaxRing + st] - 1) & 1u, nullptr, 100000000LL);
        }
    } else if (warp - kMmaWarp < I) {
        // ---------------- MMA issue: one warp per accumulator ------------------------------------------------
        const int me = warp - kMmaWarp;
        const uint32_t idesc = idesc_f16_f32(kRows, nb);
        const uint32_t d_col = tmem_base + static_cast<uint32_t>(me * nb);
        uint32_t started = 0;
        Pos xs, slot;
        for (int u = me; u < n_units && !failed; u += I) {
            const int j = I == kActive ? me : (u & 1);             // the warpgroup that dequantises the unit
            if (I != kActive) { slot.i = 0; slot.ph = static_cast<uint32_t>(u >> 1) & 1u; }
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int sub = s % XK, st = me * p.x_stages + xs.i;
                if (sub == 0 && !wait_all(&bars->x_full[st], xs.ph, abort_flag)) { failed = true; break; }
                if (!wait_all(&bars->a_full[j][slot.i], slot.ph, abort_flag)) { failed = true; break; }
                tc_fence_after_sync();
                const uint32_t a_col = tmem_base + a_col0 + static_cast<uint32_t>((j * SLOTS + slot.i) * 32);
                const uint32_t x_addr = s_u32(x_ring + st * x_bytes) + static_cast<uint32_t>(sub * nb * 128);
                const uint64_t desc = smem_desc_kmajor(x_addr, 16u, 1024u) | (static_cast<uint64_t>(kSwizzle128) << 61);
                if (elect_one()) {
                    mma_f16_ts(d_col, a_col, desc, idesc, started);
#pragma unroll
                    for (int k = 1; k < kSub / 16; ++k)
                        mma_f16_ts_acc(d_col, a_col + 8u * k, desc + static_cast<uint64_t>(2 * k), idesc);
                    mma_commit(&bars->a_empty[j][slot.i]);
                    if (sub == XK - 1) mma_commit(&bars->x_empty[st]);
                }
                __syncwarp();
                started = 1u;
                slot.next(SLOTS);
                if (sub == XK - 1) xs.next(p.x_stages);
            }
        }
        // every MMA of this issuer; also on failure, before tensor and shared memory are released
        if (elect_one()) mma_commit(&bars->d_full);
        __syncwarp();
        if (failed || *abort_flag) bar_wait(&bars->d_full, 0, nullptr, 100000000LL);
    }

    if (failed) {
        *abort_flag = 1;
        if (p.err) atomicOr(p.err, ERR_WAIT_TIMEOUT);
    }
    __syncwarp();

    // ---------------- epilogue: warp = (TMEM quadrant, every fourth block of 16 columns) ---------------------
    float* red = reinterpret_cast<float*>(smem + p.off_x);   // [nb][128], K-split partials: every operand has been read
    if (warp < kDqWarps) {
        const int q = warp & 3;
        const bool ok = wait_all(&bars->d_full, 0, abort_flag) && __all_sync(0xffffffffu, !*abort_flag);
        if (!ok && lane == 0 && !*abort_flag) {
            *abort_flag = 1;
            if (p.err) atomicOr(p.err, ERR_WAIT_TIMEOUT);
        }
        tc_fence_after_sync();
        if (ok) {
            asm volatile("griddepcontrol.wait;" ::: "memory");   // Y may still be read by the kernel before
            const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
            const int r = q * 32 + lane, row = row0 + r;
            const int used = n_units < I ? n_units : I;      // accumulators that were written
            const int m_end = p.M - m0 < nb ? p.M - m0 : nb;
            for (int c0 = (warp >> 2) * 16; c0 < m_end; c0 += 64) {
                float f[16];
                uint32_t v[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) f[e] = 0.f;
                for (int a = 0; a < used; ++a) {
                    tmem_ld16(taddr + static_cast<uint32_t>(a * nb + c0), v);
                    tmem_wait_ld();
#pragma unroll
                    for (int e = 0; e < 16; ++e) f[e] += __uint_as_float(v[e]);
                }
                if (split > 1) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) red[(c0 + e) * kRows + r] = f[e];
                } else if (row < N) {
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        if (c0 + e >= m_end) break;
                        const size_t o = static_cast<size_t>(m0 + c0 + e) * N + row;
                        if (p.y_f32) static_cast<float*>(Y)[o] = f[e];
                        else static_cast<__half*>(Y)[o] = __float2half_rn(f[e]);
                    }
                }
            }
        }
        tc_fence_before_sync();
    }
    __syncthreads();

    if (split > 1) {
        cluster_sync_all();
        if (!*abort_flag) {
            const int r_lo = kRows * crank / split, r_hi = kRows * (crank + 1) / split;
            const int rows_c = r_hi - r_lo;
            const int m_end = p.M - m0 < nb ? p.M - m0 : nb;
            const uint32_t red_addr = s_u32(red);
            for (int e = tid; e < m_end * rows_c; e += kThreads) {
                const int m = e / rows_c, r = r_lo + e % rows_c;
                const int row = row0 + r;
                if (row >= N) continue;
                // every peer's part is asked for before the first is added: one trip across the cluster, not `split`
                float part[8];
#pragma unroll
                for (int c = 0; c < 8; ++c)
                    part[c] = c < split ? ld_cluster_f32(red_addr + static_cast<uint32_t>(m * kRows + r) * 4u, c) : 0.f;
                float acc = part[0];
#pragma unroll
                for (int c = 1; c < 8; ++c) acc += part[c];
                const size_t o = static_cast<size_t>(m0 + m) * N + row;
                if (p.y_f32) static_cast<float*>(Y)[o] = acc;
                else static_cast<__half*>(Y)[o] = __float2half_rn(acc);
            }
        }
        cluster_sync_all();   // peers may still be reading this CTA's partials
    }

    if (warp == kRawWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTmemCols);
    }
}

// How many clusters of `size` CTAs the device holds at once (every instance fills an SM's shared
// memory or tensor memory, so one CTA per SM whatever the shapes); 0 when the query fails.
int max_active_clusters(int size, int smem) {
    static std::atomic<int> cache[9] = {};
    int n = cache[size].load();
    if (n == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(size * 64);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = size;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_q_tc_kernel<FMT_Q4_0, 4, 3, 4>, &cfg) != cudaSuccess || n <= 0) {
            n = -1;
            (void)cudaGetLastError();
        }
        cache[size].store(n);
    }
    return n > 0 ? n : 0;
}

using QtcKernel = void (*)(const QtcParams, const QtcMaps);
struct QtcVariant { int max_nb, issuers, active, xk; QtcKernel kernel[2]; };
const QtcVariant kVariants[] = {
    {16, 4, 4, 4, {gemm_q_tc_kernel<FMT_Q4_0, 4, 3, 4>, gemm_q_tc_kernel<FMT_Q8_0, 4, 3, 4>}},
    {32, 4, 4, 2, {gemm_q_tc_kernel<FMT_Q4_0, 4, 3, 2>, gemm_q_tc_kernel<FMT_Q8_0, 4, 3, 2>}},
    {64, 4, 4, 1, {gemm_q_tc_kernel<FMT_Q4_0, 4, 2, 1>, gemm_q_tc_kernel<FMT_Q8_0, 4, 2, 1>}},
    {128, 2, 2, 1, {gemm_q_tc_kernel<FMT_Q4_0, 2, 4, 1>, gemm_q_tc_kernel<FMT_Q8_0, 2, 4, 1>}},
    {256, 1, 2, 1, {gemm_q_tc_kernel<FMT_Q4_0, 1, 4, 1>, gemm_q_tc_kernel<FMT_Q8_0, 1, 4, 1>}},
};

}  // namespace

cudaError_t init_gemm_q_tc_kernels(int smem_optin) {
    for (const QtcVariant& v : kVariants)
        for (QtcKernel k : v.kernel) {
            const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

// Up to kMaxMats products of the same activation rows in one launch: ops[1 ..] differ from ops[0] in W, Y and N
// only.  cudaErrorNotSupported when the operation is outside this kernel's domain.
cudaError_t launch_gemm_q_tc(const GemvQArgs* ops, int n_ops, const LaunchEnv& env, cudaStream_t stream, int* launches) {
    if (n_ops < 1 || n_ops > kMaxMats) return cudaErrorNotSupported;
    const GemvQArgs& a = ops[0];
    QtcParams p{};
    p.err = env.err_word;
    p.M = a.M;
    p.y_f32 = a.y_f32 ? 1 : 0;
    p.groups = a.K / 256;
    // Activation rows in as few equal tiles of at most 256 as there can be.
    p.col_tiles = (a.M + 255) / 256;
    p.nb = ((a.M + p.col_tiles - 1) / p.col_tiles + 15) & ~15;
    long long row_tiles = 0;
    for (int i = 0; i < kMaxMats; ++i) {
        p.tile0[i] = 0x7fffffff;
        if (i >= n_ops) continue;
        const GemvQArgs& o = ops[i];
        if (o.x_f32 || o.gamma != nullptr || (o.fmt != FMT_Q4_0 && o.fmt != FMT_Q8_0) || o.M < 1 || o.K <= 0 || o.K % 256 != 0 || o.N <= 0 ||
            (reinterpret_cast<uintptr_t>(o.W) & 15u) || (reinterpret_cast<uintptr_t>(o.X) & 15u))
            return cudaErrorNotSupported;
        p.tile0[i] = static_cast<int>(row_tiles);
        p.Y[i] = o.Y;
        p.N[i] = o.N;
        row_tiles += (o.N + kRows - 1) / kRows;
    }
    const QtcVariant* v = kVariants;
    while (v->max_nb < p.nb) ++v;
    const int raw_bytes = kRows * (a.fmt == FMT_Q4_0 ? 144 : 272), x_bytes = p.nb * 128 * v->xk;
    const long long tiles_ll = row_tiles * p.col_tiles;
    if (tiles_ll > 0x0fffffff) return cudaErrorNotSupported;
    const int tiles = static_cast<int>(tiles_ll);

    // Ring depths: two raw stages per warpgroup where at least two activation stages fit beside them (one
    // being read, one in flight), else one; activations get what is left.
    const int room = env.smem_optin - kBarBytes;
    const int min_x = (v->issuers == 1 ? 4 : 2) * v->issuers * x_bytes;
    p.raw_stages = 2 * v->active * raw_bytes + min_x <= room ? 2 : 1;
    p.x_stages = (room - p.raw_stages * v->active * raw_bytes) / (v->issuers * x_bytes);
    if (p.x_stages * v->issuers > kMaxRing) p.x_stages = kMaxRing / v->issuers;
    if (p.x_stages < 2) return cudaErrorNotSupported;
    p.off_x = kBarBytes;                               // 1024-byte aligned, as are the activation stages
    p.off_raw = p.off_x + v->issuers * p.x_stages * x_bytes;
    const int smem = p.off_raw + v->active * p.raw_stages * raw_bytes;
    const int red_bytes = p.nb * kRows * 4;

    // K is split over a cluster when there are fewer tiles than SMs: the largest cluster size whose
    // clusters can all be resident at once, so that the split shortens the K loop instead of queueing, and
    // whose CTAs keep a unit for each of four warpgroups (8 rows, split 1 / 2 / 4 / 8: 4096 x 1024 3.4 / 4.5 /
    // 6.2 us, 4096 x 2048 5.1 / 5.0 / 6.5, 2048 x 4096 - / 6.5 / 4.7 / 10.5, 1024 x 8192 15.9 / 10.1 / 6.3 / 6.0).
    const char* const forced = std::getenv("TC_TC_SPLIT");
    auto split_for = [&](int n) {
        int split = 1;
        for (int s = 8; s > 1; --s) {
            if (4 * s > p.groups || static_cast<long long>(n) * s > env.sm_count) continue;
            if (n <= max_active_clusters(s, env.smem_optin)) { split = s; break; }
        }
        if (forced) split = std::atoi(forced);
        if (split > 8) split = 8;
        if (split > p.groups) split = p.groups;
        if (split < 1 || p.off_x + red_bytes > env.smem_optin) split = 1;
        return split;
    };
    // Tiles left over after whole rounds of one per SM go in a launch of their own when their K can be split
    // over the SMs that would idle beside them (22016 x 4096, 8 rows: 148 tiles, then 24 in clusters of 4,
    // 20.5 -> 18.8 us).
    int first = tiles;
    const int left = env.sm_count > 0 ? tiles % env.sm_count : 0;
    if (tiles > env.sm_count && left > 0 && !forced && split_for(left) > 1) first = tiles - left;

    QtcMaps maps;
    const int gb = a.fmt == FMT_Q4_0 ? 144 : 272;
    for (int i = 0; i < n_ops; ++i)
        if (!encode_bytes_2d(&maps.w[i], ops[i].W, ops[i].N, static_cast<uint64_t>(p.groups) * gb, gb, kRows, a.fmt == FMT_Q4_0 ? 1 : 4))
            return cudaErrorNotSupported;
    for (int i = n_ops; i < kMaxMats; ++i) maps.w[i] = maps.w[0];
    if (!encode_f16_slices_sw128(&maps.x, a.X, a.M, a.K, p.nb, v->xk)) return cudaErrorNotSupported;

    auto launch = [&](int tile, int n) {
        p.tile_base = tile;
        p.split = split_for(n);
        p.wait_first = tile == 0 && env.wait_first() ? 1 : 0;      // the second launch follows this call's first
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(n) * p.split);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = p.split > 1 && p.off_x + red_bytes > smem ? p.off_x + red_bytes : smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        cfg.attrs = attr;
        cfg.numAttrs = 0;
        if (p.split > 1) {
            attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
            attr[cfg.numAttrs].val.clusterDim.x = p.split;
            attr[cfg.numAttrs].val.clusterDim.y = 1;
            attr[cfg.numAttrs].val.clusterDim.z = 1;
            ++cfg.numAttrs;
        }
        if (env.pdl || tile > 0) {         // behind this call's own first launch in any case
            attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
            ++cfg.numAttrs;
        }
        return cudaLaunchKernelEx(&cfg, v->kernel[a.fmt == FMT_Q4_0 ? 0 : 1], p, maps);
    };
    const cudaError_t e = launch(0, first);
    if (launches) *launches += first < tiles ? 2 : 1;
    return e == cudaSuccess && first < tiles ? launch(first, tiles - first) : e;
}

}  // namespace tcb
