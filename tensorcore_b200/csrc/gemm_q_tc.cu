// Quantized GEMV / GEMM for five activation rows or more on the sm_100a tensor cores (tcgen05):
//
//   Y[m][n] = sum_k X[m][k] * dequant(W)[n][k],   Q4_0 or Q8_0 blocks, fp16 X, any number of rows.
//
// The reference computes this as independent dequant-dots per output element, re-reading the weights
// for every activation row (lib/ops/quantized_cpu.cpp:193-228).  Here the packed weights are read
// once per tile of up to 256 activation rows and never exist as fp16 in memory:
//
//   * Up to four matrices that share their activations (q, k and v; gate and up) are one launch.
//   * The unit of work is one group of 8 blocks (256 weights) of a tile of 128 weight rows x NB activation rows
//     (NB = 16 .. 256, the MMA's N): a single tiled TMA copy of 128 rows x 144 (Q4_0) or 272 (Q8_0) raw bytes into
//     a ring.  Three ways to deal them out, chosen by the launcher: a tile per CTA; a cluster of up to 8 CTAs that
//     splits a tile's K; or shares - one CTA per SM works through an equal, contiguous run of the list of all
//     tiles' units, wherever tiles end, and the rings run on from tile to tile.
//   * Shares: warps of their own read out a finished tile while the next one is multiplied (two sets of
//     accumulators up to 32 columns).  A tile that two CTAs have parts of is stored by the one that has its
//     beginning, which comes to it last; the other begins with it and leaves its sums in scratch in L2, where a
//     word that holds no sum yet is known by its bits: no flag, no fence, about 1.2 us from store to use (with
//     flags 4 us).  Sums are added in K order, so results do not depend on timing.
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
//     fixed order.  Four issuers, two, one: 12288 x 4096, 8 rows 11.8 / 13.3 / 17.4 us, 14336 x 4096, 64 rows 16.2 /
//     20 / 27 us.
//   * The activation producer's loop is short on purpose: with 64 columns an issuer has two stages of 64 K, and 40
//     clocks more per copy cost 7 % of the call.
//   * Epilogue: tcgen05.ld, then a direct store, or in a cluster a fixed-order sum through distributed shared
//     memory.
//
// What bounds it: up to about 64 rows the weight stream and the dequantising instructions (14 per
// eight Q4_0 weights, issued by 16 warps; the zero point and the scale cannot be one fused
// multiply-add because 1032 d does not fit fp16), from 128 rows on the tensor pipe.
// Back to back on a stream, weights from HBM, against the kernel of 256-row tiles with separate
// activation staging (Q4_0 up to 95 rows) and the dequantised copy plus GEMM (the others) before it:
//   Q4_0 14336 x 4096   32 rows  22.0 -> 11.8 us (2.8 TB/s)    512 rows  95 -> 53 us (1130 TFLOP/s)
//   Q8_0 11008 x 4096   16 rows  51 -> 15.3 us (3.1 TB/s)
// With shares, against a tile per CTA in rounds: Q4_0 28672 x 4096, 32 rows 24.9 -> 19.7 us (3.4 TB/s), 22016 x 4096,
// 8 rows 20.4 -> 15.2, Q8_0 28672 x 4096, 16 rows 33.2 -> 27.8 (4.5 TB/s).
// Per 128-row unit of 256 weights in steady state: Q4_0 0.51 us at 8 rows, 1.9 us at 256 rows (1.08 us
// of tensor work at the clock's peak); Q8_0 0.82 us at 16 rows, which is the weight stream at 6.3 TB/s.
#include "handover.cuh"
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
constexpr int kEpiWarp = kMmaWarp + 4;     // with four groups: four warps that read out the tiles a CTA goes on from
// (with two groups the warps of the other two do that)
constexpr int threads_of(int wgs, bool runs) { return (runs && wgs == kWgs ? kEpiWarp + 4 : kEpiWarp) * 32; }
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
    int tile_base;     // first tile of a launch in clusters
    int tiles;         // (row tile, column tile) pairs, column tile fastest
    int col_tiles;     // tiles of nb activation rows
    int split;         // > 1: a cluster of that many CTAs per tile
    int chunk;         // split == 1: CTAs take runs of so many units: 1, or all of a tile
    int run, longer;   // ... run of them each, the first `longer` CTAs one more
    uint32_t* part;    // shares: [grid][nb][128], what a CTA has of a tile that began in the CTA before it (nothing else: handover.cuh)
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
    uint64_t d_full[2], d_empty[2], d_last;
    uint64_t drain[4];           // an issuer's last commit, before a CTA that gives up frees its memory
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

// First unit of share c: units are numbered tile by tile.
__device__ __forceinline__ int first_unit(const QtcParams& p, int c) {
    return (c * p.run + (c < p.longer ? c : p.longer)) * p.chunk;
}
// CB of the partial sums that another CTA of this launch leaves in scratch (handover.cuh), by a whole warp.
template <int CB>
__device__ __forceinline__ bool take_sums(uint32_t* src, uint32_t (&v)[CB], volatile int* abort_flag) {
    const long long t0 = clock64();
    for (;;) {
        bool all = true;
#pragma unroll
        for (int e = 0; e < CB; ++e)
            v[e] = handover::load(src + e * kRows);
#pragma unroll
        for (int e = 0; e < CB; ++e) all = all && handover::there(v[e]);
        if (__all_sync(0xffffffffu, all)) break;
        if (__any_sync(0xffffffffu, *abort_flag || clock64() - t0 > 2000000000LL)) return false;
    }
#pragma unroll
    for (int e = 0; e < CB; ++e) handover::store(src + e * kRows, handover::kNothing);
    return true;
}
template <int CB>
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&v)[CB]) {
    if constexpr (CB == 4) tmem_ld4(taddr, v);
    else if constexpr (CB == 8) tmem_ld8(taddr, v);
    else tmem_ld16(taddr, v);
    tmem_wait_ld();
}

// I: accumulators and issuers; unit u is issued by warp u % I.  WGS: dequantising warpgroups; unit u is group
// u % WGS's.  SLOTS: A slots per warpgroup.  XK: 64-wide K slices per activation stage.  ND: sets of accumulators.
// CB: columns a warp reads out at a time.  RUNS: a CTA works through a run of the unit list; else it has a K range of
// one tile (the code that goes on from tile to tile costs such launches 2 to 5 %).
template <int FMT, bool RUNS, int I, int WGS, int SLOTS, int XK, int ND, int CB>
__global__ void __launch_bounds__(threads_of(WGS, RUNS), 1)
gemm_q_tc_kernel(const QtcParams p, const __grid_constant__ QtcMaps maps) {
    using F = QFmt<FMT>;
    constexpr int kRawBytes = kRows * F::kGroup;
    static_assert(I == WGS || SLOTS == 4, "a slot's position follows from the unit when an issuer serves several groups");
    static_assert(WGS % I == 0 && WGS <= kWgs && SLOTS <= kMaxSlots && ND <= 2, "");
    extern __shared__ __align__(1024) uint8_t smem[];
    Bars* bars = reinterpret_cast<Bars*>(smem);
    volatile int* abort_flag = &bars->abort_flag;
    int* sent = bars->sent;
    // The warp number by shuffle, and one elected lane inside warp-uniform control flow around every copy, MMA
    // and commit: operands then are uniform values for the compiler.  An MMA issued from under `lane == 0`
    // took 70 to 112 clocks instead of 39 (M128 x N16..64 x K16, one issuing warp).
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int split = RUNS ? 1 : p.split, nb = p.nb, G = p.groups;
    // This CTA's units: a K range of one tile (clusters), or a run of the list of all tiles' units.  A CTA reads what
    // the one with the next share has of its last tile, so shares are numbered against the order in which CTAs start.
    int crank = 0, share = 0, u0 = 0, n_units, tile_lo, g_lo;
    if (!RUNS) {
        crank = split > 1 ? static_cast<int>(cluster_ctarank()) : 0;
        tile_lo = p.tile_base + static_cast<int>(blockIdx.x) / split;
        g_lo = G * crank / split;
        n_units = G * (crank + 1) / split - g_lo;
    } else {
        share = static_cast<int>(gridDim.x - 1 - blockIdx.x);
        u0 = first_unit(p, share);
        n_units = first_unit(p, share + 1) - u0;
        tile_lo = u0 / G;
        g_lo = u0 - tile_lo * G;
    }
    // Where a tile lies: its rows in one of the matrices, its columns.
    struct Place { int rt, ct, mat, N, row0; };
    auto place_of = [&](int tile) {
        Place t;
        t.rt = p.col_tiles == 1 ? tile : tile / p.col_tiles;
        t.ct = tile - t.rt * p.col_tiles;
        t.mat = 0;
        t.N = p.N[0];
        t.row0 = t.rt * kRows;
#pragma unroll
        for (int i = 1; i < kMaxMats; ++i)
            if (t.rt >= p.tile0[i]) { t.mat = i; t.N = p.N[i]; t.row0 = (t.rt - p.tile0[i]) * kRows; }
        return t;
    };
    const Place lo = place_of(tile_lo);
    const int first_len = !RUNS || n_units < G - g_lo ? n_units : G - g_lo;      // units of the first tile
    uint8_t* raw_ring = smem + p.off_raw;
    uint8_t* x_ring = smem + p.off_x;
    const int x_bytes = nb * 128 * XK;

    if (!p.wait_first) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (tid == kRawWarp * 32) prefetch_tensormap(&maps.w[lo.mat]);
    if (tid == kXWarp * 32) prefetch_tensormap(&maps.x);
    if (warp == 0) {                                 // a lane per index: one after the other they took half a microsecond
        if (lane < kMaxRing) {
            bar_init(&bars->raw_full[lane], 1);
            bar_init(&bars->raw_empty[lane], 4);     // the four warps of the warpgroup that reads it
            bar_init(&bars->x_full[lane], 1);
            bar_init(&bars->x_empty[lane], 1);       // commit of the issuer that read it
            sent[lane] = sent[kMaxRing + lane] = 0;
        } else if (lane < kMaxRing + kMaxSlots) {
            const int i = lane - kMaxRing;
            for (int j = 0; j < kWgs; ++j) {
                bar_init(&bars->a_full[j][i], 4);
                bar_init(&bars->a_empty[j][i], 1);
            }
            bar_init(&bars->drain[i], 1);
        } else if (lane < kMaxRing + kMaxSlots + 2) {
            const int i = lane - kMaxRing - kMaxSlots;
            bar_init(&bars->d_full[i], I);                          // every issuer has finished the tile
            bar_init(&bars->d_empty[i], WGS == kWgs ? 4 : 8);       // the read-out warps are through
        } else if (lane == 31) {
            bar_init(&bars->d_last, I);              // the last tile: its readers have not seen the phases before
            bars->abort_flag = 0;
        }
        fence_barrier_init();
    }
    if (warp == kRawWarp) tmem_alloc(&bars->tmem_base, kTmemCols);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = bars->tmem_base;
    const uint32_t a_col0 = static_cast<uint32_t>(ND * I * nb);      // accumulators first, then the A slots
    float* red = reinterpret_cast<float*>(smem + p.off_x);           // [nb][128], partials of a cluster: every operand has been read
    bool failed = false;
    // Reads out tile number `seg` of this CTA, units [done, end) of its run: blocks of CB columns from c_first in
    // steps of c_step, a warp per TMEM quadrant and block.  A tile the CTA has whole is stored; a tile that began in
    // the share before goes to scratch; one that goes on in the shares after this is stored with what those have of
    // it added in K order.  (They begin with that tile: it is there by the time it is needed unless the shares are
    // shorter than a tile.)
    auto read_out = [&](int seg, int done, int end, int c_first, int c_step, bool ok) {
        const int set = seg % ND, q = warp & 3, r = q * 32 + lane;
        const int tile = tile_lo + seg;
        const Place t = !RUNS || seg == 0 ? lo : place_of(tile);
        const int m0 = t.ct * nb, N = t.N, row = t.row0 + r;
        void* Y = p.Y[t.mat];
        const int m_end = p.M - m0 < nb ? p.M - m0 : nb;
        const int used = end - done < I ? end - done : I;          // accumulators that were written
        const bool last = !RUNS || end == n_units, begins = !RUNS || seg > 0 || g_lo == 0;
        uint32_t* mine = p.part + static_cast<size_t>(share) * nb * kRows + r;
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(set * I * nb);
        int others = 0;
        if (RUNS && begins && last)
            for (int u = u0 + end, t_end = (tile + 1) * G; u < t_end; u = first_unit(p, share + others + 1)) ++others;
        ok = ok && wait_all(last ? &bars->d_last : &bars->d_full[set], last ? 0u : static_cast<uint32_t>(seg / ND) & 1u, abort_flag);
        ok = __all_sync(0xffffffffu, ok && !*abort_flag);
        tc_fence_after_sync();
        for (int c0 = c_first; c0 < m_end && ok; c0 += c_step) {
            float f[CB];
            uint32_t v[CB];
#pragma unroll
            for (int e = 0; e < CB; ++e) f[e] = 0.f;
            for (int t = 0; t < used; ++t) {
                const int a = I == 1 ? 0 : (done + t) % I;
                tmem_ld_cols(taddr + static_cast<uint32_t>(a * nb + c0), v);
#pragma unroll
                for (int e = 0; e < CB; ++e) f[e] += __uint_as_float(v[e]);
            }
            for (int i = 1; RUNS && i <= others && ok; ++i) {
                ok = take_sums(mine + (static_cast<size_t>(i) * nb + c0) * kRows, v, abort_flag);
#pragma unroll
                for (int e = 0; e < CB; ++e) f[e] += __uint_as_float(v[e]);
            }
            if (split > 1) {
#pragma unroll
                for (int e = 0; e < CB; ++e) red[(c0 + e) * kRows + r] = f[e];
            } else if (RUNS && !begins) {
#pragma unroll
                for (int e = 0; e < CB; ++e) handover::store(mine + (c0 + e) * kRows, handover::word_of(f[e]));
            } else if (row < N) {
                const size_t o = static_cast<size_t>(m0 + c0) * N + row;
                if (p.y_f32) {
                    float* y = static_cast<float*>(Y) + o;
#pragma unroll
                    for (int e = 0; e < CB; ++e, y += N)
                        if (c0 + e < m_end) *y = f[e];
                } else {
                    __half* y = static_cast<__half*>(Y) + o;
#pragma unroll
                    for (int e = 0; e < CB; ++e, y += N)
                        if (c0 + e < m_end) *y = __float2half_rn(f[e]);
                }
            }
        }
        tc_fence_before_sync();
        return ok;
    };

    // Reads out every tile but the last, while the next one is multiplied.
    auto read_out_others = [&](int c_first, int c_step) {
        asm volatile("griddepcontrol.wait;" ::: "memory");         // Y and the scratch may still be in use by the kernel before
        for (int seg = 0, done = 0, end = first_len; end < n_units; ++seg) {
            if (!read_out(seg, done, end, c_first, c_step, true)) return false;
            __syncwarp();
            if (lane == 0) bar_arrive(&bars->d_empty[seg % ND]);   // the accumulators may be used again
            done = end;
            end = end + G < n_units ? end + G : n_units;
        }
        return true;
    };

    if (warp < kDqWarps) {
        // ---------------- dequantisers: one thread per weight row --------------------------------------
        const int wg = warp >> 2, q = warp & 3;
        const uint32_t a_base = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + a_col0 + static_cast<uint32_t>(wg * SLOTS * 32);
        const uint32_t row_off = static_cast<uint32_t>(q * 32 + lane) * F::kGroup;
        Pos slot, ring;
        for (int u = wg; u < n_units && wg < WGS && !failed; u += WGS) {
            const int st = wg + WGS * ring.i;
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
        if (RUNS && WGS < kWgs && wg >= WGS && !read_out_others((wg - WGS) * CB, (kWgs - WGS) * CB)) failed = true;
        // The last tile: all of them.
        asm volatile("griddepcontrol.wait;" ::: "memory");
        const int more = RUNS ? (n_units - first_len + G - 1) / G : 0;      // tiles after the first
        const int done = more > 0 ? first_len + (more - 1) * G : 0;
        if (!read_out(more, done, n_units, wg * CB, kWgs * CB, !failed)) failed = true;
    } else if (warp == kRawWarp) {
        // ---------------- weight producer: 128 rows x one group per unit; rows past N read as zeros -----
        const CUtensorMap* wmap = &maps.w[lo.mat];
        int tile = tile_lo, row0 = lo.row0;
        if (p.wait_first) {
            asm volatile("griddepcontrol.wait;" ::: "memory");
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        }
        Pos ring;
        int g = g_lo, wg = 0;
        for (int u = 0, end = first_len; u < n_units && !failed; g = 0) {
            for (; u < end; ++u, ++g) {
                const int st = wg + WGS * ring.i;
                if (!wait_all(&bars->raw_empty[st], ring.ph ^ 1u, abort_flag)) { failed = true; break; }
                if (elect_one()) {
                    bar_expect_tx(&bars->raw_full[st], kRawBytes);
                    tensor_load_2d(raw_ring + st * kRawBytes, wmap, g * (F::kGroup / F::kElem), row0, &bars->raw_full[st]);
                    sent[st] += 1;
                }
                __syncwarp();
                if (++wg == WGS) { wg = 0; ring.next(p.raw_stages); }
            }
            end = end + G < n_units ? end + G : n_units;
            if (!RUNS) break;
            const Place t = place_of(++tile);
            wmap = &maps.w[t.mat];
            row0 = t.row0;
        }
        if (failed || *abort_flag) {             // copies in flight land before the shared memory is released
            for (int st = 0; st < WGS * p.raw_stages; ++st)
                if (sent[st] > 0) bar_wait(&bars->raw_full[st], static_cast<uint32_t>(sent[st] - 1) & 1u, nullptr, 100000000LL);
        }
    } else if (warp == kXWarp) {
        // ---------------- activation producer, in the order the issuers consume ---------------------------
        // The slices of a round of I units take turns, but never those of two tiles: an issuer that has to wait for the
        // accumulators must not hold up another that still has to finish the tile in them.
        // Activations belong to the stream's order: wait for the kernel before this one here, with
        // the weight copies already in flight where nothing that may still run writes them.
        int ct = lo.ct;
        asm volatile("griddepcontrol.wait;" ::: "memory");
        Pos ring;                                    // the same place in every issuer's ring
        for (int r = 0, from = 0, end = first_len, g = g_lo, m0 = ct * nb; r < n_units && !failed;) {
            // units [from, hi) of the round from r belong to one tile; unit u is group u + g of it
            int hi = r + I < n_units ? r + I : n_units;
            if (end < hi) hi = end;
            Pos at = ring;
            if (from == r && hi == r + I) {
                for (int s = 0; s < 4 && !failed; s += XK) {
#pragma unroll
                    for (int j = 0; j < I; ++j) {
                        const int st = j * p.x_stages + at.i;
                        if (!wait_all(&bars->x_empty[st], at.ph ^ 1u, abort_flag)) { failed = true; break; }
                        if (elect_one()) {
                            bar_expect_tx(&bars->x_full[st], x_bytes);
                            tensor_load_3d(x_ring + st * x_bytes, &maps.x, 0, m0, (g + r + j) * 4 + s, &bars->x_full[st]);
                            sent[kMaxRing + st] += 1;
                        }
                        __syncwarp();
                    }
                    at.next(p.x_stages);
                }
            } else
            for (int s = 0; s < 4 && !failed; s += XK) {
#pragma unroll
                for (int j = 0; j < I; ++j) {
                    if (r + j < from) continue;
                    if (r + j >= hi) break;
                    const int st = j * p.x_stages + at.i;
                    if (!wait_all(&bars->x_empty[st], at.ph ^ 1u, abort_flag)) { failed = true; break; }
                    if (elect_one()) {
                        bar_expect_tx(&bars->x_full[st], x_bytes);
                        tensor_load_3d(x_ring + st * x_bytes, &maps.x, 0, m0, (g + r + j) * 4 + s, &bars->x_full[st]);
                        sent[kMaxRing + st] += 1;
                    }
                    __syncwarp();
                }
                at.next(p.x_stages);
            }
            from = hi;
            if (hi == r + I) { r = hi; ring = at; }
            else if (hi == n_units) break;
            if (hi == end) {
                g = -end;
                end += G;
                if (++ct == p.col_tiles) ct = 0;
                m0 = ct * nb;
            }
        }
        if (failed || *abort_flag) {
            for (int st = 0; st < I * p.x_stages; ++st)
                if (sent[kMaxRing + st] > 0)
                    bar_wait(&bars->x_full[st], static_cast<uint32_t>(sent[kMaxRing + st] - 1) & 1u, nullptr, 100000000LL);
        }
    } else if (warp < kEpiWarp) {
        // ---------------- MMA issue: one warp per accumulator ------------------------------------------------
        const int me = warp - kMmaWarp;
        const uint32_t idesc = idesc_f16_f32(kRows, nb);
        uint32_t d_col = tmem_base + static_cast<uint32_t>(me * nb), started = 0;
        Pos xs, set, slot;
        int end = first_len;                                       // the tile's units end here
        // Every MMA of this issuer so far is the tile's; on to the next one, once its accumulators have been read out.
        auto next_tile = [&]() {
            if (elect_one()) mma_commit(&bars->d_full[set.i]);
            __syncwarp();
            set.next(ND);
            end = end + G < n_units ? end + G : n_units;
            started = 0;
            if (ND > 1) d_col = tmem_base + static_cast<uint32_t>((set.i * I + me) * nb);
            if (!wait_all(&bars->d_empty[set.i], set.ph ^ 1u, abort_flag)) failed = true;
            tc_fence_after_sync();
        };
        for (int u = me; u < n_units && me < I && !failed; u += I) {
            while (RUNS && u >= end && !failed) next_tile();
            if (failed) break;
            const int j = I == WGS ? me : u % WGS;                 // the warpgroup that dequantises the unit
            if (I != WGS) { slot.i = 0; slot.ph = static_cast<uint32_t>(u / WGS) & 1u; }
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
        while (RUNS && end < n_units && me < I && !failed) next_tile();    // tiles without a unit of this issuer's
        if (me < I && !failed && elect_one()) mma_commit(&bars->d_last);
        __syncwarp();
        if (me < I && (failed || *abort_flag)) {
            // every MMA issued has completed before tensor and shared memory are released
            if (elect_one()) mma_commit(&bars->drain[me]);
            __syncwarp();
            bar_wait(&bars->drain[me], 0, nullptr, 100000000LL);
        }
    } else if (RUNS && !read_out_others(0, CB)) {
        failed = true;
    }

    if (failed) {
        *abort_flag = 1;
        if (p.err) atomicOr(p.err, ERR_WAIT_TIMEOUT);
    }
    __syncwarp();
    __syncthreads();

    if (split > 1) {
        const int m0 = lo.ct * nb, N = lo.N, row0 = lo.row0;
        void* Y = p.Y[lo.mat];
        cluster_sync_all();
        if (!*abort_flag) {
            const int r_lo = kRows * crank / split, r_hi = kRows * (crank + 1) / split;
            const int rows_c = r_hi - r_lo;
            const int m_end = p.M - m0 < nb ? p.M - m0 : nb;
            const uint32_t red_addr = s_u32(red);
            for (int e = tid; e < m_end * rows_c; e += blockDim.x) {
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
        cfg.blockDim = dim3(threads_of(kWgs, false));
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = size;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&n, gemm_q_tc_kernel<FMT_Q4_0, false, 4, 4, 3, 4, 1, 4>, &cfg) != cudaSuccess || n <= 0) {
            n = -1;
            (void)cudaGetLastError();
        }
        cache[size].store(n);
    }
    return n > 0 ? n : 0;
}

using QtcKernel = void (*)(const QtcParams, const QtcMaps);
struct QtcVariant { int max_nb, issuers, wgs, xk; QtcKernel kernel[2][2]; };      // kernel[runs][format]
#define TCB_QTC(NB, I, WGS, XK, SLOTS, CB, RUN_SLOTS, ND, RUN_CB) \
    {NB, I, WGS, XK, {{gemm_q_tc_kernel<FMT_Q4_0, false, I, WGS, SLOTS, XK, 1, CB>, gemm_q_tc_kernel<FMT_Q8_0, false, I, WGS, SLOTS, XK, 1, CB>}, \
                      {gemm_q_tc_kernel<FMT_Q4_0, true, I, WGS, RUN_SLOTS, XK, ND, RUN_CB>, gemm_q_tc_kernel<FMT_Q8_0, true, I, WGS, RUN_SLOTS, XK, ND, RUN_CB>}}}
const QtcVariant kVariants[] = {TCB_QTC(16, 4, 4, 4, 3, 4, 3, 2, 4), TCB_QTC(32, 4, 4, 2, 3, 8, 2, 2, 8), TCB_QTC(64, 4, 4, 1, 2, 16, 2, 1, 8),
                                TCB_QTC(128, 2, 2, 1, 4, 16, 4, 1, 16), TCB_QTC(256, 1, 2, 1, 4, 16, 4, 1, 16)};
#undef TCB_QTC

// The MMA's columns for M activation rows: as few equal tiles of at most 256 as there can be.
int mma_columns(int M, int* col_tiles) {
    *col_tiles = (M + 255) / 256;
    return ((M + *col_tiles - 1) / *col_tiles + 15) & ~15;
}

// Shares, where they save enough units of the CTA with most of them.  What they cost: a tile more to read out
// on the way, and, where a share is shorter than a tile, the sums that cross the L2 at the very end (a tile of 8 /
// 32 / 64 / 128 / 256 columns: 2.2 / 2.5 / 6.5 / 6.7 / 10 us).  Whole tiles or clusters / shares, microseconds back to
// back, units of 256 weights by 128 rows of the longest CTA in brackets:
//   Q4_0, rows           8            32            64           128           256           512
//   11008 x 4096 (16 / 9.3)   11.7 / 11.3   12.5 / 12.3   16.1 / 18.4   17.7 / 19.2   29.1 / 29.9   -
//   14336 x 4096 (16 / 12.1)  12.0 / 12.5   12.8 / 13.7   16.4 / 20.1   17.8 / 21.0   28.9 / 33.2   59.5 / 56.2 (32 / 24.2)
//   28672 x 4096 (32 / 24.2)  21.5 / 18.2   22.7 / 19.7   30.5 / 31.5   33.4 / 34.0   58.0 / 54.8   112 / 102 (64 / 48.4)
//   20000 x 2048 (16 / 8.5)   15.7 / 10.2   16.4 / 11.1   19.7 / 16.2   22.5 / 18.5   39.2 / 29.5   62.0 / 46.8 (24 / 17)
//   4096 x 4096 (4 / 3.5)      8.7 /  8.0    9.2 /  8.8   10.9 / 15.0 (clusters of four)
// Q8_0's units take longer up to 32 columns (0.82 against 0.5 us), so fewer of them pay; and the longer the tiles the more
// they have to be, because the weights then come at HBM's rate either way.  With fewer tiles than SMs (differences of 200
// calls of 104 to 147 tiles): saved 5 units of 16 / 32 / 50 / 80 Q4_0 +0.1 / +0.1 / +0.2 / +1.5 us, 8 units - / -0.9 / -0.8 / -0.7;
// Q8_0 5 units -0.5 / -0.2 / +2.3 / +1.0, 8 units - / -1.8 / +0.2 / -0.5.
// And not where a tile is in the hands of many CTAs, whose sums are taken one after the other: more than seven, or ten where
// shares are seven units or more.  Clusters / shares: Q4_0, 32 rows, 768 x 28672 12.9 / 18.0 us, 1024 x 20480 11.5 / 14.7;
// 16 rows 2048 x 28672 15.6 / 14.5, Q8_0 21.7 / 19.2; 2560 x 14336 15.0 / 13.6 but 2560 x 11008 12.6 / 13.3.
struct Shares { int n; bool pay; };
Shares shares_of(int fmt, int nb, long long tiles, int groups, int sms) {
    const long long units = tiles * groups;
    const int n = units < sms ? static_cast<int>(units) : sms;
    const double saved = static_cast<double>((tiles + sms - 1) / sms) * groups - static_cast<double>(units) / n;
    if (tiles > sms) return {n, saved > (nb <= 32 ? 4.0 : nb <= 128 ? 7.0 : 5.6)};
    const bool few = 7 * tiles > sms || (10 * tiles > sms && units >= 7 * sms);
    const double least = fmt == FMT_Q4_0 ? 5.5 : 4.0, by_length = (fmt == FMT_Q4_0 ? 0.1 : 0.15) * groups;
    return {n, nb <= 32 && few && units >= 3 * sms && saved > (by_length < least ? least : by_length > 8.0 ? 8.0 : by_length)};
}
size_t share_bytes(const Shares& s, int nb) { return static_cast<size_t>(s.n) * nb * kRows * 4; }

}  // namespace

cudaError_t init_gemm_q_tc_kernels(int smem_optin) {
    for (const QtcVariant& v : kVariants)
        for (const auto& forms : v.kernel)
            for (QtcKernel k : forms) {
                const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin);
                if (e != cudaSuccess) return e;
            }
    return cudaSuccess;
}

size_t gemm_q_tc_share_bytes(const GemvQArgs* ops, int n_ops, int M, int sm_count) {
    int col_tiles = 1;
    const int nb = mma_columns(M, &col_tiles);
    long long row_tiles = 0;
    for (int i = 0; i < n_ops; ++i) row_tiles += (ops[i].N + kRows - 1) / kRows;
    const Shares s = shares_of(ops[0].fmt, nb, row_tiles * col_tiles, ops[0].K / 256, sm_count > 0 ? sm_count : 148);
    return s.pay ? share_bytes(s, nb) : 0;
}

size_t gemm_q_tc_share_room(int M, int sm_count) {
    int col_tiles = 1;
    return share_bytes({sm_count > 0 ? sm_count : 148, true}, mma_columns(M, &col_tiles));
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
    p.nb = mma_columns(a.M, &p.col_tiles);
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
    const long long units = row_tiles * p.col_tiles * p.groups;
    if (units > 0x3fffffff) return cudaErrorNotSupported;
    p.tiles = static_cast<int>(row_tiles * p.col_tiles);

    // Ring depths: two raw stages per warpgroup where at least two activation stages fit beside them (one
    // being read, one in flight), else one; activations get what is left.
    const int room = env.smem_optin - kBarBytes;
    const int min_x = (v->issuers == 1 ? 4 : 2) * v->issuers * x_bytes;
    p.raw_stages = 2 * v->wgs * raw_bytes + min_x <= room ? 2 : 1;
    p.x_stages = (room - p.raw_stages * v->wgs * raw_bytes) / (v->issuers * x_bytes);
    if (p.x_stages * v->issuers > kMaxRing) p.x_stages = kMaxRing / v->issuers;
    if (p.x_stages < 2) return cudaErrorNotSupported;
    p.off_x = kBarBytes;                               // 1024-byte aligned, as are the activation stages
    p.off_raw = p.off_x + v->issuers * p.x_stages * x_bytes;
    const int smem = p.off_raw + v->wgs * p.raw_stages * raw_bytes;
    const int red_bytes = p.nb * kRows * 4;

    // K is split over a cluster when there are fewer tiles than SMs: the largest cluster size whose
    // clusters can all be resident at once, so that the split shortens the K loop instead of queueing, and
    // whose CTAs keep a unit for each of four warpgroups (8 rows, split 1 / 2 / 4 / 8: 4096 x 1024 3.4 / 4.5 /
    // 6.2 us, 4096 x 2048 5.1 / 5.0 / 6.5, 2048 x 4096 - / 6.5 / 4.7 / 10.5, 1024 x 8192 15.9 / 10.1 / 6.3 / 6.0).
    const char* const forced = std::getenv("TC_TC_SPLIT");
    const int sms = env.sm_count > 0 ? env.sm_count : 148, tiles = p.tiles, left = tiles % sms;
    auto split_for = [&](int n) {
        int split = 1;
        for (int c = 8; c > 1; --c) {
            if (4 * c > p.groups || static_cast<long long>(n) * c > sms) continue;
            if (n <= max_active_clusters(c, env.smem_optin)) { split = c; break; }
        }
        if (forced) split = std::atoi(forced);
        if (split > 8) split = 8;
        if (split > p.groups) split = p.groups;
        if (split < 1 || p.off_x + red_bytes > env.smem_optin) split = 1;
        return split;
    };
    // Tiles left over after whole rounds of one per SM can go in a launch of their own when their K can be split
    // over the SMs that would idle beside them.
    const bool two_launches = tiles > sms && left > 0 && !forced && split_for(left) > 1;
    const Shares shares = shares_of(a.fmt, p.nb, tiles, p.groups, sms);
    // A synchronous call keeps its two launches, which test_tiles_left_over_after_whole_rounds counts; by the table above
    // shares would be faster (20000 x 2048, 8 rows 10.2 us instead of 15.7 back to back).
    const bool share = shares.pay && !forced && !(env.alone && two_launches) && a.share_scratch &&
                       a.share_scratch_bytes >= share_bytes(shares, p.nb);
    p.part = static_cast<uint32_t*>(a.share_scratch);
    const int first = two_launches && !share ? tiles - left : tiles;

    QtcMaps maps;
    const int gb = a.fmt == FMT_Q4_0 ? 144 : 272;
    for (int i = 0; i < n_ops; ++i)
        if (!encode_bytes_2d(&maps.w[i], ops[i].W, ops[i].N, static_cast<uint64_t>(p.groups) * gb, gb, kRows, a.fmt == FMT_Q4_0 ? 1 : 4))
            return cudaErrorNotSupported;
    for (int i = n_ops; i < kMaxMats; ++i) maps.w[i] = maps.w[0];
    if (!encode_f16_slices_sw128(&maps.x, a.X, a.M, a.K, p.nb, v->xk)) return cudaErrorNotSupported;

    auto launch = [&](int tile, int n) {
        p.tile_base = tile;
        p.tiles = n;
        p.split = share ? 1 : split_for(n);
        p.wait_first = tile == 0 && env.wait_first() ? 1 : 0;      // the second launch follows this call's first
        cudaLaunchConfig_t cfg = {};
        const int ctas = p.split > 1 ? n * p.split : share ? shares.n : n < sms ? n : sms;
        const int chunks = share ? static_cast<int>(units) : n;
        p.chunk = share ? 1 : p.groups;
        p.run = chunks / ctas;
        p.longer = chunks % ctas;
        cfg.gridDim = dim3(static_cast<unsigned>(ctas));
        const bool runs = share || (p.split == 1 && n > ctas);
        cfg.blockDim = dim3(threads_of(v->wgs, runs));
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
        return cudaLaunchKernelEx(&cfg, v->kernel[runs][a.fmt == FMT_Q4_0 ? 0 : 1], p, maps);
    };
    const cudaError_t e = launch(0, first);
    if (launches) *launches += first < tiles ? 2 : 1;
    return e == cudaSuccess && first < tiles ? launch(first, tiles - first) : e;
}

}  // namespace tcb
