// Quantized GEMV for rows that the tiled copies cannot describe: any K that is a multiple of 32, any
// row count, weights at any 2-byte aligned address (Q4_0 / Q8_0 blocks of 18 / 34 bytes).
//
//   Y[m][n] = sum_b d[n][b] * sum_i q[n][b][i] * X[m][32 b + i],  up to four activation rows per pass,
//
// in fp32 throughout, a block's products first and then the scale, as the reference's loop has it
// (lib/ops/quantized_cpu.cpp:111-170,193-228).
//
// A lane owns a block: the 32 lanes of a warp take neighbouring blocks of four weight rows, so a warp
// has 4 x 32 blocks in flight.  A block starts at any even byte; it is read with the 8-byte words that
// contain it (three for Q4_0, five for Q8_0 whatever the offset, none without a byte of the block) and
// shifted into place in registers.  Activations sit in shared memory as fp32, transposed so that lanes on
// neighbouring blocks read neighbouring 16-byte pieces, and every piece serves four weight rows; with
// one row per warp those reads would be the bound.  A CTA per SM owns a row range; its (4 rows x 32 blocks)
// units are dealt to 16 warps, and the partial sums of a row are added in block order: deterministic.
// HBM-bound in principle; what it reaches is set by how many units a warp gets (one to three).
// 5003 x 4128 Q8_0, three fp32 rows: 283 us before (a warp per row, byte loads, activations from L1 for
// every weight); 14.8 us before a unit's blocks were fetched while the activations are staged and the unit
// before it is computed, 14.1 us with that (in a raw call 14.7 back to back since it waits for the work before).  Error against 64 bits on that shape 1.13e-7 with a block's products in
// two chains, 1.28e-7 in one and as the warp per row had it.
#include "gemv_common.cuh"

namespace tcb {
namespace {

constexpr int kRowsThreads = 512;
constexpr int kRowsWarps = kRowsThreads / 32;
constexpr int kGroupRows = 4;

struct RowsParams {
    const uint8_t* W;
    const void* X;
    void* Y;
    const void* gamma;
    int N, K, nb;
    int nbp;          // blocks of a staged row, padded to an odd count (bank conflicts while staging)
    int cb, chunks;   // blocks per chunk (at most 32), chunks per row
    int max_rows;     // rows of a CTA, rounded up to whole groups
    EvenSplit rows_of;
    int step_c;       // whole chunks from a warp's unit to its next one, at least
    int x_f32, y_f32;
    int wait_first;   // the kernel before may write the weights
    int x_vec;        // X and gamma allow 8-byte (fp16) / 16-byte (fp32) loads
    float eps;
    int off_part;
};

template <int FMT>
struct RowBlock {
    static constexpr int kWords8 = FMT == FMT_Q4_0 ? 3 : 5;
    static constexpr int kQ = FMT == FMT_Q4_0 ? 4 : 8;       // 32-bit words of quants
    uint32_t w[2 * kWords8];
    // All loads of the block; the 8-byte words at and after floor8(address) that hold its bytes.
    __device__ __forceinline__ void load(const uint8_t* at, bool active) {
        const uint2* src = reinterpret_cast<const uint2*>(reinterpret_cast<uintptr_t>(at) & ~static_cast<uintptr_t>(7));
#pragma unroll
        for (int k = 0; k < kWords8; ++k) {
            uint2 v = make_uint2(0u, 0u);
            if (active) v = __ldg(src + k);
            w[2 * k] = v.x; w[2 * k + 1] = v.y;
        }
    }
    // Scale, and the quants as kQ words in order (the block begins `off` = 0, 2, 4 or 6 bytes into w).
    __device__ __forceinline__ float unpack(int off, uint32_t (&q)[kQ]) const {
        uint32_t s[kQ + 1];
#pragma unroll
        for (int k = 0; k <= kQ; ++k) s[k] = (off & 4) ? w[k + 1] : w[k];
        const uint32_t sh = (off & 2) ? 32u : 16u;
#pragma unroll
        for (int k = 0; k < kQ; ++k) q[k] = __funnelshift_rc(s[k], s[k + 1], sh);
        const float d = h2f((off & 2) ? hi16(s[0]) : lo16(s[0]));
        return d;
    }
};
// Quants of elements 4 i .. 4 i + 3 as floats: the unsigned byte becomes the low mantissa of 2^23 and the offset
// is subtracted, both exactly; a conversion instruction a weight has a quarter of the rate (14.1 -> 13.3 us).
template <int FMT>
__device__ __forceinline__ void four_quants(const uint32_t* q, int i, float (&f)[4]) {
    const uint32_t v = FMT == FMT_Q4_0 ? (i < 4 ? q[i & 3] : q[i & 3] >> 4) & 0x0F0F0F0Fu : q[i & 7] ^ 0x80808080u;
    const float zero = FMT == FMT_Q4_0 ? 8388608.0f + 8.0f : 8388608.0f + 128.0f;
#pragma unroll
    for (int t = 0; t < 4; ++t) f[t] = __uint_as_float(__byte_perm(v, 0x4B000000u, 0x7440 + t)) - zero;
}

template <int FMT, int MB>
__global__ void __launch_bounds__(kRowsThreads, 1) gemv_q_rows_kernel(const RowsParams p) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ double red[kRowsWarps];
    constexpr int kBlock = FMT == FMT_Q4_0 ? 18 : 34;
    float4* xs = reinterpret_cast<float4*>(smem);               // [MB][8][nbp]
    float* part = reinterpret_cast<float*>(smem + p.off_part);  // [chunks][max_rows][MB]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (p.wait_first) pdl_wait();
    pdl_launch_dependents();
    const int r0 = p.rows_of.first(blockIdx.x), r1 = p.rows_of.first(blockIdx.x + 1);
    const int groups = (r1 - r0 + kGroupRows - 1) / kGroupRows;
    const size_t row_bytes = static_cast<size_t>(p.nb) * kBlock;
    // Blocks of this warp's next unit, on their way while the activations are staged or a unit is computed.
    RowBlock<FMT> blk[kGroupRows];
    int off[kGroupRows];
    auto fetch = [&](int c, int g) {
        const int b = c * p.cb + lane;
        const bool active = c < p.chunks && lane < p.cb && b < p.nb;
#pragma unroll
        for (int r = 0; r < kGroupRows; ++r) {
            int row = r0 + g * kGroupRows + r;
            if (row >= r1) row = r1 - 1;                        // its result is not stored
            const uint8_t* at = p.W + static_cast<size_t>(row) * row_bytes + static_cast<size_t>(active ? b : 0) * kBlock;
            off[r] = static_cast<int>(reinterpret_cast<uintptr_t>(at) & 7u);
            blk[r].load(at, active);
        }
    };
    // Unit c * groups + g: chunk c of row group g.  A warp's units are kRowsWarps apart, and it goes from one to the next
    // by whole chunks that the host has counted and a subtraction or two.  Whole calls, one row: counted out of the
    // unit's number by subtractions (one per chunk, twice a unit) / by a division / so: Q4_0 4096 x 50016 71.8 / 54.9 / 52.8 us,
    // Q8_0 8192 x 28704 68.6 / 60.4 / 57.3, Q4_0 11008 x 4128 14.5 / 14.8 / 14.0, Q8_0 300 x 55008 19.5 / 17.7 / 17.5.
    // (Four rows of Q8_0, 5003 x 4128, spill: 17.3 / 19.1 / 18.0.)
    int c = 0, g = warp;
    for (; g >= groups; g -= groups) ++c;
    const int step_g = kRowsWarps - p.step_c * groups;
    fetch(c, g);
    pdl_wait();

    auto load4 = [&](const void* src, size_t at) {
        if (p.x_f32) {
            const float* f = static_cast<const float*>(src) + at;
            return p.x_vec ? *reinterpret_cast<const float4*>(f) : make_float4(f[0], f[1], f[2], f[3]);
        }
        const __half* h = static_cast<const __half*>(src) + at;
        if (p.x_vec) {
            const uint2 v = *reinterpret_cast<const uint2*>(h);
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
            return make_float4(a.x, a.y, b.x, b.y);
        }
        return make_float4(__half2float(h[0]), __half2float(h[1]), __half2float(h[2]), __half2float(h[3]));
    };
    const int quads = p.K / 4;
#pragma unroll
    for (int m = 0; m < MB; ++m) {
        const size_t row = static_cast<size_t>(m) * p.K;
        float rstd = 1.f;
        if (p.gamma != nullptr) {
            double ss = 0.0;
            for (int e = tid; e < quads; e += kRowsThreads) {
                const float4 v = load4(p.X, row + 4 * static_cast<size_t>(e));
                ss += static_cast<double>(v.x) * v.x + static_cast<double>(v.y) * v.y;
                ss += static_cast<double>(v.z) * v.z + static_cast<double>(v.w) * v.w;
            }
            ss = block_sum_f64(ss, red);
            rstd = 1.0f / sqrtf(static_cast<float>(ss / static_cast<double>(p.K)) + p.eps);
        }
        for (int e = tid; e < quads; e += kRowsThreads) {
            float4 v = load4(p.X, row + 4 * static_cast<size_t>(e));
            if (p.gamma != nullptr) {
                const float4 g = load4(p.gamma, 4 * static_cast<size_t>(e));
                v.x = __fmul_rn(__fmul_rn(v.x, rstd), g.x); v.y = __fmul_rn(__fmul_rn(v.y, rstd), g.y);
                v.z = __fmul_rn(__fmul_rn(v.z, rstd), g.z); v.w = __fmul_rn(__fmul_rn(v.w, rstd), g.w);
            }
            xs[(m * 8 + (e & 7)) * p.nbp + (e >> 3)] = v;
        }
    }
    __syncthreads();

    while (c < p.chunks) {
        const int b = c * p.cb + lane, sums_at = (c * p.max_rows + g * kGroupRows) * MB;
        const bool active = lane < p.cb && b < p.nb;
        const int bx = active ? b : 0;
        uint32_t q[kGroupRows][RowBlock<FMT>::kQ];
        float d[kGroupRows], acc[kGroupRows][MB], acc2[kGroupRows][MB];
#pragma unroll
        for (int r = 0; r < kGroupRows; ++r) {
            d[r] = blk[r].unpack(off[r], q[r]);
#pragma unroll
            for (int m = 0; m < MB; ++m) acc[r][m] = acc2[r][m] = 0.f;
        }
        c += p.step_c;
        for (g += step_g; g >= groups; g -= groups) ++c;
        if (c < p.chunks) fetch(c, g);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float4 x[MB];
#pragma unroll
            for (int m = 0; m < MB; ++m) x[m] = xs[(m * 8 + i) * p.nbp + bx];
#pragma unroll
            for (int r = 0; r < kGroupRows; ++r) {
                float f[4];
                four_quants<FMT>(q[r], i, f);
#pragma unroll
                for (int m = 0; m < MB; ++m) {
                    float& a = (i & 1) ? acc2[r][m] : acc[r][m];       // two chains of 16 products: fewer roundings on each
                    a = fmaf(x[m].x, f[0], a);
                    a = fmaf(x[m].y, f[1], a);
                    a = fmaf(x[m].z, f[2], a);
                    a = fmaf(x[m].w, f[3], a);
                }
            }
        }
#pragma unroll
        for (int r = 0; r < kGroupRows; ++r)
#pragma unroll
            for (int m = 0; m < MB; ++m) {
                float v = active ? (acc[r][m] + acc2[r][m]) * d[r] : 0.f;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) part[sums_at + r * MB + m] = v;
            }
    }
    __syncthreads();
    for (int e = tid; e < (r1 - r0) * MB; e += kRowsThreads) {
        const int m = MB == 1 ? 0 : e / (r1 - r0), r = e - m * (r1 - r0);
        float v = 0.f;
        for (int c = 0; c < p.chunks; ++c) v += part[(c * p.max_rows + r) * MB + m];
        const size_t o = static_cast<size_t>(m) * p.N + r0 + r;
        if (p.y_f32) static_cast<float*>(p.Y)[o] = v;
        else static_cast<__half*>(p.Y)[o] = __float2half_rn(v);
    }
}

using RowsKernel = void (*)(const RowsParams);
const RowsKernel kRowsKernels[2][kMaxMB] = {
    {gemv_q_rows_kernel<FMT_Q4_0, 1>, gemv_q_rows_kernel<FMT_Q4_0, 2>, gemv_q_rows_kernel<FMT_Q4_0, 3>, gemv_q_rows_kernel<FMT_Q4_0, 4>},
    {gemv_q_rows_kernel<FMT_Q8_0, 1>, gemv_q_rows_kernel<FMT_Q8_0, 2>, gemv_q_rows_kernel<FMT_Q8_0, 3>, gemv_q_rows_kernel<FMT_Q8_0, 4>}};

}  // namespace

cudaError_t init_gemv_q_rows_kernels(int smem_optin) {
    for (const auto& fmt : kRowsKernels)
        for (RowsKernel k : fmt) {
            const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_optin - 1024);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

// Up to kMaxMB rows.  cudaErrorNotSupported: weights at an odd address, or activations that do not fit
// shared memory as fp32 (fewer rows may).
cudaError_t launch_gemv_q_rows(const GemvQArgs& a, const LaunchEnv& env, cudaStream_t stream) {
    if (a.M < 1 || a.M > kMaxMB || a.K % 32 != 0 || (reinterpret_cast<uintptr_t>(a.W) & 1u)) return cudaErrorNotSupported;
    if (a.fmt != FMT_Q4_0 && a.fmt != FMT_Q8_0) return cudaErrorNotSupported;
    RowsParams p{};
    p.W = a.W; p.X = a.X; p.Y = a.Y; p.gamma = a.gamma;
    p.N = a.N; p.K = a.K; p.nb = a.K / 32;
    p.nbp = p.nb | 1;
    p.chunks = (p.nb + 31) / 32;
    p.cb = (p.nb + p.chunks - 1) / p.chunks;
    p.x_f32 = a.x_f32; p.y_f32 = a.y_f32; p.eps = a.eps; p.wait_first = env.wait_first() ? 1 : 0;
    const uintptr_t mask = a.x_f32 ? 15u : 7u;
    p.x_vec = ((reinterpret_cast<uintptr_t>(a.X) | reinterpret_cast<uintptr_t>(a.gamma)) & mask) == 0;
    const int sms = env.sm_count > 0 ? env.sm_count : 148;
    const int groups = (a.N + kGroupRows - 1) / kGroupRows;
    const int grid = groups < sms ? groups : sms;
    p.max_rows = ((a.N + grid - 1) / grid + kGroupRows) / kGroupRows * kGroupRows;
    p.rows_of.set(a.N, grid);
    p.step_c = kRowsWarps / ((p.rows_of.run + (p.rows_of.longer > 0) + kGroupRows - 1) / kGroupRows);
    const long long off = static_cast<long long>(a.M) * 8 * p.nbp * 16;
    const long long bytes = off + static_cast<long long>(p.chunks) * p.max_rows * a.M * 4;
    if (bytes > env.smem_optin - 1024) return cudaErrorNotSupported;
    p.off_part = static_cast<int>(off);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(kRowsThreads);
    cfg.dynamicSmemBytes = static_cast<size_t>(bytes);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = env.pdl ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kRowsKernels[a.fmt == FMT_Q4_0 ? 0 : 1][a.M - 1], p);
}

}  // namespace tcb
