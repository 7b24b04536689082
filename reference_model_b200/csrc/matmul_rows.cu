// MATMUL with up to four rows of A (a classifier on a few images, a decoder's single position): every element of B meets only
// those rows, so the operator reads B once and nothing else counts; a 128-row tile of the tensor core would be padding.
//
// A block takes 128 columns, a lane four neighbouring ones (one 32-bit load of int8 or one 64-bit load of 16-bit elements per K
// row: 128 or 256 contiguous bytes per warp), its eight warps share out K, and up to eight blocks of a cluster share it again
// so that all SMs read.  Sixteen rows of B are in flight per lane.  int8: four K rows are transposed (eight byte permutes) into a
// word of four K elements per column, one dp4a per row of A; zero points through the sums of A's rows and B's columns.  16-bit:
// fp32 multiply-adds, sums of sixteen rows added in a fixed order.  What bounds it: the first bytes of B on small calls (2.7 to 4 us), B's
// bytes on large ones (fp16 1x4x8192x8192: 4.0 TB/s).
#include <algorithm>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.h"
#include "ptx_sm100.cuh"

namespace tb200
{
namespace
{

constexpr int kRowsThreads = 256, kRowsWarps = 8, kRowsCols = 128;

struct RowsParams
{
    const void* a;
    const void* b;
    void* out;
    int C, W, splits, k_per_cta;
    int32_t a_zp, b_zp;
    int out_f32;
};

// Loads that stay behind the wait for the predecessor in the stream, which may have written what they read: not through the path
// for data that nobody writes while the kernel is there.  Nothing is read twice, so L1 keeps none of it.
__device__ __forceinline__ uint32_t rows_load(const int8_t* p)
{
    uint32_t v;
    asm volatile("ld.global.cg.b32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
template <typename E>
__device__ __forceinline__ uint2 rows_load(const E* p)
{
    uint2 v;
    asm volatile("ld.global.cg.v2.b32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}

// Adds up `v` (H x 4 columns per lane) over the warps of the block and the blocks of the cluster, always in the same order; `use`
// gets (row, column of the block's 128, sum) for this block's share of the columns.
template <typename T, int H, typename F>
__device__ __forceinline__ void rows_reduce(const RowsParams& p, T (&v)[H][4], T (*part)[H][kRowsCols], T (*sum)[kRowsCols], F use)
{
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int h = 0; h < H; h++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            part[warp][h][lane * 4 + j] = v[h][j];
    __syncthreads();
    for (int e = tid; e < H * kRowsCols; e += kRowsThreads)
    {
        const int h = e / kRowsCols, c = e % kRowsCols;
        T s         = 0;
#pragma unroll
        for (int w = 0; w < kRowsWarps; w++)
            s += part[w][h][c];
        sum[h][c] = s;
    }
    const int rank = p.splits > 1 ? (int)ptx::cluster_ctarank() : 0;
    if (p.splits > 1)
        ptx::cluster_sync();
    else
        __syncthreads();
    const int own = kRowsCols / p.splits;
    for (int e = tid; e < H * own; e += kRowsThreads)
    {
        const int h = e / own, c = rank * own + e % own;
        T s         = 0;
        if (p.splits > 1)
            for (int r = 0; r < p.splits; r++)
            {
                uint32_t x;
                asm volatile("ld.shared::cluster.b32 %0, [%1];" : "=r"(x) : "r"(ptx::map_to_cta(ptx::smem_u32(&sum[h][c]), (uint32_t)r)) : "memory");
                s += *reinterpret_cast<const T*>(&x);
            }
        else
            s = sum[h][c];
        use(h, c, s);
    }
    if (p.splits > 1)
        ptx::cluster_sync();    // nobody leaves while another block may still read its sums
}

// row H of the sums: the columns of B (zero points)
template <int H>
__global__ void __launch_bounds__(kRowsThreads) matmul_rows_i8_kernel(const __grid_constant__ RowsParams p)
{
    __shared__ int32_t part[kRowsWarps][H + 1][kRowsCols];
    __shared__ int32_t sum[H + 1][kRowsCols];
    constexpr int P = kRowsWarps / H;    // warps that share out a row of A
    __shared__ int32_t row_part[H][P];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = p.splits > 1 ? (int)ptx::cluster_ctarank() : 0;
    const int col0 = (int)(blockIdx.x / (unsigned)p.splits) * kRowsCols, col = col0 + lane * 4;
    const int8_t* const A = reinterpret_cast<const int8_t*>(p.a) + (int64_t)blockIdx.y * H * p.C;
    const int8_t* const B = reinterpret_cast<const int8_t*>(p.b) + (int64_t)blockIdx.y * p.C * p.W + (col < p.W ? col : 0);
    const int k0 = rank * p.k_per_cta, k1 = min(p.C, k0 + p.k_per_cta);
    if (tid == 0)
        ptx::dep_launch_trigger();
    ptx::dep_launch_wait();
    // sums of A's rows over all of K, for B's zero point: the first words are asked for here and added up behind the loop (a warp
    // each behind it added a latency per 128 elements: 2x3x500x3168 7.7 us, 7.0 so)
    const bool summing = p.b_zp != 0 && warp < H * P;
    const int sum_k = (warp / H * 32 + lane) * 4, sum_step = P * 128;
    uint32_t row_words[4] = { 0, 0, 0, 0 };
    if (summing)
    {
#pragma unroll
        for (int j = 0; j < 4; j++)
            if (sum_k + j * sum_step < p.C)
                row_words[j] = rows_load(A + (int64_t)(warp % H) * p.C + sum_k + j * sum_step);
    }
    int32_t acc[H + 1][4];
#pragma unroll
    for (int h = 0; h <= H; h++)
        acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0;
    constexpr int U = 4;    // groups of four K rows in flight
    for (int k = k0 + warp * 4; k < k1; k += 4 * kRowsWarps * U)
    {
        uint32_t w[U][4], x[U][H];
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            const int kk  = k + u * 4 * kRowsWarps;
            const bool in = kk < k1;
#pragma unroll
            for (int i = 0; i < 4; i++)
                w[u][i] = in ? rows_load(B + (int64_t)(kk + i) * p.W) : 0u;
#pragma unroll
            for (int h = 0; h < H; h++)
                x[u][h] = in ? rows_load(A + (int64_t)h * p.C + kk) : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            const uint32_t lo01 = __byte_perm(w[u][0], w[u][1], 0x5140), hi01 = __byte_perm(w[u][0], w[u][1], 0x7362);
            const uint32_t lo23 = __byte_perm(w[u][2], w[u][3], 0x5140), hi23 = __byte_perm(w[u][2], w[u][3], 0x7362);
            const uint32_t t[4] = { __byte_perm(lo01, lo23, 0x5410), __byte_perm(lo01, lo23, 0x7632), __byte_perm(hi01, hi23, 0x5410),
                                    __byte_perm(hi01, hi23, 0x7632) };
#pragma unroll
            for (int j = 0; j < 4; j++)
            {
#pragma unroll
                for (int h = 0; h < H; h++)
                    acc[h][j] = __dp4a((int)t[j], (int)x[u][h], acc[h][j]);
                acc[H][j] = __dp4a((int)t[j], 0x01010101, acc[H][j]);
            }
        }
    }
    if (summing)
    {
        int32_t s = 0;
#pragma unroll
        for (int j = 0; j < 4; j++)
            s = __dp4a((int)row_words[j], 0x01010101, s);
        for (int k = sum_k + 4 * sum_step; k < p.C; k += sum_step)
            s = __dp4a((int)rows_load(A + (int64_t)(warp % H) * p.C + k), 0x01010101, s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0)
            row_part[warp % H][warp / H] = s;
    }
    // all sums of a column meet in shared memory again (the warps' parts have been added up by then)
    int32_t* const out = reinterpret_cast<int32_t*>(p.out) + (int64_t)blockIdx.y * H * p.W;
    int32_t* const cs  = &part[0][0][0];
    rows_reduce<int32_t, H + 1>(p, acc, part, sum, [&](int h, int c, int32_t s) { cs[h * kRowsCols + c] = s; });
    __syncthreads();
    const int own = kRowsCols / p.splits;
    for (int e = tid; e < H * own; e += kRowsThreads)
    {
        const int h = e / own, c = rank * own + e % own;
        int32_t row_sum = 0;
        if (p.b_zp != 0)
        {
#pragma unroll
            for (int j = 0; j < P; j++)
                row_sum += row_part[h][j];
        }
        if (col0 + c < p.W)
            out[(int64_t)h * p.W + col0 + c] =
                (int32_t)((uint32_t)cs[h * kRowsCols + c] - (uint32_t)p.a_zp * (uint32_t)cs[H * kRowsCols + c] - (uint32_t)p.b_zp * (uint32_t)row_sum +
                          (uint32_t)p.C * (uint32_t)(p.a_zp * p.b_zp));
    }
}

template <typename E>
__device__ __forceinline__ float2 rows_pair(uint32_t w);
template <>
__device__ __forceinline__ float2 rows_pair<__half>(uint32_t w)
{
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <>
__device__ __forceinline__ float2 rows_pair<__nv_bfloat16>(uint32_t w)
{
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
}
__device__ __forceinline__ void rows_store(__half* o, float v)
{
    *o = __float2half_rn(v);
}
__device__ __forceinline__ void rows_store(__nv_bfloat16* o, float v)
{
    *o = __float2bfloat16_rn(v);
}

template <typename E, int H>
__global__ void __launch_bounds__(kRowsThreads) matmul_rows_f16_kernel(const __grid_constant__ RowsParams p)
{
    __shared__ float part[kRowsWarps][H][kRowsCols];
    __shared__ float sum[H][kRowsCols];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rank = p.splits > 1 ? (int)ptx::cluster_ctarank() : 0;
    const int col0 = (int)(blockIdx.x / (unsigned)p.splits) * kRowsCols, col = col0 + lane * 4;
    const E* const A = reinterpret_cast<const E*>(p.a) + (int64_t)blockIdx.y * H * p.C;
    const E* const B = reinterpret_cast<const E*>(p.b) + (int64_t)blockIdx.y * p.C * p.W + (col < p.W ? col : 0);
    const int k0 = rank * p.k_per_cta, k1 = min(p.C, k0 + p.k_per_cta);
    if (tid == 0)
        ptx::dep_launch_trigger();
    ptx::dep_launch_wait();
    float acc[H][4];
#pragma unroll
    for (int h = 0; h < H; h++)
        acc[h][0] = acc[h][1] = acc[h][2] = acc[h][3] = 0.f;
    constexpr int U = 4;
    for (int k = k0 + warp * 4; k < k1; k += 4 * kRowsWarps * U)
    {
        uint2 w[U][4], x[U][H];
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            const int kk  = k + u * 4 * kRowsWarps;
            const bool in = kk < k1;
#pragma unroll
            for (int i = 0; i < 4; i++)
                w[u][i] = in ? rows_load(B + (int64_t)(kk + i) * p.W) : make_uint2(0, 0);
#pragma unroll
            for (int h = 0; h < H; h++)
                x[u][h] = in ? rows_load(A + (int64_t)h * p.C + kk) : make_uint2(0, 0);
        }
        // a pass sums its sixteen rows apart: one running sum over K / 8 rows is three times as far from the exact result
        // (K = 4000, not split over a cluster: 4.0e-7 of the result's root mean square, 1.4e-7 so)
        float sums[H][4];
#pragma unroll
        for (int h = 0; h < H; h++)
            sums[h][0] = sums[h][1] = sums[h][2] = sums[h][3] = 0.f;
#pragma unroll
        for (int u = 0; u < U; u++)
        {
            float xs[H][4];
#pragma unroll
            for (int h = 0; h < H; h++)
            {
                const float2 lo = rows_pair<E>(x[u][h].x), hi = rows_pair<E>(x[u][h].y);
                xs[h][0] = lo.x; xs[h][1] = lo.y; xs[h][2] = hi.x; xs[h][3] = hi.y;
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
            {
                const float2 lo = rows_pair<E>(w[u][i].x), hi = rows_pair<E>(w[u][i].y);
#pragma unroll
                for (int h = 0; h < H; h++)
                {
                    sums[h][0] = fmaf(xs[h][i], lo.x, sums[h][0]);
                    sums[h][1] = fmaf(xs[h][i], lo.y, sums[h][1]);
                    sums[h][2] = fmaf(xs[h][i], hi.x, sums[h][2]);
                    sums[h][3] = fmaf(xs[h][i], hi.y, sums[h][3]);
                }
            }
        }
#pragma unroll
        for (int h = 0; h < H; h++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                acc[h][j] += sums[h][j];
    }
    rows_reduce<float, H>(p, acc, part, sum, [&](int h, int c, float s) {
        if (col0 + c >= p.W)
            return;
        const int64_t at = ((int64_t)blockIdx.y * H + h) * p.W + col0 + c;
        if (p.out_f32)
            reinterpret_cast<float*>(p.out)[at] = s;
        else
            rows_store(reinterpret_cast<E*>(p.out) + at, s);
    });
}

typedef void (*RowsKern)(const RowsParams);

}    // namespace

// Whole words of both operands; K deep enough to share out, and no more rows than the kernels' 32-bit indexes (which step past the
// last one) reach.  65 535 batches are a grid's limit.  Per call, against the tensor core's
// tiles (us): int8 1x1x2048x1000 5.3 / 9.5, 1x4x256x64 4.0 / 16.3, 32x3x1024x512 7.5 / 23.9, 1x4x8192x8192 23 / 51, 1000x4x256x256
// 25 / 45; fp16 1x1x2048x1000 4.5 / 24.6, 1x4x256x64 3.8 / 8.2, 8x2x4096x1024 17.1 / 42.1, 1x4x8192x8192 35 / 78, 1000x1x256x64
// 8.3 / 16.4, but 1000x4x256x256 36 / 31: with more than eight blocks per SM the tiles' own loads keep memory busy, and several
// rows of 16-bit elements cost a conversion and a multiply-add each.  Over 460 shapes the time is 0.56 of the tiles'; they are faster
// in some with about a block per SM: int8 16x1x488x880 8.2 / 6.7, fp16 34x2x3208x416 27.9 / 19.5 (but 13x2x2848x944 13.9 / 27.8).
bool matmul_rows_supported(tb200_dtype dt, const void* a, const void* b, int N, int H, int C, int W, int num_sms)
{
    const uintptr_t al = dt == TB200_INT8 ? 3 : 7;
    return (dt == TB200_INT8 || dt == TB200_FP16 || dt == TB200_BF16) && H >= 1 && H <= 4 && C >= 256 && C <= (1 << 30) && W >= 4 && C % 4 == 0 && W % 4 == 0 && N <= 65535 &&
           !(dt != TB200_INT8 && H > 1 && C % 8 == 0 && W % 8 == 0 && (int64_t)N * ((W + kRowsCols - 1) / kRowsCols) > 8 * (int64_t)num_sms) &&
           ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & al) == 0;
}

tb200_status matmul_rows_launch(tb200_ctx* ctx, tb200_dtype dt, const void* a, const void* b, void* out, tb200_dtype out_dt, int N, int H, int C, int W,
                                int32_t a_zp, int32_t b_zp)
{
    static const RowsKern kerns[3][4] = {
        { matmul_rows_i8_kernel<1>, matmul_rows_i8_kernel<2>, matmul_rows_i8_kernel<3>, matmul_rows_i8_kernel<4> },
        { matmul_rows_f16_kernel<__half, 1>, matmul_rows_f16_kernel<__half, 2>, matmul_rows_f16_kernel<__half, 3>, matmul_rows_f16_kernel<__half, 4> },
        { matmul_rows_f16_kernel<__nv_bfloat16, 1>, matmul_rows_f16_kernel<__nv_bfloat16, 2>, matmul_rows_f16_kernel<__nv_bfloat16, 3>,
          matmul_rows_f16_kernel<__nv_bfloat16, 4> } };
    RowsParams p;
    p.a = a; p.b = b; p.out = out; p.C = C; p.W = W; p.a_zp = a_zp; p.b_zp = b_zp;
    p.out_f32 = out_dt == TB200_FP32 ? 1 : 0;
    const int type      = dt == TB200_INT8 ? 0 : dt == TB200_FP16 ? 1 : 2;
    const RowsKern kern = kerns[type][H - 1];
    int& resident       = ctx->rows_blocks[type * 4 + H - 1];
    if (resident == 0)
    {
        int occ = 0;
        TB200_CUDA_CHECK(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kRowsThreads, 0));
        resident = std::max(1, occ);
    }
    // K over a cluster while that leaves a block 128 rows and the grid is below one block per SM, or still fits the SMs at once: it is
    // the bytes in flight that a grid of one or two blocks per SM lacks (int8, up to one block per SM, so, and the tensor core's tiles, us:
    // 4x1x2228x1840 16.8 / 11.1 / 10.6, 34x4x1248x288 15.0 / 10.8 / 10.5, 7x3x788x2000 11.1 / 7.5 / 8.3, 1x4x8192x8192 37 / 23 / 51).
    const int64_t blocks = (int64_t)((W + kRowsCols - 1) / kRowsCols) * N;
    p.splits = 1;
    while (p.splits < 8 && C / (2 * p.splits) >= 128 &&
           (blocks * p.splits < ctx->num_sms || blocks * p.splits * 2 <= (int64_t)resident * ctx->num_sms))
        p.splits *= 2;
    p.k_per_cta = ((C + p.splits - 1) / p.splits + 3) & ~3;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim  = dim3((unsigned)((W + kRowsCols - 1) / kRowsCols * p.splits), (unsigned)N);
    cfg.blockDim = dim3(kRowsThreads);
    cfg.stream   = ctx->stream;
    cudaLaunchAttribute at[2];
    at[0].id               = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)p.splits;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs    = at;
    cfg.numAttrs = ctx->launch_overlap ? 2 : 1;
    timer_begin(ctx);
    cudaLaunchKernelEx(&cfg, kern, p);
    timer_end(ctx);
    return post_launch(ctx, dt == TB200_INT8 ? "matmul_rows_i8" : "matmul_rows_f16");
}

}    // namespace tb200
