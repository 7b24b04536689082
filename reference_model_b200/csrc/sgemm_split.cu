// fp32 batched MATMUL and CONV2D on the tensor cores without giving up fp32: every operand is taken apart into three bf16
// values whose sum is the operand, exactly (the first two rounded to nearest: what is left has 16, then 7 significant bits),
// and a product is the six partial products that matter (a0 b0, a0 b1, a1 b0, a0 b2, a1 b1, a2 b0).  The three left out come
// to at most 2^-24 of it, of either sign: |a1| <= 2^-8, |a2| <= 2^-17 of the operand's power of two.  (Parts that are cut off
// instead leave out up to 2^-21, always of the product's sign.)  bf16 has fp32's exponent range, so nothing has to be scaled.
//
// Sums.  The tensor core cuts its running sum off instead of rounding it, so it never carries one far, and the leading
// products not beside the small ones: per stage of 64 K elements one accumulator takes a0 b0 (products of 16 bits, whose sums
// mostly fit 24), and another, over four stages, the five others (whose cut-off is 2^-8 of the result's).  Both are read back and
// added to fp32 accumulators in registers, rounded to nearest.
// Error against 64 bits, relative 2-norm, K = 256 / 1024 / 4096: normal operands 8.0e-8 / 1.1e-7 / 1.8e-7 (multiply-adds in K
// order 2.9e-7 / 5.7e-7 / 1.1e-6), positive ones 4.0e-8 / 7.7e-8 / 1.4e-7 (2.4e-7 / 4.8e-7 / 9.6e-7); one product per sum 2.52e-8
// (2.48e-8).
//
// One persistent CTA per SM, 128 x 128 output tiles, sixteen warps:
//   warps 0-7   add up stages (32 rows x 64 columns each, 64 accumulators per thread), finish and store the tile; the first
//               issues the MMAs, 24 of 128 x 128 x 16 per stage;
//   warps 8-15  load fp32 operands straight into registers (64 K elements ahead), take them apart and store three planes in
//               the tensor core's swizzled layouts.  A warp's unit is 64 elements, two neighbours per lane, so that one code
//               path serves any alignment, a gathered convolution window and both operands without bank conflicts.
// Taking operands apart inside the kernel instead of in a pass before it keeps the planes out of memory (3.2 GB for 64
// products of 1024 x 4096 x 1024).  4 x 1024 x 4096 x 1024: 257 us (FFMA kernel 828), 3 800 SM cycles per stage.  What bounds it:
// the MMAs alone take 2 680 (24 of ~107 and the hand-over), the loads 3 300 on their own: 64 KB a stage through the ~28 KB of
// L1 that two 96 KB stages leave.  Three stages of 32 K elements with more L1 lose more to commits and hand-overs (4 500).
//
// Values the split cannot carry are computed again with ordinary multiply-adds:
//   * results that are not finite (an infinite operand has no split: its lower parts are NaN, so it always shows);
//   * results so small that what parts and partial products lose below the normal range, 2^-126, could show in them.  A product
//     loses at most 2^-126 (|a| + |b| + 6), so a sum of K of them is trusted where half its last place is above K times that
//     for the largest magnitudes of its row and column: |y| >= K 2^-101 (row + column + 8).  Only a tile with a non-zero
//     operand below 2^-48 can have lost anything: without one all products are above 2^-96.
#include <algorithm>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "common.h"
#include "ptx_sm100.cuh"

namespace tb200
{
namespace
{

constexpr int kTile = 128, kHalfK = 32, kStageK = 2 * kHalfK, kStages = 2;
constexpr int kAccs = 2;           // accumulators of a0 b0, one per stage, and of the five small partial products, one per
constexpr int kSmallStages = 4;    // so many stages of a tile, behind each other in tensor memory
constexpr int kBigCol = 2 * kTile, kTmemCols = 4 * kTile;
constexpr int kPlane = kTile * kHalfK * 2;       // bytes of one bf16 plane of 32 K elements of an operand
constexpr int kHalfBytes = 6 * kPlane, kStageBytes = 2 * kHalfBytes;    // A planes, B planes of 32 K elements, twice
constexpr int kFlushWarps = 8, kSplitWarps = 8;
constexpr int kSplitThreads = 32 * (kFlushWarps + kSplitWarps);
constexpr int kStagePitch = 17;                   // staged output: 32 rows x 16 columns per warp
constexpr int kOutOff  = kStages * kStageBytes;
constexpr int kRowsOff = kOutOff + kFlushWarps * 32 * kStagePitch * 4;    // int2[128]: window origins of a convolution's rows
constexpr int kAgainSlots = 128;
constexpr int kMagOff  = kRowsOff + kTile * 8;    // for even and odd tiles: largest magnitudes of rows, of columns by warp, small_key()s
constexpr int kMinOff  = kTile + kSplitWarps * kTile, kMagWords = kMinOff + kSplitWarps;
constexpr int kSplitSmem = kMagOff + 2 * kMagWords * 4 + 1024;

struct SplitParams
{
    const float* a;
    const float* b;
    float* out;
    int M, N, K;
    int64_t a_batch, b_batch, o_batch;
    int ldb;
    int tiles_m, tiles_n, tiles, nk;
    int IH, IW, IC, OH, OW, KW, pad_t, pad_l, sy, sx, dy, dx;
    int in_sn, in_sh, in_sw;
    const float* bias;
    int bias_n;
    int has_clamp;
    float clamp_lo, clamp_hi;
    uint32_t idesc;
    uint64_t a_desc_hi, b_desc_hi;
    long long wait_limit;
    int* status;
};

// origin of an output row's window: element offset, iy0 | ix0
__device__ __forceinline__ int2 window_of(const SplitParams& p, int m)
{
    const int ox = m % p.OW, q = m / p.OW;
    const int oy = q % p.OH, n = q / p.OH;
    const int iy0 = oy * p.sy - p.pad_t, ix0 = ox * p.sx - p.pad_l;
    return make_int2(n * p.in_sn + iy0 * p.in_sh + ix0 * p.in_sw, (int)(((uint32_t)iy0 << 16) | ((uint32_t)ix0 & 0xffffu)));
}

__device__ __forceinline__ bool window_has(const SplitParams& p, int2 r, int y, int x)
{
    return (unsigned)((r.y >> 16) + y) < (unsigned)p.IH && (unsigned)((int)(short)r.y + x) < (unsigned)p.IW;
}

// Loads with a predicate and no branch around them: a branch makes the compiler wait for each load where the paths join.
__device__ __forceinline__ float2 load2_if(const float* src, bool inside)
{
    float2 v;
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %3, 0;\nmov.b32 %0, 0;\nmov.b32 %1, 0;\n@p ld.global.nc.v2.f32 {%0, %1}, [%2];\n}\n"
                 : "=&f"(v.x), "=&f"(v.y)
                 : "l"(src), "r"((int)inside));
    return v;
}

__device__ __forceinline__ float load1_if(const float* src, bool inside)
{
    float v;
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %2, 0;\nmov.b32 %0, 0;\n@p ld.global.nc.f32 %0, [%1];\n}\n"
                 : "=&f"(v)
                 : "l"(src), "r"((int)inside));
    return v;
}

__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi)
{
    const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// Two fp32 values as three packed bf16 pairs.  (A value that rounds to infinity leaves NaN: its results are computed again.)
__device__ __forceinline__ void split3(float2 v, uint32_t (&w)[3])
{
    w[0] = bf16_pair(v.x, v.y);
    const float rx = v.x - __uint_as_float(w[0] << 16), ry = v.y - __uint_as_float(w[0] & 0xffff0000u);
    w[1] = bf16_pair(rx, ry);
    const float sx = rx - __uint_as_float(w[1] << 16), sy = ry - __uint_as_float(w[1] & 0xffff0000u);
    w[2] = __byte_perm(__float_as_uint(sx), __float_as_uint(sy), 0x7632);    // exact: at most seven bits are left
}

// Largest magnitude; NaN counts for nothing.
__device__ __forceinline__ float max_abs(float m, float x, float y)
{
    asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(m) : "f"(x), "f"(y));
    return m;
}

// A value whose magnitude grows as that of x falls; NaN for zero and NaN.  (2^-48: 127 - 48 is its biased exponent.)
__device__ __forceinline__ float small_key(float x)
{
    return __uint_as_float(0x7f800001u - __float_as_uint(x));
}
constexpr uint32_t kSmallKey = 0x7f800001u - (79u << 23);

// A result: bias and CLAMP of a convolution.
template <bool CONV>
__device__ __forceinline__ float finish(const SplitParams& p, int n, float y)
{
    if (CONV)
    {
        y = (p.bias_n == 1 ? __ldg(p.bias) : n < p.N ? __ldg(p.bias + n) : 0.f) + y;
        if (p.has_clamp)
        {
            y = (y < p.clamp_lo) ? p.clamp_lo : y;
            y = (y > p.clamp_hi) ? p.clamp_hi : y;
        }
    }
    return y;
}

// 32 rows x 32 columns of the output with ordinary multiply-adds, K in order: a lane's row, column by column.  One warp, eight
// K elements at a time through `st`: A as 32 rows of nine words (no bank conflicts), then B as eight rows of 32.  Per K element
// a warp reads one word of A and eight broadcast quads of B for its 32 multiply-adds, as the FFMA kernel does.  Taps outside
// the image are skipped, whatever their weight.
// (40 x 256 x 4096 x 256, every block: 2.3 ms, where a row and sixteen columns at a time inside the pipeline took 25.)
template <bool CONV>
__device__ __noinline__ void plain_block(const SplitParams& p, int batch, int m0, int n0, float* st)
{
    const int lane = threadIdx.x & 31, kq = lane & 7, rq = lane >> 3;
    const float* const A = p.a + batch * p.a_batch;
    const float* const B = p.b + batch * p.b_batch;
    const int2 r  = !CONV ? make_int2(0, 0) : m0 + lane < p.M ? window_of(p, m0 + lane) : make_int2(0, (int)0x80008000);
    const bool in = n0 + lane < p.N;
    int ic = 0, ky = 0, kx = 0;    // CONV: of K element k + kq
    if (CONV)
    {
        const int tap = kq / p.IC;
        ic = kq - tap * p.IC;
        ky = tap / p.KW;
        kx = tap - ky * p.KW;
    }
    float ra[8], rb[8];
    uint32_t taps = 0, next_taps = 0;    // CONV: which of the piece's K elements lie inside the image, for this lane's row
    auto load = [&](int k) {
        const int y = ky * p.dy, x = kx * p.dx;
        next_taps   = 0;
#pragma unroll
        for (int i = 0; i < 8; i++)
        {
            const int row = rq + 4 * i;
            if (CONV)
            {
                const int2 o = make_int2(__shfl_sync(0xffffffffu, r.x, row), __shfl_sync(0xffffffffu, r.y, row));
                const bool inside = k + kq < p.K && window_has(p, o, y, x);
                ra[i]             = load1_if(A + (o.x + y * p.in_sh + x * p.in_sw + ic), inside);
                // (lanes 8 rq + kq: byte rq of the ballot belongs to row rq + 4 i)
                const uint32_t all = __ballot_sync(0xffffffffu, inside);
                if (lane >> 2 == i)
                    next_taps = all >> (8 * (lane & 3)) & 0xffu;
            }
            else
                ra[i] = load1_if(A + (int64_t)(m0 + row) * p.K + k + kq, k + kq < p.K && m0 + row < p.M);
            rb[i] = load1_if(B + (int64_t)(k + i) * p.ldb + n0 + lane, k + i < p.K && in);
        }
        if (CONV)
            for (ic += 8; ic >= p.IC;)
            {
                ic -= p.IC;
                if (++kx == p.KW)
                {
                    kx = 0;
                    ky++;
                }
            }
    };
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; j++)
        v[j] = 0.f;
    float* const as = st;
    float* const bs = st + 32 * 9;
    load(0);
    for (int k = 0; k < p.K; k += 8)
    {
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; i++)
        {
            as[(rq + 4 * i) * 9 + kq] = ra[i];
            bs[i * 32 + lane]         = rb[i];
        }
        __syncwarp();
        taps = next_taps;
        if (k + 8 < p.K)
            load(k + 8);
#pragma unroll
        for (int i = 0; i < 8; i++)
        {
            const float x = as[lane * 9 + i];
            if (CONV && !(taps >> i & 1))
                continue;
#pragma unroll
            for (int j = 0; j < 32; j += 4)
            {
                const float4 b = *reinterpret_cast<const float4*>(bs + i * 32 + j);
                v[j]     = fmaf(x, b.x, v[j]);
                v[j + 1] = fmaf(x, b.y, v[j + 1]);
                v[j + 2] = fmaf(x, b.z, v[j + 2]);
                v[j + 3] = fmaf(x, b.w, v[j + 3]);
            }
        }
    }
    __syncwarp();
    float* const o = p.out + batch * p.o_batch + (int64_t)(m0 + lane) * p.N + n0;
    if (m0 + lane < p.M)
#pragma unroll
        for (int j = 0; j < 32; j++)
            if (n0 + j < p.N)
                o[j] = finish<CONV>(p, n0 + j, v[j]);
}

// AVEC, BVEC: pairs of neighbouring elements of A along K (CONV: along the channels), of B along its rows, are aligned to
// eight bytes and never straddle an edge.
template <bool CONV, bool AVEC, bool BVEC>
__global__ void __launch_bounds__(kSplitThreads, 1) sgemm_split_kernel(const __grid_constant__ SplitParams p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kStages], bar_acc[kAccs], bar_free[kAccs], bar_done;
    __shared__ uint32_t tmem_base_holder;
    __shared__ uint32_t again[kAgainSlots];    // blocks of 32 x 32 to be computed again, a bit each, of tiles slot, slot + kAgainSlots, ...

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* const sm   = smem_raw + (base - ptx::smem_u32(smem_raw));
    int2* const rows    = reinterpret_cast<int2*>(sm + kRowsOff);
    float* const mags   = reinterpret_cast<float*>(sm + kMagOff);

    if (tid < kAgainSlots)
        again[tid] = 0;
    if (tid == 0)
    {
        for (int s = 0; s < kStages; s++)
            ptx::mbar_init(ptx::smem_u32(&bar_full[s]), kSplitWarps);
        for (int s = 0; s < kAccs; s++)
        {
            ptx::mbar_init(ptx::smem_u32(&bar_acc[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&bar_free[s]), kFlushWarps);
        }
        ptx::mbar_init(ptx::smem_u32(&bar_done), 1);
        ptx::fence_barrier_init();
    }
    if (warp == kFlushWarps)
    {
        ptx::tmem_alloc(ptx::smem_u32(&tmem_base_holder), kTmemCols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = tmem_base_holder;
    if (tid == 0)
        ptx::dep_launch_trigger();

    bool ok = true;
    const int per = p.tiles_m * p.tiles_n;
    const int mine  = p.tiles > (int)blockIdx.x ? (p.tiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
    const int total = mine * p.nk;
    if (warp < kFlushWarps)
    {
        // ------------------------------------------------------------------ sums
        ptx::dep_launch_wait();    // the predecessor may still read what is written here
        const int quarter = warp & 3, half = warp >> 2;
        const int row     = quarter * 32 + lane;
        const uint32_t t0 = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 64);
        float* const st   = reinterpret_cast<float*>(sm + kOutOff) + warp * 32 * kStagePitch;
        const bool v8 = (p.N & 7) == 0 && (reinterpret_cast<uintptr_t>(p.out) & 31) == 0;
        // The stage's MMAs, by the first lane of the first of these warps: issuing takes as long as the MMAs before take to make
        // room in the unit's short queue, so a splitting warp must not do it (the two then take turns: 5 600 cycles a stage), and a warp of its own, the seventeenth, would leave 96 registers per thread instead of 128.
        // These warps have time: a stage's sums take about a third of its MMAs.
        int issue_k = 0, issue_small = 0;    // stage of its tile and small accumulator of the next issue
        auto issue = [&](int c) {
            const int buf = c % kAccs, slot = c % kStages;
            if (!ptx::mbar_wait_bounded(ptx::smem_u32(&bar_free[buf]), ((uint32_t)(c / kAccs) & 1u) ^ 1u, p.wait_limit) ||
                !ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[slot]), (uint32_t)(c / kStages) & 1u, p.wait_limit))
                return false;
            ptx::tc_fence_after_sync();
            const uint32_t s = base + (uint32_t)(slot * kStageBytes);
            uint32_t accum   = issue_k % kSmallStages != 0;
            const uint32_t small = tmem + (uint32_t)(issue_small * kTile), big = tmem + (uint32_t)(kBigCol + buf * kTile);
            if (++issue_k == p.nk)
                issue_k = 0;
            if (issue_k % kSmallStages == 0)
                issue_small ^= 1;
            // smallest first: a0 b2, a1 b1, a2 b0, a0 b1, a1 b0; then a0 b0 into an accumulator of its own
            constexpr int pa[6] = { 0, 1, 2, 0, 1, 0 }, pb[6] = { 2, 1, 0, 1, 0, 0 };
#pragma unroll
            for (int q = 0; q < 6; q++)
            {
                if (q == 5)
                    accum = 0;
#pragma unroll
                for (int h = 0; h < 2; h++)
                {
                    uint64_t ad = ptx::smem_desc(p.a_desc_hi, s + (uint32_t)(h * kHalfBytes + pa[q] * kPlane));
                    uint64_t bd = ptx::smem_desc(p.b_desc_hi, s + (uint32_t)(h * kHalfBytes + (3 + pb[q]) * kPlane));
#pragma unroll
                    for (int kk = 0; kk < kHalfK / 16; kk++, ad += 2, bd += 128)    // 32 bytes along a row; sixteen K rows
                    {
                        ptx::mma_f16_ss(q == 5 ? big : small, ad, bd, p.idesc, accum);
                        accum = 1;
                    }
                }
            }
            ptx::mma_commit(ptx::smem_u32(&bar_acc[buf]));
            return true;
        };
        if (warp == 0)
        {
            if (lane == 0 && total > 0)
                ok = issue(0);
            ok = __all_sync(0xffffffffu, ok);
        }
        int c = 0, small = 0;
        for (int i = 0, tile = (int)blockIdx.x; tile < p.tiles && ok; i++, tile += (int)gridDim.x)
        {
            const int batch = tile / per, rem = tile - batch * per, tm = rem / p.tiles_n;
            const int m0 = tm * kTile, n0 = (rem - tm * p.tiles_n) * kTile + half * 64;
            float acc[64];
#pragma unroll
            for (int j = 0; j < 64; j++)
                acc[j] = 0.f;
            for (int k = 0; k < p.nk; k++, c++)
            {
                const int buf = c % kAccs;
                if (warp == 0)
                {
                    if (lane == 0 && c + 1 < total)
                        ok = ok && issue(c + 1);
                    __syncwarp();
                }
                ok = ok && ptx::mbar_wait_bounded(ptx::smem_u32(&bar_acc[buf]), (uint32_t)(c / kAccs) & 1u, p.wait_limit);
                ok = __all_sync(0xffffffffu, ok);
                if (!ok)
                    break;
                ptx::tc_fence_after_sync();
                // (bar_free of a stage also frees the small accumulator that the stage two later may start: its last use was
                // read back before)
                const bool last = (k + 1) % kSmallStages == 0 || k + 1 == p.nk;
                if (last)
                {
#pragma unroll
                    for (int h = 0; h < 2; h++)
                    {
                        uint32_t v[32];
                        ptx::tmem_ld_32x32b_x32(t0 + (uint32_t)(small * kTile + h * 32), v);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 32; j++)
                            acc[h * 32 + j] += __uint_as_float(v[j]);
                    }
                    small ^= 1;
                }
#pragma unroll
                for (int h = 0; h < 2; h++)
                {
                    uint32_t v[32];
                    ptx::tmem_ld_32x32b_x32(t0 + (uint32_t)(kBigCol + buf * kTile + h * 32), v);
                    ptx::tmem_ld_wait();
                    if (h == 1)
                    {
                        ptx::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0)
                            ptx::mbar_arrive(ptx::smem_u32(&bar_free[buf]));
                    }
#pragma unroll
                    for (int j = 0; j < 32; j++)
                        acc[h * 32 + j] += __uint_as_float(v[j]);
                }
            }
            if (!ok)
                break;
            // Magnitudes of this row and of this warp's columns.  The splitting warps come back to this half of the table two
            // tiles, at least eight stages, later; they are never more than four stages ahead (two in shared memory, two in
            // tensor memory).
            const float* const mg = mags + (i & 1) * kMagWords;
            const int m           = m0 + row;
            uint32_t odd[2]       = { 0, 0 };    // columns to be computed again
#pragma unroll
            for (int j = 0; j < 64; j++)
                odd[j >> 5] |= isfinite(acc[j]) ? 0u : 1u << (j & 31);
            float least = 0.f;
#pragma unroll
            for (int q = 0; q < kSplitWarps; q++)
                least = fmaxf(least, mg[kMinOff + q]);
            if (least > __uint_as_float(kSmallKey))
            {
                const float rmag = mg[row], lim = (float)p.K * 3.9443045e-31f;    // 2^-101
                float cmag0 = 0.f, cmag1 = 0.f;                                   // columns lane, 32 + lane
#pragma unroll
                for (int q = 0; q < kSplitWarps; q++)
                {
                    cmag0 = fmaxf(cmag0, mg[kTile + q * kTile + half * 64 + lane]);
                    cmag1 = fmaxf(cmag1, mg[kTile + q * kTile + half * 64 + 32 + lane]);
                }
#pragma unroll
                for (int j = 0; j < 64; j++)
                {
                    const float cm = __shfl_sync(0xffffffffu, j < 32 ? cmag0 : cmag1, j & 31);
                    if (rmag != 0.f && cm != 0.f && fabsf(acc[j]) < fmaf(lim, rmag + cm, 8.f * lim))
                        odd[j >> 5] |= 1u << (j & 31);
                }
            }
#pragma unroll
            for (int h = 0; h < 2; h++)
                if (n0 + h * 32 < p.N && __any_sync(0xffffffffu, odd[h] != 0) && lane == 0)
                    atomicOr(&again[i % kAgainSlots], 1u << (quarter * 4 + half * 2 + h));
#pragma unroll
            for (int g = 0; g < 4; g++)
            {
                float* const y = acc + g * 16;
                const int n    = n0 + g * 16;
                if (n >= p.N)
                    break;
#pragma unroll
                for (int j = 0; j < 16; j++)
                    y[j] = finish<CONV>(p, n + j, y[j]);
                float* const o = p.out + batch * p.o_batch + (int64_t)m * p.N + n;
                if (v8)
                {
                    if (m < p.M)
                    {
#pragma unroll
                        for (int j = 0; j < 16; j += 8)
                            if (n + j < p.N)
                                ptx::st_global_v8(o + j, __float_as_uint(y[j]), __float_as_uint(y[j + 1]), __float_as_uint(y[j + 2]),
                                                  __float_as_uint(y[j + 3]), __float_as_uint(y[j + 4]), __float_as_uint(y[j + 5]),
                                                  __float_as_uint(y[j + 6]), __float_as_uint(y[j + 7]));
                    }
                }
                else
                {
                    // rows of any alignment: through shared memory, half a warp per row and store
#pragma unroll
                    for (int j = 0; j < 16; j++)
                        st[lane * kStagePitch + j] = y[j];
                    __syncwarp();
                    const int col = lane & 15;
                    float* const og = p.out + batch * p.o_batch + (int64_t)(m0 + quarter * 32) * p.N + n;
#pragma unroll 4
                    for (int r = lane >> 4; r < 32; r += 2)
                        if (m0 + quarter * 32 + r < p.M && n + col < p.N)
                            og[(int64_t)r * p.N + col] = st[r * kStagePitch + col];
                    __syncwarp();
                }
            }
        }
        if (warp == 0 && lane == 0)
        {
            ptx::mma_commit(ptx::smem_u32(&bar_done));
            ptx::mbar_wait_bounded(ptx::smem_u32(&bar_done), 0u, 40000000LL);    // (nothing to wait for unless a role gave up)
        }
        __syncwarp();
    }
    else
    {
        // ------------------------------------------------------------------ load, take apart, store
        // A warp's unit is 64 elements: two neighbouring rows x 32 K elements of A (64-byte swizzle), 64 columns of one K row of
        // B (128-byte swizzle).  Eight units of each per stage, w, w + 8, ...: their places in the swizzle are the same.
        const int w = warp - kFlushWarps;
        const int kl = 2 * (lane & 15), odd = lane >> 4;    // this lane's K elements of a unit of A, and which row
        const uint32_t dst_a = base + (uint32_t)(w * 128 + odd * 64 + ((((lane >> 2) & 3) ^ (w & 3)) << 4) + (lane & 3) * 4);
        const uint32_t dst_b = base + (uint32_t)(3 * kPlane + w * 128 + (((lane >> 2) ^ w) << 4) + (lane & 3) * 4);
        ptx::dep_launch_wait();
        // The loads run two halves, one stage, ahead of what is being taken apart, across tiles; past the last tile they load nothing.
        int tile = (int)blockIdx.x, kstage = 0;
        const float* A = p.a;    // MATMUL: this lane's elements of its first row; CONV2D: the input
        const float* B = p.b;    // this lane's elements of K row w
        int nrows = 0;           // MATMUL: rows of the tile from this lane's first one on
        int ncols = 0;           // columns of the tile
        int kleft = 0;           // K elements from the stage's first to the end
        int ic[2] = {}, ky[2] = {}, kx[2] = {};                // CONV: channels and taps of this lane's elements (one tap for both if AVEC)
        auto next_tap = [&](int q, int step) {
            ic[q] += step;
            while (ic[q] >= p.IC)
            {
                ic[q] -= p.IC;
                if (++kx[q] == p.KW)
                {
                    kx[q] = 0;
                    ky[q]++;
                }
            }
        };
        auto start_tile = [&]() {
            kstage = 0;
            kleft  = tile < p.tiles ? p.K : 0;
            if (tile >= p.tiles)
                return;
            const int batch = tile / per, rem = tile - batch * per, tm = rem / p.tiles_n;
            const int m0 = tm * kTile, n0 = (rem - tm * p.tiles_n) * kTile;
            A     = p.a + batch * p.a_batch;
            B     = p.b + batch * p.b_batch + (int64_t)w * p.ldb + n0 + 2 * lane;
            ncols = (BVEC ? p.ldb : p.N) - n0;    // (BVEC: the same, or zeros up to an even count)
            if (CONV)
            {
                __syncwarp();
                if (lane < 16)    // (a warp reads its own rows only)
                {
                    const int r = 2 * (w + 8 * (lane >> 1)) + (lane & 1);
                    rows[r]     = m0 + r < p.M ? window_of(p, m0 + r) : make_int2(0, (int)0x80008000);
                }
                __syncwarp();
#pragma unroll
                for (int q = 0; q < 2; q++)
                {
                    ic[q] = ky[q] = kx[q] = 0;
                    next_tap(q, kl + q);
                }
            }
            else
            {
                nrows = p.M - m0 - (2 * w + odd);
                A += (int64_t)(m0 + 2 * w + odd) * p.K + kl;
            }
        };
        auto load_a = [&](float2 (&v)[8]) {
            if (CONV)
            {
                int off[2], y[2], x[2];
#pragma unroll
                for (int q = 0; q < (AVEC ? 1 : 2); q++)
                {
                    y[q]   = ky[q] * p.dy;
                    x[q]   = kx[q] * p.dx;
                    off[q] = y[q] * p.in_sh + x[q] * p.in_sw + ic[q];
                }
#pragma unroll
                for (int i = 0; i < 8; i++)
                {
                    const int2 o = rows[2 * (w + 8 * i) + odd];
                    if (AVEC)
                        v[i] = load2_if(A + (o.x + off[0]), kl < kleft && window_has(p, o, y[0], x[0]));
                    else
                        v[i] = make_float2(load1_if(A + (o.x + off[0]), kl < kleft && window_has(p, o, y[0], x[0])),
                                           load1_if(A + (o.x + off[1]), kl + 1 < kleft && window_has(p, o, y[1], x[1])));
                }
            }
            else
            {
#pragma unroll
                for (int i = 0; i < 8; i++)
                {
                    const float* s = A + (int64_t)(16 * i) * p.K;
                    const bool row = 16 * i < nrows;
                    if (AVEC)
                        v[i] = load2_if(s, row && kl < kleft);
                    else
                        v[i] = make_float2(load1_if(s, row && kl < kleft), load1_if(s + 1, row && kl + 1 < kleft));
                }
            }
        };
        auto load_b = [&](float2 (&v)[8]) {
#pragma unroll
            for (int i = 0; i < 8; i++)
            {
                const int n    = 2 * lane + (i & 1) * 64;
                const float* s = B + (int64_t)(8 * (i >> 1)) * p.ldb + (i & 1) * 64;
                const bool k   = w + 8 * (i >> 1) < kleft;
                if (BVEC)
                    v[i] = load2_if(s, k && n < ncols);
                else
                    v[i] = make_float2(load1_if(s, k && n < ncols), load1_if(s + 1, k && n + 1 < ncols));
            }
        };
        auto next_half = [&]() {
            kleft -= kHalfK;
            if (++kstage == 2 * p.nk)
            {
                tile += (int)gridDim.x;
                start_tile();
                return;
            }
            B += (int64_t)kHalfK * p.ldb;
            if (CONV)
            {
#pragma unroll
                for (int q = 0; q < (AVEC ? 1 : 2); q++)
                    next_tap(q, kHalfK);
            }
            else
                A += kHalfK;
        };
        float mag_a[8], mag_b[4];    // largest magnitudes: rows, columns of even and odd units
        float least = 0.f;           // largest small_key() of both operands
        auto clear = [&]() {
#pragma unroll
            for (int i = 0; i < 8; i++)
                mag_a[i] = 0.f;
            mag_b[0] = mag_b[1] = mag_b[2] = mag_b[3] = least = 0.f;
        };
        clear();
        auto put = [&](float2 v, uint32_t dst) {
            uint32_t x[3];
            split3(v, x);
            least = max_abs(least, small_key(v.x), small_key(v.y));
#pragma unroll
            for (int q = 0; q < 3; q++)
                asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (uint32_t)(q * kPlane)), "r"(x[q]) : "memory");
        };
        int left = p.nk, t = 0;    // stages left of the tile being taken apart, and which of this CTA's tiles it is
        // Half a stage: the loads of the half two ahead follow the use of their registers, eight at a time (interleaved with their
        // uses one by one, loads share the few scoreboards with later ones and every use waits for nearly all of them).
        auto half = [&](float2 (&va)[8], float2 (&vb)[8], uint32_t s) {
#pragma unroll
            for (int i = 0; i < 8; i++)
            {
                mag_a[i] = max_abs(mag_a[i], va[i].x, va[i].y);
                put(va[i], dst_a + s + (uint32_t)(i * 1024));
            }
            load_a(va);
#pragma unroll
            for (int i = 0; i < 8; i++)
            {
                mag_b[2 * (i & 1)]     = fmaxf(mag_b[2 * (i & 1)], fabsf(vb[i].x));
                mag_b[2 * (i & 1) + 1] = fmaxf(mag_b[2 * (i & 1) + 1], fabsf(vb[i].y));
                put(vb[i], dst_b + s + (uint32_t)((i & 1) * (kPlane / 2) + (i >> 1) * 1024));
            }
            load_b(vb);
            next_half();
        };
        float2 a0[8], b0[8], a1[8], b1[8];
        auto stage = [&](int c) {
            // the MMAs that read this stage's planes before
            if (c >= kStages)
                ok = ok && ptx::mbar_wait_bounded(ptx::smem_u32(&bar_acc[(c - kStages) % kAccs]), (uint32_t)((c - kStages) / kAccs) & 1u, p.wait_limit);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok)
                return;
            const uint32_t s = (uint32_t)(c % kStages * kStageBytes);
            half(a0, b0, s);
            half(a1, b1, s + kHalfBytes);
            if (--left == 0)
            {
                // the tile's magnitudes, before its last stage is handed over
                float* const mg = mags + (t & 1) * kMagWords;
#pragma unroll
                for (int i = 0; i < 8; i++)
                {
                    float m = mag_a[i];
#pragma unroll
                    for (int o = 8; o > 0; o >>= 1)
                        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
                    if ((lane & 15) == 0)
                        mg[2 * (w + 8 * i) + odd] = m;
                }
                // (columns 2 lane, 2 lane + 1 of the even and of the odd units)
                float* const mc = mg + kTile + w * kTile + 2 * lane;
                mc[0] = mag_b[0]; mc[1] = mag_b[1]; mc[64] = mag_b[2]; mc[65] = mag_b[3];
                // (non-negative floats order like their bits)
                const uint32_t key = __reduce_max_sync(0xffffffffu, __float_as_uint(least));
                if (lane == 0)
                    mg[kMinOff + w] = __uint_as_float(key);
                clear();
                left = p.nk;
                t++;
            }
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0)
                ptx::mbar_arrive(ptx::smem_u32(&bar_full[c % kStages]));
        };
        start_tile();
        load_a(a0);
        load_b(b0);
        next_half();
        load_a(a1);
        load_b(b1);
        next_half();
        for (int c = 0; c < total && ok; c++)
            stage(c);
    }
    if (!ok)
        atomicOr(p.status, TB200_DEV_TIMEOUT);
    ptx::tc_fence_before_sync();
    const bool all_ok = __syncthreads_and(ok);
    if (warp == kFlushWarps)
    {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem, kTmemCols);
    }
    // Results that the split does not carry, by all warps and after the pipeline: inside it the sums of a tile would have to
    // stay in registers beside those of the block (measured: 9 % of every product), and the other roles would wait as long as
    // K is deep.  Whole blocks are replaced; of more tiles than slots, those of a slot together.
    int turn = 0;
    for (int slot = 0; all_ok && slot < min(mine, kAgainSlots); slot++)
    {
        const uint32_t blocks = again[slot];
        for (int i = slot; blocks != 0 && i < mine; i += kAgainSlots)
        {
            const int tile = (int)blockIdx.x + i * (int)gridDim.x;
            const int batch = tile / per, rem = tile - batch * per, tm = rem / p.tiles_n;
            for (int b = 0; b < 16; b++)
                if (blocks >> b & 1 && turn++ % (kFlushWarps + kSplitWarps) == warp)
                    plain_block<CONV>(p, batch, tm * kTile + (b >> 2) * 32, (rem - tm * p.tiles_n) * kTile + (b & 3) * 32,
                                      reinterpret_cast<float*>(sm) + warp * 32 * kStagePitch);
        }
    }
}

template <bool CONV, bool AVEC, bool BVEC>
tb200_status launch_split(tb200_ctx* ctx, const SplitParams& p)
{
    auto kern = sgemm_split_kernel<CONV, AVEC, BVEC>;
    const tb200_status st = raise_smem_limit(ctx, 52 + (CONV ? 2 : 0) + (AVEC ? 1 : 0), reinterpret_cast<const void*>(kern), kSplitSmem);
    if (st != TB200_OK)
        return st;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim          = dim3((unsigned)std::min(p.tiles, ctx->num_sms));
    cfg.blockDim         = dim3(kSplitThreads);
    cfg.dynamicSmemBytes = kSplitSmem;
    cfg.stream           = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id                                           = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs    = at;
    cfg.numAttrs = ctx->launch_overlap ? 1 : 0;
    timer_begin(ctx);
    cudaLaunchKernelEx(&cfg, kern, p);
    timer_end(ctx);
    return TB200_OK;
}

tb200_status finish_split(tb200_ctx* ctx, SplitParams& p, int batches)
{
    p.tiles_m = (p.M + kTile - 1) / kTile;
    p.tiles_n = (p.N + kTile - 1) / kTile;
    p.tiles   = batches * p.tiles_m * p.tiles_n;
    p.nk      = (p.K + kStageK - 1) / kStageK;
    p.idesc      = ptx::make_idesc(1u, 1u, 1u, 0u, 1u, kTile, kTile);
    p.a_desc_hi  = ptx::make_smem_desc_hi(16, 512, 4u);
    p.b_desc_hi  = ptx::make_smem_desc_hi(kPlane / 2, 1024, 2u);
    p.wait_limit = ctx->wait_limit_cycles;
    p.status     = ctx->d_status;
    return TB200_OK;
}

// Shallow products stay with the FFMA kernel: its chains are short enough there to err no more than a stage's cut-off does
// (1.4e-7 at K = 64), and the tables of magnitudes rely on tiles of at least four stages.
constexpr int kMinSplitK = 256;

}    // namespace

// Estimated SM cycles of the split kernel, 0 where it does not serve.
// A stage measured 3 700 cycles, 4 500 with unaligned pairs, 4 500 - 5 600 where A is gathered (16x28x28x256 3x3 256
// channels: 181 us, 82 TFLOP/s; 32x28x28x64 3x3 128 channels: 58 us, where FFMA takes 71).
double sgemm_split_cost(const tb200_ctx* ctx, int64_t batches, int64_t M, int64_t N, int64_t K, bool conv)
{
    const int64_t tiles = batches * ((M + kTile - 1) / kTile) * ((N + kTile - 1) / kTile);
    if (K < kMinSplitK || tiles >= (1LL << 30) || (ctx->max_smem_optin > 0 && ctx->max_smem_optin < kSplitSmem + 1024) || ctx->d_status == nullptr)
        return 0.0;
    const double rounds = (double)((tiles + ctx->num_sms - 1) / ctx->num_sms);
    const double stage  = conv ? 6200.0 : (K % 2 || N % 2) ? 4600.0 : 3700.0;
    return rounds * ((double)((K + kStageK - 1) / kStageK) * stage + 1500.0) + 5000.0;
}

tb200_status sgemm_split_launch(tb200_ctx* ctx, const float* a, const float* b, float* out, int N, int H, int C, int W)
{
    SplitParams p;
    memset(&p, 0, sizeof(p));
    p.a = a; p.b = b; p.out = out;
    p.M = H; p.N = W; p.K = C; p.ldb = W;
    p.a_batch = (int64_t)H * C; p.b_batch = (int64_t)C * W; p.o_batch = (int64_t)H * W;
    finish_split(ctx, p, N);
    const bool vec = (W % 2) == 0 && (C % 2) == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 7) == 0;
    const tb200_status st = vec ? launch_split<false, true, true>(ctx, p) : launch_split<false, false, false>(ctx, p);
    return st != TB200_OK ? st : post_launch(ctx, "sgemm_f32");
}

tb200_status conv_f32_split_launch(tb200_ctx* ctx, const ConvF32Problem& q)
{
    SplitParams p;
    memset(&p, 0, sizeof(p));
    p.a = q.in; p.b = q.wt; p.out = q.out;
    p.M = q.N * q.OH * q.OW; p.N = q.OC; p.K = q.KH * q.KW * q.IC; p.ldb = conv_f32_ldb(q.OC);
    p.IH = q.IH; p.IW = q.IW; p.IC = q.IC; p.OH = q.OH; p.OW = q.OW; p.KW = q.KW;
    p.pad_t = q.pad_t; p.pad_l = q.pad_l; p.sy = q.sy; p.sx = q.sx; p.dy = q.dy; p.dx = q.dx;
    p.in_sn = (int)q.in_sn; p.in_sh = (int)q.in_sh; p.in_sw = (int)q.in_sw;
    p.bias = q.bias; p.bias_n = q.bias_n;
    p.has_clamp = q.has_clamp; p.clamp_lo = q.clamp_lo; p.clamp_hi = q.clamp_hi;
    finish_split(ctx, p, 1);
    const bool vec = (q.IC % 2) == 0 && ((q.in_sn | q.in_sh | q.in_sw) & 1) == 0 && (reinterpret_cast<uintptr_t>(q.in) & 7) == 0;
    const tb200_status st = vec ? launch_split<true, true, true>(ctx, p) : launch_split<true, false, true>(ctx, p);
    return st != TB200_OK ? st : post_launch(ctx, "conv_f32");
}

}    // namespace tb200
