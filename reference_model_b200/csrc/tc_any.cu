// Tensor-core GEMM for the shapes the TMA kernels do not take or take badly: channel runs, rows and columns of any length
// and alignment, and problems with so few output tiles that most of the chip would idle.
//
// One CTA computes one 128 x block_n tile of the output (or a share of its K range).  What differs from tc_gemm.cu is how
// the rows get into shared memory: eight warps gather them (CONV2D: pixel windows tap by tap, straight from the NHWC input;
// MATMUL: rows of A) in 16-byte pieces and write them in the swizzled layout the tensor core reads, so that
//   * the channel run of a tap needs no alignment: pieces are copied asynchronously where a run is a multiple of 16, 8 or 4
//     bytes and assembled from aligned words otherwise; a run is padded to whole pieces in K only (the weights hold zeros
//     there), never in memory;
//   * rows are consecutive output pixels whatever the image width: no tile is cut at the end of an image row, and a tile
//     that holds all channels of its pixels is one contiguous piece of the output;
//   * a tap outside the image is a piece filled with the input zero point, so that every pixel has the interior's
//     correction and the epilogue knows no borders.
// The other operand arrives by TMA (weights, K-major; B of a MATMUL with 16-byte rows, MN-major) or is gathered the same way
// (B with rows of any length).  Zero-point sums of an int8 MATMUL cost no pass over memory: a tile of ones in shared memory
// is multiplied with B (column sums, in every lane) and with A (row sums, in every column) beside the product itself.
// Problems with few tiles split K over the CTAs of a cluster; the partial accumulators are added in rank order through
// distributed shared memory.
// fp16 96 x 197 x 64 x 197: 22.4 us on the device (one thread per output 68), int8 16x57x57x24 3x3 40 channels 13.8 (136).  What
// bounds them: a block has one to three chunks of K, so set-up, gather and epilogue follow each other (issue slots 43 % busy,
// tensor pipe 2 to 3 %), in 1.3 waves.
// Every wait on a barrier in memory is bounded; one that gives up sets TB200_DEV_TIMEOUT and the CTA drains and frees its
// tensor memory.  The allocation of tensor memory and the meetings of a cluster have no limit of their own: no CTA holds
// columns while it waits for another CTA, so both end once the CTAs that run do.
#include <algorithm>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>
#include <cuda_runtime.h>

#include "common.h"
#include "ptx_sm100.cuh"
#include "rescale_math.cuh"

namespace tb200
{
namespace
{

constexpr int kRows       = 128;
constexpr int kLoaders    = 256;    // warps 0..7: gather, later the epilogue
constexpr int kThreads    = 320;    // warp 8: TMA of B, warp 9: tensor memory and MMA issue
constexpr int kMaxStages  = 4;
constexpr int kABytes     = kRows * 128;
constexpr int kOnesCols   = 32;     // accumulator columns of the row sums

struct AnyParams
{
    CUtensorMap tmB;
    const uint8_t* a;
    const uint8_t* b;       // B gathered by the loaders (b_mode 2)
    uint8_t* out;
    int es, run_bytes;      // element size of A and B; bytes of one tap's channel run
    int M, N;               // rows and columns of one batch
    uint32_t fd_ow[2], fd_oh[2];    // division by OW, OH (fastdiv_make)
    int64_t a_batch, o_batch, b_batch;    // elements between batches
    // gather of A: row m is the window of output pixel m (MATMUL: one tap, "pixel" stride = row stride)
    int conv, IH, IW, OH, OW, KH, KW, pad_t, pad_l, sy, sx, dy, dx;
    int in_sn, in_sh, in_sw;              // elements
    int skip_nan;           // float CONV2D with padding: see sum_inside()
    int b_fmt;              // element type for sum_inside(): 0 fp16, 1 bf16, 2 E4M3, 3 E5M2
    uint32_t fill4;         // the input zero point in all four bytes
    int pieces_per_tap, pieces;           // 16-byte pieces of a run; of the whole K
    int chunks, chunks_per_split;         // 128-byte chunks of K; of one CTA of a cluster
    int b_mode;             // 0: TMA, K-major; 1: TMA, MN-major; 2: gathered, MN-major
    int bK;                 // rows of B (b_mode 1, 2), elements
    int block_n, tiles_m, tiles_n, splits;
    int stages, stage_bytes, b_box_bytes, b_nbox;
    int ones_off, part_off, stage_out_off, rec_off;    // shared-memory offsets behind the 1024-byte aligned base
    int tmem_cols, csum_col, rsum_col;                 // accumulator columns of the sums (-1: not needed)
    int halves;             // ANY_SUM32: accumulators per chunk, 1 or 2
    uint32_t idesc, idesc_rsum;
    uint64_t a_desc_hi, b_desc_hi;
    int b_kstep16, kind;    // 0 i8, 1 f16, 2 f8f6f4
    int32_t a_zp, b_zp, zp_const;
    // epilogue
    const int32_t* corr;    // [N padded] int32 added to every column, or null
    const int32_t* rec;     // lean RESCALE records, or null: multipliers / shifts below
    const int* rec_ok;      // whether every record is usable, as the kernel that built them left it
    const int32_t* mult;
    const int8_t* shift;
    const float* bias_f;
    int out_es, out_bf16, direct;
    int double_round, out_zp, clamp_lo, clamp_hi, has_clamp;
    float clamp_lo_f, clamp_hi_f;
    long long wait_limit;
    int* status;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void st_shared_v4(uint32_t dst, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// `nb` bytes (1..16, or nothing when it is not positive) of a 16-byte piece, fetched into words; finish_piece() puts them
// in place.  ALIGN: what the address and the run length are multiples of (8, 4, or 0 for nothing: aligned words that hold
// at least one of the bytes, shifted into place).
template <int ALIGN>
struct Piece
{
    uint32_t w[ALIGN == 0 ? 5 : 4];
    __device__ __forceinline__ void fetch(const uint8_t* src, int nb)
    {
        if (ALIGN == 8)
        {
            uint2 a = make_uint2(0, 0), b = make_uint2(0, 0);
            if (nb > 0)
                a = *reinterpret_cast<const uint2*>(src);
            if (nb > 8)
                b = *reinterpret_cast<const uint2*>(src + 8);
            w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
        }
        else if (ALIGN == 4)
        {
#pragma unroll
            for (int i = 0; i < 4; i++)
                w[i] = nb > 4 * i ? *reinterpret_cast<const uint32_t*>(src + 4 * i) : 0u;
        }
        else
        {
            const int sh          = (int)(reinterpret_cast<uintptr_t>(src) & 3);
            const uint32_t* words = reinterpret_cast<const uint32_t*>(src - sh);
            const int last        = nb > 0 ? sh + nb : 0;
#pragma unroll
            for (int i = 0; i < 5; i++)
                w[i] = 4 * i < last ? words[i] : 0u;
        }
    }
    __device__ __forceinline__ void finish(uint32_t dst, const uint8_t* src, int nb)
    {
        if (ALIGN != 0)
        {
            st_shared_v4(dst, w[0], w[1], w[2], w[3]);
            return;
        }
        const int sh = 8 * (int)(reinterpret_cast<uintptr_t>(src) & 3);
        uint32_t o[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            o[i]           = __funnelshift_r(w[i], w[i + (ALIGN == 0 ? 1 : 0)], sh);
            const int left = nb - 4 * i;
            if (left < 4)
                o[i] = left <= 0 ? 0u : o[i] & ((1u << (8 * left)) - 1u);
        }
        st_shared_v4(dst, o[0], o[1], o[2], o[3]);
    }
};

__device__ __forceinline__ float element(const uint8_t* base, int64_t i, int fmt)
{
    switch (fmt)
    {
        case 0: return __half2float(reinterpret_cast<const __half*>(base)[i]);
        case 1: return __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(base)[i]);
        case 2: return static_cast<float>(reinterpret_cast<const __nv_fp8_e4m3*>(base)[i]);
        default: return static_cast<float>(reinterpret_cast<const __nv_fp8_e5m2*>(base)[i]);
    }
}

// A tap outside the image is a zero that is multiplied like any other; the reference skips it.  The two differ where a weight
// is infinite or NaN: zero times it is NaN, and only then.  So a NaN of a window that leaves the image is summed again here,
// over the taps inside, in ky, kx, channel order (reference_model/src/ops/tensor_ops.cpp:828-873).
__device__ __noinline__ float sum_inside(const AnyParams& p, int m, int col)
{
    const int q  = (int)fastdiv_apply((uint32_t)m, p.fd_ow), n = (int)fastdiv_apply((uint32_t)q, p.fd_oh);
    const int y0 = (q - n * p.OH) * p.sy - p.pad_t, x0 = (m - q * p.OW) * p.sx - p.pad_l;
    if (y0 >= 0 && x0 >= 0 && y0 + (p.KH - 1) * p.dy < p.IH && x0 + (p.KW - 1) * p.dx < p.IW)
        return __uint_as_float(0x7fffffffu);    // every tap is inside: the NaN stands
    const uint8_t* const w = p.b + (int64_t)col * p.pieces * 16;
    float sum = 0.f;
    for (int ky = 0; ky < p.KH; ky++)
        for (int kx = 0; kx < p.KW; kx++)
        {
            const int y = y0 + ky * p.dy, x = x0 + kx * p.dx;
            if ((unsigned)y >= (unsigned)p.IH || (unsigned)x >= (unsigned)p.IW)
                continue;
            const int64_t at = (int64_t)n * p.in_sn + (int64_t)y * p.in_sh + (int64_t)x * p.in_sw;
            const uint8_t* const wt = w + (int64_t)(ky * p.KW + kx) * p.pieces_per_tap * 16;
            for (int c = 0; c < p.run_bytes / p.es; c++)
                sum = fmaf(element(p.a, at + c, p.b_fmt), element(wt, c, p.b_fmt), sum);
        }
    return sum;
}

// The NaNs among sixteen neighbouring columns of one row, `mask`, by sum_inside().
__device__ __noinline__ void mend_nans(const AnyParams& p, int m, int col, uint32_t mask, uint32_t* v)
{
    for (; mask; mask &= mask - 1)
    {
        const int at = __ffs((int)mask) - 1;
        v[at]        = __float_as_uint(sum_inside(p, m, col + at));
    }
}

// Sixteen neighbouring columns of one row: corrections, RESCALE or bias, CLAMP, packing.  w: the packed output bytes.
enum : int
{
    ANY_I32     = 0,
    ANY_RESCALE = 1,
    ANY_FLOAT   = 2,
    ANY_SUM32   = 3,    // floating-point operands, fp32 output
    ANY_CONV    = 4,    // ANY_FLOAT of a CONV2D: NaNs of windows that leave the image are looked at (MATMUL would pay 3 % for it)
};

template <int EPI>
__device__ __forceinline__ void epilogue16(const AnyParams& p, int col, const uint32_t (&v)[16], const int32_t (*rec)[8],
                                           uint32_t (&w)[16], bool& bad)
{
    if (EPI == ANY_I32)
    {
#pragma unroll
        for (int i = 0; i < 16; i++)
            w[i] = v[i] + (p.corr ? (uint32_t)__ldg(p.corr + col + i) : 0u);
    }
    else if (EPI == ANY_RESCALE)
    {
        if (rec != nullptr)
        {
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                int32_t z[4];
#pragma unroll
                for (int j = 0; j < 4; j++)
                {
                    const int4 r0 = *reinterpret_cast<const int4*>(&rec[4 * q + j][0]);
                    const int2 r1 = *reinterpret_cast<const int2*>(&rec[4 * q + j][4]);
                    z[j] = rescale_rec_apply((int32_t)v[4 * q + j], r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, p.double_round != 0);
                }
                asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w[q]) : "r"(z[3]), "r"(z[2]), "r"(0));
                asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w[q]) : "r"(z[1]), "r"(z[0]), "r"(w[q]));
                if (p.clamp_lo > -128 || p.clamp_hi < 127)
                    w[q] = __vmins4(__vmaxs4(w[q], (uint32_t)(p.clamp_lo & 0xff) * 0x01010101u), (uint32_t)(p.clamp_hi & 0xff) * 0x01010101u);
            }
            return;
        }
        // any multiplier, shift and output type: apply_scale_32 with its REQUIRE checks
#pragma unroll
        for (int i = 0; i < 16; i++)
        {
            int32_t z = 0;
            if (col + i < p.N)
            {
                const int32_t acc = (int32_t)(v[i] + (uint32_t)__ldg(p.corr + col + i));
                z = apply_scale_32_dev(acc, __ldg(p.mult + col + i), (int32_t)__ldg(p.shift + col + i), p.double_round != 0, bad);
                const int64_t zz = (int64_t)z + p.out_zp;
                bad |= zz > 2147483647LL || zz < -2147483648LL;
                z = (int32_t)(zz < p.clamp_lo ? p.clamp_lo : zz > p.clamp_hi ? p.clamp_hi : zz);
            }
            w[i] = (uint32_t)z;
        }
        if (p.out_es == 1)
#pragma unroll
            for (int q = 0; q < 4; q++)
                w[q] = (w[4 * q] & 0xffu) | ((w[4 * q + 1] & 0xffu) << 8) | ((w[4 * q + 2] & 0xffu) << 16) | (w[4 * q + 3] << 24);
        else if (p.out_es == 2)
#pragma unroll
            for (int q = 0; q < 8; q++)
                w[q] = (w[2 * q] & 0xffffu) | (w[2 * q + 1] << 16);
    }
    else
    {
        float f[16];
#pragma unroll
        for (int i = 0; i < 16; i++)
            f[i] = __uint_as_float(v[i]);
        if (p.bias_f)
        {
#pragma unroll
            for (int q = 0; q < 4; q++)
            {
                const float4 b = __ldg(reinterpret_cast<const float4*>(p.bias_f + col) + q);
                f[4 * q] += b.x; f[4 * q + 1] += b.y; f[4 * q + 2] += b.z; f[4 * q + 3] += b.w;
            }
        }
        if (p.has_clamp)
        {
#pragma unroll
            for (int i = 0; i < 16; i++)
            {
                f[i] = (f[i] < p.clamp_lo_f) ? p.clamp_lo_f : f[i];
                f[i] = (f[i] > p.clamp_hi_f) ? p.clamp_hi_f : f[i];
            }
        }
        if (p.out_es == 4)
        {
#pragma unroll
            for (int i = 0; i < 16; i++)
                w[i] = __float_as_uint(f[i]);
        }
        else if (p.out_bf16)
        {
#pragma unroll
            for (int q = 0; q < 8; q++)
            {
                const __nv_bfloat162 h = __floats2bfloat162_rn(f[2 * q], f[2 * q + 1]);
                w[q] = *reinterpret_cast<const uint32_t*>(&h);
            }
        }
        else
        {
#pragma unroll
            for (int q = 0; q < 8; q++)
            {
                const __half2 h = __floats2half2_rn(f[2 * q], f[2 * q + 1]);
                w[q] = *reinterpret_cast<const uint32_t*>(&h);
            }
        }
    }
}

// Sixteen finished columns of one row, to global memory in 16-byte pieces (whole rows are multiples of 16 bytes then), or
// to the staging tile, element by element.
__device__ __forceinline__ void put16(const AnyParams& p, uint8_t* dst, int ncols, const uint32_t (&w)[16])
{
    // (static indices only: the sixteen words stay in registers)
#pragma unroll
    for (int q = 0; q < 4; q++)
        if (q < p.out_es && (q * 16) < ncols * p.out_es)
            *reinterpret_cast<uint4*>(dst + q * 16) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
}

// (any element-aligned address: whole words where they lie inside the sixteen columns, single elements at the two ends)
template <int EPI>
__device__ __forceinline__ void stage16(const AnyParams& p, uint8_t* dst, int ncols, const uint32_t (&w)[16])
{
    if (p.out_es == 4)
    {
        uint32_t* const o = reinterpret_cast<uint32_t*>(dst);
#pragma unroll
        for (int i = 0; i < 16; i++)
            if (i < ncols)
                o[i] = w[i];
    }
    else if (EPI != ANY_I32 && p.out_es == 2)
    {
        const bool odd    = (reinterpret_cast<uintptr_t>(dst) & 2) != 0;
        uint32_t* const o = reinterpret_cast<uint32_t*>(dst + (odd ? 2 : 0));
        if (odd)
            *reinterpret_cast<uint16_t*>(dst) = (uint16_t)w[0];
#pragma unroll
        for (int q = 0; q < 8; q++)
        {
            // columns 2q, 2q + 1 (2q + 1, 2q + 2 where the address is odd)
            const uint32_t v = odd ? __funnelshift_r(w[q], w[q + 1], 16) : w[q];
            const int c      = odd ? 2 * q + 1 : 2 * q;
            if (c + 1 < ncols)
                o[q] = v;
            else if (c < ncols)
                *reinterpret_cast<uint16_t*>(o + q) = (uint16_t)v;
        }
    }
    else if (EPI == ANY_RESCALE)
    {
        const int sh   = (int)(reinterpret_cast<uintptr_t>(dst) & 3);
        const int head = sh ? min(ncols, 4 - sh) : 0;
#pragma unroll
        for (int b = 0; b < 3; b++)
            if (b < head)
                dst[b] = (uint8_t)(w[0] >> (8 * b));
        uint32_t* const o = reinterpret_cast<uint32_t*>(dst + head);
        const int left    = ncols - head;
#pragma unroll
        for (int q = 0; q < 4; q++)
        {
            const uint32_t v = __funnelshift_r(w[q], q < 3 ? w[q + 1] : 0u, 8 * head);
            if (4 * q + 4 <= left)
                o[q] = v;
            else if (4 * q < left)
            {
#pragma unroll
                for (int b = 0; b < 3; b++)
                    if (4 * q + b < left)
                        reinterpret_cast<uint8_t*>(o + q)[b] = (uint8_t)(v >> (8 * b));
            }
        }
    }
}

// ANY_SUM32.  The tensor core cuts its running sum off at every step instead of rounding it, which a 16-bit result hides and
// an fp32 result shows: with operands of one sign the sum of K = 4001 was 2.6e-6 off where rounded multiply-adds are 9e-7 off.
// So no sum is carried there for more than one 128-byte chunk of K (64 or 128 elements): each stage has its own accumulator,
// started from zero, and the gathering warps read a finished chunk back and add it to fp32 registers (64 of them at 128
// columns: one CTA per SM) while later chunks are in flight.  Sums of up to two chunks of 16-bit operands, which rounded
// multiply-adds do not get far wrong either, have an accumulator for each half of a chunk (K = 65: 1.6e-7 with one).
template <int EPI, int ALIGN>
__global__ void __launch_bounds__(kThreads, EPI == ANY_SUM32 ? 1 : 2) tc_any_kernel(const __grid_constant__ AnyParams p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kMaxStages], bar_empty[kMaxStages], bar_acc;
    __shared__ uint32_t tmem_base_holder;
    __shared__ int abort_flag;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* const sm   = smem_raw + (base - ptx::smem_u32(smem_raw));

    const int rank  = p.splits > 1 ? (int)ptx::cluster_ctarank() : 0;
    const int tile  = (int)(blockIdx.x / (unsigned)p.splits);
    const int per   = p.tiles_m * p.tiles_n;
    const int batch = tile / per;
    const int rem   = tile - batch * per;
    const int tm    = rem / p.tiles_n;
    const int m0 = tm * kRows, n0 = (rem - tm * p.tiles_n) * p.block_n;
    const int rows  = min(kRows, p.M - m0);
    const int c_lo  = rank * p.chunks_per_split;
    const int nk    = max(0, min(p.chunks, c_lo + p.chunks_per_split) - c_lo);    // 128-byte chunks of K this CTA takes (at least one)

    if (tid == 0)
    {
        for (int s = 0; s < p.stages; s++)
        {
            ptx::mbar_init(ptx::smem_u32(&bar_full[s]), kLoaders + (p.b_mode != 2 ? 1 : 0));
            ptx::mbar_init(ptx::smem_u32(&bar_empty[s]), 1);
        }
        ptx::mbar_init(ptx::smem_u32(&bar_acc), 1);
        abort_flag = 0;
        ptx::fence_barrier_init();
        if (p.b_mode != 2)
            ptx::prefetch_tmap(&p.tmB);
    }
    if (warp == 9)
    {
        ptx::tmem_alloc(ptx::smem_u32(&tmem_base_holder), (uint32_t)p.tmem_cols);
        ptx::tmem_relinquish();
    }
    // (set-up of the gathering warps, while tensor memory is being allocated)
    const int j = tid & 7, r0 = (tid & 255) >> 3;    // piece of a row's 128 bytes; rows r0, r0 + 32, r0 + 64, r0 + 96
    int off[4], oy_[4], ox_[4];
    if (warp < 8)
    {
#pragma unroll
        for (int i = 0; i < 4; i++)
        {
            const int m = m0 + r0 + 32 * i;
            oy_[i] = ox_[i] = 0;
            if (p.conv)
            {
                const int q  = (int)fastdiv_apply((uint32_t)m, p.fd_ow), ox = m - q * p.OW;
                const int n  = (int)fastdiv_apply((uint32_t)q, p.fd_oh), oy = q - n * p.OH;
                oy_[i] = oy * p.sy - p.pad_t;
                ox_[i] = ox * p.sx - p.pad_l;
                off[i] = n * p.in_sn + oy_[i] * p.in_sh + ox_[i] * p.in_sw;
            }
            else
                off[i] = m * p.in_sw;
        }
        if (EPI == ANY_I32 && (p.csum_col >= 0 || p.rsum_col >= 0))
            for (int e = tid; e < kABytes / 16; e += kLoaders)
                st_shared_v4(base + (uint32_t)(p.ones_off + e * 16), 0x01010101u, 0x01010101u, 0x01010101u, 0x01010101u);
        if (EPI == ANY_RESCALE && p.rec != nullptr)
        {
            const uint8_t* const src = reinterpret_cast<const uint8_t*>(p.rec + (int64_t)n0 * 8);
            for (int e = tid; e < p.block_n * 2; e += kLoaders)
                cp_async16(base + (uint32_t)(p.rec_off + e * 16), src + e * 16);
        }
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem = tmem_base_holder;
    // (after the tensor memory is held: a successor's CTA on this SM then waits for this one, never the other way round)
    if (tid == 0)
        ptx::dep_launch_trigger();

    bool ok = true, lean = false;
    constexpr int kSumGroups = EPI == ANY_SUM32 ? 4 : 1;    // sixteen columns each, of up to 128
    float acc[kSumGroups * 16];
#pragma unroll
    for (int i = 0; i < kSumGroups * 16; i++)
        acc[i] = 0.f;
    if (warp < 8)
    {
        // ------------------------------------------------------------------ gather
        const uint32_t a_dst   = (uint32_t)(r0 * 128 + ((j ^ (r0 & 7)) << 4));
        const uint8_t* const a = p.a + (int64_t)batch * p.a_batch * p.es;
        const int esl          = p.es - 1;             // log2 of the element size
        ptx::dep_launch_wait();
        // The verdict is read here and not by the host: no first call waits for it, and a captured graph follows constants that
        // are replaced under it.
        if (EPI == ANY_RESCALE && p.rec != nullptr)
            lean = *p.rec_ok != 0;

        int pk = c_lo * 8 + j;                         // this thread's piece of K, its tap and place in the tap's run
        int cp = pk, kx = 0, ky = 0;
        if (pk >= p.pieces_per_tap)
        {
            const int tap = pk / p.pieces_per_tap;
            cp -= tap * p.pieces_per_tap;
            ky = tap / p.KW;
            kx = tap - ky * p.KW;
        }
        int stage = 0;
        uint32_t phase = 0;
        // the running chunk's source: offset inside the window, how many bytes of the piece exist
        auto here = [&](int& toff, int& nb, int& y, int& x) {
            const int c0 = cp << 4;
            y    = ky * p.dy;
            x    = kx * p.dx;
            toff = y * p.in_sh + x * p.in_sw + (c0 >> esl);
            nb   = pk < p.pieces ? min(16, p.run_bytes - c0) : 0;
        };
        auto inside = [&](int q, int y, int x) {
            return !p.conv || ((unsigned)(oy_[q] + y) < (unsigned)p.IH && (unsigned)(ox_[q] + x) < (unsigned)p.IW);
        };
        auto advance = [&]() {
            pk += 8;
            cp += 8;
            while (cp >= p.pieces_per_tap)
            {
                cp -= p.pieces_per_tap;
                if (++kx == p.KW)
                {
                    kx = 0;
                    ky++;
                }
            }
        };
        auto hand_over = [&](int s) {
            ptx::fence_proxy_async_smem();
            ptx::mbar_arrive(ptx::smem_u32(&bar_full[s]));
        };
        auto gather_b = [&](int i) {
            // B of a MATMUL with rows of any length: four pieces in flight per thread
            const uint32_t sB  = base + (uint32_t)(stage * p.stage_bytes + kABytes);
            const int krows    = 128 >> esl;
            const int pw_log   = 31 - __clz((p.block_n * p.es) >> 4);    // pieces of a row, a power of two
            const uint8_t* bb  = p.b + (int64_t)batch * p.b_batch * p.es;
            const int total    = krows << pw_log;
            for (int e0 = tid; e0 < total; e0 += 4 * kLoaders)
            {
                Piece<0> pc[4];
                const uint8_t* src[4];
                int nb[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                {
                    const int e  = e0 + u * kLoaders;
                    const int k  = (c_lo + i) * krows + (e >> pw_log), n = n0 + ((e & ((1 << pw_log) - 1)) << (4 - esl));
                    nb[u]  = e < total && k < p.bK && n < p.N ? min(16, (p.N - n) << esl) : 0;
                    src[u] = bb + (((int64_t)k * p.N + n) << esl);
                    pc[u].fetch(src[u], nb[u]);
                }
#pragma unroll
                for (int u = 0; u < 4; u++)
                {
                    const int e = e0 + u * kLoaders, k = e >> pw_log, c = e & ((1 << pw_log) - 1);
                    if (e < total)
                        pc[u].finish(sB + (uint32_t)((c >> 3) * p.b_box_bytes + k * 128 + (((c & 7) ^ (k & 7)) << 4)), src[u], nb[u]);
                }
            }
        };
        auto wait_empty = [&]() {
            const bool got = ptx::mbar_wait_bounded(ptx::smem_u32(&bar_empty[stage]), phase ^ 1u, p.wait_limit);
            return EPI == ANY_SUM32 ? (bool)__all_sync(0xffffffffu, got) : got;    // (what follows there is done by whole warps)
        };
        // ANY_SUM32: the next chunk's sums into the registers.  Its accumulator is written again `stages` chunks later, which
        // this thread hands over only after it has been here.
        int summed = 0, sum_stage = 0;
        uint32_t sum_phase = 0;
        auto sum_chunk = [&]() {
            ok = __all_sync(0xffffffffu, ok && ptx::mbar_wait_bounded(ptx::smem_u32(&bar_empty[sum_stage]), sum_phase, p.wait_limit));
            if (!ok)
                return;
            ptx::tc_fence_after_sync();
            const uint32_t t = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(sum_stage * p.halves * p.block_n + (warp >> 2) * 16);
            // (a second half that got no MMA was not written)
            const int halves = p.halves == 2 && p.pieces - (c_lo + summed) * 8 > 4 ? 2 : 1;
            for (int h = 0; h < halves; h++)
#pragma unroll
                for (int g = 0; g < kSumGroups; g++)
                    if (g * 32 < p.block_n)
                    {
                        uint32_t v[16];
                        ptx::tmem_ld_32x32b_x16(t + (uint32_t)(h * p.block_n + g * 32), v);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            acc[g * 16 + i] += __uint_as_float(v[i]);
                    }
            ptx::tc_fence_before_sync();
            summed++;
            if (++sum_stage == p.stages)
            {
                sum_stage = 0;
                sum_phase ^= 1u;
            }
        };
        if (ALIGN == 16)
        {
            // asynchronous copies; a stage is handed over once this thread's copies into it have landed: two stages
            // behind the one being filled
            int done = 0, done_stage = 0;
            for (int i = 0; i < nk && ok; i++)
            {
                if (!wait_empty())
                {
                    ok = false;
                    break;
                }
                int toff, nb, y, x;
                here(toff, nb, y, x);
                const uint32_t sA = base + (uint32_t)(stage * p.stage_bytes) + a_dst;
#pragma unroll
                for (int q = 0; q < 4; q++)
                {
                    if (r0 + 32 * q >= rows)
                        break;
                    const uint32_t dst = sA + (uint32_t)(q * 32 * 128);
                    if (nb > 0 && inside(q, y, x))
                        cp_async16(dst, a + ((int64_t)(off[q] + toff) << esl));
                    else
                    {
                        const uint32_t f = nb > 0 ? p.fill4 : 0u;
                        st_shared_v4(dst, f, f, f, f);
                    }
                }
                advance();
                if (p.b_mode == 2)
                    gather_b(i);
                asm volatile("cp.async.commit_group;" ::: "memory");
                if (++stage == p.stages)
                {
                    stage = 0;
                    phase ^= 1u;
                }
                if (i >= 2)
                {
                    asm volatile("cp.async.wait_group 2;" ::: "memory");
                    hand_over(done_stage);
                    done++;
                    done_stage = done_stage + 1 == p.stages ? 0 : done_stage + 1;
                }
                if (EPI == ANY_SUM32 && i >= 3)
                    sum_chunk();
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            for (; ok && done < nk; done++)
            {
                hand_over(done_stage);
                done_stage = done_stage + 1 == p.stages ? 0 : done_stage + 1;
            }
        }
        else
        {
            // through registers: the next chunk's loads are issued as soon as this one's pieces are stored (a second set of
            // registers for them spilled and measured slower)
            constexpr int AL = ALIGN == 16 ? 8 : ALIGN;
            struct Chunk
            {
                Piece<AL> piece[4];
                const uint8_t* src[4];
                int nb[4];    // bytes of the piece; -1: outside the image
            };
            auto fetch = [&](Chunk& c) {
                int toff, nb, y, x;
                here(toff, nb, y, x);
#pragma unroll
                for (int q = 0; q < 4; q++)
                {
                    if (r0 + 32 * q >= rows)
                        break;    // rows past the last pixel keep whatever the stage holds: their results are not stored
                    c.nb[q]  = nb > 0 && !inside(q, y, x) ? -1 : nb;
                    c.src[q] = a + ((int64_t)(off[q] + toff) << esl);
                    c.piece[q].fetch(c.src[q], c.nb[q]);
                }
                advance();
            };
            Chunk cur;
            fetch(cur);
            for (int i = 0; i < nk && ok; i++)
            {
                if (!wait_empty())
                {
                    ok = false;
                    break;
                }
                if (p.b_mode == 2)
                    gather_b(i);
                const uint32_t sA = base + (uint32_t)(stage * p.stage_bytes) + a_dst;
#pragma unroll
                for (int q = 0; q < 4; q++)
                {
                    if (r0 + 32 * q >= rows)
                        break;
                    const uint32_t dst = sA + (uint32_t)(q * 32 * 128);
                    if (cur.nb[q] < 0)
                        st_shared_v4(dst, p.fill4, p.fill4, p.fill4, p.fill4);
                    else
                        cur.piece[q].finish(dst, cur.src[q], cur.nb[q]);
                }
                hand_over(stage);
                if (i + 1 < nk)
                    fetch(cur);
                if (++stage == p.stages)
                {
                    stage = 0;
                    phase ^= 1u;
                }
                if (EPI == ANY_SUM32 && i >= 2)
                    sum_chunk();
            }
        }
        if (EPI == ANY_SUM32)
            while (ok && summed < nk)
                sum_chunk();
        if (EPI == ANY_RESCALE)
        {
            // the records have landed for every gathering warp
            asm volatile("cp.async.wait_all;" ::: "memory");
            asm volatile("bar.sync 1, 256;" ::: "memory");
        }
        ok = ok && ptx::mbar_wait_bounded(ptx::smem_u32(&bar_acc), 0u, p.wait_limit);
        ptx::tc_fence_after_sync();
    }
    else if (warp == 8)
    {
        // ------------------------------------------------------------------ B by TMA
        if (lane == 0 && p.b_mode != 2)
        {
            if (p.b_mode == 1)
                ptx::dep_launch_wait();    // B of a MATMUL may be the predecessor's output; weights are constants
            const uint32_t bytes = (uint32_t)(p.stage_bytes - kABytes);
            const int elems      = 128 / p.es;
            int stage = 0;
            uint32_t phase = 0;
            for (int i = 0; i < nk; i++)
            {
                if (!ptx::mbar_wait_bounded(ptx::smem_u32(&bar_empty[stage]), phase ^ 1u, p.wait_limit))
                {
                    ok = false;
                    break;
                }
                const uint32_t full = ptx::smem_u32(&bar_full[stage]);
                const uint32_t sB   = base + (uint32_t)(stage * p.stage_bytes + kABytes);
                ptx::mbar_arrive_expect_tx(full, bytes);
                const int k = (c_lo + i) * elems;
                if (p.b_mode == 0)
                    ptx::tma_load_3d(sB, &p.tmB, full, k, n0, 0);
                else
                    for (int bx = 0; bx < p.b_nbox; bx++)
                        ptx::tma_load_3d(sB + (uint32_t)(bx * p.b_box_bytes), &p.tmB, full, n0 + bx * elems, k, batch);
                if (++stage == p.stages)
                {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
    }
    else
    {
        // ------------------------------------------------------------------ MMA issue
        if (lane == 0)
        {
            int stage = 0;
            uint32_t phase = 0, accum = 0;
            const uint64_t ones_a = ptx::smem_desc(p.a_desc_hi, base + (uint32_t)p.ones_off);
            for (int i = 0; i < nk; i++)
            {
                if (!ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[stage]), phase, p.wait_limit))
                {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint32_t sA = base + (uint32_t)(stage * p.stage_bytes);
                uint64_t ad = ptx::smem_desc(p.a_desc_hi, sA), bd = ptx::smem_desc(p.b_desc_hi, sA + kABytes);
                uint32_t d = tmem + (EPI == ANY_SUM32 ? (uint32_t)(stage * p.halves * p.block_n) : 0u);
                if (EPI == ANY_SUM32)
                    accum = 0;
                const int mmas = min(4, (p.pieces - (c_lo + i) * 8 + 1) >> 1);    // 32 bytes of K each
                for (int m = 0; m < mmas; m++, ad += 2, bd += (uint64_t)p.b_kstep16)
                {
                    if (EPI == ANY_SUM32 && m == 2 && p.halves == 2)
                    {
                        d += (uint32_t)p.block_n;
                        accum = 0;
                    }
                    if (EPI < ANY_FLOAT)
                    {
                        ptx::mma_i8_ss(tmem, ad, bd, p.idesc, accum);
                        if (p.csum_col >= 0)
                            ptx::mma_i8_ss(tmem + (uint32_t)p.csum_col, ones_a, bd, p.idesc, accum);
                        if (p.rsum_col >= 0)
                            ptx::mma_i8_ss(tmem + (uint32_t)p.rsum_col, ad, ones_a, p.idesc_rsum, accum);
                    }
                    else if (p.kind == 2)
                        ptx::mma_f8_ss(d, ad, bd, p.idesc, accum);
                    else
                        ptx::mma_f16_ss(d, ad, bd, p.idesc, accum);
                    accum = 1;
                }
                ptx::mma_commit(ptx::smem_u32(&bar_empty[stage]));
                if (++stage == p.stages)
                {
                    stage = 0;
                    phase ^= 1u;
                }
            }
            ptx::mma_commit(ptx::smem_u32(&bar_acc));    // (also after a wait gave up: whoever waits for the MMAs issued so far gets through)
        }
    }
    if (!ok)
    {
        atomicOr(p.status, TB200_DEV_TIMEOUT);
        atomicExch(&abort_flag, 1);
    }

    // ---------------------------------------------------------------------- epilogue (the gathering warps)
    const int32_t(*const rec)[8] = lean ? reinterpret_cast<const int32_t(*)[8]>(sm + p.rec_off) : nullptr;
    const int groups = p.block_n >> 4;    // sixteen columns each
    const int row_a  = p.splits > 1 ? rank * (kRows / p.splits) : 0;    // rows of the tile this CTA finishes
    const int row_b  = min(rows, p.splits > 1 ? row_a + kRows / p.splits : kRows);
    const int ncols  = min(p.block_n, p.N - n0);
    uint8_t* const g0 = p.out + ((int64_t)batch * p.o_batch + (int64_t)(m0 + row_a) * p.N + n0) * p.out_es;
    // staged output: laid out as in memory, at the same offset inside 16 bytes
    uint8_t* const s0 = sm + p.stage_out_off + (p.tiles_n == 1 ? (reinterpret_cast<uintptr_t>(g0) & 15) : 0);
    const int s_pitch = p.tiles_n == 1 ? ncols * p.out_es : (ncols * p.out_es + 7) & ~3;
    bool bad = false;
    auto finish = [&](int row, int c, uint32_t (&v)[16]) {
        if (EPI == ANY_CONV && p.skip_nan)
        {
            uint32_t nans = 0;
#pragma unroll
            for (int i = 0; i < 16; i++)
                nans |= (v[i] & 0x7fffffffu) > 0x7f800000u && c * 16 + i < ncols ? 1u << i : 0u;
            if (nans)
            {
                uint32_t t[16];
#pragma unroll
                for (int i = 0; i < 16; i++)
                    t[i] = v[i];
                mend_nans(p, m0 + row, n0 + c * 16, nans, t);
#pragma unroll
                for (int i = 0; i < 16; i++)
                    v[i] = t[i];
            }
        }
        uint32_t w[16];
        epilogue16<EPI>(p, n0 + c * 16, v, rec ? rec + c * 16 : nullptr, w, bad);
        const int left = min(16, ncols - c * 16);
        if (p.direct)
            put16(p, g0 + ((int64_t)(row - row_a) * p.N + c * 16) * p.out_es, left, w);
        else
            stage16<EPI>(p, s0 + (row - row_a) * s_pitch + c * 16 * p.out_es +
                           (p.tiles_n == 1 ? 0 : (int)(reinterpret_cast<uintptr_t>(g0 + (int64_t)(row - row_a) * p.N * p.out_es) & 3)), left, w);
    };
    if (warp < 8)
    {
        ok = __all_sync(0xffffffffu, ok);
        const int quarter = warp & 3;
        const int row     = quarter * 32 + lane;
        const uint32_t t0 = tmem + ((uint32_t)(quarter * 32) << 16);
        uint32_t* const part = reinterpret_cast<uint32_t*>(sm + p.part_off) + row * (p.block_n + 4);
        if (ok)
        {
            uint32_t rterm = 0;
            if (EPI == ANY_I32 && p.rsum_col >= 0)
            {
                uint32_t v[16];
                ptx::tmem_ld_32x32b_x16(t0 + (uint32_t)p.rsum_col, v);
                ptx::tmem_ld_wait();
                rterm = (uint32_t)p.b_zp * v[0];
            }
            if (EPI == ANY_I32 && rank == 0)
                rterm -= (uint32_t)p.zp_const;
            auto emit = [&](int c, uint32_t (&v)[16]) {
                if (p.splits > 1)
                {
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        *reinterpret_cast<uint4*>(part + c * 16 + 4 * q) = make_uint4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
                else if (row < rows)
                    finish(row, c, v);
            };
            if (EPI == ANY_SUM32)
            {
#pragma unroll
                for (int g = 0; g < kSumGroups; g++)
                {
                    const int c = (warp >> 2) + 2 * g;
                    uint32_t v[16];
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        v[i] = __float_as_uint(acc[g * 16 + i]);
                    if (c < groups && c * 16 < ncols)
                        emit(c, v);
                }
            }
            for (int c = warp >> 2; EPI != ANY_SUM32 && c < groups && c * 16 < ncols; c += 2)
            {
                uint32_t v[16];
                ptx::tmem_ld_32x32b_x16(t0 + (uint32_t)(c * 16), v);
                ptx::tmem_ld_wait();
                if (EPI == ANY_I32)
                {
                    if (p.csum_col >= 0)
                    {
                        uint32_t cs[16];
                        ptx::tmem_ld_32x32b_x16(t0 + (uint32_t)(p.csum_col + c * 16), cs);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i++)
                            v[i] -= (uint32_t)p.a_zp * cs[i];
                    }
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        v[i] -= rterm;
                }
                emit(c, v);
            }
        }
    }
    auto release = [&]() {
        ptx::tc_fence_before_sync();
        __syncthreads();
        if (tid == 0 && abort_flag)
        {
            // a role gave up: let copies in flight land and MMAs already issued retire before memory is released
            if (p.b_mode != 2)
                for (int s = 0; s < p.stages; s++)
                {
                    ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[s]), 0u, 2000000LL);
                    ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[s]), 1u, 2000000LL);
                }
            ptx::mbar_wait_bounded(ptx::smem_u32(&bar_acc), 0u, 40000000LL);
        }
        __syncthreads();
        if (warp == 9)
        {
            ptx::tc_fence_after_sync();
            ptx::tmem_dealloc(tmem, (uint32_t)p.tmem_cols);
        }
    };
    if (p.splits > 1)
    {
        // Tensor memory goes back before this CTA waits for its peers.  Its allocation is the one wait of the kernel without a
        // limit, and another launch's CTAs may hold columns of the same SM: two clusters that each held the columns the
        // other's CTA waits for would wait for ever.  This way whoever holds columns gives them back without waiting for a CTA
        // that may still be asking for some.
        release();
        __syncwarp();
        ptx::cluster_sync();    // every CTA's partial tile is in its shared memory
        if (warp < 8 && ok)
        {
            const int live = (ncols + 15) >> 4;
            for (int e = tid; e < (row_b - row_a) * live; e += kLoaders)
            {
                const int r = e / live, c = e - r * live, row = row_a + r;
                const uint32_t at = ptx::smem_u32(sm + p.part_off) + (uint32_t)((row * (p.block_n + 4) + c * 16) * 4);
                uint32_t v[16];
#pragma unroll
                for (int i = 0; i < 16; i++)
                    v[i] = 0;
                for (int s = 0; s < p.splits; s++)
                {
                    const uint32_t src = ptx::map_to_cta(at, (uint32_t)s);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                    {
                        uint32_t x0, x1, x2, x3;
                        asm volatile("ld.shared::cluster.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x0), "=r"(x1), "=r"(x2), "=r"(x3) : "r"(src + 16 * q) : "memory");
                        if (EPI >= ANY_FLOAT)
                        {
                            v[4 * q + 0] = __float_as_uint(__uint_as_float(v[4 * q + 0]) + __uint_as_float(x0));
                            v[4 * q + 1] = __float_as_uint(__uint_as_float(v[4 * q + 1]) + __uint_as_float(x1));
                            v[4 * q + 2] = __float_as_uint(__uint_as_float(v[4 * q + 2]) + __uint_as_float(x2));
                            v[4 * q + 3] = __float_as_uint(__uint_as_float(v[4 * q + 3]) + __uint_as_float(x3));
                        }
                        else
                        {
                            v[4 * q + 0] += x0;
                            v[4 * q + 1] += x1;
                            v[4 * q + 2] += x2;
                            v[4 * q + 3] += x3;
                        }
                    }
                }
                finish(row, c, v);
            }
        }
    }
    if (!p.direct && warp < 8)
    {
        asm volatile("bar.sync 1, 256;" ::: "memory");
        const int nrows = max(0, row_b - row_a);
        if (ok && p.tiles_n == 1)
        {
            const int total = nrows * s_pitch;
            const int head  = min(total, (int)((16 - (reinterpret_cast<uintptr_t>(g0) & 15)) & 15));
            const int body  = (total - head) >> 4, tail = total - head - 16 * body;
            if (tid < head)
                g0[tid] = s0[tid];
            for (int e = tid; e < body; e += kLoaders)
                *reinterpret_cast<uint4*>(g0 + head + 16 * e) = *reinterpret_cast<const uint4*>(s0 + head + 16 * e);
            if (tid < tail)
                g0[total - tail + tid] = s0[total - tail + tid];
        }
        else if (ok)
        {
            // a row at a time, in words that are aligned in both places (the staged row sits at the row's offset inside a
            // word), elements at its ends
            for (int r = warp; r < nrows; r += 8)
            {
                uint8_t* const g       = g0 + (int64_t)r * p.N * p.out_es;
                const uint8_t* const s = s0 + r * s_pitch + (int)(reinterpret_cast<uintptr_t>(g) & 3);
                const int total = ncols * p.out_es;
                const int head  = min(total, (int)((4 - (reinterpret_cast<uintptr_t>(g) & 3)) & 3));
                const int body  = (total - head) >> 2, tail = total - head - 4 * body;
                if (lane < head)
                    g[lane] = s[lane];
#pragma unroll 2
                for (int e = lane; e < body; e += 32)
                    *reinterpret_cast<uint32_t*>(g + head + 4 * e) = *reinterpret_cast<const uint32_t*>(s + head + 4 * e);
                if (lane < tail)
                    g[total - tail + lane] = s[total - tail + lane];
            }
        }
    }
    if (bad)
        atomicOr(p.status, TB200_DEV_UNPREDICTABLE);

    // ---------------------------------------------------------------------- teardown
    __syncwarp();
    if (p.splits > 1)
        ptx::cluster_sync();    // nobody leaves while another CTA may still read its shared memory
    else
        release();
}

struct AnyPlan
{
    AnyParams k;
    int align;    // of A's channel runs: 16, 8, 4 bytes, 0 = less
    int smem_bytes;
    int64_t ctas;
    bool sum32;    // ANY_SUM32
};

int64_t any_align(int64_t a, int64_t b)
{
    while (b)
    {
        const int64_t t = a % b;
        a = b;
        b = t;
    }
    return a;
}

// Lays a problem out for one tile width and one split of K; false when it does not fit.
bool any_layout(const TcProblem& q, int max_smem, int block_n, int splits, AnyPlan* plan)
{
    AnyParams& k = plan->k;
    memset(&k, 0, sizeof(k));
    const bool matmul = q.b_mn_major != 0;
    k.es        = (int)dtype_size(q.in_dtype);
    k.conv      = matmul ? 0 : 1;
    k.run_bytes = q.IC * k.es;
    const int64_t rows = matmul ? (int64_t)q.OW : (int64_t)q.N * q.OH * q.OW;
    if (rows > 0x7fffffff - 2 * kRows)
        return false;    // row numbers, past the end of the last tile too, are 32 bits
    k.M         = (int)rows;
    k.N         = q.OC;
    const int64_t sw = matmul || !q.a_stride_w ? q.IC : q.a_stride_w, sh = matmul ? 0 : q.a_stride_h ? q.a_stride_h : sw * q.IW,
                  sn = matmul ? 0 : q.a_stride_n ? q.a_stride_n : sh * q.IH;
    if ((matmul ? sw * q.OW : sn * q.N) >= (1LL << 31))
        return false;    // offsets inside the input are 32 bits
    k.in_sw = (int)sw; k.in_sh = (int)sh; k.in_sn = (int)sn;
    k.IH = q.IH; k.IW = q.IW; k.OH = matmul ? 1 : q.OH; k.OW = matmul ? 1 : q.OW; k.KH = q.KH; k.KW = q.KW;
    fastdiv_make((uint32_t)k.OW, k.fd_ow);
    fastdiv_make((uint32_t)k.OH, k.fd_oh);
    k.pad_t = q.pad_t; k.pad_l = q.pad_l; k.sy = q.stride_y; k.sx = q.stride_x; k.dy = q.dil_y; k.dx = q.dil_x;
    k.a_batch = (int64_t)q.OW * q.IC; k.b_batch = (int64_t)q.IC * q.OC; k.o_batch = (int64_t)q.OW * q.OC;
    if (!matmul)
        k.a_batch = k.b_batch = k.o_batch = 0;
    k.pieces_per_tap = (k.run_bytes + 15) / 16;
    const int64_t pieces = (int64_t)q.KH * q.KW * k.pieces_per_tap;
    if (pieces <= 0 || pieces >= (1 << 26) || k.M <= 0 || k.N <= 0)
        return false;
    k.pieces = (int)pieces;
    k.chunks = (k.pieces + 7) / 8;
    const int64_t al = any_align(any_align(16, k.run_bytes), any_align(any_align(sw * k.es, sh * k.es), sn * k.es));
    plan->align = al >= 4 ? (int)al : 0;
    k.b_mode = !matmul ? 0 : ((int64_t)k.N * k.es) % 16 == 0 && (reinterpret_cast<uintptr_t>(q.b) & 15) == 0 ? 1 : 2;
    k.bK     = q.IC;
    if (k.b_mode != 0 && (block_n * k.es) % 128 != 0)
        return false;
    k.block_n = block_n;
    k.tiles_m = (k.M + kRows - 1) / kRows;
    k.tiles_n = (k.N + block_n - 1) / block_n;
    k.splits  = splits;
    k.chunks_per_split = (k.chunks + splits - 1) / splits;
    if (k.chunks_per_split * (splits - 1) >= k.chunks)
        return false;    // every CTA of a cluster has work
    k.stages      = std::min(k.chunks_per_split, kMaxStages);
    k.stage_bytes = kABytes + block_n * 128;
    k.b_box_bytes = k.b_mode ? 128 / k.es * 128 : 0;
    k.b_nbox      = k.b_mode ? block_n * k.es / 128 : 1;
    k.out_es      = (int)dtype_size(q.out_dtype);
    k.direct      = ((int64_t)k.N * k.out_es) % 16 == 0 && (reinterpret_cast<uintptr_t>(q.out) & 15) == 0;
    k.a_zp = q.a_zp; k.b_zp = q.b_zp;
    k.csum_col = k.rsum_col = -1;
    plan->sum32 = q.epi == TC_EPI_FLOAT && q.out_dtype == TB200_FP32;
    if (plan->sum32 && block_n > 128)
        return false;
    k.halves   = plan->sum32 && k.chunks <= 2 && k.es == 2 ? 2 : 1;
    int cols   = plan->sum32 ? k.stages * k.halves * block_n : block_n;
    if (matmul && q.in_dtype == TB200_INT8)
    {
        if (q.a_zp != 0)
        {
            k.csum_col = cols;
            cols += block_n;
        }
        if (q.b_zp != 0)
        {
            k.rsum_col = cols;
            cols += kOnesCols;
        }
        k.zp_const = (int32_t)((uint32_t)q.IC * (uint32_t)(q.a_zp * q.b_zp));
    }
    if (cols > 512)
        return false;
    k.tmem_cols = 32;
    while (k.tmem_cols < cols)
        k.tmem_cols *= 2;
    const int part    = splits > 1 ? kRows * (block_n + 4) * 4 : 0;
    const int staging = k.direct ? 0 : kRows / splits * (std::min(block_n, k.N) * k.out_es + 8) + 32;
    k.part_off      = 0;
    k.stage_out_off = part;
    int at          = (std::max(k.stages * k.stage_bytes, part + staging) + 1023) & ~1023;
    k.ones_off      = at;
    if (k.csum_col >= 0 || k.rsum_col >= 0)
        at += kABytes;
    k.rec_off        = at;
    at += q.epi == TC_EPI_RESCALE && q.rec ? block_n * 32 : 0;
    plan->smem_bytes = at + 1024;
    plan->ctas       = 0;
    // tensor memory of co-resident CTAs of one launch must fit together: one that waits for columns would idle its SM's share
    const int per_sm = std::min(3, (max_smem + 1024) / (plan->smem_bytes + 1024));
    if (per_sm * k.tmem_cols > 512)
        plan->smem_bytes = std::max(plan->smem_bytes, max_smem / 2 + 1024);
    return plan->smem_bytes <= max_smem;
}

// Tile width and split of K with the smallest estimated time.
bool any_choose(const TcProblem& q, int num_sms, int max_smem, AnyPlan* best)
{
    const int batches = q.b_mn_major ? q.OH : 1;
    double best_cost  = 0;
    for (int bn = 32; bn <= 256; bn *= 2)
        for (int s = 1; s <= 8; s *= 2)
        {
            AnyPlan plan;
            if ((bn > 32 && bn / 2 >= q.OC && best_cost > 0) || !any_layout(q, max_smem, bn, s, &plan))
                continue;
            const AnyParams& k = plan.k;
            const int64_t ctas = (int64_t)batches * k.tiles_m * k.tiles_n * s;
            if (ctas >= (1LL << 31))
                continue;
            const int per_sm     = plan.sum32 ? 1 : std::max(1, std::min(2, (max_smem + 1024) / (plan.smem_bytes + 1024)));
            const double rounds  = (double)((ctas + (int64_t)num_sms * per_sm - 1) / ((int64_t)num_sms * per_sm));
            const double stage_c = 500.0 + 2.0 * bn;
            const double cost    = rounds * (3000.0 + k.chunks_per_split * stage_c + bn * 20.0 / s + (s > 1 ? 2000.0 + 8.0 * bn : 0.0));
            if (best_cost == 0 || cost < best_cost)
            {
                best_cost  = cost;
                *best      = plan;
                best->ctas = ctas;
            }
        }
    return best_cost > 0;
}

}    // namespace

bool tc_any_supported(const tb200_ctx* ctx, const TcProblem& q)
{
    if (!(q.in_dtype == TB200_INT8 || q.in_dtype == TB200_FP16 || q.in_dtype == TB200_BF16 || dtype_is_fp8(q.in_dtype)))
        return false;
    if (q.xpar || q.out_sy || q.tile_end || (reinterpret_cast<uintptr_t>(q.out) & 3))
        return false;
    // (one layout that fits is enough: the launch then has one to choose)
    const int max_smem = ctx->max_smem_optin > 0 ? ctx->max_smem_optin - 1024 /* static */ : 200 * 1024;
    for (int bn = 32; bn <= 256; bn *= 2)
    {
        AnyPlan plan;
        if (any_layout(q, max_smem, bn, 1, &plan) && (int64_t)(q.b_mn_major ? q.OH : 1) * plan.k.tiles_m * plan.k.tiles_n < (1LL << 31))
            return true;
    }
    return false;
}

tb200_status tc_any_launch(tb200_ctx* ctx, const TcProblem& q)
{
    AnyPlan plan;
    const int max_smem = ctx->max_smem_optin > 0 ? ctx->max_smem_optin - 1024 /* static */ : 200 * 1024;
    if (!any_choose(q, ctx->num_sms, max_smem, &plan))
        return fail(ctx, TB200_ERROR, "shape does not fit the gathering tensor-core kernel");
    AnyParams& k      = plan.k;
    const bool matmul = q.b_mn_major != 0;
    k.a   = reinterpret_cast<const uint8_t*>(q.a);
    k.b   = reinterpret_cast<const uint8_t*>(q.b);
    k.out = reinterpret_cast<uint8_t*>(q.out);
    k.fill4 = (uint32_t)(q.a_fill & 0xff) * 0x01010101u;
    k.skip_nan = !matmul && q.epi == TC_EPI_FLOAT && q.padded;
    k.b_fmt    = q.in_dtype == TB200_FP16 ? 0 : q.in_dtype == TB200_BF16 ? 1 : q.in_dtype == TB200_FP8E4M3 ? 2 : 3;
    const bool is_f8 = dtype_is_fp8(q.in_dtype), is_i8 = q.in_dtype == TB200_INT8;
    k.kind = is_i8 ? 0 : is_f8 ? 2 : 1;
    uint32_t cf = is_i8 ? 2u : 1u, af, bf;
    if (is_f8)
    {
        af = q.in_dtype == TB200_FP8E5M2 ? 1u : 0u;
        bf = (q.b_fp8_dtype ? (tb200_dtype)q.b_fp8_dtype : q.in_dtype) == TB200_FP8E5M2 ? 1u : 0u;
    }
    else
        af = bf = is_i8 ? 1u : q.in_dtype == TB200_BF16 ? 1u : 0u;
    k.idesc      = ptx::make_idesc(cf, af, bf, 0u, matmul ? 1u : 0u, kRows, (uint32_t)k.block_n);
    k.idesc_rsum = ptx::make_idesc(cf, af, bf, 0u, 0u, kRows, kOnesCols);
    k.a_desc_hi  = ptx::make_smem_desc_hi(16, 1024, 2u);
    k.b_desc_hi  = matmul ? ptx::make_smem_desc_hi(k.b_box_bytes, 1024, 2u) : k.a_desc_hi;
    k.b_kstep16  = matmul ? (32 / k.es) * 128 / 16 : 2;
    if (k.b_mode != 2)
    {
        auto enc = reinterpret_cast<CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                                 const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill)>(tensor_map_encode_fn());
        if (!enc)
            return fail(ctx, TB200_INTERNAL, "cuTensorMapEncodeTiled is not available from the driver");
        const CUtensorMapDataType dt = is_i8 || is_f8 ? CU_TENSOR_MAP_DATA_TYPE_UINT8
                                       : q.in_dtype == TB200_FP16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
        const cuuint64_t kel = (cuuint64_t)k.pieces * 16 / k.es;
        const cuuint64_t d0[3] = { kel, (cuuint64_t)k.N, 1 }, d1[3] = { (cuuint64_t)k.N, (cuuint64_t)q.IC, (cuuint64_t)q.OH };
        const cuuint64_t s0[2] = { kel * k.es, kel * k.es * k.N }, s1[2] = { (cuuint64_t)k.N * k.es, (cuuint64_t)k.N * k.es * q.IC };
        const cuuint32_t b0[3] = { (cuuint32_t)(128 / k.es), (cuuint32_t)k.block_n, 1 }, b1[3] = { (cuuint32_t)(128 / k.es), (cuuint32_t)(128 / k.es), 1 };
        const cuuint32_t one[3] = { 1, 1, 1 };
        const CUresult r = enc(&k.tmB, dt, 3, const_cast<void*>(q.b), matmul ? d1 : d0, matmul ? s1 : s0, matmul ? b1 : b0, one,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
            return fail(ctx, TB200_INTERNAL, "tensor map for B rejected (CUresult %d)", (int)r);
    }
    if (!matmul && q.corr)
    {
        // every tap is in scope (the gather fills the border): the interior's correction row
        const int interior = q.corr_classes ? (q.KH * (q.KW + 1)) * (q.KW + 1) + q.KW : 0;
        k.corr = q.corr + (int64_t)interior * q.corr_stride;
    }
    k.rec    = q.epi == TC_EPI_RESCALE && q.out_dtype == TB200_INT8 ? q.rec : nullptr;
    k.rec_ok = q.rec_ok;
    k.mult   = q.mult_pad;
    k.shift  = q.shift_pad;
    k.bias_f = q.bias_f_pad;
    k.out_bf16     = q.out_dtype == TB200_BF16;
    k.double_round = q.double_round;
    k.out_zp       = q.out_zp;
    k.clamp_lo = q.clamp_lo; k.clamp_hi = q.clamp_hi; k.has_clamp = q.has_clamp;
    k.clamp_lo_f = q.clamp_lo_f; k.clamp_hi_f = q.clamp_hi_f;
    k.wait_limit = ctx->wait_limit_cycles;
    k.status     = ctx->d_status;
    const int al = plan.align == 16 ? 0 : plan.align == 8 ? 1 : plan.align == 4 ? 2 : 3;
    const int variant = plan.sum32 ? ANY_SUM32 : q.epi == TC_EPI_FLOAT && !matmul ? ANY_CONV : q.epi;
    static void (*const kernels[5][4])(const AnyParams) = {
        { tc_any_kernel<ANY_I32, 16>, tc_any_kernel<ANY_I32, 8>, tc_any_kernel<ANY_I32, 4>, tc_any_kernel<ANY_I32, 0> },
        { tc_any_kernel<ANY_RESCALE, 16>, tc_any_kernel<ANY_RESCALE, 8>, tc_any_kernel<ANY_RESCALE, 4>, tc_any_kernel<ANY_RESCALE, 0> },
        { tc_any_kernel<ANY_FLOAT, 16>, tc_any_kernel<ANY_FLOAT, 8>, tc_any_kernel<ANY_FLOAT, 4>, tc_any_kernel<ANY_FLOAT, 0> },
        { tc_any_kernel<ANY_SUM32, 16>, tc_any_kernel<ANY_SUM32, 8>, tc_any_kernel<ANY_SUM32, 4>, tc_any_kernel<ANY_SUM32, 0> },
        { tc_any_kernel<ANY_CONV, 16>, tc_any_kernel<ANY_CONV, 8>, tc_any_kernel<ANY_CONV, 4>, tc_any_kernel<ANY_CONV, 0> } };
    void (*const kern)(const AnyParams) = kernels[variant][al];
    const tb200_status st = raise_smem_limit(ctx, (variant >= ANY_SUM32 ? 56 - 4 * ANY_SUM32 : 20) + variant * 4 + al, reinterpret_cast<const void*>(kern), plan.smem_bytes);
    if (st != TB200_OK)
        return st;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim          = dim3((unsigned)plan.ctas);
    cfg.blockDim         = dim3(kThreads);
    cfg.dynamicSmemBytes = (size_t)plan.smem_bytes;
    cfg.stream           = ctx->stream;
    cudaLaunchAttribute at[2];
    int na = 0;
    if (ctx->launch_overlap)
    {
        at[na].id                                            = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[na++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (k.splits > 1)
    {
        at[na].id                 = cudaLaunchAttributeClusterDimension;
        at[na].val.clusterDim.x   = (unsigned)k.splits;
        at[na].val.clusterDim.y   = 1;
        at[na++].val.clusterDim.z = 1;
    }
    cfg.attrs    = at;
    cfg.numAttrs = (unsigned)na;
    timer_begin(ctx);
    cudaLaunchKernelEx(&cfg, kern, k);
    timer_end(ctx);
    static const char* const names[] = { "tc_gemm_any_i8_i32", "tc_gemm_any_i8_rescale", "tc_gemm_any_f16", "tc_gemm_any_f8" };
    return post_launch(ctx, names[q.epi == TC_EPI_I32 ? 0 : q.epi == TC_EPI_RESCALE ? 1 : is_f8 ? 3 : 2]);
}

}    // namespace tb200
