// int8 CONV2D + RESCALE (+ CLAMP, + residual join) to int8 on tcgen05 with the CHANNELS on the accumulator's rows.
//
// The product is taken transposed: A = 128 output channels of the weights, B = up to 256 output pixels, so a thread of the
// epilogue owns one channel (its TMEM lane) and walks over pixels (the columns).  What that gives over one pixel per thread
// (tc_conv_lean.cuh):
//   * a channel's RESCALE record is six registers of the thread that owns it.  With a pixel per thread every output read
//     its record from shared memory, and those reads and the scattered 32-byte stores were what the kernel waited for
//     (LSU pipe: 5 wavefronts per 32 outputs);
//   * pixels are columns, and the number of columns is free: 256, 192, 128 or 64 per tile, whichever fills the SMs;
//   * results leave through shared memory, a slot of [pixel][32 channels] per warp, by a tensor store that the warp issues itself.
// The bytes of four pixels are transposed between the four threads of a quad (two shuffles and two byte permutes per four
// outputs) into words of four channels of one pixel.  A residual join works on those words: its other operand's tile
// is loaded into the slot the result will be written to.
//
// Pixels are numbered flat over [N][OH][OW].  A 1x1 stride-1 convolution of a dense tensor reads a plain [pixels][IC] matrix;
// anything else goes through an im2col tensor map: one copy per filter tap brings any run of consecutive output pixels,
// across rows and images, zero outside the image (which is the padding), so no tile works on rows that are cut off.
//
// Roles (576 threads, one CTA per SM): warp 0 lane 0 issues the loads, warp 1 lane 0 the MMAs, warps 2..17 are the
// epilogue: quarter warp % 4 of the TMEM lanes, four groups of four warps, each with a quarter of a tile's pixels.  No warp waits for
// another: each has slots, stores and residual loads of its own (64 to 256 channels on 256x56x56: 98.7 us with a barrier for all
// sixteen, which kept them in step, 86.9 with one per group, 84).  Two accumulators alternate.  Weights stay
// in shared memory when the K extent of a channel block fits beside the ring (the grid is then a multiple of the channel blocks
// and a CTA keeps its block).  Every wait is bounded (p.wait_limit); a wait that gives up sets TB200_DEV_TIMEOUT, the roles
// leave their loops, copies and MMAs in flight are waited for, tensor memory is freed.
#include <algorithm>
#include <cuda.h>
#include <cuda_runtime.h>
#include <mutex>

#include "common.h"
#include "ptx_sm100.cuh"
#include "rescale_math.cuh"

namespace tb200
{

namespace
{

constexpr int kChanThreads   = 576;
constexpr int kChanMaxStages = 8;
constexpr int kChanStaging   = 3;      // most output / residual slots of a warp

struct ChanParams
{
    CUtensorMap tmW, tmX, tmO, tmR;
    int tiles, cbs;                    // tile = pixel block * cbs + channel block
    int px;                            // pixels per tile: 256, 192, 128 or 64
    int pixels, OC;
    int im2col;
    uint32_t fd_ohow[2], fd_ow[2], fd_cbs[2];
    int OH, OW, IH, IW, KH, KW, pad_t, pad_l, stride_y, stride_x, dil_y, dil_x;
    int chunk, chunks_per_tap, total_chunks, ksub, mmas;
    int x_chunk_bytes, w_chunk_bytes, stage_bytes, num_stages, resident;
    int slots;                         // output slots of a warp: 1 or 2, with a join 2 or 3
    int w_off, ring_off;               // from the 1024-byte aligned base; the staging slots come first
    uint64_t desc_hi;
    uint32_t idesc;
    int tmem_cols;
    const int32_t* rec;                // [channels padded to 256][8], rescale_rec_build
    const int32_t* delta;              // [classes][corr_stride] class row minus interior row
    int corr_stride;
    int clamp_lo, clamp_hi;
    const int32_t* join;               // block of kJoinWords words, or null
    int join_lo, join_hi;
    // conv_split_kernel
    int split, chunks_per_cta, red_off, double_round;
    int8_t* out;
    const int8_t* res;
    long long wait_limit;
    int* status;
};

__device__ __forceinline__ uint32_t chan_pack4(int a, int b, int c, int d)
{
    uint32_t hi, r;
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(d), "r"(c), "r"(0));
    asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(b), "r"(a), "r"(hi));
    return r;
}

// One pair of a join through the tabulated legs (indexes: byte ^ 0x80) and the exact arithmetic
__device__ __forceinline__ int32_t chan_join_general_one(const int32_t* blk, int ia, int ib, int32_t m, int32_t sh, int32_t zp, int lo, int hi, bool& bad)
{
    bad = bad || blk[kJoinBadA + ia] != 0 || blk[kJoinBadB + ib] != 0;
    return join_general(blk[kJoinLutA + ia], blk[kJoinLutB + ib], m, sh, blk[kJoinOutDouble] != 0, zp, lo, hi, bad);
}

// A join whose record is not usable (constants uploaded under a captured graph): the pairs of four words through the tabulated
// legs and the exact arithmetic, REQUIRE conditions reported for the words of `real`.  Reads the other operand from the slot and
// stores the results there.
__device__ __noinline__ void chan_join_general(uint32_t dst, uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3, const int32_t* blk, int lo, int hi,
                                               uint32_t real, int* status)
{
    const int32_t m = blk[kJoinOutMult], sh = blk[kJoinOutShift], zp = blk[kJoinOutZp];
    bool any = false;
    for (int q = 0; q < 4; q++)
    {
        const uint32_t qa = q == 0 ? w0 : q == 1 ? w1 : q == 2 ? w2 : w3;
        uint32_t qb, w = 0;
        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(qb) : "r"(dst + (uint32_t)q * 128u));
        bool bad = false;
        for (int j = 0; j < 4; j++)
        {
            const int32_t z = chan_join_general_one(blk, (int)((qa >> (8 * j)) & 0xffu) ^ 0x80, (int)((qb >> (8 * j)) & 0xffu) ^ 0x80, m, sh, zp, lo, hi, bad);
            w |= (uint32_t)(z & 0xff) << (8 * j);
        }
        asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (uint32_t)q * 128u), "r"(w) : "memory");
        any = any || (bad && (real >> q & 1u));
    }
    if (any)
        atomicOr(status, TB200_DEV_UNPREDICTABLE);
}

// One word of the same where nothing is held in registers for it (conv_split_kernel): four results of the convolution with
// the four of the other operand.
__device__ __forceinline__ uint32_t chan_join_word(uint32_t w, uint32_t r, const int32_t* blk, int lo, int hi, int* status)
{
    const int usable = __ldg(blk + kJoinUsable);
    if (usable == 0)
    {
        const int32_t m = blk[kJoinOutMult], sh = blk[kJoinOutShift], zp = blk[kJoinOutZp];
        uint32_t o      = 0;
        bool bad        = false;
        for (int j = 0; j < 4; j++)
        {
            const int32_t z = chan_join_general_one(blk, (int)((w >> (8 * j)) & 0xffu) ^ 0x80, (int)((r >> (8 * j)) & 0xffu) ^ 0x80, m, sh, zp, lo, hi, bad);
            o |= (uint32_t)(z & 0xff) << (8 * j);
        }
        if (bad && status != nullptr)
            atomicOr(status, TB200_DEV_UNPREDICTABLE);
        return o;
    }
    const int4 c0 = __ldg(reinterpret_cast<const int4*>(blk));        // coefficients, constant, m or S, shift or d
    const int2 c1 = __ldg(reinterpret_cast<const int2*>(blk + 4));    // R, or base
    const uint32_t i01 = __byte_perm(w, r, 0x5140), i23 = __byte_perm(w, r, 0x7362);
    int32_t s[4], z[4];
    asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(s[0]) : "r"(c0.x), "r"(i01), "r"(c0.y));
    asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(s[1]) : "r"(c0.x), "r"(i01), "r"(c0.y));
    asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(s[2]) : "r"(c0.x), "r"(i23), "r"(c0.y));
    asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(s[3]) : "r"(c0.x), "r"(i23), "r"(c0.y));
    const bool fix = __ldg(blk + kJoinOutDouble) != 0;
#pragma unroll
    for (int e = 0; e < 4; e++)
    {
        if (usable == 0x01010101)
            z[e] = join_f32_apply(s[e], __int_as_float(c0.z), __int_as_float(c0.w), __int_as_float(c1.x));
        else
        {
            const int64_t P = (int64_t)s[e] * (int64_t)c0.z + (int64_t)(((uint64_t)(uint32_t)c1.y << 32) | (uint32_t)c1.x);
            z[e] = ((int32_t)(P >> 32) + (fix ? s[e] >> 31 : 0)) >> c0.w;
        }
    }
    w = chan_pack4(z[0], z[1], z[2], z[3]);
    if (lo > -128 || hi < 127)
        w = __vmins4(__vmaxs4(w, (uint32_t)(lo & 0xff) * 0x01010101u), (uint32_t)(hi & 0xff) * 0x01010101u);
    return w;
}

// The class of a pixel's clipped window (the rectangle of filter taps inside the image); *border: it is clipped.
__device__ __forceinline__ int chan_border_class(const ChanParams& p, int oy, int ox, bool* border)
{
    const int iy0 = oy * p.stride_y - p.pad_t, ix0 = ox * p.stride_x - p.pad_l;
    *border = iy0 < 0 || ix0 < 0 || iy0 + (p.KH - 1) * p.dil_y >= p.IH || ix0 + (p.KW - 1) * p.dil_x >= p.IW;
    if (!*border)
        return 0;
    int ky_lo = 0, ky_hi = p.KH, kx_lo = 0, kx_hi = p.KW;
    if (iy0 < 0)
        ky_lo = (-iy0 + p.dil_y - 1) / p.dil_y;
    if (ix0 < 0)
        kx_lo = (-ix0 + p.dil_x - 1) / p.dil_x;
    if (iy0 + (p.KH - 1) * p.dil_y >= p.IH)
        ky_hi = iy0 >= p.IH ? 0 : (p.IH - 1 - iy0) / p.dil_y + 1;
    if (ix0 + (p.KW - 1) * p.dil_x >= p.IW)
        kx_hi = ix0 >= p.IW ? 0 : (p.IW - 1 - ix0) / p.dil_x + 1;
    ky_lo = min(ky_lo, p.KH);
    kx_lo = min(kx_lo, p.KW);
    ky_hi = max(ky_hi, ky_lo);
    kx_hi = max(kx_hi, kx_lo);
    return ((ky_lo * (p.KH + 1) + ky_hi) * (p.KW + 1) + kx_lo) * (p.KW + 1) + kx_hi;
}

// CLASSES: padding with a non-zero input zero point, border pixels add what their clipped window leaves out.  FIX: the
// RESCALE has double_round.  JOIN: 0 none, 1 residual join in integers, 2 in single precision.
template <bool CLASSES, bool FIX, int JOIN>
__global__ void __launch_bounds__(kChanThreads, 1) conv_chan_kernel(const __grid_constant__ ChanParams p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kChanMaxStages], bar_empty[kChanMaxStages];
    __shared__ __align__(8) uint64_t bar_acc_full[2], bar_acc_empty[2];
    __shared__ __align__(8) uint64_t bar_res[16 * kChanStaging];
    __shared__ __align__(8) uint64_t bar_w, bar_drain;
    __shared__ uint32_t tmem_base_holder;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t s_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t s_w = s_base + (uint32_t)p.w_off, s_ring = s_base + (uint32_t)p.ring_off;

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < p.num_stages; s++)
        {
            ptx::mbar_init(ptx::smem_u32(&bar_full[s]), 1);
            ptx::mbar_init(ptx::smem_u32(&bar_empty[s]), 1);
        }
        for (int a = 0; a < 2; a++)
        {
            ptx::mbar_init(ptx::smem_u32(&bar_acc_full[a]), 1);
            ptx::mbar_init(ptx::smem_u32(&bar_acc_empty[a]), 16);
        }
        for (int s = 0; s < 16 * kChanStaging; s++)
            ptx::mbar_init(ptx::smem_u32(&bar_res[s]), 1);
        ptx::mbar_init(ptx::smem_u32(&bar_w), 1);
        ptx::mbar_init(ptx::smem_u32(&bar_drain), 1);
        abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::prefetch_tmap(&p.tmW);
        ptx::prefetch_tmap(&p.tmX);
        ptx::prefetch_tmap(&p.tmO);
    }
    if (warp == 1)
    {
        ptx::tmem_alloc(ptx::smem_u32(&tmem_base_holder), (uint32_t)p.tmem_cols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_holder;
    const int my_tiles = (p.tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
    // the successor kernel may be scheduled from here on: its CTAs take an SM as soon as this grid's leave it
    if (threadIdx.x == 0)
        ptx::dep_launch_trigger();

    if (warp == 0)
    {
        // ------------------------------------------------------------------ loads
        if (lane == 0)
        {
            bool ok = true;
            if (p.resident)
            {
                const int cb = (int)blockIdx.x % p.cbs;
                ptx::mbar_arrive_expect_tx(ptx::smem_u32(&bar_w), (uint32_t)(p.total_chunks * 128 * p.chunk));
                for (int ch = 0; ch < p.total_chunks; ch++)
                    ptx::tma_load_3d(s_w + (uint32_t)(ch * p.w_chunk_bytes), &p.tmW, ptx::smem_u32(&bar_w), ch * p.chunk, cb * 128, 0);
            }
            // weights and tables are constants (a kernel that prepares them never lets its successor start early); the
            // activations are the predecessor's output
            ptx::dep_launch_wait();
            int stage      = 0;
            uint32_t phase = 0;
            int tile       = (int)blockIdx.x;
            const uint32_t tx_chunk = (uint32_t)((p.px + (p.resident ? 0 : 128)) * p.chunk);
            for (int i = 0; i < my_tiles && ok; i++, tile += (int)gridDim.x)
            {
                const int pb = (int)fastdiv_apply((uint32_t)tile, p.fd_cbs), cb = tile - pb * p.cbs;
                const int p0 = pb * p.px;
                int n0 = 0, y0 = 0, x0 = 0;
                if (p.im2col)
                {
                    n0           = (int)fastdiv_apply((uint32_t)p0, p.fd_ohow);
                    const int r  = p0 - n0 * (p.OH * p.OW);
                    const int oy = (int)fastdiv_apply((uint32_t)r, p.fd_ow);
                    y0           = oy * p.stride_y - p.pad_t;
                    x0           = (r - oy * p.OW) * p.stride_x - p.pad_l;
                }
                int cc = 0, ky = 0, kx = 0, left = p.total_chunks, ck = 0;
                while (left > 0)
                {
                    if (!ptx::mbar_wait_bounded(ptx::smem_u32(&bar_empty[stage]), phase ^ 1u, p.wait_limit))
                    {
                        ok = false;
                        break;
                    }
                    const int nch = min(p.ksub, left);
                    left -= nch;
                    const uint32_t full = ptx::smem_u32(&bar_full[stage]);
                    uint32_t sx = s_ring + (uint32_t)(stage * p.stage_bytes);
                    uint32_t sw = sx + (uint32_t)(p.ksub * p.x_chunk_bytes);
                    ptx::mbar_arrive_expect_tx(full, (uint32_t)nch * tx_chunk);
                    for (int j = 0; j < nch; j++)
                    {
                        if (p.im2col)
                            ptx::tma_load_im2col_4d(sx, &p.tmX, full, cc * p.chunk, x0, y0, n0, (uint16_t)(kx * p.dil_x), (uint16_t)(ky * p.dil_y));
                        else
                            ptx::tma_load_2d(sx, &p.tmX, full, cc * p.chunk, p0);
                        if (!p.resident)
                            ptx::tma_load_3d(sw, &p.tmW, full, ck, cb * 128, 0);
                        sx += (uint32_t)p.x_chunk_bytes;
                        sw += (uint32_t)p.w_chunk_bytes;
                        ck += p.chunk;
                        if (++cc == p.chunks_per_tap)
                        {
                            cc = 0;
                            if (++kx == p.KW)
                            {
                                kx = 0;
                                ky++;
                            }
                        }
                    }
                    if (++stage == p.num_stages)
                    {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            if (!ok)
            {
                atomicOr(p.status, TB200_DEV_TIMEOUT);
                atomicExch(&abort_flag, 1);
            }
        }
    }
    else if (warp == 1)
    {
        // ------------------------------------------------------------------ MMAs
        if (lane == 0)
        {
            bool ok = true;
            if (p.resident)
            {
                ok = ptx::mbar_wait_bounded(ptx::smem_u32(&bar_w), 0u, p.wait_limit);
                ptx::tc_fence_after_sync();
            }
            int stage      = 0;
            uint32_t phase = 0;
            const uint64_t x16 = (uint64_t)(p.x_chunk_bytes >> 4), w16 = (uint64_t)(p.w_chunk_bytes >> 4);
            for (int i = 0; i < my_tiles && ok; i++)
            {
                if (!ptx::mbar_wait_bounded(ptx::smem_u32(&bar_acc_empty[i & 1]), ((uint32_t)(i >> 1) & 1u) ^ 1u, p.wait_limit))
                {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint32_t d = tmem_base + (uint32_t)((i & 1) * p.px);
                uint32_t accum = 0;
                int left = p.total_chunks, done = 0;
                while (left > 0)
                {
                    if (!ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[stage]), phase, p.wait_limit))
                    {
                        ok = false;
                        break;
                    }
                    ptx::tc_fence_after_sync();
                    const int nch = min(p.ksub, left);
                    left -= nch;
                    const uint32_t sx = s_ring + (uint32_t)(stage * p.stage_bytes);
                    uint64_t bd = ptx::smem_desc(p.desc_hi, sx);
                    uint64_t ad = p.resident ? ptx::smem_desc(p.desc_hi, s_w + (uint32_t)(done * p.w_chunk_bytes))
                                             : ptx::smem_desc(p.desc_hi, sx + (uint32_t)(p.ksub * p.x_chunk_bytes));
                    for (int j = 0; j < nch; j++)
                    {
                        ptx::mma_i8_ss_chunk(d, ad, bd, p.idesc, accum, p.mmas);
                        accum = 1;
                        ad += w16;
                        bd += x16;
                    }
                    done += nch;
                    ptx::mma_commit(ptx::smem_u32(&bar_empty[stage]));
                    if (++stage == p.num_stages)
                    {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (!ok)
                    break;
                ptx::mma_commit(ptx::smem_u32(&bar_acc_full[i & 1]));
            }
            if (!ok)
            {
                atomicOr(p.status, TB200_DEV_TIMEOUT);
                atomicExch(&abort_flag, 1);
            }
        }
    }
    else
    {
        // ------------------------------------------------------------------ epilogue
        const int quarter = warp & 3, group = (warp - 2) >> 2;
        const int cols    = p.px >> 2;             // columns of a tile that this warp's group takes
        const int t       = lane & 3;
        const uint32_t sel1 = t < 2 ? 0x5410u : 0x3276u;
        const uint32_t sel2 = (t & 1) ? 0x3715u : 0x6240u;
        const int ew      = warp - 2;
        const bool boss   = lane == 0;    // issues its warp's stores and residual loads
        const bool narrow = p.clamp_lo > -128 || p.clamp_hi < 127;
        const uint32_t lo4 = (uint32_t)(p.clamp_lo & 0xff) * 0x01010101u, hi4 = (uint32_t)(p.clamp_hi & 0xff) * 0x01010101u;
        const uint32_t jlo4 = (uint32_t)(p.join_lo & 0xff) * 0x01010101u, jhi4 = (uint32_t)(p.join_hi & 0xff) * 0x01010101u;
        const bool jnarrow  = p.join_lo > -128 || p.join_hi < 127;
        const int nslots  = p.slots;
        const uint32_t slot_bytes = (uint32_t)cols * 32u;
        const uint32_t s_mine     = s_base + (uint32_t)(ew * nslots) * slot_bytes;    // this warp's slots: [column][32 channels]
        // word q of sixteen columns holds columns 4 q .. 4 q + 3; after the transposition this thread has four channels of
        // column 4 q + t, and a warp's word is 128 contiguous bytes of the slot
        const uint32_t off = (uint32_t)(t * 32 + (lane >> 2) * 4);
        int32_t rm = 0, rpk = 0, rcpk = 0, rsh = 0, rlo = 0, rhi = 0;
        uint32_t jcoef = 0;
        int32_t jc = 0, jm = 0, jsh = 0, jrlo = 0, jrhi = 0;
        bool jusable = true;
        if (JOIN)
        {
            jcoef = (uint32_t)p.join[kJoinCoef];
            jc    = p.join[kJoinC];
            jm    = p.join[kJoinM];
            jsh   = p.join[kJoinSh];
            jrlo  = p.join[kJoinRlo];
            jrhi  = p.join[kJoinRhi];
            // (the coefficients of the two forms differ)
            jusable = JOIN == 2 ? p.join[kJoinUsable] == 0x01010101 : p.join[kJoinUsable] == 1;
        }
        const int32_t jfix = JOIN && p.join[kJoinOutDouble] ? -1 : 0;
        int cur_cb = -1;
        bool ok    = true;
        int tile   = (int)blockIdx.x;
        if (boss)
        {
            ptx::dep_launch_wait();
            if (JOIN)
                for (int i = 0; i < nslots - 1 && i < my_tiles; i++)
                {
                    const int rt = tile + i * (int)gridDim.x;
                    const int pb = (int)fastdiv_apply((uint32_t)rt, p.fd_cbs), cb = rt - pb * p.cbs;
                    const uint32_t bar = ptx::smem_u32(&bar_res[ew * kChanStaging + i]);
                    ptx::mbar_arrive_expect_tx(bar, slot_bytes);
                    ptx::tma_load_2d(s_mine + (uint32_t)i * slot_bytes, &p.tmR, bar, cb * 128 + quarter * 32, pb * p.px + group * cols);
                }
        }
        int slot = 0;
        uint32_t slot_phase = 0;
        for (int i = 0; i < my_tiles; i++, tile += (int)gridDim.x)
        {
            const int pb = (int)fastdiv_apply((uint32_t)tile, p.fd_cbs), cb = tile - pb * p.cbs;
            const int ch = cb * 128 + quarter * 32 + lane;
            if (cb != cur_cb)
            {
                const int4 r0 = __ldg(reinterpret_cast<const int4*>(p.rec + (int64_t)ch * 8));
                const int2 r1 = __ldg(reinterpret_cast<const int2*>(p.rec + (int64_t)ch * 8 + 4));
                rm = r0.x; rpk = r0.y; rcpk = r0.z; rsh = r0.w; rlo = r1.x; rhi = r1.y;
                cur_cb = cb;
            }
            // classes of this warp's columns, two per lane at most; bits of `border` are columns whose window is clipped
            int cls[2]         = { 0, 0 };
            uint32_t border[2] = { 0, 0 };
            if (CLASSES)
            {
#pragma unroll
                for (int k = 0; k < 2; k++)
                {
                    const int pix = pb * p.px + group * cols + k * 32 + lane;
                    const int n   = (int)fastdiv_apply((uint32_t)pix, p.fd_ohow);
                    const int r   = pix - n * (p.OH * p.OW);
                    const int oy  = (int)fastdiv_apply((uint32_t)r, p.fd_ow);
                    bool b;
                    cls[k] = chan_border_class(p, oy, r - oy * p.OW, &b);
                    border[k] = __ballot_sync(0xffffffffu, b);
                }
            }
            const uint32_t s_slot = s_mine + (uint32_t)slot * slot_bytes;
            ok = ptx::mbar_wait_bounded(ptx::smem_u32(&bar_acc_full[i & 1]), (uint32_t)(i >> 1) & 1u, p.wait_limit);
            if (JOIN && ok)
                ok = ptx::mbar_wait_bounded(ptx::smem_u32(&bar_res[ew * kChanStaging + slot]), slot_phase, p.wait_limit);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok)
                break;
            if (!JOIN && nslots == 1)
            {
                // one slot: the store of the tile before has had this tile's MMAs to read it
                if (boss)
                    ptx::bulk_wait_read();
                __syncwarp();
            }
            {
                ptx::tc_fence_after_sync();
                const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((i & 1) * p.px + group * cols);
                // sixteen columns: RESCALE, transpose, join, store into the slot
                auto work = [&](uint32_t(&v)[16], int c0) {
                    if (CLASSES)
                    {
                        const uint32_t bm = (c0 & 32 ? border[1] : border[0]) >> (c0 & 16) & 0xffffu;
                        if (bm != 0)
                        {
                            const int my = c0 & 32 ? cls[1] : cls[0];
                            int32_t d[16];
#pragma unroll
                            for (int j = 0; j < 16; j++)
                            {
                                const int cj = __shfl_sync(0xffffffffu, my, (c0 & 16) + j);
                                d[j] = (bm >> j & 1u) ? __ldg(p.delta + (int64_t)cj * p.corr_stride + ch) : 0;
                            }
#pragma unroll
                            for (int j = 0; j < 16; j++)
                                v[j] += (uint32_t)d[j];
                        }
                    }
                    // four words at a time through every step: their shuffles and loads are in flight together
                    uint32_t w[4], y[4];
                    const uint32_t dst = s_slot + (uint32_t)c0 * 32u + off;
#pragma unroll
                    for (int q = 0; q < 4; q++)
                    {
                        int32_t z[4];
#pragma unroll
                        for (int e = 0; e < 4; e++)
                            z[e] = rescale_rec_apply((int32_t)v[4 * q + e], rm, rpk, rcpk, rsh, rlo, rhi, FIX);
                        w[q] = chan_pack4(z[0], z[1], z[2], z[3]);
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        y[q] = __shfl_xor_sync(0xffffffffu, w[q], 2);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        w[q] = __byte_perm(w[q], y[q], sel1);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        y[q] = __shfl_xor_sync(0xffffffffu, w[q], 1);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        w[q] = __byte_perm(w[q], y[q], sel2);
                    if (narrow)
                    {
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            w[q] = __vmins4(__vmaxs4(w[q], lo4), hi4);
                    }
                    if (JOIN)
                    {
                        if (!jusable)
                        {
                            // (pixels and channels past the end hold no operands: whatever they give is not stored and says nothing)
                            uint32_t real = 0;
                            for (int q = 0; q < 4; q++)
                                if (pb * p.px + group * cols + c0 + 4 * q + t < p.pixels && cb * 128 + quarter * 32 + (lane & ~3) < p.OC)
                                    real |= 1u << q;
                            chan_join_general(dst, w[0], w[1], w[2], w[3], p.join, p.join_lo, p.join_hi, real, p.status);
                            return;
                        }
                        uint32_t r[4];
#pragma unroll
                        for (int q = 0; q < 4; q++)
                            asm volatile("ld.shared.b32 %0, [%1];" : "=r"(r[q]) : "r"(dst + (uint32_t)q * 128u));
                        {
#pragma unroll
                            for (int q = 0; q < 4; q++)
                            {
                                const uint32_t i01 = __byte_perm(w[q], r[q], 0x5140), i23 = __byte_perm(w[q], r[q], 0x7362);
                                int32_t s[4], z[4];
                                asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(s[0]) : "r"(jcoef), "r"(i01), "r"(jc));
                                asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(s[1]) : "r"(jcoef), "r"(i01), "r"(jc));
                                asm("dp2a.lo.s32.s32 %0, %1, %2, %3;" : "=r"(s[2]) : "r"(jcoef), "r"(i23), "r"(jc));
                                asm("dp2a.hi.s32.s32 %0, %1, %2, %3;" : "=r"(s[3]) : "r"(jcoef), "r"(i23), "r"(jc));
#pragma unroll
                                for (int e = 0; e < 4; e++)
                                {
                                    if (JOIN == 2)
                                        z[e] = join_f32_apply(s[e], __int_as_float(jm), __int_as_float(jsh), __int_as_float(jrlo));
                                    else
                                    {
                                        const int64_t P = (int64_t)s[e] * (int64_t)jm + (int64_t)(((uint64_t)(uint32_t)jrhi << 32) | (uint32_t)jrlo);
                                        z[e] = ((int32_t)(P >> 32) + ((s[e] >> 31) & jfix)) >> jsh;
                                    }
                                }
                                w[q] = chan_pack4(z[0], z[1], z[2], z[3]);
                            }
                            if (jnarrow)
                            {
#pragma unroll
                                for (int q = 0; q < 4; q++)
                                    w[q] = __vmins4(__vmaxs4(w[q], jlo4), jhi4);
                            }
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        asm volatile("st.shared.b32 [%0], %1;" ::"r"(dst + (uint32_t)q * 128u), "r"(w[q]) : "memory");
                };
                auto release = [&] {    // this warp has read its part of the accumulator
                    ptx::tc_fence_before_sync();
                    __syncwarp();
                    if (lane == 0)
                        ptx::mbar_arrive(ptx::smem_u32(&bar_acc_empty[i & 1]));
                };
                // the next sixteen columns are on their way from tensor memory while sixteen are worked on
                uint32_t va[16], vb[16];
                ptx::tmem_ld_32x32b_x16(taddr, va);
                for (int c0 = 0; c0 < cols; c0 += 32)
                {
                    const bool second = c0 + 16 < cols;
                    ptx::tmem_ld_wait_x16(va);
                    if (second)
                        ptx::tmem_ld_32x32b_x16(taddr + (uint32_t)(c0 + 16), vb);
                    else
                        release();
                    work(va, c0);
                    if (second)
                    {
                        ptx::tmem_ld_wait_x16(vb);
                        if (c0 + 32 < cols)
                            ptx::tmem_ld_32x32b_x16(taddr + (uint32_t)(c0 + 32), va);
                        else
                            release();
                        work(vb, c0 + 16);
                    }
                }
            }
            // The slot goes out as one tensor store; the slot of the tile before this one may be filled again once its store
            // has read it.
            ptx::fence_proxy_async_smem();
            if (boss && nslots > 1)
                ptx::bulk_wait_read();
            __syncwarp();
            if (boss)
            {
                ptx::tma_store_2d(&p.tmO, s_slot, cb * 128 + quarter * 32, pb * p.px + group * cols);
                ptx::bulk_commit();
                if (JOIN && i + nslots - 1 < my_tiles)
                {
                    const int rt = tile + (nslots - 1) * (int)gridDim.x;
                    const int rpb = (int)fastdiv_apply((uint32_t)rt, p.fd_cbs), rcb = rt - rpb * p.cbs;
                    const int s2 = slot == 0 ? nslots - 1 : slot - 1;    // (i + nslots - 1) % nslots
                    const uint32_t bar = ptx::smem_u32(&bar_res[ew * kChanStaging + s2]);
                    ptx::mbar_arrive_expect_tx(bar, slot_bytes);
                    ptx::tma_load_2d(s_mine + (uint32_t)s2 * slot_bytes, &p.tmR, bar, rcb * 128 + quarter * 32, rpb * p.px + group * cols);
                }
            }
            if (++slot == nslots)
            {
                slot = 0;
                slot_phase ^= 1u;
            }
        }
        if (boss)
            ptx::bulk_wait_all();
        if (!ok && lane == 0)
        {
            atomicOr(p.status, TB200_DEV_TIMEOUT);
            atomicExch(&abort_flag, 1);
        }
    }

    // ---------------------------------------------------------------------- teardown
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (threadIdx.x == 0 && abort_flag)
    {
        // a role gave up: let copies that may still be in flight land before the CTA's shared memory is released
        for (int s = 0; s < p.num_stages; s++)
        {
            ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[s]), 0u, 2000000LL);
            ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[s]), 1u, 2000000LL);
        }
        if (JOIN)
            for (int s = 0; s < 16 * kChanStaging; s++)
            {
                ptx::mbar_wait_bounded(ptx::smem_u32(&bar_res[s]), 0u, 2000000LL);
                ptx::mbar_wait_bounded(ptx::smem_u32(&bar_res[s]), 1u, 2000000LL);
            }
        if (p.resident)
            ptx::mbar_wait_bounded(ptx::smem_u32(&bar_w), 0u, 2000000LL);
    }
    if (warp == 1 && lane == 0 && abort_flag)
    {
        // ... and let the tensor-core work already issued retire before its accumulators' tensor memory is freed
        ptx::mma_commit(ptx::smem_u32(&bar_drain));
        ptx::mbar_wait_bounded(ptx::smem_u32(&bar_drain), 0u, 40000000LL);
    }
    __syncthreads();
    if (warp == 1)
    {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }
}

// ------------------------------------------------------------------------------------------------ small problems
// The same product where there are fewer tiles than SMs: a chain of latencies, in which the load and the multiplication of
// a whole K by one SM were the longest link (3x3 512 to 512 on one 7x7 map: 590 KB and 144 MMAs in 8 CTAs, 13 of 14 us).
// A cluster of S CTAs shares a tile of 128 channels by PX pixels: each multiplies its part of K, hands every other
// one the columns that one owns (PX / S of them, written to its shared memory) and finishes its own columns.  All
// chunks of a CTA are in flight at once, the weights before the predecessor in the stream has finished.  192 threads and at most
// half of an SM's shared memory, so that two grids fit an SM and the successor's set-up hides behind this one.
// One 128-thread epilogue; results are stored from registers, four channels of a pixel per thread.
// Tensor memory is given back before the CTAs meet: none holds columns that a cluster on another stream waits for.
constexpr int kSplitThreads   = 192;
constexpr int kSplitMaxChunks = 16;

template <int PX>
__global__ void __launch_bounds__(kSplitThreads, 2) conv_split_kernel(const __grid_constant__ ChanParams p)
{
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bar_full[kSplitMaxChunks];
    __shared__ __align__(8) uint64_t bar_acc, bar_drain;
    __shared__ uint32_t tmem_base_holder;
    __shared__ int abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t s_base = (ptx::smem_u32(smem_raw) + 1023u) & ~1023u;
    const int S      = p.split;
    const int rank   = S > 1 ? (int)ptx::cluster_ctarank() : 0;
    const int tile   = (int)blockIdx.x / S;
    const int pb     = (int)fastdiv_apply((uint32_t)tile, p.fd_cbs), cb = tile - pb * p.cbs;
    const int p0     = pb * PX;
    const int first  = rank * p.chunks_per_cta;
    const int chunks = max(0, min(p.chunks_per_cta, p.total_chunks - first));

    if (S > 1)
        ptx::cluster_arrive();    // this CTA has started: waited for before its shared memory is written to
    if (threadIdx.x == 0)
    {
        for (int c = 0; c < chunks; c++)
            ptx::mbar_init(ptx::smem_u32(&bar_full[c]), 1);
        ptx::mbar_init(ptx::smem_u32(&bar_acc), 1);
        ptx::mbar_init(ptx::smem_u32(&bar_drain), 1);
        abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::prefetch_tmap(&p.tmW);
        ptx::prefetch_tmap(&p.tmX);
    }
    if (warp == 1)
    {
        ptx::tmem_alloc(ptx::smem_u32(&tmem_base_holder), (uint32_t)p.tmem_cols);
        ptx::tmem_relinquish();
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_holder;
    // (behind the allocation: a successor may take what is left of this SM's tensor memory)
    if (threadIdx.x == 0)
        ptx::dep_launch_trigger();

    const int quarter = warp & 3, t = lane & 3;
    const int own     = PX / S;                   // columns of the tile that this CTA finishes
    const int col0    = rank * own;
    const int ch4     = cb * 128 + quarter * 32 + (lane & ~3);    // this thread's four channels after the transposition
    const int64_t at0 = (int64_t)(p0 + col0 + t) * p.OC + ch4;    // ... of column col0 + t
    uint32_t v[PX];
    uint32_t res[PX / 4];
    int cls[2]         = { 0, 0 };
    uint32_t border[2] = { 0, 0 };
    int32_t rm = 0, rpk = 0, rcpk = 0, rsh = 0, rlo = 0, rhi = 0;
    const int ch = cb * 128 + quarter * 32 + lane;
    bool ok      = true;

    if (warp == 0)
    {
        if (lane == 0)
        {
            for (int c = 0; c < chunks; c++)
            {
                const uint32_t full = ptx::smem_u32(&bar_full[c]);
                ptx::mbar_arrive_expect_tx(full, (uint32_t)((PX + 128) * p.chunk));
                ptx::tma_load_3d(s_base + (uint32_t)(c * p.stage_bytes + p.x_chunk_bytes), &p.tmW, full, (first + c) * p.chunk, cb * 128, 0);
            }
            ptx::dep_launch_wait();
            int n0 = 0, y0 = 0, x0 = 0;
            if (p.im2col)
            {
                n0           = (int)fastdiv_apply((uint32_t)p0, p.fd_ohow);
                const int r  = p0 - n0 * (p.OH * p.OW);
                const int oy = (int)fastdiv_apply((uint32_t)r, p.fd_ow);
                y0           = oy * p.stride_y - p.pad_t;
                x0           = (r - oy * p.OW) * p.stride_x - p.pad_l;
            }
            const int tap = first / p.chunks_per_tap;
            int cc = first - tap * p.chunks_per_tap, ky = tap / p.KW, kx = tap - ky * p.KW;
            for (int c = 0; c < chunks; c++)
            {
                const uint32_t full = ptx::smem_u32(&bar_full[c]), dst = s_base + (uint32_t)(c * p.stage_bytes);
                if (p.im2col)
                    ptx::tma_load_im2col_4d(dst, &p.tmX, full, cc * p.chunk, x0, y0, n0, (uint16_t)(kx * p.dil_x), (uint16_t)(ky * p.dil_y));
                else
                    ptx::tma_load_2d(dst, &p.tmX, full, cc * p.chunk, p0);
                if (++cc == p.chunks_per_tap)
                {
                    cc = 0;
                    if (++kx == p.KW)
                    {
                        kx = 0;
                        ky++;
                    }
                }
            }
        }
    }
    else if (warp == 1)
    {
        if (lane == 0)
        {
            uint32_t accum = 0;
            for (int c = 0; c < chunks; c++)
            {
                if (!ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[c]), 0u, p.wait_limit))
                {
                    ok = false;
                    break;
                }
                ptx::tc_fence_after_sync();
                const uint32_t sx = s_base + (uint32_t)(c * p.stage_bytes);
                ptx::mma_i8_ss_chunk(tmem_base, ptx::smem_desc(p.desc_hi, sx + (uint32_t)p.x_chunk_bytes), ptx::smem_desc(p.desc_hi, sx), p.idesc, accum,
                                     p.mmas);
                accum = 1;
            }
            if (ok && chunks > 0)
                ptx::mma_commit(ptx::smem_u32(&bar_acc));
            if (!ok)
                atomicExch(&abort_flag, 1);
        }
    }
    else
    {
        // constants, and what does not depend on the product, while it is on its way
        const int4 r0 = __ldg(reinterpret_cast<const int4*>(p.rec + (int64_t)ch * 8));
        const int2 r1 = __ldg(reinterpret_cast<const int2*>(p.rec + (int64_t)ch * 8 + 4));
        rm = r0.x; rpk = r0.y; rcpk = r0.z; rsh = r0.w; rlo = r1.x; rhi = r1.y;
        if (p.delta != nullptr)
        {
#pragma unroll
            for (int k = 0; k < (PX > 32 ? 2 : 1); k++)
            {
                const int pix = p0 + col0 + k * 32 + lane;
                const int n   = (int)fastdiv_apply((uint32_t)pix, p.fd_ohow);
                const int r   = pix - n * (p.OH * p.OW);
                const int oy  = (int)fastdiv_apply((uint32_t)r, p.fd_ow);
                bool b;
                cls[k]    = chan_border_class(p, oy, r - oy * p.OW, &b);
                border[k] = __ballot_sync(0xffffffffu, b);
            }
        }
        // the other operand of a join is the predecessor's (an ordinary load, which stays behind this); the output may still be read by it
        ptx::dep_launch_wait();
        if (p.join != nullptr)
        {
#pragma unroll
            for (int q = 0; q < PX / 4; q++)
                if (4 * q < own)
                    res[q] = p0 + col0 + 4 * q + t < p.pixels && ch4 < p.OC
                                 ? *reinterpret_cast<const uint32_t*>(p.res + at0 + (int64_t)(4 * q) * p.OC)
                                 : 0u;
        }
        if (chunks > 0)
        {
            ok = ptx::mbar_wait_bounded(ptx::smem_u32(&bar_acc), 0u, p.wait_limit);
            ok = __all_sync(0xffffffffu, ok);
        }
        if (ok && chunks > 0)
        {
            ptx::tc_fence_after_sync();
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
            for (int c = 0; c < PX; c += 16)
            {
                uint32_t x[16];
                ptx::tmem_ld_32x32b_x16(taddr + (uint32_t)c, x);
                ptx::tmem_ld_wait_x16(x);
#pragma unroll
                for (int j = 0; j < 16; j++)
                    v[c + j] = x[j];
            }
        }
        else
        {
#pragma unroll
            for (int c = 0; c < PX; c++)
                v[c] = 0;
        }
        if (!ok && lane == 0)
            atomicExch(&abort_flag, 1);
    }

    // ---------------------------------------------------------------------- tensor memory goes back before the CTAs meet
    ptx::tc_fence_before_sync();
    __syncthreads();
    const bool aborted = abort_flag != 0;
    if (aborted)
    {
        if (threadIdx.x == 0)
        {
            atomicOr(p.status, TB200_DEV_TIMEOUT);
            // let copies that may still be in flight land before the CTA's shared memory is released
            for (int c = 0; c < chunks; c++)
                ptx::mbar_wait_bounded(ptx::smem_u32(&bar_full[c]), 0u, 2000000LL);
        }
        if (warp == 1 && lane == 0)
        {
            ptx::mma_commit(ptx::smem_u32(&bar_drain));
            ptx::mbar_wait_bounded(ptx::smem_u32(&bar_drain), 0u, 40000000LL);
        }
        __syncthreads();
    }
    if (warp == 1)
    {
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, (uint32_t)p.tmem_cols);
    }

    // ---------------------------------------------------------------------- columns to their owners
    const uint32_t s_red = s_base + (uint32_t)p.red_off;    // [source rank][own columns][128 channels]
    if (S > 1)
    {
        ptx::cluster_wait();
        if (warp >= 2)
        {
            const uint32_t mine = s_red + (uint32_t)(rank * own) * 512u + (uint32_t)(quarter * 32 + lane) * 4u;
#pragma unroll
            for (int c = 0; c < PX; c++)
            {
                const int d = c >> (__ffs(own) - 1);    // (own is a power of two of at least 4)
                ptx::st_shared_cluster(ptx::map_to_cta(mine + (uint32_t)(c & (own - 1)) * 512u, (uint32_t)d), v[c]);
            }
        }
        ptx::cluster_arrive();
        ptx::cluster_wait();
    }
    if (warp < 2 || aborted)
        return;

    // ---------------------------------------------------------------------- RESCALE, join, store
    const uint32_t sel1 = t < 2 ? 0x5410u : 0x3276u, sel2 = (t & 1) ? 0x3715u : 0x6240u;
    const bool narrow  = p.clamp_lo > -128 || p.clamp_hi < 127;
    const uint32_t lo4 = (uint32_t)(p.clamp_lo & 0xff) * 0x01010101u, hi4 = (uint32_t)(p.clamp_hi & 0xff) * 0x01010101u;
    auto emit = [&](int q, int32_t(&x)[4], uint32_t other) {
        if (p.delta != nullptr)
        {
            const uint32_t bm = (q >= 8 ? border[1] : border[0]) >> ((4 * q) & 31) & 15u;
            if (bm != 0)
            {
#pragma unroll
                for (int e = 0; e < 4; e++)
                {
                    const int cj = __shfl_sync(0xffffffffu, q >= 8 ? cls[1] : cls[0], (4 * q + e) & 31);
                    if (bm >> e & 1u)
                        x[e] += __ldg(p.delta + (int64_t)cj * p.corr_stride + ch);
                }
            }
        }
        int32_t z[4];
#pragma unroll
        for (int e = 0; e < 4; e++)
            z[e] = p.double_round ? rescale_rec_apply(x[e], rm, rpk, rcpk, rsh, rlo, rhi, true)
                                  : rescale_rec_apply(x[e], rm, rpk, rcpk, rsh, rlo, rhi, false);
        uint32_t w = chan_pack4(z[0], z[1], z[2], z[3]);
        uint32_t y = __shfl_xor_sync(0xffffffffu, w, 2);
        w          = __byte_perm(w, y, sel1);
        y          = __shfl_xor_sync(0xffffffffu, w, 1);
        w          = __byte_perm(w, y, sel2);
        if (narrow)
            w = __vmins4(__vmaxs4(w, lo4), hi4);
        const bool real = p0 + col0 + 4 * q + t < p.pixels && ch4 < p.OC;
        if (p.join != nullptr)
            w = chan_join_word(w, other, p.join, p.join_lo, p.join_hi, real ? p.status : nullptr);
        if (real)
            *reinterpret_cast<uint32_t*>(p.out + at0 + (int64_t)(4 * q) * p.OC) = w;
    };
    if (S == 1)
    {
#pragma unroll
        for (int q = 0; q < PX / 4; q++)
        {
            int32_t x[4] = { (int32_t)v[4 * q], (int32_t)v[4 * q + 1], (int32_t)v[4 * q + 2], (int32_t)v[4 * q + 3] };
            emit(q, x, res[q]);
        }
    }
    else
    {
        const uint32_t mine = s_red + (uint32_t)(quarter * 32 + lane) * 4u;
#pragma unroll
        for (int q = 0; q < PX / 8; q++)
            if (4 * q < own)
            {
                int32_t x[4] = { 0, 0, 0, 0 };
                for (int r = 0; r < S; r++)
#pragma unroll
                    for (int e = 0; e < 4; e++)
                    {
                        int32_t y;
                        asm volatile("ld.shared.b32 %0, [%1];" : "=r"(y) : "r"(mine + (uint32_t)(r * own + 4 * q + e) * 512u));
                        x[e] += y;
                    }
                emit(q, x, res[q]);
            }
    }
}

// ------------------------------------------------------------------------------------------------ planning
typedef CUresult (*PFN_encodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                    const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                    CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
typedef CUresult (*PFN_encodeIm2col)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                     const int*, const int*, cuuint32_t, cuuint32_t, const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

PFN_encodeIm2col im2col_encode_fn()
{
    static PFN_encodeIm2col fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &f, cudaEnableDefault, &st) == cudaSuccess && st == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_encodeIm2col>(f);
    });
    return fn;
}

struct ChanPlan
{
    ChanParams kp;
    int grid, smem_bytes;
    int64_t sw, sh, sn;
    int lower[2], upper[2];    // im2col corners (x, y)
    CUtensorMapSwizzle swz;
};

// SM cycles of a small problem on conv_split_kernel, in the measure of chan_choose's estimates (fitted to device times of layers on
// one and two images): a chunk costs its MMAs, an exchange the columns that a CTA hands out and finishes; 0: not worth trying.
double split_cost(int px, int S, int chunks, int mmas)
{
    const double chunk = 130.0 * mmas + 50;
    if (px == 32)
        return chunks * chunk + (S == 2 ? 4800 : 3600);
    return S == 8 ? chunks * chunk + 5600 : S == 4 ? chunks * chunk + 6600 : 0;
}

// Which kernel takes a problem of these sizes, if any, and in which layout: a function of the sizes alone.
ChanChoice chan_choose(int num_sms, int max_smem, int64_t pixels, int OC, int IC, int KH, int KW, bool join)
{
    ChanChoice c;
    memset(&c, 0, sizeof(c));
    const int swz = IC % 128 == 0 ? 128 : IC % 64 == 0 ? 64 : 32, mmas = swz / 32, w_chunk_bytes = 128 * swz;
    const int total_chunks = KH * KW * (IC / swz), cbs = (OC + 127) / 128;
    const int budget = (max_smem > 0 ? max_smem : 232448) - 2048;

    // Pixels per tile, where the weights live, slots and stages: the smallest estimate of a first tile from its loads
    // to its store, and the longest of MMAs, epilogue and loads for every further round.  SM cycles: an MMA of 128 channels by 256 / 192 / 128 / 64 pixels and
    // 32 bytes of K 171 / 139 / 107 / 104, a commit 60; loads bring 50 bytes per cycle to an SM, 32 when all SMs load (3x3 512 to
    // 512 on 256x7x7: 8.9 TB/s in tiles of 128 and of 240 pixels alike), and no more than what is in flight (the ring less the
    // stage in use) per 2900 cycles of latency.
    double best = 0;
    for (const int px : { 256, 192, 128, 64 })
        for (int res = 1; res >= 0; res--)
            for (int slots = join ? 3 : 2; slots >= (join ? 2 : 1); slots--)
            {
                const int64_t pbs = (pixels + px - 1) / px, tiles = pbs * cbs;
                if (tiles >= (1LL << 30))
                    continue;
                const int staging = slots * px * 128;
                const int w_bytes = res ? total_chunks * w_chunk_bytes : 0;
                int grid = (int)std::min<int64_t>(tiles, num_sms);
                if (res)
                {
                    if (cbs > num_sms || w_bytes > budget)
                        continue;
                    grid = (int)std::min<int64_t>(tiles, (int64_t)num_sms / cbs * cbs);
                }
                const int per_chunk = px * swz + (res ? 0 : w_chunk_bytes);
                const int avail     = budget - 1024 - staging - w_bytes;
                if (avail < 2 * per_chunk)
                    continue;
                int ksub = std::max(1, std::min(total_chunks, 48 * 1024 / per_chunk));
                while (ksub > 1 && avail / (ksub * per_chunk) < 3)
                    ksub--;
                const int stages = std::min(kChanMaxStages, avail / (ksub * per_chunk));
                const double rate = std::min(std::min(50.0, 32.0 * num_sms / grid), (double)(stages - 1) * ksub * per_chunk / 2900.0);
                const double mma  = (double)total_chunks * mmas * (px == 256 ? 171 : px == 192 ? 139 : px == 128 ? 107 : 104) +
                                   60.0 * ((total_chunks + ksub - 1) / ksub + 1);
                const double epi  = px * (join ? 26.0 : 14.7) + 500;
                const double load = (double)total_chunks * per_chunk / rate + (join ? px * 128 / 50.0 : 0.0);
                const int64_t rounds = (tiles + grid - 1) / grid;
                // the store, or the residual's load, is not overlapped.  (With a join two slots take as long as three where the tile is the
                // same, 256 channels 3x3 on 128x14x14x256 24.4 / 24.3 us, 512 on 256x7x7x512 37.9 / 38.0, and less where they make room
                // for a larger one, 128 on 128x28x28x128 24.9 / 27.5.)
                const bool few       = slots == (join ? 2 : 1);
                const double cost = 1200 + std::max(mma, load + w_bytes / 50.0) + epi + (double)(rounds - 1) * (std::max(mma, std::max(epi, load)) + (few ? 300 : 0));
                if (best == 0 || cost < best * 0.98)
                {
                    best            = cost;
                    c.px            = px;
                    c.resident      = res;
                    c.slots         = slots;
                    c.ksub          = ksub;
                    c.num_stages    = stages;
                    c.x_chunk_bytes = px * swz;
                    c.stage_bytes   = ksub * per_chunk;
                    c.tiles         = (int)tiles;
                    c.w_off         = staging;
                    c.ring_off      = staging + w_bytes;
                    c.grid      = grid;
                    c.smem_bytes = 1024 + staging + w_bytes + stages * ksub * per_chunk;
                }
            }
    // One tile per cluster of S CTAs, where that fills one wave at most (conv_split_kernel).
    for (int px = 64; px >= 32; px >>= 1)
        for (int S = 1; S <= 8 && px / S >= 4 && S <= total_chunks; S *= 2)
        {
            const int64_t tiles = (pixels + px - 1) / px * cbs;
            const int cpc       = (total_chunks + S - 1) / S;
            const int stage     = (px + 128) * swz;
            const int smem      = 1024 + cpc * stage + (S > 1 ? px * 512 : 0);
            // one wave: clusters of 8 and 4 leave SMs of a GPC over when a CTA fills its SM
            const int room = smem <= 110 * 1024 || S == 1 ? num_sms : num_sms * (S == 8 ? 3 : 4) / (S == 8 ? 4 : 5);
            if (tiles * S > room || cpc > kSplitMaxChunks || smem > budget)
                continue;
            const double cost = split_cost(px, S, cpc, mmas);
            if (cost > 0 && (best == 0 || cost < best))
            {
                best             = cost;
                c.split          = S;
                c.chunks_per_cta = cpc;
                c.px             = px;
                c.x_chunk_bytes  = px * swz;
                c.stage_bytes    = stage;
                c.red_off        = cpc * stage;
                c.tiles          = (int)tiles;
                c.grid       = (int)tiles * S;
                c.smem_bytes = smem;
            }
        }
    if (best == 0)
        return c;
    // Channel blocks less than three quarters full leave rows of the product and threads of the epilogue idle: 160 channels on
    // 21x102x13x96 7.6 us against 6.6 with a pixel per thread, 32 channels 3x3 on 13x32x12x32 8.5 against 5.9; 192 channels 3x3 on
    // 8x26x10x192 10.4 against 13.5.  Where the products are long and the pixels many they are what counts, and there this kernel
    // needs fewer of them (K, pixels, us here / with a pixel per thread): 64 channels 3200, 14 850 15.0 / 19.6, 4320, 26 884 35.7 / 91.5,
    // 3744, 25 688 31.7 / 42.3, but 3456, 12 312 15.9 / 12.6, 4608, 13 392 18.7 / 14.6, 4320, 9 085 31.1 / 26.0; 32 channels 4000, 61 950
    // 92 / 125, 4800, 16 302 26.3 / 32.9, but 3456, 27 360 27.0 / 20.2, 3168, 81 576 116 / 85, 4000, 6 912 42.9 / 24.0.
    // A residual join pays for itself at any width.
    const int rows = (OC + 127) / 128 * 128;
    if (!c.split && !join && OC * 4 < rows * 3 &&
        ((int64_t)KH * KW * IC < (OC * 4 <= rows ? 4000 : 3072) || pixels < 96 * (int64_t)num_sms))
        return c;
    // Windows over 32-byte pieces, loaded again for each of several channel blocks: 512 channels 3x3 on 24x34x49x96 23.7 / 19.9, 256
    // 5x5 on 22x18x50x32 25.9 / 18.9, 448 3x3 on 54x11x18x32 16.4 / 12.0, 416 5x5 on 9x64x25x96 41.3 / 38.4.
    if (!c.split && !join && KH * KW > 1 && IC % 64 != 0 && OC >= 256)
        return c;
    c.taken = 1;
    return c;
}

bool chan_plan(tb200_ctx* ctx, const TcProblem& q, ChanPlan* plan)
{
    if (q.epi != TC_EPI_RESCALE || !q.lean_ok || q.rec == nullptr || q.rec_ok == nullptr || q.b_mn_major || q.in_dtype != TB200_INT8 ||
        q.out_dtype != TB200_INT8 || q.out_sy != 0 || q.xpar || q.tile_begin != 0 || q.tile_end != 0)
        return false;
    if (q.OC % 32 != 0 || q.IC % 32 != 0 || ((reinterpret_cast<uintptr_t>(q.out) | reinterpret_cast<uintptr_t>(q.a) |
                                               reinterpret_cast<uintptr_t>(q.b) | reinterpret_cast<uintptr_t>(q.res)) & 15) != 0)
        return false;
    if (q.clamp_lo < -128 || q.clamp_hi > 127 || q.clamp_lo > q.clamp_hi || q.out_zp < -128 || q.out_zp > 127)
        return false;
    if (q.corr_classes && q.delta == nullptr)
        return false;
    const int64_t pixels = (int64_t)q.N * q.OH * q.OW;
    if (pixels >= (1LL << 30))
        return false;
    const int64_t sw = q.a_stride_w ? q.a_stride_w : (int64_t)q.IC;
    const int64_t sh = q.a_stride_h ? q.a_stride_h : sw * q.IW;
    const int64_t sn = q.a_stride_n ? q.a_stride_n : sh * q.IH;
    if (sw % 16 != 0 || sh % 16 != 0 || sn % 16 != 0 || sn >= (1LL << 40) || sh >= (1LL << 40))
        return false;
    const bool flat = q.KH == 1 && q.KW == 1 && q.stride_y == 1 && q.stride_x == 1 && q.pad_t == 0 && q.pad_l == 0 && q.OH == q.IH &&
                      q.OW == q.IW && sw == q.IC && sh == sw * q.IW && sn == sh * q.IH;
    memset(&plan->kp, 0, sizeof(plan->kp));
    ChanParams& k = plan->kp;
    plan->sw = sw; plan->sh = sh; plan->sn = sn;
    if (!flat)
    {
        // corners of the box that a window's first tap walks over, relative to the image; tap offsets; strides
        plan->lower[0] = -q.pad_l;
        plan->lower[1] = -q.pad_t;
        plan->upper[0] = -q.pad_l + q.stride_x * (q.OW - 1) - (q.IW - 1);
        plan->upper[1] = -q.pad_t + q.stride_y * (q.OH - 1) - (q.IH - 1);
        for (int d = 0; d < 2; d++)
            if (plan->lower[d] < -128 || plan->lower[d] > 127 || plan->upper[d] < -128 || plan->upper[d] > 127)
                return false;
        if (q.stride_x > 8 || q.stride_y > 8 || (q.KW - 1) * q.dil_x > 255 || (q.KH - 1) * q.dil_y > 255 || im2col_encode_fn() == nullptr)
            return false;
    }
    k.im2col = flat ? 0 : 1;
    k.pixels = (int)pixels;
    k.OC     = q.OC;
    k.OH = q.OH; k.OW = q.OW; k.IH = q.IH; k.IW = q.IW; k.KH = q.KH; k.KW = q.KW;
    k.pad_t = q.pad_t; k.pad_l = q.pad_l; k.stride_y = q.stride_y; k.stride_x = q.stride_x; k.dil_y = q.dil_y; k.dil_x = q.dil_x;
    const int swz    = q.IC % 128 == 0 ? 128 : q.IC % 64 == 0 ? 64 : 32;
    plan->swz        = swz == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : swz == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B;
    k.chunk          = swz;
    k.chunks_per_tap = q.IC / swz;
    k.total_chunks   = q.KH * q.KW * k.chunks_per_tap;
    k.mmas           = swz / 32;
    k.cbs            = (q.OC + 127) / 128;
    k.w_chunk_bytes  = 128 * swz;
    k.desc_hi        = ptx::make_smem_desc_hi(16, 8 * swz, swz == 128 ? 2u : swz == 64 ? 4u : 6u);
    bool known = false;
    if (!ctx->chan_memo)
        ctx->chan_memo.reset(new SizeMemo<ChanChoice>());
    auto& memo = ctx->chan_memo->at(pixels, (int64_t)q.OC << 32 | q.IC, (int64_t)q.KH << 32 | q.KW << 1 | (q.join ? 1 : 0), &known);
    if (!known)
        memo.value = chan_choose(ctx->num_sms, ctx->max_smem_optin, pixels, q.OC, q.IC, q.KH, q.KW, q.join != nullptr);
    const ChanChoice& c = memo.value;
    if (!c.taken)
        return false;
    k.px = c.px; k.resident = c.resident; k.slots = c.slots; k.ksub = c.ksub; k.num_stages = c.num_stages;
    k.x_chunk_bytes = c.x_chunk_bytes; k.stage_bytes = c.stage_bytes; k.tiles = c.tiles; k.w_off = c.w_off; k.ring_off = c.ring_off;
    k.split = c.split; k.chunks_per_cta = c.chunks_per_cta; k.red_off = c.red_off;
    plan->grid = c.grid; plan->smem_bytes = c.smem_bytes;
    k.idesc     = ptx::make_idesc(2u, 1u, 1u, 0u, 0u, 128u, (uint32_t)k.px);
    k.tmem_cols = k.split ? k.px : k.px == 192 ? 512 : 2 * k.px;
    fastdiv_make((uint32_t)(q.OH * q.OW), k.fd_ohow);
    fastdiv_make((uint32_t)q.OW, k.fd_ow);
    fastdiv_make((uint32_t)k.cbs, k.fd_cbs);
    return true;
}

}    // namespace

bool conv_chan_supported(tb200_ctx* ctx, const TcProblem& q)
{
    ChanPlan plan;
    return chan_plan(ctx, q, &plan);
}

tb200_status conv_chan_launch(tb200_ctx* ctx, const TcProblem& q, bool* taken)
{
    ChanPlan plan;
    *taken = chan_plan(ctx, q, &plan);
    if (!*taken)
        return TB200_OK;
    PFN_encodeTiled enc = reinterpret_cast<PFN_encodeTiled>(tensor_map_encode_fn());
    if (!enc)
        return fail(ctx, TB200_INTERNAL, "cuTensorMapEncodeTiled is not available from the driver");
    ChanParams& k = plan.kp;
    const cuuint32_t ones[4] = { 1, 1, 1, 1 };
    const cuuint64_t pixels  = (cuuint64_t)q.N * q.OH * q.OW;
    auto matrix = [&](CUtensorMap* m, const void* base, cuuint64_t rows, cuuint64_t row_bytes, cuuint32_t bx, cuuint32_t by,
                      CUtensorMapSwizzle s) {
        const cuuint64_t dims[2] = { row_bytes, rows }, strides[1] = { row_bytes };
        const cuuint32_t box[2]  = { bx, by };
        return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void*>(base), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, s,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r;
    if (k.im2col)
    {
        const cuuint64_t dims[4]    = { (cuuint64_t)q.IC, (cuuint64_t)q.IW, (cuuint64_t)q.IH, (cuuint64_t)q.N };
        const cuuint64_t strides[3] = { (cuuint64_t)plan.sw, (cuuint64_t)plan.sh, (cuuint64_t)plan.sn };
        const cuuint32_t estr[4]    = { 1, (cuuint32_t)q.stride_x, (cuuint32_t)q.stride_y, 1 };
        r = im2col_encode_fn()(&k.tmX, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<void*>(q.a), dims, strides, plan.lower, plan.upper,
                               (cuuint32_t)k.chunk, (cuuint32_t)k.px, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, plan.swz,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    else
        r = matrix(&k.tmX, q.a, pixels, (cuuint64_t)q.IC, (cuuint32_t)k.chunk, (cuuint32_t)k.px, plan.swz);
    if (r != CUDA_SUCCESS)
        return fail(ctx, TB200_INTERNAL, "tensor map for the activations rejected (CUresult %d)", (int)r);
    {
        const cuuint64_t ktot = (cuuint64_t)q.KH * q.KW * q.IC;
        const cuuint64_t dims[3] = { ktot, (cuuint64_t)q.OC, 1 }, strides[2] = { ktot, ktot * q.OC };
        const cuuint32_t box[3]  = { (cuuint32_t)k.chunk, 128, 1 };
        r = enc(&k.tmW, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void*>(q.b), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE, plan.swz,
                CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    }
    if (r == CUDA_SUCCESS && !k.split)
        r = matrix(&k.tmO, q.out, pixels, (cuuint64_t)q.OC, 32, (cuuint32_t)k.px / 4, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (r == CUDA_SUCCESS && !k.split && q.join)
        r = matrix(&k.tmR, q.res, pixels, (cuuint64_t)q.OC, 32, (cuuint32_t)k.px / 4, CU_TENSOR_MAP_SWIZZLE_NONE);
    if (r != CUDA_SUCCESS)
        return fail(ctx, TB200_INTERNAL, "tensor map rejected (CUresult %d)", (int)r);
    k.rec = q.rec; k.delta = q.delta; k.corr_stride = q.corr_stride;
    k.clamp_lo = q.clamp_lo; k.clamp_hi = q.clamp_hi;
    k.join = q.join; k.join_lo = q.join_lo; k.join_hi = q.join_hi;
    k.wait_limit = ctx->wait_limit_cycles;
    k.status     = ctx->d_status;
    k.double_round = q.double_round;
    k.out          = reinterpret_cast<int8_t*>(q.out);
    k.res          = reinterpret_cast<const int8_t*>(q.res);
    if (!q.corr_classes)
        k.delta = nullptr;

    typedef void (*Kern)(const ChanParams);
    if (k.split)
    {
        const Kern kern        = k.px == 64 ? conv_split_kernel<64> : conv_split_kernel<32>;
        const tb200_status ast = raise_smem_limit(ctx, 76 + (k.px == 64 ? 1 : 0), reinterpret_cast<const void*>(kern), plan.smem_bytes);
        if (ast != TB200_OK)
            return ast;
        timer_begin(ctx);
        cudaLaunchConfig_t cfg;
        memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim          = dim3((unsigned)plan.grid);
        cfg.blockDim         = dim3((unsigned)kSplitThreads);
        cfg.dynamicSmemBytes = (size_t)plan.smem_bytes;
        cfg.stream           = ctx->stream;
        cudaLaunchAttribute at[2];
        at[0].id               = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = (unsigned)k.split;
        at[0].val.clusterDim.y = 1;
        at[0].val.clusterDim.z = 1;
        at[1].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs    = at;
        cfg.numAttrs = ctx->launch_overlap ? 2 : 1;
        cudaLaunchKernelEx(&cfg, kern, k);
        timer_end(ctx);
        const tb200_status st = post_launch(ctx, q.join ? "tc_conv_lean_i8_join" : "tc_conv_lean_i8");
        ctx->form             = { "conv_split", k.px, 0, k.split, 1 };
        return st;
    }
    static const Kern kerns[2][2][3] = {
        { { conv_chan_kernel<false, false, 0>, conv_chan_kernel<false, false, 1>, conv_chan_kernel<false, false, 2> },
          { conv_chan_kernel<false, true, 0>, conv_chan_kernel<false, true, 1>, conv_chan_kernel<false, true, 2> } },
        { { conv_chan_kernel<true, false, 0>, conv_chan_kernel<true, false, 1>, conv_chan_kernel<true, false, 2> },
          { conv_chan_kernel<true, true, 0>, conv_chan_kernel<true, true, 1>, conv_chan_kernel<true, true, 2> } } };
    const int ci = q.corr_classes ? 1 : 0, fi = q.double_round ? 1 : 0, ji = q.join ? (q.join_f32 ? 2 : 1) : 0;
    const Kern kern = kerns[ci][fi][ji];
    const tb200_status ast = raise_smem_limit(ctx, 64 + (ci * 2 + fi) * 3 + ji, reinterpret_cast<const void*>(kern), plan.smem_bytes);
    if (ast != TB200_OK)
        return ast;
    timer_begin(ctx);
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim          = dim3((unsigned)plan.grid);
    cfg.blockDim         = dim3((unsigned)kChanThreads);
    cfg.dynamicSmemBytes = (size_t)plan.smem_bytes;
    cfg.stream           = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs    = at;
    cfg.numAttrs = ctx->launch_overlap ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, k);
    timer_end(ctx);
    const tb200_status st = post_launch(ctx, q.join ? "tc_conv_lean_i8_join" : "tc_conv_lean_i8");
    ctx->form             = { "conv_chan", k.px, k.slots, 0, 1 };
    return st;
}

}    // namespace tb200
