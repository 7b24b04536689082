// int8 DEPTHWISE_CONV2D + RESCALE (+ CLAMP) to int8, 3 x 3 and 5 x 5 windows, stride 1 or 2.
//
// A depthwise layer multiplies each channel with its own few weights: no contraction for the tensor cores, and with int8
// operands the integer instructions bound it long before memory does.  What a thread does here is chosen to need few of
// them.  It owns four neighbouring channels (one 32-bit word per pixel) and walks along x:
//   * the words of the window's rows at one x are transposed (6 to 8 byte permutes) into one word per channel that holds
//     that channel's column of the window, and a column serves every output that looks at it: one dp4a per output, channel
//     and column instead of one multiply-add per tap;
//   * at stride 1 a 3 x 3 thread makes two output rows: four rows fill the column words, and the second row's weights are
//     the first's shifted by a byte;
//   * weights, packed by columns, and the lean RESCALE records (rescale_rec_build) are prepared once per layer and sit in
//     registers for the whole walk; taps outside the image read the input zero point, so that all pixels share them.  Where a
//     record is not usable a thread makes its outputs one by one with the general arithmetic (beside the walk, which it would
//     cost 20 registers).  The kernel reads that verdict itself, so no call waits for it and a captured graph follows
//     constants that are replaced under it.
// Channel counts that are no multiple of four read each word as two aligned ones.
// 32 x 56 x 56 x 144, 3 x 3: 18.4 us per call with operands that come from DRAM, 16.6 from L2 (24.5 and 20.0 where each load was
// used as soon as it was asked for and a row's pieces were made without regard to the waves of blocks);
// 32 x 57 x 57 x 144 stride 2 14.3 -> 9.2, 16 x 28 x 28 x 240 5 x 5 stride 2 9.9 -> 5.3.  What bounds it: 17 instructions per
// output of four channels and row, issued in 40 % of the slots by the 14 warps per SM that registers and pieces leave.
#include <algorithm>
#include <cuda_runtime.h>

#include "common.h"
#include "rescale_math.cuh"

namespace tb200
{
namespace
{

struct DwSlideParams
{
    const int8_t* in;
    const int8_t* in_end;    // one past the input's last byte
    int8_t* out;
    const int4* wcol;        // [K][C4 / 4]: per channel the window column's first four rows, one byte each
    const int4* wrow5;       // [K][C4 / 4]: 5 x 5 only, the fifth row's weight at the channel's own byte
    const int4* rec;         // [C4][2]
    const int* usable;       // whether every record may be used; else (walk_general):
    const int8_t* w;         // [K][K][C]
    const int32_t* corr;     // [C4] bias less the zero point's share
    const int32_t* mult;
    const int8_t* shift;
    int per_channel, out_zp;
    int* status;
    int N, IH, IW, C, OH, OW, pad_t, pad_l;
    int c4, strips, row_groups, len;    // channel words, pieces of a row, groups of rows, outputs of a piece
    uint32_t fd_c4[2], fd_strips[2], fd_rg[2];
    int total;               // threads with work
    uint32_t fill4;
    int clamp_lo, clamp_hi;
};

// Outputs [ox0, ox1) x `rows` rows of four channels, tap by tap, by apply_scale_32 with its checks.
__device__ __noinline__ void walk_general(const DwSlideParams& p, int K, int S, int double_round, int n, int oy, int rows, int c, int ox0, int ox1)
{
    const int live = min(4, p.C - c), zp = (int)(int8_t)(p.fill4 & 0xffu);
    bool bad       = false;
    for (int y = oy; y < min(p.OH, oy + rows); y++)
        for (int ox = ox0; ox < ox1; ox++)
            for (int i = 0; i < live; i++)
            {
                int32_t acc = p.corr[c + i];
                for (int k = 0; k < K * K; k++)
                {
                    const int iy = y * S - p.pad_t + k / K, ix = ox * S - p.pad_l + k % K;
                    const bool inside = (unsigned)iy < (unsigned)p.IH && (unsigned)ix < (unsigned)p.IW;
                    const int v = inside ? (int)p.in[(((int64_t)n * p.IH + iy) * p.IW + ix) * p.C + c + i] : zp;
                    acc += v * (int)p.w[k * p.C + c + i];
                }
                const int at = p.per_channel ? c + i : 0;
                int64_t z    = (int64_t)apply_scale_32_dev(acc, p.mult[at], p.shift[at], double_round != 0, bad) + p.out_zp;
                bad |= z > 2147483647LL || z < -2147483648LL;
                z = z < p.clamp_lo ? p.clamp_lo : z > p.clamp_hi ? p.clamp_hi : z;
                p.out[(((int64_t)n * p.OH + y) * p.OW + ox) * p.C + c + i] = (int8_t)z;
            }
    if (bad)
        atomicOr(p.status, TB200_DEV_UNPREDICTABLE);
}

template <int K, int S, bool ALIGNED, bool FIX>
__global__ void __launch_bounds__(128) depthwise_slide_i8_kernel(const __grid_constant__ DwSlideParams p)
{
    constexpr int R  = (K == 3 && S == 1) ? 2 : 1;    // output rows per thread
    constexpr int NR = (R - 1) * S + K;               // input rows they look at
    const int item = (int)(blockIdx.x * 128 + threadIdx.x);
    if (item >= p.total)
        return;
    const int r1 = (int)fastdiv_apply((uint32_t)item, p.fd_c4), cw = item - r1 * p.c4;
    const int r2 = (int)fastdiv_apply((uint32_t)r1, p.fd_strips), strip = r1 - r2 * p.strips;
    const int n  = (int)fastdiv_apply((uint32_t)r2, p.fd_rg), oy = (r2 - n * p.row_groups) * R;
    const int c  = cw * 4;
    const int ox0 = strip * p.len, ox1 = min(p.OW, ox0 + p.len);

    const bool usable = *p.usable != 0;    // (asked below, behind the loads that a usable layer waits for as well)
    int wc[K][4], w5[K == 5 ? K : 1][4];
#pragma unroll
    for (int k = 0; k < K; k++)
    {
        const int4 t = __ldg(p.wcol + k * p.c4 + cw);
        wc[k][0] = t.x; wc[k][1] = t.y; wc[k][2] = t.z; wc[k][3] = t.w;
        if (K == 5)
        {
            const int4 u = __ldg(p.wrow5 + k * p.c4 + cw);
            w5[K == 5 ? k : 0][0] = u.x; w5[K == 5 ? k : 0][1] = u.y; w5[K == 5 ? k : 0][2] = u.z; w5[K == 5 ? k : 0][3] = u.w;
        }
    }
    // the second row's weights, kept (the compiler would shift them again for every output)
    int wd[R == 2 ? K : 1][4];
    if (R == 2)
    {
#pragma unroll
        for (int k = 0; k < K; k++)
#pragma unroll
            for (int i = 0; i < 4; i++)
                asm volatile("shl.b32 %0, %1, 8;" : "=r"(wd[R == 2 ? k : 0][i]) : "r"(wc[k][i]));
    }
    int4 ra[4];
    int2 rb[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
    {
        ra[i] = __ldg(p.rec + (c + i) * 2);
        rb[i] = __ldg(reinterpret_cast<const int2*>(p.rec + (c + i) * 2 + 1));
    }

    if (!usable)
    {
        walk_general(p, K, S, FIX, n, oy, R, c, ox0, ox1);
        return;
    }

    // Rows and columns outside the image are the zero point.  An aligned word's load is predicated and leaves a register that
    // holds it already: a select after the load would wait for the load where it is asked for.
    const int8_t* const img = p.in + (int64_t)n * p.IH * p.IW * p.C + c;
    const int8_t* row[NR];
    bool row_in[NR];
#pragma unroll
    for (int r = 0; r < NR; r++)
    {
        const int y = oy * S - p.pad_t + r;
        row_in[r]   = (unsigned)y < (unsigned)p.IH;
        row[r]      = img + (int64_t)(row_in[r] ? y : 0) * p.IW * p.C;
    }
    auto fetch_column = [&](int x, uint32_t(&a)[NR]) {
        const bool in = (unsigned)x < (unsigned)p.IW;
        const int xo  = ALIGNED ? x * p.C : min(max(x, 0), p.IW - 1) * p.C;
#pragma unroll
        for (int r = 0; r < NR; r++)
        {
            const int8_t* at = row[r] + xo;
            if (ALIGNED)
            {
                uint32_t v = p.fill4;
                asm("{\n\t.reg .pred in;\n\tsetp.ne.s32 in, %2, 0;\n\t@in ld.global.nc.b32 %0, [%1];\n\t}" : "+r"(v) : "l"(at), "r"((int)(in && row_in[r])));
                a[r] = v;
            }
            else
            {
                const int sh      = (int)(reinterpret_cast<uintptr_t>(at) & 3);
                const int8_t* lo  = at - sh;
                const uint32_t w0 = *reinterpret_cast<const uint32_t*>(lo);
                const uint32_t w1 = sh && lo + 4 < p.in_end ? *reinterpret_cast<const uint32_t*>(lo + 4) : 0u;
                a[r] = in && row_in[r] ? __funnelshift_r(w0, w1, 8 * sh) : p.fill4;
            }
        }
    };
    // column x of the window's rows: t[0..3] one word per channel (rows 0..3), t[4] the fifth row's four channels
    struct Column
    {
        uint32_t t[K == 5 ? 5 : 4];
    };
    auto column = [&](const uint32_t(&a)[NR], Column& q) {
        const uint32_t lo01 = __byte_perm(a[0], a[1], 0x5140), hi01 = __byte_perm(a[0], a[1], 0x7362);
        if (NR == 3)
        {
            // (the fourth byte meets a zero weight)
            q.t[0] = __byte_perm(lo01, a[2], 0x4410);
            q.t[1] = __byte_perm(lo01, a[2], 0x5532);
            q.t[2] = __byte_perm(hi01, a[2], 0x6610);
            q.t[3] = __byte_perm(hi01, a[2], 0x7732);
        }
        else
        {
            const uint32_t a3   = a[NR > 3 ? 3 : 0];
            const uint32_t lo23 = __byte_perm(a[2], a3, 0x5140), hi23 = __byte_perm(a[2], a3, 0x7362);
            q.t[0] = __byte_perm(lo01, lo23, 0x5410);
            q.t[1] = __byte_perm(lo01, lo23, 0x7632);
            q.t[2] = __byte_perm(hi01, hi23, 0x5410);
            q.t[3] = __byte_perm(hi01, hi23, 0x7632);
        }
        if (K == 5)
            q.t[K == 5 ? 4 : 0] = a[NR > 4 ? 4 : 0];
    };
    const bool narrow  = p.clamp_lo > -128 || p.clamp_hi < 127;
    const uint32_t lo4 = (uint32_t)(p.clamp_lo & 0xff) * 0x01010101u, hi4 = (uint32_t)(p.clamp_hi & 0xff) * 0x01010101u;
    int8_t* o0         = p.out + (((int64_t)n * p.OH + oy) * p.OW + ox0) * p.C + c;
    const int64_t o_row = (int64_t)p.OW * p.C;
    const bool two     = R == 2 && oy + 1 < p.OH;
    auto emit = [&](int8_t* o, const int (&acc)[4]) {
        uint32_t w;
        int z[4];
#pragma unroll
        for (int i = 0; i < 4; i++)
            z[i] = rescale_rec_apply(acc[i], ra[i].x, ra[i].y, ra[i].z, ra[i].w, rb[i].x, rb[i].y, FIX);
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(z[3]), "r"(z[2]), "r"(0));
        asm("cvt.pack.sat.s8.s32.b32 %0, %1, %2, %3;" : "=r"(w) : "r"(z[1]), "r"(z[0]), "r"(w));
        if (narrow)
            w = __vmins4(__vmaxs4(w, lo4), hi4);
        if (ALIGNED)
            *reinterpret_cast<uint32_t*>(o) = w;
        else
        {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (c + i < p.C)
                    o[i] = (int8_t)(w >> (8 * i));
        }
    };

    // The last K columns, as a ring whose positions are compile-time constants: the loop over x is unrolled K times.  An
    // output's new columns are asked for K outputs before they are used; those that are put together from two words when they are used
    // (the words kept ahead would be twice as many registers: 80 shapes took 1.2 times as long, 10 x 15 x 11 x 361 5 x 5 stride 2
    // 14.4 us against 7.1).
    Column q[K];
    uint32_t raw[ALIGNED ? K * S : 1][NR], head[K - S][NR];
    int x = ox0 * S - p.pad_l;
#pragma unroll
    for (int k = 0; k < K - S; k++)
        fetch_column(x + k, head[k]);
    x += K - S;
    if (ALIGNED)
    {
#pragma unroll
        for (int k = 0; k < K * S; k++)
            fetch_column(x + k, raw[ALIGNED ? k : 0]);
    }
#pragma unroll
    for (int k = 0; k < K - S; k++)
        column(head[k], q[k]);
    for (int ox = ox0; ox < ox1; ox += K)
    {
#pragma unroll
        for (int u = 0; u < K; u++)
        {
            if (ox + u < ox1)
            {
                // ring position of window column k at output ox + u: (u S + k) mod K
#pragma unroll
                for (int s = 0; s < S; s++)
                {
                    if (!ALIGNED)
                        fetch_column(x + u * S + s, raw[0]);
                    column(raw[ALIGNED ? u * S + s : 0], q[(u * S + K - S + s) % K]);
                }
                if (ALIGNED && ox + u + K < ox1)
                {
#pragma unroll
                    for (int s = 0; s < S; s++)
                        fetch_column(x + (u + K) * S + s, raw[ALIGNED ? u * S + s : 0]);
                }
                int acc[4], acc2[4];
#pragma unroll
                for (int i = 0; i < 4; i++)
                    acc[i] = acc2[i] = 0;
#pragma unroll
                for (int k = 0; k < K; k++)
                {
                    const Column& w = q[(u * S + k) % K];
#pragma unroll
                    for (int i = 0; i < 4; i++)
                    {
                        acc[i] = __dp4a((int)w.t[i], wc[k][i], acc[i]);
                        if (K == 5)
                            acc[i] = __dp4a((int)w.t[K == 5 ? 4 : 0], w5[K == 5 ? k : 0][i], acc[i]);
                        if (R == 2)
                            acc2[i] = __dp4a((int)w.t[i], wd[R == 2 ? k : 0][i], acc2[i]);
                    }
                }
                emit(o0, acc);
                if (two)
                    emit(o0 + o_row, acc2);
                o0 += p.C;
            }
        }
        x += K * S;
    }
}

// Weights [K][K][C] packed by window columns, RESCALE records; one thread per channel (of C rounded up to four).
__global__ void depthwise_pack_kernel(const int8_t* __restrict__ w, const int32_t* __restrict__ bias, int bias_n, int C, int C4, int K, int32_t in_zp,
                                      const int32_t* __restrict__ mult, const int8_t* __restrict__ shift, int per_channel, int double_round,
                                      int32_t out_zp, int32_t* __restrict__ wcol, int32_t* __restrict__ wrow5, int32_t* __restrict__ rec,
                                      int32_t* __restrict__ corr, int* all_ok)
{
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C4)
        return;
    int32_t sum = 0;
    for (int kx = 0; kx < K; kx++)
    {
        uint32_t col = 0, five = 0;
        for (int ky = 0; ky < K && c < C; ky++)
        {
            const int v = w[(ky * K + kx) * C + c];
            sum += v;
            if (ky < 4)
                col |= (uint32_t)(v & 0xff) << (8 * ky);
            else
                five = (uint32_t)(v & 0xff) << (8 * (c & 3));
        }
        wcol[kx * C4 + c] = (int32_t)col;
        if (K == 5)
            wrow5[kx * C4 + c] = (int32_t)five;
    }
    int32_t r8[8] = { 0, 0, 0, 0, 0, 0, 0, 1 };
    if (c < C)
    {
        const int32_t b    = bias[bias_n == 1 ? 0 : c];
        const int64_t vmax = (int64_t)K * K * 255 * 128 + (b < 0 ? -(int64_t)b : (int64_t)b);
        rescale_rec_build(mult[per_channel ? c : 0], (int32_t)shift[per_channel ? c : 0], double_round, out_zp, b - in_zp * sum, vmax, r8);
        if (r8[7] == 0)
            *all_ok = 0;
        corr[c] = (int32_t)((uint32_t)b - (uint32_t)in_zp * (uint32_t)sum);
    }
    for (int i = 0; i < 8; i++)
        rec[c * 8 + i] = r8[i];
}

size_t pack_words(int C, int K)
{
    const size_t C4 = (size_t)((C + 3) & ~3);
    return C4 * (size_t)(K == 5 ? 2 * K : K) + C4 * 9;    // weights, records, corrections
}

}    // namespace

bool depthwise_slide_supported(const DepthwiseI8Problem& q)
{
    // 32-bit item numbers and offsets inside a row; two rows of a window never wrap around an image smaller than it
    return (q.K == 3 || q.K == 5) && (q.S == 1 || q.S == 2) && (int64_t)q.N * q.OH * q.OW * ((q.C + 3) / 4) < (1LL << 31) &&
           (int64_t)q.OW * 2 * q.C < (1LL << 31) && (int64_t)q.IW * q.C < (1LL << 31);
}

size_t depthwise_slide_pack_bytes(int C, int K)
{
    return pack_words(C, K) * 4 + 64;
}

size_t depthwise_slide_flag_offset(int C, int K)
{
    return pack_words(C, K) * 4;
}

tb200_status depthwise_slide_pack(tb200_ctx* ctx, const DepthwiseI8Problem& q, void* block)
{
    const int C4  = (q.C + 3) & ~3;
    int32_t* wcol = reinterpret_cast<int32_t*>(block);
    int32_t* five = wcol + C4 * q.K;
    int32_t* rec  = five + (q.K == 5 ? C4 * q.K : 0);
    int32_t* corr = rec + C4 * 8;
    int* flag     = reinterpret_cast<int*>(corr + C4);
    TB200_CUDA_CHECK(ctx, cudaMemsetAsync(flag, 1, sizeof(int), ctx->stream));
    depthwise_pack_kernel<<<(C4 + 127) / 128, 128, 0, ctx->stream>>>(q.w, q.bias, q.bias_n, q.C, C4, q.K, q.in_zp, q.mult, q.shift, q.per_channel,
                                                                    q.double_round, q.out_zp, wcol, five, rec, corr, flag);
    return post_launch(ctx, "depthwise_pack");
}

// Pieces of a row: a thread is a chain of columns, so a call takes a chain's length times the waves of blocks, or the time its
// instructions take where that is longer.  SM cycles: 350 per column of a 3 x 3 chain, 600 of a 5 x 5
// one, 1500 to 2500 for the first output; 5 per 32 outputs.  32 x 56 x 56 x 144, 3 x 3, by outputs per piece: 56 24.3 us, 28
// and 14 18.4, 19, 12 and 8 20.5, 5 26.6.  Tried is each piece count that gives another length; on rows of more than 256 outputs a
// quarter more pieces at a time, some twenty counts (all of them took the host 5 us for 4801 outputs).  Returns how many.
static int dw_pieces(int64_t lines, int OW, int K, int S, int R, int num_sms, int blocks_per_sm, int* best_len, int* best_strips)
{
    const int64_t room = (int64_t)num_sms * blocks_per_sm;
    double best        = 0;
    int tried          = 0;
    for (int strips = std::max(1, OW / 256), next; strips <= std::max(1, OW / 2); strips = next, tried++)
    {
        const int len = (OW + strips - 1) / strips;
        next          = len > 1 ? (OW + len - 2) / (len - 1) : OW + 1;
        if (OW > 256)
            next = std::max(next, strips + strips / 4);
        const int64_t threads = lines * ((OW + len - 1) / len);
        const double waves    = (double)((threads + 128 * room - 1) / (128 * room));
        const double chain    = K == 3 ? (len + 3 - S) * 350.0 + 2500 : (len + 5 - S) * 600.0 + 1500;
        const double work     = (double)threads / 32 / num_sms * (len + 3) * R * 4 * 5;
        const double cost     = std::max(waves * chain, work);
        if (best == 0 || cost < best * 0.99)
        {
            best         = cost;
            *best_len    = len;
            *best_strips = (OW + len - 1) / len;
        }
    }
    return tried;
}

tb200_status depthwise_slide_launch(tb200_ctx* ctx, const DepthwiseI8Problem& q, const void* block, const char* name)
{
    const int C4 = (q.C + 3) & ~3;
    DwSlideParams p;
    memset(&p, 0, sizeof(p));
    p.in     = q.in;
    p.in_end = q.in + (int64_t)q.N * q.IH * q.IW * q.C;
    p.out    = q.out;
    p.wcol   = reinterpret_cast<const int4*>(block);
    p.wrow5  = p.wcol + C4 / 4 * q.K;
    p.rec    = p.wrow5 + (q.K == 5 ? C4 / 4 * q.K : 0);
    p.corr   = reinterpret_cast<const int32_t*>(p.rec + C4 * 2);
    p.usable = reinterpret_cast<const int*>(p.corr + C4);
    p.w = q.w; p.mult = q.mult; p.shift = q.shift; p.per_channel = q.per_channel; p.out_zp = q.out_zp; p.status = ctx->d_status;
    p.N = q.N; p.IH = q.IH; p.IW = q.IW; p.C = q.C; p.OH = q.OH; p.OW = q.OW; p.pad_t = q.pad_t; p.pad_l = q.pad_l;
    p.c4         = C4 / 4;
    const int R  = q.K == 3 && q.S == 1 ? 2 : 1;
    p.row_groups = (q.OH + R - 1) / R;
    const bool al = q.C % 4 == 0 && ((reinterpret_cast<uintptr_t>(q.in) | reinterpret_cast<uintptr_t>(q.out)) & 3) == 0;
    typedef void (*Kern)(const DwSlideParams);
    static const Kern kerns[16] = {
#define TB200_DW(KK, SS)                                                                                                     \
    depthwise_slide_i8_kernel<KK, SS, false, false>, depthwise_slide_i8_kernel<KK, SS, false, true>,                         \
        depthwise_slide_i8_kernel<KK, SS, true, false>, depthwise_slide_i8_kernel<KK, SS, true, true>
        TB200_DW(3, 1), TB200_DW(3, 2), TB200_DW(5, 1), TB200_DW(5, 2)
#undef TB200_DW
    };
    const int which = (q.K == 5 ? 8 : 0) + (q.S == 2 ? 4 : 0) + (al ? 2 : 0) + (q.double_round ? 1 : 0);
    if (ctx->dw_blocks[which] == 0)
    {
        int occ = 0;
        TB200_CUDA_CHECK(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kerns[which], 128, 0));
        ctx->dw_blocks[which] = std::max(1, occ);
    }
    const int64_t lines = (int64_t)q.N * p.row_groups * p.c4;
    bool known          = false;
    if (!ctx->dw_memo)
        ctx->dw_memo.reset(new SizeMemo<DwPieces>());
    auto& memo = ctx->dw_memo->at(lines, q.OW, which, &known);
    if (!known)
        dw_pieces(lines, q.OW, q.K, q.S, R, ctx->num_sms, ctx->dw_blocks[which], &memo.value.len, &memo.value.strips);
    p.len    = memo.value.len;
    p.strips = memo.value.strips;
    fastdiv_make((uint32_t)p.c4, p.fd_c4);
    fastdiv_make((uint32_t)p.strips, p.fd_strips);
    fastdiv_make((uint32_t)p.row_groups, p.fd_rg);
    p.total    = (int)(lines * p.strips);
    p.fill4    = (uint32_t)(q.in_zp & 0xff) * 0x01010101u;
    p.clamp_lo = q.clamp_lo;
    p.clamp_hi = q.clamp_hi;
    kerns[which]<<<(p.total + 127) / 128, 128, 0, ctx->stream>>>(p);
    return post_launch(ctx, name);
}

}    // namespace tb200
