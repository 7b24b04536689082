// fp32 batched MATMUL and CONV2D on CUDA cores (deep and large ones go to sgemm_split.cu where that is estimated to be
// faster): FFMA only, no TF32, so every product and sum is an IEEE fp32 operation
// and the result stays inside the reference's dot-product error bound.
//
// One tiled kernel for both.  A block owns a BM x BN tile of the output and walks K sixteen elements at a time through a
// ring of shared-memory stages filled with asynchronous copies:
//   * A (MATMUL: [N,H,C]; CONV2D: the input, gathered tap by tap) is read along K and keeps that order, As[row][k]: a
//     thread takes four K elements of each of its rows with one 128-bit read.  Copies are 16 bytes wide where C (the
//     channel count) is a multiple of four and 4 bytes wide otherwise; a tap outside the image, a row past the last
//     pixel and a K tail are all a copy of zero bytes (zero fill).  (A first version transposed A with 4-byte copies: their
//     address and bounds arithmetic, once per element, took a quarter of a convolution's instructions.)
//   * B ([N,C,W], or the CONV2D weights re-ordered once to [K][OC]) keeps its layout: 16-byte copies where its rows allow.
// A warp covers a (4 TM) x (8 TN) part of the tile, four lanes down and eight across: the rows' pitch of 20 words and the
// 128 contiguous bytes of B make both operands' 128-bit reads one shared-memory wavefront each.  Accumulators are pairs of
// neighbouring columns for the packed multiply-add (fma.rn.f32x2: two IEEE operations).
// Problems with few tiles split K over the CTAs of a cluster; the partial tiles are added in rank order through
// distributed shared memory, so a result does not depend on timing.
#include <algorithm>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "common.h"

namespace tb200
{
namespace
{

constexpr int BK = 16;

struct SgemmParams
{
    const float* a;
    const float* b;
    float* out;
    int M, N, K;             // rows, columns, depth of one batch
    int64_t a_batch, b_batch, o_batch;
    int ldb;                 // elements between rows of B
    int tiles_m, tiles_n;
    int k_per_split;         // K range of one CTA of a cluster, a multiple of BK
    // CONV2D: A is gathered from an NHWC input
    int IH, IW, IC, OH, OW, KH, KW, pad_t, pad_l, sy, sx, dy, dx;
    int in_sn, in_sh, in_sw;
    int padded;              // some window may leave the image
    const float* bias;
    int bias_n;              // CONV2D bias length (OC or 1), 0 = none
    int has_clamp;
    float clamp_lo, clamp_hi;
};

// A tap outside the image is a zero that is multiplied like any other, where the reference skips it
// (reference_model/src/ops/tensor_ops.cpp:828-873).  They differ where a weight is infinite or NaN: zero times it is NaN, and
// only then.  A NaN of a window that leaves the image is summed again here, over the taps inside.
__device__ __noinline__ float sum_inside(const SgemmParams& p, int m, int n)
{
    const int ox = m % p.OW, q = m / p.OW, oy = q % p.OH;
    const int y0 = oy * p.sy - p.pad_t, x0 = ox * p.sx - p.pad_l;
    if (y0 >= 0 && x0 >= 0 && y0 + (p.KH - 1) * p.dy < p.IH && x0 + (p.KW - 1) * p.dx < p.IW)
        return __uint_as_float(0x7fffffffu);    // every tap is inside: the NaN stands
    const float* const in = p.a + (int64_t)(q / p.OH) * p.in_sn;
    float sum = 0.f;
    for (int ky = 0; ky < p.KH; ky++)
        for (int kx = 0; kx < p.KW; kx++)
        {
            const int y = y0 + ky * p.dy, x = x0 + kx * p.dx;
            if ((unsigned)y >= (unsigned)p.IH || (unsigned)x >= (unsigned)p.IW)
                continue;
            for (int c = 0; c < p.IC; c++)
                sum = fmaf(in[(int64_t)y * p.in_sh + (int64_t)x * p.in_sw + c], p.b[((int64_t)(ky * p.KW + kx) * p.IC + c) * p.ldb + n], sum);
        }
    return sum;
}

// asynchronous copy of RUN floats, or zero fill
template <int RUN>
__device__ __forceinline__ void cp(uint32_t dst, const float* src, bool inside)
{
    if (RUN == 4)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(inside ? 16 : 0) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(inside ? 4 : 0) : "memory");
}

template <int BM, int BN, int TM, int TN, int ST>
struct SgemmShape
{
    static constexpr int kWarpsM  = BM / (4 * TM), kWarpsN = BN / (8 * TN);
    static constexpr int kThreads = 32 * kWarpsM * kWarpsN;
    static constexpr int kAPitch  = BK + 4;    // rows 16-byte aligned, four neighbouring rows in different banks
    static constexpr int kBOff    = BM * kAPitch, kStage = kBOff + BK * BN;
    static constexpr int kFloats  = ST * kStage > BM * BN ? ST * kStage : BM * BN;    // stages, later a partial tile
    static constexpr int kSmem    = kFloats * 4 + BM * 8;
};

// CONV: A is gathered from a convolution's input.  AVEC, BVEC: runs of four elements of A along K, of B along its rows, are
// whole aligned 16-byte pieces.
template <int BM, int BN, int TM, int TN, int ST, int OCC, bool CONV, bool AVEC, bool BVEC>
__global__ void __launch_bounds__(SgemmShape<BM, BN, TM, TN, ST>::kThreads, OCC) sgemm_f32_kernel(const __grid_constant__ SgemmParams p)
{
    using S = SgemmShape<BM, BN, TM, TN, ST>;
    constexpr int T = S::kThreads;
    constexpr int kRun  = AVEC ? 4 : 1;            // K elements per copy of A
    constexpr int kRowStep = T / (BK / kRun);      // rows the block copies at a time
    constexpr int kRowCopies = BM >= kRowStep ? BM / kRowStep : 1;    // (a tile shorter than that leaves threads idle)
    static_assert((BM % kRowStep == 0 || BM < kRowStep) && (BK * BN / 4) % T == 0, "copies divide evenly over the block");
    extern __shared__ __align__(16) float smem[];
    int2* const rows = reinterpret_cast<int2*>(smem + S::kFloats);    // CONV: {element offset of the row's window, iy0 | ix0}

    namespace cg      = cooperative_groups;
    const int splits  = (int)cg::this_cluster().num_blocks();
    const int rank    = splits > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int tile    = (int)(blockIdx.x / (unsigned)splits);
    const int per     = p.tiles_m * p.tiles_n;
    const int batch   = tile / per;
    const int rem     = tile - batch * per;
    const int m0 = (rem / p.tiles_n) * BM, n0 = (rem % p.tiles_n) * BN;
    const float* const A = p.a + batch * p.a_batch;
    const float* const B = p.b + batch * p.b_batch;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (CONV)
    {
        for (int r = tid; r < BM; r += T)
        {
            const int m = m0 + r;
            int2 v      = make_int2(0, (int)0x80008000);    // a row past the last pixel: every tap is outside
            if (m < p.M)
            {
                const int ox = m % p.OW, q = m / p.OW;
                const int oy = q % p.OH, n = q / p.OH;
                const int iy0 = oy * p.sy - p.pad_t, ix0 = ox * p.sx - p.pad_l;
                v.x = n * p.in_sn + iy0 * p.in_sh + ix0 * p.in_sw;
                v.y = (int)(((uint32_t)iy0 << 16) | ((uint32_t)ix0 & 0xffffu));
            }
            rows[r] = v;
        }
        __syncthreads();
    }

    // this thread's copies: K elements ak .. ak + kRun - 1 of the A stage's rows ar, ar + kRowStep, ..., and its share of B
    const int ak = tid % (BK / kRun) * kRun, ar = tid / (BK / kRun);
    const int k_lo = rank * p.k_per_split;
    const int k_hi = min(p.K, k_lo + p.k_per_split);
    const int nk   = max(0, (k_hi - k_lo + BK - 1) / BK);
    int ka = k_lo + ak;                    // running K index of this thread's A copies
    int ic = 0, ky = 0, kx = 0;            // CONV: its channel and tap
    if (CONV)
    {
        const int tap = ka / p.IC;
        ic = ka - tap * p.IC;
        ky = tap / p.KW;
        kx = tap - ky * p.KW;
    }
    const uint32_t s0 = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    auto load_stage = [&](int kt, int st) {
        const uint32_t sa = s0 + (uint32_t)((st * S::kStage + ar * S::kAPitch + ak) * 4);
        const bool kin = ka < k_hi;
        if (CONV)
        {
            const int y = ky * p.dy, x = kx * p.dx;
            const int off = y * p.in_sh + x * p.in_sw + ic;
#pragma unroll
            for (int i = 0; i < kRowCopies; i++)
            {
                if (BM < kRowStep && ar >= BM)
                    break;
                const int2 r = rows[ar + i * kRowStep];
                const bool inside = kin && (unsigned)((r.y >> 16) + y) < (unsigned)p.IH && (unsigned)((int)(short)r.y + x) < (unsigned)p.IW;
                cp<kRun>(sa + i * kRowStep * S::kAPitch * 4, inside ? A + (r.x + off) : A, inside);
            }
            ic += BK;
            while (ic >= p.IC)
            {
                ic -= p.IC;
                if (++kx == p.KW)
                {
                    kx = 0;
                    ky++;
                }
            }
        }
        else
        {
            const float* src = A + (int64_t)(m0 + ar) * p.K + ka;
#pragma unroll
            for (int i = 0; i < kRowCopies; i++)
            {
                if (BM < kRowStep && ar >= BM)
                    break;
                const bool inside = kin && m0 + ar + i * kRowStep < p.M;
                cp<kRun>(sa + i * kRowStep * S::kAPitch * 4, inside ? src + (int64_t)i * kRowStep * p.K : A, inside);
            }
        }
        ka += BK;
        const uint32_t sb = s0 + (uint32_t)((st * S::kStage + S::kBOff) * 4);
        const int kb0     = k_lo + kt * BK;
        if (BVEC)
        {
#pragma unroll
            for (int i = 0; i < BK * BN / 4 / T; i++)
            {
                const int e = tid + i * T, k = kb0 + e / (BN / 4), n = n0 + (e % (BN / 4)) * 4;
                const bool inside = k < k_hi && n < p.N;
                cp<4>(sb + (uint32_t)e * 16, inside ? B + (int64_t)k * p.ldb + n : B, inside);
            }
        }
        else
        {
#pragma unroll
            for (int i = 0; i < BK * BN / T; i++)
            {
                const int e = tid + i * T, k = kb0 + e / BN, n = n0 + e % BN;
                const bool inside = k < k_hi && n < p.N;
                cp<1>(sb + (uint32_t)e * 4, inside ? B + (int64_t)k * p.ldb + n : B, inside);
            }
        }
    };

    float2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int j = 0; j < TN / 2; j++)
            acc[i][j] = make_float2(0.f, 0.f);

#pragma unroll
    for (int s = 0; s < ST - 1; s++)
    {
        if (s < nk)
            load_stage(s, s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int wm = (warp / S::kWarpsN) * 4 * TM, wn = (warp % S::kWarpsN) * 8 * TN;
    const int ly = lane >> 3, lx = lane & 7;
    int rd = 0, wr = ST - 1;
    for (int kt = 0; kt < nk; kt++)
    {
        asm volatile("cp.async.wait_group %0;" ::"n"(ST - 2) : "memory");
        __syncthreads();    // the stage has landed for everyone, and everyone is done with the stage filled next
        if (kt + ST - 1 < nk)
            load_stage(kt + ST - 1, wr);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* as = smem + rd * S::kStage + (wm + ly) * S::kAPitch;
        const float* bs = smem + rd * S::kStage + S::kBOff + wn + lx * 4;
#pragma unroll
        for (int kq = 0; kq < BK; kq += 4)
        {
            float4 a4[TM];    // rows wm + ly, wm + ly + 4, ...
#pragma unroll
            for (int i = 0; i < TM; i++)
                a4[i] = *reinterpret_cast<const float4*>(as + i * 4 * S::kAPitch + kq);
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
            {
                float2 bv[TN / 2];
#pragma unroll
                for (int g = 0; g < TN / 4; g++)
                {
                    const float4 t = *reinterpret_cast<const float4*>(bs + (kq + kk) * BN + g * 32);
                    bv[2 * g] = make_float2(t.x, t.y); bv[2 * g + 1] = make_float2(t.z, t.w);
                }
#pragma unroll
                for (int i = 0; i < TM; i++)
                {
                    const float a   = kk == 0 ? a4[i].x : kk == 1 ? a4[i].y : kk == 2 ? a4[i].z : a4[i].w;
                    const float2 a2 = make_float2(a, a);
#pragma unroll
                    for (int j = 0; j < TN / 2; j++)
                        acc[i][j] = __ffma2_rn(a2, bv[j], acc[i][j]);
                }
            }
        }
        rd = rd + 1 == ST ? 0 : rd + 1;
        wr = wr + 1 == ST ? 0 : wr + 1;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");

    float* const O   = p.out + batch * p.o_batch;
    const bool ovec  = (p.N & 3) == 0 && (reinterpret_cast<uintptr_t>(O) & 15) == 0;
    auto store4 = [&](int m, int n, float4 v) {
        if (m >= p.M || n >= p.N)
            return;
        float f[4] = { v.x, v.y, v.z, v.w };
        if (CONV && p.padded && (isnan(v.x) || isnan(v.y) || isnan(v.z) || isnan(v.w)))
            for (int j = 0; j < 4; j++)
            {
                const float x = j == 0 ? f[0] : j == 1 ? f[1] : j == 2 ? f[2] : f[3];
                if (isnan(x) && n + j < p.N)
                {
                    const float s = sum_inside(p, m, n + j);
                    f[0] = j == 0 ? s : f[0]; f[1] = j == 1 ? s : f[1]; f[2] = j == 2 ? s : f[2]; f[3] = j == 3 ? s : f[3];
                }
            }
        if (CONV)
        {
#pragma unroll
            for (int j = 0; j < 4; j++)
            {
                if (p.bias_n)
                    f[j] = (p.bias_n == 1 ? __ldg(p.bias) : n + j < p.N ? __ldg(p.bias + n + j) : 0.f) + f[j];
                if (p.has_clamp)
                {
                    f[j] = (f[j] < p.clamp_lo) ? p.clamp_lo : f[j];
                    f[j] = (f[j] > p.clamp_hi) ? p.clamp_hi : f[j];
                }
            }
        }
        float* o = O + (int64_t)m * p.N + n;
        if (ovec)
            *reinterpret_cast<float4*>(o) = make_float4(f[0], f[1], f[2], f[3]);
        else
        {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (n + j < p.N)
                    o[j] = f[j];
        }
    };
    if (splits == 1)
    {
#pragma unroll
        for (int i = 0; i < TM; i++)
#pragma unroll
            for (int g = 0; g < TN / 4; g++)
                store4(m0 + wm + i * 4 + ly, n0 + wn + g * 32 + lx * 4,
                       make_float4(acc[i][2 * g].x, acc[i][2 * g].y, acc[i][2 * g + 1].x, acc[i][2 * g + 1].y));
        return;
    }
    // partial tiles meet in shared memory: every CTA adds up its share of the tile's float4s over all ranks, in rank order
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TM; i++)
#pragma unroll
        for (int g = 0; g < TN / 4; g++)
            *reinterpret_cast<float4*>(smem + (wm + i * 4 + ly) * BN + wn + g * 32 + lx * 4) =
                make_float4(acc[i][2 * g].x, acc[i][2 * g].y, acc[i][2 * g + 1].x, acc[i][2 * g + 1].y);
    auto cluster = cg::this_cluster();
    cluster.sync();
    for (int e = rank * T + tid; e < BM * BN / 4; e += splits * T)
    {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int r = 0; r < splits; r++)
        {
            const float4 v = *reinterpret_cast<const float4*>(cluster.map_shared_rank(smem, r) + e * 4);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        store4(m0 + e / (BN / 4), n0 + (e % (BN / 4)) * 4, sum);
    }
    cluster.sync();    // nobody leaves while another CTA may still read its shared memory
}

// Tile configurations and what they measured.  `step`: cycles one K step of a tile takes from a full SM, in units of the
// 128 multiply-adds per cycle an SM can start (1 = peak): packed multiply-adds are bound by register operand bandwidth, and
// wide thread tiles reuse more operands.  Over 32 x 1024 x 4096 x 1024: 128 x 128 with 8 x 16 accumulators per thread 57.6
// TFLOP/s (8 x 8: 52.6, scalar multiply-adds: 48), 64 x 64 50.0, 128 x 32 48.9, 32 x 64 42.2, 16 x 128 39.3.
// `chain`: cycles a K step takes when a CTA has its SM to itself (1 x 64 x 4096 x 64).
struct SgemmConfig
{
    int bm, bn, tm, tn, stages, occ;
    double step, chain;
};
constexpr SgemmConfig kConfigs[] = {
    { 128, 128, 8, 16, 3, 2, 1.29, 2940.0 },
    { 64, 64, 8, 4, 4, 4, 1.48, 1060.0 },
    { 32, 64, 4, 4, 4, 4, 1.76, 710.0 },
    { 16, 128, 4, 4, 4, 4, 1.89, 770.0 },
    { 128, 32, 8, 4, 4, 4, 1.52, 1085.0 },
};
constexpr int kNumConfigs = (int)(sizeof(kConfigs) / sizeof(kConfigs[0]));

template <int I, bool CONV, bool VEC>
tb200_status launch_config(tb200_ctx* ctx, const SgemmParams& p, int splits, int64_t tiles)
{
    constexpr SgemmConfig c = kConfigs[I];
    using S   = SgemmShape<c.bm, c.bn, c.tm, c.tn, c.stages>;
    auto kern = sgemm_f32_kernel<c.bm, c.bn, c.tm, c.tn, c.stages, c.occ, CONV, VEC, CONV || VEC>;
    const tb200_status st = raise_smem_limit(ctx, 32 + I * 4 + (CONV ? 2 : 0) + (VEC ? 1 : 0), reinterpret_cast<const void*>(kern), S::kSmem);
    if (st != TB200_OK)
        return st;
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim          = dim3((unsigned)(tiles * splits));
    cfg.blockDim         = dim3(S::kThreads);
    cfg.dynamicSmemBytes = S::kSmem;
    cfg.stream           = ctx->stream;
    cudaLaunchAttribute at[1];
    at[0].id               = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)splits;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs    = at;
    cfg.numAttrs = splits > 1 ? 1 : 0;
    timer_begin(ctx);
    cudaLaunchKernelEx(&cfg, kern, p);
    timer_end(ctx);
    return TB200_OK;
}

// Tile size and split of K: the pair with the smallest estimated time, which is the larger of the multiply-adds of the
// fullest SM and the serial chain of K steps of one CTA, plus what starting a CTA (and meeting the cluster) costs.
struct SgemmPlan
{
    int config, splits;
    double cost;    // SM cycles
};

SgemmPlan choose(const tb200_ctx* ctx, const SgemmParams& p, int batches)
{
    int best = 0, best_split = 1;
    double best_cost = 0;
    const int steps  = std::max(1, (p.K + BK - 1) / BK);
    for (int i = 0; i < kNumConfigs; i++)
    {
        const SgemmConfig& c = kConfigs[i];
        const int64_t tiles  = (int64_t)batches * ((p.M + c.bm - 1) / c.bm) * ((p.N + c.bn - 1) / c.bn);
        for (int s = 1; s <= 8 && (s == 1 || steps >= 4 * s); s *= 2)
        {
            const int64_t ctas   = tiles * s;
            const double per_sm  = (double)((ctas + ctx->num_sms - 1) / ctx->num_sms);
            const double waves   = (double)((ctas + (int64_t)ctx->num_sms * c.occ - 1) / ((int64_t)ctx->num_sms * c.occ));
            const double ksteps  = (double)((steps + s - 1) / s);
            const double work    = per_sm * ksteps * c.step * (c.bm * c.bn * BK / 128.0);
            const double cost    = std::max(work, waves * ksteps * c.chain) + waves * 1500.0 + (s > 1 ? 1500.0 : 0.0);
            if (best_cost == 0 || cost < best_cost)
            {
                best_cost  = cost;
                best       = i;
                best_split = s;
            }
        }
    }
    return { best, best_split, best_cost };
}

template <bool CONV, bool VEC>
tb200_status launch_any(tb200_ctx* ctx, SgemmParams p, int batches, const SgemmPlan& plan)
{
    const SgemmConfig& c = kConfigs[plan.config];
    const int best_split = plan.splits, steps = std::max(1, (p.K + BK - 1) / BK);
    p.tiles_m = (p.M + c.bm - 1) / c.bm;
    p.tiles_n = (p.N + c.bn - 1) / c.bn;
    p.k_per_split = (steps + best_split - 1) / best_split * BK;
    const int64_t tiles = (int64_t)batches * p.tiles_m * p.tiles_n;
    if (tiles * best_split >= (1LL << 31))
        return fail(ctx, TB200_ERROR, "fp32 product with too many tiles");
    switch (plan.config)
    {
        case 0: return launch_config<0, CONV, VEC>(ctx, p, best_split, tiles);
        case 1: return launch_config<1, CONV, VEC>(ctx, p, best_split, tiles);
        case 2: return launch_config<2, CONV, VEC>(ctx, p, best_split, tiles);
        case 3: return launch_config<3, CONV, VEC>(ctx, p, best_split, tiles);
        default: return launch_config<4, CONV, VEC>(ctx, p, best_split, tiles);
    }
}

// CONV2D weights [OC][K] -> [K][ldb] (ldb = OC rounded up to four; the pad columns are zero), and whether they are all
// finite (see sum_inside(): layers whose weights are not are faster on a kernel that skips taps in the first place).
__global__ void transpose_weights_f32_kernel(const float* __restrict__ w, float* __restrict__ wt, int OC, int K, int ldb, int* all_finite)
{
    __shared__ float t[32][33];
    const int k0 = blockIdx.x * 32, o0 = blockIdx.y * 32;
    bool finite = true;
    for (int r = threadIdx.y; r < 32; r += 8)
    {
        const int oc = o0 + r, k = k0 + threadIdx.x;
        const float v = oc < OC && k < K ? w[(int64_t)oc * K + k] : 0.f;
        finite        = finite && isfinite(v);
        t[r][threadIdx.x] = v;
    }
    if (!finite)
        atomicExch(all_finite, 0);
    __syncthreads();
    for (int r = threadIdx.y; r < 32; r += 8)
    {
        const int oc = o0 + threadIdx.x, k = k0 + r;
        if (oc < ldb && k < K)
            wt[(int64_t)k * ldb + oc] = t[threadIdx.x][r];
    }
}

}    // namespace

tb200_status sgemm_f32_launch(tb200_ctx* ctx, const float* a, const float* b, float* out, int N, int H, int C, int W)
{
    SgemmParams p;
    memset(&p, 0, sizeof(p));
    p.a = a; p.b = b; p.out = out;
    p.M = H; p.N = W; p.K = C; p.ldb = W;
    p.a_batch = (int64_t)H * C; p.b_batch = (int64_t)C * W; p.o_batch = (int64_t)H * W;
    const SgemmPlan plan = choose(ctx, p, N);
    const double split   = sgemm_split_cost(ctx, N, H, W, C, false);
    if (split > 0 && split < plan.cost)
        return sgemm_split_launch(ctx, a, b, out, N, H, C, W);
    const bool vec = (W % 4) == 0 && (C % 4) == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15) == 0;
    const tb200_status st = vec ? launch_any<false, true>(ctx, p, N, plan) : launch_any<false, false>(ctx, p, N, plan);
    return st != TB200_OK ? st : post_launch(ctx, "sgemm_f32");
}

int conv_f32_ldb(int OC)
{
    return (OC + 3) & ~3;
}

tb200_status conv_f32_weights_launch(tb200_ctx* ctx, const float* w, float* wt, int OC, int K, int* all_finite)
{
    const int ldb = conv_f32_ldb(OC);
    TB200_CUDA_CHECK(ctx, cudaMemsetAsync(all_finite, 1, sizeof(int), ctx->stream));
    transpose_weights_f32_kernel<<<dim3((K + 31) / 32, (ldb + 31) / 32), dim3(32, 8), 0, ctx->stream>>>(w, wt, OC, K, ldb, all_finite);
    return post_launch(ctx, "conv_f32_weights");
}

tb200_status conv_f32_launch(tb200_ctx* ctx, const ConvF32Problem& q)
{
    SgemmParams p;
    memset(&p, 0, sizeof(p));
    p.a = q.in; p.b = q.wt; p.out = q.out;
    p.M = q.N * q.OH * q.OW; p.N = q.OC; p.K = q.KH * q.KW * q.IC; p.ldb = conv_f32_ldb(q.OC);
    p.IH = q.IH; p.IW = q.IW; p.IC = q.IC; p.OH = q.OH; p.OW = q.OW; p.KH = q.KH; p.KW = q.KW; p.padded = q.padded;
    p.pad_t = q.pad_t; p.pad_l = q.pad_l; p.sy = q.sy; p.sx = q.sx; p.dy = q.dy; p.dx = q.dx;
    p.in_sn = (int)q.in_sn; p.in_sh = (int)q.in_sh; p.in_sw = (int)q.in_sw;
    p.bias = q.bias; p.bias_n = q.bias_n;
    p.has_clamp = q.has_clamp; p.clamp_lo = q.clamp_lo; p.clamp_hi = q.clamp_hi;
    const SgemmPlan plan = choose(ctx, p, 1);
    const double split   = sgemm_split_cost(ctx, 1, p.M, p.N, p.K, true);
    if (split > 0 && split < plan.cost)
        return conv_f32_split_launch(ctx, q);
    const bool vec = (q.IC % 4) == 0 && ((q.in_sn | q.in_sh | q.in_sw) & 3) == 0 && (reinterpret_cast<uintptr_t>(q.in) & 15) == 0;
    const tb200_status st = vec ? launch_any<true, true>(ctx, p, 1, plan) : launch_any<true, false>(ctx, p, 1, plan);
    return st != TB200_OK ? st : post_launch(ctx, "conv_f32");
}

}    // namespace tb200
