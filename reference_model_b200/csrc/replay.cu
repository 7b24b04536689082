// Captured convolutions follow their constants.
//
// tc_conv_lean_kernel and conv_chan.cu's kernels run on RESCALE records that the host has seen usable (rescale_rec_build's
// static bound on the values).  An upload of multipliers, shifts, weights or biases rebuilds the records under a captured
// graph, which holds the launch, and the new ones may not be usable.  The host then exchanges that launch for
// conv_general_kernel, one thread per output with the RESCALE's own arithmetic, and back when the records are usable again.
// The fast kernels carry no trace of it: a verdict read by them and a branch to the general arithmetic behind their loops
// cost 0.1 to 0.5 us a launch (one image of the ResNet-shaped graph 267 us, then 275 to 280, in five forms of it).
#include <cuda_runtime.h>

#include "common.h"
#include "ptx_sm100.cuh"
#include "rescale_math.cuh"

namespace tb200
{

// Outputs one after the other, with every REQUIRE condition reported.  The grid is that of the launch it stands for.
__global__ void __launch_bounds__(576) conv_general_kernel(const __grid_constant__ ConvGeneral p)
{
    ptx::dep_launch_wait();
    const int64_t total = (int64_t)p.N * p.OH * p.OW * p.OC;
    bool bad            = false;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
    {
        const int ch    = (int)(i % p.OC);
        const int64_t r = i / p.OC;
        const int ox = (int)(r % p.OW), oy = (int)(r / p.OW % p.OH), n = (int)(r / p.OW / p.OH);
        // parity-split problems: batch index 2 n + parity holds the output columns 2 ox + parity of image n
        const int no = p.xpar ? n >> 1 : n, xo = p.xpar ? 2 * ox + (n & 1) : ox, wo = p.xpar ? p.out_ow : p.OW;
        if (xo >= wo)
            continue;
        const int iy0 = oy * p.stride_y - p.pad_t, ix0 = ox * p.stride_x - p.pad_l;
        int32_t acc = 0;
        int ky_lo = p.KH, ky_hi = 0, kx_lo = p.KW, kx_hi = 0;    // the taps inside the image
        for (int ky = 0; ky < p.KH; ky++)
            if ((unsigned)(iy0 + ky * p.dil_y) < (unsigned)p.IH)
            {
                ky_lo = min(ky_lo, ky);
                ky_hi = ky + 1;
            }
        for (int kx = 0; kx < p.KW; kx++)
            if ((unsigned)(ix0 + kx * p.dil_x) < (unsigned)p.IW)
            {
                kx_lo = min(kx_lo, kx);
                kx_hi = kx + 1;
            }
        for (int ky = ky_lo; ky < ky_hi; ky++)
            for (int kx = kx_lo; kx < kx_hi; kx++)
            {
                const int* x = reinterpret_cast<const int*>(p.a + n * p.a_stride_n + (iy0 + ky * p.dil_y) * p.a_stride_h + (ix0 + kx * p.dil_x) * p.a_stride_w);
                const int* w = reinterpret_cast<const int*>(p.w + (((int64_t)ch * p.KH + ky) * p.KW + kx) * p.IC);
                for (int c = 0; c < p.IC / 4; c++)
                    acc = __dp4a(x[c], w[c], acc);
            }
        int64_t cls = 0;
        if (p.classes)
        {
            if (ky_hi <= ky_lo || kx_hi <= kx_lo)    // no tap inside: every such rectangle leaves the same (the bias)
                ky_lo = ky_hi = kx_lo = kx_hi = 0;
            cls = ((ky_lo * (p.KH + 1) + ky_hi) * (p.KW + 1) + kx_lo) * (p.KW + 1) + kx_hi;
        }
        acc += p.corr[cls * p.corr_stride + ch];
        int32_t z        = rescale_general(acc, p.mult[ch], p.shift[ch], p.double_round != 0, p.out_zp, p.clamp_lo, p.clamp_hi, bad);
        const int64_t at = (((int64_t)no * p.OH + oy) * wo + xo) * p.OC + ch;
        if (p.join != nullptr)
        {
            const int ia = (z & 0xff) ^ 0x80, ib = (p.res[at] & 0xff) ^ 0x80;
            bad = bad || p.join[kJoinBadA + ia] != 0 || p.join[kJoinBadB + ib] != 0;
            z   = join_general(p.join[kJoinLutA + ia], p.join[kJoinLutB + ib], p.join[kJoinOutMult], p.join[kJoinOutShift], p.join[kJoinOutDouble] != 0,
                               p.join[kJoinOutZp], p.join_lo, p.join_hi, bad);
        }
        p.out[at] = (int8_t)z;
    }
    if (bad)
        atomicOr(p.status, TB200_DEV_UNPREDICTABLE);
}

void replay_note_launch(tb200_ctx* ctx, const TcProblem& q)
{
    if (!ctx->capturing)
        return;
    ReplaySwap s;
    s.verdict = q.rec_ok;
    ConvGeneral& g = s.general;
    g.a = reinterpret_cast<const int8_t*>(q.a);
    g.w = reinterpret_cast<const int8_t*>(q.b);
    g.a_stride_w = q.a_stride_w ? q.a_stride_w : (int64_t)q.IC;
    g.a_stride_h = q.a_stride_h ? q.a_stride_h : g.a_stride_w * q.IW;
    g.a_stride_n = q.a_stride_n ? q.a_stride_n : g.a_stride_h * q.IH;
    g.N = q.N; g.OH = q.OH; g.OW = q.OW; g.OC = q.OC; g.IH = q.IH; g.IW = q.IW; g.IC = q.IC; g.KH = q.KH; g.KW = q.KW;
    g.pad_t = q.pad_t; g.pad_l = q.pad_l; g.stride_y = q.stride_y; g.stride_x = q.stride_x; g.dil_y = q.dil_y; g.dil_x = q.dil_x;
    g.xpar = q.xpar; g.out_ow = q.out_ow_real;
    g.corr = q.corr; g.corr_stride = q.corr_stride; g.classes = q.corr_classes;
    g.mult = q.mult_pad; g.shift = q.shift_pad;
    g.double_round = q.double_round; g.out_zp = q.out_zp; g.clamp_lo = q.clamp_lo; g.clamp_hi = q.clamp_hi;
    g.join = q.join; g.res = reinterpret_cast<const int8_t*>(q.res); g.join_lo = q.join_lo; g.join_hi = q.join_hi;
    g.out    = reinterpret_cast<int8_t*>(q.out);
    g.status = ctx->d_status;
    // the launch just recorded is what the stream's next one will depend on
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    const cudaGraphNode_t* at  = nullptr;
    const cudaGraphEdgeData* edges = nullptr;
    size_t n = 0;
    cudaGraphNodeType type = cudaGraphNodeTypeEmpty;
    if (cudaStreamGetCaptureInfo_v3(ctx->stream, &st, nullptr, nullptr, &at, &edges, &n) == cudaSuccess && n == 1 &&
        cudaGraphNodeGetType(at[0], &type) == cudaSuccess && type == cudaGraphNodeTypeKernel)
        s.node = at[0];
    cudaGetLastError();
    ctx->capture_swaps.push_back(s);
}

tb200_status replay_follow(tb200_ctx* ctx, const void* block, size_t bytes)
{
    const char* lo = reinterpret_cast<const char*>(block);
    int usable     = -1;
    for (tb200_graph* g : ctx->graphs)
        for (ReplaySwap& s : g->swaps)
        {
            const char* v = reinterpret_cast<const char*>(s.verdict);
            if (v < lo || v >= lo + bytes)
                continue;
            if (usable < 0)    // one verdict per block
            {
                TB200_CUDA_CHECK(ctx, cudaMemcpyAsync(ctx->h_status, v, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
                TB200_CUDA_CHECK(ctx, cudaStreamSynchronize(ctx->stream));
                usable = *ctx->h_status != 0 ? 1 : 0;
            }
            if (s.swapped == (usable == 0))
                continue;
            s.swapped = usable == 0;
            cudaKernelNodeParams np;
            void* args[1] = { &s.general };
            cudaError_t e = s.node ? cudaGraphKernelNodeGetParams(s.node, &np) : cudaErrorInvalidValue;
            if (e == cudaSuccess && s.swapped)
            {
                np.func           = reinterpret_cast<void*>(&conv_general_kernel);
                np.sharedMemBytes = 0;
                np.kernelParams   = args;
                np.extra          = nullptr;
            }
            if (e == cudaSuccess)
                e = cudaGraphExecKernelNodeSetParams(g->exec, s.node, &np);
            s.stuck = e != cudaSuccess && s.swapped;
            cudaGetLastError();
        }
    return TB200_OK;
}

}    // namespace tb200
