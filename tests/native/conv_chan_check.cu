// The layouts of conv_chan.cu on the host, over random problems: one context that remembers what it worked out for sizes gives what a
// new one gives, and every layout fits its limits (shared memory, one wave of clusters, whole tiles).
#include <cstdio>
#include <random>

#include "../../reference_model_b200/csrc/conv_chan.cu"

namespace tb200
{
tb200_status post_launch(tb200_ctx*, const char*, int) { return TB200_OK; }
void timer_begin(tb200_ctx*) {}
void timer_end(tb200_ctx*) {}
tb200_status raise_smem_limit(tb200_ctx*, int, const void*, int) { return TB200_OK; }
void* tensor_map_encode_fn() { return nullptr; }
}    // namespace tb200

int main()
{
    using namespace tb200;
    std::mt19937 rng(7);
    auto pick = [&](int lo, int hi) { return lo + (int)(rng() % (unsigned)(hi - lo + 1)); };
    tb200_ctx one;
    one.max_smem_optin = 232448;
    long long taken = 0, split = 0, wrong = 0;
    TcProblem seen[512];
    for (int i = 0; i < 4000; i++)
    {
        TcProblem& q = seen[i % 512];
        if (i < 512 || i % 3 == 0)    // else: one of the earlier ones again
        {
            memset(&q, 0, sizeof(q));
            q.in_dtype = q.out_dtype = TB200_INT8;
            q.N = pick(1, 64); q.IH = q.OH = pick(1, 112); q.IW = q.OW = pick(1, 112);
            q.IC = 32 * pick(1, 16); q.OC = 32 * pick(1, 20);
            q.KH = q.KW = 1;    // a flat problem: no tap map is asked for, which the host has not
            q.stride_x = q.stride_y = q.dil_x = q.dil_y = 1;
            q.epi = TC_EPI_RESCALE; q.lean_ok = 1; q.clamp_lo = -128; q.clamp_hi = 127;
            const int32_t* some = reinterpret_cast<const int32_t*>(static_cast<uintptr_t>(256));
            q.rec = q.rec_ok = some; q.a = q.b = some; q.out = const_cast<int32_t*>(some);
            if (pick(0, 1))
                q.join = some;
        }
        tb200_ctx fresh;
        fresh.max_smem_optin = 232448;
        ChanPlan a, b;
        const bool ta = chan_plan(&one, q, &a), tb = chan_plan(&fresh, q, &b);
        if (ta != tb || (ta && (memcmp(&a.kp, &b.kp, sizeof(a.kp)) != 0 || a.grid != b.grid || a.smem_bytes != b.smem_bytes)))
            wrong++;
        if (!ta)
            continue;
        taken++;
        const int64_t pixels = (int64_t)q.N * q.OH * q.OW, pbs = (pixels + a.kp.px - 1) / a.kp.px;
        if (a.smem_bytes > 232448 - 1024 || a.kp.tiles != pbs * a.kp.cbs || a.grid < 1)
            wrong++;
        if (a.kp.split)
        {
            split++;
            if (a.grid > 148 || a.grid != a.kp.tiles * a.kp.split || a.kp.chunks_per_cta * a.kp.split < a.kp.total_chunks)
                wrong++;
        }
        else if (a.grid > 148 || (a.kp.resident && a.grid % a.kp.cbs != 0 && a.grid != a.kp.tiles) || a.kp.num_stages < 2)
            wrong++;
    }
    std::printf("taken=%lld split=%lld wrong=%lld\n", taken, split, wrong);
    return wrong != 0 || taken == 0 || split == 0;
}
