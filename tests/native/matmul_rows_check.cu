// The rule that sends a MATMUL to matmul_rows.cu, on the host: what it takes must leave the kernels' 32-bit indexes over K in
// range (the main loop steps by 512 rows behind the last one, the sums of A's rows by 1024).
#include <cstdio>

#include "../../reference_model_b200/csrc/matmul_rows.cu"

namespace tb200
{
tb200_status post_launch(tb200_ctx*, const char*, int) { return TB200_OK; }
void timer_begin(tb200_ctx*) {}
void timer_end(tb200_ctx*) {}
}    // namespace tb200

int main()
{
    using namespace tb200;
    const void* p = reinterpret_cast<const void*>(static_cast<uintptr_t>(4096));
    long long taken = 0, wrong = 0;
    for (tb200_dtype dt : { TB200_INT8, TB200_FP16, TB200_BF16 })
        for (long long c : { 256LL, 4096LL, 1LL << 20, (1LL << 30) - 4, 1LL << 30, (1LL << 30) + 4, (1LL << 31) - 1024, (1LL << 31) - 4 })
        {
            if (!matmul_rows_supported(dt, p, p, 1, 1, (int)c, 4, 148))
                continue;
            taken++;
            for (int splits = 1; splits <= 8; splits *= 2)
            {
                const long long per = ((c + splits - 1) / splits + 3) & ~3LL;
                // first row of a rank's share, its end, and the rows that the last pass looks at
                if ((splits - 1) * per + per > 0x7fffffffLL || c + 4 * 8 * 4 + 4 * 8 * 3 + 3 > 0x7fffffffLL || c + splits - 1 + 3 > 0x7fffffffLL)
                    wrong++;
            }
            if (c + 5 * 1024 > 0x7fffffffLL)
                wrong++;
        }
    std::printf("taken=%lld wrong=%lld\n", taken, wrong);
    return wrong != 0 || taken == 0;
}
