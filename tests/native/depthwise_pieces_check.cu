// How the sliding depthwise kernels cut rows into pieces, on the host: a launch looks at few counts however long the rows are, the
// pieces cover the row without an empty one, and up to 256 outputs every count that gives another length is looked at.
#include <cstdio>
#include <set>

#include "../../reference_model_b200/csrc/depthwise_i8.cu"

namespace tb200
{
tb200_status post_launch(tb200_ctx*, const char*, int) { return TB200_OK; }
}    // namespace tb200

int main()
{
    long long checked = 0, wrong = 0;
    for (int K : { 3, 5 })
        for (int S : { 1, 2 })
            for (long long lines : { 4LL, 1000LL, 200000LL })
                for (int OW = 1; OW < 2000000; OW += OW < 600 ? 1 : OW / 7)
                {
                    int len = 0, strips = 0;
                    const int tried = tb200::dw_pieces(lines, OW, K, S, K == 3 && S == 1 ? 2 : 1, 148, 4, &len, &strips);
                    std::set<int> lens;
                    for (int s = 1; s <= std::max(1, OW / 2) && OW <= 256; s++)
                        lens.insert((OW + s - 1) / s);
                    checked++;
                    if (tried > 48 || len < 1 || (long long)len * strips < OW || (long long)len * (strips - 1) >= OW || (OW <= 256 && tried < (int)lens.size()))
                        wrong++;
                }
    std::printf("checked=%lld wrong=%lld\n", checked, wrong);
    return wrong != 0;
}
