// Test harness (CPU only): the block sizes of the optimizer's chains.  Every number of
// chains up to two full blocks an SM: whole warps, at most 256 threads, few enough
// blocks for the sums' workspace (two an SM and one, or the full blocks' number), and in
// 3 dimensions and more, where an SM's time goes with its chains, no SM with over 5/4 of
// what full blocks dealt out evenly give it (5/4: two blocks of 160, which were faster).
#include <algorithm>
#include <cstdio>

#include "chain_blocks.h"

int main() {
    for (int sms : {132, 148, 152}) {
        for (int d = 1; d <= 6; ++d) {
            for (int chains = 1; chains <= 512 * sms; ++chains) {
                const int t = ncvis_gpu::chain_block_threads(chains, d, sms, 256);
                const int blocks = (chains + t - 1) / t, full = (chains + 255) / 256;
                const int load = (blocks + sms - 1) / sms * t;
                const int full_load = (full + sms - 1) / sms * 256;
                if (t < 32 || t > 256 || t % 32 || blocks > std::max(2 * sms + 1, full) ||
                    (d >= 3 && 4 * load > 5 * full_load)) {
                    std::printf("%d chains, d = %d, %d SMs: %d blocks of %d\n", chains, d, sms,
                                blocks, t);
                    return 1;
                }
            }
        }
    }
    std::printf("ok\n");
    return 0;
}
