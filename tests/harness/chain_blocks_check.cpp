// Test harness (CPU only): the block sizes of the optimizer's chains.  Every number of
// chains up to two full blocks an SM: whole warps, at most 256 threads, few enough
// blocks for the sums' workspace (two an SM and one, or the full blocks' number), and no
// SM with more chains than blocks of 256 dealt out evenly give it.
#include <algorithm>
#include <cstdio>

#include "chain_blocks.h"

int main() {
    for (int sms : {1, 3, 132, 148, 152}) {
        for (int chains = 1; chains <= 512 * sms; ++chains) {
            const int t = ncvis_gpu::chain_block_threads(chains, sms, 256);
            const int blocks = (chains + t - 1) / t, full = (chains + 255) / 256;
            const int load = (blocks + sms - 1) / sms * t, full_load = (full + sms - 1) / sms * 256;
            if (t < 32 || t > 256 || t % 32 || load > full_load ||
                blocks > std::max(2 * sms + 1, full)) {
                std::printf("%d chains on %d SMs: %d blocks of %d\n", chains, sms, blocks, t);
                return 1;
            }
        }
    }
    std::printf("ok\n");
    return 0;
}
