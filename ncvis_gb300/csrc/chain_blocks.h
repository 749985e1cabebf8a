// Block size of the unstaged optimizer's chains (sgd.cu).
#pragma once

namespace ncvis_gpu {

// Threads per block for `chains` chains, one a thread, on `sms` SMs, at most `most` (a
// multiple of 32).  Few chains are spread over all SMs: a sample's row gather and its
// reduction each take an SM's load unit a cycle a lane, so that 5,000 chains in blocks
// of 256 waited for 20 SMs (547 us an epoch of 20 noise samples at 10,000 points; 474 in
// blocks of 32).  Up to most / 2 chains an SM the blocks are a little smaller than an
// SM's share and a few SMs have two (30,000 points in 3 dimensions, 5 epochs: 4,397 us
// in blocks of 256, 3,486 so, 3,560 in larger ones); beyond, a few SMs with two are what
// the others wait for, and the blocks are at least the share (75,000 points in 4
// dimensions: 3,853, 5,775 and 3,650).  No SM gets more chains than blocks of `most`
// give it.
inline int chain_block_threads(int chains, int sms, int most) {
    const int down = chains / sms / 32 * 32, up = ((chains + sms - 1) / sms + 31) / 32 * 32;
    if (chains / sms < most / 2) return down < 32 ? 32 : down;
    return up < most ? up : most;
}

}  // namespace ncvis_gpu
