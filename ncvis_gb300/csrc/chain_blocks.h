// Block size of the unstaged optimizer's chains (sgd.cu).
#pragma once

namespace ncvis_gpu {

// Threads per block for `chains` chains of a d-dimensional embedding, one a thread, on
// `sms` SMs, at most `most` (a multiple of 32).  Few chains are spread over all SMs: a
// sample's row gather and its reduction each take an SM's load unit a cycle a lane, so
// that 5,000 chains in blocks of 256 waited for 20 SMs (547 us an epoch of 20 noise
// samples at 10,000 points; 474 in blocks of 32).  The blocks are a little smaller than
// an SM's share, so that a few SMs have two; from 3 dimensions on and 11/16 of a full
// block an SM those are what the others wait for, and the blocks are full ones (5
// epochs, full and smaller: 50,000 points in 3 and 4 dimensions 4,434 and 4,051, 3,668 and
// 3,243 us, 55,000 4,655 and 5,332, 3,697 and 4,315, 75,000 6,001 and 7,888, 3,853 and
// 5,775; in 1 and 2 dimensions the smaller ones stay ahead, 75,000 3,201 and 2,931, 3,281
// and 2,991).
inline int chain_block_threads(int chains, int d, int sms, int most) {
    const int share = chains / sms;
    if (share >= most || (d >= 3 && 16 * share >= 11 * most)) return most;
    return share < 32 ? 32 : share / 32 * 32;
}

}  // namespace ncvis_gpu
