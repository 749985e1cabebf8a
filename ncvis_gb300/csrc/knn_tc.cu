// K2: kNN candidate selection on the 5th-generation tensor cores (tcgen05),
// BF16 operands with FP32 accumulation; the candidates are re-ranked exactly
// in FP32 afterwards (K4, knn_simt.cu), which restores the reference's
// distances (src/ncvis.cpp:72-153) on the selected set.
//
// Work decomposition (one persistent CTA per SM, 11 warps):
//   * a query tile is 256 preprocessed points (two M=128 halves), held in
//     shared memory for the whole sweep (TMA, 128-byte swizzle, K-major);
//   * candidate tiles of 128 points stream through a TMA ring, a stage per part
//     of a tile;
//   * warp 0 issues TMA; warps 1 and 10 issue tcgen05.mma (M=128, N=128,
//     K=16 steps), one query half each, into one of two double-buffered
//     2x128-column FP32 accumulators (512 TMEM columns; warp 1 allocates);
//     each half hands its accumulators to its own four epilogue warps;
//   * warps 2..9 own one query row each (TMEM lane = row; warp % 4 selects
//     the lane quadrant): they read the accumulator with tcgen05.ld in
//     32-column chunks, turn dot products into ranking scores (-<q,c> for the
//     inner-product spaces, |c|^2 - 2<q,c> for squared L2), reduce each chunk
//     with 3-input min/max trees and compare its best with the row's worst;
//     a group of 4 columns that holds a qualifying candidate goes whole to a
//     per-row queue in shared memory; when a queue is full the warp looks all its
//     rows' queues over and inserts what qualifies into the rows'
//     register-resident sorted lists in lockstep rounds (the first tiles of a
//     short sweep: single candidates, merged in 16 at a time by a network);
//   * a CTA takes items from its own work list: an item is a query tile's rows
//     and one candidate range (masked at both ends), and may continue the
//     previous item's tile, so one tile's lists are built over several ranges
//     (batched problems: the tile's own problem; the inverted file: the tile's
//     probed cells), with an optional map from sorted rows back to the caller's
//     numbering; items of several CTAs may share a query tile, each writing a
//     list of its own, with its scores, of which the best are kept afterwards
//     (sweep_items, merge_lists: the last wave of one problem's tiles);
//   * squared L2 with D <= 126 folds the candidate norms into the product:
//     candidates come from a second BF16 copy whose columns D, D + 1 hold
//     -|c|^2 / 2 as a BF16 high and low part, the queries' copy 1, 1 there, so
//     the accumulator holds <q, c> - |c|^2 / 2 and the scan is the
//     inner-product one (otherwise the scan adds the FP32 norms per column);
//   * kParts = 2 is the FP32 search's form (launch_knn_select_split): every row
//     is an FP16 high and low part (split_rows, preprocess.cu), a candidate
//     tile is taken in two parts, and its product is the sum of three FP16
//     products accumulated in FP32, the small ones first: q_hi c_lo, then
//     q_lo c_hi and q_hi c_hi (q_lo c_lo as well for rows of up to 32 columns,
//     where it is not below the others' rounding, and for plans with low_low).
// Every mbarrier wait is bounded in time: on expiry the CTA sets *err,
// stops, drains its MMAs and in-flight TMA copies, frees TMEM and returns.
// The waits between roles use the plan's limit (default ~2 s); the drain
// waits always use the long one.  An epilogue warp decides as a warp (votes)
// whether to stop, so its lanes never part at a warp-collective instruction.
// A diagnostic stall makes the producer first wait on a barrier that nothing
// completes, so that the timeout path runs deterministically.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cfloat>
#include <string>
#include <type_traits>

#include "common.cuh"
#include "stages.cuh"

namespace ncvis_gpu {

namespace {

constexpr int kQueryTile = 256;   // queries per CTA tile (2 x M=128)
constexpr int kCandTile = 128;    // candidates per tile (N=128)
constexpr int kAtomBytes = 128 * 128;  // 128 rows x 128 bytes (64 bf16) per swizzle atom column
constexpr int kMaxAtoms = 2;      // K <= 128
constexpr int kThreads = 352;
constexpr int kEpiWarp0 = 2;
constexpr int kEpiWarps = 8;
constexpr int kMmaWarp1 = 10;  // issues the second query half's MMAs (warp 1 the first)
constexpr uint32_t kTmemCols = 512;
constexpr int kLowLowSteps = 2;  // K steps up to which the low parts' product is taken too
constexpr long long kWaitCycles = 4000000000LL;  // ~2 s at 2 GHz

// One queued group of 4 accumulator columns of a warp's rows: the values and the
// candidate index of the first column.
constexpr int kGroup = 4;
constexpr uint32_t kFlushAt = 4;  // slots past which a queue is flushed after a tile
// Pending entries past which lists are merged after a tile: 10,000 x 64 144, 134, 129 us
// with 5, 8 and 11.
constexpr uint32_t kMergeAt = 11;
// Candidate tiles that fill a list: 131,072 x 100 4.53, 4.55 and 4.69 ms with 16, 32 and
// 64, 60,013 x 100 FP32 1.76, 1.78 and 1.86.
constexpr int kFillTiles = 16;
struct QueueSlot {
    float4 v[32];
    int32_t first[32];
};

// Shared memory by the number of parts a row is held in: the query tile takes
// 64 KB a part, so the two-part form has a ring of 2 stages and 6 queue slots
// per row where the one-part form has 3 and 12 (both 224 KB in all).  Stages of
// 64 columns (half a part, twice as many) made the BF16 sweep of 1,024,000 x 100
// 18% slower: the MMA warps then wait within a tile too.
template <int kParts>
struct SharedStorage {
    static constexpr int kStages = kParts == 1 ? 3 : 2;  // candidate ring (32 KB each)
    static constexpr int kQueue = kParts == 1 ? 12 : 6;  // column groups queued per row
    // 1024-byte aligned tiles first (128B swizzle atoms repeat every 1024 B).
    uint8_t a[2][kParts][kMaxAtoms][kAtomBytes];
    uint8_t b[kStages][kMaxAtoms][kAtomBytes];
    QueueSlot queue[kEpiWarps][kQueue];  // each warp's own: it may hold entries instead
    uint64_t full[kStages];
    uint64_t empty[kStages];
    uint64_t a_full, a_empty;
    uint64_t acc_full[2][2], acc_empty[2][2];  // [buffer][query half]
    uint64_t drain;
    uint64_t never;  // completed by nothing: the diagnostic stall waits on it
    uint32_t tmem_base;
    volatile int abort;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait (`limit` SM cycles) for the phase of `parity`; false if it
// expired or the CTA aborted.
__device__ __forceinline__ bool mbar_wait(volatile int &abort, uint64_t *bar, uint32_t parity,
                                          int *err, int code, long long limit) {
    const long long t0 = clock64();
    while (!mbar_try_wait(bar, parity)) {
        if (abort) return false;
        if (clock64() - t0 > limit) {
            abort = 1;
            atomicExch(err, code);
            return false;
        }
    }
    return true;
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x,
                                            int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes "
        "[%0], [%1, {%3, %4}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (stride byte offset), descriptor version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr) {
    uint64_t d = (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;             // leading byte offset (unused with 128B swizzle, K-major)
    d |= (uint64_t)(1024 >> 4) << 32;   // stride byte offset
    d |= (uint64_t)1 << 46;             // version
    d |= (uint64_t)2 << 61;             // 128-byte swizzle
    return d;
}

// Instruction descriptor, kind::f16: D f32, A and B both bf16 (type 1) or both
// f16 (type 0), both K-major, M=128, N=128.
constexpr uint32_t idesc(uint32_t type) {
    return (1u << 4) | (type << 7) | (type << 10) | ((uint32_t)(kCandTile >> 3) << 17) |
           ((uint32_t)(128 >> 4) << 24);
}

template <uint32_t kIdesc>
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %4, p;\n\t}" ::"r"(tmem_d),
        "l"(a), "l"(b), "r"(acc), "r"(kIdesc));
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tmem_fence_after() {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_before() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ float max3f(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Minimum (kMax false) or maximum of n values, as a tree of 3-input operations.
template <bool kMax, int n>
__device__ __forceinline__ float tree_reduce(const float (&a)[n]) {
    if constexpr (n == 1) {
        return a[0];
    } else if constexpr (n == 2) {
        return kMax ? fmaxf(a[0], a[1]) : fminf(a[0], a[1]);
    } else {
        constexpr int m = (n + 2) / 3;
        float b[m];
#pragma unroll
        for (int j = 0; j < m; ++j) {
            if (3 * j + 2 < n)
                b[j] = kMax ? max3f(a[3 * j], a[3 * j + 1], a[3 * j + 2])
                            : min3f(a[3 * j], a[3 * j + 1], a[3 * j + 2]);
            else if (3 * j + 1 < n)
                b[j] = kMax ? fmaxf(a[3 * j], a[3 * j + 1]) : fminf(a[3 * j], a[3 * j + 1]);
            else
                b[j] = a[3 * j];
        }
        return tree_reduce<kMax, m>(b);
    }
}

__device__ __forceinline__ uint32_t ld_shared(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float4 ld_shared_v4(uint32_t a) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(a)
                 : "memory");
    return v;
}

// Insert (v, vi) into the ascending list (ls, li) of R entries, dropping the
// largest.  Every slot's new entry comes from the old ones alone (its own, its
// left neighbour's or the new value, by two compares), so the R slots are
// independent: passing the displaced entry on from slot to slot instead is a
// chain of R dependent compares, which cost the sweeps 6% (131,072 x 100) to 30%
// (65,536 x 50 with 64 entries).
template <int R>
__device__ __forceinline__ void list_push(float (&ls)[R], int32_t (&li)[R], float v, int32_t vi) {
#pragma unroll
    for (int t = R - 1; t > 0; --t) {
        const bool here = v < ls[t], left = v < ls[t - 1];
        li[t] = here ? (left ? li[t - 1] : vi) : li[t];
        ls[t] = fminf(fmaxf(ls[t - 1], v), ls[t]);
    }
    if (v < ls[0]) ls[0] = v, li[0] = vi;
}

// Queues the 4 columns v[0..4) of a row, the first being candidate `first`, when
// their best score gb is below the row's worst: `off` is the byte offset of the
// row's next slot, and moves on; the columns are stored where it lies within the
// queue (predicated stores, no branch).
__device__ __forceinline__ void queue_group(uint32_t queue_v, uint32_t queue_i, uint32_t &off,
                                            uint32_t bytes, float gb, float worst, const float *v,
                                            int32_t first) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t.reg .u32 a, b;\n\t"
        "setp.lt.f32 p, %1, %2;\n\t"
        "setp.lt.and.u32 q, %0, %11, p;\n\t"
        "add.u32 a, %3, %0;\n\t"
        "add.u32 b, %4, %0;\n\t"
        "@q st.shared.v4.f32 [a], {%5, %6, %7, %8};\n\t"
        "@q st.shared.s32 [b], %9;\n\t"
        "@p add.u32 %0, %0, %10;\n\t}"
        : "+r"(off)
        : "f"(gb), "f"(worst), "r"(queue_v), "r"(queue_i), "f"(v[0]), "f"(v[1]), "f"(v[2]),
          "f"(v[3]), "r"(first), "n"(sizeof(QueueSlot)), "r"(bytes)
        : "memory");
}

// Every queued candidate of the warp's rows that still beats its row's worst
// goes into its row's list; queues end empty.  Each lane first marks its
// qualifying values (a bit per queued column), then the warp inserts in lockstep
// rounds, one marked value per row a round, so that a round serves every row
// that has one left.
template <int R, bool kIP, int kQueue>
__device__ __forceinline__ void flush_queue(float (&ls)[R], int32_t (&li)[R], float &worst,
                                            uint32_t &off, uint32_t queue_v, uint32_t queue_i) {
    constexpr uint32_t kSlot = sizeof(QueueSlot);
    const uint32_t most = __reduce_max_sync(0xffffffffu, off);
    uint32_t marks[2] = {0u, 0u};  // slot b's columns: bits 4 (b % 8) .. of marks[b / 8]
#pragma unroll
    for (int b = 0; b < kQueue; ++b) {
        if (b * kSlot >= most) break;
        if (b * kSlot < off) {
            const float4 x = ld_shared_v4(queue_v + b * kSlot);
            const float w[kGroup] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < kGroup; ++j)
                if ((kIP ? -w[j] : w[j]) < worst) marks[b >> 3] |= 1u << (4 * (b & 7) + j);
        }
    }
#pragma unroll 1
    while (__any_sync(0xffffffffu, (marks[0] | marks[1]) != 0u)) {
        if ((marks[0] | marks[1]) != 0u) {
            uint32_t pos;
            if (marks[0] != 0u) {
                pos = __ffs(marks[0]) - 1;
                marks[0] &= marks[0] - 1u;
            } else {
                pos = 31 + __ffs(marks[1]);
                marks[1] &= marks[1] - 1u;
            }
            const uint32_t slot = (pos >> 2) * kSlot, j = pos & 3;
            const float raw = __uint_as_float(ld_shared(queue_v + slot + 4 * j));
            uint32_t first = 0u;  // loaded ahead where there are registers for it
            if (R <= 32) first = ld_shared(queue_i + slot);
            const float x = kIP ? -raw : raw;
            if (x < worst) {
                if (R > 32) first = ld_shared(queue_i + slot);
                list_push<R>(ls, li, x, (int32_t)(first + j));
                worst = ls[R - 1];
            }
        }
    }
    off = 0u;
    __syncwarp();
}

// ---- the filling of a list of 32 --------------------------------------------------
// While a row's list fills, its qualifying candidates wait in shared memory, an entry
// (raw score, index) each, and are merged into the list up to kPending at a time: a
// sorting network over the pending ones, then a bitonic merge, the same instructions
// in every lane.  Inserting them one by one in lockstep rounds (flush_queue) takes
// 180 instructions a round, and the fullest of a warp's 32 rows sets the number of
// rounds: about 570 in the first 80 tiles, where the average row inserts 270.  Later,
// when a tile brings a few rows one candidate each, queueing whole column groups
// and inserting is the faster way (131,072 x 100 in the caller's order 4.6 ms, 5.4 with
// merging all along), as it is for lists of 64, whose networks do not fit the registers.
// The filling is the kernel's form kFill.  Selection without and with it: 1,000 x 32
// 68 and 43 us, 10,000 x 64 175 and 133, 48 problems of 200 to 9,000 1,717 and 1,430,
// 131,072 x 100 3,800 and 3,600.  Sweeps over kFillMaxRows rows or more (TcWork::fill)
// go without: its loop beside theirs costs them more than the filling gives (whole
// calls without and with it: 150,000 x 100 5.98 and 5.92 ms, 150,000 x 32 4.90 and
// 5.08, 250,000 x 64 11.4 and 12.0, 500,000 x 64 38.0 and 41.5).  That rule is for the
// sweeps of one problem's rows (launch_sweep_work, the ordered sweep); the lists of the
// inverted file and of batched problems take short sweeps each and always fill, and so
// does squared L2 without folded norms (127 and 128 columns), which has no other form
// (before the filling and now: inverted file of 1,000,000 x 100 33.9 and 21.2 ms, squared
// L2 of 100,000 x 127 6.20 and 4.79, 300,000 x 127 44.2 and 43.0).
constexpr int kPending = 16;

// Orders entries a and b by score, equal scores by index (the order they are met
// in, but for a sweep that wraps around).
__device__ __forceinline__ bool entry_less(float av, int32_t ai, float bv, int32_t bi) {
    return (av < bv) | ((av == bv) & (ai < bi));
}
__device__ __forceinline__ void order_pair(float &av, int32_t &ai, float &bv, int32_t &bi) {
    const bool swap = entry_less(bv, bi, av, ai);
    const float lv = swap ? bv : av, hv = swap ? av : bv;
    const int32_t li = swap ? bi : ai, hi = swap ? ai : bi;
    av = lv, ai = li, bv = hv, bi = hi;
}

// Queues the 4 columns v[0..4) of a row, the first being candidate `first`: those
// that beat the row's worst (for raw inner products: `limit` is its negative) take
// the entry at byte offset `off`, which moves on; an entry is stored where it lies
// within the first `cap` bytes (predicated stores, no branch).
template <bool kIP>
__device__ __forceinline__ void push_group(uint32_t pend_v, uint32_t pend_i, uint32_t &off,
                                           uint32_t cap, float limit, const float *v,
                                           int32_t first) {
    constexpr int kEntry = 32 * 4;
#pragma unroll
    for (int j = 0; j < kGroup; ++j) {
        if constexpr (kIP)
            asm volatile(
                "{\n\t.reg .pred p, q;\n\t.reg .u32 a, b;\n\t"
                "setp.gt.f32 p, %1, %2;\n\t"
                "setp.lt.and.u32 q, %0, %6, p;\n\t"
                "add.u32 a, %3, %0;\n\t"
                "add.u32 b, %4, %0;\n\t"
                "@q st.shared.f32 [a], %1;\n\t"
                "@q st.shared.s32 [b], %5;\n\t"
                "@p add.u32 %0, %0, %7;\n\t}"
                : "+r"(off)
                : "f"(v[j]), "f"(limit), "r"(pend_v), "r"(pend_i), "r"(first + j), "r"(cap),
                  "n"(kEntry)
                : "memory");
        else
            asm volatile(
                "{\n\t.reg .pred p, q;\n\t.reg .u32 a, b;\n\t"
                "setp.lt.f32 p, %1, %2;\n\t"
                "setp.lt.and.u32 q, %0, %6, p;\n\t"
                "add.u32 a, %3, %0;\n\t"
                "add.u32 b, %4, %0;\n\t"
                "@q st.shared.f32 [a], %1;\n\t"
                "@q st.shared.s32 [b], %5;\n\t"
                "@p add.u32 %0, %0, %7;\n\t}"
                : "+r"(off)
                : "f"(v[j]), "f"(limit), "r"(pend_v), "r"(pend_i), "r"(first + j), "r"(cap),
                  "n"(kEntry)
                : "memory");
    }
}

// Batcher's odd-even merge sort of the pending entries, from its step (p, k) on.
template <int p, int k>
__device__ __forceinline__ void sort_pending(float (&pv)[kPending], int32_t (&pi)[kPending]) {
#pragma unroll
    for (int x = k % p; x + k < kPending; ++x)
        if ((x - k % p) / k % 2 == 0 && x / (2 * p) == (x + k) / (2 * p))
            order_pair(pv[x], pi[x], pv[x + k], pi[x + k]);
    if constexpr (k > 1)
        sort_pending<p, k / 2>(pv, pi);
    else if constexpr (2 * p < kPending)
        sort_pending<2 * p, 2 * p>(pv, pi);
}

// The bitonic merge of R entries, from distance st on.
template <int st, int R>
__device__ __forceinline__ void merge_bitonic(float (&ls)[R], int32_t (&li)[R]) {
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (!(i & st)) order_pair(ls[i], li[i], ls[i + st], li[i + st]);
    if constexpr (st > 1) merge_bitonic<st / 2, R>(ls, li);
}

// The row's `off` bytes of pending entries (at most kEntries) into its ascending
// list of 32: the pending ones sorted, the smaller of list entry 31 - t and pending
// entry t for the 16 last places (the 32 best of both, a bitonic sequence), merged.
template <int R, bool kIP, int kEntries>
__device__ __forceinline__ void merge_pending(float (&ls)[R], int32_t (&li)[R], float &worst,
                                              uint32_t &off, uint32_t pend_v,
                                              uint32_t pend_i) {
    static_assert(kEntries <= kPending, "pending entries");
    constexpr uint32_t kEntry = 32 * 4;
    float pv[kPending];
    int32_t pi[kPending];
#pragma unroll
    for (int b = 0; b < kPending; ++b) {
        pv[b] = FLT_MAX;
        pi[b] = -1;
        if (b < kEntries && b * kEntry < off) {
            const float raw = __uint_as_float(ld_shared(pend_v + b * kEntry));
            pv[b] = kIP ? -raw : raw;
            pi[b] = (int32_t)ld_shared(pend_i + b * kEntry);
        }
    }
    sort_pending<1, 1>(pv, pi);
#pragma unroll
    for (int t = 0; t < kPending; ++t) {
        const int at = R - 1 - t;
        const bool take = entry_less(pv[t], pi[t], ls[at], li[at]);
        ls[at] = take ? pv[t] : ls[at];
        li[at] = take ? pi[t] : li[at];
    }
    merge_bitonic<R / 2>(ls, li);
    if (off > 0u) worst = ls[R - 1];
    off = 0u;
}

// One item of work (TcItem): the query tile of 256 rows from row0 (rows at or
// past qend are not outputs) against candidate rows [lo, hi); `cont`: the item
// extends the previous item's query tile (no reload, lists carry over);
// `more`: a later item extends this one (lists written after the last).
struct QueryTile {
    int32_t row0, qend, lo, hi;  // N < 2^31
    bool cont, more;
};

__device__ __forceinline__ QueryTile work_item(const TcItem *__restrict__ work, int64_t it) {
    const TcItem w = work[it];
    QueryTile q;
    q.row0 = w.row0;
    q.qend = w.qend;
    q.lo = w.lo;
    q.hi = w.hi;
    q.cont = (w.flags & kTcContinue) != 0;
    q.more = (w.flags & kTcMore) != 0;
    return q;
}

// The work list of one problem of N rows spread as `w` says: CTA b takes the
// whole query tiles b, b + ctas, ... below full_qt, then its run of the other
// tiles' (query tile, candidate tile) pairs, an item per query tile it meets.
__global__ void sweep_items(int64_t N, TcSweep w, int stride, int64_t *__restrict__ begin,
                            int64_t *__restrict__ end, TcItem *__restrict__ items) {
    const int64_t b = blockIdx.x;
    const TcRun run(N, w);
    const int64_t n_ct = run.n_ct;
    const int64_t r0 = b < run.G ? run.begin(b) : 0, r1 = b < run.G ? run.begin(b + 1) : 0;
    const int64_t whole = b < w.full_qt ? (w.full_qt - 1 - b) / w.ctas + 1 : 0;
    const int64_t n = whole + (r1 > r0 ? (r1 - 1) / n_ct - r0 / n_ct + 1 : 0);
    TcItem *mine = items + b * stride;
    for (int64_t it = threadIdx.x; it < n; it += blockDim.x) {
        TcItem q{};
        q.qend = q.hi = (int32_t)N;
        if (it < whole) {
            q.row0 = (int32_t)((b + it * w.ctas) * kQueryTile);
        } else {
            const int64_t t = r0 / n_ct + (it - whole);  // query tile among the rest
            const int64_t u0 = max(r0, t * n_ct), u1 = min(r1, (t + 1) * n_ct);
            q.row0 = (int32_t)((w.full_qt + t) * kQueryTile);
            q.lo = (int32_t)((u0 - t * n_ct) * kCandTile);
            q.hi = (int32_t)min(N, (u1 - t * n_ct) * kCandTile);
            // The tile's first pair is in the run of the last CTA that begins
            // at or before it; the CTAs after it write the next lists.
            q.slot = (int32_t)(b - run.first_cta(t));
        }
        mine[it] = q;
    }
    if (threadIdx.x == 0) {
        begin[b] = b * stride;
        end[b] = b * stride + n;
    }
}

// Items of one CTA at most: its whole tiles and the query tiles its run meets.
int sweep_stride(int64_t N, const TcSweep &w) {
    const int64_t n_qt = (N + kQueryTile - 1) / kQueryTile, n_ct = (N + kCandTile - 1) / kCandTile;
    const int64_t run = ((n_qt - w.full_qt) * n_ct + w.rest_ctas - 1) / w.rest_ctas;
    return (int)((w.full_qt + w.ctas - 1) / w.ctas + (run + n_ct - 1) / n_ct + 1);
}

// Rows of the operands' parts in their tensor maps: part p of row r is row
// part[p] + r (part 0 the high or only one, part 1 the low one).
struct TcParts {
    int32_t q[2], c[2];
};

template <int R, bool kIP, int kParts, bool kFill>
__global__ void __launch_bounds__(kThreads, 1)
    knn_select_tc(const __grid_constant__ CUtensorMap tmap,
                  const __grid_constant__ CUtensorMap tmap_c, const TcParts parts,
                  const float *__restrict__ sqnorm, int ksteps, int katoms, int low_low_steps,
                  const int64_t *__restrict__ work_begin, const int64_t *__restrict__ work_end,
                  const TcItem *__restrict__ work, const int32_t *__restrict__ row_map,
                  int32_t *__restrict__ cand_i, const TcLists lists, int *__restrict__ err,
                  long long wait_limit, int stall) {
    using Shared = SharedStorage<kParts>;
    constexpr int kStages = Shared::kStages;
    constexpr int kQueue = Shared::kQueue;
    extern __shared__ uint8_t smem_raw[];
    Shared &s = *reinterpret_cast<Shared *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                            ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t n_items = work_end[blockIdx.x] - work_begin[blockIdx.x];
    const TcItem *const mine = work + work_begin[blockIdx.x];
    const uint32_t a_bytes = 2u * kParts * katoms * kAtomBytes;
    const uint32_t b_bytes = (uint32_t)katoms * kAtomBytes;

    if (threadIdx.x == 0) {
        // Barriers the MMA issuers commit to take one arrival from each of the two.
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&s.full[i], 1);
            mbar_init(&s.empty[i], 2);
        }
        mbar_init(&s.a_full, 1);
        mbar_init(&s.a_empty, 2);
        // Each query half has its own accumulator hand-off: its MMA warp and
        // its four epilogue warps, so one half's slow tile does not hold the other.
        for (int i = 0; i < 2; ++i)
            for (int hh = 0; hh < 2; ++hh) {
                mbar_init(&s.acc_full[i][hh], 1);
                mbar_init(&s.acc_empty[i][hh], kEpiWarps / 2);
            }
        mbar_init(&s.drain, 2);
        mbar_init(&s.never, 1);
        s.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(&s.tmem_base)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tmem_fence_before();
    __syncthreads();
    tmem_fence_after();
    const uint32_t tmem = s.tmem_base;

    if (warp == 0 && lane == 0) {
        // ---------------------------------------------------------- TMA producer
        int stage = 0;
        uint32_t phase = 0, a_phase = 0;
        uint32_t issued_parity[kStages];
        bool issued[kStages];
        for (int i = 0; i < kStages; ++i) issued[i] = false, issued_parity[i] = 0;
        bool a_issued = false;
        uint32_t a_parity = 0;
        if (stall) mbar_wait(s.abort, &s.never, 0, err, 7, wait_limit);
        for (int64_t it = 0; it < n_items && !s.abort; ++it) {
            const QueryTile q = work_item(mine, it);
            if (!q.cont) {
                if (!mbar_wait(s.abort, &s.a_empty, a_phase ^ 1, err, 1, wait_limit)) break;
                mbar_expect_tx(&s.a_full, a_bytes);
                for (int h = 0; h < 2; ++h)
                    for (int p = 0; p < kParts; ++p)
                        for (int at = 0; at < katoms; ++at)
                            tma_load_2d(s.a[h][p][at], &tmap, &s.a_full, at * 64,
                                        (int)(parts.q[p] + q.row0 + h * 128));
                a_issued = true;
                a_parity = a_phase;
                a_phase ^= 1;
            }
            bool ok = true;
            for (int64_t ct = q.lo / kCandTile; ok && ct * kCandTile < q.hi; ++ct) {
                // The low part of a tile first, then the high one.
                for (int p = kParts - 1; p >= 0; --p) {
                    if (!mbar_wait(s.abort, &s.empty[stage], phase ^ 1, err, 2, wait_limit)) {
                        ok = false;
                        break;
                    }
                    mbar_expect_tx(&s.full[stage], b_bytes);
                    for (int at = 0; at < katoms; ++at)
                        tma_load_2d(s.b[stage][at], &tmap_c, &s.full[stage], at * 64,
                                    (int)(parts.c[p] + ct * kCandTile));
                    issued[stage] = true;
                    issued_parity[stage] = phase;
                    if (++stage == kStages) stage = 0, phase ^= 1;
                }
            }
        }
        // Copies still in flight must land before the CTA's shared memory goes away.
        const long long t0 = clock64();
        for (int i = 0; i < kStages; ++i)
            if (issued[i])
                while (!mbar_try_wait(&s.full[i], issued_parity[i]) && clock64() - t0 < kWaitCycles) {
                }
        if (a_issued)
            while (!mbar_try_wait(&s.a_full, a_parity) && clock64() - t0 < kWaitCycles) {
            }
    } else if ((warp == 1 || warp == kMmaWarp1) && lane == 0) {
        // ---------------------------------------------------------- MMA issuers
        // Warp 1 issues query half 0's MMAs, warp kMmaWarp1 half 1's: two
        // schedulers share the descriptor work of a tile.
        const int h = (warp == 1) ? 0 : 1;
        int stage = 0;
        uint32_t phase = 0, a_phase = 0, acc_phase = 0;
        int acc = 0;
        for (int64_t it = 0; it < n_items && !s.abort; ++it) {
            const QueryTile q = work_item(mine, it);
            if (!q.cont) {
                if (!mbar_wait(s.abort, &s.a_full, a_phase, err, 3, wait_limit)) break;
                a_phase ^= 1;
            }
            tmem_fence_after();
            bool ok = true;
            for (int64_t ct = q.lo / kCandTile; ok && ct * kCandTile < q.hi; ++ct) {
                if (!mbar_wait(s.abort, &s.acc_empty[acc][h], acc_phase ^ 1, err, 4, wait_limit))
                    break;
                const uint32_t d_tmem = tmem + (uint32_t)(acc * 256 + h * 128);
                uint32_t accumulate = 0u;
                for (int p = kParts - 1; p >= 0; --p) {
                    if (!mbar_wait(s.abort, &s.full[stage], phase, err, 5, wait_limit)) {
                        ok = false;
                        break;
                    }
                    tmem_fence_after();
                    auto product = [&](int qp) {
                        for (int ks = 0; ks < ksteps; ++ks) {
                            const int at = ks >> 2;
                            const uint32_t off = (uint32_t)(ks & 3) * 32;
                            const uint64_t ad = smem_desc(smem_u32(s.a[h][qp][at]) + off);
                            const uint64_t bd = smem_desc(smem_u32(s.b[stage][at]) + off);
                            umma_f16<idesc(kParts == 1 ? 1u : 0u)>(d_tmem, ad, bd, accumulate);
                            accumulate = 1u;
                        }
                    };
                    if (kParts == 2 && (p == 0 || ksteps <= low_low_steps)) product(kParts - 1);
                    product(0);
                    umma_commit(&s.empty[stage]);
                    if (++stage == kStages) stage = 0, phase ^= 1;
                }
                if (!ok) break;
                umma_commit(&s.acc_full[acc][h]);
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
            if (!q.more) umma_commit(&s.a_empty);
        }
        // Every issued MMA completes before TMEM is released.
        umma_commit(&s.drain);
        const long long t0 = clock64();
        while (!mbar_try_wait(&s.drain, 0) && clock64() - t0 < kWaitCycles) {
        }
    } else if (warp >= kEpiWarp0 && warp < kEpiWarp0 + kEpiWarps) {
        // ---------------------------------------------------------- epilogue
        const int h = (warp - kEpiWarp0) >> 2;
        const int quad = warp & 3;
        const int row_in_tile = h * 128 + quad * 32 + lane;
        // Accumulator columns per tcgen05.ld: 32 with 32-entry lists; 64-entry
        // lists leave registers for 16.
        constexpr int kC = R <= 32 ? 32 : 16;
        constexpr int kG = kC / kGroup;  // column groups per load
        // A list's first tiles (lists of 32): its row's pending candidates, else
        // queued column groups, in the same memory.
        constexpr bool kMerge = R == 32 && kFill;
        constexpr int kFits = sizeof(s.queue[0]) / (8 * 32);
        constexpr int kEntries = kFits < kPending ? kFits : kPending;
        constexpr uint32_t kQueueBytes = kQueue * sizeof(QueueSlot);
        constexpr uint32_t kPendBytes = kEntries * 32 * 4;
        const uint32_t queue_v = smem_u32(&s.queue[warp - kEpiWarp0][0].v[lane]);
        const uint32_t queue_i = smem_u32(&s.queue[warp - kEpiWarp0][0].first[lane]);
        auto flush = [&](float (&ls)[R], int32_t (&li)[R], float &worst, uint32_t &off) {
            flush_queue<R, kIP, kQueue>(ls, li, worst, off, queue_v, queue_i);
        };
        uint32_t acc_phase = 0;
        int acc = 0;
        float ls[R];
        int32_t li[R];
        float worst = FLT_MAX;
        uint32_t qoff = 0u;
        const int32_t it_end = (int32_t)work_end[blockIdx.x];
        for (int32_t it = (int32_t)work_begin[blockIdx.x]; it < it_end; ++it) {
            // Lanes read the abort flag at different times: the warp stops as one.
            if (__any_sync(0xffffffffu, s.abort != 0)) break;
            const QueryTile q = work_item(work, it);
            if (!q.cont) {
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    ls[t] = FLT_MAX;
                    li[t] = -1;
                }
                // Nothing qualifies in rows that are not outputs.
                worst = q.row0 + row_in_tile < q.qend ? FLT_MAX : -INFINITY;
                qoff = 0u;
            }
            // Candidate tiles [ct, ct_end), the first ones of a list (kFilling) or later
            // ones; false if a wait ran out.  Two loops: in one loop with a branch for
            // each the later tiles took 25% longer.
            auto scan = [&](auto filling, int32_t ct, const int32_t ct_end) {
                constexpr bool kFilling = decltype(filling)::value;
                for (; ct < ct_end; ++ct) {
                    const bool got = mbar_wait(s.abort, &s.acc_full[acc][h], acc_phase, err, 6, wait_limit);
                    if (!__all_sync(0xffffffffu, got)) return false;
                    tmem_fence_after();
                    const int32_t c0 = ct * kCandTile;
                    // A tile reaching outside [lo, hi): its outside columns are masked.
                    const bool tail = c0 < q.lo || c0 + kCandTile > q.hi;
#pragma unroll 1
                    for (int chunk = 0; chunk < kCandTile / kC; ++chunk) {
                        float v[kC];
                        __syncwarp();
                        tmem_ld(tmem + ((uint32_t)(quad * 32) << 16) +
                                    (uint32_t)(acc * 256 + h * 128 + chunk * kC),
                                v);
                        if (chunk == kCandTile / kC - 1) {
                            // The tile's last columns are in registers: the
                            // accumulator goes back to the MMA warp before their
                            // scan, so the next MMAs into it start meanwhile.
                            tmem_fence_before();
                            __syncwarp();
                            if (lane == 0) mbar_arrive(&s.acc_empty[acc][h]);
                        }
                        const int32_t cb = c0 + chunk * kC;
                        // Scores, lower is better: |c|^2 - 2<q,c> (squared L2) or
                        // -<q,c> (kept as +<q,c>, compared against -worst).
                        if constexpr (!kIP) {
                            // The chunk's candidate norms, the same for every lane:
                            // 16-byte loads where the chunk lies inside the rows.
                            if (cb >= q.lo && cb + kC <= q.hi) {
#pragma unroll
                                for (int j = 0; j < kC; j += 4) {
                                    const float4 nc =
                                        __ldg(reinterpret_cast<const float4 *>(sqnorm + cb + j));
                                    v[j] = fmaf(-2.f, v[j], nc.x);
                                    v[j + 1] = fmaf(-2.f, v[j + 1], nc.y);
                                    v[j + 2] = fmaf(-2.f, v[j + 2], nc.z);
                                    v[j + 3] = fmaf(-2.f, v[j + 3], nc.w);
                                }
                            } else {
#pragma unroll
                                for (int j = 0; j < kC; ++j) {
                                    const int32_t c = cb + j;
                                    const float nc =
                                        (c >= q.lo && c < q.hi) ? __ldg(sqnorm + c) : 0.f;
                                    v[j] = fmaf(-2.f, v[j], nc);
                                }
                            }
                        }
                        if (tail) {
#pragma unroll
                            for (int j = 0; j < kC; ++j)
                                if (cb + j < q.lo || cb + j >= q.hi) v[j] = kIP ? -FLT_MAX : FLT_MAX;
                        }
                        // Best score of each group of columns, then of the chunk.
                        float gb[kG];
#pragma unroll
                        for (int g = 0; g < kG; ++g) {
                            const float *w = v + kGroup * g;
                            gb[g] = kIP ? -fmaxf(max3f(w[0], w[1], w[2]), w[3])
                                        : fminf(min3f(w[0], w[1], w[2]), w[3]);
                        }
                        const float best = tree_reduce<false, kG>(gb);
                        if constexpr (R == 1) {
                            // The best alone: its column is looked for when it wins.
                            if (!__any_sync(0xffffffffu, best < worst)) continue;
                            if (best < worst) {
                                const float raw = kIP ? -best : best;
#pragma unroll
                                for (int j = kC - 1; j >= 0; --j)
                                    if (v[j] == raw) li[0] = cb + j;
                                ls[0] = worst = best;
                            }
                        } else if constexpr (kFilling) {
                            // The columns that beat the row's worst are queued one by
                            // one, and merged into the lists when a row's queue would
                            // overflow, after a tile when one has more than kMergeAt,
                            // and after the last tile.
                            const bool hit = __any_sync(0xffffffffu, best < worst);
                            const bool tile_end = chunk == kCandTile / kC - 1;
                            if (!hit && !tile_end) continue;
                            const uint32_t limit = !tile_end           ? kPendBytes
                                                   : ct + 1 == ct_end ? 0u
                                                                       : kMergeAt * 32 * 4;
                            const uint32_t pend_v = smem_u32(s.queue[warp - kEpiWarp0]) + 4 * lane;
                            const uint32_t pend_i = pend_v + kPendBytes;
                            const float before = worst;
                            uint32_t start = qoff;
                            for (;;) {
                                if (hit) {
                                    qoff = start;
#pragma unroll
                                    for (int g = 0; g < kG; ++g)
                                        if (__any_sync(0xffffffffu, gb[g] < before))
                                            push_group<kIP>(pend_v, pend_i,
                                                            qoff, kPendBytes,
                                                            kIP ? -before : before, v + kGroup * g,
                                                            cb + kGroup * g);
                                    if ((int32_t)qoff < 0) qoff = 0u;
                                }
                                if (!__any_sync(0xffffffffu, qoff > limit)) break;
                                // Past the end: the chunk is gone over again after the
                                // merge: what was stored now lies below offset 0 (and
                                // is not stored again), what was not follows.
                                const bool over = __any_sync(0xffffffffu, qoff > kPendBytes);
                                qoff = min(qoff, kPendBytes);
                                merge_pending<R, kIP, kEntries>(ls, li, worst, qoff, pend_v,
                                                             pend_i);
                                if (!over) break;
                                start -= kPendBytes;
                            }
                        } else {
                            // The groups whose best beats the row's worst are queued
                            // whole: about 7 instructions a group, where looking at
                            // each column of them here held the accumulator for longer.
                            // A queue that would overflow: as above.
                            if (!__any_sync(0xffffffffu, best < worst)) continue;
                            const float before = worst;
                            uint32_t start = qoff;
                            for (;;) {
                                qoff = start;
#pragma unroll
                                for (int g = 0; g < kG; ++g)
                                    queue_group(queue_v, queue_i, qoff, kQueueBytes, gb[g], before,
                                                v + kGroup * g, cb + kGroup * g);
                                if ((int32_t)qoff < 0) qoff = 0u;
                                if (!__any_sync(0xffffffffu, qoff > kQueueBytes)) break;
                                qoff = min(qoff, kQueueBytes);
                                flush(ls, li, worst, qoff);
                                start -= kQueueBytes;
                            }
                        }
                    }
                    acc ^= 1;
                    if (acc == 0) acc_phase ^= 1;
                    // Here, with the accumulator released, queues past kFlushAt slots
                    // are flushed.  Fewer slots insert for fewer rows a round, more
                    // hold the warp up for longer than the accumulators' two buffers
                    // cover: 131,072 x 100 BF16 6.54, 6.44, 6.45 and 6.53 ms with 1, 2, 4
                    // and 6, 60,013 x 100 FP32 2.59, 2.57, 2.54 and 2.65.
                    if constexpr (!kFilling)
                        if (__any_sync(0xffffffffu, qoff > kFlushAt * sizeof(QueueSlot)))
                            flush(ls, li, worst, qoff);
                }
                return true;
            };
            int32_t ct = q.lo / kCandTile;
            const int32_t ct_end = (q.hi - 1) / kCandTile + 1;
            bool ok = true;
            if (kMerge && !q.cont) {
                const int32_t filled = min(ct_end, ct + kFillTiles);
                ok = scan(std::true_type(), ct, filled);
                ct = filled;
            }
            if (ok) ok = scan(std::false_type(), ct, ct_end);
            if (!ok) break;
            // The item read again: its rows, its flags and where its lists go are not
            // held in registers over the sweep (the barrier keeps the two reads apart).
            int32_t again = it;
            asm volatile("" : "+r"(again));
            const TcItem o = work[again];
            const int64_t grow = o.row0 + row_in_tile;
            const bool seed = (o.flags & kTcSeed) != 0;
            if ((o.flags & kTcMore) && !seed) continue;  // the next item extends this tile
            flush(ls, li, worst, qoff);
            if (seed) {
                // R candidates score `worst` or better, so that the row's R best do:
                // entries from the next larger score on are as good as empty ones.
                const float bound = worst < FLT_MAX ? nextafterf(worst, FLT_MAX) : FLT_MAX;
#pragma unroll
                for (int t = 0; t < R; ++t) {
                    ls[t] = bound;
                    li[t] = -1;
                }
                if (grow < o.qend) worst = bound;
                continue;
            }
            if (grow < o.qend) {
                const int64_t orow = row_map ? (int64_t)row_map[grow] : grow + o.out_off;
                int32_t *out = cand_i + orow * R;
                if (lists.count > 0 && grow >= lists.row0) {
                    const int64_t at = ((grow - lists.row0) * lists.count + o.slot) * R;
                    out = lists.idx + at;
#pragma unroll
                    for (int t = 0; t < R; ++t) lists.score[at + t] = ls[t];
                }
#pragma unroll
                for (int t = 0; t < R; ++t)
                    out[t] = li[t] < 0 ? -1
                                       : (row_map ? row_map[li[t]] : (int32_t)(li[t] + o.out_off));
            }
        }
    }
    __syncthreads();
    if (warp == 1) {
        tmem_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(kTmemCols));
    }
}

// The driver's tensor-map encoder, looked up once (thread-safe static
// initialisation; a failed lookup throws and is retried on the next call).
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        NCVIS_CUDA(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000,
                                                    cudaEnableDefault, &q));
        require(q == cudaDriverEntryPointSuccess && p != nullptr,
                "knn: cuTensorMapEncodeTiled is unavailable", kCudaError);
        return (PFN_cuTensorMapEncodeTiled_v12000)p;
    }();
    return fn;
}

}  // namespace

KnnTcPlan plan_knn_tc(int64_t N, int D, int k, int rerank_factor, int dist) {
    KnnTcPlan p;
    // Default: 2k candidates (32 for k = 15), which measured recall@15 = 1.0
    // against FP64 search at 1,024,000 x 100; rerank_factor = 4 keeps 64.
    if (rerank_factor <= 0) rerank_factor = 2;
    const int64_t want = std::max<int64_t>((int64_t)rerank_factor * k, (int64_t)k + 1);
    p.R = want <= 32 ? 32 : 64;  // the kernel keeps 32 or 64 candidates per point
    // Squared L2 folds -|c|^2 / 2 into two extra K columns when they fit (D <= 126).
    p.fold = (dist == kSquaredL2) && D + 2 <= 64 * kMaxAtoms;
    p.ldb = (D + (p.fold ? 2 : 0) + 7) / 8 * 8;
    (void)N;
    return p;
}

KnnTcPlan plan_knn_split(int D, int R, int dist) {
    KnnTcPlan p;
    p.parts = 2;
    p.R = R <= 32 ? 32 : 64;
    // Squared L2 folds -|c|^2 / 2 into three extra columns.
    p.fold = dist == kSquaredL2;
    p.ldb = (D + (p.fold ? 3 : 0) + 7) / 8 * 8;
    return p;
}

// Scores against 64 bits (rms over 500 queries' 32 best of 20,000, the three
// products against K3's FP32 sums): 0.46 to 0.94 times K3's error for 8 to 126
// columns, raw and unit rows, products and squared L2; 1.04 times at 4 columns
// and 1.4 at 2 (the parts' own rounding), which therefore stay on the CUDA cores.
constexpr int kSplitMinCols = 8;

bool knn_split_supported(int64_t N, int D, int R, int dist) {
    return N < (int64_t(1) << 30) && R <= 64 && D >= kSplitMinCols &&
           D + (dist == kSquaredL2 ? 3 : 0) <= 64 * kMaxAtoms;
}

TcSweep plan_sweep(int64_t N, int ctas) {
    TcSweep w;
    const int64_t n_qt = (N + kQueryTile - 1) / kQueryTile, n_ct = (N + kCandTile - 1) / kCandTile;
    w.full_qt = n_qt / ctas * ctas;
    const int64_t left = n_qt - w.full_qt;
    w.ctas = ctas;
    if (left == 0) return w;
    // The last wave's tiles whole, in p equal runs each (of at least two candidate
    // tiles, and a sixth of a sweep), or in ctas equal runs, which then mostly reach
    // over two tiles and fill two sets of lists: filling one from nothing takes
    // about as long as scanning kFill candidate tiles afterwards.  Selection in us,
    // whole / p runs / ctas runs, before lists were filled by merging: 10,000 x 64 BF16
    // (40 tiles, p = 3) 271 / 183 / 243, 131,072 x 100 (56 left, p = 2) 4,255 / 3,918 /
    // 4,081, 20,000 x 100 (79) 386 / - / 420, 32,768 x 100 (128) 487 / - / 885, 60,013 x
    // 100 FP32 (83 left) 2,082 / - / 1,838, 30,000 x 100 FP32 (118) 595 / - / 650; since
    // then 131,072 x 100 - / 3,786 / 3,600.  A last wave more than three
    // quarters full stays whole: 500,000 x 64 (130 left) 39.1 ms whole, 40.4 in runs
    // (300,000 x 100, 108 left, 18.8 and 18.7).
    constexpr int64_t kFill = 100;
    const int64_t rest = left * n_ct;
    const int64_t p = std::max<int64_t>(1, std::min<int64_t>({ctas / left, 6, n_ct / 2}));
    int64_t G = p * left, cost = n_ct / p + kFill;
    if (ctas > G && 4 * left < 3 * ctas && ctas <= 6 * left && ctas <= rest / 2 && rest / ctas + 2 * kFill < cost) G = ctas;
    if (G == left) return whole_tiles(N, ctas);
    w.rest_ctas = (int)G;
    if (w.full_qt == 0) w.ctas = w.rest_ctas;
    const TcRun run(N, w);
    for (int64_t t = 0; t < left; ++t)
        w.lists = std::max<int>(w.lists, (int)(run.last_cta(t) - run.first_cta(t) + 1));
    w.split_rows = N - w.full_qt * kQueryTile;
    return w;
}

TcSweep whole_tiles(int64_t N, int ctas) {
    TcSweep w;
    w.full_qt = (N + kQueryTile - 1) / kQueryTile;
    w.ctas = (int)std::min<int64_t>(w.full_qt, ctas);
    return w;
}

namespace {

size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

// The best `keep` of a split row's lists, a warp a row: every entry's place is its
// own in its list and, by a binary search in each other one, the number of entries
// before it there (equal scores: those of the lists before its own).  Bound by the
// latency of the searches' steps: 14,336 rows x 2 lists 9 us, 10,000 x 3 11 us, 6,144
// x 7 22 us; re-ranking all the lists instead took 100 us more at 10,000 x 3.
template <int R>
__global__ void __launch_bounds__(128) merge_lists(int64_t N, TcSweep w, TcLists lists, int keep,
                                                   const int32_t *__restrict__ order,
                                                   int32_t *__restrict__ cand_i) {
    extern __shared__ float scores[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t row = lists.row0 + (int64_t)blockIdx.x * (blockDim.x >> 5) + warp;
    if (row >= N) return;
    const TcRun run(N, w);
    const int64_t tile = row / kQueryTile - w.full_qt;
    const int n = (int)(run.last_cta(tile) - run.first_cta(tile)) + 1;
    const int64_t at = (row - lists.row0) * lists.count * R;
    float *sc = scores + (size_t)warp * lists.count * R;
    for (int c = lane; c < n * R; c += 32) sc[c] = lists.score[at + c];
    __syncwarp();
    int32_t *out = cand_i + (order ? (int64_t)order[row] : row) * keep;
    for (int c = lane; c < n * R; c += 32) {
        const int a = c / R;
        const float x = sc[c];
        int place = c % R;
        for (int b = 0; b < n; ++b) {
            if (b == a) continue;
            const float *y = sc + b * R;
            int before = 0;
#pragma unroll
            for (int step = R; step > 0; step >>= 1) {
                const int i = before + step - 1;
                if (i < R && (b < a ? y[i] <= x : y[i] < x)) before += step;
            }
            place += before;
        }
        if (place < keep) out[place] = lists.idx[at + c];
    }
    for (int c = n * R + lane; c < keep; c += 32) out[c] = -1;
}

}  // namespace

size_t sweep_lists_bytes(const TcSweep &w, int R) {
    return w.lists > 1 ? 2 * align256(sizeof(int32_t) * (size_t)w.split_rows * w.lists * R) : 0;
}

size_t sweep_bytes(int64_t N, const TcSweep &w, int R) {
    return sweep_lists_bytes(w, R) +
           align256(16 * (((size_t)w.ctas + 1) / 2 * 2) +
                    sizeof(TcItem) * (size_t)w.ctas * sweep_stride(N, w));
}

TcLists sweep_lists(int64_t N, const TcSweep &w, int R, void *workspace) {
    TcLists l;
    if (w.lists <= 1) return l;
    l.count = w.lists;
    l.row0 = N - w.split_rows;
    l.idx = (int32_t *)workspace;
    l.score = (float *)((char *)workspace + sweep_lists_bytes(w, R) / 2);
    return l;
}

TcWork launch_sweep_work(int64_t N, const TcSweep &w, int R, void *workspace, cudaStream_t s) {
    TcWork work;
    work.ctas = w.ctas;
    work.lists = sweep_lists(N, w, R, workspace);
    int64_t *begin = (int64_t *)((char *)workspace + sweep_lists_bytes(w, R));
    int64_t *end = begin + (w.ctas + 1) / 2 * 2;
    TcItem *items = (TcItem *)(end + (w.ctas + 1) / 2 * 2);
    NCVIS_LAUNCH(sweep_items, (unsigned)w.ctas, 32, 0, s, N, w, sweep_stride(N, w), begin, end,
                 items);
    work.begin = begin;
    work.end = end;
    work.items = items;
    work.fill = N < kFillMaxRows;
    return work;
}

void launch_merge_lists(int64_t N, const TcSweep &w, const TcLists &lists, int R, int keep,
                        const int32_t *order, int32_t *cand_i, cudaStream_t s) {
    if (lists.count == 0) return;
    require(R == 32 || R == 64, "knn: lists of 32 or 64 candidates", kInternal);
    require(!order || keep <= R, "knn: more candidates than seeded lists hold", kInternal);
    const int warps = 4;
    const size_t smem = sizeof(float) * warps * lists.count * R;  // at most 8 lists: 8 KB
    const unsigned grid = (unsigned)ceil_div(N - lists.row0, warps);
    if (R == 32)
        NCVIS_LAUNCH(merge_lists<32>, grid, warps * 32, smem, s, N, w, lists, keep, order, cand_i);
    else
        NCVIS_LAUNCH(merge_lists<64>, grid, warps * 32, smem, s, N, w, lists, keep, order, cand_i);
}

bool knn_tc_supported(int D, int R) { return D >= 1 && D <= 64 * kMaxAtoms && (R == 32 || R == 64); }


namespace {

void encode_rows(const void *base, int64_t rows, int ldb, bool half, CUtensorMap &map) {
    cuuint64_t dims[2] = {(cuuint64_t)ldb, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ldb * 2};
    cuuint32_t box[2] = {64, 128};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = tensor_map_encoder()(&map,
                                      half ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16
                                           : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16,
                                      2, (void *)base,
                                      dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      CU_TENSOR_MAP_SWIZZLE_128B,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    require(r == CUDA_SUCCESS,
            "knn: cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")", kCudaError);
}

void launch_select(const CUtensorMap &map, const CUtensorMap &map_c, const TcParts &parts,
                   const float *sqnorm, const KnnTcPlan &plan, bool ip, int32_t *cand_i,
                   int *timeout_flag, cudaStream_t s, const TcWork &work) {
    const int ksteps = (plan.ldb + 15) / 16;
    const int katoms = (ksteps * 16 + 63) / 64;
    const unsigned grid = (unsigned)work.ctas;
    if (grid == 0) return;
    auto go = [&](auto kernel, size_t shared) {
        const size_t smem = shared + 1024;
        NCVIS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
        NCVIS_LAUNCH(kernel, grid, kThreads, smem, s, map, map_c, parts, sqnorm, ksteps, katoms,
                     plan.low_low ? ksteps : kLowLowSteps, work.begin, work.end, work.items, work.map, cand_i, work.lists, timeout_flag,
                     plan.wait_cycles > 0 ? plan.wait_cycles : kWaitCycles, plan.stall ? 1 : 0);
    };
    constexpr size_t one = sizeof(SharedStorage<1>), two = sizeof(SharedStorage<2>);
    if (plan.parts == 2) {
        if (plan.R == 64)
            go(knn_select_tc<64, true, 2, false>, two);
        else if (work.fill)
            go(knn_select_tc<32, true, 2, true>, two);
        else
            go(knn_select_tc<32, true, 2, false>, two);
    } else if (plan.R == 1) {
        go(knn_select_tc<1, true, 1, false>, one);
    } else if (plan.R == 64) {
        ip ? go(knn_select_tc<64, true, 1, false>, one) : go(knn_select_tc<64, false, 1, false>, one);
    } else if (!ip) {
        go(knn_select_tc<32, false, 1, true>, one);
    } else if (work.fill) {
        go(knn_select_tc<32, true, 1, true>, one);
    } else {
        go(knn_select_tc<32, true, 1, false>, one);
    }
}

void check_plan(const KnnTcPlan &plan) {
    const int ksteps = (plan.ldb + 15) / 16;
    const int katoms = (ksteps * 16 + 63) / 64;
    require(katoms <= kMaxAtoms, "knn: the tensor-core path supports D <= 128", kUnsupported);
    require(plan.R == 1 || plan.R == 32 || plan.R == 64,
            "knn: the tensor-core kernel keeps 1, 32 or 64 candidates");
}

}  // namespace

void launch_knn_select_tc(const __nv_bfloat16 *Xb, const float *sqnorm, int64_t N,
                          const KnnTcPlan &plan, int dist, int32_t *cand_i, int *timeout_flag,
                          cudaStream_t s, const TcWork &work, const __nv_bfloat16 *Xc) {
    require(N < (int64_t(1) << 31), "knn: N must be below 2^31");
    check_plan(plan);
    require(((uintptr_t)Xb & 15) == 0, "knn: BF16 rows must be 16-byte aligned");
    require(((uintptr_t)sqnorm & 15) == 0, "knn: squared norms must be 16-byte aligned");
    require(!plan.fold || (Xc && ((uintptr_t)Xc & 15) == 0),
            "knn: the folded squared-L2 mode needs a 16-byte aligned candidate copy");
    // Queries come from Xb, candidates from Xc in the folded mode (else Xb).
    CUtensorMap map, map_c;
    encode_rows(Xb, N, plan.ldb, false, map);
    encode_rows(plan.fold ? Xc : Xb, N, plan.ldb, false, map_c);
    // The folded squared-L2 product <q, c> - |c|^2 / 2 ranks like an inner product.
    const bool ip = dist != kSquaredL2 || plan.fold;
    launch_select(map, map_c, TcParts{}, sqnorm, plan, ip, cand_i, timeout_flag, s, work);
}

void launch_knn_select_split(const __half *rows, int64_t N, const KnnTcPlan &plan,
                             int32_t *cand_i, int *timeout_flag, cudaStream_t s,
                             const TcWork &work) {
    require(plan.parts == 2 && N < (int64_t(1) << 30), "knn: N must be below 2^30");
    check_plan(plan);
    require(((uintptr_t)rows & 15) == 0, "knn: FP16 rows must be 16-byte aligned");
    // Blocks of N rows: the high parts, the low parts and, folded, the
    // candidates' high parts; the candidates' map starts at the low parts then.
    const int32_t n = (int32_t)N;
    CUtensorMap map, map_c;
    encode_rows(rows, 2 * N, plan.ldb, true, map);
    encode_rows(plan.fold ? rows + (size_t)N * plan.ldb : rows, 2 * N, plan.ldb, true, map_c);
    const TcParts parts = plan.fold ? TcParts{{0, n}, {n, 0}} : TcParts{{0, n}, {0, n}};
    launch_select(map, map_c, parts, nullptr, plan, true, cand_i, timeout_flag, s, work);
}

void launch_knn_select_tc_pair(const __nv_bfloat16 *Q, int64_t nq, const __nv_bfloat16 *Cm,
                               int64_t nc, const float *c_sqnorm, const KnnTcPlan &plan, bool ip,
                               int32_t *cand_i, int *timeout_flag, cudaStream_t s,
                               const TcWork &work) {
    require(nq < (int64_t(1) << 31) && nc < (int64_t(1) << 31), "knn: rows must be below 2^31");
    check_plan(plan);
    require((((uintptr_t)Q | (uintptr_t)Cm) & 15) == 0, "knn: BF16 rows must be 16-byte aligned");
    require(ip || (c_sqnorm && ((uintptr_t)c_sqnorm & 15) == 0),
            "knn: squared L2 without folded norms needs 16-byte aligned candidate norms");
    CUtensorMap map, map_c;
    encode_rows(Q, nq, plan.ldb, false, map);
    encode_rows(Cm, nc, plan.ldb, false, map_c);
    launch_select(map, map_c, TcParts{}, c_sqnorm, plan, ip, cand_i, timeout_flag, s, work);
}

}  // namespace ncvis_gpu
