// K6: NCVis::init_embedding (src/ncvis.cpp:184-273) over the CSR graph.
//
//   Y ~ U(0,1), element t from draw t of the one-thread pcg64(seed) stream
//       (src/ncvis.cpp:195-200); each thread jumps to its own offset;
//   repeat n_init_epochs times (src/ncvis.cpp:203-261):
//       Y_new[i] = sum over row i, in CSR order, of alpha * Y_old[j]
//                  (FP32, multiply then add as the reference's build does: no
//                  fused multiply-add);
//       mean, population std per dimension (FP64 block partial sums, cast to
//       FP32 and divided by N in FP32 as the reference does; or, on request,
//       the reference's one-thread FP32 sums in row order, whose rounding
//       drifts ~1e-4 relative from the exact statistics at a million rows);
//       Y_new = (Y_new - mean) / sigma;
//   ping-pong buffers, result left in Y (src/ncvis.cpp:262-267).
// An epoch is three launches: the sums and the mean, the deviation, and the
// standardisation; a statistic is finished by the last block of its launch.
#include <algorithm>
#include <cfloat>

#include "common.cuh"
#include "rng.cuh"
#include "stages.cuh"

namespace ncvis_gpu {

namespace {

constexpr int kThreads = 256;
constexpr int kMaxDim = 32;  // dimensions held in registers by the row kernels

// n = N d draws into rows of `pitch` floats.
__global__ void uniform_init(float *__restrict__ Y, int64_t n, int d, int pitch, uint64_t seed,
                             int per_thread) {
    const int64_t t0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) * per_thread;
    if (t0 >= n) return;
    Pcg64 g(seed);
    g.advance((uint64_t)t0);
    const int64_t t1 = min(n, t0 + per_thread);
    for (int64_t t = t0; t < t1; ++t)
        Y[pitch == d ? t : t / d * pitch + t % d] = unit_float(g.next());
}

// Rows of the internal buffers, P floats apart: d = 3 is padded to 4, so that a
// row is one 16-byte load that lies in one sector.
template <int D>
constexpr int kPitch = D == 3 ? 4 : D;

template <int D>
struct RowVec {
    float v[D];
};

template <int D>
__device__ __forceinline__ RowVec<D> load_row(const float *__restrict__ Y, int64_t i) {
    RowVec<D> r;
    if constexpr (D == 1) {
        r.v[0] = __ldg(Y + i);
    } else if constexpr (D == 2) {
        const float2 t = __ldg(reinterpret_cast<const float2 *>(Y) + i);
        r.v[0] = t.x, r.v[1] = t.y;
    } else {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(Y) + i);
        r.v[0] = t.x, r.v[1] = t.y, r.v[2] = t.z;
        if constexpr (D == 4) r.v[3] = t.w;
    }
    return r;
}

template <int D>
__device__ __forceinline__ void store_row(float *__restrict__ Y, int64_t i, const RowVec<D> &r) {
    if constexpr (D == 1) {
        Y[i] = r.v[0];
    } else if constexpr (D == 2) {
        reinterpret_cast<float2 *>(Y)[i] = make_float2(r.v[0], r.v[1]);
    } else {
        float w = 0.f;
        if constexpr (D == 4) w = r.v[3];
        reinterpret_cast<float4 *>(Y)[i] = make_float4(r.v[0], r.v[1], r.v[2], w);
    }
}

// Which rows a block handles and whose statistics they are: one problem of N
// rows, block b rows [b * rows, ..); or B problems, problem p owning rows
// [off[p], off[p+1]) and blocks [tp[p], tp[p+1]).
struct RowBlocks {
    int64_t N, rows;
    const int64_t *off, *tp;
    int B;
};
struct BlockRows {
    int64_t row, end;       // the block's rows
    int64_t first, blocks;  // its problem's blocks
    int64_t n;              // and points
    int problem;
};
__device__ __forceinline__ BlockRows block_rows(const RowBlocks &w) {
    BlockRows r;
    if (w.off) {
        const int p = segment_of(w.tp, w.B, blockIdx.x);
        r.problem = p;
        r.first = w.tp[p];
        r.blocks = w.tp[p + 1] - w.tp[p];
        r.row = w.off[p] + ((int64_t)blockIdx.x - r.first) * w.rows;
        r.n = w.off[p + 1] - w.off[p];
        r.end = min(w.off[p + 1], r.row + w.rows);
    } else {
        r.problem = 0;
        r.first = 0;
        r.blocks = gridDim.x;
        r.row = (int64_t)blockIdx.x * w.rows;
        r.n = w.N;
        r.end = min(w.N, r.row + w.rows);
    }
    return r;
}

// stat[c] of one problem from its blocks' FP64 sums, by the last of them to
// arrive: kMean the sum / n, else sqrt(sum / n), in FP32 as the reference does.
// Every block leaves its sums in part; the last one adds them up in the order of
// the blocks, so the result does not depend on who is last.  sum: in thread
// c < d the block's sum of dimension c.
template <bool kMean>
__device__ __forceinline__ void finish_stat(int d, double sum, double *__restrict__ part,
                                            int *__restrict__ done, const BlockRows &b,
                                            float *__restrict__ stat) {
    __shared__ double red[kThreads / 32];
    __shared__ bool last;
    if (threadIdx.x < d) {
        part[(int64_t)blockIdx.x * d + threadIdx.x] = sum;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done + b.problem, 1) == (int)b.blocks - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = 0; c < d; ++c) {
        double s = 0.0;
        for (int64_t t = threadIdx.x; t < b.blocks; t += kThreads)
            s += __ldcg(part + (b.first + t) * d + c);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) red[warp] = s;
        __syncthreads();
        if (threadIdx.x == 0) {
            s = 0.0;
            for (int w = 0; w < kThreads / 32; ++w) s += red[w];
            const float v = __fdiv_rn((float)s, (float)b.n);
            stat[b.problem * d + c] = kMean ? v : sqrtf(v);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) done[b.problem] = 0;  // for the next statistic
}

// A sum held as two FP32 numbers, hi + lo to about 48 bits (Knuth's TwoSum): the
// statistics' FP64 sums up to a warp's are formed in it, because an FP64 add of a
// warp takes 16 cycles of an SM here, which with the conversions was 13 of the
// deviation pass's 20 us at 500,001 x 3.
// kSquares: where the sum leaves FP32's range it is infinite, as an FP64 one is by the
// time it is rounded, not the NaN that the parts' differences make (a sum of values
// that leaves it makes the mean infinite or NaN, and either every row NaN).
template <bool kSquares>
struct Sum2 {
    float hi = 0.f, lo = 0.f;
    __device__ __forceinline__ void add(float h, float l) {
        const float s = __fadd_rn(hi, h);
        const float t = __fsub_rn(s, hi);
        const float e = __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(h, t));
        const float r = __fadd_rn(e, __fadd_rn(lo, l));
        const bool keep = kSquares && !(s <= FLT_MAX);
        hi = keep ? s : __fadd_rn(s, r);
        lo = keep ? 0.f : __fsub_rn(r, __fsub_rn(hi, s));
    }
};

// Thread c < D gets the block's sum of sum[c]: over the warps' lanes, then over
// the warps in FP64.
template <int D, bool kSquares>
__device__ __forceinline__ double block_sum(Sum2<kSquares> (&sum)[D]) {
    __shared__ double red[D][kThreads / 32];
#pragma unroll
    for (int c = 0; c < D; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float h = __shfl_xor_sync(0xffffffffu, sum[c].hi, o);
            const float l = __shfl_xor_sync(0xffffffffu, sum[c].lo, o);
            sum[c].add(h, l);
        }
        if ((threadIdx.x & 31) == 0)
            red[c][threadIdx.x >> 5] = (double)sum[c].hi + (double)sum[c].lo;
    }
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < D)
        for (int w = 0; w < kThreads / 32; ++w) s += red[threadIdx.x][w];
    return s;
}

// One init epoch's neighbour sums for d <= 4 and their means, one thread per row:
// the columns and then the rows of eight edges are loaded together before they
// are added in CSR order.  Bound by the L2's 32-byte sectors, one per gathered
// row, at 25 M edges (130 us at 1,000,000 x 2, 6.3 TB/s of sectors).  Tried and not
// kept at that size: 16-byte loads of the columns (159 us), the next columns in
// flight during the gathers (183), 8 lanes per row with the values passed round by
// shuffles (226), long rows by whole warps (147).
constexpr int kStep = 8;

template <int D>
__device__ __forceinline__ RowVec<D> row_sum(int64_t p0, int64_t p1,
                                             const int32_t *__restrict__ cols, float alpha,
                                             const float *__restrict__ Yold) {
    RowVec<D> acc{};
    for (int64_t p = p0; p < p1; p += kStep) {
        int32_t col[kStep];
#pragma unroll
        for (int u = 0; u < kStep; ++u) col[u] = p + u < p1 ? __ldg(cols + p + u) : -1;
        RowVec<D> y[kStep];
#pragma unroll
        for (int u = 0; u < kStep; ++u)
            if (col[u] >= 0) y[u] = load_row<D>(Yold, col[u]);
#pragma unroll
        for (int u = 0; u < kStep; ++u)
            if (col[u] >= 0) {
#pragma unroll
                for (int c = 0; c < D; ++c)
                    acc.v[c] = __fadd_rn(acc.v[c], __fmul_rn(alpha, y[u].v[c]));
            }
    }
    return acc;
}

template <int D>
__global__ void __launch_bounds__(kThreads) spmm_mean(
    RowBlocks blocks, const int64_t *__restrict__ row_ptr, const int32_t *__restrict__ cols,
    float alpha, const float *__restrict__ Yold, float *__restrict__ Ynew,
    double *__restrict__ part, int *__restrict__ done, float *__restrict__ mean) {
    const BlockRows b = block_rows(blocks);
    const int64_t i = b.row + threadIdx.x;
    Sum2<false> sum[D];
    if (i < b.end) {
        const RowVec<D> acc = row_sum<D>(row_ptr[i], row_ptr[i + 1], cols, alpha, Yold);
        store_row<D>(Ynew, i, acc);
#pragma unroll
        for (int c = 0; c < D; ++c) sum[c].hi = acc.v[c];
    }
    finish_stat<true>(D, block_sum(sum), part, done, b, mean);
}

// The same for few rows, where the longest row is what an epoch waits for: a row's
// next columns are loaded while the eight before them are gathered, 16 bytes at a
// time (kVec: cols 16-byte aligned), and rows of more than kLong columns (hubs) are
// listed and taken by the block's warps afterwards, one warp each with 128 columns
// in flight, the values passed round by shuffles to be added in the same order.
// 10,000 x 64 Gaussian mixture, whose hubs have up to 800 edges: 23 us an epoch by
// spmm_mean, 15 so; 48 such problems of 230,000 rows in all 63 and 50; 300,000 rows
// without long hubs 43.7 and 44.8, and 1,000,000 130 and 232.
constexpr int kLong = 64, kLongStep = 4;
constexpr int64_t kShareRows = 300000;

template <bool kVec>
__device__ __forceinline__ void load_cols(int32_t (&col)[kStep], const int32_t *__restrict__ cols,
                                          int64_t p, int64_t p0, int64_t p1, int64_t E) {
    if constexpr (kVec) {
#pragma unroll
        for (int v = 0; v < kStep / 4; ++v) {
            const int64_t at = p + 4 * v;
            int4 t = make_int4(-1, -1, -1, -1);
            if (at < p1) {
                if (at + 4 <= E) {
                    t = __ldg(reinterpret_cast<const int4 *>(cols + at));
                } else {  // the array's last few columns
                    t.x = __ldg(cols + at);
                    if (at + 1 < E) t.y = __ldg(cols + at + 1);
                    if (at + 2 < E) t.z = __ldg(cols + at + 2);
                }
            }
            const int32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
                col[4 * v + u] = at + u >= p0 && at + u < p1 ? w[u] : -1;
        }
    } else {
#pragma unroll
        for (int u = 0; u < kStep; ++u) col[u] = p + u < p1 ? __ldg(cols + p + u) : -1;
    }
}

// A long row by one warp: acc the same in every lane.
template <int D>
__device__ __forceinline__ RowVec<D> long_row_sum(int64_t p0, int n, const int32_t *__restrict__ cols,
                                                  float alpha, const float *__restrict__ Yold) {
    const int lane = threadIdx.x & 31;
    RowVec<D> acc{};
    for (int q = 0; q < n; q += 32 * kLongStep) {
        int32_t col[kLongStep];
        RowVec<D> y[kLongStep];
#pragma unroll
        for (int u = 0; u < kLongStep; ++u) {
            const int e = q + u * 32 + lane;
            col[u] = e < n ? __ldg(cols + p0 + e) : -1;
        }
#pragma unroll
        for (int u = 0; u < kLongStep; ++u) {
            y[u] = RowVec<D>{};
            if (col[u] >= 0) y[u] = load_row<D>(Yold, col[u]);
#pragma unroll
            for (int c = 0; c < D; ++c) y[u].v[c] = __fmul_rn(alpha, y[u].v[c]);
        }
#pragma unroll
        for (int u = 0; u < kLongStep; ++u) {
            const int m = min(32, n - (q + u * 32));
#pragma unroll 8
            for (int e = 0; e < m; ++e) {
#pragma unroll
                for (int c = 0; c < D; ++c)
                    acc.v[c] = __fadd_rn(acc.v[c], __shfl_sync(0xffffffffu, y[u].v[c], e));
            }
        }
    }
    return acc;
}

template <int D, bool kVec>
__global__ void __launch_bounds__(kThreads) spmm_mean_share(
    RowBlocks blocks, const int64_t *__restrict__ row_ptr, int64_t n_rows,
    const int32_t *__restrict__ cols, float alpha, const float *__restrict__ Yold,
    float *__restrict__ Ynew, double *__restrict__ part, int *__restrict__ done,
    float *__restrict__ mean) {
    constexpr int kWarps = kThreads / 32;
    __shared__ int64_t long_row[kThreads];
    __shared__ int n_long[kWarps];
    const BlockRows b = block_rows(blocks);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Sum2<false> sum[D];
    auto finish = [&](int64_t i, const RowVec<D> &acc) {
        store_row<D>(Ynew, i, acc);
#pragma unroll
        for (int c = 0; c < D; ++c) sum[c].add(acc.v[c], 0.f);
    };
    const int64_t i = b.row + threadIdx.x;
    const int64_t p0 = i < b.end ? row_ptr[i] : 0, p1 = i < b.end ? row_ptr[i + 1] : 0;
    const bool is_long = p1 - p0 > kLong;
    const unsigned longs = __ballot_sync(0xffffffffu, is_long);
    if (lane == 0) n_long[warp] = __popc(longs);
    if (!is_long && i < b.end) {
        const int64_t E = kVec ? row_ptr[n_rows] : 0;
        RowVec<D> acc{};
        int32_t col[kStep];
        int64_t p = kVec ? p0 & ~(int64_t)3 : p0;
        load_cols<kVec>(col, cols, p, p0, p1, E);
        for (; p < p1; p += kStep) {
            RowVec<D> y[kStep];
#pragma unroll
            for (int u = 0; u < kStep; ++u)
                if (col[u] >= 0) y[u] = load_row<D>(Yold, col[u]);
            int32_t next[kStep];
            load_cols<kVec>(next, cols, p + kStep, p0, p1, E);
#pragma unroll
            for (int u = 0; u < kStep; ++u) {
                if (col[u] >= 0) {
#pragma unroll
                    for (int c = 0; c < D; ++c)
                        acc.v[c] = __fadd_rn(acc.v[c], __fmul_rn(alpha, y[u].v[c]));
                }
                col[u] = next[u];
            }
        }
        finish(i, acc);
    }
    // The long rows, listed in the order of the rows.
    __syncthreads();
    int before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
        before += w < warp ? n_long[w] : 0;
        all += n_long[w];
    }
    if (is_long) long_row[before + __popc(longs & ((1u << lane) - 1u))] = i;
    __syncthreads();
    for (int t = warp; t < all; t += kWarps) {
        const int64_t li = long_row[t], lp = row_ptr[li];
        const RowVec<D> acc = long_row_sum<D>(lp, (int)(row_ptr[li + 1] - lp), cols, alpha, Yold);
        if (lane == 0) finish(li, acc);
    }
    finish_stat<true>(D, block_sum(sum), part, done, b, mean);
}

// sigma from the rows and their mean: (y - mean)^2 rounded to FP32 as the
// reference's terms are, summed in FP64.
template <int D>
__global__ void __launch_bounds__(kThreads) centred_sigma(RowBlocks blocks,
                                                          const float *__restrict__ Y,
                                                          const float *__restrict__ mean,
                                                          double *__restrict__ part,
                                                          int *__restrict__ done,
                                                          float *__restrict__ sigma) {
    const BlockRows b = block_rows(blocks);
    Sum2<true> sum[D];
    float m[D];
#pragma unroll
    for (int c = 0; c < D; ++c) m[c] = mean[b.problem * D + c];
    for (int64_t i = b.row + threadIdx.x; i < b.end; i += kThreads) {
        const RowVec<D> y = load_row<D>(Y, i);
#pragma unroll
        for (int c = 0; c < D; ++c) {
            const float dev = __fsub_rn(y.v[c], m[c]);
            sum[c].add(__fmul_rn(dev, dev), 0.f);
        }
    }
    finish_stat<false>(D, block_sum(sum), part, done, b, sigma);
}

// The two for any d, one thread per row and dimension: neighbouring threads read
// one neighbour's row together.  Thread c < d gets the block's sum.
__device__ __forceinline__ double block_sum_any(int d, double sum) {
    __shared__ double all[kThreads];
    all[threadIdx.x] = sum;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < d)
        for (int t = 0; t < kThreads / d; ++t) s += all[t * d + threadIdx.x];
    return s;
}

__global__ void __launch_bounds__(kThreads) spmm_mean_any(
    RowBlocks blocks, int d, const int64_t *__restrict__ row_ptr,
    const int32_t *__restrict__ cols, float alpha, const float *__restrict__ Yold,
    float *__restrict__ Ynew, double *__restrict__ part, int *__restrict__ done,
    float *__restrict__ mean) {
    const BlockRows b = block_rows(blocks);
    const int per = kThreads / d, r = threadIdx.x / d, c = threadIdx.x - r * d;
    double sum = 0.0;
    if (r < per) {
        for (int64_t i = b.row + r; i < b.end; i += per) {
            float acc = 0.f;
            const int64_t p1 = row_ptr[i + 1];
#pragma unroll 8
            for (int64_t p = row_ptr[i]; p < p1; ++p)
                acc = __fadd_rn(acc,
                                __fmul_rn(alpha, __ldg(Yold + (int64_t)__ldg(cols + p) * d + c)));
            Ynew[i * d + c] = acc;
            sum += (double)acc;
        }
    }
    finish_stat<true>(d, block_sum_any(d, sum), part, done, b, mean);
}

__global__ void __launch_bounds__(kThreads) centred_sigma_any(RowBlocks blocks, int d,
                                                              const float *__restrict__ Y,
                                                              const float *__restrict__ mean,
                                                              double *__restrict__ part,
                                                              int *__restrict__ done,
                                                              float *__restrict__ sigma) {
    const BlockRows b = block_rows(blocks);
    const int per = kThreads / d, r = threadIdx.x / d, c = threadIdx.x - r * d;
    double sum = 0.0;
    if (r < per) {
        const float m = mean[b.problem * d + c];
        for (int64_t i = b.row + r; i < b.end; i += per) {
            const float dev = __fsub_rn(Y[i * d + c], m);
            sum += (double)__fmul_rn(dev, dev);
        }
    }
    finish_stat<false>(d, block_sum_any(d, sum), part, done, b, sigma);
}

// The reference's one-thread statistics (src/ncvis.cpp:226-254 on one
// thread): per dimension an FP32 sum over the rows in order, mode 0 of the
// values (stat = sum / N), mode 1 of (y - mean)^2 (stat = sqrt(sum / N)).
// One block: all threads stage chunks of rows into shared memory with
// asynchronous copies, the next chunk in flight while lane c < d adds up
// dimension c of the current one; the adds form one dependent chain per
// dimension (N FP32 adds, ~2 ms per pass at a million rows).
constexpr int kSeqFloats = 8192;  // floats per staged chunk (32 KB; whole rows)

__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(dst)),
                 "l"(src)
                 : "memory");
}

__global__ void __launch_bounds__(kThreads) sequential_stat(const float *__restrict__ Y, int64_t N,
                                                            int d, int mode,
                                                            const float *__restrict__ mean,
                                                            float *__restrict__ stat) {
    extern __shared__ float chunk[];  // [2][rows_per * d]
    const int64_t rows_per = kSeqFloats / d;
    const int64_t per = rows_per * d;
    const int64_t n = N * d;
    const int64_t chunks = (n + per - 1) / per;
    auto issue = [&](int64_t k) {
        float *dst = chunk + (k & 1) * per;
        const int64_t base = k * per;
        const int64_t len = min(per, n - base);
        for (int64_t t = threadIdx.x; t < len; t += blockDim.x) cp_async4(dst + t, Y + base + t);
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int c = threadIdx.x;
    const float m = (mode == 1 && c < d) ? mean[c] : 0.f;
    float s = 0.f;
    issue(0);
    for (int64_t k = 0; k < chunks; ++k) {
        if (k + 1 < chunks) {
            issue(k + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        if (c < d) {
            const float *v = chunk + (k & 1) * per;
            const int64_t rows = min(rows_per, N - k * rows_per);
#pragma unroll 8
            for (int64_t r = 0; r < rows; ++r) {
                float t = v[r * d + c];
                if (mode == 1) {
                    t = __fsub_rn(t, m);
                    t = __fmul_rn(t, t);
                }
                s = __fadd_rn(s, t);
            }
        }
        __syncthreads();
    }
    if (c < d) {
        const float v = __fdiv_rn(s, (float)N);
        stat[c] = (mode == 0) ? v : __fsqrt_rn(v);
    }
}

// out = (Y - mean) / sigma, rows of kPitch<D> floats in and kPitch<D> or D out.
template <int D>
__global__ void __launch_bounds__(kThreads) standardize_rows(RowBlocks blocks, const float *Y,
                                                             const float *__restrict__ mean,
                                                             const float *__restrict__ sigma,
                                                             float *out, int packed) {
    const BlockRows b = block_rows(blocks);
    float m[D], s[D];
#pragma unroll
    for (int c = 0; c < D; ++c) m[c] = mean[b.problem * D + c], s[c] = sigma[b.problem * D + c];
    for (int64_t i = b.row + threadIdx.x; i < b.end; i += kThreads) {
        // Not through the read-only path: out may be Y.
        RowVec<D> y;
        const float *row = Y + i * kPitch<D>;
        if constexpr (D == 2) {
            const float2 t = *reinterpret_cast<const float2 *>(row);
            y.v[0] = t.x, y.v[1] = t.y;
        } else if constexpr (D >= 3) {
            const float4 t = *reinterpret_cast<const float4 *>(row);
            y.v[0] = t.x, y.v[1] = t.y, y.v[2] = t.z;
            if constexpr (D == 4) y.v[3] = t.w;
        } else {
            y.v[0] = row[0];
        }
#pragma unroll
        for (int c = 0; c < D; ++c) y.v[c] = __fdiv_rn(__fsub_rn(y.v[c], m[c]), s[c]);
        if (packed && kPitch<D> != D) {
#pragma unroll
            for (int c = 0; c < D; ++c) out[i * D + c] = y.v[c];
        } else {
            store_row<D>(out, i, y);
        }
    }
}

__global__ void __launch_bounds__(kThreads) standardize_any(RowBlocks blocks, int d, const float *Y,
                                                            const float *__restrict__ mean,
                                                            const float *__restrict__ sigma,
                                                            float *out) {
    const BlockRows b = block_rows(blocks);
    for (int64_t t = b.row * d + threadIdx.x; t < b.end * d; t += kThreads) {
        const int c = (int)(t % d) + b.problem * d;
        out[t] = __fdiv_rn(__fsub_rn(Y[t], mean[c]), sigma[c]);
    }
}

// ---- batched problems: problem p owns rows [off[p], off[p+1]), its own
// seed, and row tiles [tp[p], tp[p+1]) of kThreads rows each.

__global__ void uniform_init_batched(float *__restrict__ Y, int64_t total, int d, int pitch,
                                     const int64_t *__restrict__ off, int B,
                                     const uint64_t *__restrict__ seeds) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= total) return;
    const int p = segment_of(off, B, t / d);
    Pcg64 g(seeds[p]);
    g.advance((uint64_t)(t - off[p] * d));
    Y[pitch == d ? t : t / d * pitch + t % d] = unit_float(g.next());
}

inline size_t align256(size_t v) { return (v + 255) & ~(size_t)255; }

// Rows per block: a block per SM as soon as there are 32 rows each (a few long rows
// a warp), whole warps of rows up to one row a thread.
int64_t rows_per_block(int64_t N) {
    const int64_t few = (N + num_sms() - 1) / num_sms();
    return few <= kThreads ? std::max<int64_t>(1, (few + 31) / 32) * 32 : kThreads;
}

// The same for the passes over the rows alone: at most four blocks per SM.
int64_t rows_per_block_light(int64_t N) {
    const int64_t most = 4 * num_sms();
    return std::max(rows_per_block(N), (N + kThreads * most - 1) / (kThreads * most) * kThreads);
}

// Epochs of neighbour averaging and standardisation from the uniform start in
// bufs[0]; `packed` buffers hold rows of d floats, the others of kPitch<d>.  The
// result goes to Y, whichever buffer that is.
struct InitRun {
    RowBlocks blocks, light;  // of the neighbour sums, and of the passes over the rows
    unsigned grid, light_grid;
    int d, epochs;
    bool by_row;  // d <= 4, aligned rows: one thread per row
    bool share;   // long rows by all warps of the block
    const int64_t *row_ptr;
    const int32_t *cols;
    float alpha;
    double *part;
    int *done;
    float *mean, *sigma;
};

template <int D>
void epoch_by_row(const InitRun &r, const float *from, float *to, float *out, bool packed,
                  cudaStream_t s) {
    if (r.share) {
        auto go = [&](auto kernel) {
            NCVIS_LAUNCH(kernel, r.grid, kThreads, 0, s, r.blocks, r.row_ptr, r.blocks.N, r.cols,
                         r.alpha, from, to, r.part, r.done, r.mean);
        };
        ((uintptr_t)r.cols & 15) == 0 ? go(spmm_mean_share<D, true>)
                                      : go(spmm_mean_share<D, false>);
    } else {
        NCVIS_LAUNCH(spmm_mean<D>, r.grid, kThreads, 0, s, r.blocks, r.row_ptr, r.cols, r.alpha,
                     from, to, r.part, r.done, r.mean);
    }
    NCVIS_LAUNCH(centred_sigma<D>, r.light_grid, kThreads, 0, s, r.light, to, r.mean, r.part, r.done,
                 r.sigma);
    NCVIS_LAUNCH(standardize_rows<D>, r.light_grid, kThreads, 0, s, r.light, to, r.mean, r.sigma, out,
                 packed ? 1 : 0);
}

void run_epochs(const InitRun &r, float *Y, float *bufs[2], cudaStream_t s) {
    for (int ep = 0; ep < r.epochs; ++ep) {
        const float *from = bufs[ep % 2];
        float *to = bufs[(ep + 1) % 2];
        const bool last = ep + 1 == r.epochs;
        float *out = last ? Y : to;
        if (!r.by_row) {
            NCVIS_LAUNCH(spmm_mean_any, r.grid, kThreads, 0, s, r.blocks, r.d, r.row_ptr, r.cols,
                         r.alpha, from, to, r.part, r.done, r.mean);
            NCVIS_LAUNCH(centred_sigma_any, r.light_grid, kThreads, 0, s, r.light, r.d, to, r.mean,
                         r.part, r.done, r.sigma);
            NCVIS_LAUNCH(standardize_any, r.light_grid, kThreads, 0, s, r.light, r.d, to, r.mean,
                         r.sigma, out);
            continue;
        }
        switch (r.d) {
            case 1: epoch_by_row<1>(r, from, to, out, last, s); break;
            case 2: epoch_by_row<2>(r, from, to, out, last, s); break;
            case 3: epoch_by_row<3>(r, from, to, out, last, s); break;
            default: epoch_by_row<4>(r, from, to, out, last, s);
        }
    }
}

// Rows of Y whose vector loads and stores are aligned.
bool aligned_rows(const float *Y, int d) {
    return ((uintptr_t)Y & (d == 4 ? 15 : d == 2 ? 7 : 3)) == 0;
}

// Buffers beside Y: one of Y's layout, or two padded ones for d = 3.
size_t buffer_bytes(int64_t rows, int d) {
    return d == 3 ? 2 * align256(sizeof(float) * 4 * rows) : align256(sizeof(float) * rows * d);
}

}  // namespace

int init_tile_rows() { return kThreads; }

size_t init_batched_workspace_bytes(int64_t total_rows, int64_t n_tiles, int B, int d) {
    return buffer_bytes(total_rows, d) + align256(sizeof(double) * n_tiles * d) +
           2 * align256(sizeof(float) * B * d) + align256(sizeof(int) * B);
}

void run_init_embedding_batched(int64_t total_rows, int d, const int64_t *off, const int64_t *tp,
                                int B, int64_t n_tiles, const uint64_t *seeds,
                                const int64_t *row_ptr, const int32_t *cols, int n_init_epochs,
                                float alpha, float *Y, void *workspace, cudaStream_t s) {
    require(d >= 1 && d <= kMaxDim, "init_embedding: d must be in [1, 32]");
    char *p = (char *)workspace;
    float *other = (float *)p;
    p += buffer_bytes(total_rows, d);
    double *part = (double *)p;  p += align256(sizeof(double) * n_tiles * d);
    float *mean = (float *)p;    p += align256(sizeof(float) * B * d);
    float *sigma = (float *)p;   p += align256(sizeof(float) * B * d);
    int *done = (int *)p;
    const int64_t n = total_rows * d;
    const bool padded = d == 3 && n_init_epochs > 0;
    float *bufs[2] = {padded ? other : Y, padded ? other + align256(16 * total_rows) / 4 : other};
    NCVIS_CUDA(cudaMemsetAsync(done, 0, sizeof(int) * B, s));
    NCVIS_LAUNCH(uniform_init_batched, ceil_div(n, kThreads), kThreads, 0, s, bufs[0], n, d,
                 padded ? 4 : d, off, B, seeds);
    const RowBlocks tiles{total_rows, kThreads, off, tp, B};
    InitRun r{tiles, tiles, (unsigned)n_tiles, (unsigned)n_tiles, d, n_init_epochs,
              d <= 4 && aligned_rows(Y, d), total_rows <= kShareRows, row_ptr, cols, alpha, part, done, mean, sigma};
    run_epochs(r, Y, bufs, s);
}

size_t init_workspace_bytes(int64_t N, int d) {
    const int64_t rows = rows_per_block(N), blocks = (N + rows - 1) / rows;
    return buffer_bytes(N, d) + align256(sizeof(double) * blocks * d) +
           2 * align256(sizeof(float) * d) + align256(sizeof(int));
}

void run_init_embedding(int64_t N, int d, const int64_t *row_ptr, const int32_t *cols,
                        uint64_t seed, int n_init_epochs, float alpha, float *Y, void *workspace,
                        cudaStream_t s, bool sequential_stats) {
    require(d >= 1 && d <= kMaxDim, "init_embedding: d must be in [1, 32]");
    const int64_t rows = rows_per_block(N), blocks = (N + rows - 1) / rows;
    char *p = (char *)workspace;
    float *other = (float *)p;
    p += buffer_bytes(N, d);
    double *part = (double *)p;  p += align256(sizeof(double) * blocks * d);
    float *mean = (float *)p;    p += align256(sizeof(float) * d);
    float *sigma = (float *)p;   p += align256(sizeof(float) * d);
    int *done = (int *)p;

    const int64_t n = N * d;
    const bool padded = d == 3 && n_init_epochs > 0 && !sequential_stats;
    float *bufs[2] = {padded ? other : Y, padded ? other + align256(16 * N) / 4 : other};
    // Draws per thread: each jump costs about as much as 40 draws, and few
    // points need every thread they can have.
    const int per_thread = n >= (int64_t)64 * kThreads * num_sms() ? 64 : 8;
    NCVIS_CUDA(cudaMemsetAsync(done, 0, sizeof(int), s));
    NCVIS_LAUNCH(uniform_init, ceil_div(ceil_div(n, per_thread), kThreads), kThreads, 0, s,
                 bufs[0], n, d, padded ? 4 : d, seed, per_thread);
    const int64_t light = rows_per_block_light(N);
    InitRun r{{N, rows, nullptr, nullptr, 0}, {N, light, nullptr, nullptr, 0}, (unsigned)blocks,
              (unsigned)((N + light - 1) / light), d, n_init_epochs, d <= 4 && aligned_rows(Y, d) && !sequential_stats, N <= kShareRows, row_ptr, cols, alpha, part, done, mean, sigma};
    if (!sequential_stats) {
        run_epochs(r, Y, bufs, s);
        return;
    }
    const size_t seq_smem = sizeof(float) * 2 * (size_t)(kSeqFloats / d) * d;
    NCVIS_CUDA(cudaFuncSetAttribute(sequential_stat, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)seq_smem));
    for (int ep = 0; ep < n_init_epochs; ++ep) {
        float *to = bufs[(ep + 1) % 2];
        NCVIS_LAUNCH(spmm_mean_any, r.grid, kThreads, 0, s, r.blocks, d, row_ptr, cols, alpha,
                     bufs[ep % 2], to, part, done, mean);
        NCVIS_LAUNCH(sequential_stat, 1, kThreads, seq_smem, s, to, N, d, 0, nullptr, mean);
        NCVIS_LAUNCH(sequential_stat, 1, kThreads, seq_smem, s, to, N, d, 1, mean, sigma);
        NCVIS_LAUNCH(standardize_any, r.light_grid, kThreads, 0, s, r.light, d, to, mean, sigma,
                     ep + 1 == n_init_epochs ? Y : to);
    }
}

}  // namespace ncvis_gpu
