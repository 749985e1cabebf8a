// K1: per-point preprocessing of NCVis::preprocess (src/ncvis.cpp:32-70).
// correlation: subtract the row mean; cosine and correlation: divide by the
// row's Euclidean norm when it is non-zero; squared_L2 and inner_product:
// copy.  One warp per row; the squared norm of the result (for the
// |x|^2 + |y|^2 - 2<x,y> form of squared L2) and the zero-padded BF16
// copies for the tensor-core kNN are produced in the same pass.
#include <cmath>
#include <cstring>

#include "common.cuh"
#include "stages.cuh"

namespace ncvis_gpu {

namespace {

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// The value of x's lowest set bit (0 for 0).
__device__ __forceinline__ float low_bit(float x) {
    const uint32_t b = __float_as_uint(x) & 0x7fffffffu;
    const float v = __uint_as_float(b);
    return (b & 0x7fffffu) ? v - __uint_as_float(b & (b - 1u)) : v;
}

// A row whose coordinates are multiples of u and whose squared norm is at most
// kExactNorm u^2 has exact FP32 sums with every other such row: their products and
// squared norms are whole numbers of u^2 below 2^24.  Integers, one-hot columns and
// 8-bit pixels are such rows; ties among their distances are exact and go by index.
constexpr float kExactNorm = 0x1p24f;

__global__ void __launch_bounds__(256) preprocess_rows(const float *__restrict__ X, int64_t N,
                                                       int D, int dist, float *__restrict__ Xp,
                                                       float *__restrict__ sqnorm,
                                                       __nv_bfloat16 *__restrict__ Xb,
                                                       __nv_bfloat16 *__restrict__ Xc, int ldb,
                                                       int *__restrict__ bad_flag,
                                                       uint32_t *__restrict__ norms) {
    const int lane = threadIdx.x & 31;
    const int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= N) return;
    const float *x = X + row * D;
    float *out = Xp + row * D;

    float mean = 0.f;
    bool finite = true;
    if (dist == kCorrelation) {
        float s = 0.f;
        for (int t = lane; t < D; t += 32) s += x[t];
        mean = warp_sum(s) / (float)D;
    }
    float sq = 0.f;
    for (int t = lane; t < D; t += 32) {
        float v = x[t];
        finite &= isfinite(v);
        v = v - mean;
        sq += v * v;
    }
    sq = warp_sum(sq);
    float scale_div = 1.f;
    const bool normalise = (dist == kCorrelation || dist == kCosine) && sq != 0.f;
    if (normalise) scale_div = sqrtf(sq);
    float sq_out = 0.f;
    bool bits12 = false;  // a coordinate of exactly 12 significant bits
    for (int t = lane; t < D; t += 32) {
        float v = x[t] - mean;
        if (normalise) v = v / scale_div;
        out[t] = v;
        sq_out += v * v;
        bits12 |= (__float_as_uint(v) & 0x1fffu) == 0x1000u;
        if (Xb) Xb[row * ldb + t] = __float2bfloat16_rn(v);
        if (Xc) Xc[row * ldb + t] = __float2bfloat16_rn(v);
    }
    // With Xc (squared L2 on the tensor cores) columns D and D + 1 hold 1, 1 in
    // the query copy and -|x|^2 / 2 split into a BF16 high and low part in the
    // candidate copy, so that a row pair's product is <q, c> - |c|^2 / 2.
    const int extra = Xc ? 2 : 0;
    if (Xb)
        for (int t = D + extra + lane; t < ldb; t += 32) Xb[row * ldb + t] = __float2bfloat16_rn(0.f);
    if (Xc)
        for (int t = D + extra + lane; t < ldb; t += 32) Xc[row * ldb + t] = __float2bfloat16_rn(0.f);
    sq_out = warp_sum(sq_out);
    if (norms && __any_sync(0xffffffffu, bits12)) {
        // One row in eighty of arbitrary numbers comes here; its lowest bit is
        // far too low.
        float u = INFINITY;
        for (int t = lane; t < D; t += 32)
            if (out[t] != 0.f) u = fminf(u, low_bit(out[t]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) u = fminf(u, __shfl_xor_sync(0xffffffffu, u, o));
        if (lane == 0 && sq_out <= kExactNorm * u * u) norms[2] = 1u;
    }
    if (lane == 0) {
        sqnorm[row] = sq_out;
        if (norms) {
            // Most rows find both words past their norm already: a read, no atomic.
            const uint32_t bits = __float_as_uint(sq_out);
            if (bits > __ldcg(norms)) atomicMax(norms, bits);
            if (bits != 0u && bits <= kInfBits && kInfBits - bits > __ldcg(norms + 1))
                atomicMax(norms + 1, kInfBits - bits);
        }
        if (Xc) {
            const float h = -0.5f * sq_out;
            const __nv_bfloat16 hi = __float2bfloat16_rn(h);
            const __nv_bfloat16 lo = __float2bfloat16_rn(h - __bfloat162float(hi));
            Xb[row * ldb + D] = __float2bfloat16_rn(1.f);
            Xb[row * ldb + D + 1] = __float2bfloat16_rn(1.f);
            Xc[row * ldb + D] = hi;
            Xc[row * ldb + D + 1] = lo;
        }
    }
    if (!__all_sync(0xffffffffu, finite) && lane == 0) atomicOr(bad_flag, 1);
}

// FP16 parts of s * x for the FP32 search on the tensor cores: 8 columns of one
// row per thread, 16-byte stores.  hi is s x rounded to 11 bits; s x - hi is
// exact in FP32 and its 11 bits are lo, so hi + lo holds s x to at most one unit
// in FP32's last place.  The tensor cores' FP32 accumulator truncates: a product
// loses about 0.6 units in its 24th place per 16 columns (measured: 0.36 on unit
// rows to 0.85 on rows far from the origin), which lo makes up for on both sides
// (`lift` = half of that, relative).  A coordinate that may belong to a row of exact
// sums (kExactNorm) takes no lift: nothing is truncated there, and a lift would tell
// equal distances apart (60,000 rows of 32 zeros and ones: 8% of the rows had other
// neighbours than (distance, index) says).  Squared L2 (fold): w = -|s c|^2 / 2 goes into three
// columns, w = 2^14 a + 2^3 b + 2^-8 c with a, b, c in FP16, each part's
// remainder exact; the powers keep all three within FP16's normal range for
// norms from 2^1 to 2^14.
__global__ void __launch_bounds__(256) split_rows(
    const float *__restrict__ Xp, const float *__restrict__ sqnorm, int64_t N, int D, int ldb,
    float scale, float lift, bool fold, __half *__restrict__ hi, __half *__restrict__ lo,
    __half *__restrict__ cand, const int64_t *__restrict__ off, const int64_t *__restrict__ pad,
    int B) {
    const int per = ldb >> 3;
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= N * per) return;
    const int64_t row = t / per;
    const int c0 = (int)(t - row * per) * 8;
    int64_t to = row;
    if (off) {
        const int p = segment_of(off, B, row);
        to = pad[p] + (row - off[p]);
    }
    const float *x = Xp + row * D;
    const float sq = __ldg(sqnorm + row);
    float v[8];
    if ((D & 3) == 0 && c0 + 8 <= D) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(x + c0));
        const float4 b = __ldg(reinterpret_cast<const float4 *>(x + c0 + 4));
        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
        v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = c0 + j < D ? __ldg(x + c0 + j) : 0.f;
    }
    __align__(16) __half h[8], l[8], c[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float y = v[j] * scale;
        const float low = low_bit(v[j]);
        const bool exact = sq <= kExactNorm * low * low;
        h[j] = __float2half_rn(y);
        l[j] = __float2half_rn(fmaf(y, exact ? 0.f : lift, y - __half2float(h[j])));
        c[j] = h[j];
    }
    if (fold && c0 + 8 > D) {
        const float w = -0.5f * sq * scale * scale;
        const __half a = __float2half_rn(w * 0x1p-14f);
        const float r1 = w - __half2float(a) * 0x1p14f;
        const __half b = __float2half_rn(r1 * 0x1p-3f);
        const float r2 = r1 - __half2float(b) * 0x1p3f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (c0 + j == D) c[j] = a, h[j] = __float2half_rn(0x1p14f);
            if (c0 + j == D + 1) c[j] = b, h[j] = __float2half_rn(0x1p3f);
            if (c0 + j == D + 2) c[j] = __float2half_rn(r2 * 0x1p8f), h[j] = __float2half_rn(0x1p-8f);
        }
    }
    const int64_t o = to * ldb + c0;
    *reinterpret_cast<uint4 *>(hi + o) = *reinterpret_cast<const uint4 *>(h);
    *reinterpret_cast<uint4 *>(lo + o) = *reinterpret_cast<const uint4 *>(l);
    if (fold) *reinterpret_cast<uint4 *>(cand + o) = *reinterpret_cast<const uint4 *>(c);
}

}  // namespace

float split_scale(const uint32_t norms[3], int dist, bool one_problem) {
    // Unit rows (and rows of zeros).
    if (dist == kCosine || dist == kCorrelation) return 0x1p14f;
    if (norms[0] == 0u) return 1.f;
    if (norms[0] >= kInfBits) return 0.f;
    const uint32_t low_bits = kInfBits - norms[1];
    float top, low;
    std::memcpy(&top, &norms[0], 4);
    std::memcpy(&low, &low_bits, 4);
    // Squared norms must keep their own precision in FP32.
    if (low < 0x1p-100f || top > 0x1p100f) return 0.f;
    // Distances 1 - <q, c> are rounded to 2^-24, and equal ones go by index.  Where a
    // row's products all lie within 2^-14 many distances are equal though their
    // products are not, and the CUDA cores' search ranks by the distance: 20,000 x 64
    // at products of 2^-18 and 1,000 x 16 at 2^-20 held other neighbours from the tensor
    // cores, none at 2^-16.  A problem of a batch may hold the smallest norms only.
    if (dist == kInnerProduct && (one_problem ? std::sqrt(low * top) : low) < 0x1p-14f) return 0.f;
    const int e = std::ilogb(std::sqrt(top)) + 1;  // norms < 2^e (1 + rounding)
    const float scale = std::ldexp(1.f, 14 - e);
    return std::sqrt(low) * scale >= 2.f ? scale : 0.f;
}

void launch_split_rows(const float *Xp, const float *sqnorm, int64_t N, int D, float scale,
                       const KnnTcPlan &plan, __half *rows, int64_t rows_per_part, cudaStream_t s,
                       const int64_t *off, const int64_t *pad, int B) {
    const size_t part = (size_t)rows_per_part * plan.ldb;
    const float lift = 0.5f * 0.6f * (float)D / 16.f * 0x1p-24f;
    NCVIS_LAUNCH(split_rows, ceil_div((size_t)N * (plan.ldb / 8), 256), 256, 0, s, Xp, sqnorm, N, D,
                 plan.ldb, scale, lift, plan.fold, rows, rows + part,
                 plan.fold ? rows + 2 * part : nullptr, off, pad, B);
}

void launch_preprocess(const float *X, int64_t N, int D, int dist, float *Xp, float *sqnorm,
                       __nv_bfloat16 *Xb, int ldb, int *bad_flag, cudaStream_t s,
                       __nv_bfloat16 *Xc, uint32_t *norms) {
    const int warps_per_block = 8;
    NCVIS_LAUNCH(preprocess_rows, ceil_div(N, warps_per_block), 32 * warps_per_block, 0, s, X, N,
                 D, dist, Xp, sqnorm, Xb, Xc, ldb, bad_flag, norms);
}

}  // namespace ncvis_gpu
