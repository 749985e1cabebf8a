// Test harness (CPU only): rows that hold NaN distances.  std::sort's steps as the
// engine states them (merge_row.cuh) stay within the row, which a checked view of it
// watches, and give std::sort's own result and the reference's deduplication
// (src/knntable.cpp:81-93), so the sequential merge takes such rows.  The ranks by
// which the data-parallel merge sorts a leaf (the keys below one's own, equal ones to
// the left) are no permutation there: counted, and expected.
// Prints "ok <rows> <rows whose ranks collide>" or the first mismatch.  As a shared
// library: nan_symmetrize, the reference's symmetrization of a whole table (the oracle
// is built as the reference is, with -ffast-math, where comparisons need not honour NaN).
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <numeric>
#include <random>
#include <vector>

#include "merge_row.cuh"

using ncvis_gpu::SortItem;

template <class T>
struct Checked {
    T *v;
    int32_t n;
    T &operator[](int32_t i) const {
        if (i < 0 || i >= n) {
            std::printf("index %d of %d\n", i, n);
            std::exit(1);
        }
        return v[i];
    }
};

// The reference's steps on one row: indices `orig` and distances `key`.
static void reference_row(const std::vector<int32_t> &orig, const std::vector<float> &key,
                          std::vector<int32_t> &cols, std::vector<float> &vals) {
    std::vector<long> idx(key.size());
    std::iota(idx.begin(), idx.end(), 0L);
    std::sort(idx.begin(), idx.end(), [&key](long a, long b) { return key[a] < key[b]; });
    std::vector<int32_t> row(orig);
    cols.clear();
    vals.clear();
    for (size_t j = 0; j < idx.size(); ++j) {
        if (j > 0 && row[idx[j]] == row[idx[j - 1]]) continue;
        row[cols.size()] = orig[idx[j]];
        cols.push_back(orig[idx[j]]);
        vals.push_back(key[idx[j]]);
    }
}

// row_ptr [N + 1], cols and vals [2 N k]; returns the number of entries.
extern "C" int64_t nan_symmetrize(int64_t N, int64_t k, const int32_t *inds, const float *dists,
                                  int64_t *row_ptr, int32_t *cols, float *vals) {
    std::vector<std::vector<int64_t>> in(N);
    for (int64_t e = 0; e < N * k; ++e) in[inds[e]].push_back(e);
    std::vector<int32_t> orig, c;
    std::vector<float> key, v;
    int64_t at = row_ptr[0] = 0;
    for (int64_t i = 0; i < N; ++i) {
        orig.assign(inds + i * k, inds + i * k + k);
        key.assign(dists + i * k, dists + i * k + k);
        for (int64_t e : in[i]) orig.push_back((int32_t)(e / k)), key.push_back(dists[e]);
        reference_row(orig, key, c, v);
        std::copy(c.begin(), c.end(), cols + at);
        std::copy(v.begin(), v.end(), vals + at);
        row_ptr[i + 1] = at += (int64_t)c.size();
    }
    return at;
}

int main(int argc, char **argv) {
    const int rows = argc > 1 ? std::atoi(argv[1]) : 20000;
    std::mt19937_64 rng(5);
    int collide = 0;
    for (int r = 0; r < rows; ++r) {
        const int32_t n = 1 + (int32_t)(rng() % (r % 4 == 0 ? 1200 : 140));
        const int32_t levels = 1 + (int32_t)(rng() % (r % 2 == 0 ? 5 : 100000));
        const uint32_t share = 1 + (uint32_t)(rng() % 100);  // per cent of NaN, at least one
        const float nan = std::numeric_limits<float>::quiet_NaN();
        std::vector<float> key(n);
        std::vector<int32_t> orig(n);
        for (int32_t i = 0; i < n; ++i) {
            key[i] = rng() % 100 < share ? nan : (float)(rng() % levels);
            if (rng() % 50 == 0) key[i] = std::numeric_limits<float>::infinity();
            orig[i] = (int32_t)(rng() % (1 + n / 2));
        }
        key[rng() % n] = nan;
        std::vector<int32_t> cols;
        std::vector<float> vals;
        reference_row(orig, key, cols, vals);
        std::vector<SortItem> v(n);
        for (int32_t i = 0; i < n; ++i) v[i] = SortItem{key[i], i};
        const int32_t n_out = ncvis_gpu::sort_and_dedup(Checked<SortItem>{v.data(), n},
                                                        Checked<int32_t>{orig.data(), n}, n);
        bool same = n_out == (int32_t)cols.size();
        for (int32_t q = 0; same && q < n_out; ++q)
            same = orig[v[q].pos] == cols[q] && std::memcmp(&v[q].key, &vals[q], 4) == 0;
        if (!same) {
            std::printf("row %d n=%d: kept %d vs %zu\n", r, n, n_out, cols.size());
            return 1;
        }
        std::vector<int> hit(n, 0);
        for (int32_t x = 0; x < std::min(n, 16); ++x) {
            int rank = 0;
            for (int32_t y = 0; y < std::min(n, 16); ++y)
                rank += (key[y] < key[x]) || (key[y] == key[x] && y < x);
            collide += ++hit[rank] == 2;
        }
    }
    std::printf("ok %d %d\n", rows, collide);
    return 0;
}
