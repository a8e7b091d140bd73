// Merge of the partial results of attention over split key ranges: [split][hd + 2] = (m, l, o[hd]), o relative to the split's maximum m
// and not divided by its denominator l. Splits without keys carry m = -inf, l = 0, o = 0.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace sp {

constexpr int MERGE_MAX_SPLITS = 32;  // of merge_splits

// Coordinate e of the merged row; n_splits <= NS. All of a thread's loads are requested before the first is used (with a test per
// split around them they came one after another, a round trip each: 16 splits took 7.5 to 8.8 us of a launch).
template <int NS>
__device__ __forceinline__ float merge_splits(const float* __restrict__ src, int n_splits, int hd, int e) {
    float m[NS], l[NS], o[NS], M = -INFINITY, L = 0.f, v = 0.f;
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const float* p = src + (int64_t)min(s, n_splits - 1) * (hd + 2);
        m[s] = p[0];
        l[s] = p[1];
        o[s] = p[2 + e];
    }
#pragma unroll
    for (int s = 0; s < NS; ++s) M = fmaxf(M, s < n_splits ? m[s] : -INFINITY);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const float c = s >= n_splits || m[s] == -INFINITY ? 0.f : expf(m[s] - M);
        L = fmaf(c, l[s], L);
        v = fmaf(c, o[s], v);
    }
    return v * ((L == 0.f) ? 0.f : 1.0f / L);
}

// The same for any number of splits, a few loads ahead: no engine has more than 32, a caller of the paged entry point may.
__device__ __forceinline__ float merge_many_splits(const float* __restrict__ src, int n_splits, int hd, int e) {
    float M = -INFINITY, L = 0.f, v = 0.f;
#pragma unroll 8
    for (int s = 0; s < n_splits; ++s) M = fmaxf(M, src[(int64_t)s * (hd + 2)]);
#pragma unroll 8
    for (int s = 0; s < n_splits; ++s) {
        const float* p = src + (int64_t)s * (hd + 2);
        const float c = p[0] == -INFINITY ? 0.f : expf(p[0] - M);
        L = fmaf(c, p[1], L);
        v = fmaf(c, p[2 + e], v);
    }
    return v * ((L == 0.f) ? 0.f : 1.0f / L);
}

}  // namespace sp
