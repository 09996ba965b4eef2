// bucket_math.h -- positions of (view, tile) buckets in the sorted list.
//
// Positions are int32 and the list has at most 2^31 - 1 entries, but what a
// frame asks for can be more: the fused path learns the total on the device
// and reports it after the launches are queued.  Positions past the list
// therefore saturate instead of wrapping to negative ones.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define UBS_HD __host__ __device__ __forceinline__
#else
#define UBS_HD inline
#endif

namespace ubs {

UBS_HD int64_t imin64(int64_t a, int64_t b) { return a < b ? a : b; }

// A position as it is stored.
UBS_HD int32_t bucket_start(int64_t at) { return (int32_t)imin64(at, INT32_MAX); }

// A scanned value: an int32 one is a position.
template <typename T> UBS_HD T scan_value(int64_t v);
template <> UBS_HD int32_t scan_value<int32_t>(int64_t v) { return bucket_start(v); }
template <> UBS_HD int64_t scan_value<int64_t>(int64_t v) { return v; }

// The entries [lo, hi) of a bucket between the stored positions `start` and
// `end` (INT32_MAX for the last bucket) in a list of T: 0 <= lo <= hi <= T
// whatever is stored.
UBS_HD void bucket_bounds(int32_t start, int32_t end, int64_t T, int64_t &lo, int64_t &hi) {
    lo = imin64(start > 0 ? start : 0, T);
    hi = imin64(end, T);
    if (hi < lo) hi = lo;
}

} // namespace ubs
