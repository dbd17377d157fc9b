// What the unit form's scan does with a range, as the warps that improve its champion publish it
// and the load warp reads it, without a lock and at any time: one word a range, so that no order
// of the two sides' accesses can show half of a change.  (A threshold and a full-form bit in two
// words could be read as "threshold +inf, not in the full form" between the two writes, and the
// range's next tiles were then looked at by nobody.)
#pragma once

#if defined(__CUDACC__)
#define MARS_SCAN_FN __host__ __device__ __forceinline__
#else
#define MARS_SCAN_FN inline
#endif

namespace mars {
namespace tc {

constexpr float kScanFull = 0.0f;         // the range takes the full form (thresholds are positive)
constexpr float kScanNothing = __builtin_huge_valf();  // nothing to scan for: no block, or a flat one

struct ScanState {
    bool full;
    float threshold;  // of the scan's test; +inf for ranges that it passes by
};

// words: the ranges' words, with load(i) and store(i, value) that are made where they stand.
template <class Words>
MARS_SCAN_FN void scan_publish(const Words& words, int range, bool full, float threshold) {
    words.store(range, full ? kScanFull : threshold);
}

template <class Words>
MARS_SCAN_FN ScanState scan_read(const Words& words, int range) {
    const float v = words.load(range);
    const bool full = v == kScanFull;
    return ScanState{full, full ? kScanNothing : v};
}

}  // namespace tc
}  // namespace mars
