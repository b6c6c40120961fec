// Accumulated bins of a set of points, from its largest distance (host code without CUDA).
#pragma once
#include <algorithm>
#include <cmath>

namespace ausaxs_b200 {

struct BinSpan {
    int bins;      // bins that are accumulated: at most bin_count, at least 11 where that allows it
    bool covered;  // no pair's distance lies beyond them
};

// The count is formed and compared in double: a distance of 2^31 bins or more (or one that is not a number) has no
// int, and converted all the same it would come out as few bins that seem to cover everything.
inline BinSpan bin_span(double dmax, float inv_w, int bin_count) {
    const double n = std::ceil(dmax * inv_w) + 2;
    if (!(n <= bin_count)) return {bin_count, false};
    const int bins = std::max(static_cast<int>(n), 11);
    return {std::min(bins, bin_count), bins <= bin_count};
}

}  // namespace ausaxs_b200
