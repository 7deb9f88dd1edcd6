// Append binning's row lists (k_bin.cu), as the host sees them.
#pragma once

#include "kernels.hpp"

namespace b200 {

// Bin b's list starts at b * m (the device only counts rows).
inline void list_offsets(Plan* plan, int nb, int32_t m) {
    for (int b = 0; b < nb; b++) plan->bin_off[b] = b * m;
}

// The limits append binning counts one-pass rows by: the fill ladder's, and,
// where the fill may expand, sort and compress, kEscSplit, kEscCtaSmall and
// kEscCtaMid too.  Which kernel takes which list is decided when the sample is
// known: src[e] is the fill bin limit e comes from (kFromSplit, kFromSmall:
// inserted).
constexpr int kFromSplit = -1;
constexpr int kFromSmall = -2;
struct ListLadder {
    Ladder lad;
    int src[kMaxBins];
    // the fill bin that list e belongs to
    int fill_bin(int e, bool split) const {
        if (src[e] == kFromSplit) return kEscBins - 1;
        if (src[e] == kFromSmall) return kEscBins;
        return split && src[e] == kEscBins - 1 ? kEscBins : src[e];
    }
};

// False when the limits are more than the scratch has lists (the device would
// write row ids past them): the caller reports it.
inline bool list_ladder(const Ladder& fill, bool esc, ListLadder* out) {
    ListLadder l = {};
    int nb = 0;
    auto put = [&](int32_t limit, int from) {
        if (nb < kListBins) {
            l.lad.limit[nb] = limit;
            l.src[nb] = from;
        }
        nb++;
    };
    for (int b = 0; b < fill.nb; b++) {
        if (esc && b == kEscBins - 1) put(kEscSplit, kFromSplit);
        if (esc && b == kEscBins) put(kEscCtaSmall, kFromSmall);
        if (esc && b == kEscBins) put(kEscCtaMid, kFromSmall);
        put(fill.limit[b], b);
        // rows forced to bin min_bin or above: to the lists past the bin below
        if (b == fill.min_bin - 1) l.lad.min_bin = nb;
    }
    if (nb > kListBins) return false;
    l.lad.nb = nb;
    *out = l;
    return true;
}

}  // namespace b200
