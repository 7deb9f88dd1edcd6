// Host driver of gpuspgemm_b200/csrc/lists.hpp for tests/test_lists.py.
//
// Usage: lists_host NB ESC MIN_BIN: a fill ladder of NB bins with the limits of
// the one-pass ladder's first five.  Prints one JSON object.
#include <cstdio>
#include <cstdlib>

#include "lists.hpp"

int main(int argc, char** argv) {
    using namespace b200;
    if (argc != 4) return 2;
    Ladder fill = {};
    fill.nb = std::atoi(argv[1]);
    fill.min_bin = std::atoi(argv[3]);
    const int32_t first[] = {12, 48, 192, 768, 3072};
    for (int b = 0; b < fill.nb; b++) fill.limit[b] = b < 5 ? first[b] : 4096 * (b - 3);
    ListLadder l = {};
    l.lad.nb = -1;
    const bool ok = list_ladder(fill, std::atoi(argv[2]) != 0, &l);
    std::printf("{\"ok\": %d, \"lists\": %d, \"nb\": %d, \"min\": %d, \"limits\": [", ok, kListBins,
                l.lad.nb, l.lad.min_bin);
    for (int e = 0; e < l.lad.nb; e++) std::printf("%s%d", e ? ", " : "", l.lad.limit[e]);
    std::printf("], \"hash_bin\": [");
    for (int e = 0; e < l.lad.nb; e++) std::printf("%s%d", e ? ", " : "", l.fill_bin(e, false));
    std::printf("], \"sort_bin\": [");
    for (int e = 0; e < l.lad.nb; e++) std::printf("%s%d", e ? ", " : "", l.fill_bin(e, true));
    std::printf("]}\n");
    return 0;
}
