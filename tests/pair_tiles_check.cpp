// Host-side check of the tapered pair plan (plan_pair_tiles in libkhrr), run on
// the CPU by tests/test_pair_tiles.py: replays every item as the kernel
// executes it.  Tiles of an item's own block ([j_begin, diag_end)) count once,
// (i tile, j tile); later tiles twice, (i, j) and (j, i).  Every ordered pair
// of 128-body tiles of one system must be hit exactly once and none across
// systems, with block-aligned i blocks, and the sums must end at the system's
// real bodies.  Prints "ok <items> <largest chunk in tiles>" or the violation.
#include <cstdint>
#include <cstdio>
#include <algorithm>
#include <cstdlib>
#include <vector>

#include "khrr_runtime.h"

using namespace khrr;

int main(int argc, char** argv) {
    if (argc < 3) return 2;
    const int ctas = std::atoi(argv[1]);
    std::vector<int64_t> cnt, poff{0};
    for (int a = 2; a < argc; ++a) {
        cnt.push_back(std::atoll(argv[a]));
        poff.push_back(poff.back() + (cnt.back() + kPad - 1) / kPad * kPad);
    }
    ForcePlan p;
    plan_pair_tiles(poff, cnt, ctas, p);
    const int64_t ntiles = poff.back() / kPad;
    std::vector<int> sys(ntiles);
    for (size_t k = 0; k < cnt.size(); ++k)
        for (int64_t t = poff[k] / kPad; t < poff[k + 1] / kPad; ++t) sys[t] = static_cast<int>(k);
    std::vector<unsigned char> cover(static_cast<size_t>(ntiles * ntiles), 0);
    int64_t largest = 0;
    for (const PairItem& w : p.pair_items) {
        const int64_t i0 = w.i_begin / kPad, i1 = w.i_end / kPad, j0 = w.j_begin / kPad, j1 = w.j_end / kPad;
        const int k = sys[i0];
        const bool aligned = w.i_begin % kPad == 0 && w.j_begin % kPad == 0 && w.j_end % kPad == 0;
        if (!aligned || (w.i_begin - poff[k]) % kPairBlock || i1 <= i0 || j1 <= j0 || w.i_end - w.i_begin > kPairBlock ||
            w.diag_end != w.i_end || j0 < i0 || w.real_end != poff[k] + cnt[k]) {
            std::printf("FAIL item %d %d %d %d %d\n", w.i_begin, w.i_end, w.j_begin, w.j_end, w.diag_end);
            return 1;
        }
        largest = std::max(largest, j1 - j0);
        for (int64_t i = i0; i < i1; ++i)
            for (int64_t j = j0; j < j1; ++j) {
                ++cover[i * ntiles + j];
                if (j * kPad >= w.diag_end) ++cover[j * ntiles + i];
            }
    }
    for (int64_t a = 0; a < ntiles; ++a)
        for (int64_t b = 0; b < ntiles; ++b)
            if (cover[a * ntiles + b] != (sys[a] == sys[b] ? 1 : 0)) {
                std::printf("FAIL tile pair %lld %lld covered %d times\n", (long long)a, (long long)b, cover[a * ntiles + b]);
                return 1;
            }
    std::printf("ok %zu %lld\n", p.pair_items.size(), (long long)largest);
    return 0;
}
