// Host-only check of the staged split search's table plans (stage_tables): whole 32-feature tiles that cover the
// features, no table above the limit except one tile of unflipped rows, the widest first, and where flipped rows have
// their own bins. Prints "<n> failures".
#include <algorithm>
#include <cstdio>

#include "../../curfil_b200/csrc/split_eval.h"

using namespace cf;

static int failures = 0;

static void check(long long rows, bool flips, int F, long long max_bytes) {
    const std::vector<StageTable> t = stage_tables(rows, flips, F, max_bytes);
    const int tiles = (F + kStageTile - 1) / kStageTile;
    bool ok = !t.empty();
    for (size_t i = 0; ok && i < t.size(); i++) {
        const long long bytes = (t[i].both ? 2 : 1) * rows * t[i].chunk;
        ok = t[i].chunk >= kStageTile && t[i].chunk % kStageTile == 0;
        ok = ok && static_cast<long long>(t[i].n_chunks) * t[i].chunk >= F && (t[i].n_chunks - 1ll) * t[i].chunk < F;
        ok = ok && (bytes <= max_bytes || (!t[i].both && t[i].chunk == kStageTile));
        ok = ok && (flips || !t[i].both);
        if (i > 0) ok = ok && (t[i].both == t[i - 1].both ? t[i].chunk < t[i - 1].chunk : !t[i].both);
    }
    ok = ok && t.back().chunk == kStageTile && !t.back().both;
    // the unflipped rows take as few chunks as the limit allows
    const auto one = std::find_if(t.begin(), t.end(), [](const StageTable& x) { return !x.both; });
    const long long most = std::max(1ll, std::min<long long>(tiles, max_bytes / rows / kStageTile));
    ok = ok && one != t.end() && one->n_chunks <= (tiles + most - 1) / most;
    if (flips) {   // flipped rows are staged where they cost no chunks, or leave wide ones
        const long long both = max_bytes / (2 * rows) / kStageTile;
        const bool fits = both >= tiles || both >= kWideChunk / kStageTile;
        ok = ok && (!fits || t[0].both) && (!t[0].both || t[0].n_chunks == one->n_chunks || t[0].chunk >= kWideChunk / 2);
    }
    if (!ok) {
        failures++;
        std::printf("FAIL rows %lld flips %d F %d limit %lld\n", rows, flips, F, max_bytes);
    }
}

int main() {
    for (long long rows : {1ll, 31ll, 2363ll, 5200ll, 32768ll, 32769ll, 266600ll, 8000000ll, 1073741823ll, 2147483646ll})
        for (int F : {1, 31, 32, 33, 64, 255, 256, 257, 331, 500, 2000, 4000, 100000})
            for (long long mb : {1ll, 2ll, 3ll, 64ll, 8192ll, 65536ll})
                for (bool flips : {false, true}) check(rows, flips, F, mb << 20);
    std::printf("%d failures\n", failures);
    return failures != 0;
}
