// The staged split search under failing device allocations: the library's objects are linked with --wrap=cudaMalloc, so
// allocations of this program's choice fail on the host. Prints one line per check and "<n> failures".
//   1. each allocation of a call in turn fails once: the call gives the unlimited call's splits, or CF_ERR_OOM only
//      where the search in one pass needs that allocation too, and the same call works again afterwards;
//   2. allocations of a size and more fail: a smaller table, then the search in one pass;
//   3. an allocation refused while a context keeps preprocessing scratch works again with that memory given back;
//   4. stage_max_mb bounds the table whether or not samples are evaluated both ways, and the splits stay the same.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "../../include/curfil_b200.h"

static bool armed = false;
static int calls = 0, fail_at = -1;
static size_t fail_from = ~size_t(0), largest = 0;

extern "C" cudaError_t __real_cudaMalloc(void** p, size_t bytes);
extern "C" cudaError_t __wrap_cudaMalloc(void** p, size_t bytes) {
    if (armed && (calls++ == fail_at || bytes >= fail_from)) return cudaErrorMemoryAllocation;
    if (armed && bytes > largest) largest = bytes;
    return __real_cudaMalloc(p, bytes);
}

static int failures = 0;
static void check(bool ok, const char* what, int flips, long long detail) {
    if (!ok) failures++;
    if (!ok) std::printf("FAIL %s (flips %d): %lld\n", what, flips, detail);
}

struct Level {
    static constexpr int kFrames = 3, kW = 96, kH = 72, kC = 11, kNodes = 5, kT = 20, kRows = 3000;
    std::vector<uint8_t> rgb;
    std::vector<uint16_t> depth;
    std::vector<cf_sample> samples;
    std::vector<int64_t> offsets{0, 700, 701, 1500, 2900, kRows};
    std::vector<int8_t> features;
    std::vector<float> thresholds;
    int F;

    explicit Level(bool flips, int kF = 64) : rgb(size_t(kFrames) * kW * kH * 3), depth(size_t(kFrames) * kW * kH), samples(kRows),
                                 features(11 * kF), thresholds(kT * kF), F(kF) {
        std::mt19937 gen(7);
        auto pick = [&](int lo, int hi) { return std::uniform_int_distribution<int>(lo, hi)(gen); };
        for (auto& v : rgb) v = static_cast<uint8_t>(pick(0, 255));
        for (auto& v : depth) v = static_cast<uint16_t>(pick(0, 9) ? pick(700, 4000) : 0);
        for (auto& s : samples) {
            std::memset(&s, 0, sizeof(s));
            s.x = static_cast<uint16_t>(pick(0, kW - 1));
            s.y = static_cast<uint16_t>(pick(0, kH - 1));
            s.image = static_cast<uint32_t>(pick(0, kFrames - 1));
            s.depth = static_cast<float>(pick(700, 4000)) / 1000.0f;
            s.label = static_cast<uint8_t>(pick(0, kC - 1));
            s.flip = static_cast<uint8_t>(flips ? pick(0, 2) : 0);
        }
        for (int f = 0; f < kF; f++) {
            const bool color = f >= kF / 2;
            features[f] = color;
            for (int r = 1; r <= 4; r++) features[r * kF + f] = static_cast<int8_t>(pick(-30, 30));
            for (int r = 5; r <= 8; r++) features[r * kF + f] = static_cast<int8_t>(pick(1, 8));
            for (int r = 9; r <= 10; r++) features[r * kF + f] = static_cast<int8_t>(color ? pick(0, 2) : 0);
            for (int t = 0; t < kT; t++)
                thresholds[t * kF + f] = color ? static_cast<float>(pick(-3000, 3000)) : static_cast<float>(pick(-400, 400)) / 500.0f;
        }
    }
};

struct Run {
    cf_context* ctx = nullptr;
    cf_dataset* ds = nullptr;
    const Level& level;
    Run(const Level& l, int stage_bins, int stage_max_mb = 8192) : level(l) {
        cf_eval_tuning t;
        if (cf_context_create(0, &ctx) != CF_OK || cf_context_get_tuning(ctx, &t) != CF_OK) std::printf("FAIL context\n");
        t.stage_bins = stage_bins;
        t.stage_max_mb = stage_max_mb;
        if (cf_context_set_tuning(ctx, &t) != CF_OK || cf_dataset_create(ctx, Level::kFrames, Level::kW, Level::kH, &ds) != CF_OK ||
            cf_dataset_upload_raw(ds, 0, Level::kFrames, l.rgb.data(), l.depth.data(), 0) != CF_OK)
            std::printf("FAIL set-up\n");
    }
    ~Run() {
        cf_dataset_destroy(ds);
        cf_context_destroy(ctx);
    }
    cf_status call(std::vector<cf_split>& best, int64_t* staged = nullptr) {
        best.assign(Level::kNodes, cf_split{});
        cf_context_set_timing(ctx, 1);
        cf_context_reset_timing(ctx);
        const cf_status s = cf_evaluate_best_splits(ds, Level::kNodes, level.offsets.data(), level.samples.data(), Level::kC, level.F,
                                                    Level::kT, level.features.data(), level.thresholds.data(), best.data());
        double ms = 0;
        int64_t n = 0;
        cf_context_kernel_time(ctx, "stage_bins", &ms, &n);
        if (staged) *staged = n;
        return s;
    }
};

static bool same(const std::vector<cf_split>& a, const std::vector<cf_split>& b) {
    for (size_t i = 0; i < a.size(); i++)
        if (a[i].score != b[i].score || a[i].feature != b[i].feature || a[i].threshold_index != b[i].threshold_index ||
            a[i].threshold != b[i].threshold)
            return false;
    return true;
}

static int count_calls(const Level& level, int stage_bins, std::vector<cf_split>& best, int64_t* staged) {
    Run r(level, stage_bins);
    armed = true;
    calls = 0;
    const cf_status s = r.call(best, staged);
    armed = false;
    if (s != CF_OK) std::printf("FAIL unlimited call\n");
    return calls;
}

int main() {
    for (int flips = 0; flips < 2; flips++) {
        const Level level(flips != 0);
        std::vector<cf_split> want, best;
        int64_t staged = 0;
        const int one_pass = count_calls(level, 0, want, &staged);
        check(staged == 0, "one pass", flips, staged);
        const int two_passes = count_calls(level, 2, best, &staged);
        check(staged == 1 && same(best, want), "two passes", flips, staged);
        check(two_passes > one_pass + 10, "allocations of the two passes", flips, two_passes);
        int oom = 0;
        for (int n = 0; n < two_passes; n++) {
            Run r(level, 2);
            armed = true;
            calls = 0;
            fail_at = n;
            const cf_status s = r.call(best);
            armed = false;
            fail_at = -1;
            if (s == CF_OK) check(same(best, want), "splits with one allocation refused", flips, n);
            else check(s == CF_ERR_OOM, "status with one allocation refused", flips, n);
            oom += s != CF_OK;
            check(r.call(best) == CF_OK && same(best, want), "the call after a refused allocation", flips, n);
        }
        check(oom <= one_pass, "calls refused", flips, oom);
        // the table: 64 features x 3000 rows, twice that with flipped rows
        const size_t tile = size_t(32) * Level::kRows;
        struct {
            size_t from;
            int64_t staged;
        } limits[] = {{2 * tile + 1, 1}, {2 * tile, 2}, {tile + 1, 2}, {tile, 0}};
        for (const auto& l : limits) {
            Run r(level, 2);
            armed = true;
            calls = 0;
            fail_from = l.from;
            const cf_status s = r.call(best, &staged);
            armed = false;
            fail_from = ~size_t(0);
            check(s == CF_OK, "status under a limit", flips, static_cast<long long>(l.from));
            check(same(best, want), "splits under a limit", flips, static_cast<long long>(l.from));
            std::printf("flips %d, allocations below %zu bytes: %lld launches of pass 1\n", flips, l.from, static_cast<long long>(staged));
            check((staged == 0) == (l.staged == 0), "passes under a limit", flips, static_cast<long long>(l.from));
        }
        {
            Run r(level, 0);
            const int w = 640, h = 480, frames = 4;   // L*a*b* scratch: 36 bytes a pixel, 44 MB
            std::vector<uint8_t> rgb(size_t(frames) * w * h * 3, 90);
            std::vector<uint16_t> depth(size_t(frames) * w * h, 1500);
            cf_dataset* lab = nullptr;
            check(cf_dataset_create(r.ctx, frames, w, h, &lab) == CF_OK &&
                      cf_dataset_upload_raw_ex(lab, 0, frames, rgb.data(), depth.data(), 0, 1, 1) == CF_OK &&
                      cf_context_synchronize(r.ctx) == CF_OK,
                  "preprocessing", flips, 0);
            size_t before = 0, after = 0, total = 0;
            cudaMemGetInfo(&before, &total);
            armed = true;
            calls = 0;
            fail_at = 0;
            const cf_status s = r.call(best);
            armed = false;
            fail_at = -1;
            cudaMemGetInfo(&after, &total);
            check(s == CF_OK && same(best, want), "a refused allocation with scratch kept", flips, s);
            check(after > before + (size_t(16) << 20), "scratch given back", flips, static_cast<long long>(after) - static_cast<long long>(before));
            check(cf_dataset_upload_raw_ex(lab, 0, frames, rgb.data(), depth.data(), 0, 1, 1) == CF_OK, "preprocessing again", flips, 0);
            cf_dataset_destroy(lab);
        }
        // 20 tiles of 96 kB; the other allocations of the call are smaller
        const Level wide(flips != 0, 640);
        count_calls(wide, 0, want, &staged);
        check(staged == 0, "one pass of the wide level", flips, staged);
        for (int mb : {1, 2, 4}) {
            Run r(wide, 2, mb);
            armed = true;
            largest = 0;
            const cf_status s = r.call(best, &staged);
            armed = false;
            check(s == CF_OK && same(best, want), "splits with a bounded table", flips, mb);
            check(staged >= 1 && largest <= size_t(mb) << 20, "bytes of a bounded table", flips, static_cast<long long>(largest));
            std::printf("flips %d, stage_max_mb %d: %lld launches of pass 1, largest allocation %zu\n", flips, mb,
                        static_cast<long long>(staged), largest);
        }
    }
    std::printf("%d failures\n", failures);
    return failures != 0;
}
