// Pass 1 of the staged split search: every (sample, feature) of a level gets its threshold bin.
//
// A response reads eight corners of the sample's integral images, and the lanes of a corner load (one sample
// each) fall in as many 128-byte lines, so a load of 32 lanes takes 8 cycles of the L1 tag pipe however its
// data lies: 64 of them per 32 evaluations, 80 with the parameters and the threshold search. That pipe is
// what bounds the pass (75 % of its peak, issue 55 %); the kernel is laid out to need little else:
//   - 170 instructions per 32 evaluations (feature_bin of eval_fast.cuh: 311). Depth scaling is the
//     reference's trunc(RN(v / d)): every sample brings a float i with floor(v i) = trunc(RN(v / d)) for every
//     magnitude v that the level's candidates hold, checked value by value (RN(1 / d) or the next float serves
//     99.9 % of the depths in whole millimetres; rows of other depths take the general kernel). v i + 2^23
//     rounded toward zero is then one instruction for two values, and corner offsets are computed as floats
//     whose bits are the integer;
//   - an SM keeps 32 neighbouring samples at a time (frame and Morton order), and its 24 warps walk their features
//     side by side, so the patch that the corners lie in stays in L1: misses cost cycles of the same pipe.
// 800 000 samples, 4000 features x 32 thresholds (100 frames 640x480, a sample per 38 pixels): 49.0 ms with 256
// samples x 64 features a CTA, 31.5 ms with two CTAs of 64 samples and a barrier per 128 features, 28.2 ms this way.
// A tree of 266 600 samples, 2000 x 20 (200 frames, a sample per 230 pixels; hit rate 54 % with the barriers): 145.6 ms,
// then 103.2 ms over its 19 levels; 8 M samples on 1000 frames: 519, 320 and 294 ms.
//
// The bin is the one feature_bin gives, in every case: depth means are compared in float with an error
// bound and a threshold within it is decided by the exact division; colour sums are exact in double.
#include <algorithm>
#include <climits>
#include <cmath>

#include <cub/device/device_radix_sort.cuh>

#include "box_fast.cuh"
#include "stage.h"

namespace cf {

namespace {

constexpr int kThreads = 768;         // 24 warps of 80 registers (512: 2 %, 1024 with 64 registers: 1 % slower)
constexpr int kRows = 32;             // samples of a CTA, one to a lane (64, or two CTAs of 32: 10-20 % slower)
constexpr int kStep = 2;              // features of a copy to shared memory (4: more of it, 2 % slower)
// Features per work item of the general kernel. Where it takes the few rows without a checked reciprocal, 64 kept one
// CTA 45-90 us on those of a small level, 16 do not. Where it takes all rows, 32 set up a tile and fetch a sample half
// as often, once there are kManyItems work items of 32 features per resident CTA. Of 16 / 32 / 64, in ms: 20 000 rows x
// 300 features 0.261 / 0.363 / 0.537, x 1000 (5.7 items a CTA) 0.572 / 0.578 / 0.963; 50 000 x 500 (7.1) 0.791 / 0.728 /
// 0.947; 266 600 x 1000 6.25 / 5.88 / 5.90 (100 thresholds); 100 000 x 500 of 1920x1080 1.50 / 1.35 / 1.57.
constexpr int kSmallTile = 16, kLargeTile = 32;
constexpr long long kManyItems = 6;
constexpr int kGeneralCtasPerSm = 3;

// Floats of a feature's row: eight parameters, +-2^23 with the sign of each offset, then the ascending
// thresholds padded with +inf: 32 entries serve T <= 31, 36 T = 32, 64 T <= 63.
constexpr int kRowParams = 12;
constexpr int kMaxPaddedT = 63;
int feature_row(int T) { return T < 32 ? kRowParams + 32 : T == 32 ? kRowParams + 36 : kRowParams + 64; }
// Entries of all feature rows, in whole units; where there are no rows (row = 0) their parameters alone are walked.
long long feature_floats(int F, int row) {
    return (F + kStageUnit - 1ll) / kStageUnit * kStageUnit * std::max(row, kRowParams);
}

// Unit lists: depth features, the nine channel pairs, the rest (channels past 2).
__device__ __forceinline__ int pair_code(const FeatParams& f) {
    if (f.type == kDepthFeature) return 0;
    return f.ch1 < 3 && f.ch2 < 3 ? 1 + f.ch1 * 3 + f.ch2 : kStageCodes - 1;
}

// The candidates laid out for the kernels below. Blocks past `row_blocks` take a feature chunk each: the
// 8-feature blocks of every code (a block with features of several codes is listed in each, with the mask of its
// features), by one warp in block order. The others write the feature rows (row = 0: none) and find the largest
// magnitude that a candidate of the level scales by a depth.
__global__ void __launch_bounds__(256)
stage_plan_kernel(int F, int T, int row, int row_blocks, int chunk, int cap, const FeatParams* __restrict__ packs,
                  const float* __restrict__ sorted_thr, float* __restrict__ rows, int* __restrict__ reach,
                  uint32_t* __restrict__ units, int* __restrict__ unit_count) {
    const int lane = threadIdx.x & 31;
    if (static_cast<int>(blockIdx.x) < row_blocks) {
        const long long i = blockIdx.x * 256ll + threadIdx.x;
        const int per = max(row, kRowParams);
        const int f = static_cast<int>(i / per), k = static_cast<int>(i - static_cast<long long>(f) * per);
        float v = 0.0f;
        if (f < (F + kStageUnit - 1) / kStageUnit * kStageUnit) {
            if (k < kRowParams) {
                const FeatParams p = f < F ? packs[f] : FeatParams{};   // whole units: the rows past F hold zeros
                const int8_t par[8] = {p.o1x, p.o1y, p.o2x, p.o2y, p.r1x, p.r1y, p.r2x, p.r2y};
                v = k < 8 ? static_cast<float>(par[k]) : par[k - 8] < 0 ? -8388608.0f : 8388608.0f;
            } else {
                const int t = k - kRowParams;
                v = t < T && f < F ? sorted_thr[static_cast<long long>(f) * T + t] : INFINITY;
            }
            if (row > 0) rows[i] = v;
        }
        const int m = __reduce_max_sync(0xffffffffu, k < 8 ? static_cast<int>(fabsf(v)) : 0);
        if (lane == 0) atomicMax(reach, m);
        return;
    }
    const int ch = static_cast<int>(blockIdx.x) - row_blocks;
    const int f0 = ch * chunk, n = min(chunk, F - f0);
    const int blocks = (n + kStageUnit - 1) / kStageUnit;
    uint32_t* mine = units + static_cast<long long>(ch) * kStageCodes * cap;
    if (threadIdx.x >= 32) return;
    int count = 0;   // of code `lane`
    for (int b0 = 0; b0 < blocks; b0 += 32) {
        const int b = b0 + lane;
        u64 codes = ~0ull;   // 4 bits per feature, 15: none
        for (int j = 0; j < kStageUnit; j++) {
            const int f = b * kStageUnit + j;
            const u64 c = b < blocks && f < n ? pair_code(packs[f0 + f]) : 15;
            codes = (codes & ~(15ull << (4 * j))) | (c << (4 * j));
        }
        for (int c = 0; c < kStageCodes; c++) {
            uint32_t mask = 0;
            for (int j = 0; j < kStageUnit; j++)
                if (((codes >> (4 * j)) & 15ull) == static_cast<u64>(c)) mask |= 1u << j;
            const unsigned bal = __ballot_sync(0xffffffffu, mask != 0);
            const int at = __shfl_sync(0xffffffffu, count, c) + __popc(bal & ((1u << lane) - 1u));
            if (mask) mine[c * cap + at] = static_cast<uint32_t>(b) << 8 | mask;
            if (lane == c) count += __popc(bal);
        }
    }
    if (lane < kStageCodes) unit_count[ch * kStageCodes + lane] = count;
}

// Rows of the table: row_base[n] + k is sample k of node n; with `both`, row rows + r is the flipped response of
// row r's sample, used where that sample is evaluated both ways (flip 2). Pass 1 takes them frame by frame and
// within a frame in Morton (Z) order of (y, x), so that the rows a CTA takes lie in a compact patch; rows without
// a checked reciprocal come after the others in the same order, unused rows last.
__global__ void stage_rows_kernel(const NodeDesc* __restrict__ nodes, const long long* __restrict__ row_base, int M,
                                  long long rows, int both, const Sample* __restrict__ samples,
                                  const int* __restrict__ reach, int padded, int morton_bits, int frame_bits,
                                  int* __restrict__ row_pos, uint8_t* __restrict__ row_label,
                                  uint8_t* __restrict__ row_both, u64* __restrict__ key, int* __restrict__ row_ids,
                                  float* __restrict__ row_inv) {
    const long long r = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (r >= rows) return;
    int lo = 0, hi = M - 1;   // the last node n with row_base[n] <= r
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (row_base[mid] <= r) lo = mid;
        else hi = mid - 1;
    }
    const long long p = nodes[lo].start + (r - row_base[lo]);
    const Sample s = samples[p];
    row_pos[r] = static_cast<int>(p);
    row_label[r] = s.label;
    row_ids[r] = static_cast<int>(r);
    float inv = 1.0f;   // an invalid depth scales nothing
    if (s.depth > 0.0f)
        inv = s.depth >= 1e-3f && s.depth <= 1e6f ? checked_reciprocal(s.depth, *reach) : 0.0f;   // |v / d| < 2^18
    if (!padded) inv = 0.0f;
    row_inv[r] = inv;
    const int general_bit = morton_bits + frame_bits;
    const u64 k = (inv == 0.0f ? 1ull << general_bit : 0ull) | static_cast<u64>(s.image) << morton_bits |
                  spread_bits(s.y) << 1 | spread_bits(s.x);
    key[r] = k;
    if (both) {
        row_both[r] = s.flip == 2 ? 1 : 0;
        row_ids[rows + r] = static_cast<int>(rows + r);
        key[rows + r] = s.flip == 2 ? k : 3ull << general_bit;
    }
}

// The rows in key order; ends[0]: the first without a checked reciprocal, ends[1]: the first unused one.
__global__ void stage_list_kernel(long long rows, long long list_rows, int general_bit, const u64* __restrict__ key,
                                  const int* __restrict__ order, const int* __restrict__ row_pos,
                                  const Sample* __restrict__ samples, const float* __restrict__ row_inv,
                                  int* __restrict__ ends, StageSample* __restrict__ out) {
    const long long k = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    if (k >= list_rows) return;
    const int row = order[k];
    const int from = row < rows ? row : row - static_cast<int>(rows);
    const Sample s = samples[row_pos[from]];
    StageSample o;
    o.x = s.x;
    o.y = s.y;
    o.image = s.image;
    o.row = static_cast<uint32_t>(row) | (s.flip == 1 || row >= rows ? 0x80000000u : 0u);
    o.inv_d = s.depth > 0.0f ? row_inv[from] : 0.0f;
    out[k] = o;
    // 0: gathered, 1: general, 3: unused; the first position of what follows each
    const int kind = static_cast<int>(key[k] >> general_bit);
    const int before = k > 0 ? static_cast<int>(key[k - 1] >> general_bit) : 0;
    if (kind >= 1 && (k == 0 || before < 1)) ends[0] = static_cast<int>(k);
    if (kind >= 3 && (k == 0 || before < 3)) ends[1] = static_cast<int>(k);
    if (k == list_rows - 1) {
        if (kind < 1) ends[0] = static_cast<int>(list_rows);
        if (kind < 3) ends[1] = static_cast<int>(list_rows);
    }
}

struct StageArgs {
    DsView ds;
    const Sample* samples;    // the level's samples
    const int* row_pos;
    long long rows;           // of the table
    long long sample_rows;    // rows past these hold flipped responses
    const StageSample* list;
    const int* order;
    const int* ends;          // list positions: first row without a checked reciprocal, first unused row
    const FeatParams* packs;
    const float* sorted_thr;  // [F][T]
    const float* feature_rows;
    int T;
    int f_first, n_feat;      // the chunk's features [f_first, f_first + n_feat)
    const uint32_t* units;    // [codes][cap]
    const int* unit_count;    // [codes]
    int cap;
    int parts;                // work items per block of rows
    uint8_t* out;             // [n_feat / 32 blocks][rows][32]
};

__device__ __forceinline__ uint8_t* bin_place(const StageArgs& a, int g, long long row) {
    return a.out + (((g >> 5) * a.rows + row) << 5) + (g & 31);
}

__device__ __forceinline__ void cp_async16(void* shared, const void* global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(shared))),
                 "l"(global)
                 : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

// Thresholds below v of a padded row (32 entries serve T <= 31, 36 T = 32, 64 T <= 63): halving, on a byte
// offset so that a step is a read, a compare and an addition.
template <int kRow>
__device__ __forceinline__ int row_below(const float* t, float v) {
    const char* at = reinterpret_cast<const char*>(t);
    auto entry = [&](int k) { return *reinterpret_cast<const float*>(at + 4 * k); };
    constexpr int kEntries = kRow - kRowParams;
    if (kEntries == 64) {
        if (t[31] < v) at += 128;
    }
    if (entry(15) < v) at += 64;
    if (entry(7) < v) at += 32;
    if (entry(3) < v) at += 16;
    if (entry(1) < v) at += 8;
    if (entry(0) < v) at += 4;
    const int k = static_cast<int>(at - reinterpret_cast<const char*>(t)) >> 2;
    return kEntries == 36 ? k + (t[31] < v ? 1 : 0) : k;
}

__device__ __forceinline__ Corners row_corners(const BoxLane& l, const float* row, const FrameView& p) {
    const ulonglong2 o = *reinterpret_cast<const ulonglong2*>(row);          // o1, o2
    const ulonglong2 g = *reinterpret_cast<const ulonglong2*>(row + 4);      // r1, r2
    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(row + 8);      // 2^23 with the offsets' signs
    return corners(l, o.x, o.y, g.x, g.y, b.x, b.y, p);
}

// Bin of a depth feature; `open` where it still has to be found from the boxes (a threshold lies between the
// bounds, or a count is no plain one).
template <int kRow>
__device__ __forceinline__ int depth_bin(const BoxLane& l, const float* row, const unsigned char* frame,
                                         const FrameView& p, int T, DepthBoxes& box, bool& open) {
    const Corners k = row_corners(l, row, p);
    box = depth_boxes(k, frame);
    const DepthBounds d = depth_bounds(box);
    const float* t = row + kRowParams;
    const int bin = row_below<kRow>(t, d.lo);
    const bool some = k.in && box.n1 != 0 && box.n2 != 0;
    open = some && !(t[bin] > d.hi && d.plain);
    return some ? bin : T;
}

template <int kRow>
__device__ __noinline__ int open_bin(int s1, int n1, int s2, int n2, const float* t) {
    return row_below<kRow>(t, __double2float_ru(exact_depth_response(s1, n1, s2, n2)));
}

template <int kRow>
__device__ __forceinline__ int color_bin(const BoxLane& l, const float* row, const unsigned char* frame,
                                         const FrameView& p, int T) {
    const Corners k = row_corners(l, row, p);
    const double r = color_response(k, frame);
    const int bin = row_below<kRow>(row + kRowParams, __double2float_ru(r));
    return k.in && !isnan(r) ? bin : T;
}

// One work item = 32 rows of the list x the chunk's features (in `parts` parts where there are few rows), its
// features in units of eight. A warp's lanes keep the 32 samples. The warps of a CTA take the next unit of its items
// in turn: they stay on the same rows and on neighbouring features, so that their corners share L1, without waiting
// for one another (with a barrier per 128 features: 17 % slower on 500 features). The rows of the next two features
// are copied to the warp's own shared memory while two are evaluated, whose gathers overlap; a unit's bins are stored
// as one 8-byte word.
template <int kRow>
__global__ void __launch_bounds__(kThreads, 1)
stage_gather_kernel(const __grid_constant__ StageArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ unsigned s_next;   // units of this CTA's items that are taken
    const int T = a.T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    float* rows = reinterpret_cast<float*>(smem) + warp * 2 * kStep * kRow;   // two steps of the warp's
    if (threadIdx.x == 0) s_next = 0;
    __syncthreads();
    // lane c: the units of codes 0 .. c
    int upto = lane < kStageCodes - 1 ? a.unit_count[lane] : 0;
    for (int o = 1; o < kStageCodes; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += v;
    }
    const int n_units = __shfl_sync(0xffffffffu, upto, kStageCodes - 2);
    const unsigned per = (n_units + a.parts - 1) / a.parts;   // units of an item; a last part may hold fewer
    const int end = a.ends[0];
    const int items = static_cast<int>((end + kRows - 1ll) / kRows) * a.parts;
    if (n_units == 0) return;

    BoxLane l;
    FrameView view;
    view.xmax = static_cast<float>(a.ds.width - 1);
    view.ymax = static_cast<float>(a.ds.height - 1);
    const int plane = static_cast<int>(a.ds.plane) * 4;
    const unsigned char *depth = nullptr, *color = nullptr;
    bool have = false, valid = false;
    int row = 0, block = -1;

    // the next unit of this CTA's items: its item, and the entry of its list with the code above bit 28
    auto take = [&](int& item, uint32_t& unit) {
        for (;;) {
            unsigned q = 0;
            if (lane == 0) q = atomicAdd(&s_next, 1u);
            q = __shfl_sync(0xffffffffu, q, 0);
            const unsigned turn = q / per;
            const long long at = blockIdx.x + static_cast<long long>(turn) * gridDim.x;
            item = at < items ? static_cast<int>(at) : -1;
            if (item < 0) return;
            const int u = static_cast<int>(item % a.parts * per + (q - turn * per));
            if (u >= n_units) continue;
            const int c = __popc(__ballot_sync(0xffffffffu, lane < kStageCodes - 1 && upto <= u));
            const int first = __shfl_sync(0xffffffffu, upto, max(c - 1, 0));
            unit = __ldg(a.units + c * a.cap + u - (c > 0 ? first : 0)) | static_cast<uint32_t>(c) << 28;
            return;
        }
    };
    auto fetch = [&](uint32_t unit, int step) {
        const int f0 = a.f_first + static_cast<int>(unit >> 8 & 0xFFFFFu) * kStageUnit + step * kStep;
        const float* from = a.feature_rows + static_cast<long long>(f0) * kRow;
        float* to = rows + (step & 1) * kStep * kRow;
        for (int i = lane; i < kStep * kRow / 4; i += 32) cp_async16(to + 4 * i, from + 4 * i);
    };

    int next_item;
    uint32_t next = 0;
    take(next_item, next);
    if (next_item >= 0) fetch(next, 0);
    cp_async_commit();
    while (next_item >= 0) {
        const uint32_t unit = next;
        const int blk = next_item / a.parts;
        if (blk != block) {
            block = blk;
            const long long k = static_cast<long long>(blk) * kRows + lane;
            have = k < end;
            const StageSample s = a.list[have ? k : end - 1];
            valid = s.inv_d > 0.0f;
            const float inv = valid ? s.inv_d : 1.0f;
            l.pos = pack_f2(static_cast<float>(s.x), static_cast<float>(s.y));
            l.inv = pack_f2(inv, inv);
            l.side = pack_f2(s.row >> 31 ? -1.0f : 1.0f, 1.0f);
            row = static_cast<int>(s.row & 0x7FFFFFFFu);
            depth = reinterpret_cast<const unsigned char*>(a.ds.depth + s.image * a.ds.plane);
            color = reinterpret_cast<const unsigned char*>(a.ds.color + s.image * 3ll * a.ds.plane);
        }
        take(next_item, next);
        const int code = unit >> 28;
        uint32_t lo = 0, hi = 0;
#pragma unroll 1
        for (int step = 0; step < kStageUnit / kStep; step++) {
            if (step + 1 < kStageUnit / kStep) fetch(unit, step + 1);
            else if (next_item >= 0) fetch(next, 0);
            cp_async_commit();
            cp_async_wait<1>();
            __syncwarp();
            const float* r = rows + (step & 1) * kStep * kRow;
            int b0, b1;
            if (code == 0) {
                view.size = __int_as_float(8);
                view.pitch = __int_as_float(8 * a.ds.width);
                view.base1 = view.base2 = 0.0f;
                DepthBoxes x0, x1;
                bool open0, open1;
                b0 = depth_bin<kRow>(l, r, depth, view, T, x0, open0);
                b1 = depth_bin<kRow>(l, r + kRow, depth, view, T, x1, open1);
                if (open0) b0 = open_bin<kRow>(x0.s1, x0.n1, x0.s2, x0.n2, r + kRowParams);
                if (open1) b1 = open_bin<kRow>(x1.s1, x1.n1, x1.s2, x1.n2, r + kRow + kRowParams);
            } else {
                view.size = __int_as_float(4);
                view.pitch = __int_as_float(4 * a.ds.width);
                view.base1 = __int_as_float((code - 1) / 3 * plane);
                view.base2 = __int_as_float((code - 1) % 3 * plane);
                b0 = color_bin<kRow>(l, r, color, view, T);
                b1 = color_bin<kRow>(l, r + kRow, color, view, T);
            }
            lo = __byte_perm(lo, hi, 0x5432);                        // (hi, lo) moves down two bytes
            hi = __byte_perm(hi, __byte_perm(b0, b1, 0x0040), 0x5432);
            __syncwarp();   // the step is read: the next copy may overwrite it
        }
        if (!valid) lo = hi = static_cast<uint32_t>(T) * 0x01010101u;
        if (have) {
            const uint32_t mask = unit & 255u;
            uint8_t* to = bin_place(a, static_cast<int>(unit >> 8 & 0xFFFFFu) * kStageUnit, row);
            if (mask == 255u) {
                *reinterpret_cast<uint2*>(to) = make_uint2(lo, hi);
            } else {
                const u64 word = static_cast<u64>(hi) << 32 | lo;
                for (int i = 0; i < kStageUnit; i++)
                    if (mask >> i & 1u) to[i] = static_cast<uint8_t>(word >> (8 * i));
            }
        }
    }
}

// feature_bin itself: rows without a checked reciprocal with all features, then all rows with the features of
// other channels. One work item = 256 consecutive rows of the list x up to kTile features.
template <int kPad, int kTile>
__global__ void __launch_bounds__(256, kGeneralCtasPerSm)
stage_general_kernel(const __grid_constant__ StageArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    EvalFeat* s_params = reinterpret_cast<EvalFeat*>(smem);
    float* s_thr = reinterpret_cast<float*>(smem + sizeof(EvalFeat) * kTile);
    __shared__ uint32_t s_unit[kTile / kStageUnit];
    constexpr int kUnits = kTile / kStageUnit;
    const int T = a.T;
    const int TP = kPad ? kPad : T;
    const int W = a.ds.width, H = a.ds.height;
    for (int seg = 0; seg < 2; seg++) {
        const int code_a = seg == 0 ? 0 : kStageCodes - 1, code_b = seg == 0 ? kStageCodes - 1 : kStageCodes;
        int n_units = 0;
        for (int c = code_a; c < code_b; c++) n_units += a.unit_count[c];
        const long long begin = seg == 0 ? a.ends[0] : 0, end = a.ends[1];
        const int tiles = (n_units + kUnits - 1) / kUnits;
        const long long items = (end - begin + 255) / 256 * tiles;
        for (long long q = blockIdx.x; q < items; q += gridDim.x) {
            const long long blk = q / tiles;
            const int j = static_cast<int>(q - blk * tiles);
            const int nu = min(kUnits, n_units - j * kUnits);
            __syncthreads();   // the previous item's reads of the tile are done
            if (static_cast<int>(threadIdx.x) < nu) {
                int v = j * kUnits + threadIdx.x, c = code_a;
                while (v >= a.unit_count[c]) v -= a.unit_count[c++];
                s_unit[threadIdx.x] = a.units[c * a.cap + v];
            }
            __syncthreads();
            for (int i = threadIdx.x; i < nu * kStageUnit; i += blockDim.x) {
                const int g = static_cast<int>(s_unit[i / kStageUnit] >> 8) * kStageUnit + i % kStageUnit;
                if (g < a.n_feat) s_params[i] = make_eval_feat(a.packs[a.f_first + g]);
            }
            for (int i = threadIdx.x; i < nu * kStageUnit * TP; i += blockDim.x) {
                const int f = i / TP, t = i - f * TP;
                const int g = static_cast<int>(s_unit[f / kStageUnit] >> 8) * kStageUnit + f % kStageUnit;
                s_thr[i] = t < T && g < a.n_feat ? a.sorted_thr[static_cast<long long>(a.f_first + g) * T + t] : INFINITY;
            }
            __syncthreads();
            const long long k = begin + blk * 256 + threadIdx.x;
            if (k >= end) continue;
            const int row = a.order[k];
            const int from = row < a.sample_rows ? row : row - static_cast<int>(a.sample_rows);
            const Sample smp = a.samples[a.row_pos[from]];
            const EvalPixel px = make_eval_pixel(a.ds, smp);
            const bool flip = smp.flip == 1 || row >= a.sample_rows;
            for (int u = 0; u < nu; u++) {
                const uint32_t unit = s_unit[u];
                const uint32_t mask = unit & 255u;
                uint8_t* to = bin_place(a, static_cast<int>(unit >> 8) * kStageUnit, row);
                u64 word = 0;
                for (int i = 0; i < kStageUnit; i += 2) {
                    const int f = u * kStageUnit + i;
                    int b0 = 0, b1 = 0;
                    if (mask >> i & 1u) b0 = feature_bin(px, W, H, s_params[f], flip, SortedBins<kPad>{s_thr + f * TP, T});
                    if (mask >> i & 2u)
                        b1 = feature_bin(px, W, H, s_params[f + 1], flip, SortedBins<kPad>{s_thr + (f + 1) * TP, T});
                    word |= static_cast<u64>(static_cast<uint32_t>(b0 | b1 << 8)) << (8 * i);
                }
                if (mask == 255u) {
                    *reinterpret_cast<u64*>(to) = word;
                } else {
                    for (int i = 0; i < kStageUnit; i++)
                        if (mask >> i & 1u) to[i] = static_cast<uint8_t>(word >> (8 * i));
                }
            }
        }
    }
}

template <typename K>
void set_smem(K kernel, size_t smem, int ctas) {
    // the carveout that just holds the resident CTAs; the rest of the unified memory caches the gathers
    const double need = ctas * (smem + 2048.0);
    CF_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    CF_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       std::min(100, static_cast<int>(std::ceil(100.0 * need / (228.0 * 1024))))));
}

template <int kPad, int kTile>
void launch_general(cf_context* ctx, const char* name, const StageArgs& a) {
    const int TP = kPad ? kPad : a.T;
    const size_t smem = sizeof(EvalFeat) * kTile + sizeof(float) * kTile * TP;
    set_smem(stage_general_kernel<kPad, kTile>, smem, kGeneralCtasPerSm);
    launch(ctx, name, dim3(ctx->num_sms * kGeneralCtasPerSm), dim3(256), smem, stage_general_kernel<kPad, kTile>, a);
}

template <int kTile>
void launch_general(cf_context* ctx, const char* name, const StageArgs& a) {
    switch (padded_row(a.T)) {
        case 32: launch_general<32, kTile>(ctx, name, a); break;
        case 64: launch_general<64, kTile>(ctx, name, a); break;
        default: launch_general<0, kTile>(ctx, name, a); break;
    }
}

}  // namespace

// The padded threshold rows serve T <= 63, the float offsets frames of up to 2^24 bytes of colour integrals
// (1280x960: 14.7 MB); otherwise every row takes the general kernel.
bool BinStager::gathers(const DsView& ds, int T) { return T <= kMaxPaddedT && ds.plane <= kMaxBoxPlane; }

void BinStager::reserve(cf_context* ctx, const DsView& ds, long long rows, bool both, const LevelFeatures& lf, int chunk,
                        int n_chunks) {
    sample_rows_ = rows;
    list_rows_ = both ? 2 * rows : rows;
    chunk_ = chunk;
    n_chunks_ = n_chunks;
    cap_ = (chunk + kStageUnit - 1) / kStageUnit;
    padded_ = gathers(ds, lf.T);
    int frame_bits = 1, pixel_bits = 1;
    while ((1ll << frame_bits) < ds.n) frame_bits++;
    while ((1 << pixel_bits) < std::max(ds.width, ds.height)) pixel_bits++;
    morton_bits_ = 2 * pixel_bits;
    frame_bits_ = frame_bits;
    reach_.reserve(1);
    units_.reserve(static_cast<size_t>(n_chunks) * kStageCodes * cap_);
    unit_count_.reserve(static_cast<size_t>(n_chunks) * kStageCodes);
    if (padded_) rows_f_.reserve(feature_floats(lf.F, feature_row(lf.T)));
    row_pos_.reserve(rows);
    row_inv_.reserve(rows);
    row_ids_.reserve(list_rows_);
    key_.reserve(list_rows_);
    key_sorted_.reserve(list_rows_);
    order_.reserve(list_rows_);
    list_.reserve(list_rows_);
    ends_.reserve(2);
    sort_bytes_ = 0;
    CF_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes_, key_.get(), key_sorted_.get(), row_ids_.get(),
                                                  order_.get(), static_cast<int>(list_rows_), 0, end_bit(), ctx->stream));
    sort_temp_.reserve(sort_bytes_);
}

void BinStager::release() {
    reach_.release();
    units_.release();
    unit_count_.release();
    rows_f_.release();
    row_pos_.release();
    row_inv_.release();
    row_ids_.release();
    key_.release();
    key_sorted_.release();
    order_.release();
    list_.release();
    ends_.release();
    sort_temp_.release();
}

void BinStager::prepare(cf_context* ctx, const DsView& ds, const Sample* samples, const NodeDesc* nodes_dev, int M,
                        const long long* row_base_dev, const LevelFeatures& lf, uint8_t* row_label, uint8_t* row_both) {
    const long long rows = sample_rows_;
    const bool both = list_rows_ > rows;
    cudaStream_t st = ctx->stream;
    const int row = padded_ ? feature_row(lf.T) : 0;
    const int row_blocks = static_cast<int>((feature_floats(lf.F, row) + 255) / 256);
    CF_CUDA_CHECK(cudaMemsetAsync(reach_.get(), 0, sizeof(int), st));
    launch(ctx, "stage_plan", dim3(row_blocks + n_chunks_), dim3(256), 0, stage_plan_kernel, lf.F, lf.T, row, row_blocks,
           chunk_, cap_, lf.packs.get(), lf.sorted_thr.get(), rows_f_.get(), reach_.get(), units_.get(),
           unit_count_.get());
    launch(ctx, "stage_rows", dim3(static_cast<unsigned>((rows + 255) / 256)), dim3(256), 0, stage_rows_kernel, nodes_dev,
           row_base_dev, M, rows, both ? 1 : 0, samples, static_cast<const int*>(reach_.get()), padded_ ? 1 : 0,
           morton_bits_, frame_bits_, row_pos_.get(), row_label, row_both, key_.get(), row_ids_.get(), row_inv_.get());
    CF_CUDA_CHECK(cub::DeviceRadixSort::SortPairs(sort_temp_.get(), sort_bytes_, key_.get(), key_sorted_.get(),
                                                  row_ids_.get(), order_.get(), static_cast<int>(list_rows_), 0, end_bit(),
                                                  st));
    launch(ctx, "stage_rows", dim3(static_cast<unsigned>((list_rows_ + 255) / 256)), dim3(256), 0, stage_list_kernel, rows,
           list_rows_, morton_bits_ + frame_bits_, static_cast<const u64*>(key_sorted_.get()), order_.get(), row_pos_.get(),
           samples, row_inv_.get(), ends_.get(), list_.get());
}

void BinStager::run(cf_context* ctx, const DsView& ds, const Sample* samples, const LevelFeatures& lf, int c,
                    uint8_t* out) {
    StageArgs a;
    a.ds = ds;
    a.samples = samples;
    a.row_pos = row_pos_.get();
    a.rows = list_rows_;
    a.sample_rows = sample_rows_;
    a.list = list_.get();
    a.order = order_.get();
    a.ends = ends_.get();
    a.packs = lf.packs.get();
    a.sorted_thr = lf.sorted_thr.get();
    a.feature_rows = rows_f_.get();
    a.T = lf.T;
    a.f_first = c * chunk_;
    a.n_feat = std::min(chunk_, lf.F - a.f_first);
    a.units = units_.get() + static_cast<size_t>(c) * kStageCodes * cap_;
    a.unit_count = unit_count_.get() + c * kStageCodes;
    a.cap = cap_;
    a.out = out;
    if (padded_) {
        auto kernel = lf.T < 32 ? stage_gather_kernel<kRowParams + 32>
                                : lf.T == 32 ? stage_gather_kernel<kRowParams + 36> : stage_gather_kernel<kRowParams + 64>;
        const size_t smem = sizeof(float) * (kThreads / 32) * 2 * kStep * feature_row(lf.T);
        set_smem(kernel, smem, 1);
        // few rows: their features in parts of at least 128, for about eight work items per CTA
        const long long blocks = (list_rows_ + kRows - 1) / kRows, slots = ctx->num_sms;
        a.parts = static_cast<int>(std::max<long long>(1, std::min<long long>((a.n_feat + 127) / 128, 8 * slots / blocks)));
        launch(ctx, "stage_bins", dim3(static_cast<unsigned>(std::min(slots, blocks * a.parts))), dim3(kThreads), smem,
               kernel, a);
    }
    const long long items = (list_rows_ + 255) / 256 * ((a.n_feat + kLargeTile - 1) / kLargeTile);
    const bool many = !padded_ && items >= kManyItems * ctx->num_sms * kGeneralCtasPerSm;
    const char* name = padded_ ? "stage_general" : "stage_bins";
    if (many) launch_general<kLargeTile>(ctx, name, a);
    else launch_general<kSmallTile>(ctx, name, a);
}

}  // namespace cf
