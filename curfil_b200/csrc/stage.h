// Pass 1 of the staged split search: the threshold bin of every (sample, feature) of a level.
#pragma once

#include "features.h"

namespace cf {

// One open node of a level: its samples are [start, start + count) of the level's sample array.
struct NodeDesc {
    long long start;
    int count;
    int tree_index;
};

constexpr int kStageTile = 32;     // features per table block
constexpr int kStageUnit = 8;      // features a lane takes at a time
constexpr int kStageCodes = 11;    // unit lists: depth, the nine colour channel pairs, the rest

// One row of the pass-1 order.
struct __align__(16) StageSample {
    uint16_t x, y;
    uint32_t image;
    uint32_t row;                  // table row; bit 31: the flipped response is wanted
    float inv_d;                   // checked reciprocal of the depth; 0: invalid depth, every response is NaN
};

class BinStager {
public:
    // Whether the gather kernel serves such frames and thresholds.
    static bool gathers(const DsView& ds, int T);
    // Lays out a level of `rows` samples and n_chunks feature chunks of `chunk` features, and allocates everything that
    // prepare() and run() use. With `both` the table has twice the rows: row rows + r is the flipped response of row r
    // where row_both[r] (its sample has flip 2).
    void reserve(cf_context* ctx, const DsView& ds, long long rows, bool both, const LevelFeatures& lf, int chunk,
                 int n_chunks);
    void release();
    // Orders the level's rows (row_base[n] + k is sample k of node n) and lays out the candidates of its chunks.
    void prepare(cf_context* ctx, const DsView& ds, const Sample* samples, const NodeDesc* nodes_dev, int M,
                 const long long* row_base_dev, const LevelFeatures& lf, uint8_t* row_label, uint8_t* row_both);
    // The bins of chunk c: feature f of the chunk and table row r at out[((f / 32) * table rows + r) * 32 + f % 32].
    void run(cf_context* ctx, const DsView& ds, const Sample* samples, const LevelFeatures& lf, int c, uint8_t* out);

private:
    // key bits that are sorted: kind 0 (gathered) or 1 (general) above the frame, with flipped rows also 3 (unused)
    int end_bit() const { return morton_bits_ + frame_bits_ + (list_rows_ > sample_rows_ ? 2 : 1); }
    long long sample_rows_ = 0, list_rows_ = 0;
    int chunk_ = 0, n_chunks_ = 0, cap_ = 0;
    int morton_bits_ = 0, frame_bits_ = 0;   // of a row's sort key
    size_t sort_bytes_ = 0;
    bool padded_ = false;          // the level's thresholds and frames suit the gather kernel
    DevArray<unsigned long long> key_, key_sorted_;
    DevArray<int> row_pos_, row_ids_, order_;
    DevArray<float> row_inv_;      // [rows] checked reciprocal of each row's depth, 0 if there is none
    DevArray<StageSample> list_;   // [rows] in pass-1 order
    DevArray<int> ends_;           // list positions: first without a checked reciprocal, first unused
    DevArray<float> rows_f_;       // [F][row] scaled parameters and padded thresholds
    DevArray<uint32_t> units_;     // [chunks][codes][cap] first feature / 8 and the mask of its features
    DevArray<int> unit_count_;     // [chunks][codes]
    DevArray<int> reach_;          // largest magnitude of the level's candidates
    DevArray<unsigned char> sort_temp_;
};

}  // namespace cf
