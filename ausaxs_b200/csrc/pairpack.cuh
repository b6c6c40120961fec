// Pair-distance histograms with one shared-memory atomic per pair (the unweighted O(N^2) stage).
#pragma once
#include "common.cuh"

namespace ausaxs_b200 {

// One pass of pair binning: outer set A (index i) against inner set B (index j).  The count row of a
// pair is the outer point's type (rows > 1) or row 0; an atom-atom pass is therefore one job per inner
// type, over the list of that type's atoms (typed_lists_launch) in ascending atom index.
struct alignas(16) PackJob {
    const float4* A;
    const float4* B;
    int32_t na, nb;
    int32_t self;         // 1: only pairs whose inner point has the larger index in the (shared) set
    int32_t indexed;      // 1: the index of an inner point in its set is its w (ascending); 0: its position
    const int32_t* pre;   // self && indexed: pre[c] = inner points with index < 256 c
    int64_t tile_begin;   // first tile id of the job
    int32_t tiles_i, tiles_j;  // outer tiles, inner tiles (self: an upper bound for every outer tile)
    int32_t rows, nbins;
    float inv_w;          // float(1 / bin_width)
    float c, scale;       // fixed-point offsets (pair_residual)
    int32_t seg_pairs;    // pairs of the first segments (pack_segment_pairs)
    // where the pairs sit in the reference's loops (PairJob)
    int32_t a_base, b_base, tail_end, tail_from_outer;
    // Jobs of a group keep their counts and offset sums on chip side by side (same nbins): group_rows count
    // rows, this job's from cnt_row on, and group_sums offset sums, this job's sum_slot.  Row r of the
    // group goes to out[group_out + r], offset sum s to out[group_out + group_rows + s].
    int32_t group, group_out, group_rows, group_sums;
    int32_t cnt_row, sum_slot;
    int32_t mult;         // multiplicity of every pair (jobs of a group share it)
    int32_t copies;       // packed words of every row: a power of two, lanes take turns (pack_copies)
};
static_assert(sizeof(PackJob) == 128, "copied in 16-byte words");

struct PackLaunch {
    const PackJob* jobs;
    unsigned long long* const* out;  // u64 accumulators [nbins] of every group's rows and offset sums
    int32_t n_jobs;
    int64_t total_tiles;
    int32_t rows;         // most packed rows (rows x copies) of a job
    int32_t group_rows, group_sums;  // most rows and offset sums of a group
    int32_t bins;         // most bins of a job
    int32_t tile_j;       // inner points per tile (a multiple of 4, at most kPackMaxTileJ)
    unsigned long long* tile_counter;
    unsigned long long* overflow;
    int32_t nr;           // 1: every job's width is verified for the Newton-Raphson root; 2: and is a power of two
    int32_t offsets;      // 0: no job has offset sums (counts only)
    int32_t many;         // 1: some job keeps several copies of its words
    int32_t covered;      // 1: no pair's distance lies beyond its job's bins
    int32_t max_tiles;    // > 0: a CTA exits after this many tiles (grid * max_tiles >= total_tiles)
};

constexpr int kPackMaxTileJ = 512;
constexpr int kPackPre = 256;      // granularity of PackJob::pre; outer tiles are multiples of it
constexpr int kPackCountShift = 23;
constexpr int kPackMaxPairs = 65536 - 1;  // pairs of a segment: what the check of a segment needs (pairpack.cu)

// CTA shapes: threads, thread groups that split a tile's inner points, outer points per tile
struct PackShape {
    int threads, groups;
    int outer() const { return threads / groups * 2; }
};
constexpr PackShape kPackShapes[] = {{128, 1}, {256, 1}, {256, 2}, {512, 2}};

// footprint of a launch with L's rows, bins and tile_j
size_t pack_smem_bytes(const PackLaunch& L);
// resident CTAs per SM of a shape with L's footprint (0: does not fit)
int pack_ctas_per_sm(int shape, const PackLaunch& L);
// shape of a launch by its footprint, -1 when it does not fit (pairpack.cu)
int pack_shape(const PackLaunch& L);
// pairs of a job's first segments: the most frequent cell of a protein-like distance distribution
// then holds about 100 pairs
int pack_segment_pairs(int bins, double largest_row_share);
// copies of the packed words of a job of `rows` rows whose distances spread over `spread` of the launch's bins
int pack_copies(int rows, int bins, int spread, double largest_row_share);
// Adds the pairs of a sample whose packed evaluation differs from the scalar one to *mismatches.
void pack_check_launch(float inv_w, int bins, bool power_of_two, unsigned long long* mismatches, cudaStream_t s);
void pack_launch(const PackLaunch& L, int shape, int grid, cudaStream_t s);

}  // namespace ausaxs_b200
