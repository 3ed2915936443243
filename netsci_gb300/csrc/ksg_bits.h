// KSG joint search on rank bitmaps (ksg_bits.cuh): launch configuration.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "ksg_grid.h"

namespace nsg {

constexpr int kBitTries = 12;     // search radii tried before a query scans all frames
// Bitmap hits per wanted frame from which a first radius is cut back unseen,
// and the next ones (another look takes as long as evaluating 400 frames, and
// three times that in rows of four words a lane).
constexpr int kCrowd = 10, kCrowdTries = 3;
__host__ __device__ constexpr int crowds(int words) { return words == 4 ? 200 : 60; }
// A k-th distance below this share of a crowded radius cuts the warp's scale,
// which stays between kLeastScale and its inverse; the least radius looked at.
constexpr float kFar = 0.45f;
constexpr float kLeastScale = 0.05f;
constexpr float kLeastH = 1e-30f;
// Queries a warp takes at a time, at most: a lane per query and coordinate.
__host__ __device__ constexpr int bit_queries(int d) { return d == 3 ? 4 : 8; }
// Shared words per warp: queries, the 32 n nearest frames' distances, bins, bit_of_rank's table.
__host__ __device__ constexpr int bit_warp_words(int d, int n) {
    return bit_queries(d) * 8 + 96 * n + 4 + bit_queries(d) * 4 * d + 32;
}

// Words of one bitmap row over m frames: whole 16-byte groups, an odd number
// of them, so that the lanes that store one word each of successive rows
// spread over the banks.
__host__ __device__ inline int bit_row_words(int m) { return ((((m + 31) / 32 + 3) / 4) | 1) * 4; }

struct BitsArgs {
    GridArgs g;
    int chunks;                 // work items: g.npairs * chunks
    int grab;                   // queries a warp takes at a time (at most bit_queries)
    int rows, step;             // rows per coordinate, bins per row
    int rows_words, perm_words; // shared-memory layout (words)
};

struct BitsConfig {
    bool ok = false;
    int words = 0;              // words a lane ANDs at a time: 1, 2 or 4
    int keep = 0;               // frames within the search radius a query keeps, in 32s
    int threads = 0, ctas_per_sm = 0;
    int rows = 0, step = 0, rows_words = 0, perm_words = 0;
    size_t smem = 0;
};
// Shared-memory layout and CTA size for pairs of up to max_m frames; not ok
// where the rows of such a pair do not fit.
BitsConfig bits_config(int d, int k, int max_m);
// Runs of pairs (sorted by falling m) that share a configuration, for a
// batch whose longest pair has one: one search launch each, at most
// kBitSegments.
struct BitsSegment {
    int first, npairs, max_m;
    BitsConfig config;
};
constexpr int kBitSegments = 4;
std::vector<BitsSegment> bits_segments(const KsgPairDesc* descs, int npairs, int d, int k);
// Scale estimates of node grids (grid_launch_nodes) of up to max_m frames.
void bits_launch_est(const GridNode* nodes, int nnodes, int max_m, int d, cudaStream_t s);
// The search of one segment of a batch (the nodes carry scale estimates);
// takes what grid_launch_search takes for the batch, but no pair grids, and a
// counter of the segment's own, zero before the launch.
void bits_launch_search(const GridArgs& g, const BitsSegment& seg, int* counter, int d, cudaStream_t s);

}  // namespace nsg
