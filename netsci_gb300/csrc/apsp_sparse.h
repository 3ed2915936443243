// Min-plus steps and path walks over the finite entries of A only
// (apsp_sparse.cu); apsp.cu decides when a solve takes them.
#pragma once

#include <cuda_runtime.h>

namespace nsg {

// Rows of a matrix in slices of kSellRows rows: slice s holds
// ptr[s+1] - ptr[s] entries per row, entry e of row r of the slice at
// edges[(ptr[s] + e) * kSellRows + r] as (column, weight bits), columns
// ascending. Widths are multiples of kSellUnroll; shorter rows are padded
// with (0, +inf).
constexpr int kSellRows = 8;
constexpr int kSellUnroll = 4;
struct SellView {
    const int2* edges;
    const int* ptr;
    int nslices;
};
inline int sell_slices(int n) { return (n + kSellRows - 1) / kSellRows; }

// Largest n the sparse steps take (a column block of H has to fit in shared
// memory).
constexpr int kSparseMaxN = 14000;

// What a solve asks about A before it chooses its kernels (device words).
struct GraphInfo {
    int flags;      // bit 0 asymmetric, 1 non-zero diagonal, 2 negative or NaN, 3 non-integer
    int wmax;       // bits of the largest finite non-negative weight
    int width;      // sum of the slice widths: width * kSellRows entries with padding
    int entries;    // finite entries, without padding
};
// Fills *info, the per-row counts (n ints, zeroed by the caller together with
// *info) and the slice offsets ptr (sell_slices(n) + 1 ints).
void sparse_analyze(const float* A, int n, GraphInfo* info, int* counts, int* ptr, cudaStream_t s);
// Counts and slice offsets of an n x n matrix of row stride ld.
void sparse_count(const float* A, int ld, int n, GraphInfo* info, int* counts, int* ptr, cudaStream_t s);
void sparse_fill(const float* A, int ld, int n, const int* ptr, int2* edges, cudaStream_t s);

// Vertices by falling number of entries: order[r] is the vertex of rank r,
// rank its inverse (counts as sparse_analyze left them). Rows of one slice
// then have nearly the same length. The slice offsets and the entries of the
// relabelled matrix, and matrices in and out of the new labels.
void sparse_sort(const int* counts, int n, int* order, int* rank, cudaStream_t s);
void sparse_slices_sorted(const int* counts, const int* order, int n, GraphInfo* info, int* ptr, cudaStream_t s);
void sparse_fill_sorted(const float* A, int n, const int* order, const int* rank, const int* ptr, int2* edges,
                        cudaStream_t s);
void sparse_relabel(const float* A, float* out, int n, const int* order, cudaStream_t s);    // out[r][c] = A[order[r]][order[c]]
void sparse_restore(const float* A, float* out, int n, const int* order, const int* rank, cudaStream_t s);

// Hn[i][j] = min over the entries (k, a) of row j of fl(a + H[k][i]);
// changed[step] is set when an entry differs from H[i][j]. A step whose
// predecessor changed nothing returns at once, or, with `fill`, copies H.
void sparse_step(const SellView& g, const float* H, float* Hn, int n, int* changed, int step, bool fill,
                 cudaStream_t s);
// Estimated seconds of one such step.
double sparse_step_seconds(long long width, int n);
// Whether relabelled slices save more than they cost over `steps` steps (16 at
// most are counted on: a solve may converge early).
bool sparse_sort_pays(long long width, long long entries, int n, int steps);

// hedetniemi_walk_kernel (apsp.cu) over the columns of A; cols: the slices
// of A's transpose.
void sparse_walk(const SellView& cols, const float* H, const float* Hi, int* paths, float tolerance, int n, int L,
                 cudaStream_t s);

}  // namespace nsg
