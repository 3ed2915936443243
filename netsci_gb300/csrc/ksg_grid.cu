// Cell-grid KSG: grid construction kernels, the instantiations of the grid
// pass-1 / count kernels and their launchers (ksg_grid.cuh has the search).
#include <cuda_runtime.h>

#include <algorithm>

#include "errors.h"
#include "ksg_grid.cuh"
#include "ksg_grid.h"

namespace nsg {
namespace {

int device_sms() {
    int dev = 0, sms = 0;
    NSG_CUDA(cudaGetDevice(&dev));
    NSG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return sms;
}

constexpr int kPrepThreads = 1024;
constexpr int kSample = 2048;       // frames sampled per coordinate for the quantiles

// In-place ascending bitonic sort of n = kSample floats in shared memory.
__device__ void bitonic_sort(float* v) {
    for (int size = 2; size <= kSample; size <<= 1) {
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            __syncthreads();
            for (int t = threadIdx.x; t < kSample / 2; t += blockDim.x) {
                const int lo = 2 * t - (t & (stride - 1));
                const int hi = lo + stride;
                const bool asc = (lo & size) == 0;
                const float a = v[lo], b = v[hi];
                if ((a > b) == asc) {
                    v[lo] = b;
                    v[hi] = a;
                }
            }
        }
    }
    __syncthreads();
}

// Number of edges <= x among e[0..n) (sorted ascending): the bin of x.
__device__ __forceinline__ int bin_of(const float* e, int n, float x) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (e[mid] <= x) lo = mid + 1;
        else hi = mid;
    }
    return lo;
}

// Exclusive scan of cnt[0..n) (n <= 1024) into out[0..n], out[n] = total.
__device__ void block_scan(const int* cnt, int* out, int n) {
    __shared__ int s_warp[32];
    const int t = threadIdx.x;
    const int v = t < n ? cnt[t] : 0;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if ((t & 31) >= o) x += y;
    }
    if ((t & 31) == 31) s_warp[t >> 5] = x;
    __syncthreads();
    if (t < 32) {
        int w = t < (blockDim.x >> 5) ? s_warp[t] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (t >= o) w += y;
        }
        s_warp[t] = w;
    }
    __syncthreads();
    const int incl = x + ((t >> 5) ? s_warp[(t >> 5) - 1] : 0);
    if (t < n) out[t] = incl - v;
    if (t == n - 1) out[n] = incl;
    __syncthreads();
}

// Query order of a grid's cells (the layout is described in ksg_grid.h):
// cnt[c] holds the frames of row-major cell c. The Z-order codes of a
// Gp x Gp square (Gp = G rounded up to a power of two, at most 32) are
// ranked, skipping cells outside G x G, and the counts accumulated in that
// order. tmp1, tmp2: shared scratch of 1024 and 1025 ints.
__device__ void build_query_order(const int* cnt, int G, int* start, int* tmp1, int* tmp2) {
    int* qstart = start + grid_qoff(G);
    unsigned short* qcell = reinterpret_cast<unsigned short*>(qstart + grid_qoff(G));
    int Gp = 1;
    while (Gp < G) Gp <<= 1;
    const int ncode = Gp * Gp;
    const int t = threadIdx.x;
    int row = 0, col = 0;
#pragma unroll
    for (int b = 0; b < 5; ++b) {
        row |= ((t >> (2 * b + 1)) & 1) << b;
        col |= ((t >> (2 * b)) & 1) << b;
    }
    const bool valid = t < ncode && row < G && col < G;
    if (t < ncode) tmp1[t] = valid ? 1 : 0;
    __syncthreads();
    block_scan(tmp1, tmp2, ncode);
    const int rank = t < ncode ? tmp2[t] : 0;
    __syncthreads();
    if (valid) {
        qcell[rank] = static_cast<unsigned short>(row * G + col);
        tmp1[rank] = cnt[row * G + col];
    }
    __syncthreads();
    block_scan(tmp1, tmp2, G * G);
    for (int c = t; c <= G * G; c += blockDim.x) qstart[c] = tmp2[c];
}

// Quantiles of coordinate c of a node (kQuantFloats) from a sorted sample;
// v: kSample floats of shared memory.
__device__ void node_quantiles(const GridNode& nd, int c, float* v, float* out) {
    for (int s = threadIdx.x; s < kSample; s += blockDim.x) {
        const int j = static_cast<int>((static_cast<long long>(s) * nd.m) / kSample);
        v[s] = __ldg(nd.x + static_cast<long long>(c) * nd.ld + j);
    }
    bitonic_sort(v);
    const int t = threadIdx.x;
    if (t < kGridMaxG) out[t] = t < nd.G - 1 ? v[((t + 1) * kSample) / nd.G] : __int_as_float(0x7f800000);
    if (t < 64) out[kGridMaxG + t] = v[min((t * kSample) / kBitBins, kSample - 1)];
    if (t == 0) out[kGridMaxG + 64] = v[(kSample * 9) / 10] - v[kSample / 10];
    __syncthreads();
}

// Coordinates by their spread: the widest, the second widest (-1 if none),
// and the other one.
template <int D>
__device__ __forceinline__ void node_axes(const float* quant, int (&axis)[3]) {
    float w[D];
#pragma unroll
    for (int c = 0; c < D; ++c) w[c] = quant[c * kQuantFloats + kGridMaxG + 64];
    int c1 = 0;
    for (int c = 1; c < D; ++c)
        if (w[c] > w[c1]) c1 = c;
    int c2 = -1;
    for (int c = 0; c < D; ++c)
        if (c != c1 && (c2 < 0 || w[c] > w[c2])) c2 = c;
    axis[0] = c1;
    axis[1] = c2;
    axis[2] = D == 3 ? 3 - c1 - c2 : 0;
}

// Cell and bitmap bins of frames [lo, hi) of a node, and their coordinates in
// the bitmap search's layout.
template <int D>
__device__ void node_bins(GridNode* node, const GridNode& nd, const float* quant, int lo, int hi) {
    __shared__ float s_e1[kGridMaxG], s_e2[kGridMaxG];
    __shared__ float s_be[D][64];
    const int G = nd.G, t = threadIdx.x;
    int axis[3];
    node_axes<D>(quant, axis);
    const int c1 = axis[0], c2 = axis[1];
    if (t < kGridMaxG) {
        s_e1[t] = quant[c1 * kQuantFloats + t];
        s_e2[t] = c2 >= 0 ? quant[c2 * kQuantFloats + t] : __int_as_float(0x7f800000);
        if (lo == 0) {
            nd.e1[t] = s_e1[t];
            nd.e2[t] = s_e2[t];
        }
    }
    if (t == 0 && lo == 0) {
        node->c1 = c1;
        node->c2 = c2;
    }
    for (int e = t; e < 64 * D; e += blockDim.x) {
        const int c = e >> 6;
        const int ax = c == 0 ? axis[0] : c == 1 ? axis[1] : axis[2];
        s_be[c][e & 63] = quant[ax * kQuantFloats + kGridMaxG + (e & 63)];
        if (lo == 0) nd.bedges[e] = s_be[c][e & 63];
    }
    __syncthreads();
    bool bad = false;
    for (int j = lo + t; j < hi; j += blockDim.x) {
        float x[D];
        unsigned bins = 0;
#pragma unroll
        for (int c = 0; c < D; ++c) {
            const int ax = c == 0 ? axis[0] : c == 1 ? axis[1] : axis[2];
            x[c] = __ldg(nd.x + static_cast<long long>(ax) * nd.ld + j);
            bad |= !isfinite(x[c]);
            bins |= static_cast<unsigned>(bin_of(s_be[c] + 1, kBitBins - 1, x[c])) << (8 * c);
        }
        int cell = bin_of(s_e1, G - 1, x[0]) * G;
        if constexpr (D > 1) cell += bin_of(s_e2, G - 1, x[1]);
        nd.cell[j] = static_cast<unsigned short>(cell);
        if constexpr (D == 1) nd.aos[j] = x[0];
        else if constexpr (D == 2) reinterpret_cast<float2*>(nd.aos)[j] = make_float2(x[0], x[1]);
        else reinterpret_cast<float4*>(nd.aos)[j] = make_float4(x[0], x[1], x[2], 0.f);
        nd.bins[j] = bins;
    }
    if (bad) nd.ostart[63] = 1;
}

// Counting sort of a node's frames by cell.
template <int D>
__device__ void node_cells(const GridNode& nd) {
    __shared__ int s_cnt[kGridMaxG * kGridMaxG];
    __shared__ int s_start[kGridMaxG * kGridMaxG + 1];
    __shared__ int s_tmp1[kGridMaxG * kGridMaxG], s_tmp2[kGridMaxG * kGridMaxG + 1];
    const int m = nd.m, G = nd.G, t = threadIdx.x;
    for (int c = t; c < G * G; c += blockDim.x) s_cnt[c] = 0;
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) atomicAdd(&s_cnt[nd.cell[j]], 1);
    __syncthreads();
    block_scan(s_cnt, s_start, G * G);
    for (int c = t; c <= G * G; c += blockDim.x) nd.start[c] = s_start[c];
    for (int c = t; c < G * G; c += blockDim.x) s_cnt[c] = 0;
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) {
        const int cell = nd.cell[j];
        const int pos = s_start[cell] + atomicAdd(&s_cnt[cell], 1);
        nd.perm[pos] = j;
#pragma unroll
        for (int c = 0; c < D; ++c) {
            nd.sx[static_cast<long long>(c) * m + pos] = __ldg(nd.x + static_cast<long long>(c) * nd.ld + j);
        }
    }
    __syncthreads();
    build_query_order(s_cnt, G, nd.start, s_tmp1, s_tmp2);
}

// Counting sort of a node's frames by their bitmap bin of c1.
__device__ void node_order(const GridNode& nd) {
    __shared__ int s_ocnt[64], s_ostart[65];
    const int m = nd.m, t = threadIdx.x;
    if (m > kBitMaxM) return;
    if (t < 64) s_ocnt[t] = 0;
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) atomicAdd(&s_ocnt[nd.bins[j] & 0xffu], 1);
    __syncthreads();
    block_scan(s_ocnt, s_ostart, 64);
    if (t < 64) {
        if (t < 63) nd.ostart[t] = s_ostart[t];
        s_ocnt[t] = 0;
    }
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) {
        const int b = nd.bins[j] & 0xffu;
        nd.order[s_ostart[b] + atomicAdd(&s_ocnt[b], 1)] = static_cast<unsigned short>(j);
    }
}

// Everything for one node by a cluster of kNodeCtas CTAs: a coordinate's
// quantiles each, a share of the bins each, then one counting sort each in
// two of them. One CTA doing it in sequence took 87 us for a pair's two nodes
// at m = 10000.
constexpr int kNodeCtas = 4;

__device__ __forceinline__ void cluster_wait() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int D>
__global__ void __cluster_dims__(kNodeCtas, 1, 1) __launch_bounds__(kPrepThreads) grid_node_kernel(GridNode* nodes) {
    __shared__ float s_val[kSample];
    GridNode* node = nodes + blockIdx.x / kNodeCtas;
    const int part = blockIdx.x % kNodeCtas;
    const GridNode nd = *node;
    if (threadIdx.x == 0 && part == 0) nd.ostart[63] = 0;
    if (part < D) node_quantiles(nd, part, s_val, nd.quant + part * kQuantFloats);
    cluster_wait();
    const int share = (nd.m + kNodeCtas - 1) / kNodeCtas;
    const int lo = min(nd.m, part * share);
    node_bins<D>(node, nd, nd.quant, lo, min(nd.m, lo + share));
    cluster_wait();
    if (part == 0) node_cells<D>(nd);
    else if (part == 1) node_order(nd);
}

// The same in four kernels for plans of many nodes: the sample sort waits on
// barriers, the counting sorts on atomics, and the bins on binary searches;
// small CTAs of one kind overlap better than 1024 threads doing one after the
// other.
constexpr int kSplitThreads = 512;

__global__ void __launch_bounds__(kSplitThreads) node_quantiles_kernel(const GridNode* nodes) {
    __shared__ float s_val[kSample];
    const GridNode nd = nodes[blockIdx.x];
    if (threadIdx.x == 0 && blockIdx.y == 0) nd.ostart[63] = 0;
    node_quantiles(nd, blockIdx.y, s_val, nd.quant + blockIdx.y * kQuantFloats);
}

template <int D>
__global__ void __launch_bounds__(kSplitThreads) node_bins_kernel(GridNode* nodes) {
    const GridNode nd = nodes[blockIdx.x];
    const int share = (nd.m + gridDim.y - 1) / gridDim.y;
    const int lo = blockIdx.y * share;
    if (lo < nd.m) node_bins<D>(nodes + blockIdx.x, nd, nd.quant, lo, min(nd.m, lo + share));
}

template <int D>
__global__ void __launch_bounds__(kPrepThreads) node_cells_kernel(const GridNode* nodes) {
    node_cells<D>(nodes[blockIdx.x]);
}

__global__ void __launch_bounds__(kSplitThreads) node_order_kernel(const GridNode* nodes) {
    node_order(nodes[blockIdx.x]);
}

// One CTA per pair of the batch: cells over (bin of a on its c1, bin of b on
// its c1), counting sort, both nodes' coordinates copied in that order.
template <int D>
__global__ void __launch_bounds__(kPrepThreads) grid_pair_kernel(const KsgPairDesc* pairs,
                                                                GridPair* gps,
                                                                const GridNode* nodes) {
    __shared__ int s_cnt[kGridMaxG * kGridMaxG];
    __shared__ int s_start[kGridMaxG * kGridMaxG + 1];
    __shared__ int s_tmp1[kGridMaxG * kGridMaxG], s_tmp2[kGridMaxG * kGridMaxG + 1];
    const KsgPairDesc P = pairs[blockIdx.x];
    const GridPair gp = gps[blockIdx.x];
    const GridNode na = nodes[gp.a], nb = nodes[gp.b];
    const int m = P.m, G = na.G, t = threadIdx.x;
    for (int c = t; c < G * G; c += blockDim.x) s_cnt[c] = 0;
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) {
        const int cell = (na.cell[j] / G) * G + nb.cell[j] / G;
        atomicAdd(&s_cnt[cell], 1);
    }
    __syncthreads();
    block_scan(s_cnt, s_start, G * G);
    for (int c = t; c <= G * G; c += blockDim.x) gp.start[c] = s_start[c];
    for (int c = t; c < G * G; c += blockDim.x) s_cnt[c] = 0;
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) {
        const int cell = (na.cell[j] / G) * G + nb.cell[j] / G;
        const int pos = s_start[cell] + atomicAdd(&s_cnt[cell], 1);
        gp.perm[pos] = j;
#pragma unroll
        for (int c = 0; c < D; ++c) {
            gp.sx[static_cast<long long>(c) * m + pos] = __ldg(P.xa + static_cast<long long>(c) * P.ld + j);
            gp.sx[static_cast<long long>(D + c) * m + pos] =
                __ldg(P.xb + static_cast<long long>(c) * P.ld + j);
        }
    }
    __syncthreads();
    build_query_order(s_cnt, G, gp.start, s_tmp1, s_tmp2);
}

// The same pair grid, written plane by plane through shared memory: each
// frame's position is computed once, then every output plane (the original
// indices and the 2d coordinates) is scattered into a shared-memory buffer
// and written out with coalesced stores, instead of scattering 2d + 1 values
// per frame across global memory. Dynamic shared memory: 8 * mpad bytes
// (positions, then the plane buffer) with mpad >= m.
template <int D>
__global__ void __launch_bounds__(kPrepThreads) grid_pair_staged_kernel(const KsgPairDesc* pairs,
                                                                       GridPair* gps,
                                                                       const GridNode* nodes, int mpad) {
    extern __shared__ int s_dyn[];
    __shared__ int s_cnt[kGridMaxG * kGridMaxG];
    __shared__ int s_start[kGridMaxG * kGridMaxG + 1];
    __shared__ int s_tmp1[kGridMaxG * kGridMaxG], s_tmp2[kGridMaxG * kGridMaxG + 1];
    int* s_pos = s_dyn;
    int* s_buf = s_dyn + mpad;
    const KsgPairDesc P = pairs[blockIdx.x];
    const GridPair gp = gps[blockIdx.x];
    const GridNode na = nodes[gp.a], nb = nodes[gp.b];
    const int m = P.m, G = na.G, t = threadIdx.x;
    for (int c = t; c < G * G; c += blockDim.x) s_cnt[c] = 0;
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) {
        const int cell = (na.cell[j] / G) * G + nb.cell[j] / G;
        s_pos[j] = cell;
        atomicAdd(&s_cnt[cell], 1);
    }
    __syncthreads();
    block_scan(s_cnt, s_start, G * G);
    for (int c = t; c <= G * G; c += blockDim.x) gp.start[c] = s_start[c];
    for (int c = t; c < G * G; c += blockDim.x) s_cnt[c] = 0;
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) {
        const int cell = s_pos[j];
        s_pos[j] = s_start[cell] + atomicAdd(&s_cnt[cell], 1);
    }
    __syncthreads();
    for (int j = t; j < m; j += blockDim.x) s_buf[s_pos[j]] = j;
    __syncthreads();
    for (int q = t; q < m; q += blockDim.x) gp.perm[q] = s_buf[q];
    float* fbuf = reinterpret_cast<float*>(s_buf);
#pragma unroll 1
    for (int c = 0; c < 2 * D; ++c) {
        const float* src = c < D ? P.xa + static_cast<long long>(c) * P.ld : P.xb + static_cast<long long>(c - D) * P.ld;
        __syncthreads();
        for (int j = t; j < m; j += blockDim.x) fbuf[s_pos[j]] = __ldg(src + j);
        __syncthreads();
        float* dst = gp.sx + static_cast<long long>(c) * m;
        for (int q = t; q < m; q += blockDim.x) dst[q] = fbuf[q];
    }
    __syncthreads();
    build_query_order(s_cnt, G, gp.start, s_tmp1, s_tmp2);
}

// psi[n_x] + psi[n_y] per sample from the raw counts (self included), as
// write_outputs does in the exhaustive kernel.
__global__ void grid_combine_kernel(const KsgPairDesc* pairs, const int* cnt_a, const int* cnt_b,
                                    const float* psi, float* psum, int* nx_out, int* ny_out) {
    const KsgPairDesc P = pairs[blockIdx.x];
    for (int i = blockIdx.y * blockDim.x + threadIdx.x; i < P.m; i += gridDim.y * blockDim.x) {
        const long long o = P.scratch + i;
        const int nx = min(max(cnt_a[o] - 1, 0), P.m);
        const int ny = min(max(cnt_b[o] - 1, 0), P.m);
        psum[o] = __fadd_rn(__ldg(psi + nx), __ldg(psi + ny));
        if (nx_out) nx_out[o] = nx;
        if (ny_out) ny_out[o] = ny;
    }
}

// Query orders (see kOrderBits and kOrderBlock). A warp's queries then have
// boxes of nearly the same cells, so the union of their boxes is smaller
// than in a grid's Z order of cells. Any order gives the same results;
// these only shorten the scans.
constexpr int kOrderThreads = 256;
constexpr int kOrderKeyBits = 4 * kOrderBits;          // Z code of the four box corners
constexpr int kOrderBins = 1 << (kOrderKeyBits - 4);   // counting-sort bins: the top bits
constexpr int kOrderSortMax = 32;
// Counts orders sort their bins on the low key bits up to this m (keys and
// bins: 8 bytes per query of shared memory).
constexpr int kOrderSortLowMaxM = 20480;
static_assert(2 * kOrderSortLowMaxM <= kOrderMaxM, "the attribute covers both arrays");
static_assert(kOrderBins % kOrderThreads == 0, "bins split evenly over the CTA");

// Coarse cell (cell >> 1: kOrderBits bits) of x on an axis whose edges give
// the thresholds t[L - 1] = e[2L - 1], L = 1..15, padded with +inf where the
// grid has fewer cells and ended by a NaN (never <= x): the number of
// thresholds <= x, by four branch-free steps over the 16 sorted entries.
static_assert(kOrderBits == 4 && kGridMaxG <= 32, "coarse cells are cell pairs of a grid of <= 32 cells");
__device__ __forceinline__ unsigned coarse_cell(const float* t, float x) {
    unsigned b = t[7] <= x ? 8u : 0u;
    b += t[b + 3] <= x ? 4u : 0u;
    b += t[b + 1] <= x ? 2u : 0u;
    b += t[b] <= x ? 1u : 0u;
    return b;
}

// Bits of v < 16 spread to positions 0, 4, 8, 12.
__device__ __forceinline__ unsigned spread4(unsigned v) {
    return (v & 1u) | (v & 2u) << 3 | (v & 4u) << 6 | (v & 8u) << 9;
}

// Z code of the box [x - h, x + h] x [y - h, y + h] in coarse cells: bit b
// of corner q (low row, low column, high row, high column) at bit 4b + q.
__device__ __forceinline__ unsigned box_key(const float* t1, const float* t2, float x, float y, float h) {
    return spread4(coarse_cell(t1, x - h)) | spread4(coarse_cell(t2, y - h)) << 1 |
           spread4(coarse_cell(t1, x + h)) << 2 | spread4(coarse_cell(t2, y + h)) << 3;
}

// Writes out[rank] = pos for every position pos < m of a grid, ranks in
// ascending order of the 16-bit keys s_key[pos]: a counting sort on the top
// twelve bits (shared-memory atomics). With s_tmp (m more words of shared
// memory; m <= 65536) each bin of at most kOrderSortMax positions, most
// bins, is then sorted on the low four bits by one thread in shared memory;
// larger bins, where many queries share one box, keep the atomics' order,
// so the work stays O(m). Without s_tmp the low bits are ignored. Called by
// the whole CTA after it has written s_key.
__device__ void write_key_order(const unsigned* s_key, int m, int* out, unsigned* s_tmp) {
    __shared__ int s_bin[kOrderBins];
    __shared__ int s_part[kOrderThreads];
    for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x) s_bin[b] = 0;
    __syncthreads();
    for (int pos = threadIdx.x; pos < m; pos += blockDim.x) atomicAdd(&s_bin[s_key[pos] >> 4], 1);
    __syncthreads();
    // exclusive prefix over the bins: kPer bins per thread
    constexpr int kPer = kOrderBins / kOrderThreads;
    int acc = 0;
    for (int q = 0; q < kPer; ++q) acc += s_bin[threadIdx.x * kPer + q];
    s_part[threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int t = 0; t < kOrderThreads; ++t) {
            const int v = s_part[t];
            s_part[t] = run;
            run += v;
        }
    }
    __syncthreads();
    int run = s_part[threadIdx.x];
    for (int q = 0; q < kPer; ++q) {
        const int b = threadIdx.x * kPer + q;
        const int v = s_bin[b];
        s_bin[b] = run;
        run += v;
    }
    __syncthreads();
    if (!s_tmp) {
        for (int pos = threadIdx.x; pos < m; pos += blockDim.x) out[atomicAdd(&s_bin[s_key[pos] >> 4], 1)] = pos;
        return;
    }
    // entries (low key bits << 16 | pos): their order is the order wanted
    for (int pos = threadIdx.x; pos < m; pos += blockDim.x) {
        const unsigned key = s_key[pos];
        s_tmp[atomicAdd(&s_bin[key >> 4], 1)] = (key & 15u) << 16 | static_cast<unsigned>(pos);
    }
    __syncthreads();
    // s_bin[b] is now the end of bin b
    for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x) {
        const int lo = b == 0 ? 0 : s_bin[b - 1], hi = s_bin[b];
        if (hi - lo > kOrderSortMax) continue;
        for (int r = lo + 1; r < hi; ++r) {
            const unsigned v = s_tmp[r];
            int t = r;
            while (t > lo && s_tmp[t - 1] > v) {
                s_tmp[t] = s_tmp[t - 1];
                --t;
            }
            s_tmp[t] = v;
        }
    }
    __syncthreads();
    for (int r = threadIdx.x; r < m; r += blockDim.x) out[r] = static_cast<int>(s_tmp[r] & 0xffffu);
}

// Count order of one count group per CTA: boxes of the largest eps of the
// group's pairs on the node grid. Dynamic shared memory: corder_ld keys,
// then, with `sort_low`, corder_ld words for write_key_order's bins.
__global__ void __launch_bounds__(kOrderThreads) grid_count_order_kernel(GridArgs A, int sort_low) {
    extern __shared__ unsigned s_key[];
    __shared__ float s_t[2][16];
    const CountGroup grp = A.groups[blockIdx.x];
    const GridNode nd = A.nodes[grp.node];
    const int m = nd.m;
    if (threadIdx.x < 32) {
        const int L = threadIdx.x & 15;
        const float* e = threadIdx.x < 16 ? nd.e1 : nd.e2;
        s_t[threadIdx.x >> 4][L] = L < 15 ? e[2 * L + 1] : __int_as_float(0x7fc00000);
    }
    __syncthreads();
    const float* eps[kCountGroup];
#pragma unroll
    for (int p = 0; p < kCountGroup; ++p) {  // unused slots repeat the first variable
        const int v = grp.vars[p];
        eps[p] = (v & 1 ? A.eps_b : A.eps_a) + A.pairs[v >> 1].scratch;
    }
    // the grid's coordinates in storage order (coalesced)
    const float* x1 = nd.sx + static_cast<long long>(nd.c1) * m;
    const float* x2 = nd.c2 >= 0 ? nd.sx + static_cast<long long>(nd.c2) * m : nullptr;
    for (int pos = threadIdx.x; pos < m; pos += blockDim.x) {
        const int j = __ldg(nd.perm + pos);
        float e = __ldg(eps[0] + j);
#pragma unroll
        for (int p = 1; p < kCountGroup; ++p)
            if (p < grp.nvars) e = fmaxf(e, __ldg(eps[p] + j));
        s_key[pos] = box_key(s_t[0], s_t[1], __ldg(x1 + pos), x2 ? __ldg(x2 + pos) : 0.f, e);
    }
    __syncthreads();
    write_key_order(s_key, m, A.corder + static_cast<long long>(blockIdx.x) * A.corder_ld,
                    sort_low ? s_key + A.corder_ld : nullptr);
}

// Search order: cells in kOrderBlock x kOrderBlock blocks, blocks in Z
// order, and within a block the queries by size class. Box Z codes of the
// estimates, which serve the counts, made the search slower (197 against
// 175 ms per 8192-pair batch at m = 10000): a warp's queries then spread
// over more cells than its seed rectangle allows, and its lists fill later.
constexpr int kOrderBlocks = (kGridMaxG + kOrderBlock - 1) / kOrderBlock;  // per axis
constexpr int kOrderClasses = 64;
static_assert(kOrderBlocks * kOrderBlocks * kOrderClasses == kOrderBins, "one counting-sort bin per class");

__device__ __forceinline__ unsigned block_zcode(int bx, int by) {
    unsigned z = 0;
#pragma unroll
    for (int b = 0; b < 3; ++b) z |= ((bx >> b) & 1u) << (2 * b + 1) | ((by >> b) & 1u) << (2 * b);
    return z;
}

// Size class of a box size e >= 0: its quarter octave (the float's exponent
// and top two mantissa bits; +inf and NaN land in the top class).
__device__ __forceinline__ unsigned size_bits(float e) {
    return isnan(e) ? 0xffffffffu : __float_as_uint(fmaxf(e, 0.f)) >> 21;
}

// Search order of one pair per CTA: the size class of the geometric mean of
// the two nodes' scale estimates, which follows the k-th joint distance
// closely enough to group queries with similar boxes (rank correlation 0.89
// with it, against 0.86 for the larger estimate, in a CPU model of the
// protein trajectories); the smallest class present becomes class 0. Dynamic
// shared memory: m keys.
__global__ void __launch_bounds__(kOrderThreads) grid_pair_order_kernel(const KsgPairDesc* pairs,
                                                                       const GridPair* gps,
                                                                       const GridNode* nodes) {
    extern __shared__ unsigned s_key[];
    __shared__ unsigned s_lo;
    const GridPair gp = gps[blockIdx.x];
    const GridNode na = nodes[gp.a], nb = nodes[gp.b];
    const int m = pairs[blockIdx.x].m, G = na.G;
    if (threadIdx.x == 0) s_lo = 0xffffffffu;
    __syncthreads();
    unsigned lo = 0xffffffffu;
    for (int pos = threadIdx.x; pos < m; pos += blockDim.x) {
        const int j = __ldg(gp.perm + pos);
        s_key[pos] = size_bits(sqrtf(__ldg(na.est + j) * __ldg(nb.est + j)));
        lo = min(lo, s_key[pos]);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    if ((threadIdx.x & 31) == 0) atomicMin(&s_lo, lo);
    __syncthreads();
    lo = s_lo;
    for (int pos = threadIdx.x; pos < m; pos += blockDim.x) {
        const int j = __ldg(gp.perm + pos);
        const int row = __ldg(na.cell + j) / G, col = __ldg(nb.cell + j) / G;
        const unsigned d = s_key[pos] - lo;
        const unsigned cls = d < static_cast<unsigned>(kOrderClasses) ? d : kOrderClasses - 1;
        s_key[pos] = (block_zcode(row / kOrderBlock, col / kOrderBlock) * kOrderClasses + cls) << 4;
    }
    __syncthreads();
    write_key_order(s_key, m, gp.qpos, nullptr);
}

// One CTA per row.
__global__ void grid_gather_kernel(const GatherRow* rows, int d, int* fault) {
    const GatherRow g = rows[blockIdx.x];
    const float inf = __int_as_float(0x7f800000);
    for (int s = threadIdx.x; s < g.ld_out; s += blockDim.x) {
        int f = 0;
        if (s < g.m) {
            f = __ldg(g.fmap + s);
            if (f < 0 || f >= g.ld) {
                atomicOr(fault, FAULT_BAD_INDEX);
                f = 0;
            }
        }
        for (int c = 0; c < d; ++c) {
            g.out[static_cast<long long>(c) * g.ld_out + s] =
                s < g.m ? __ldg(g.x + static_cast<long long>(c) * g.ld + f) : inf;
        }
    }
}

template <int D>
void launch_pass1(const GridArgs& a, int kmax, int grid, cudaStream_t st) {
    const dim3 b(32 * kGridWarps);
    switch (kmax) {
        case 6: ksg_grid_pass1_kernel<D, 6, false><<<grid, b, 0, st>>>(a); break;
        case 8: ksg_grid_pass1_kernel<D, 8, false><<<grid, b, 0, st>>>(a); break;
        case 16: ksg_grid_pass1_kernel<D, 16, false><<<grid, b, 0, st>>>(a); break;
        case 32: ksg_grid_pass1_kernel<D, 32, false><<<grid, b, 0, st>>>(a); break;
        case 64: ksg_grid_pass1_kernel<D, 64, false><<<grid, b, 0, st>>>(a); break;
        default: fail(NSG_ERR_UNSUPPORTED, "no grid kernel for this k");
    }
}

}  // namespace

CountWork count_work(const GridPair* gps, const KsgPairDesc* descs, int npairs, bool ordered) {
    CountWork w;
    // variables by node, in first-appearance order within a node
    std::vector<std::pair<int, int>> keyed(2 * static_cast<size_t>(npairs));
    for (int p = 0; p < npairs; ++p) {
        keyed[p] = {gps[p].a, 2 * p};
        keyed[static_cast<size_t>(npairs) + p] = {gps[p].b, 2 * p + 1};
    }
    std::stable_sort(keyed.begin(), keyed.end(),
                     [](const std::pair<int, int>& x, const std::pair<int, int>& y) { return x.first < y.first; });
    long long rows = 0;  // queries: samples of the distinct nodes
    for (size_t s = 0; s < keyed.size(); ++s) {
        if (s == 0 || keyed[s].first != keyed[s - 1].first) rows += descs[keyed[s].second >> 1].m;
    }
    const bool few = !ordered && rows <= kRankFewRows;
    int gitems = 0, ritems = 0;
    for (size_t s = 0; s < keyed.size();) {
        size_t e = s;
        while (e < keyed.size() && keyed[e].first == keyed[s].first) ++e;
        const int node = keyed[s].first, m = descs[keyed[s].second >> 1].m;
        const int vars = static_cast<int>(e - s);
        if (ordered ? vars >= kRankMinVars : few && vars <= kRankDirect) {
            w.ranks.push_back({node, static_cast<int>(w.refs.size()), static_cast<int>(e - s), m});
            w.rprefix.push_back(ritems);
            ritems += (m + kRankBlock - 1) / kRankBlock;
            for (; s < e; ++s) {
                const int v = keyed[s].second;
                w.refs.push_back(descs[v >> 1].scratch * 2 + (v & 1));
            }
        }
        while (s < e) {
            // the rest in groups of equal size (8 variables: 4 + 4)
            const int left = static_cast<int>(e - s);
            const int take = (left + (left + kCountGroup - 1) / kCountGroup - 1) / ((left + kCountGroup - 1) / kCountGroup);
            CountGroup g{};
            g.node = node;
            g.nvars = take;
            for (int q = 0; q < kCountGroup; ++q) g.vars[q] = keyed[s + (q < take ? q : 0)].second;
            s += take;
            w.groups.push_back(g);
            w.gprefix.push_back(gitems);
            gitems += (m + kCountQueries - 1) / kCountQueries;
        }
    }
    w.gprefix.push_back(gitems);
    w.rprefix.push_back(ritems);
    return w;
}

int grid_cells_per_axis(int m) {
    int g = 1;
    while ((g + 1) * (g + 1) * 10 <= m && g < kGridMaxG) ++g;
    return g;
}

namespace {

template <int D>
void launch_nodes(GridNode* nodes, int nnodes, bool split, cudaStream_t st) {
    if (split) {
        node_quantiles_kernel<<<dim3(nnodes, D), kSplitThreads, 0, st>>>(nodes);
        node_bins_kernel<D><<<dim3(nnodes, 4), kSplitThreads, 0, st>>>(nodes);
        node_cells_kernel<D><<<nnodes, kPrepThreads, 0, st>>>(nodes);
        node_order_kernel<<<nnodes, kSplitThreads, 0, st>>>(nodes);
    } else {
        grid_node_kernel<D><<<nnodes * kNodeCtas, kPrepThreads, 0, st>>>(nodes);
    }
    NSG_CUDA(cudaGetLastError());
}

}  // namespace

void grid_launch_nodes(GridNode* nodes, int nnodes, int d, bool split, cudaStream_t st) {
    if (nnodes <= 0) return;
    switch (d) {
        case 1: launch_nodes<1>(nodes, nnodes, split, st); break;
        case 2: launch_nodes<2>(nodes, nnodes, split, st); break;
        case 3: launch_nodes<3>(nodes, nnodes, split, st); break;
        default: invalid("d must be 1, 2 or 3");
    }
}

bool grid_split_pays(int nnodes, int sms) { return nnodes * kNodeCtas >= sms; }

bool grid_orders_pay(long long search_warps, int sms) {
    return search_warps >= static_cast<long long>(kOrderMinWaves) * 32 * sms;
}

size_t grid_node_bytes(int m, int d) {
    auto a16 = [](size_t b) { return (b + 15) & ~size_t(15); };
    const size_t mm = static_cast<size_t>(m);
    return a16(2 * kGridMaxG * sizeof(float)) + grid_index_bytes(grid_cells_per_axis(m)) +
           a16(mm * sizeof(unsigned short)) + a16(mm * sizeof(int)) + a16(mm * sizeof(float)) +
           a16(static_cast<size_t>(d) * mm * sizeof(float)) + grid_node_bitmap_bytes(m, d);
}

size_t grid_node_bitmap_bytes(int m, int d) {
    auto a16 = [](size_t b) { return (b + 15) & ~size_t(15); };
    const size_t mm = static_cast<size_t>(m);
    // frames, bins, order, edges, starts
    return a16((d == 3 ? 4 : d) * mm * sizeof(float)) + a16(mm * sizeof(unsigned)) + a16(mm * sizeof(unsigned short)) +
           static_cast<size_t>(d) * (64 + kQuantFloats) * sizeof(float) + 64 * sizeof(int);
}

GridNode grid_node_at(unsigned char* base, const float* x, int ld, int m, int d) {
    auto a16 = [](size_t b) { return (b + 15) & ~size_t(15); };
    const size_t mm = static_cast<size_t>(m);
    GridNode n{};
    n.x = x;
    n.ld = ld;
    n.m = m;
    n.G = grid_cells_per_axis(m);
    n.e1 = reinterpret_cast<float*>(base);
    n.e2 = n.e1 + kGridMaxG;
    base += a16(2 * kGridMaxG * sizeof(float));
    n.start = reinterpret_cast<int*>(base);
    base += grid_index_bytes(n.G);
    n.cell = reinterpret_cast<unsigned short*>(base);
    base += a16(mm * sizeof(unsigned short));
    n.perm = reinterpret_cast<int*>(base);
    base += a16(mm * sizeof(int));
    n.est = reinterpret_cast<float*>(base);
    base += a16(mm * sizeof(float));
    n.sx = reinterpret_cast<float*>(base);
    base += a16(static_cast<size_t>(d) * mm * sizeof(float));
    n.aos = reinterpret_cast<float*>(base);
    base += a16((d == 3 ? 4 : d) * mm * sizeof(float));
    n.bins = reinterpret_cast<unsigned*>(base);
    base += a16(mm * sizeof(unsigned));
    n.order = reinterpret_cast<unsigned short*>(base);
    base += a16(mm * sizeof(unsigned short));
    n.bedges = reinterpret_cast<float*>(base);
    n.quant = n.bedges + 64 * d;
    n.ostart = reinterpret_cast<int*>(n.quant + kQuantFloats * d);
    return n;
}

size_t grid_pair_place(GridPair& g, size_t off, int m, int d) {
    auto a16 = [](size_t b) { return (b + 15) & ~size_t(15); };
    const size_t mm = static_cast<size_t>(m);
    g.start = reinterpret_cast<int*>(off);
    off += grid_index_bytes(grid_cells_per_axis(m));
    g.perm = reinterpret_cast<int*>(off);
    off += a16(mm * sizeof(int));
    g.qpos = reinterpret_cast<int*>(off);
    off += a16(mm * sizeof(int));
    g.sx = reinterpret_cast<float*>(off);
    off += a16(static_cast<size_t>(2 * d) * mm * sizeof(float));
    return off;
}

void grid_pair_rebase(GridPair& g, const void* base) {
    const uintptr_t b = reinterpret_cast<uintptr_t>(base);
    g.start = reinterpret_cast<int*>(b + reinterpret_cast<uintptr_t>(g.start));
    g.perm = reinterpret_cast<int*>(b + reinterpret_cast<uintptr_t>(g.perm));
    g.qpos = reinterpret_cast<int*>(b + reinterpret_cast<uintptr_t>(g.qpos));
    g.sx = reinterpret_cast<float*>(b + reinterpret_cast<uintptr_t>(g.sx));
}

namespace {

// Largest dynamic shared memory the staged pair-grid kernel asks for.
constexpr size_t kPairStagedSmem = size_t(160) << 10;

template <int D>
void launch_pairs(const KsgPairDesc* pairs, GridPair* gps, const GridNode* nodes, int npairs, int max_m,
                  cudaStream_t st) {
    const int mpad = (max_m + 3) & ~3;
    const size_t smem = sizeof(int) * 2 * static_cast<size_t>(mpad);
    if (smem <= kPairStagedSmem) {
        // set on every launch: the attribute belongs to the current device
        NSG_CUDA(cudaFuncSetAttribute(grid_pair_staged_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(kPairStagedSmem)));
        grid_pair_staged_kernel<D><<<npairs, kPrepThreads, smem, st>>>(pairs, gps, nodes, mpad);
    } else {
        grid_pair_kernel<D><<<npairs, kPrepThreads, 0, st>>>(pairs, gps, nodes);
    }
}

}  // namespace

int grid_launch_pairs(const KsgPairDesc* pairs, GridPair* gps, const GridNode* nodes, int npairs,
                      int max_m, int d, bool order, cudaStream_t st) {
    if (npairs <= 0) return 0;
    switch (d) {
        case 1: launch_pairs<1>(pairs, gps, nodes, npairs, max_m, st); break;
        case 2: launch_pairs<2>(pairs, gps, nodes, npairs, max_m, st); break;
        case 3: launch_pairs<3>(pairs, gps, nodes, npairs, max_m, st); break;
        default: invalid("d must be 1, 2 or 3");
    }
    NSG_CUDA(cudaGetLastError());
    if (!order || max_m > kOrderMaxM) return 0;
    // set on every launch: the attribute belongs to the current device
    NSG_CUDA(cudaFuncSetAttribute(grid_pair_order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(sizeof(unsigned) * kOrderMaxM)));
    grid_pair_order_kernel<<<npairs, kOrderThreads, sizeof(unsigned) * static_cast<size_t>(max_m), st>>>(
        pairs, gps, nodes);
    NSG_CUDA(cudaGetLastError());
    return 1;
}

void grid_launch_search(const GridArgs& a, int d, int kmax, int grid, bool tie_record, cudaStream_t st) {
    if (tie_record) {
        grid_launch_search_rec(a, d, kmax, grid, st);
        return;
    }
    switch (d) {
        case 1: launch_pass1<1>(a, kmax, grid, st); break;
        case 2: launch_pass1<2>(a, kmax, grid, st); break;
        case 3: launch_pass1<3>(a, kmax, grid, st); break;
        default: invalid("d must be 1, 2 or 3");
    }
    NSG_CUDA(cudaGetLastError());
}

GridArgs grid_launch_count_order(const GridArgs& a, cudaStream_t st) {
    GridArgs c = a;
    if (c.corder && c.corder_ld <= kOrderMaxM && c.ngroups > 0) {
        // keys, and up to kOrderSortLowMaxM the bins' second copy
        const int sort_low = c.corder_ld <= kOrderSortLowMaxM ? 1 : 0;
        const size_t smem = sizeof(unsigned) * static_cast<size_t>(c.corder_ld) * (1 + sort_low);
        // set on every launch: the attribute belongs to the current device
        NSG_CUDA(cudaFuncSetAttribute(grid_count_order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      static_cast<int>(sizeof(unsigned) * kOrderMaxM)));
        grid_count_order_kernel<<<c.ngroups, kOrderThreads, smem, st>>>(c, sort_low);
        NSG_CUDA(cudaGetLastError());
    } else {
        c.corder = nullptr;
    }
    return c;
}

namespace {

template <int D>
void launch_counts(const GridArgs& c, int grid, cudaStream_t st) {
    if (c.ngroups > 0) {
        ksg_grid_count_kernel<D><<<grid, 32 * kGridWarps, 0, st>>>(c);
        NSG_CUDA(cudaGetLastError());
    }
    if (c.nranks > 0) {
        const int ctas = std::min(device_sms() * (40 / kRankWarps), (c.rank_items + kRankWarps - 1) / kRankWarps);
        ksg_grid_rank_kernel<D><<<ctas, 32 * kRankWarps, 0, st>>>(c);
        NSG_CUDA(cudaGetLastError());
    }
}

}  // namespace

void grid_launch_count_kernel(const GridArgs& c, int d, int grid, cudaStream_t st) {
    switch (d) {
        case 1: launch_counts<1>(c, grid, st); break;
        case 2: launch_counts<2>(c, grid, st); break;
        case 3: launch_counts<3>(c, grid, st); break;
        default: invalid("d must be 1, 2 or 3");
    }
}

void grid_launch_counts(const GridArgs& a, int d, int grid, cudaStream_t st) {
    grid_launch_count_kernel(grid_launch_count_order(a, st), d, grid, st);
}

void grid_launch_combine(const KsgPairDesc* pairs, int npairs, int max_m, const int* cnt_a, const int* cnt_b,
                         const float* psi, float* psum, int* nx, int* ny, cudaStream_t st) {
    if (npairs <= 0) return;
    // few pairs: spread each over CTAs
    const int parts = std::max(1, std::min((max_m + 255) / 256, 2 * device_sms() / npairs));
    grid_combine_kernel<<<dim3(npairs, parts), 256, 0, st>>>(pairs, cnt_a, cnt_b, psi, psum, nx, ny);
    NSG_CUDA(cudaGetLastError());
}

void grid_launch_gather(const GatherRow* rows, int nrows, int d, int* fault, cudaStream_t st) {
    if (nrows <= 0) return;
    grid_gather_kernel<<<nrows, 256, 0, st>>>(rows, d, fault);
    NSG_CUDA(cudaGetLastError());
}

int grid_search_ctas_per_sm(int d, int kmax) {
    int n = 0;
    const int b = 32 * kGridWarps;
    cudaError_t e = cudaSuccess;
#define NSG_OCC(D_, K_) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ksg_grid_pass1_kernel<D_, K_, false>, b, 0)
    switch (d * 100 + kmax) {
        case 106: NSG_OCC(1, 6); break;
        case 108: NSG_OCC(1, 8); break;
        case 116: NSG_OCC(1, 16); break;
        case 132: NSG_OCC(1, 32); break;
        case 164: NSG_OCC(1, 64); break;
        case 206: NSG_OCC(2, 6); break;
        case 208: NSG_OCC(2, 8); break;
        case 216: NSG_OCC(2, 16); break;
        case 232: NSG_OCC(2, 32); break;
        case 264: NSG_OCC(2, 64); break;
        case 306: NSG_OCC(3, 6); break;
        case 308: NSG_OCC(3, 8); break;
        case 316: NSG_OCC(3, 16); break;
        case 332: NSG_OCC(3, 32); break;
        case 364: NSG_OCC(3, 64); break;
        default: return 1;
    }
#undef NSG_OCC
    cuda_check(e, "occupancy query");
    return n > 0 ? n : 1;
}

int grid_count_ctas_per_sm(int d) {
    int n = 0;
    const int b = 32 * kGridWarps;
    cudaError_t e = cudaSuccess;
    switch (d) {
        case 1: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ksg_grid_count_kernel<1>, b, 0); break;
        case 2: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ksg_grid_count_kernel<2>, b, 0); break;
        case 3: e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, ksg_grid_count_kernel<3>, b, 0); break;
        default: return 1;
    }
    cuda_check(e, "occupancy query");
    return n > 0 ? n : 1;
}

}  // namespace nsg
