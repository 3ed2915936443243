// Hedetniemi steps on sparse weight matrices.
//
// A step is Hn[i][j] = min_k fl(A[j][k] + H[k][i]) (apsp.cu). An entry
// A[j][k] = +inf adds +inf or a NaN, neither of which lowers a minimum that
// starts at +inf, so only the other entries of row j are visited: the result
// is the dense step's bit for bit, in whatever order they come. Contact
// graphs and geometric graphs hold about a dozen entries per row, where the
// dense product visits n.
#include <cuda_runtime.h>

#include <algorithm>

#include "apsp_sparse.h"
#include "common.cuh"

namespace nsg {
namespace {

constexpr int kInfBits = 0x7f800000;

// Flags, largest weight and entries per row, one 32 x 32 tile of A and its
// mirror tile per CTA (32 x 8 threads), so that both are read in rows.
__global__ void analyze_kernel(const float* __restrict__ A, int n, GraphInfo* info, int* counts) {
    if (blockIdx.x < blockIdx.y) return;
    __shared__ float t1[32][33], t2[32][33];
    const float inf = __int_as_float(kInfBits);
    const int r0 = blockIdx.y * 32, c0 = blockIdx.x * 32, lane = threadIdx.x;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
        t1[y][lane] = (r0 + y < n && c0 + lane < n) ? __ldg(A + (size_t)(r0 + y) * n + c0 + lane) : inf;
        t2[y][lane] = (c0 + y < n && r0 + lane < n) ? __ldg(A + (size_t)(c0 + y) * n + r0 + lane) : inf;
    }
    __syncthreads();
    int f = 0, w = 0;
    for (int y = threadIdx.y; y < 32; y += blockDim.y) {
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            if (side && r0 == c0) break;
            const float a = side ? t2[y][lane] : t1[y][lane];
            const int row = (side ? c0 : r0) + y, col = (side ? r0 : c0) + lane;
            const bool in = row < n && col < n;
            const unsigned keep = __ballot_sync(0xffffffffu, in && __float_as_int(a) != kInfBits);
            if (lane == 0 && keep) atomicAdd(counts + row, __popc(keep));
            if (!in) continue;
            if (__float_as_int(a) != __float_as_int(side ? t1[lane][y] : t2[lane][y])) f |= 1;
            if (row == col && a != 0.f) f |= 2;
            if (!(a >= 0.f)) f |= 4;
            if (a >= 0.f && a < inf) {
                if (a != rintf(a)) f |= 8;
                w = max(w, __float_as_int(a));
            }
        }
    }
    f = __reduce_or_sync(0xffffffffu, f);
    w = __reduce_max_sync(0xffffffffu, w);
    if (lane == 0) {
        if (f) atomicOr(&info->flags, f);
        atomicMax(&info->wmax, w);
    }
}

// Entries per row of a matrix of row stride ld, one warp per row.
__global__ void count_kernel(const float* __restrict__ A, int ld, int n, int* counts) {
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= n) return;
    int c = 0;
    for (int k = lane; k < n; k += 32) c += __float_as_int(__ldg(A + (size_t)row * ld + k)) != kInfBits;
    c = __reduce_add_sync(0xffffffffu, c);
    if (lane == 0) counts[row] = c;
}

// Slice widths (the longest row of each slice, in whole groups of
// kSellUnroll) and their exclusive prefix; one CTA of 1024 threads.
// order: the vertex of each row, or null for the matrix's own order.
__global__ void __launch_bounds__(1024) slice_kernel(const int* __restrict__ counts, const int* __restrict__ order,
                                                     int n, int nslices, int* ptr, GraphInfo* info) {
    __shared__ int s_warp[32];
    const int t = threadIdx.x, lane = t & 31;
    int base = 0, entries = 0;
    for (int s0 = 0; s0 < nslices; s0 += 1024) {
        const int s = s0 + t;
        int w = 0;
        for (int r = 0; r < kSellRows; ++r) {
            const int row = s * kSellRows + r;
            if (s < nslices && row < n) {
                const int c = counts[order ? order[row] : row];
                w = max(w, c);
                entries += c;
            }
        }
        w = (w + kSellUnroll - 1) / kSellUnroll * kSellUnroll;
        int x = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) s_warp[t >> 5] = x;
        __syncthreads();
        int before = base, all = base;
        for (int q = 0; q < 32; ++q) {
            if (q < (t >> 5)) before += s_warp[q];
            all += s_warp[q];
        }
        if (s < nslices) ptr[s] = before + x - w;
        base = all;
        __syncthreads();
    }
    if (!order) {  // the second pass over the same counts adds nothing new
        entries = __reduce_add_sync(0xffffffffu, entries);
        if (lane == 0) atomicAdd(&info->entries, entries);
    }
    if (t == 0) {
        ptr[nslices] = base;
        info->width = base;
    }
}

// One warp per row (of whole slices): its entries in ascending columns, then
// the padding up to the slice's width. With order and rank, row r is vertex
// order[r]'s and columns are ranks.
__global__ void fill_kernel(const float* __restrict__ A, int ld, int n, int nslices, const int* __restrict__ order,
                            const int* __restrict__ rank, const int* __restrict__ ptr, int2* __restrict__ edges) {
    const int row = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (row >= nslices * kSellRows) return;
    const int s = row / kSellRows, r = row % kSellRows;
    const int end = ptr[s + 1];
    int e = ptr[s];
    if (row < n) {
        const int vertex = order ? order[row] : row;
        for (int k0 = 0; k0 < n; k0 += 32) {
            const int k = k0 + lane;
            const float a = k < n ? __ldg(A + (size_t)vertex * ld + k) : __int_as_float(kInfBits);
            const bool keep = __float_as_int(a) != kInfBits;
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (keep) {
                const int at = e + __popc(mask & ((1u << lane) - 1u));
                edges[(size_t)at * kSellRows + r] = make_int2(rank ? rank[k] : k, __float_as_int(a));
            }
            e += __popc(mask);
        }
    }
    for (int p = e + lane; p < end; p += 32) edges[(size_t)p * kSellRows + r] = make_int2(0, kInfBits);
}

// Rank of every vertex by falling count, ties in index order: a thread per
// vertex compares it with all others (n^2 compares from shared memory).
__global__ void __launch_bounds__(256) sort_kernel(const int* __restrict__ counts, int n, int* order, int* rank) {
    __shared__ int s_c[1024];
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int mine = i < n ? counts[i] : 0;
    int r = 0;
    for (int base = 0; base < n; base += 1024) {
        __syncthreads();
        for (int q = threadIdx.x; q < 1024; q += blockDim.x) s_c[q] = base + q < n ? counts[base + q] : -1;
        __syncthreads();
        for (int q = 0; q < min(1024, n - base); ++q) r += s_c[q] > mine || (s_c[q] == mine && base + q < i);
    }
    if (i < n) {
        rank[i] = r;
        order[r] = i;
    }
}

// One row per CTA through shared memory: row to[r] of out takes the elements
// pick[c] of row from[r] (null: the row or element itself).
__global__ void __launch_bounds__(256) pick_kernel(const float* __restrict__ A, float* __restrict__ out, int n,
                                                   const int* __restrict__ from, const int* __restrict__ to,
                                                   const int* __restrict__ pick) {
    extern __shared__ float s_row[];
    const int r = blockIdx.x;
    const float* src = A + (size_t)(from ? from[r] : r) * n;
    float* dst = out + (size_t)(to ? to[r] : r) * n;
    for (int c = threadIdx.x; c < n; c += blockDim.x) s_row[c] = __ldg(src + c);
    __syncthreads();
    for (int c = threadIdx.x; c < n; c += blockDim.x) dst[c] = s_row[pick[c]];
}

__device__ __forceinline__ void cp_async(void* smem, const void* gmem, int bytes16) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    if (bytes16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gmem) : "memory");
}

// One step. A CTA owns the C columns i0 .. i0+C-1 of H, staged in shared
// memory once (all n rows: n * C floats), and a range of slices; every
// neighbour row read is then a shared-memory read. C/4 lanes take a row,
// four columns each, so 32/(C/4) rows are reduced per warp at a time and the
// entries of a slice arrive as one 64-byte load per entry index. Results go
// out transposed (Hn[i][j], j along the lanes). The compare against H stops
// reading H once a difference was seen in the CTA. The entries' latency and
// the conflicts of the row reads (64-byte rows, two to a shared-memory line)
// bound it: the next group of entries loads while one is reduced, across the
// slices of a warp, their offsets from shared memory (n = 2000, degree 12:
// 1.81 -> 1.73 ms for 61 steps, n = 8000 32.0 -> 30.2 ms for 64; two groups
// ahead 1.74 and 30.6 ms, three 1.78 and 31.7 ms: the registers run out).
template <int C>
__global__ void __launch_bounds__(1024) sparse_step_kernel(SellView g, const float* __restrict__ H,
                                                           float* __restrict__ Hn, int n, int per_split, int vec,
                                                           int* changed, int step, int fill) {
    extern __shared__ __align__(16) float hs[];
    __shared__ int s_diff;
    int* s_ptr = reinterpret_cast<int*>(hs + (size_t)n * C);  // offsets of this CTA's slices
    constexpr int kLanes = C / 4;           // lanes per row
    constexpr int kRows = 32 / kLanes;      // rows per warp
    constexpr int kSlices = kRows / kSellRows;
    const float inf = __int_as_float(kInfBits);
    const int tid = threadIdx.x, lane = tid & 31;
    const int i0 = blockIdx.x * C;
    const int first = blockIdx.y * per_split, last = min(g.nslices, first + per_split);
    if (step > 0 && changed[step - 1] == 0) {  // fixed point reached earlier
        if (!fill) return;
        const int j0 = first * kSellRows, w = min(n, last * kSellRows) - j0;
        for (int idx = tid; idx < C * w; idx += blockDim.x) {
            const int i = i0 + idx / w, j = j0 + idx % w;
            if (i < n) Hn[(size_t)i * n + j] = H[(size_t)i * n + j];
        }
        return;
    }
    if (tid == 0) s_diff = 0;
    if (vec && i0 + C <= n) {
        for (int idx = tid; idx < n * kLanes; idx += blockDim.x) {
            const int k = idx / kLanes, q = idx % kLanes;
            cp_async(hs + 4 * idx, H + (size_t)k * n + i0 + 4 * q, 1);
        }
    } else {
        for (int idx = tid; idx < n * C; idx += blockDim.x) {
            const int k = idx / C, c = idx % C;
            if (i0 + c < n) cp_async(hs + idx, H + (size_t)k * n + i0 + c, 0);
            else hs[idx] = inf;
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    for (int idx = tid; idx <= last - first; idx += blockDim.x) s_ptr[idx] = __ldg(g.ptr + first + idx);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    const float4* h4 = reinterpret_cast<const float4*>(hs);
    const int q = lane % kLanes, rw = lane / kLanes, r = rw % kSellRows;
    const int stride = (blockDim.x >> 5) * kSlices;
    // this lane's columns: rows i0 + 4q .. of the transposed result
    const int cols = n - (i0 + 4 * q);
    float* out = Hn + (size_t)(i0 + 4 * q) * n;
    const float* old = H + (size_t)(i0 + 4 * q) * n;
    bool diff = false;
    int s = first + (tid >> 5) * kSlices + rw / kSellRows;
    // a group of entries is loaded while the one before it is reduced, on into the next slice
    int ls = s, left = 0;
    const int2* ed = nullptr;
    auto open = [&] {  // first slice from ls on that has entries
        for (; ls < last; ls += stride) {
            const int e0 = s_ptr[ls - first];
            left = (s_ptr[ls - first + 1] - e0) / kSellUnroll;
            ed = g.edges + (size_t)e0 * kSellRows + r;
            if (left > 0) return;
        }
    };
    open();
    int2 p[kSellUnroll];
    auto load = [&] {
        if (left == 0) return;
#pragma unroll
        for (int e = 0; e < kSellUnroll; ++e) p[e] = __ldg(ed + e * kSellRows);
        ed += kSellUnroll * kSellRows;
        if (--left == 0) {
            ls += stride;
            open();
        }
    };
    load();
    for (; s < last; s += stride) {
        int groups = (s_ptr[s - first + 1] - s_ptr[s - first]) / kSellUnroll;
        float acc[4] = {inf, inf, inf, inf};
        for (; groups > 0; --groups) {
            float4 v[kSellUnroll];
            float a[kSellUnroll];
#pragma unroll
            for (int e = 0; e < kSellUnroll; ++e) {
                v[e] = h4[p[e].x * kLanes + q];
                a[e] = __int_as_float(p[e].y);
            }
            load();
#pragma unroll
            for (int e = 0; e < kSellUnroll; e += 2) {
                acc[0] = nsg_min3(acc[0], __fadd_rn(a[e], v[e].x), __fadd_rn(a[e + 1], v[e + 1].x));
                acc[1] = nsg_min3(acc[1], __fadd_rn(a[e], v[e].y), __fadd_rn(a[e + 1], v[e + 1].y));
                acc[2] = nsg_min3(acc[2], __fadd_rn(a[e], v[e].z), __fadd_rn(a[e + 1], v[e + 1].z));
                acc[3] = nsg_min3(acc[3], __fadd_rn(a[e], v[e].w), __fadd_rn(a[e + 1], v[e + 1].w));
            }
        }
        const int j = s * kSellRows + r;
        if (j >= n) continue;
        const bool look = !diff && *reinterpret_cast<volatile int*>(&s_diff) == 0;
        float* on = out + j;
        const float* oh = old + j;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (u < cols) {
                if (look && __float_as_int(acc[u]) != __float_as_int(*oh)) diff = true;
                *on = acc[u];
            }
            on += n;
            oh += n;
        }
        if (diff) s_diff = 1;
    }
    if (__syncthreads_or(diff) && tid == 0) changed[step] = 1;
}

// The back-walk of netcalc/src/hedetniemi_gpu.cu:70-107, as
// hedetniemi_walk_kernel (apsp.cu): the first q (ascending, q != j) with
// H_p[i][q] + A[q][k] - len < tolerance. An entry A[q][k] = +inf never
// passes that test, so only the other entries of column k are looked at.
__global__ void sparse_walk_kernel(SellView cols, const float* __restrict__ H, const float* __restrict__ Hi,
                                   int* __restrict__ paths, float tolerance, int n, int L) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y * blockDim.y + threadIdx.y;
    if (i >= n || j >= n) return;
    int* cell = paths + (size_t)i * L * n + (size_t)j * L;
    if (i == j) {
        for (int p = 0; p < L; ++p) cell[p] = i;
        return;
    }
    float len = H[(size_t)i * n + j];
    int k = j;
    for (int p = L - 1; p >= 0; --p) {
        const float* hp = Hi + (size_t)p * n * n + (size_t)i * n;
        const int s = k / kSellRows;
        const int end = __ldg(cols.ptr + s + 1);
        const int2* ed = cols.edges + k % kSellRows;
        for (int e = __ldg(cols.ptr + s); e < end; ++e) {
            const int2 c = __ldg(ed + (size_t)e * kSellRows);
            if (c.x == j) continue;
            const float a = __int_as_float(c.y);
            if (__fsub_rn(__fadd_rn(hp[c.x], a), len) < tolerance) {
                len = __fsub_rn(len, a);
                k = c.x;
                break;
            }
        }
        cell[p] = k;
    }
}

int sm_count_now() {
    int dev = 0, sms = 0;
    NSG_CUDA(cudaGetDevice(&dev));
    NSG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return sms;
}

// Columns per CTA: 16 while n rows of them fit in shared memory, then 8 and 4.
constexpr int kMax16 = 3500, kMax8 = 7000;
constexpr int kStepSmem = 227 * 1024 - 64;
constexpr int step_smem(int n, int columns, int slices) { return 4 * (n * columns + slices + 1); }
static_assert(step_smem(kMax16, 16, kMax16 / 8 + 1) <= kStepSmem && step_smem(kMax8, 8, kMax8 / 8 + 1) <= kStepSmem &&
                  step_smem(kSparseMaxN, 4, kSparseMaxN / 8 + 1) <= kStepSmem,
              "a column block fits in shared memory");

template <int C>
void launch_step(const SellView& g, const float* H, float* Hn, int n, int* changed, int step, bool fill,
                 cudaStream_t s) {
    static_assert(C % 4 == 0 && 32 / (C / 4) >= kSellRows, "whole slices per warp");
    constexpr int kSlices = 32 / (C / 4) / kSellRows;
    const int blocks = (n + C - 1) / C;
    // slices split over CTAs until there is one per SM, at least one warp's worth each
    const int splits = std::max(1, std::min(sm_count_now() / blocks, g.nslices / (4 * kSlices)));
    const int per = (g.nslices + splits - 1) / splits;
    const int warps = std::min(32, std::max(4, (per + kSlices - 1) / kSlices));
    const int vec = (n % 4 == 0) && (reinterpret_cast<uintptr_t>(H) % 16 == 0);
    // set on every launch: the attribute belongs to the current device. One
    // value for all sizes: another thread may set it before this launch.
    NSG_CUDA(cudaFuncSetAttribute(sparse_step_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, kStepSmem));
    const int smem = step_smem(n, C, per);
    sparse_step_kernel<C><<<dim3(blocks, (g.nslices + per - 1) / per), 32 * warps, smem, s>>>(
        g, H, Hn, n, per, vec, changed, step, fill ? 1 : 0);
    NSG_CUDA(cudaGetLastError());
}

}  // namespace

void sparse_analyze(const float* A, int n, GraphInfo* info, int* counts, int* ptr, cudaStream_t s) {
    const int t = (n + 31) / 32;
    analyze_kernel<<<dim3(t, t), dim3(32, 8), 0, s>>>(A, n, info, counts);
    slice_kernel<<<1, 1024, 0, s>>>(counts, nullptr, n, sell_slices(n), ptr, info);
    NSG_CUDA(cudaGetLastError());
}

void sparse_count(const float* A, int ld, int n, GraphInfo* info, int* counts, int* ptr, cudaStream_t s) {
    count_kernel<<<(n + 7) / 8, 256, 0, s>>>(A, ld, n, counts);
    slice_kernel<<<1, 1024, 0, s>>>(counts, nullptr, n, sell_slices(n), ptr, info);
    NSG_CUDA(cudaGetLastError());
}

void sparse_fill(const float* A, int ld, int n, const int* ptr, int2* edges, cudaStream_t s) {
    const int ns = sell_slices(n);
    fill_kernel<<<ns, 32 * kSellRows, 0, s>>>(A, ld, n, ns, nullptr, nullptr, ptr, edges);
    NSG_CUDA(cudaGetLastError());
}

void sparse_sort(const int* counts, int n, int* order, int* rank, cudaStream_t s) {
    sort_kernel<<<(n + 255) / 256, 256, 0, s>>>(counts, n, order, rank);
    NSG_CUDA(cudaGetLastError());
}

void sparse_slices_sorted(const int* counts, const int* order, int n, GraphInfo* info, int* ptr, cudaStream_t s) {
    slice_kernel<<<1, 1024, 0, s>>>(counts, order, n, sell_slices(n), ptr, info);
    NSG_CUDA(cudaGetLastError());
}

void sparse_fill_sorted(const float* A, int n, const int* order, const int* rank, const int* ptr, int2* edges,
                        cudaStream_t s) {
    const int ns = sell_slices(n);
    fill_kernel<<<ns, 32 * kSellRows, 0, s>>>(A, n, n, ns, order, rank, ptr, edges);
    NSG_CUDA(cudaGetLastError());
}

namespace {
void launch_pick(const float* A, float* out, int n, const int* from, const int* to, const int* pick, cudaStream_t s) {
    const size_t smem = sizeof(float) * n;
    // set on every launch: the attribute belongs to the current device
    NSG_CUDA(cudaFuncSetAttribute(pick_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(sizeof(float) * kSparseMaxN)));
    pick_kernel<<<n, 256, smem, s>>>(A, out, n, from, to, pick);
    NSG_CUDA(cudaGetLastError());
}
}  // namespace

void sparse_relabel(const float* A, float* out, int n, const int* order, cudaStream_t s) {
    launch_pick(A, out, n, order, nullptr, order, s);
}

void sparse_restore(const float* A, float* out, int n, const int* order, const int* rank, cudaStream_t s) {
    launch_pick(A, out, n, nullptr, order, rank, s);
}

void sparse_step(const SellView& g, const float* H, float* Hn, int n, int* changed, int step, bool fill,
                 cudaStream_t s) {
    if (n <= kMax16) launch_step<16>(g, H, Hn, n, changed, step, fill, s);
    else if (n <= kMax8) launch_step<8>(g, H, Hn, n, changed, step, fill, s);
    else launch_step<4>(g, H, Hn, n, changed, step, fill, s);
}

double sparse_step_seconds(long long width, int n) {
    // start-up, H in and out, entries: 28 us measured at n = 2000 (width 3260),
    // 9 to 12 at n = 800, 85 to 110 at n = 4000
    return 5.5e-6 + 8.0 * n * n / 2.2e12 + 8.0 * static_cast<double>(width) * n / 6e12;
}

// Sorted slices hold the entries and about two of padding per row group (their
// widths are rounded up to kSellUnroll). Measured per solve: the sort, the
// slices and the fill 25 us, the two passes over the matrix 2.7 TB/s. Random
// geometric graphs of mean degree 12, without -> with: n = 1200 350 -> 353 us
// after 16 steps (not taken), n = 2000 602 -> 587 us after 16 and 2.00 ->
// 1.81 ms after 61, n = 8000 9.42 -> 8.72 ms after 16. A ring of degree 6 has
// nothing to gain: n = 4000 1.55 -> 1.65 ms (not taken).
bool sparse_sort_pays(long long width, long long entries, int n, int steps) {
    const long long sorted = entries / kSellRows + (kSellUnroll / 2) * sell_slices(n);
    if (sorted >= width) return false;
    const double saved = sparse_step_seconds(width, n) - sparse_step_seconds(sorted, n);
    return std::min(steps, 16) * saved > 25e-6 + 16.0 * n * n / 2.7e12;
}

void sparse_walk(const SellView& cols, const float* H, const float* Hi, int* paths, float tolerance, int n, int L,
                 cudaStream_t s) {
    dim3 block(32, 8);
    dim3 grid((n + 31) / 32, (n + 7) / 8);
    sparse_walk_kernel<<<grid, block, 0, s>>>(cols, H, Hi, paths, tolerance, n, L);
    NSG_CUDA(cudaGetLastError());
}

}  // namespace nsg
