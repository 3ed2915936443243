// Hedetniemi all-pairs shortest paths on the GPU.
//
// One step computes, for every (i, j),
//     Hn[i][j] = min_k fl(A[j][k] + H[k][i])
// the update of netcalc/src/hedetniemi_gpu.cu:28-45, as a Jacobi step from H
// into a second buffer (the reference updates H in place). Every entry is a
// minimum of single roundings, so the result does not depend on the order k
// is visited in and matches the CPU restatement bit for bit.
//
// The iterate is kept transposed, X = H^T, so both operands of a step are
// contiguous along k:
//     Xn[j][i] = Hn[i][j] = min_k fl(X[i][k] + A[j][k]).
// X and a copy of A live in P x P buffers (P = n rounded up to 128, +inf
// outside n x n, so padded k contribute nothing and no load needs a bound
// check); the result is transposed back into H once at the end.
//
// Kernel shape: a 64 x 64 output tile per CTA of 256 threads, 4 x 4 outputs
// per thread (four CTAs per SM, 64 registers; 128 x 64 tiles at 8 x 4 per
// thread and two CTAs per SM took 12% longer). k runs in slabs of 32 (16
// took 6% longer: twice the barriers): both operand tiles (64 rows of 32
// floats each) are copied into shared memory with 16-byte cp.async into two
// buffers, so the next slab loads while this one is reduced. Rows are padded
// to 36 floats, which keeps the 16-byte reads of a quarter-warp on distinct
// banks. Each thread reads four consecutive k of a
// row at once; one packed add (add.rn.f32x2) forms the sums for (k, k+1) and
// one three-input min folds both into the running minimum: two instructions
// per two (i, j, k) terms. The work is FADD/FMNMX issue-bound on CUDA cores;
// a min-plus product has no tensor-core form.
//
// Convergence: step t writes changed[t] = 1 when any entry differs from the
// previous iterate; step t+1 returns at once when changed[t] == 0 (the
// iterate is then a fixed point and both buffers hold it).
//
// Repeated squaring. When the path length is unbounded (maxPathLength >=
// n-1) and A is symmetric with a zero diagonal and no negative weight, the
// iteration's fixed point is the all-pairs shortest-path matrix A*, and
// H <- H (x) H reaches it in ceil(log2(hop diameter)) products instead of
// one step per hop (H_t = A^(2^t); once a product changes nothing, every
// higher power is equal). The same step kernel does the product with the
// iterate as both operands. A squared entry sums two partial paths, where a
// Jacobi step adds one edge to a path, so on float weights the roundings can
// differ from the reference's in the last bits. On integer-valued weights
// whose path sums stay below 2^24 every sum is exact in float, and squaring
// gives the reference's fixed point bit for bit; the automatic mode squares
// only then (analyze_kernel checks A on the device) and runs Jacobi steps
// otherwise.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "apsp.h"
#include "apsp_sparse.h"
#include "common.cuh"
#include "engine.h"

namespace nsg {
namespace {

constexpr int kTileI = 64;  // output rows i per CTA (rows of X)
constexpr int kTileJ = 64;   // output columns j per CTA (rows of A)
constexpr int kSlab = 32;    // k values per stage
constexpr int kRow = 36;     // shared-memory row stride (floats)
constexpr int kThreads = 256;
constexpr int kPad = 128;    // P is a multiple of this (and of kTileJ, kSlab)

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// S CTAs of a cluster share a tile (blockIdx.z), each reducing 1/S of k; the
// partial minima meet in distributed shared memory, 1/S of the tile's
// outputs per CTA. A minimum does not depend on the order, so the result is
// the same. Matrices of few tiles leave most SMs idle otherwise: at n = 500 64
// tiles took 25 us per step on 64 of 152 SMs.
template <int S>
__global__ void __launch_bounds__(kThreads, 4)
hedetniemi_step_kernel(const float* __restrict__ X, const float* __restrict__ Ap,
                       float* __restrict__ Xn, int n, int P, int* changed, int step) {
    if (step > 0 && changed[step - 1] == 0) return;  // fixed point reached earlier
    __shared__ __align__(16) float Xs[2][kTileI][kRow];
    __shared__ __align__(16) float As[2][kTileJ][kRow];
    const float inf = __int_as_float(0x7f800000);
    const int tid = threadIdx.x;
    // rows i = i0 + tx + 16u (u < 4), columns j = j0 + ty + 16v (v < 4)
    const int tx = tid & 15;
    const int ty = tid >> 4;
    const int i0 = blockIdx.y * kTileI;
    const int j0 = blockIdx.x * kTileJ;
    const float* xg = X + (size_t)i0 * P;
    const float* ag = Ap + (size_t)j0 * P;
    // 64 + 64 rows of eight 16-byte chunks: four chunks per thread
    auto load_slab = [&](int buf, int k0) {
#pragma unroll
        constexpr int kChunks = kSlab / 4;  // 16-byte chunks per row
        static_assert((kChunks * (kTileI + kTileJ)) % kThreads == 0, "whole chunks per thread");
        for (int e = 0; e < (kChunks * (kTileI + kTileJ)) / kThreads; ++e) {
            const int c = tid + kThreads * e;
            if (c < kChunks * kTileI) {
                const int r = c / kChunks, q = c % kChunks;
                cp_async16(&Xs[buf][r][4 * q], xg + (size_t)r * P + k0 + 4 * q);
            } else {
                const int c2 = c - kChunks * kTileI;
                const int r = c2 / kChunks, q = c2 % kChunks;
                cp_async16(&As[buf][r][4 * q], ag + (size_t)r * P + k0 + 4 * q);
            }
        }
        cp_async_commit();
    };

    float acc[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) acc[u][v] = inf;

    const int nslab = P / kSlab / S;
    const int k_first = S > 1 ? static_cast<int>(blockIdx.z) * nslab * kSlab : 0;
    load_slab(0, k_first);
    for (int sl = 0; sl < nslab; ++sl) {
        if (sl + 1 < nslab) {
            load_slab((sl + 1) & 1, k_first + (sl + 1) * kSlab);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const int b = sl & 1;
#pragma unroll
        for (int kq = 0; kq < kSlab / 4; ++kq) {
            float4 x[4], a[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) x[u] = *reinterpret_cast<const float4*>(&Xs[b][tx + 16 * u][4 * kq]);
#pragma unroll
            for (int v = 0; v < 4; ++v) a[v] = *reinterpret_cast<const float4*>(&As[b][ty + 16 * v][4 * kq]);
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    const float2 s0 = nsg_add2(make_float2(x[u].x, x[u].y), make_float2(a[v].x, a[v].y));
                    const float2 s1 = nsg_add2(make_float2(x[u].z, x[u].w), make_float2(a[v].z, a[v].w));
                    acc[u][v] = nsg_min3(acc[u][v], s0.x, s0.y);
                    acc[u][v] = nsg_min3(acc[u][v], s1.x, s1.y);
                }
        }
        __syncthreads();  // the buffer is refilled two slabs on
    }

    bool diff = false;
    if constexpr (S == 1) {
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int i = i0 + tx + 16 * u;
            if (i >= n) continue;
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int j = j0 + ty + 16 * v;
                if (j >= n) continue;
                const size_t o = (size_t)j * P + i;
                if (__float_as_int(acc[u][v]) != __float_as_int(__ldg(X + o))) diff = true;
                Xn[o] = acc[u][v];
            }
        }
    } else {
        static_assert(sizeof(Xs) >= sizeof(float) * kTileI * kTileJ, "a tile's partial minima fit one stage pair");
        auto cluster = cooperative_groups::this_cluster();
        float* part = &Xs[0][0][0];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) part[(ty + 16 * v) * kTileI + tx + 16 * u] = acc[u][v];
        cluster.sync();
        constexpr int kShare = kTileI * kTileJ / S;
        for (int e = blockIdx.z * kShare + tid; e < (static_cast<int>(blockIdx.z) + 1) * kShare; e += kThreads) {
            float m = inf;
#pragma unroll
            for (int r = 0; r < S; ++r) m = fminf(m, cluster.map_shared_rank(part, r)[e]);
            const int i = i0 + e % kTileI, j = j0 + e / kTileI;
            if (i >= n || j >= n) continue;
            const size_t o = (size_t)j * P + i;
            if (__float_as_int(m) != __float_as_int(__ldg(X + o))) diff = true;
            Xn[o] = m;
        }
        cluster.sync();  // the others may still read this CTA's part
    }
    if (__syncthreads_or(diff) && tid == 0) changed[step] = 1;
}

// dst (P x P) = src (n x n, stride n) or its transpose, +inf outside n x n.
__global__ void pad_copy_kernel(const float* __restrict__ src, float* __restrict__ dst, int n, int P,
                                int transpose) {
    __shared__ float t[32][33];
    const float inf = __int_as_float(0x7f800000);
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;  // dst tile: rows by.., columns bx..
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const int sr = transpose ? bx + yy : by + yy;
        const int sc = transpose ? by + threadIdx.x : bx + threadIdx.x;
        t[yy][threadIdx.x] = (sr < n && sc < n) ? __ldg(src + (size_t)sr * n + sc) : inf;
    }
    __syncthreads();
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const int r = by + yy, c = bx + threadIdx.x;
        dst[(size_t)r * P + c] = transpose ? t[threadIdx.x][yy] : t[yy][threadIdx.x];
    }
}

// The three padded matrices of a solve from one read of src: a copy, and its
// transpose twice.
__global__ void pad_iterates_kernel(const float* __restrict__ src, float* __restrict__ Ap, float* __restrict__ X0,
                                    float* __restrict__ X1, int n, int P) {
    __shared__ float t[32][33];
    const float inf = __int_as_float(0x7f800000);
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;  // tile of Ap: rows by.., columns bx..
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const int r = by + yy, c = bx + threadIdx.x;
        const float v = (r < n && c < n) ? __ldg(src + (size_t)r * n + c) : inf;
        t[yy][threadIdx.x] = v;
        Ap[(size_t)r * P + c] = v;
    }
    __syncthreads();
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const size_t o = (size_t)(bx + yy) * P + by + threadIdx.x;
        X0[o] = X1[o] = t[threadIdx.x][yy];
    }
}

// H (n x n) = the n x n corner of X (stride P), transposed.
__global__ void unpad_transpose_kernel(const float* __restrict__ X, float* __restrict__ H, int n, int P) {
    __shared__ float t[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32;  // H tile: rows by.., columns bx..
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y)
        t[yy][threadIdx.x] = __ldg(X + (size_t)(bx + yy) * P + by + threadIdx.x);
    __syncthreads();
    for (int yy = threadIdx.y; yy < 32; yy += blockDim.y) {
        const int r = by + yy, c = bx + threadIdx.x;
        if (r < n && c < n) H[(size_t)r * n + c] = t[threadIdx.x][yy];
    }
}

// Back-walk of netcalc/src/hedetniemi_gpu.cu:70-107 over snapshots Hi[p]
// (H before step p). Diagonal cells hold i.
__global__ void hedetniemi_walk_kernel(const float* __restrict__ H, const float* __restrict__ Hi,
                                       const float* __restrict__ A, int* __restrict__ paths,
                                       float tolerance, int n, int L) {
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
        for (int q = 0; q < n; ++q) {
            if (q == j) continue;
            const float a = A[(size_t)q * n + k];
            if (__fsub_rn(__fadd_rn(hp[q], a), len) < tolerance) {
                len = __fsub_rn(len, a);
                k = q;
                break;
            }
        }
        cell[p] = k;
    }
}

// mode 0: 1/r adjacency (netcalc/src/hedetniemi_gpu.cu:10-26);
// mode 1: -ln(r) adjacency, evaluated in double and rounded to float.
__global__ void corr_to_adj_kernel(const float* __restrict__ C, float* __restrict__ A, int n,
                                   int mode) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)n * n) return;
    const int i = static_cast<int>(idx / n), j = static_cast<int>(idx % n);
    const float c = C[idx];
    const float inf = __int_as_float(0x7f800000);
    float v;
    if (i == j) {
        v = 0.f;
    } else if (mode == 0) {
        v = (c == 0.f) ? inf : __fdiv_rn(1.f, c);
    } else {
        v = (c > 0.f) ? __double2float_rn(-log(static_cast<double>(c))) : inf;
    }
    A[idx] = v;
}

template <int S>
void launch_split_step(const float* Ap, const float* X, float* Xn, int n, int P, int* changed, int step,
                       cudaStream_t s) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(P / kTileJ, P / kTileI, S);
    c.blockDim = dim3(kThreads);
    c.stream = s;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim = {1, 1, S};
    c.attrs = &a;
    c.numAttrs = 1;
    NSG_CUDA(cudaLaunchKernelEx(&c, hedetniemi_step_kernel<S>, X, Ap, Xn, n, P, changed, step));
}

// CTAs of a cluster that share a tile: four up to 160 tiles (n <= 768), two up
// to 320 (n <= 1024), as the GPU holds 608 CTAs of this kernel.
int step_split(int tiles) { return tiles <= 160 ? 4 : tiles <= 320 ? 2 : 1; }

void launch_step(const float* Ap, const float* X, float* Xn, int n, int P, int* changed, int step,
                 cudaStream_t s) {
    const int split = step_split((P / kTileJ) * (P / kTileI));
    if (split == 4) {
        launch_split_step<4>(Ap, X, Xn, n, P, changed, step, s);
    } else if (split == 2) {
        launch_split_step<2>(Ap, X, Xn, n, P, changed, step, s);
    } else {
        hedetniemi_step_kernel<1><<<dim3(P / kTileJ, P / kTileI), kThreads, 0, s>>>(X, Ap, Xn, n, P, changed, step);
        NSG_CUDA(cudaGetLastError());
    }
}

void launch_pad(const float* src, float* dst, int n, int P, bool transpose, cudaStream_t s) {
    pad_copy_kernel<<<dim3(P / 32, P / 32), dim3(32, 8), 0, s>>>(src, dst, n, P, transpose ? 1 : 0);
    NSG_CUDA(cudaGetLastError());
}

void launch_unpad(const float* X, float* H, int n, int P, cudaStream_t s) {
    unpad_transpose_kernel<<<dim3((n + 31) / 32, (n + 31) / 32), dim3(32, 8), 0, s>>>(X, H, n, P);
    NSG_CUDA(cudaGetLastError());
}

// The device's pool of solver workspace. The driver's default pool gives its
// memory back at every synchronisation, so each small solve mapped its
// matrices anew; this one keeps up to kPoolKeep bytes between solves and gives
// them back through apsp_release_pools.
constexpr unsigned long long kPoolKeep = 1ull << 30;
std::mutex g_pool_mu;
std::map<int, cudaMemPool_t> g_pools;

cudaMemPool_t workspace_pool() {
    int dev = 0;
    NSG_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_pool_mu);
    cudaMemPool_t& pool = g_pools[dev];
    if (!pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        NSG_CUDA(cudaMemPoolCreate(&pool, &props));
        unsigned long long keep = kPoolKeep;
        NSG_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
    }
    return pool;
}

// Workspace allocated and freed in the order of the solver's stream, so a
// solve does not wait for kernels on other streams.
struct DevMem {
    void* p = nullptr;
    cudaStream_t s;
    DevMem(size_t bytes, cudaStream_t st) : s(st) {
        if (bytes) alloc(bytes, st);
    }
    void alloc(size_t bytes, cudaStream_t st) {
        s = st;
        NSG_CUDA(cudaMallocFromPoolAsync(&p, bytes, workspace_pool(), st));
    }
    ~DevMem() { if (p) cudaFreeAsync(p, s); }
    // For what a kernel is about to write or read: a block that was not
    // allocated ends the solve with an error.
    float* floats() const {
        if (!p) fail(NSG_ERR_CUDA, "shortest paths: a workspace block is not there");
        return static_cast<float*>(p);
    }
    DevMem(const DevMem&) = delete;
    DevMem& operator=(const DevMem&) = delete;
};

// Padded copy of A and the two transposed iterates X = H^T, both starting at A^T.
struct Iterates {
    int P;
    DevMem mem;
    float* Ap;
    float* X[2];
    Iterates(const float* A, int n, cudaStream_t s)
        : P((n + kPad - 1) / kPad * kPad), mem(sizeof(float) * 3 * (size_t)P * P, s) {
        const size_t pp = (size_t)P * P;
        Ap = static_cast<float*>(mem.p);
        X[0] = Ap + pp;
        X[1] = Ap + 2 * pp;
        pad_iterates_kernel<<<dim3(P / 32, P / 32), dim3(32, 8), 0, s>>>(A, Ap, X[0], X[1], n, P);
        NSG_CUDA(cudaGetLastError());
    }
};

std::atomic<int> g_method{-1};

int ceil_log2(int v) {
    int b = 0;
    while ((1 << b) < v) ++b;
    return b;
}

// Seconds of a dense step: what the step of a small matrix takes anyway, and
// 34.2 ns per k of a tile for the SM with the most tiles (measured at P = 512 to
// 2048: within 6%, where P^3 alone was off by a quarter).
double dense_step_seconds(int n) {
    const int P = (n + kPad - 1) / kPad * kPad, tiles = (P / kTileJ) * (P / kTileI), split = step_split(tiles);
    const int sms = sm_count();
    return 6e-6 + 34.2e-9 * ((tiles * split + sms - 1) / sms) * (P / split);
}

// A sparse step of a solve: a row's entries are a chain of their own.
double sparse_solve_step_seconds(long long width, int n) {
    return sparse_step_seconds(width, n) + 40e-9 * static_cast<double>(width) / sell_slices(n);
}

// Whether a solve of few dense steps is over before the analysis of A (25 us
// with its wait) could pay: n = 300, one to three steps 73 to 96 us without it,
// against 82 to 100 with it for a sparse A and 94 to 118 for a full one. Node
// sequences: every step is kept, and a back-walk looks at n entries instead of a
// row's. Up to three steps of those gain less on a sparse symmetric A (n = 64,
// three steps: 108 us against 131) than full or asymmetric ones lose (150).
bool analysis_pays(int n, int steps, bool walk) {
    const double dense = dense_step_seconds(n);
    if (walk) return steps * (dense - 2.5e-6 + 0.1e-6 * (n - 10)) > (steps <= 3 ? 45e-6 : 20e-6);
    return std::min(steps, 8) * (dense - 5.6e-6) > 15e-6;
}

// Whether the steps go over the entries: the fill of their lists (12 us, and the
// transpose's for a walk over an asymmetric A) and the steps, against the
// padded copies and the dense steps. Four steps are counted on: full matrices
// converge in about that many, and sparse ones gain with every further step.
// N = 200, full, five steps: 153 us over the entries, 133 dense; degree 16: 106
// and 126.
bool sparse_pays(long long width, int n, int steps, bool walk, bool symmetric) {
    const double row = static_cast<double>(width) / sell_slices(n);
    const double sparse = sparse_solve_step_seconds(width, n), dense = dense_step_seconds(n);
    if (!walk) return 12e-6 + std::min(steps, 4) * sparse < 22e-6 + std::min(steps, 4) * dense;
    const double fill = (symmetric ? 12e-6 : 48e-6) + 0.4e-6 * row;
    return fill + steps * (sparse + 0.1e-6 * row) < 25e-6 + steps * (dense + 3.3e-6 + 0.1e-6 * n);
}

// Exact squaring on a sparse A: every A^(t+1) is the same matrix whichever way
// it is reached, so 2^f - 1 sparse steps can stand for the first f products.
// They cost a detour (the fill, the flags' wait and a copy, 25 us) and pay
// where products are long. The f with the least time for a graph of points in
// space (about 3.3 N^(1/3) (10 / degree)^(1/4) hops, N = 64 to 2000, degree 6 to
// 16; other graphs go on with products where the steps end): none up to about
// n = 700 (N = 200: 150 us against 185 with one step), three or four up to 1300,
// all steps beyond (N = 2000: 1.3 ms against 3.6).
int steps_before_products(long long width, long long entries, int n) {
    const double step = sparse_solve_step_seconds(width, n), product = dense_step_seconds(n);
    const double degree = std::max(1.0, static_cast<double>(entries) / n - 1);
    const double hops = std::min(n - 1.0, 3.3 * std::cbrt(n) * std::pow(10 / degree, 0.25));
    const int products = ceil_log2(static_cast<int>(std::ceil(hops)) + 1) + 1;
    int best = 0;
    double least = products * product;
    for (int f = 1; f <= 6 && f <= ceil_log2(n); ++f) {
        const double steps = (1 << f) - 1;
        const double rest = steps >= 1.15 * hops ? 0 : std::max(1, products - f) * product;
        const double t = 25e-6 + std::min(steps, 1.15 * hops) * step + rest;
        if (t < least) {
            least = t;
            best = f;
        }
    }
    return best;
}

// A and how a solve of it runs.
struct Graph {
    int squaring = 0;  // repeated squaring reaches the result: 1 exactly, 2 within rounding (requested)
    bool symmetric = false;
    int first = 0;        // powers of A taken by sparse steps before products go on (exact squaring)
    bool sparse = false;  // steps over the finite entries; rounded squaring takes dense products alone
    long long width = 0;
    DevMem words, edges;  // GraphInfo, counts, slice offsets, order, rank; the entries
    SellView rows{};
    const int* order = nullptr;  // vertices by falling degree, where the entries are in those labels
    const int* rank = nullptr;

    // unbounded: every shortest path may be taken (maxPathLength >= n - 1);
    // steps: the most the solve takes; walk: for node sequences (the labels
    // stay the matrix's own)
    Graph(const float* A, int n, bool unbounded, int steps, bool walk, cudaStream_t s)
        : words(sizeof(GraphInfo) + sizeof(int) * (4 * (size_t)n + 2), s), edges(0, nullptr) {
        const int method = g_method.load();
        const bool may_square = method != 0 && n >= 2 && unbounded;
        if (!may_square && !analysis_pays(n, steps, walk)) return;
        GraphInfo* info = static_cast<GraphInfo*>(words.p);
        int* counts = reinterpret_cast<int*>(info + 1);
        int* ptr = counts + n;
        NSG_CUDA(cudaMemsetAsync(words.p, 0, sizeof(GraphInfo) + sizeof(int) * (size_t)n, s));
        sparse_analyze(A, n, info, counts, ptr, s);
        GraphInfo h{};
        NSG_CUDA(cudaMemcpyAsync(&h, info, sizeof(h), cudaMemcpyDeviceToHost, s));
        NSG_CUDA(cudaStreamSynchronize(s));
        symmetric = !(h.flags & 1);
        width = h.width;
        if (may_square && !(h.flags & 7)) {
            float wmax;
            std::memcpy(&wmax, &h.wmax, sizeof(float));
            // integer weights with every path sum (at most n-1 edges) exact in float
            if (!(h.flags & 8) && static_cast<double>(wmax) * (n - 1) < 16777216.0) squaring = 1;
            else if (method == 1) squaring = 2;  // squaring requested on any weights
        }
        if (n > kSparseMaxN || squaring == 2) return;
        if (squaring == 1) first = steps_before_products(width, h.entries, n);
        sparse = squaring == 1 ? first > 0 : sparse_pays(width, n, steps, walk, symmetric);
        if (!sparse) return;
        edges.alloc(sizeof(int2) * kSellRows * (size_t)std::max<long long>(1, width), s);
        if (!walk && sparse_sort_pays(width, h.entries, n, steps)) {  // shorter slices, so the entries fit
            int* ord = ptr + n + 2;
            sparse_sort(counts, n, ord, ord + n, s);
            sparse_slices_sorted(counts, ord, n, info, ptr, s);
            sparse_fill_sorted(A, n, ord, ord + n, ptr, static_cast<int2*>(edges.p), s);
            order = ord;
            rank = ord + n;
        } else {
            sparse_fill(A, n, n, ptr, static_cast<int2*>(edges.p), s);
        }
        rows = {static_cast<const int2*>(edges.p), ptr, sell_slices(n)};
    }
};

// Jacobi steps launched in chunks; a chunk's flags are read before the next, so
// long runs stop shortly after the fixed point (steps past it return at once)
// and the later chunks, which hide a read each, are longer. launch(t) enqueues
// step t; finish(), if the last chunk is reached, what follows all steps. Returns
// the steps run up to and including the one that changed nothing, *launched the
// steps enqueued, *converged whether there was such a step.
template <class F, class G>
int run_steps(int most, int* changed, cudaStream_t s, F&& launch, G&& finish, int* launched, bool* converged) {
    std::vector<int> flags;
    int chunk = 8, t = 0;
    *converged = false;
    while (t < most && !*converged) {
        const int begin = t, end = t + std::min(most - t, chunk);
        for (; t < end; ++t) launch(t);
        if (t == most) finish();
        flags.resize(t);
        NSG_CUDA(cudaMemcpyAsync(flags.data() + begin, changed + begin, sizeof(int) * (t - begin), cudaMemcpyDeviceToHost, s));
        NSG_CUDA(cudaStreamSynchronize(s));
        *converged = flags[t - 1] == 0;
        chunk = std::min(2 * chunk, 64);
    }
    *launched = t;
    if (!*converged) return t;
    int q = 0;
    while (flags[q]) ++q;
    return q + 1;
}

bool overlap(const float* a, const float* b, size_t nn) { return a < b + nn && b < a + nn; }

// Sparse Jacobi steps between H and T, the first one reading A (or T, if A is
// null). Returns as run_steps; *at is the iterate after *launched steps, in T
// where both hold it.
int sparse_steps(const Graph& g, const float* A, float* H, float* T, int n, int most, cudaStream_t s, int* launched,
                 bool* converged, float** at) {
    DevMem changed(sizeof(int) * most, s);
    NSG_CUDA(cudaMemsetAsync(changed.p, 0, sizeof(int) * most, s));
    int* ch = static_cast<int*>(changed.p);
    const int steps = run_steps(most, ch, s, [&](int t) {
        sparse_step(g.rows, t == 0 && A ? A : (t & 1) ? H : T, (t & 1) ? T : H, n, ch, t, false, s);
    }, [] {}, launched, converged);
    // step t writes H for even t; after a step that changed nothing both
    // matrices hold the fixed point (H alone, if it was the first and A not T)
    if (*converged) *at = A ? H : T;
    else *at = (*launched & 1) ? H : T;
    return steps;
}

}  // namespace

void apsp_release_pools() {
    std::lock_guard<std::mutex> lk(g_pool_mu);
    for (auto& [dev, pool] : g_pools)
        if (pool) cudaMemPoolTrimTo(pool, 0);
}

void apsp_set_method(int method) {
    if (method < -1 || method > 1) invalid("method must be -1, 0 or 1");
    g_method.store(method);
}

int apsp_lengths(const float* A, float* H, int n, int max_path_length, cudaStream_t s) {
    if (n < 0 || max_path_length < 0) invalid("negative size or path length");
    const size_t nn = (size_t)n * n;
    if (max_path_length == 0 || n == 0) {
        NSG_CUDA(cudaMemcpyAsync(H, A, nn * sizeof(float), cudaMemcpyDeviceToDevice, s));
        return 0;
    }
    const Graph g(A, n, max_path_length >= n - 1, max_path_length, false, s);
    const bool sparse = g.sparse;
    DevMem T(sparse ? nn * sizeof(float) : 0, s);
    DevMem copy(sparse && !g.order && overlap(A, H, nn) ? nn * sizeof(float) : 0, s);
    const float* from = A;
    if (g.order) {  // the steps start from the relabelled matrix in T
        sparse_relabel(A, T.floats(), n, g.order, s);
        from = nullptr;
    } else if (copy.p) {
        NSG_CUDA(cudaMemcpyAsync(copy.p, A, nn * sizeof(float), cudaMemcpyDeviceToDevice, s));
        from = copy.floats();
    }
    auto deliver = [&](float* at) {  // into H, in the matrix's own labels
        if (g.order) {
            if (at == H) {
                at = T.floats();
                NSG_CUDA(cudaMemcpyAsync(at, H, nn * sizeof(float), cudaMemcpyDeviceToDevice, s));
            }
            sparse_restore(at, H, n, g.order, g.rank, s);
        } else if (at != H) {
            NSG_CUDA(cudaMemcpyAsync(H, at, nn * sizeof(float), cudaMemcpyDeviceToDevice, s));
        }
    };
    int launched = 0, first = 0;
    bool converged = false;
    float* at = nullptr;
    if (g.squaring) {
        // A symmetric: X = A^T = A; each product X <- X (x) X. A fixed point
        // that single steps find at step h (the hop diameter) is the one that
        // ceil(log2 h) products reach and one more confirms.
        first = g.first;
        if (first > 0) {
            const int h = sparse_steps(g, from, H, T.floats(), n, (1 << first) - 1, s, &launched, &converged, &at);
            deliver(at);
            if (converged) {
                NSG_CUDA(cudaStreamSynchronize(s));
                return ceil_log2(h) + 1;
            }
            A = H;  // A^(2^first)
        }
        Iterates it(A, n, s);
        // Exact sums: powers up to 2^t >= n - 1, then the product that changes
        // nothing. Rounded sums: once every shortest path is covered, a product
        // can still lower an entry by an ulp through another split of a path's
        // sum; those descents are bounded and short, and products that find
        // nothing to change return at once.
        const int cap = g.squaring == 1 ? ceil_log2(n) + 2 : ceil_log2(n) + 64;
        DevMem changed(sizeof(int) * cap, s);
        NSG_CUDA(cudaMemsetAsync(changed.p, 0, sizeof(int) * cap, s));
        int* ch = static_cast<int*>(changed.p);
        const int products = cap - first;
        for (int t = 0; t < products; ++t)
            launch_step(it.X[t & 1], it.X[t & 1], it.X[(t + 1) & 1], n, it.P, ch, t, s);
        launch_unpad(it.X[products & 1], H, n, it.P, s);
        std::vector<int> flags(products);
        NSG_CUDA(cudaMemcpyAsync(flags.data(), ch, sizeof(int) * products, cudaMemcpyDeviceToHost, s));
        NSG_CUDA(cudaStreamSynchronize(s));
        int q = 0;
        while (q < products && flags[q]) ++q;
        if (q == products) fail(NSG_ERR_CUDA, "shortest-path squaring did not converge");
        return first + q + 1;
    }
    if (sparse) {
        const int steps = sparse_steps(g, from, H, T.floats(), n, max_path_length, s, &launched,
                                       &converged, &at);
        deliver(at);
        NSG_CUDA(cudaStreamSynchronize(s));
        return steps;
    }
    Iterates it(A, n, s);
    DevMem changed(sizeof(int) * max_path_length, s);
    NSG_CUDA(cudaMemsetAsync(changed.p, 0, sizeof(int) * max_path_length, s));
    int* ch = static_cast<int*>(changed.p);
    // The result of t steps lives in X[t & 1]; when converged both buffers hold it.
    bool unpadded = false;
    auto unpad = [&](int t) {
        launch_unpad(it.X[t & 1], H, n, it.P, s);
        unpadded = true;
    };
    const int steps = run_steps(max_path_length, ch, s, [&](int t) {
        launch_step(it.Ap, it.X[t & 1], it.X[(t + 1) & 1], n, it.P, ch, t, s);
    }, [&] { unpad(max_path_length); }, &launched, &converged);
    if (!unpadded) {
        unpad(launched);
        NSG_CUDA(cudaStreamSynchronize(s));
    }
    return steps;
}

void apsp_paths(const float* A, float* H, int* paths, int n, int L, float tolerance,
                cudaStream_t s) {
    if (n < 0 || L < 1) invalid("paths need n >= 0 and maxPathLength >= 1");
    const size_t nn = (size_t)n * n;
    NSG_CUDA(cudaMemsetAsync(paths, 0xff, sizeof(int) * nn * L, s));  // -1
    if (n == 0) return;
    const Graph g(A, n, false, L, true, s);
    DevMem snaps(nn * (L + 1) * sizeof(float), s);  // H before each step, and after the last
    DevMem changed(sizeof(int) * L, s);
    NSG_CUDA(cudaMemsetAsync(changed.p, 0, sizeof(int) * L, s));
    float* Hi = static_cast<float*>(snaps.p);
    int* ch = static_cast<int*>(changed.p);
    float* last = Hi + nn * L;
    if (g.sparse) {
        NSG_CUDA(cudaMemcpyAsync(Hi, A, nn * sizeof(float), cudaMemcpyDeviceToDevice, s));
        for (int p = 0; p < L; ++p) sparse_step(g.rows, Hi + nn * p, Hi + nn * (p + 1), n, ch, p, true, s);
        SellView cols = g.rows;
        DevMem words(0, s), edges(0, s);
        DevMem At(0, s);
        if (!g.symmetric) {
            // the columns of A as rows of its transpose
            const int P = (n + kPad - 1) / kPad * kPad;
            At.alloc(sizeof(float) * (size_t)P * P, s);
            float* at = static_cast<float*>(At.p);
            launch_pad(A, at, n, P, true, s);
            words.alloc(sizeof(GraphInfo) + sizeof(int) * (2 * (size_t)n + 2), s);
            GraphInfo* info = static_cast<GraphInfo*>(words.p);
            int* counts = reinterpret_cast<int*>(info + 1);
            sparse_count(at, P, n, info, counts, counts + n, s);
            GraphInfo h{};
            NSG_CUDA(cudaMemcpyAsync(&h, info, sizeof(h), cudaMemcpyDeviceToHost, s));
            NSG_CUDA(cudaStreamSynchronize(s));
            edges.alloc(sizeof(int2) * kSellRows * (size_t)std::max(1, h.width), s);
            sparse_fill(at, P, n, counts + n, static_cast<int2*>(edges.p), s);
            cols = {static_cast<const int2*>(edges.p), counts + n, sell_slices(n)};
        }
        sparse_walk(cols, last, Hi, paths, tolerance, n, L, s);
        NSG_CUDA(cudaMemcpyAsync(H, last, nn * sizeof(float), cudaMemcpyDeviceToDevice, s));
        NSG_CUDA(cudaStreamSynchronize(s));
        return;
    }
    Iterates it(A, n, s);
    for (int p = 0; p < L; ++p) {
        launch_unpad(it.X[p & 1], Hi + nn * p, n, it.P, s);  // H before step p
        launch_step(it.Ap, it.X[p & 1], it.X[(p + 1) & 1], n, it.P, ch, p, s);
    }
    launch_unpad(it.X[L & 1], last, n, it.P, s);
    dim3 block(32, 8);
    dim3 grid((n + 31) / 32, (n + 7) / 8);
    hedetniemi_walk_kernel<<<grid, block, 0, s>>>(last, Hi, A, paths, tolerance, n, L);
    NSG_CUDA(cudaGetLastError());
    NSG_CUDA(cudaMemcpyAsync(H, last, nn * sizeof(float), cudaMemcpyDeviceToDevice, s));
    NSG_CUDA(cudaStreamSynchronize(s));
}

void corr_to_adjacency(const float* C, float* A, int n, int mode, cudaStream_t s) {
    if (n <= 0) return;
    const size_t nn = (size_t)n * n;
    const int threads = 256;
    corr_to_adj_kernel<<<static_cast<unsigned>((nn + threads - 1) / threads), threads, 0, s>>>(
        C, A, n, mode);
    NSG_CUDA(cudaGetLastError());
}

}  // namespace nsg
