// Tie resolution for the KSG count kernel.
//
// A sample whose k-th and (k+1)-th nearest joint distances are equal (and
// non-zero) has a neighbour set that the reference CPU path picks by the
// order its std::sort leaves equal distances in
// (netcalc/src/mutual_information_cpu.cpp:48-77). The search kernels append
// such samples to a list, unless every frame at the tied distance has the same
// marginal pair (then any order gives the same eps); the kernels here take the
// list one sample at a time, a CTA each while the row fits in shared memory, a
// warp each beyond:
//
//   1. the sample's full joint-distance row (the reference's arithmetic) and
//      the identity index array;
//   2. the reference sort's order replayed on the prefix that holds the
//      neighbours (the steps sort_prefix.h restates, each partition's stoppers
//      found all at once, or 32 at a time with ballots);
//   3. eps_a / eps_b over sorted positions 1..k;
//   4. the marginal counts again over all frames, and the sample's psi term.
//
// Runs between the count kernel and the finalize kernel, with a fixed grid
// that walks the tie list through an atomic counter (an empty list costs one
// launch that returns at once).
#include <algorithm>

#include "common.cuh"
#include "engine.h"
#include "ksg.cuh"
#include "sort_prefix.h"

namespace nsg {
namespace {

constexpr int kWarpsPerCta = 8;
constexpr int kCtasPerSm = 6;  // latency-bound: 48 warps per SM (40 registers) replays about 6% faster than 32
constexpr int kStack = 64;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ int tie_frame(const int* __restrict__ fmap, int s, int ld, int* fault) {
    if (!fmap) return s;
    const int f = __ldg(fmap + s);
    if (f < 0 || f >= ld) {
        atomicOr(fault, FAULT_BAD_INDEX);
        return 0;
    }
    return f;
}

template <int D>
__device__ __forceinline__ float tie_marginal(const float (&q)[D], const float* __restrict__ x,
                                              int ld, int src) {
    float v = fabsf(q[0] - __ldg(x + src));
#pragma unroll
    for (int c = 1; c < D; ++c) v = fmaxf(v, fabsf(q[c] - __ldg(x + (size_t)c * ld + src)));
    return v;
}

// sort_prefix_like_reference (sort_prefix.h) run by a whole warp: the same
// segments, pivots and swaps, with each unguarded partition found 32
// positions at a time. The partition of [first+1, last) around pk swaps the
// t-th element from the left that is not below pk (a left stopper) with the
// t-th element from the right that is not above pk (a right stopper, the
// scan may reach the pivot itself at `first`) while the former lies left of
// the latter; the elements between them are untouched until then, so the
// stoppers can be read from the array as it was. The cut is the first left
// stopper past the last swap, or that swap's right position if it comes
// first. The pairs found by one round of ballots touch distinct positions,
// so lane t swaps the round's t-th pair, all at once. Lane 0 holds the
// segment stack; all lanes load and vote. A segment whose depth budget runs
// out is heapsorted by lane 0 (heap_sort_like_reference). Same result as the
// serial routine, element for element.
// ranked: 64 bytes of shared memory of the warp's own.
__device__ bool sort_prefix_warp(const float* key, int* idx, int n, int T, SortSegment* stack,
                                 int cap, unsigned char* ranked, int lane) {
    if (n <= 1) return true;
    constexpr int kThreshold = 16;
    int top = 0;
    if (lane == 0) stack[0] = {0, n, 2 * floor_log2(n)};
    top = 1;
    int prefix_end = 0;
    while (top > 0) {
        --top;
        SortSegment sg{};
        if (lane == 0) sg = stack[top];
        int first = __shfl_sync(kFull, sg.first, 0);
        int last = __shfl_sync(kFull, sg.last, 0);
        int depth = __shfl_sync(kFull, sg.depth, 0);
        while (last - first > kThreshold) {
            if (depth == 0) {
                if (lane == 0) heap_sort_like_reference(key, idx + first, last - first);
                __syncwarp();
                break;
            }
            --depth;
            // median of three moved to `first` (lane 0)
            if (lane == 0) {
                const int a = first + 1, b = first + (last - first) / 2, c = last - 1;
                const float ka = key[idx[a]], kb = key[idx[b]], kc = key[idx[c]];
                int pick;
                if (ka < kb) {
                    if (kb < kc) pick = b;
                    else if (ka < kc) pick = c;
                    else pick = a;
                } else if (ka < kc) {
                    pick = a;
                } else if (kb < kc) {
                    pick = c;
                } else {
                    pick = b;
                }
                const int t = idx[first];
                idx[first] = idx[pick];
                idx[pick] = t;
            }
            __syncwarp();
            const float pk = key[idx[first]];
            // left stoppers from first+1 up, right stoppers from last-1 down
            int lbase = first + 1, rbase = last - 1;  // next chunk starts
            int lchunk = 0, rchunk = 0;               // current chunk starts
            unsigned lmask = 0, rmask = 0;
            bool lend = false, rend = false;
            int prev_r = -1;                          // right position of the last swap
            int cut;
            for (;;) {
                while (lmask == 0 && !lend) {
                    if (lbase >= last) {
                        lend = true;
                        break;
                    }
                    const int p = lbase + lane;
                    const bool st = p < last && !(key[idx[p]] < pk);
                    lmask = __ballot_sync(kFull, st);
                    lchunk = lbase;
                    lbase += 32;
                }
                while (rmask == 0 && !rend) {
                    if (rbase < first) {
                        rend = true;
                        break;
                    }
                    const int p = rbase - lane;
                    const bool st = p >= first && !(pk < key[idx[p]]);
                    rmask = __ballot_sync(kFull, st);
                    rchunk = rbase;
                    rbase -= 32;
                }
                // the median of three leaves stoppers on both sides; running
                // out of either means a broken invariant, reported as failure
                if (rend) return false;
                // the t-th left stopper of lmask pairs with the t-th right
                // stopper of rmask while it lies left of it; those pairs form
                // a prefix of t and are swapped together, lane t taking pair t
                const int npair = lend ? 0 : min(__popc(lmask), __popc(rmask));
                // (each stopper's lane writes itself down at its rank)
                const unsigned before = (1u << lane) - 1u;
                if (lmask >> lane & 1u) ranked[__popc(lmask & before)] = static_cast<unsigned char>(lane);
                if (rmask >> lane & 1u) ranked[32 + __popc(rmask & before)] = static_cast<unsigned char>(lane);
                __syncwarp();
                int lp = 0x7fffffff, rp = -1;
                if (lane < npair) {
                    lp = lchunk + ranked[lane];
                    rp = rchunk - ranked[32 + lane];
                }
                const bool swap = lane < npair && lp < rp;
                const int c = __popc(__ballot_sync(kFull, swap));
                const int llast = c ? ranked[c - 1] : 0, rlast = c ? ranked[32 + c - 1] : 0;
                if (swap) {
                    const int t = idx[lp];
                    idx[lp] = idx[rp];
                    idx[rp] = t;
                }
                __syncwarp();
                if (c > 0) prev_r = __shfl_sync(kFull, rp, c - 1);
                if (c == npair && !lend) {
                    // every pair of the round swapped: drop them, continue
                    lmask &= kFull << llast << 1;
                    rmask &= kFull << rlast << 1;
                    continue;
                }
                // pair c crosses (or no left stopper is left)
                const int lpos = lend ? 0x7fffffff : __shfl_sync(kFull, lp, c);
                cut = prev_r < 0 ? lpos : min(lpos, prev_r);
                break;
            }
            __syncwarp();
            if (cut >= last) return false;
            if (cut < T) {
                if (top >= cap) return false;
                if (lane == 0) stack[top] = {cut, last, depth};
                ++top;
            }
            last = cut;
        }
        if (first < T && last > prefix_end) prefix_end = last;
    }
    __syncwarp();
    // The insertion sort of [0, prefix_end), a few dozen elements, is a stable
    // sort: an element's place is the number of smaller keys plus the equal
    // ones before it. Longer prefixes (heapsorted segments among them) are left
    // to lane 0, and so are those with a NaN, which no key is smaller than and
    // none larger: where it ends up follows from the sort's steps alone.
    int v[2] = {0, 0};
    float kv[2] = {0.f, 0.f};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int i = 32 * h + lane;
        if (i < prefix_end) {
            v[h] = idx[i];
            kv[h] = key[v[h]];
        }
    }
    const bool odd = __any_sync(kFull, kv[0] != kv[0] || kv[1] != kv[1]);
    if (prefix_end <= 64 && !odd) {
        int place[2] = {0, 0};
        for (int j = 0; j < prefix_end; ++j) {
            const float kj = __shfl_sync(kFull, j < 32 ? kv[0] : kv[1], j & 31);
#pragma unroll
            for (int h = 0; h < 2; ++h) place[h] += kj < kv[h] || (kj == kv[h] && j < 32 * h + lane);
        }
        __syncwarp();
#pragma unroll
        for (int h = 0; h < 2; ++h)
            if (32 * h + lane < prefix_end) idx[place[h]] = v[h];
    } else if (lane == 0) {
        for (int i = 1; i < prefix_end; ++i) {
            const int moved = idx[i];
            const float km = key[moved];
            int j = i;
            while (j > 0 && km < key[idx[j - 1]]) {
                idx[j] = idx[j - 1];
                --j;
            }
            idx[j] = moved;
        }
    }
    __syncwarp();
    return true;
}

// Longest row whose distances, order and partition lists fit in shared memory
// (10.5 bytes a frame); longer ones keep a warp per sample.
constexpr int kSmemRow = 20480;
constexpr int kTieThreads = 512;  // most per CTA

__host__ __device__ constexpr int tie_chunks(int m) { return (m + 31) / 32; }
__host__ __device__ constexpr int tie_list(int m) { return (m / 2 + 2 + 7) & ~7; }  // entries of one list
constexpr int tie_smem(int m) { return 8 * ((m + 3) & ~3) + 2 * 2 * tie_list(m) + 16 * tie_chunks(m); }

// What the CTA of one sample shares beside its rows.
struct TieShared {
    SortSegment stack[kStack];
    int item, nl, nr, swaps, ca, cb;
};

// sort_prefix_like_reference (sort_prefix.h) run by a CTA: the same segments,
// pivots and swaps. The partition of [first+1, last) around pk swaps the t-th
// element from the left that is not below pk (a left stopper) with the t-th
// element from the right that is not above pk (a right stopper, the scan may
// reach the pivot itself at `first`) while the former lies left of the latter;
// the elements between them are untouched until then, so all stoppers can be
// read from the array as it was. The cut is the first left stopper past the
// last swap, or that swap's right position if it comes first. Per partition:
// the stoppers' masks, 32 positions a word; their prefix counts from either
// side; the positions by rank (pairs that swap lie within the first half of
// the ranks); all swaps. A segment whose depth budget runs out is heapsorted
// by thread 0 (heap_sort_like_reference). Same result as the serial routine,
// element for element.
__device__ bool sort_prefix_cta(const float* key, int* idx, int n, int T, TieShared& sh, unsigned short* left,
                                unsigned short* right, unsigned* words) {
    if (n <= 1) return true;
    constexpr int kThreshold = 16;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nthreads = blockDim.x, nwarps = nthreads >> 5;  // two warps at least: one counts from each side
    unsigned* lm = words;
    unsigned* rm = lm + tie_chunks(n);
    int* lp = reinterpret_cast<int*>(rm + tie_chunks(n));
    int* rp = lp + tie_chunks(n);
    if (tid == 0) sh.stack[0] = {0, n, 2 * floor_log2(n)};
    int top = 1;
    int prefix_end = 0;
    while (top > 0) {
        --top;
        __syncthreads();
        const SortSegment sg = sh.stack[top];
        const int first = sg.first;
        int last = sg.last, depth = sg.depth;
        while (last - first > kThreshold) {
            if (depth == 0) {
                if (tid == 0) heap_sort_like_reference(key, idx + first, last - first);
                __syncthreads();
                break;
            }
            --depth;
            // median of three moved to `first`
            if (tid == 0) {
                const int a = first + 1, b = first + (last - first) / 2, c = last - 1;
                const float ka = key[idx[a]], kb = key[idx[b]], kc = key[idx[c]];
                int pick;
                if (ka < kb) {
                    if (kb < kc) pick = b;
                    else if (ka < kc) pick = c;
                    else pick = a;
                } else if (ka < kc) {
                    pick = a;
                } else if (kb < kc) {
                    pick = c;
                } else {
                    pick = b;
                }
                const int t = idx[first];
                idx[first] = idx[pick];
                idx[pick] = t;
            }
            __syncthreads();
            const float pk = key[idx[first]];
            const int len = last - first, nc = tie_chunks(len), half = len / 2;
#pragma unroll 4
            for (int w = wid; w < nc; w += nwarps) {
                const int i = 32 * w + lane;
                const float kv = i < len ? key[idx[first + i]] : 0.f;
                const unsigned ml = __ballot_sync(kFull, i > 0 && i < len && !(kv < pk));
                const unsigned mr = __ballot_sync(kFull, i < len && !(pk < kv));
                if (lane == 0) {
                    lm[w] = ml;
                    rm[w] = mr;
                }
            }
            __syncthreads();
            if (wid < 2) {  // warp 0 from the left, warp 1 from the right
                int run = 0;
                for (int w0 = 0; w0 < nc; w0 += 32) {
                    const int w = wid == 0 ? w0 + lane : nc - 1 - (w0 + lane);
                    const bool in = w0 + lane < nc;
                    const int v = in ? __popc(wid == 0 ? lm[w] : rm[w]) : 0;
                    int x = v;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int y = __shfl_up_sync(kFull, x, o);
                        if (lane >= o) x += y;
                    }
                    if (in) (wid == 0 ? lp : rp)[w] = run + x - v;
                    run += __shfl_sync(kFull, x, 31);
                }
                if (lane == 0) (wid == 0 ? sh.nl : sh.nr) = run;
                if (tid == 0) sh.swaps = 0;
            }
            __syncthreads();
            for (int w = wid; w < nc; w += nwarps) {
                const unsigned ml = lm[w], mr = rm[w];
                const int rl = lp[w] + __popc(ml & ((1u << lane) - 1u));
                const int rr = rp[w] + __popc(mr & ~(kFull >> (31 - lane)));
                if ((ml >> lane & 1u) && rl <= half) left[rl] = static_cast<unsigned short>(32 * w + lane);
                if ((mr >> lane & 1u) && rr <= half) right[rr] = static_cast<unsigned short>(32 * w + lane);
            }
            __syncthreads();
            const int nl = sh.nl, nr = sh.nr, np = min(min(nl, nr), half + 1);
            for (int t = tid; t < np; t += nthreads) {
                const int l = left[t], r = right[t];
                if (l >= r) break;
                const int u = idx[first + l];
                idx[first + l] = idx[first + r];
                idx[first + r] = u;
                if (t + 1 == np || left[t + 1] >= right[t + 1]) sh.swaps = t + 1;
            }
            __syncthreads();
            const int c = sh.swaps;
            // the median of three leaves stoppers on both sides; running out of
            // either means a broken invariant, reported as failure
            if (nr <= c) return false;
            const int lpos = c < nl ? first + left[c] : 0x7fffffff;
            const int cut = c > 0 ? min(lpos, first + right[c - 1]) : lpos;
            if (cut >= last) return false;
            if (cut < T) {
                if (top >= kStack) return false;
                if (tid == 0) sh.stack[top] = {cut, last, depth};
                ++top;
            }
            last = cut;
        }
        if (first < T && last > prefix_end) prefix_end = last;
    }
    // The insertion sort of [0, prefix_end), a few dozen elements, is a stable
    // sort: an element's place is the number of smaller keys plus the equal
    // ones before it. Longer prefixes (heapsorted segments among them) are left
    // to thread 0, and so are those with a NaN (sort_prefix_warp). All swaps lie
    // before the last barrier.
    int v = 0;
    float kv = 0.f;
    if (tid < prefix_end) {
        v = idx[tid];
        kv = key[v];
    }
    const bool odd = __syncthreads_or(kv != kv);
    if (prefix_end <= nthreads && !odd) {
        int place = 0;
        if (tid < prefix_end) {
#pragma unroll 4
            for (int j = 0; j < prefix_end; ++j) {
                const float kj = key[idx[j]];
                place += kj < kv || (kj == kv && j < tid);
            }
        }
        __syncthreads();
        if (tid < prefix_end) idx[place] = v;
    } else if (tid == 0) {
        for (int i = 1; i < prefix_end; ++i) {
            const int moved = idx[i];
            const float km = key[moved];
            int j = i;
            while (j > 0 && km < key[idx[j - 1]]) {
                idx[j] = idx[j - 1];
                --j;
            }
            idx[j] = moved;
        }
    }
    __syncthreads();
    return true;
}

// A tied sample of pair P: its coordinates, and joint and marginal distances.
template <int D>
struct TieSample {
    const float* __restrict__ xa;
    const float* __restrict__ xb;
    const int* __restrict__ fmap;
    int ld;
    int* fault;
    float qa[D], qb[D];
    __device__ __forceinline__ TieSample(const KsgPairDesc& P, int q, int* f)
        : xa(P.xa), xb(P.xb), fmap(P.fmap), ld(P.ld), fault(f) {
        const int s = tie_frame(fmap, q, ld, fault);
#pragma unroll
        for (int c = 0; c < D; ++c) {
            qa[c] = __ldg(xa + (size_t)c * ld + s);
            qb[c] = __ldg(xb + (size_t)c * ld + s);
        }
    }
    __device__ __forceinline__ void marginals(int j, float& a, float& b) const {
        const int s = tie_frame(fmap, j, ld, fault);
        a = tie_marginal<D>(qa, xa, ld, s);
        b = tie_marginal<D>(qb, xb, ld, s);
    }
    // eps over sorted positions 1..k (k can exceed a warp's 31 lanes), in every lane
    __device__ __forceinline__ void eps(const int* idx, int k, float& ea, float& eb) const {
        const int lane = threadIdx.x & 31;
        ea = eb = 0.f;
        for (int p = 1 + lane; p <= k; p += 32) {
            float a, b;
            marginals(idx[p], a, b);
            ea = fmaxf(ea, a);
            eb = fmaxf(eb, b);
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            ea = fmaxf(ea, __shfl_xor_sync(kFull, ea, off));
            eb = fmaxf(eb, __shfl_xor_sync(kFull, eb, off));
        }
    }
};

// Results of a sample from its counts (self included); one thread.
__device__ __forceinline__ void write_tie(const KsgTieArgs& A, long long o, int m, int ca, int cb, float ea, float eb) {
    const int nx = min(max(ca - 1, 0), m);
    const int ny = min(max(cb - 1, 0), m);
    A.psum[o] = __fadd_rn(__ldg(A.psi + nx), __ldg(A.psi + ny));
    if (A.nx) A.nx[o] = nx;
    if (A.ny) A.ny[o] = ny;
    if (A.eps_x) A.eps_x[o] = ea;
    if (A.eps_y) A.eps_y[o] = eb;
}

// Rows too long for shared memory: a warp per sample, dz and idx in global memory.
template <int D>
__global__ void __launch_bounds__(kWarpsPerCta * 32, kCtasPerSm) ksg_tie_kernel(KsgTieArgs A) {
    __shared__ SortSegment s_stack[kWarpsPerCta][kStack];
    __shared__ unsigned char s_ranked[kWarpsPerCta][64];
    const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    float* dz = A.dz + warp * A.stride;
    int* idx = A.idx + warp * A.stride;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int total = min(*A.tie_count, A.tie_cap);
    for (;;) {
        int e = 0;
        if (lane == 0) e = atomicAdd(A.tie_next, 1);
        e = __shfl_sync(kFull, e, 0);
        if (e >= total) return;
        const KsgTie t = A.ties[e];
        const KsgPairDesc P = A.pairs[t.pair];
        const int m = P.m;
        if (m > A.stride) {  // the planner sizes rows for every pair
            if (lane == 0) atomicOr(A.fault, FAULT_BAD_INDEX);
            continue;
        }
        const TieSample<D> S(P, t.q, A.fault);
        for (int j = lane; j < m; j += 32) {
            float a, b;
            S.marginals(j, a, b);
            dz[j] = fmaxf(a, b);
            idx[j] = j;
        }
        __syncwarp();
        const bool ok = sort_prefix_warp(dz, idx, m, A.k + 1, s_stack[wid], kStack, s_ranked[wid], lane);
        __syncwarp();
        if (!ok) {
            if (lane == 0) atomicOr(A.fault, FAULT_TIE_UNRESOLVED);
            continue;
        }
        float ea, eb;
        S.eps(idx, A.k, ea, eb);
        int ca = 0, cb = 0;
        for (int j = lane; j < m; j += 32) {
            float a, b;
            S.marginals(j, a, b);
            ca += a <= ea;
            cb += b <= eb;
        }
        ca = __reduce_add_sync(kFull, ca);
        cb = __reduce_add_sync(kFull, cb);
        if (lane == 0) write_tie(A, P.scratch + t.q, m, ca, cb, ea, eb);
        __syncwarp();
    }
}

// A CTA per sample, rows in shared memory. Few samples tie and a replay is a
// chain of partitions, so its latency counts. From a warp per sample that
// finds 32 stoppers a round (rows in shared memory up to m = 3400): ties of a
// 56-node list at m = 1000 49 -> 25 us, of 101 nodes 156 -> 43 us, of
// 8,192 pairs at m = 10000 (8,559 samples) 3.19 -> 1.21 ms, of two resamples
// of 100 nodes 2.70 -> 0.33 ms.
template <int D>
__global__ void __launch_bounds__(kTieThreads) ksg_tie_smem_kernel(KsgTieArgs A) {
    extern __shared__ __align__(16) float s_rows[];
    __shared__ TieShared sh;
    const int padded = (A.stride + 3) & ~3, tid = threadIdx.x;
    float* dz = s_rows;
    int* idx = reinterpret_cast<int*>(dz + padded);
    unsigned* words = reinterpret_cast<unsigned*>(idx + padded);
    unsigned short* left = reinterpret_cast<unsigned short*>(words + 4 * tie_chunks(A.stride));
    unsigned short* right = left + tie_list(A.stride);
    const int total = min(*A.tie_count, A.tie_cap);
    for (;;) {
        if (tid == 0) {
            sh.item = atomicAdd(A.tie_next, 1);
            sh.ca = sh.cb = 0;
        }
        __syncthreads();
        const int e = sh.item;
        if (e >= total) return;
        const KsgTie t = A.ties[e];
        const KsgPairDesc P = A.pairs[t.pair];
        const int m = P.m;
        bool ok = m <= A.stride;  // the planner sizes rows for every pair
        if (!ok && tid == 0) atomicOr(A.fault, FAULT_BAD_INDEX);
        if (ok) {
            const TieSample<D> S(P, t.q, A.fault);
#pragma unroll 8
            for (int j = tid; j < m; j += blockDim.x) {
                float a, b;
                S.marginals(j, a, b);
                dz[j] = fmaxf(a, b);
                idx[j] = j;
            }
            __syncthreads();
            ok = sort_prefix_cta(dz, idx, m, A.k + 1, sh, left, right, words);
            if (!ok && tid == 0) atomicOr(A.fault, FAULT_TIE_UNRESOLVED);
            if (ok) {
                float ea, eb;
                S.eps(idx, A.k, ea, eb);
                int ca = 0, cb = 0;
#pragma unroll 8
                for (int j = tid; j < m; j += blockDim.x) {
                    float a, b;
                    S.marginals(j, a, b);
                    ca += a <= ea;
                    cb += b <= eb;
                }
                ca = __reduce_add_sync(kFull, ca);
                cb = __reduce_add_sync(kFull, cb);
                if ((tid & 31) == 0) {
                    atomicAdd(&sh.ca, ca);
                    atomicAdd(&sh.cb, cb);
                }
                __syncthreads();
                if (tid == 0) write_tie(A, P.scratch + t.q, m, sh.ca, sh.cb, ea, eb);
            }
        }
        __syncthreads();
    }
}

template <int D>
void launch_ties(const KsgTieArgs& a, long long samples, cudaStream_t st) {
    // at most a warp per eight samples: the list is short, and empty CTAs are
    // what the kernel costs on small plans (8 us for a pair)
    auto ctas = [&](int warps, int per_sm) {
        const long long most = (samples + 8 * warps - 1) / (8 * warps);
        return static_cast<int>(std::min<long long>(sm_count() * per_sm, std::max<long long>(most, 1)));
    };
    if (a.stride <= kSmemRow) {
        const int smem = tie_smem(a.stride);
        // set on every launch: the attribute belongs to the current device. One
        // value for all plans: another thread may set it before this launch.
        NSG_CUDA(cudaFuncSetAttribute(ksg_tie_smem_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      tie_smem(kSmemRow)));
        // as many CTAs as fit, with about 1024 threads per SM in all (m = 10000,
        // two CTAs: 2.40 ms with 128 threads each, 1.21 with 512)
        const int per_sm = std::max(1, std::min(12, (220 << 10) / (smem + 2048)));
        const int threads = per_sm >= 8 ? 128 : per_sm >= 4 ? 256 : kTieThreads;
        ksg_tie_smem_kernel<D><<<ctas(threads / 32, per_sm), threads, smem, st>>>(a);
    } else {
        ksg_tie_kernel<D><<<ctas(kWarpsPerCta, kCtasPerSm), kWarpsPerCta * 32, 0, st>>>(a);
    }
    NSG_CUDA(cudaGetLastError());
}

}  // namespace

bool ksg_ties_in_smem(int m) { return m <= kSmemRow; }

int ksg_tie_warps() { return sm_count() * kCtasPerSm * kWarpsPerCta; }

void ksg_launch_ties(const KsgTieArgs& a, int d, long long samples, cudaStream_t st) {
    switch (d) {
        case 1: launch_ties<1>(a, samples, st); break;
        case 2: launch_ties<2>(a, samples, st); break;
        case 3: launch_ties<3>(a, samples, st); break;
        default: fail(NSG_ERR_INVALID, "d must be 1, 2 or 3");
    }
}

// The kernel over global rows on a caller-chosen number of CTAs (the caller's scratch
// holds kWarpsPerCta * ctas rows).
void ksg_launch_ties_ctas(const KsgTieArgs& a, int d, int ctas, cudaStream_t st) {
    const int threads = kWarpsPerCta * 32;
    switch (d) {
        case 1: ksg_tie_kernel<1><<<ctas, threads, 0, st>>>(a); break;
        case 2: ksg_tie_kernel<2><<<ctas, threads, 0, st>>>(a); break;
        case 3: ksg_tie_kernel<3><<<ctas, threads, 0, st>>>(a); break;
        default: fail(NSG_ERR_INVALID, "d must be 1, 2 or 3");
    }
    NSG_CUDA(cudaGetLastError());
}

}  // namespace nsg
