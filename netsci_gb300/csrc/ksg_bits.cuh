// KSG joint search on rank bitmaps: the same results as the other searches,
// one warp per query, 32 frames per logic instruction.
//
// Every frame a query accepts lies within U (its k-th distance) of it in
// each of the 2d coordinates. Each node splits every coordinate's range at
// kBitBins - 1 quantile edges; for a pair, row t of a coordinate is the
// bitmap of the frames whose bin is below t. The frames that may lie within h
// of the query in that coordinate are then row[hi + 1] ^ row[lo], with lo and
// hi the first and last bin the interval can reach (exact: rounding is
// monotone, see ksg_grid.cuh), and the AND over the coordinates leaves the few
// frames that can lie within h in all of them: at m = 10000, d = 3, about 12
// for h = U and 25 for the h used. Only those are evaluated.
//
//   * Rows of a pair live in shared memory, over the frames in the order of
//     node a's bins of its widest coordinate, so that coordinate needs no
//     rows: its interval is a range of words (a third of them, typically).
//     One CTA owns one pair at a time (or a share of its queries) and builds
//     the rows with ballots: 2% of its time at m = 10000.
//   * A warp takes a few queries at a time: one lane per query and
//     coordinate finds the bins its interval reaches. Then, query by query,
//     each lane ANDs one to eight words of 2d - 1 row pairs, finds the set
//     bit of its rank, and evaluates that frame exactly (one 16-byte gather
//     per node); the frames within h are listed in shared memory with their
//     distances. A lane per listed frame counts the smaller distances;
//     the frames with at most k smaller ones are the query and its k nearest
//     (and whatever ties with the k-th), and warp reductions over them give
//     the k-th distance, eps and the tie test.
//   * h comes from the two nodes' scale estimates: sqrt(est_a est_b) follows
//     the k-th joint distance with a spread of 8 to 14%. Each warp scales it
//     so that about one query in fifteen finds fewer than k frames within h and
//     tries again with a larger h; whatever h is, the accepted set is complete
//     (every frame within h was evaluated, and at least k others were). Where
//     the frames fill fewer dimensions than the nodes have coordinates (nodes
//     that depend on each other, drift, long tails) the estimates are off by
//     factors: a neighbour far inside a crowded radius moves the scale by a
//     tenth, and radii that still miss or crowd change faster look by look.
//   * A full list of frames within h gives a smaller h, its own k-th distance.
//     Queries that do not settle (heavy ties, coordinates that are not finite)
//     scan all frames (scan_all), up to k + 1 of them at distance 0.
//
// Ties come out exactly: all frames at the k-th distance are among those
// evaluated. What bounds the kernel: 635 instructions per query at m = 10000,
// about 0.76 of the issue slots with the one CTA of 1024 threads that the rows
// leave room for, and about 110 shared-memory wavefronts beside the gathers.
// 8192 pairs at m = 10000: 54.1 ms, against 175 ms for the cell-grid scan, which
// spent about 2000 instructions per query.
#pragma once

#include "common.cuh"
#include "ksg.cuh"
#include "ksg_bits.h"
#include "ksg_grid.h"

namespace nsg {
namespace bitk {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float inf_f() { return __int_as_float(0x7f800000); }

template <int D>
__device__ __forceinline__ float dist(const float (&q)[D], const float (&x)[D]) {
    if constexpr (D == 1) return fabsf(q[0] - x[0]);
    else if constexpr (D == 2) return fmaxf(fabsf(q[0] - x[0]), fabsf(q[1] - x[1]));
    else return nsg_max3(fabsf(q[0] - x[0]), fabsf(q[1] - x[1]), fabsf(q[2] - x[2]));
}

// Frame j of a node's coordinates as stored by the node kernel (1, 2 or 4
// floats per frame).
template <int D>
__device__ __forceinline__ void load_frame(const float* __restrict__ aos, int j, float (&x)[D]) {
    if constexpr (D == 1) {
        x[0] = __ldg(aos + j);
    } else if constexpr (D == 2) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(aos) + j);
        x[0] = v.x;
        x[1] = v.y;
    } else {
        const float4 v = __ldg(reinterpret_cast<const float4*>(aos) + j);
        x[0] = v.x;
        x[1] = v.y;
        x[2] = v.z;
    }
}

struct Found {
    float ea, eb, wk;
    bool tie;  // frames at wk with different marginals: the reference's order decides
};

// The first part of [q - h, q + h] and one past its last among the parts
// that 63 ascending edges e (padded with +inf) cut an axis into. With an
// infinite h, hi passes the last part: such bins are never used.
__device__ __forceinline__ void reach(const float* e, float q, float h, int& lo, int& hi) {
    lo = hi = 0;
#pragma unroll
    for (int s = 32; s > 0; s >>= 1) {
        if (__fsub_rn(q, e[lo + s - 1]) > h) lo += s;
        if (__fsub_rn(e[hi + s - 1], q) <= h) hi += s;
    }
    ++hi;
}

// Inclusive prefix sum over the lanes.
__device__ __forceinline__ int lane_prefix(int v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b32 t;\n\t"
            "shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff;\n\t"
            "@p add.s32 %0, %0, t;\n\t}"
            : "+r"(v)
            : "r"(o));
    }
    return v;
}

// W words at a byte offset (a multiple of 4 W).
template <int W>
__device__ __forceinline__ void load_words(const unsigned* rows, unsigned at, unsigned (&w)[W]) {
    const char* p = reinterpret_cast<const char*>(rows) + at;
    if constexpr (W == 1) {
        w[0] = *reinterpret_cast<const unsigned*>(p);
    } else if constexpr (W == 2) {
        const uint2 v = *reinterpret_cast<const uint2*>(p);
        w[0] = v.x;
        w[1] = v.y;
    } else {
        const uint4 v = *reinterpret_cast<const uint4*>(p);
        w[0] = v.x;
        w[1] = v.y;
        w[2] = v.z;
        w[3] = v.w;
    }
}

// Position of the bit of rank win + lane among the set bits of the lanes'
// words (lane order, then word order): word g of lane l covers positions
// base + l span + 32 g for g < 4 and 4096 - 128 more above. off: set bits of
// the lanes before; cnt: of this lane; n: of all; table: 32 words of shared memory.
// Lanes whose rank does not exist get an arbitrary position.
template <int W>
__device__ __forceinline__ int bit_of_rank(const unsigned (&w)[W], int base, int span, int off, int cnt, int win, int n, int lane,
                                           unsigned* table) {
    // lanes with a bit in the window, in order, and where their bits start in it
    const int first = off - win;
    const bool here = cnt > 0 && first < 32 && first + cnt > 0;
    const unsigned owners = __ballot_sync(kFull, here);
    const unsigned starts = __reduce_or_sync(kFull, here ? 1u << max(first, 0) : 0u);
    if (here) table[__popc(owners & ((1u << lane) - 1u))] = static_cast<unsigned>(lane);
    __syncwarp();
    const int src = static_cast<int>(table[__popc(starts & (kFull >> (31 - lane))) - 1] & 31u);
    int r = win + lane - __shfl_sync(kFull, off, src);  // rank within the owner's words
    if (win + lane >= n) r = 0;
    int pos = base + span * src;
    unsigned bits = __shfl_sync(kFull, w[0], src);
#pragma unroll
    for (int g = 1; g < W; ++g) {
        // past the words before: the remaining rank moves on to word g
        const unsigned x = __shfl_sync(kFull, w[g], src);
        const int c = __popc(bits);
        if (r >= c) {
            r -= c;
            bits = x;
            pos += g == 4 ? 4096 - 96 : 32;
        } else {
            r -= 0x10000;  // found: no later word is taken
        }
    }
    r &= 0xffff;
    for (; r > 0; --r) bits &= bits - 1;
    __syncwarp();
    return pos + __ffs(bits) - 1;
}

// Rows of one coordinate for frames 32 w .. 32 w + 31: lane l holds the bin
// of frame 32 w + l where `frame` says that there is one, and then writes
// rows l and 32 + l, the frames whose bin is below that row's. The six bits
// of the bins become six ballots, and each lane compares them with its row's
// limit bit by bit (a ballot per row took three times the instructions).
__device__ __forceinline__ void build_rows(unsigned* rows, int WS, int w, int R, int step, unsigned bin, bool frame,
                                           int lane) {
    static_assert(kBitBins < 64, "bins and limits have six bits");
    unsigned plane[6];
#pragma unroll
    for (int b = 0; b < 6; ++b) plane[b] = __ballot_sync(kFull, bin >> b & 1u);
    const unsigned have = __ballot_sync(kFull, frame);
    for (int r = lane; r < R; r += 32) {
        const int limit = min(r * step, kBitBins);
        unsigned below = 0, equal = have;
#pragma unroll
        for (int b = 5; b >= 0; --b) {
            const unsigned bit = limit >> b & 1 ? kFull : 0u;
            below |= equal & bit & ~plane[b];
            equal &= ~(bit ^ plane[b]);
        }
        rows[r * WS + w] = below;
    }
}

// (k+1)-th smallest key over the lanes (at least k + 1 of them below kFull).
__device__ __forceinline__ unsigned kth_lane(unsigned u, int k) {
    unsigned last = 0;
    int cnt = 0;
    for (;;) {
        const unsigned mn = __reduce_min_sync(kFull, u > last || cnt == 0 ? u : kFull);
        cnt += __popc(__ballot_sync(kFull, u == mn));
        if (cnt > k || mn == kFull) return mn;
        last = mn;
    }
}

// From the first n listed frames within h (n <= 32 N, n > k): the (k+1)-th
// smallest distance (the query itself is listed, at distance 0), eps over
// the frames at or below it, and whether frames beyond the k-th tie with it.
// Lane i of part c counts the distances smaller than that of entry 32 c + i;
// v holds +inf up to the next multiple of four entries.
template <int N>
__device__ __forceinline__ Found select_nearest(const float* v, const float* da, const float* db, int n, int k, int lane) {
    float x[N], less[N];
#pragma unroll
    for (int c = 0; c < N; ++c) {
        x[c] = 32 * c + lane < n ? v[32 * c + lane] : inf_f();
        less[c] = 0.f;
    }
    for (int t = 0; t < n; t += 4) {
        const float4 y = *reinterpret_cast<const float4*>(v + t);
#pragma unroll
        for (int c = 0; c < N; ++c)
            less[c] += (nsg_lt_f32(y.x, x[c]) + nsg_lt_f32(y.y, x[c])) + (nsg_lt_f32(y.z, x[c]) + nsg_lt_f32(y.w, x[c]));
    }
    unsigned ea = 0, eb = 0;
    int le = 0;
#pragma unroll
    for (int c = 0; c < N; ++c) {
        const bool in = 32 * c + lane < n && less[c] <= static_cast<float>(k);
        le += __popc(__ballot_sync(kFull, in));
        if (in) {
            ea = max(ea, __float_as_uint(da[32 * c + lane]));
            eb = max(eb, __float_as_uint(db[32 * c + lane]));
        }
    }
    Found r;
    ea = __reduce_max_sync(kFull, ea);
    eb = __reduce_max_sync(kFull, eb);
    const unsigned wk = max(ea, eb);  // a joint distance is the larger of its marginals
    r.wk = __uint_as_float(wk);
    r.ea = __uint_as_float(ea);
    r.eb = __uint_as_float(eb);
    r.tie = false;
    if (le > k + 1 && wk != 0) {
        unsigned alo = kFull, ahi = 0, blo = kFull, bhi = 0;
#pragma unroll
        for (int c = 0; c < N; ++c) {
            if (32 * c + lane >= n || __float_as_uint(x[c]) != wk) continue;
            const unsigned a = __float_as_uint(da[32 * c + lane]), b = __float_as_uint(db[32 * c + lane]);
            alo = min(alo, a);
            ahi = max(ahi, a);
            blo = min(blo, b);
            bhi = max(bhi, b);
        }
        alo = __reduce_min_sync(kFull, alo);
        ahi = __reduce_max_sync(kFull, ahi);
        blo = __reduce_min_sync(kFull, blo);
        bhi = __reduce_max_sync(kFull, bhi);
        r.tie = alo != ahi || blo != bhi;
    }
    return r;
}

// Keeps the entries that are not beyond the (k+1)-th smallest (n > k) and
// returns how many; *wk is that distance.
template <int N>
__device__ __forceinline__ int keep_nearest(float* v, float* da, float* db, int n, int k, int lane, float* wk) {
    if (lane < 4) v[n + lane] = inf_f();
    __syncwarp();
    const float w = select_nearest<N>(v, da, db, n, k, lane).wk;
    int kept = 0;
#pragma unroll
    for (int c = 0; c < N; ++c) {
        const int t = 32 * c + lane;
        const bool in = t < n && v[t] <= w;
        const float x = in ? v[t] : 0.f, a = in ? da[t] : 0.f, b = in ? db[t] : 0.f;
        const unsigned mask = __ballot_sync(kFull, in);
        __syncwarp();
        if (in) {
            const int to = kept + __popc(mask & ((1u << lane) - 1u));
            v[to] = x;
            da[to] = a;
            db[to] = b;
        }
        kept += __popc(mask);
        __syncwarp();
    }
    *wk = w;
    return kept;
}

// The same over all m frames: the k + 1 smallest distances in a list spread
// over the lanes (two entries each), then a second pass for eps and ties.
template <int D>
__device__ __noinline__ Found scan_all(const float* __restrict__ xa, const float* __restrict__ xb, int m, int k,
                                       int query, int lane, unsigned long long* evals) {
    float qa[D], qb[D];
    load_frame<D>(xa, query, qa);
    load_frame<D>(xb, query, qb);
    float l0 = inf_f(), l1 = inf_f();
    float U = inf_f();
    for (int j0 = 0; j0 < m; j0 += 32) {
        const int j = j0 + lane;
        float v = inf_f();
        if (j < m) {
            float a[D], b[D];
            load_frame<D>(xa, j, a);
            load_frame<D>(xb, j, b);
            v = fmaxf(dist<D>(qa, a), dist<D>(qb, b));
        }
        unsigned todo = __ballot_sync(kFull, v < U);
        while (todo) {
            const int src = __ffs(todo) - 1;
            todo &= todo - 1;
            const float x = __shfl_sync(kFull, v, src);
            float p0 = __shfl_up_sync(kFull, l0, 1), p1 = __shfl_up_sync(kFull, l1, 1);
            const float top = __shfl_sync(kFull, l0, 31);
            if (lane == 0) {
                p0 = -inf_f();
                p1 = top;
            }
            if (l0 > x) l0 = fmaxf(p0, x);
            if (l1 > x) l1 = fmaxf(p1, x);
        }
        U = k < 32 ? __shfl_sync(kFull, l0, k) : __shfl_sync(kFull, l1, k - 32);
        if (U == 0.f) {  // k others at distance 0
            if (evals && lane == 0) atomicAdd(evals, static_cast<unsigned long long>(min(j0 + 32, m)));
            return Found{0.f, 0.f, 0.f, false};
        }
    }
    // As the tiled kernels have it: a marginal that is not a number adds nothing
    // to eps but differs from every other one at U, and with fewer than k finite
    // distances the frames at +inf are no neighbours yet: any of them makes the
    // sample a tie.
    const bool few = U == inf_f();
    unsigned ea = 0, eb = 0, alo = kFull, ahi = 0, blo = kFull, bhi = 0;
    int le = 0;
    for (int j0 = 0; j0 < m; j0 += 32) {
        const int j = j0 + lane;
        if (j >= m) break;
        float a[D], b[D];
        load_frame<D>(xa, j, a);
        load_frame<D>(xb, j, b);
        const float da = dist<D>(qa, a), db = dist<D>(qb, b), v = fmaxf(da, db);
        if (few ? v < U : v <= U) {
            ++le;
            ea = max(ea, __float_as_uint(fmaxf(da, 0.f)));
            eb = max(eb, __float_as_uint(fmaxf(db, 0.f)));
        }
        if (v == U) {
            alo = min(alo, __float_as_uint(da));
            ahi = max(ahi, __float_as_uint(da));
            blo = min(blo, __float_as_uint(db));
            bhi = max(bhi, __float_as_uint(db));
        }
    }
    le = __reduce_add_sync(kFull, le);
    ea = __reduce_max_sync(kFull, ea);
    eb = __reduce_max_sync(kFull, eb);
    alo = __reduce_min_sync(kFull, alo);
    ahi = __reduce_max_sync(kFull, ahi);
    blo = __reduce_min_sync(kFull, blo);
    bhi = __reduce_max_sync(kFull, bhi);
    const unsigned inf_bits = __float_as_uint(inf_f());
    const bool mixed = alo != ahi || blo != bhi || ahi > inf_bits || bhi > inf_bits;
    if (evals && lane == 0) atomicAdd(evals, static_cast<unsigned long long>(m));
    return Found{__uint_as_float(ea), __uint_as_float(eb), U,
                 few ? alo != kFull : le > k + 1 && U > 0.f && mixed};
}

}  // namespace bitk

// A work item is a pair and a share of its queries (B.chunks shares per
// pair). Dynamic shared memory: rows, node a's frame order, then per warp its
// queries, their bins and the two lists (bits_config sizes it for the batch's
// largest m). Up to 32 N frames within h are kept; each lane ANDs W words
// (32 W frames), of 32 W lanes' worth or, with W = 4, of twice that.
template <int D, int N, int W>
__global__ void __launch_bounds__(1024, 1) ksg_bits_search_kernel(BitsArgs B) {
    using namespace bitk;
    const GridArgs& A = B.g;
    constexpr int NC = 2 * D - 1;  // coordinates with rows: a's other D - 1, b's D
    constexpr int Q = bit_queries(D);
    constexpr int kKeep = 32 * N;
    extern __shared__ __align__(16) unsigned s_dyn[];
    __shared__ int s_start[64];
    __shared__ float s_edge[2 * D][65];
    __shared__ int s_item, s_next;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    unsigned short* s_perm = reinterpret_cast<unsigned short*>(s_dyn + B.rows_words);
    float* s_query = reinterpret_cast<float*>(s_dyn + B.rows_words + B.perm_words) + wid * bit_warp_words(D, N);
    float* s_v = s_query + Q * 8;                  // distances within h, +inf up to a multiple of four
    float* s_da = s_v + kKeep + 4;
    float* s_db = s_da + kKeep;
    unsigned* s_bins = reinterpret_cast<unsigned*>(s_db + kKeep);
    unsigned* s_table = s_bins + Q * 4 * D;
    const int R = B.rows, step = B.step, k = A.k;
    int cur_a = -1;
    float scale = 1.f;               // this warp's share in h, see the file comment
    unsigned evals = 0;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            s_item = atomicAdd(A.counter, 1);
            s_next = 0;
        }
        __syncthreads();
        const int item = s_item;
        if (item >= A.npairs * B.chunks) break;
        const int p = item / B.chunks, ch = item - p * B.chunks;
        const KsgPairDesc* P = A.pairs + p;
        const int m = P->m;
        const int share = ((m + B.chunks - 1) / B.chunks + B.grab - 1) / B.grab * B.grab;
        const int qlo = ch * share, qhi = min(m, qlo + share);
        if (qlo >= qhi) continue;
        const int na_id = A.gp[p].a, nb_id = A.gp[p].b;
        const GridNode* na = A.nodes + na_id;
        const GridNode* nb = A.nodes + nb_id;
        const float* __restrict__ xa = na->aos;
        const float* __restrict__ xb = nb->aos;
        const int WS = bit_row_words(m);
        const bool new_a = na_id != cur_a;
        cur_a = na_id;
        if (new_a) {
            for (int q = tid; q < m; q += blockDim.x) s_perm[q] = __ldg(na->order + q);
            if (tid < 64) s_start[tid] = __ldg(na->ostart + tid);
            __syncthreads();
        }
        // the edges between whole steps of bins (the first coordinate's: all)
        for (int e = tid; e < 128 * D; e += blockDim.x) {
            const int c = e >> 6, t = ((e & 63) + 1) * (c == 0 ? 1 : step);
            const float* edges = c < D ? na->bedges + c * 64 : nb->bedges + (c - D) * 64;
            s_edge[c][e & 63] = t < kBitBins ? __ldg(edges + t) : inf_f();
        }
        // rows
        {
            // the next word's bins load while this one's rows are made
            const unsigned* __restrict__ ba = na->bins;
            const unsigned* __restrict__ bb = nb->bins;
            unsigned va = 0, vb = 0;
            auto fetch = [&](int w) {
                const int pos = 32 * w + lane;
                va = vb = 0;
                if (w < WS && pos < m) {
                    const int j = s_perm[pos];
                    if (D > 1 && new_a) va = __ldg(ba + j);
                    vb = __ldg(bb + j);
                }
            };
            fetch(wid);
            for (int w = wid; w < WS; w += nwarps) {
                const bool frame = 32 * w + lane < m;
                const unsigned ca = va, cb = vb;
                fetch(w + nwarps);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (c < D - 1 && !new_a) continue;
                    const unsigned bin = c < D - 1 ? ca >> (8 * (c + 1)) : cb >> (8 * (c - (D - 1)));
                    build_rows(s_dyn + c * R * WS, WS, w, R, step, bin, frame, lane);
                }
            }
        }
        const bool bad = __ldg(na->ostart + 63) != 0 || __ldg(nb->ostart + 63) != 0;
        // ratio of the k-th joint distance to the geometric mean of the scale
        // estimates for independent nodes of uniform density; scale follows the rest
        const float rank = est_rank(m);
        const float base = exp2f(__log2f(static_cast<float>(k) * m / (rank * rank)) * (0.5f / D) + 0.3f);
        __syncthreads();
        // bins of coordinate c of query t: c = 0 the range of columns of W
        // words, else the byte offsets of its two rows
        auto set_bins = [&](int t, int c) {
            int lo, hi;
            reach(s_edge[c], s_query[8 * t + (c < D ? c : 4 + c - D)], s_query[8 * t + 3], lo, hi);
            if (c == 0) {
                lo = s_start[lo] / (32 * W);
                hi = (s_start[min(hi, kBitBins)] + 32 * W - 1) / (32 * W);
            } else {
                lo = ((c - 1) * R + lo) * WS * 4;
                hi = ((c - 1) * R + hi) * WS * 4;
            }
            *reinterpret_cast<int2*>(s_bins + 4 * D * t + 2 * c) = make_int2(lo, hi);
        };
        for (;;) {
            int q0 = 0;
            if (lane == 0) q0 = atomicAdd(&s_next, B.grab);
            q0 = __shfl_sync(kFull, q0, 0) + qlo;
            if (q0 >= qhi) break;
            const int nq = min(B.grab, qhi - q0);
            __syncwarp();
            if (lane < 2 * Q && lane % Q < nq) {
                const int t = lane % Q, i = q0 + t;
                float x[D];
                load_frame<D>(lane < Q ? xa : xb, i, x);
                float* dst = s_query + 8 * t + (lane < Q ? 0 : 4);
#pragma unroll
                for (int c = 0; c < D; ++c) dst[c] = x[c];
                dst[3] = 0.f;  // of b: the radius that was crowded
                if (lane < Q) {
                    // a node that does not move has no scale of its own
                    const float ea = __ldg(na->est + i), eb = __ldg(nb->est + i);
                    dst[3] = fmaxf(sqrtf((ea > 0.f ? ea : eb) * (eb > 0.f ? eb : ea)) * (base * scale), kLeastH);
                }
            }
            __syncwarp();
            if (lane < 2 * D * nq) set_bins(lane / (2 * D), lane % (2 * D));
            __syncwarp();
            for (int t = 0; t < nq; ++t) {
                const float4 fa = *reinterpret_cast<const float4*>(s_query + 8 * t);
                const float4 fb = *reinterpret_cast<const float4*>(s_query + 8 * t + 4);
                float qa[D], qb[D];
                qa[0] = fa.x;
                qb[0] = fb.x;
                if constexpr (D > 1) {
                    qa[1] = fa.y;
                    qb[1] = fb.y;
                }
                if constexpr (D > 2) {
                    qa[2] = fa.z;
                    qb[2] = fb.z;
                }
                float h = fa.w;
                Found r;
                bool done = false;
                for (int tries = 0; tries < kBitTries && !bad && h > 0.f && h < 1e30f; ++tries) {
                    const uint4* bins = reinterpret_cast<const uint4*>(s_bins + 4 * D * t);
                    const uint4 b0 = bins[0];
                    const int x0 = static_cast<int>(b0.x), x1 = static_cast<int>(b0.y);
                    int inside = 0;
                    int crowd = 0;
                    bool stuck = false;
                    // the AND of the row pairs over column x
                    auto column = [&](int x, auto& acc) {
#pragma unroll
                        for (int g = 0; g < W; ++g) acc[g] = 0;
                        if (x < x1) {
                            const unsigned at = 4 * W * x;
                            auto rows_of = [&](bool start, unsigned lo, unsigned hi) {
                                unsigned u[W], v[W];
                                load_words<W>(s_dyn, hi + at, u);
                                load_words<W>(s_dyn, lo + at, v);
#pragma unroll
                                for (int g = 0; g < W; ++g) acc[g] = start ? u[g] ^ v[g] : acc[g] & (u[g] ^ v[g]);
                            };
                            rows_of(true, b0.z, b0.w);
#pragma unroll
                            for (int q = 1; q < D; ++q) {
                                const uint4 b = bins[q];
                                rows_of(false, b.x, b.y);
                                rows_of(false, b.z, b.w);
                            }
                        }
                    };
                    // Evaluates the frames of the set bits, 32 at a time; false: too many ties.
                    auto consume = [&](auto& w, int base, int cnt, bool last) {
                        const int incl = lane_prefix(cnt);
                        const int n = __shfl_sync(kFull, incl, 31);
                        if (last && inside + n <= k) {  // too few whatever their distances
                            inside += n;
                            return true;
                        }
                        if (n > (tries == 0 ? kCrowd : crowds(W)) * (k + 1) && tries < kCrowdTries) {
                            // another look at the rows is cheaper than that many frames
                            crowd = n;
                            return true;
                        }
                        evals += n;
                        for (int win = 0; win < n; win += 32) {
                            const int pos = bit_of_rank(w, base, 32 * W, incl - cnt, cnt, win, n, lane, s_table);
                            float da = 0.f, db = 0.f, v = inf_f();
                            if (win + lane < n) {
                                const int j = s_perm[pos];
                                float a[D], b[D];
                                load_frame<D>(xa, j, a);
                                load_frame<D>(xb, j, b);
                                da = dist<D>(qa, a);
                                db = dist<D>(qb, b);
                                v = fmaxf(da, db);
                            }
                            unsigned in = __ballot_sync(kFull, v <= h);
                            if (inside + __popc(in) > kKeep) {
                                // k others lie within a smaller h
                                if (inside > k) {
                                    inside = keep_nearest<N>(s_v, s_da, s_db, inside, k, lane, &h);
                                    in = __ballot_sync(kFull, v <= h);
                                }
                                if (inside + __popc(in) > kKeep) {
                                    if (__popc(in) > k) h = __uint_as_float(kth_lane(v <= h ? __float_as_uint(v) : kFull, k));
                                    in = __ballot_sync(kFull, v <= h);
                                    if (inside + __popc(in) > kKeep) return false;
                                }
                            }
                            if (v <= h) {
                                const int slot = inside + __popc(in & ((1u << lane) - 1u));
                                s_v[slot] = v;
                                s_da[slot] = da;
                                s_db[slot] = db;
                            }
                            inside += __popc(in);
                            __syncwarp();
                        }
                        return true;
                    };
                    constexpr int kSpan = W == 4 ? 64 : 32;  // columns at a time
                    for (int xf = x0; xf < x1 && !stuck && !crowd; xf += kSpan) {
                        const int x = xf + lane;
                        const bool last = xf + kSpan >= x1;
                        unsigned u[W];
                        column(x, u);
                        int cnt = 0;
#pragma unroll
                        for (int g = 0; g < W; ++g) cnt += __popc(u[g]);
                        if (W < 4 || xf + 32 >= x1) {
                            stuck = !consume(u, 32 * W * xf, cnt, last);
                        } else {
                            unsigned v[W], w[2 * W];
                            column(x + 32, v);
#pragma unroll
                            for (int g = 0; g < W; ++g) {
                                w[g] = u[g];
                                w[W + g] = v[g];
                                cnt += __popc(v[g]);
                            }
                            stuck = !consume(w, 32 * W * xf, cnt, last);
                        }
                    }
                    if (stuck) break;
                    if (crowd) {
                        if (lane == 0) s_query[8 * t + 7] = h;
                        scale *= 0.9985f;
                        h *= exp2f(__log2f(0.5f * kCrowd * (k + 1) / crowd) * ((tries + 1) * (0.5f / D)));
                    } else if (inside > k) {
                        if (lane < 4) s_v[inside + lane] = inf_f();
                        __syncwarp();
                        r = select_nearest<N>(s_v, s_da, s_db, inside, k, lane);
                        __syncwarp();
                        if (tries == 0) scale *= 0.9985f;
                        else if (r.wk < kFar * s_query[8 * t + 7]) scale = fmaxf(0.9f * scale, kLeastScale);
                        done = true;
                        break;
                    } else {
                        if (tries == 0) scale = fminf(1.02f * scale, 1.f / kLeastScale);
                        const int faster = max(1, tries - 1);  // an estimate off by factors
                        h *= fminf(static_cast<float>(1 << faster),
                                   exp2f(__log2f(2.f * (k + 1) / (inside + 0.5f)) * (faster * (0.5f / D))));
                    }
                    if (lane == 0) s_query[8 * t + 3] = h;
                    __syncwarp();
                    if (lane < 2 * D) set_bins(t, lane);
                    __syncwarp();
                }
                if (!done) {
                    r = scan_all<D>(xa, xb, m, k, q0 + t, lane, A.evals);
                }
                const long long o = P->scratch + q0 + t;
                if (lane < 2) (lane ? A.eps_b : A.eps_a)[o] = lane ? r.eb : r.ea;
                if (A.eps_x && lane == 0) A.eps_x[o] = r.ea;
                if (A.eps_y && lane == 0) A.eps_y[o] = r.eb;
                if (A.kdist && lane == 0) A.kdist[o] = r.wk;
                if (r.tie && lane == 0) {
                    const int slot = atomicAdd(A.tie_count, 1);
                    if (slot < A.tie_cap) A.ties[slot] = KsgTie{A.pair_base + p, q0 + t};
                    else atomicOr(A.fault, FAULT_TIE_OVERFLOW);
                }
            }
        }
        if (A.evals && lane == 0) atomicAdd(A.evals, static_cast<unsigned long long>(evals));
        evals = 0;
    }
}

// Scale estimates of one node's frames (GridNode::est), a share of them per
// CTA (blockIdx.y). The width of the bins around a frame gives each
// coordinate's density, and their product a first radius that would hold
// R = est_rank(m) frames if the coordinates were independent; the frames
// within that radius, counted on the node's own rows (in whole bins and
// words: a few percent of the radius), correct it. With one coordinate the
// density alone is the estimate. In a CPU model of m = 10000 trajectories the
// geometric mean of two nodes' estimates follows the k-th joint distance to
// 8% (nearly independent coordinates) and 12% (correlated ones), as well as
// the exact 64th-neighbour distances do.
constexpr int kEstThreads = 1024;

template <int D>
__global__ void __launch_bounds__(kEstThreads) bits_est_kernel(const GridNode* nodes, int step) {
    using namespace bitk;
    extern __shared__ __align__(16) unsigned s_dyn[];
    __shared__ float s_edge[D][65];
    __shared__ float s_whole[D][64];
    __shared__ int s_start[64];
    __shared__ float s_out[D][2];
    const GridNode nd = nodes[blockIdx.x];
    const int m = nd.m;
    if (m > kBitMaxM) return;
    const int share = (m + gridDim.y - 1) / gridDim.y;
    const int lo = blockIdx.y * share, hi = min(m, lo + share);
    if (lo >= hi) return;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nwarps = blockDim.x >> 5;
    const int R = (kBitBins + step - 1) / step + 1;
    const int WS = bit_row_words(m);
    for (int e = tid; e < 64 * D; e += blockDim.x) {
        const int c = e >> 6, t = e & 63;
        s_edge[c][t] = __ldg(nd.bedges + e);
        s_whole[c][t] = (t + 1) * step < kBitBins ? __ldg(nd.bedges + c * 64 + (t + 1) * step) : inf_f();
    }
    if (tid < 64) s_start[tid] = __ldg(nd.ostart + tid);
    // The outermost edges no further out than three times the two bins before
    // them are wide: a frame far from all others stretched its bin, and the
    // least width of all, by any factor.
    int live = 0;  // coordinates that are not the same in nearly all frames
#pragma unroll
    for (int c = 0; c < D; ++c) {
        const float* e = nd.bedges + 64 * c;
        const float lo = __ldg(e + 1), hi = __ldg(e + kBitBins - 1);
        live += hi > lo;
        if (tid == c) {
            s_out[c][0] = fmaxf(__ldg(e), lo - 3.f * (__ldg(e + 3) - lo));
            s_out[c][1] = fminf(__ldg(e + kBitBins), hi + 3.f * (hi - __ldg(e + kBitBins - 3)));
        }
    }
    const float inv = 1.f / max(1, live);
    if constexpr (D > 1) {
        // the next word's bins load while this one's rows are made
        auto bins_of = [&](int w) {
            const int pos = 32 * w + lane;
            return w < WS && pos < m ? __ldg(nd.bins + __ldg(nd.order + pos)) : 0u;
        };
        unsigned next = bins_of(wid);
        for (int w = wid; w < WS; w += nwarps) {
            const int pos = 32 * w + lane;
            const unsigned v = next;
            next = bins_of(w + nwarps);
#pragma unroll
            for (int c = 1; c < D; ++c)
                build_rows(s_dyn + (c - 1) * R * WS, WS, w, R, step, v >> (8 * c), pos < m, lane);
        }
    }
    __syncthreads();
    const float rank = est_rank(m);
    // lane 4 t + c: coordinate c of the warp's query t
    for (int q0 = lo + 8 * wid; q0 < hi; q0 += 8 * nwarps) {
        const int t = lane >> 2, c = lane & 3;
        const int i = min(q0 + t, hi - 1);
        float x = 0.f, width = 1.f;
        if (c < D) {
            float f[D];
            load_frame<D>(nd.aos, i, f);
            x = f[0];
            if constexpr (D > 1) x = c == 1 ? f[1] : x;
            if constexpr (D > 2) x = c == 2 ? f[2] : x;
            const int b = __ldg(nd.bins + i) >> (8 * c) & 0xffu;
            const int b0 = max(b - 2, 0), b1 = min(b + 3, kBitBins);
            const float e0 = b0 == 0 ? s_out[c][0] : s_edge[c][b0], e1 = b1 == kBitBins ? s_out[c][1] : s_edge[c][b1];
            width = fmaxf((e1 - e0) * (static_cast<float>(kBitBins) / (b1 - b0)), 2e-3f * (s_out[c][1] - s_out[c][0]));
            if (!(s_edge[c][kBitBins - 1] > s_edge[c][1])) width = 1.f;
        }
        width *= __shfl_xor_sync(kFull, width, 1);
        width *= __shfl_xor_sync(kFull, width, 2);
        float est = live ? 0.5f * exp2f(__log2f(width * rank / m) * inv) : 0.f;
        if constexpr (D > 1) {
            // first and one past the last whole bin within est, as in the search
            unsigned pack = 0;
            if (c < D) {
                int a = 0, b = 0;
#pragma unroll
                for (int s = 32; s > 0; s >>= 1) {
                    if (__fsub_rn(x, s_whole[c][a + s - 1]) > est) a += s;
                    if (__fsub_rn(s_whole[c][b + s - 1], x) <= est) b += s;
                }
                b = min(b + 1, R - 1);  // an infinite estimate reaches past the padded edges
                if (c == 0) {
                    a = s_start[min(a * step, kBitBins)] >> 5;
                    b = (s_start[min(b * step, kBitBins)] + 31) >> 5;
                }
                pack = static_cast<unsigned>(b) << 16 | static_cast<unsigned>(a);
            }
            float within = 0.f;
            for (int u = 0; u < 8; ++u) {
                const unsigned range = __shfl_sync(kFull, pack, 4 * u);
                const unsigned r1 = __shfl_sync(kFull, pack, 4 * u + 1);
                const unsigned r2 = __shfl_sync(kFull, pack, 4 * u + 2);
                int n = 0;
                for (int w = static_cast<int>(range & 0xffffu) + lane; w < static_cast<int>(range >> 16); w += 32) {
                    unsigned bits = s_dyn[(r1 >> 16) * WS + w] ^ s_dyn[(r1 & 0xffffu) * WS + w];
                    if constexpr (D > 2) bits &= s_dyn[(R + (r2 >> 16)) * WS + w] ^ s_dyn[(R + (r2 & 0xffffu)) * WS + w];
                    n += __popc(bits);
                }
                n = __reduce_add_sync(kFull, n);
                if (t == u) within = static_cast<float>(n);
            }
            est *= exp2f(__log2f(rank / fmaxf(within, 1.f)) * inv);
        }
        if (c == 0 && q0 + t < hi) nd.est[i] = est;
    }
}

}  // namespace nsg
