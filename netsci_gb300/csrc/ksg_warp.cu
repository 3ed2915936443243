// Exhaustive KSG counts for small plans, one warp per query.
//
// The tiled kernels (ksg_kernels.cuh) give a thread to every query, so a
// single pair of 2,000 samples keeps 32 small CTAs busy while each thread
// walks 2,000 frames twice: 101 us whatever the GPU could do beside it. Here
// a CTA copies the pair's frames into shared memory and each of its warps
// takes one query, its lanes the frames:
//   * every lane keeps the least joint distance of its frames; the (k+1)-th
//     smallest of the 32 minima bounds the k-th neighbour's (the query itself
//     is one frame, at distance 0), and few other frames pass that bound;
//   * the frames within it are listed with their marginal distances and the
//     k nearest selected as in the bitmap search, ties included; samples with
//     too many ties, fewer than k finite distances or a neighbour whose
//     marginal is not a number count their distances up instead;
//   * the marginal counts are warp sums over all frames.
// Per query and frame that is two to three times the tiled kernels' work, so
// it serves small plans (warp_us in engine.cpp), where the GPU is mostly idle
// otherwise.
#include "common.cuh"
#include "ksg_bits.cuh"
#include "ksg_kernels.cuh"
#include "ksg_warp.h"

namespace nsg {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr size_t kMaxSmem = 200 << 10;
constexpr int kList = 96;  // frames within the bound a query keeps

template <int D>
__global__ void __launch_bounds__(32 * kWarpsPerCta) ksg_warp_kernel(KsgCountArgs A) {
    using namespace bitk;
    extern __shared__ __align__(16) float s_x[];  // 2D planes of mp floats, then the lists
    const KsgItem w = A.items[blockIdx.x];
    const KsgPairDesc P = A.pairs[w.pair];
    const int m = P.m, mp = (m + 31) / 32 * 32, k = A.k;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    // frames past the end are NaN: no comparison lets them in
    for (int j = threadIdx.x; j < mp; j += blockDim.x) {
        const int src = j < m ? ksgk::frame_of(P.fmap, j, P.ld, A.fault) : 0;
#pragma unroll
        for (int c = 0; c < D; ++c) {
            s_x[c * mp + j] = j < m ? __ldg(P.xa + static_cast<size_t>(c) * P.ld + src) : __int_as_float(0x7fc00000);
            s_x[(D + c) * mp + j] = j < m ? __ldg(P.xb + static_cast<size_t>(c) * P.ld + src) : __int_as_float(0x7fc00000);
        }
    }
    float* s_v = s_x + 2 * D * mp + wid * (3 * kList + 4);
    float* s_da = s_v + kList + 4;
    float* s_db = s_da + kList;
    __syncthreads();
    for (int i = w.q0 + wid; i < w.q1; i += kWarpsPerCta) {
        float qa[D], qb[D];
#pragma unroll
        for (int c = 0; c < D; ++c) {
            qa[c] = s_x[c * mp + i];
            qb[c] = s_x[(D + c) * mp + i];
        }
        auto distances = [&](int j, float& da, float& db) {
            float a[D], b[D];
#pragma unroll
            for (int c = 0; c < D; ++c) {
                a[c] = s_x[c * mp + j];
                b[c] = s_x[(D + c) * mp + j];
            }
            da = dist<D>(qa, a);
            db = dist<D>(qb, b);
        };
        float least = inf_f();
#pragma unroll 4
        for (int j = lane; j < mp; j += 32) {
            float da, db;
            distances(j, da, db);
            least = fminf(least, fmaxf(da, db));
        }
        float h = __uint_as_float(kth_lane(__float_as_uint(least), k));
        int inside = 0;
        bool stuck = !(h < inf_f());
        for (int j = lane; j < mp && !stuck; j += 32) {
            float da, db;
            distances(j, da, db);
            const float v = fmaxf(da, db);
            unsigned in = __ballot_sync(kFull, v <= h);
            if (!in) continue;
            if (__any_sync(kFull, v <= h && (da != da || db != db))) {  // the other marginal stands for both
                stuck = true;
                break;
            }
            if (inside + __popc(in) > kList) {
                if (inside > k) inside = keep_nearest<kList / 32>(s_v, s_da, s_db, inside, k, lane, &h);
                in = __ballot_sync(kFull, v <= h);
                if (inside + __popc(in) > kList) {  // heavy ties
                    stuck = true;
                    break;
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
        Found r;
        if (!stuck) {
            if (lane < 4) s_v[inside + lane] = inf_f();
            __syncwarp();
            r = select_nearest<kList / 32>(s_v, s_da, s_db, inside, k, lane);
            __syncwarp();
        } else {
            // without the list: the (k+1)-th smallest by counting up distinct distances
            float U = -1.f;
            int le = 0;
            while (le <= k) {
                float next = inf_f();
                for (int j = lane; j < mp; j += 32) {
                    float da, db;
                    distances(j, da, db);
                    const float v = fmaxf(da, db);
                    if (v > U) next = fminf(next, v);
                }
                U = __uint_as_float(__reduce_min_sync(kFull, __float_as_uint(next)));
                le = 0;
                for (int j = lane; j < mp; j += 32) {
                    float da, db;
                    distances(j, da, db);
                    le += fmaxf(da, db) <= U;
                }
                le = __reduce_add_sync(kFull, le);
                if (U == inf_f()) break;
            }
            // As the tiled kernels have it: a marginal that is not a number
            // adds nothing to eps but differs from every other one at U, and
            // with fewer than k finite distances the frames at +inf are no
            // neighbours yet: any of them makes the sample a tie.
            const bool few = U == inf_f();
            unsigned ea = 0, eb = 0, alo = kFull, ahi = 0, blo = kFull, bhi = 0;
            for (int j = lane; j < mp; j += 32) {
                float da, db;
                distances(j, da, db);
                const float v = fmaxf(da, db);
                if (few ? v < U : v <= U) {
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
            r.ea = __uint_as_float(__reduce_max_sync(kFull, ea));
            r.eb = __uint_as_float(__reduce_max_sync(kFull, eb));
            r.wk = U;
            alo = __reduce_min_sync(kFull, alo);
            ahi = __reduce_max_sync(kFull, ahi);
            blo = __reduce_min_sync(kFull, blo);
            bhi = __reduce_max_sync(kFull, bhi);
            const unsigned inf_bits = __float_as_uint(inf_f());
            const bool mixed = alo != ahi || blo != bhi || ahi > inf_bits || bhi > inf_bits;
            r.tie = few ? alo != kFull : le > k + 1 && U > 0.f && mixed;
        }
        float ca = 0.f, cb = 0.f;
#pragma unroll 4
        for (int j = lane; j < mp; j += 32) {
            float da, db;
            distances(j, da, db);
            ca += nsg_le_f32(da, r.ea);
            cb += nsg_le_f32(db, r.eb);
        }
        const int na = __reduce_add_sync(kFull, static_cast<int>(ca)), nb = __reduce_add_sync(kFull, static_cast<int>(cb));
        if (lane == 0) {
            const long long o = P.scratch + i;
            // as ksgk::write_outputs: non-finite inputs stay inside the table
            const int nx = min(max(na - 1, 0), m), ny = min(max(nb - 1, 0), m);
            A.psum[o] = __fadd_rn(__ldg(A.psi + nx), __ldg(A.psi + ny));
            if (A.nx) A.nx[o] = nx;
            if (A.ny) A.ny[o] = ny;
            if (A.eps_x) A.eps_x[o] = r.ea;
            if (A.eps_y) A.eps_y[o] = r.eb;
            if (A.kdist) A.kdist[o] = r.wk;
            if (r.tie) {
                const int slot = atomicAdd(A.tie_count, 1);
                if (slot < A.tie_cap) A.ties[slot] = KsgTie{w.pair, i};
                else atomicOr(A.fault, FAULT_TIE_OVERFLOW);
            }
        }
        __syncwarp();
    }
}

template <int D>
void launch(const KsgCountArgs& a, size_t smem, cudaStream_t st) {
    // set on every launch: the attribute belongs to the current device. One
    // value for all plans: another thread may set it before this launch.
    NSG_CUDA(cudaFuncSetAttribute(ksg_warp_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(kMaxSmem)));
    ksg_warp_kernel<D><<<a.nitems, 32 * kWarpsPerCta, smem, st>>>(a);
    NSG_CUDA(cudaGetLastError());
}

size_t smem_bytes(int d, int max_m) {
    const size_t mp = (static_cast<size_t>(max_m) + 31) / 32 * 32;
    return sizeof(float) * (2 * d * mp + static_cast<size_t>(kWarpsPerCta) * (3 * kList + 4));
}

}  // namespace

bool ksg_warp_fits(int d, int k, int max_m) {
    return k <= 30 && smem_bytes(d, max_m) <= kMaxSmem;  // the bound comes from 32 lane minima
}

void ksg_launch_warp(const KsgCountArgs& a, int d, int max_m, cudaStream_t st) {
    if (a.nitems <= 0) return;
    const size_t smem = smem_bytes(d, max_m);
    switch (d) {
        case 1: launch<1>(a, smem, st); break;
        case 2: launch<2>(a, smem, st); break;
        case 3: launch<3>(a, smem, st); break;
        default: invalid("d must be 1, 2 or 3");
    }
}

}  // namespace nsg
