// Instantiations and launch of the bitmap search (ksg_bits.cuh).
#include "ksg_bits.cuh"

#include <algorithm>
#include <cmath>

#include "engine.h"
#include "errors.h"

namespace nsg {

// Shared memory of an SM, and what a CTA takes beside its dynamic part.
static constexpr size_t kSm = 228 << 10, kStatic = 2048, kReserved = 1024;

BitsConfig bits_config(int d, int k, int max_m) {
    BitsConfig c;
    if (d < 1 || d > 3 || max_m < 1 || max_m > kBitMaxM) return c;
    const int nc = 2 * d - 1, ws = bit_row_words(max_m);
    c.keep = k <= 12 ? 1 : 3;
    // The first coordinate's interval covers about (k/m)^(1/2d) of the frames,
    // a little more for the search's margin and the bins: one, two or four
    // words a lane, whichever covers it in one go. Fewer words a lane leave
    // fewer instructions per query (m = 1000: one word against four).
    const double part = std::min(1.0, 1.15 * std::pow(static_cast<double>(k) / max_m, 0.5 / d) + 0.04);
    const double span = part * max_m / 32;
    c.words = span <= 28 ? 1 : span <= 56 ? 2 : 4;
    c.perm_words = ((max_m + 1) / 2 + 3) & ~3;
    auto fits = [&](int step, int threads, int ctas) {
        c.step = step;
        c.threads = threads;
        c.ctas_per_sm = ctas;
        c.rows = (kBitBins + step - 1) / step + 1;
        c.rows_words = nc * c.rows * ws;
        c.smem = sizeof(unsigned) * (static_cast<size_t>(c.rows_words) + c.perm_words +
                                     static_cast<size_t>(threads / 32) * bit_warp_words(d, c.keep));
        c.ok = ctas * (c.smem + kStatic + kReserved) <= kSm;
        return c.ok;
    };
    // a row per bin or per two, as many CTAs per SM as fit (1024 threads in
    // all): a row per bin leaves a sixth fewer candidates (m = 1000: 20.4
    // against 23.9 per query, 3% less time even with half the CTAs)
    for (int step : {1, 2}) {
        for (int n : {8, 4, 2, 1}) {
            if (fits(step, 1024 / n, n)) return c;
        }
    }
    // long rows or lists: fewer warps, then four and six bins per row (wider
    // intervals, more candidates)
    for (int step : {2, 4, 6}) {
        for (int threads : {1024, 768, 512}) {
            if (fits(step, threads, 1)) return c;
        }
    }
    return c;
}

namespace {

template <int D, int N, int W>
void launch(const BitsArgs& a, const BitsConfig& c, int grid, cudaStream_t s) {
    // set on every launch: the attribute belongs to the current device. One
    // value for all plans: another thread may set it before this launch.
    NSG_CUDA(cudaFuncSetAttribute(ksg_bits_search_kernel<D, N, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  static_cast<int>(kSm - kStatic - kReserved)));
    ksg_bits_search_kernel<D, N, W><<<grid, c.threads, c.smem, s>>>(a);
    NSG_CUDA(cudaGetLastError());
}

template <int D, int N>
void launch(const BitsArgs& a, const BitsConfig& c, int grid, cudaStream_t s) {
    if (c.words == 1) launch<D, N, 1>(a, c, grid, s);
    else if (c.words == 2) launch<D, N, 2>(a, c, grid, s);
    else launch<D, N, 4>(a, c, grid, s);
}

template <int D>
void launch(const BitsArgs& a, const BitsConfig& c, int grid, cudaStream_t s) {
    if (c.keep == 1) launch<D, 1>(a, c, grid, s);
    else launch<D, 3>(a, c, grid, s);
}

}  // namespace

void bits_launch_est(const GridNode* nodes, int nnodes, int max_m, int d, cudaStream_t s) {
    if (nnodes <= 0) return;
    max_m = std::min(max_m, kBitMaxM);  // longer nodes take neither bitmaps nor orders (kOrderMaxM)
    const size_t most = 200 << 10;
    int step = 1;
    size_t smem = 0;
    for (;; step *= 2) {
        smem = sizeof(unsigned) * (d - 1) * ((kBitBins + step - 1) / step + 1) * static_cast<size_t>(bit_row_words(max_m));
        if (smem <= most) break;
    }
    // A node's frames split over CTAs (one per SM: 1024 threads of 57
    // registers), 256 frames at a time in each; every share builds the rows
    // again, two rounds' worth.
    const int sms = sm_count();
    int parts = 1, best = 1 << 30;
    for (int p = 1; p <= std::max(1, max_m / 256); ++p) {
        const int waves = (nnodes * p + sms - 1) / sms;
        const int cost = waves * ((max_m / p + 255) / 256 + 2);
        if (cost < best) {
            best = cost;
            parts = p;
        }
    }
    const dim3 grid(nnodes, parts);
    switch (d) {
        case 1: bits_est_kernel<1><<<grid, kEstThreads, 0, s>>>(nodes, step); break;
        case 2:
            NSG_CUDA(cudaFuncSetAttribute(bits_est_kernel<2>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(most)));
            bits_est_kernel<2><<<grid, kEstThreads, smem, s>>>(nodes, step);
            break;
        case 3:
            NSG_CUDA(cudaFuncSetAttribute(bits_est_kernel<3>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          static_cast<int>(most)));
            bits_est_kernel<3><<<grid, kEstThreads, smem, s>>>(nodes, step);
            break;
        default: invalid("d must be 1, 2 or 3");
    }
    NSG_CUDA(cudaGetLastError());
}

std::vector<BitsSegment> bits_segments(const KsgPairDesc* descs, int npairs, int d, int k) {
    std::vector<BitsSegment> out;
    if (npairs <= 0) return out;
    BitsConfig c = bits_config(d, k, descs[0].m);
    if (!c.ok) return out;
    out.push_back({0, 0, descs[0].m, c});
    const int enough = 4 * sm_count();
    int m = descs[0].m;
    for (int p = 0; p < npairs; ++p) {
        if (descs[p].m != m) {
            m = descs[p].m;
            c = bits_config(d, k, m);
        }
        // a pair that would take other words starts a segment, if the last
        // one is long enough to fill the GPU
        if (c.words != out.back().config.words && out.back().npairs >= enough &&
            static_cast<int>(out.size()) < kBitSegments) {
            out.push_back({p, 0, m, c});
        }
        ++out.back().npairs;
    }
    return out;
}

void bits_launch_search(const GridArgs& g, const BitsSegment& seg, int* counter, int d, cudaStream_t s) {
    const BitsConfig& c = seg.config;
    const int max_m = seg.max_m;
    BitsArgs a{};
    a.g = g;
    a.g.pairs += seg.first;
    a.g.gp += seg.first;
    a.g.pair_base += seg.first;
    a.g.npairs = seg.npairs;
    a.g.counter = counter;
    a.rows = c.rows;
    a.step = c.step;
    a.rows_words = c.rows_words;
    a.perm_words = c.perm_words;
    // Pairs are split while there are fewer than four items per resident CTA:
    // every share builds the pair's rows again.
    const int slots = sm_count() * c.ctas_per_sm;
    const int most = std::max(1, max_m / (2 * (c.threads / 32)));
    a.chunks = seg.npairs >= 4 * slots ? 1 : std::min(most, (4 * slots + seg.npairs - 1) / seg.npairs);
    // a share of few queries is spread over all warps
    const int per_warp = max_m / (a.chunks * (c.threads / 32));
    a.grab = std::max(1, std::min(bit_queries(d), per_warp));
    const long long items = static_cast<long long>(seg.npairs) * a.chunks;
    const int grid = static_cast<int>(std::min<long long>(items, slots));
    switch (d) {
        case 1: launch<1>(a, c, grid, s); break;
        case 2: launch<2>(a, c, grid, s); break;
        case 3: launch<3>(a, c, grid, s); break;
        default: invalid("d must be 1, 2 or 3");
    }
}

}  // namespace nsg
