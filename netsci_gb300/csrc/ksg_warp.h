// Exhaustive counts of small plans, one warp per query (ksg_warp.cu).
#pragma once

#include "ksg.cuh"

namespace nsg {

constexpr int kWarpsPerCta = 16;
// Whether a plan whose pairs' squared sample counts add up to `work` (max_m:
// the largest) takes it: its time, about 1.5, 2.2 and 2.9 us per million
// frame visits at d = 1, 2, 3, stays below what the cell grids' chain of small
// kernels takes for such a plan (100 to 130 us; the tiled kernels take 100 to
// 340 us per pair at m = 1000 to 4000). 1000 samples, 10 pairs, d = 3: 49 us
// against 107 on grids and 115 tiled; 4000 samples, 3 pairs: 144, 176, 345.
bool ksg_warp_fits(int d, int k, int max_m, double work);
// One CTA per work item of `a` (KsgItem slices of kWarpsPerCta queries or a
// multiple).
void ksg_launch_warp(const KsgCountArgs& a, int d, int max_m, cudaStream_t st);

}  // namespace nsg
