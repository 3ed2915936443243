// Exhaustive counts of small plans, one warp per query (ksg_warp.cu).
#pragma once

#include "ksg.cuh"

namespace nsg {

constexpr int kWarpsPerCta = 16;
// Whether the kernel can run pairs of up to max_m samples; the planner takes it
// where its estimate (warp_us) is the smallest.
bool ksg_warp_fits(int d, int k, int max_m);
// One CTA per work item of `a` (KsgItem slices of kWarpsPerCta queries or a
// multiple).
void ksg_launch_warp(const KsgCountArgs& a, int d, int max_m, cudaStream_t st);

}  // namespace nsg
