// The reference sort's order restated serially (sort_prefix.h), for tests that
// compare the tie kernels with it: the first T positions of one row.
#include "sort_prefix.h"

extern "C" int sort_prefix_row(const float* key, int* idx, int n, int T) {
    nsg::SortSegment stack[64];
    for (int i = 0; i < n; ++i) idx[i] = i;
    return nsg::sort_prefix_like_reference(key, idx, n, T, stack, 64) ? 1 : 0;
}
