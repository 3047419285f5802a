// ljclus.cuh -- what the next evaluation of the cluster gather does.
#pragma once
#include <cmath>

#include "kernels.h"
#include "ljprune.cuh"

namespace fmd {

enum LJClusMode { CLUS_FULL = 0, CLUS_PRUNE = 1, CLUS_WALK = 2 };

// Cluster rows need the molecule builder's bitmaps, a diagonal cell and edges
// wide enough that at most one image of an atom is within rc + delta of
// another (ljclus.cu).  Evaluated on the same inputs by
// every block of the gather and by the step's reduction.
__device__ __forceinline__ int lj_clus_mode(const LJClus& c, const unsigned long long* words, const double* hh,
                                            const double* hb, double delta, double rc) {
    const int flag = c.flag[0];
    const bool stale = lj_prune_needed(words, hh, hb, delta, rc, kRowsClusters);
    const bool diag = hh[1] == 0.0 && hh[2] == 0.0 && hh[3] == 0.0 && hh[5] == 0.0 && hh[6] == 0.0 && hh[7] == 0.0;
    const double edge = fmin(hh[0], fmin(hh[4], hh[8]));
    if (flag == 0 || !diag || !(edge > 2.0 * (rc + delta) + 0.1)) return CLUS_FULL;
    return stale ? CLUS_PRUNE : CLUS_WALK;
}

}  // namespace fmd
