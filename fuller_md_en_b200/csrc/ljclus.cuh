// ljclus.cuh -- what the next evaluation of the cluster gather does.
#pragma once
#include <cmath>

#include "kernels.h"
#include "ljprune.cuh"

namespace fmd {

// Rows of atoms or of clusters; built from the lists now, or walked as the last
// prune left them; the full rows of atoms as they are.
enum LJClusMode { ATOMS_PRUNE = 0, ATOMS_WALK = 1, CLUS_PRUNE = 2, CLUS_WALK = 3, ATOMS_FULL = 4, LJ_MODES = 5 };
__device__ __forceinline__ bool lj_clus_prunes(int mode) { return mode == ATOMS_PRUNE || mode == CLUS_PRUNE; }
__device__ __forceinline__ unsigned long long lj_clus_kind(int mode) {
    return mode == CLUS_PRUNE || mode == CLUS_WALK ? kRowsClusters : kRowsAtoms;
}

// Cluster rows need the molecule builder's bitmaps, a diagonal cell and edges
// wide enough that at most one image of an atom is within rc + delta of
// another (ljclus.cu); the list build may have chosen rows of atoms
// (MolLists::flag[3]).  Evaluated on the same inputs by every block of the
// gather and by the step's reduction.
__device__ __forceinline__ int lj_clus_mode(const LJClus& c, const unsigned long long* words, const double* hh,
                                            const double* hb, double delta, double rc) {
    const int4 flag = *reinterpret_cast<const int4*>(c.flag);      // with the loads of the bound
    const bool built = flag.x != 0 && flag.w == 0;
    const bool diag = hh[1] == 0.0 && hh[2] == 0.0 && hh[3] == 0.0 && hh[5] == 0.0 && hh[6] == 0.0 && hh[7] == 0.0;
    const double edge = fmin(hh[0], fmin(hh[4], hh[8]));
    const bool clusters = built && diag && edge > 2.0 * (rc + delta) + 0.1;
    const bool stale = lj_prune_needed(words, hh, hb, delta, rc, clusters ? kRowsClusters : kRowsAtoms);
    if (flag.w > 1 && flag.z == 0) return ATOMS_FULL;
    return clusters ? (stale ? CLUS_PRUNE : CLUS_WALK) : (stale ? ATOMS_PRUNE : ATOMS_WALK);
}

}  // namespace fmd
