// ljclus.h -- host side of the cluster gather (ljclus.cu).
#pragma once
#include <vector>

#include "kernels.h"

namespace fmd {

// Atoms of one molecule (S positions x[3 S]) in clusters of kClusG near
// neighbours: perm[cluster * kClusG + k], the first the most central, -1
// beyond the last.
std::vector<int> lj_clus_assign(const double* x, int S);

}  // namespace fmd
