// rigidpair.cuh -- sums of the rigid pair kernel's records (rigidpair.cu).
#pragma once
#include "geom.cuh"
#include "kernels.h"

namespace fmd {

constexpr int kRigidRec = 13;   // F T W(xx xy xz yy yz zz) E of a molecule's part

__device__ __forceinline__ int rigid_owner(int i, int j) { return ((i + j) & 1) ? min(i, j) : max(i, j); }

// Force and torque v[6] of molecule i (in every lane), its energy and virial
// added to the lanes' tot {E, W9}; the whole warp calls it.
__device__ __forceinline__ void rigid_pair_sum(const RigidPair& r, const int* __restrict__ cnt,
                                               const int* __restrict__ list, int cap, int i, int lane, double (&v)[6],
                                               double (&tot)[kNV]) {
#pragma unroll
    for (int c = 0; c < 6; c++) v[c] = 0.0;
    const int nn = cnt[i];
    for (int k = lane; k < nn; k += 32) {
        const size_t t = (size_t)i * cap + k;
        const int j = list[t], b = r.back[t];
        if (b < 0 || rigid_owner(i, j) == i) continue;
        const double* o = r.rec + ((size_t)j * cap + b) * r.chunks * 6;
        for (int q = 0; q < r.chunks; q++)
#pragma unroll
            for (int c = 0; c < 6; c++) v[c] += o[6 * q + c];
    }
    for (int s = lane; s < r.parts; s += 32) {
        const double* o = r.out + ((size_t)i * r.parts + s) * kRigidRec;
#pragma unroll
        for (int c = 0; c < 6; c++) v[c] += o[c];
        const double xy = o[7], xz = o[8], yz = o[10];
        tot[0] += o[12];
        tot[1] += o[6]; tot[2] += xy; tot[3] += xz;
        tot[4] += xy; tot[5] += o[9]; tot[6] += yz;
        tot[7] += xz; tot[8] += yz; tot[9] += o[11];
    }
#pragma unroll
    for (int c = 0; c < 6; c++) v[c] = warp_sum(v[c]);
}

}  // namespace fmd
