// molquad.h -- which atoms the half-row walk of equal molecules reads
// (k_mol_half_quad, molnlist.cu), in a header of plain C++ so that the bounds
// are checked on the host.
#pragma once

#ifdef __CUDACC__
#define FMD_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FMD_HOST_DEVICE inline
#endif

namespace fmd {

// The atom that a lane reads in slice u of partner t of ns: atom lane + 32 u of
// the partner molecule, whose S atoms start at j0.  Lanes past S, and every
// lane of a load beyond the last partner, read i0, the warp's own first atom.
FMD_HOST_DEVICE int quad_atom(int t, int ns, int j0, int i0, int S, int lane, int u) {
    const int b = lane + 32 * u;
    return t < ns && b < S ? j0 + b : i0;
}

}  // namespace fmd
