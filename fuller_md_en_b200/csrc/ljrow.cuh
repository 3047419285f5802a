// ljrow.cuh -- one atom's row of the LJ gather: entries fetched by the lanes of
// a warp, the pair terms of a chunk, and the end of the row.  Used by the row
// gathers (airebo.cu) and by the cluster gather's rows of atoms (ljclus.cu).
#pragma once
#include "geom.cuh"
#include "kernels.h"
#include "ljpair.cuh"

namespace fmd {
namespace {

// Entries per lane in flight (U): the index loads of U entries are issued
// together, then their positions, then the pair arithmetic, so one warp has
// U dependent load chains outstanding instead of one.  PIPE additionally
// software-pipelines the lane's loop: the indices and positions of the next
// U entries are loaded before the current U are computed, so their latency
// overlaps the arithmetic.
template <int U>
__device__ __forceinline__ void lj_fetch(const double* __restrict__ pos, const int* __restrict__ row, int tot,
                                         int b, int i, int (&jj)[U], double (&qx)[U], double (&qy)[U],
                                         double (&qz)[U]) {
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int k = b + 32 * u;
        jj[u] = k < tot ? row[k] : -1;
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int j = jj[u] < 0 ? i : jj[u];
        qx[u] = pos[3 * j]; qy[u] = pos[3 * j + 1]; qz[u] = pos[3 * j + 2];
    }
}

// Pair terms of one chunk (U entries per lane; jc < 0: none) seen from atom i.
// A pruning gather (po.cnt set) also appends the chunk's entries with
// r^2 <= po.r2 to prow in row order (entry b0 + 32 u + lane, u then lane
// ascending); every lane of the warp must call this.
template <bool FULL_VIRIAL, bool F32, int U>
__device__ __forceinline__ void lj_chunk(const int (&jc)[U], const double (&cx)[U], const double (&cy)[U],
                                         const double (&cz)[U], int i, double px, double py, double pz,
                                         const double* h, const double* hi, bool diag, bool wide, const LJP& p,
                                         const LJF& pf,
                                         double& fx, double& fy, double& fz, double* acc, const LJPruneOut& po,
                                         int* __restrict__ prow, int& pc, int lane) {
    bool keep[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
        keep[u] = false;
        if (jc[u] < 0) continue;
        double dx = __dsub_rn(cx[u], px), dy = __dsub_rn(cy[u], py), dz = __dsub_rn(cz[u], pz);
        if (wide) {
            dx = mimg1_rint(dx, h[0], hi[0]);
            dy = mimg1_rint(dy, h[4], hi[4]);
            dz = mimg1_rint(dz, h[8], hi[8]);
        } else if (diag) {
            dx = mimg1(dx, h[0], hi[0]);
            dy = mimg1(dy, h[4], hi[4]);
            dz = mimg1(dz, h[8], hi[8]);
        } else {
            mimg(dx, dy, dz, hi, h);
        }
        if (po.cnt) keep[u] = norm2_rn(dx, dy, dz) <= po.r2;
        if (jc[u] > i) lj_pair<FULL_VIRIAL, F32, true>(dx, dy, dz, p, pf, fx, fy, fz, acc);
        else lj_pair<FULL_VIRIAL, F32, false>(dx, dy, dz, p, pf, fx, fy, fz, acc);
    }
    if (po.cnt) {
#pragma unroll
        for (int u = 0; u < U; u++) {
            const unsigned m = __ballot_sync(kFull, keep[u]);
            if (keep[u]) prow[pc + __popc(m & ((1u << lane) - 1u))] = jc[u];
            pc += __popc(m);
        }
    }
}

// Facc[i] for lj_atom_done, read by lane 0 when the atom's row starts so the
// load is not on the row's tail.
struct LJAcc {
    double x = 0.0, y = 0.0, z = 0.0;
};
__device__ __forceinline__ LJAcc lj_acc_load(const double* __restrict__ Facc, int i, int lane) {
    LJAcc a;
    if (lane == 0) { a.x = Facc[3 * i]; a.y = Facc[3 * i + 1]; a.z = Facc[3 * i + 2]; }
    return a;
}

// End of atom i's row: F[i] = Facc[i] (fa, read at the row's start) + the
// warp's sum (Facc cleared), and for a pruning gather the pruned row's length
// and i's fractional position.
__device__ __forceinline__ void lj_atom_done(int i, double fx, double fy, double fz, double px, double py,
                                             double pz, const double* hi, double* __restrict__ F,
                                             double* __restrict__ Facc, const LJPruneOut& po, int pc, int lane,
                                             const LJAcc& fa) {
    fx = warp_sum(fx); fy = warp_sum(fy); fz = warp_sum(fz);
    if (lane == 0) {
        F[3 * i] = fa.x + fx;
        F[3 * i + 1] = fa.y + fy;
        F[3 * i + 2] = fa.z + fz;
        if (Facc != F) { Facc[3 * i] = 0.0; Facc[3 * i + 1] = 0.0; Facc[3 * i + 2] = 0.0; }
        if (po.cnt) {
            po.cnt[i] = pc;
            po.sb[3 * i] = hi[0] * px + hi[1] * py + hi[2] * pz;
            po.sb[3 * i + 1] = hi[3] * px + hi[4] * py + hi[5] * pz;
            po.sb[3 * i + 2] = hi[6] * px + hi[7] * py + hi[8] * pz;
        }
    }
}

}  // namespace
}  // namespace fmd
