// ljprune.cuh -- the device-side decision of the pruned LJ rows (ljprune.cu).
#pragma once
#include <cuda_runtime.h>

#include <cmath>

namespace fmd {

// What the pruned rows' memory holds (words[1]): rows of single atoms or of
// clusters, and the buffer they were built with.  A gather that finds other
// rows there than its own (a replica batch and its system may use different
// ones) builds its own first.
constexpr unsigned long long kRowsAtoms = 1ull, kRowsClusters = 2ull;
__host__ __device__ inline unsigned long long lj_rows_tag(unsigned long long kind, double delta) {
    union { double d; unsigned long long u; } b;
    b.d = delta;
    return (b.u & ~3ull) | kind;
}

// 1 when the memory does not hold rows of this kind, or the pruned rows may miss a pair now within the cutoff: the cell is
// not diagonal (now or at the prune), or k (rc + delta) + 2u >= delta less a
// rounding margin, u the largest displacement since the last prune (bits in
// words[0], raised by the drift; a list build stores a huge value) and k the
// largest relative change of a cell edge since then.  Every block of the
// gather and the step's reduction evaluate it on the same, unchanged inputs.
__device__ __forceinline__ bool lj_prune_needed(const unsigned long long* words, const double* hh, const double* hb,
                                                double delta, double rc, unsigned long long kind) {
    // every load first, so that they cost one latency together
    const unsigned long long tag = words[1];
    const double u = __longlong_as_double((long long)words[0]);
    double h[9], b[9];
#pragma unroll
    for (int a = 0; a < 9; a++) { h[a] = hh[a]; b[a] = hb[a]; }
    double k = 0.0;
#pragma unroll
    for (int a = 0; a < 3; a++) k = fmax(k, fabs(h[4 * a] - b[4 * a]) / fabs(b[4 * a]));
    bool diag = true;
#pragma unroll
    for (int a = 0; a < 9; a++)
        if (a % 4 != 0) diag = diag && h[a] == 0.0 && b[a] == 0.0;
    return tag != lj_rows_tag(kind, delta) || !(diag && k * (rc + delta) + 2.0 * u < delta - 1e-6);
}

}  // namespace fmd
