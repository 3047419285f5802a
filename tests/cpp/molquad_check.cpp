// Every atom index of the half-row walk (csrc/molquad.h) for M equal molecules
// of S atoms: each group of G atoms of each molecule, each number of partners,
// each load from the first to the one beyond the last.
#include <algorithm>
#include <cstdio>

#include "molquad.h"

int main() {
    long long reads = 0;
    for (int S = 32; S <= 64; S++)
        for (int G : {1, 4})
            for (int M : {1, 2, 5}) {
                const int n = M * S;
                for (int A = 0; A < M; A++)
                    for (int a0 = 0; a0 < S; a0 += G) {
                        const int i0 = A * S + a0;
                        for (int ns = 0; ns < M - A; ns++)                 // partners A + 1 ..
                            for (int t = 0; t <= ns; t++) {
                                const int j0 = t < ns ? (A + 1 + t) * S : i0;
                                for (int lane = 0; lane < 32; lane++)
                                    for (int u = 0; u < 2; u++, reads++) {
                                        const int j = fmd::quad_atom(t, ns, j0, i0, S, lane, u);
                                        const bool wanted = t < ns && lane + 32 * u < S;
                                        if (j < 0 || j >= n || (wanted && j != j0 + lane + 32 * u)) {
                                            std::printf("S %d G %d M %d: molecule %d, first atom %d, partner %d of %d, "
                                                        "lane %d, slice %d reads atom %d of %d\n",
                                                        S, G, M, A, a0, t, ns, lane, u, j, n);
                                            return 1;
                                        }
                                    }
                            }
                    }
            }
    std::printf("%lld reads within the atoms\n", reads);
    return 0;
}
