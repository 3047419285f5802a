// rebomol.h -- the REBO term by molecules (rebomol.cu).
#pragma once
#include "kernels.h"

namespace fmd {

constexpr int kReboMolAtoms = 128;         // atoms of a molecule, at most

int rebo_mol_blocks(const ReboMol& mol);   // a grid for the molecules
cudaError_t rebo_mol_launch(const ReboMol& mol, const double* pos, const double* hh, const int* cnt, const int* list,
                            int cap, double* F, double* part, int nblocks, const int* gate, int want, bool phys,
                            cudaStream_t st);

}  // namespace fmd
