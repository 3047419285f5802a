// mmmol.h -- MM bonded terms of a system of identical molecules (mmmol.cu).
#pragma once
#include <cstddef>
#include <vector>

#include "../../include/fullermd.h"
#include "kernels.h"

namespace fmd {

struct StepArrays;

// Shared memory of a block, at most: two blocks fit an SM.
constexpr size_t kMolMaxShared = 108u << 10;

// One molecule's terms on the host, as MMTpl holds them on the device.
struct MMTplHost {
    MMTpl dims;
    std::vector<ushort4> id;
    std::vector<double4> torp;
    std::vector<double2> angp, bondp;
    std::vector<int> inc_off;
    std::vector<ushort4> inc;              // inc_off counts these
};

// Atoms per molecule when the flat topology t of na atoms is that of equal
// molecules, copies in order and each term kind molecule-major; else 0.
int mm_copies(const fmd_mm_topology& t, int na, const int* mol_id);
// The plan of the first of the copies in t (its terms come first in each
// kind); false when a block's shared memory does not hold a molecule's force
// slots.
bool mm_tpl_build(const fmd_mm_topology& t, int copies, int natom, MMTplHost& o);

size_t mm_mol_shared(const MMTpl& t);
int mm_mol_blocks(const MMTpl& t);         // partial records
cudaError_t mm_mol_launch(const MMTpl& t, int physical, const double* pos, const double* hh, double* Facc,
                          double* part, cudaStream_t st);
// Every replica by molecules; smem: the largest of the replicas' blocks.
cudaError_t batch_mm_mol_launch(const StepArrays* As, const int* off, int R, int nblocks, size_t smem,
                                cudaStream_t st);

}  // namespace fmd
