// mmmol.cu -- MM bonded terms of a system of identical molecules.
//
// The term-wise kernel (mm.cu) gives every term a thread that gathers its
// atoms, takes three minimum images, adds up to 12 FP64 atomics into L2 and
// reads its own copy of the term's parameters: per C60 molecule 6,300 atomics
// and 25 KB of indices and constants that are the same for all of them.  Here
// a block takes a molecule: positions go to shared memory once, relative to
// the molecule's first atom, so a bond vector is three subtractions; the
// terms' constants are one molecule's and stay in the L1; each term stores
// its forces in slots of shared memory, and then four lanes per atom sum the
// atom's slots (listed once per topology) and add them to the accumulator.
// No atomics, and the same sums on every run.  A torsion takes cos and sin of
// m phi - gamma from cos phi and sin phi by m - 1 complex products and the
// stored cos and sin of gamma, instead of atan2, cos and sin.
// Term-wise -> by molecules (B200, C60 crystals of 690 terms a molecule, warm):
// 256 molecules 17.5 -> 9.5 us, a batch of 7,168 molecules 392 -> 188 us.  It is
// bound by latency: 16 warps an SM, FP64 pipe busy 19 %, issue slots 34 %, the
// waits spread over barriers, shared and global loads and dependent FP64.
#include <algorithm>
#include <cmath>
#include <vector>

#include "geom.cuh"
#include "mmmol.h"
#include "pdl.cuh"
#include "step.h"

namespace fmd {
namespace {

// Threads and blocks per SM.  32 replicas of 1,920 to 30,000 atoms: 256 x 2
// (128 registers) 188 us, 320 x 2 194, 256 x 3 (80 registers, spilling) 212,
// 128 x 3 213, 512 x 1 303 us (one molecule at a time waits at its barriers).
constexpr int kMolThreads = 256, kMolBlocks = 2;
constexpr int kGather = 4;                 // lanes per atom of the slot sums
static_assert(kMolThreads >= 32 * kMMNV, "a warp per field of the partials");
constexpr int kPowMax = 8;                 // multiplicities taken by products

struct MolShared {
    double2* xy;                           // [natom] positions
    double *z, *f;                         // [natom], [3][slots + 1] forces
    ushort4* inc;
};
__device__ __forceinline__ MolShared mol_shared(const MMTpl& t, double* dyn) {
    MolShared s;
    s.xy = reinterpret_cast<double2*>(dyn);
    s.z = dyn + 2 * t.natom;
    s.inc = reinterpret_cast<ushort4*>(s.z + t.natom);
    s.f = reinterpret_cast<double*>(s.inc + t.ninc);
    return s;
}

struct Cell {
    double h[9], hi[9];
};

// The terms' view of a molecule: bond vectors and force slots.
struct MolTerms {
    const double2* xy;
    const double* uz;
    double* f;
    int fs;                                // doubles of a force component
    bool far;                              // some atom a quarter of the cell or more from the first
    const Cell* cell;
    __device__ __forceinline__ void vec(int a, int b, double& x, double& y, double& z) const {
        const double2 p = xy[a], q = xy[b];
        x = q.x - p.x; y = q.y - p.y; z = uz[b] - uz[a];
        if (far) mimg(x, y, z, cell->hi, cell->h);
    }
    __device__ __forceinline__ void put(int s, double x, double y, double z) const {
        f[s] = x; f[fs + s] = y; f[2 * fs + s] = z;
    }
};

__device__ __noinline__ double2 multiple_by_angle(double cp, double sp, int mult) {
    double2 v;
    sincos(mult * atan2(sp, cp), &v.y, &v.x);
    return v;
}

// Torsion t of n (MM:503-601, the sign sg as in mm.cu's torsion()): forces
// into slots t + {0, 1, 2, 3} n; returns the energy.
__device__ __forceinline__ double mol_torsion(const MolTerms& m, ushort4 id, double4 c, int t, int n, double sg) {
    double b1x, b1y, b1z, b2x, b2y, b2z, b3x, b3y, b3z;
    m.vec(id.x, id.y, b1x, b1y, b1z);
    m.vec(id.y, id.z, b2x, b2y, b2z);
    m.vec(id.z, id.w, b3x, b3y, b3z);
    const double mx = b1y * b2z - b1z * b2y, my = b1z * b2x - b1x * b2z, mz = b1x * b2y - b1y * b2x;
    const double nx = b2y * b3z - b2z * b3y, ny = b2z * b3x - b2x * b3z, nz = b2x * b3y - b2y * b3x;
    const double mm = mx * mx + my * my + mz * mz, nn = nx * nx + ny * ny + nz * nz;
    if (mm < 1e-20 || nn < 1e-20) {
#pragma unroll
        for (int k = 0; k < 4; k++) m.put(t + k * n, 0.0, 0.0, 0.0);
        return 0.0;
    }
    const double rm = rsqrt(mm), rn = rsqrt(nn), bb = b2x * b2x + b2y * b2y + b2z * b2z, rb = rsqrt(bb);
    const double b2len = bb * rb, rmn = rm * rn;
    double cp = (mx * nx + my * ny + mz * nz) * rmn, sp = (mx * b3x + my * b3y + mz * b3z) * b2len * rmn;
    const double unit = fma(-0.5, fma(cp, cp, sp * sp), 1.5);      // to unit length, as the angle from atan2 is
    cp *= unit; sp *= unit;
    const int mult = (int)c.w, am = abs(mult);
    double cm = 1.0, sm = 0.0;
    if (am <= kPowMax) {
        if (am > 0) { cm = cp; sm = sp; }
        for (int k = 1; k < am; k++) {
            const double x = cm * cp - sm * sp;
            sm = sm * cp + cm * sp;
            cm = x;
        }
        if (mult < 0) sm = -sm;
    } else {
        const double2 v = multiple_by_angle(cp, sp, mult);
        cm = v.x; sm = v.y;
    }
    const double e = 0.5 * c.x * (1.0 + (cm * c.y + sm * c.z));
    const double dphi = -0.5 * c.x * c.w * (sm * c.y - cm * c.z);
    const double g1 = dphi * b2len * (rm * rm), g4 = -dphi * b2len * (rn * rn);
    const double f1x = g1 * mx, f1y = g1 * my, f1z = g1 * mz;
    const double f4x = g4 * nx, f4y = g4 * ny, f4z = g4 * nz;
    const double ib = sg * (rb * rb);
    const double ci = ib * (b1x * b2x + b1y * b2y + b1z * b2z), ck = ib * (b2x * b3x + b2y * b3y + b2z * b3z);
    const double dx = ci * f1x - ck * f4x, dy = ci * f1y - ck * f4y, dz = ci * f1z - ck * f4z;
    m.put(t, f1x, f1y, f1z);
    m.put(t + n, dx - f1x, dy - f1y, dz - f1z);
    m.put(t + 2 * n, -f4x - dx, -f4y - dy, -f4z - dz);
    m.put(t + 3 * n, f4x, f4y, f4z);
    return e;
}

// Angle t of n (MM:455-492): forces into slots s + t + {0, 1, 2} n.
__device__ __forceinline__ double mol_angle(const MolTerms& m, ushort4 id, double2 c, int s, int n, double sg) {
    double u0, u1, u2, v0, v1, v2;
    m.vec(id.y, id.x, u0, u1, u2);
    m.vec(id.y, id.z, v0, v1, v2);
    const double uu = u0 * u0 + u1 * u1 + u2 * u2, vv = v0 * v0 + v1 * v1 + v2 * v2;
    if (sqrt(uu) < 1e-10 || sqrt(vv) < 1e-10) {
#pragma unroll
        for (int k = 0; k < 3; k++) m.put(s + k * n, 0.0, 0.0, 0.0);
        return 0.0;
    }
    const double ru = rsqrt(uu), rv = rsqrt(vv), ruv = ru * rv;
    double cc = (u0 * v0 + u1 * v1 + u2 * v2) * ruv;
    cc = cc > 0.999999 ? 0.999999 : (cc < -0.999999 ? -0.999999 : cc);
    const double dth = acos(cc) - c.y;
    const double dV = sg * (-c.x * dth * rsqrt(1.0 - cc * cc + 1e-30));
    const double a = dV * ruv, bu = dV * cc * (ru * ru), bv = dV * cc * (rv * rv);
    const double i0 = a * v0 - bu * u0, i1 = a * v1 - bu * u1, i2 = a * v2 - bu * u2;
    const double k0 = a * u0 - bv * v0, k1 = a * u1 - bv * v1, k2 = a * u2 - bv * v2;
    m.put(s, i0, i1, i2);
    m.put(s + n, -(i0 + k0), -(i1 + k1), -(i2 + k2));
    m.put(s + 2 * n, k0, k1, k2);
    return 0.5 * c.x * dth * dth;
}

// Molecules blk, blk + nblk, ...; partials into part[blk].
__device__ __forceinline__ void mol_bonded_body(const MMTpl& t, int physical, const double* __restrict__ pos,
                                                const double* __restrict__ hh, double* __restrict__ F,
                                                double* __restrict__ part, int blk, int nblk, double* dyn,
                                                Cell& cell) {
    const int tid = threadIdx.x;
    const MolShared sh = mol_shared(t, dyn);
    for (int k = tid; k < t.ninc; k += kMolThreads) sh.inc[k] = t.inc[k];
    const int fs = t.slots + 1;
    if (tid < 3) sh.f[tid * fs + t.slots] = 0.0;
    double acc[kMMNV];                     // Eb Ea Ed Ei W00 W11 W22
#pragma unroll
    for (int k = 0; k < kMMNV; k++) acc[k] = 0.0;
    const double sg = physical ? -1.0 : 1.0;
    const int total = t.ntor + t.nang + t.nb;
    FMD_PDL_WAIT();
    if (tid < 9) { cell.h[tid] = hh[tid]; cell.hi[tid] = hh[9 + tid]; }
    __syncthreads();
    MolTerms mt;
    mt.xy = sh.xy; mt.uz = sh.z; mt.f = sh.f; mt.fs = fs; mt.cell = &cell;
    const int s_ang = 4 * t.ntor, s_bond = s_ang + 3 * t.nang;
    for (int m = blk; m < t.nmol; m += nblk) {
        const size_t base = 3 * (size_t)m * t.natom;
        const double p0 = pos[base], p1 = pos[base + 1], p2 = pos[base + 2];
        int far = 0;
        for (int a = tid; a < t.natom; a += kMolThreads) {
            const double* p = pos + base + 3 * a;
            double x = p[0] - p0, y = p[1] - p1, z = p[2] - p2, s[3];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                s[k] = dot3_rn(cell.hi[3 * k], cell.hi[3 * k + 1], cell.hi[3 * k + 2], x, y, z);
                const double r = round(s[k]);
                far |= !(fabs(s[k] - r) < 0.25 - 1e-9);
                s[k] = r;
            }
            x -= dot3_rn(cell.h[0], cell.h[1], cell.h[2], s[0], s[1], s[2]);
            y -= dot3_rn(cell.h[3], cell.h[4], cell.h[5], s[0], s[1], s[2]);
            z -= dot3_rn(cell.h[6], cell.h[7], cell.h[8], s[0], s[1], s[2]);
            sh.xy[a] = make_double2(x, y);
            sh.z[a] = z;
        }
        // within a quarter of the cell of the first atom, the atoms' differences are nearest images
        mt.far = __syncthreads_or(far) != 0;
#pragma unroll 1
        for (int q = tid; q < total; q += kMolThreads) {
            const ushort4 id = t.id[q];
            if (q < t.ntor) {
                const double e = mol_torsion(mt, id, t.torp[q], q, t.ntor, sg);
                acc[2] += q < t.ndih ? e : 0.0;
                acc[3] += q < t.ndih ? 0.0 : e;
            } else if (q < t.ntor + t.nang) {
                const int a = q - t.ntor;
                acc[1] += mol_angle(mt, id, t.angp[a], s_ang + a, t.nang, sg);
            } else {                                              // MM:384-447
                const int b = q - t.ntor - t.nang;
                const double2 c = t.bondp[b];
                double dx, dy, dz;
                mt.vec(id.x, id.y, dx, dy, dz);
                const double r = sqrt(dx * dx + dy * dy + dz * dz);
                const bool on = !(r < 1e-10);
                const double dr = on ? r - c.y : 0.0, fm = on ? sg * (-c.x * dr / r) : 0.0;
                const double fx = fm * dx, fy = fm * dy, fz = fm * dz;
                acc[0] += 0.5 * c.x * dr * dr;
                acc[4] += dx * fx; acc[5] += dy * fy; acc[6] += dz * fz;
                mt.put(s_bond + b, fx, fy, fz);
                mt.put(s_bond + t.nb + b, -fx, -fy, -fz);
            }
        }
        __syncthreads();
        for (int q = tid; q < ((kGather * t.natom + 31) & ~31); q += kMolThreads) {
            const int a = q / kGather, k = q % kGather;
            const bool mine = a < t.natom && k < 3;
            const double f0 = mine ? F[base + 3 * a + k] : 0.0;
            double x = 0.0, y = 0.0, z = 0.0;
            if (a < t.natom)
                for (int g = t.inc_off[a] + k, end = t.inc_off[a + 1]; g < end; g += kGather) {
                    const ushort4 j = sh.inc[g];
                    const double* f = sh.f;
                    x += (f[j.x] + f[j.y]) + (f[j.z] + f[j.w]);
                    f += fs;
                    y += (f[j.x] + f[j.y]) + (f[j.z] + f[j.w]);
                    f += fs;
                    z += (f[j.x] + f[j.y]) + (f[j.z] + f[j.w]);
                }
#pragma unroll
            for (int o = 1; o < kGather; o <<= 1) {
                x += __shfl_xor_sync(kFull, x, o);
                y += __shfl_xor_sync(kFull, y, o);
                z += __shfl_xor_sync(kFull, z, o);
            }
            if (mine) F[base + 3 * a + k] = f0 + (k == 0 ? x : (k == 1 ? y : z));
        }
    }
    // partials: a warp per field
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kMMNV; k++) dyn[k * kMolThreads + tid] = acc[k];
    __syncthreads();
    if (tid < 32 * kMMNV) {
        double v = 0.0;
#pragma unroll
        for (int k = 0; k < kMolThreads / 32; k++) v += dyn[(tid >> 5) * kMolThreads + 32 * k + (tid & 31)];
        v = warp_sum(v);
        if ((tid & 31) == 0) part[(size_t)blk * kMMNV + (tid >> 5)] = v;
    }
}

__global__ void __launch_bounds__(kMolThreads, kMolBlocks)
k_mm_mol(MMTpl t, int physical, const double* __restrict__ pos, const double* __restrict__ hh, double* __restrict__ F,
         double* __restrict__ part) {
    extern __shared__ double dyn[];
    __shared__ Cell cell;
    mol_bonded_body(t, physical, pos, hh, F, part, blockIdx.x, gridDim.x, dyn, cell);
}

__global__ void __launch_bounds__(kMolThreads, kMolBlocks)
k_b_mm_mol(const StepArrays* __restrict__ As, const int* __restrict__ off, int R) {
    extern __shared__ double dyn[];
    __shared__ Cell cell;
    const int r = batch_rep(off, R, blockIdx.x);
    const StepArrays& a = As[r];
    __shared__ MMTpl tpl;                  // shared: not in registers beside the terms
    if (threadIdx.x == 0) tpl = a.topo.tpl;
    __syncthreads();
    mol_bonded_body(tpl, a.topo.physical, a.pos, a.S->h, a.Facc, a.part_f1, blockIdx.x - off[r],
                    off[r + 1] - off[r], dyn, cell);
}

template <class K>
cudaError_t allow_smem(K kernel, size_t bytes) {
    return bytes > (48u << 10)
               ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMolMaxShared)
               : cudaSuccess;
}

}  // namespace

size_t mm_mol_shared(const MMTpl& t) {
    return std::max(sizeof(double) * 3 * ((size_t)t.slots + 1 + t.natom) + sizeof(ushort4) * (size_t)t.ninc,
                    sizeof(double) * kMMNV * kMolThreads);
}

int mm_mol_blocks(const MMTpl& t) { return std::max(1, std::min(kForceBlocks, t.nmol)); }

cudaError_t mm_mol_launch(const MMTpl& t, int physical, const double* pos, const double* hh, double* Facc,
                          double* part, cudaStream_t st) {
    const size_t smem = mm_mol_shared(t);
    cudaError_t e = allow_smem(k_mm_mol, smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(k_mm_mol, dim3(mm_mol_blocks(t)), dim3(kMolThreads), smem, st, t, physical, pos, hh, Facc, part);
}

cudaError_t batch_mm_mol_launch(const StepArrays* As, const int* off, int R, int nblocks, size_t smem,
                                cudaStream_t st) {
    cudaError_t e = allow_smem(k_b_mm_mol, smem);
    if (e != cudaSuccess) return e;
    k_b_mm_mol<<<nblocks, kMolThreads, smem, st>>>(As, off, R);
    return cudaGetLastError();
}

int mm_copies(const fmd_mm_topology& t, int na, const int* mol_id) {
    int natom = 1;
    while (natom < na && mol_id[natom] == mol_id[0]) natom++;
    if (na % natom) return 0;
    const int nmol = na / natom;
    auto idx = [&](const int* a, int n) {
        const int per = n / nmol;
        for (int k = 0; k < n; k++) {
            const int m = k / per;
            if (a[k] != a[k - m * per] + m * natom || a[k - m * per] >= natom) return false;
        }
        return true;
    };
    auto same = [&](const auto* a, int n) {
        const int per = n / nmol;
        for (int k = per; k < n; k++)
            if (!(a[k] == a[k - per])) return false;
        return true;
    };
    if (t.nb % nmol || t.nang % nmol || t.ndih % nmol || t.nimp % nmol) return 0;
    const bool ok = idx(t.b_i0, t.nb) && idx(t.b_i1, t.nb) && same(t.b_kb, t.nb) && same(t.b_r0, t.nb) &&
                    idx(t.ang_i0, t.nang) && idx(t.ang_i1, t.nang) && idx(t.ang_i2, t.nang) &&
                    same(t.ang_kth, t.nang) && same(t.ang_th0, t.nang) && idx(t.dih_i0, t.ndih) &&
                    idx(t.dih_i1, t.ndih) && idx(t.dih_i2, t.ndih) && idx(t.dih_i3, t.ndih) &&
                    same(t.dih_vn, t.ndih) && same(t.dih_mult, t.ndih) && same(t.dih_gamma, t.ndih) &&
                    idx(t.imp_i0, t.nimp) && idx(t.imp_i1, t.nimp) && idx(t.imp_i2, t.nimp) &&
                    idx(t.imp_i3, t.nimp) && same(t.imp_ki, t.nimp) && same(t.imp_gamma, t.nimp);
    return ok ? natom : 0;
}

bool mm_tpl_build(const fmd_mm_topology& t, int copies, int natom, MMTplHost& o) {
    const int nb = t.nb / copies, nang = t.nang / copies, ndih = t.ndih / copies, nimp = t.nimp / copies;
    MMTpl& d = o.dims;
    d = MMTpl{};
    const long long slots = 4LL * (ndih + nimp) + 3LL * nang + 2LL * nb;
    if (slots < 1 || slots > 65534) return false;
    d.natom = natom; d.nb = nb; d.nang = nang; d.ndih = ndih; d.ntor = ndih + nimp; d.slots = (int)slots;
    std::vector<std::vector<unsigned short>> at(natom);
    auto list = [&](int atom, int slot) { at[atom].push_back((unsigned short)slot); };
    auto atoms = [&](int a, int b, int c, int e) {
        o.id.push_back(make_ushort4((unsigned short)a, (unsigned short)b, (unsigned short)c, (unsigned short)e));
    };
    auto torsion = [&](int a1, int a2, int a3, int a4, double v, double gamma, int mult) {
        const int q = (int)o.torp.size();
        atoms(a1, a2, a3, a4);
        o.torp.push_back(make_double4(v, std::cos(gamma), std::sin(gamma), (double)mult));
        list(a1, q); list(a2, q + d.ntor); list(a3, q + 2 * d.ntor); list(a4, q + 3 * d.ntor);
    };
    for (int k = 0; k < ndih; k++)
        torsion(t.dih_i0[k], t.dih_i1[k], t.dih_i2[k], t.dih_i3[k], t.dih_vn[k], t.dih_gamma[k], t.dih_mult[k]);
    for (int k = 0; k < nimp; k++)                                // MM:610-709, order c1,c0,c2,c3
        torsion(t.imp_i1[k], t.imp_i0[k], t.imp_i2[k], t.imp_i3[k], t.imp_ki[k], t.imp_gamma[k], 2);
    const int s_ang = 4 * d.ntor, s_bond = s_ang + 3 * nang;
    for (int k = 0; k < nang; k++) {
        atoms(t.ang_i0[k], t.ang_i1[k], t.ang_i2[k], 0);
        o.angp.push_back(make_double2(t.ang_kth[k], t.ang_th0[k]));
        list(t.ang_i0[k], s_ang + k); list(t.ang_i1[k], s_ang + nang + k); list(t.ang_i2[k], s_ang + 2 * nang + k);
    }
    for (int k = 0; k < nb; k++) {
        atoms(t.b_i0[k], t.b_i1[k], 0, 0);
        o.bondp.push_back(make_double2(t.b_kb[k], t.b_r0[k]));
        list(t.b_i0[k], s_bond + k); list(t.b_i1[k], s_bond + nb + k);
    }
    o.inc_off.push_back(0);
    for (auto& l : at) {
        while (l.size() % (4 * kGather)) l.push_back((unsigned short)d.slots);
        for (size_t k = 0; k < l.size(); k += 4) o.inc.push_back(make_ushort4(l[k], l[k + 1], l[k + 2], l[k + 3]));
        o.inc_off.push_back((int)o.inc.size());
    }
    d.ninc = (int)o.inc.size();
    return mm_mol_shared(d) <= kMolMaxShared;
}

}  // namespace fmd
