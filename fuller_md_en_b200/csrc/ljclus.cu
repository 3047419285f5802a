// ljclus.cu -- the atomistic LJ gather over cluster rows.
//
// The row gather (airebo.cu) gives each atom a warp that reads every partner
// position for one pair.  At 30,000 atoms that is 10.9 M scattered 24-byte
// reads a step, and the L1's rate for them (about one entry a cycle and SM)
// alone takes 37 us.  Here kClusG neighbouring atoms of one molecule form a
// cluster with one row, the union of their pruned rows: a partner is read
// once and meets all atoms of the cluster, whose pair terms are independent
// chains in one instruction stream.  Walk over pruned rows, row gather ->
// cluster gather (B200, C60 crystals, warm): 67.5 -> 38.0 us at 30,000 atoms,
// 259 -> 139 us at 122,880; FP32 pairs at 122,880: 297 -> 157 us.  It is bound
// by FP64 issue and latency: the FP64 pipe is busy 57 % of the time, half of
// the instructions are FP64.  Clusters of 3 and 5 atoms took 156 and 159 us
// where 4 took 149: fewer atoms share a partner less often, more spill.
//
// Row entry: bits 0-21 the partner j, bits 22-26 the cluster's atoms whose
// row lists j (so the reference's truncated rows stay exactly that), bits
// 27-31 the image of j (its three cell offsets -1, 0, 1 in base 3).
// Partners of higher molecules come first (j > i: these entries count energy
// and virial), filled up to whole slices of 32 with idle entries, then those
// of lower molecules.
//
// Images.  The offsets are those of the nearest image when the row is built.
// Until the next build the gather reads positions that the drift follows
// without wrapping (upos), so an entry's image, and those of the cluster's
// atoms from its first, stay what they were and a pair costs three
// subtractions instead of a rounding per axis.  With edges beyond 2 R, R = rc
// + delta (lj_clus_mode), at most one image of j is within R of an atom.  The
// nearest image from the cluster's first atom serves all its atoms when the
// edges also exceed 2 (R + their distance from it); otherwise j may need an
// entry for each of two images.
//
// Rows are built from the list builder's candidate bitmaps (molnlist.cu), one
// warp per cluster: for each partner molecule the lanes take its atoms, the
// bitmaps say which of the cluster's rows list them, and the entries within
// rc + delta now are kept.  When they may be used and must be rebuilt is the
// pruned rows' rule (ljprune.cu).
//
// Rows of atoms.  Where cluster rows cannot be had (a build by cells, a cell that
// is not diagonal or too narrow) or do not pay (atoms so fast that most
// evaluations build rows: molnlist.cu decides at each list build), the same
// kernel does what the row gather does, an atom a warp over full and pruned
// rows (atom_rows), with the pair terms of a chunk free of branches: with 12
// warps an SM the chunk's independent chains stand in for the row gather's
// warps.  30,000 atoms, pruning / walking: 126 / 66 us (the row gather 122 /
// 67; with its branches here 155 / 82), FP32 pairs 132 / 72 (200 / 109).  Where
// nearly every evaluation prunes, the full rows are walked without writing
// pruned ones, and the block's last atoms then split their rows over its warps:
// 1,920 atoms 13.5 us instead of 16.7.
//
// Virial: sum over pairs of fm d (x) d with d = d0 - x_g, d0 the partner
// from the cluster's first atom and x_g atom g from it, is
// sum d0 (x) (sum_g fm d) - sum_g x_g (x) (sum fm d): per entry one product of
// the cluster's summed force instead of one per pair.
#include <algorithm>
#include <cmath>
#include <limits>
#include <type_traits>
#include <vector>

#include "ljclus.cuh"
#include "ljclus.h"
#include "ljpair.cuh"
#include "ljrow.cuh"
#include "pdl.cuh"
#include "step.h"

namespace fmd {
namespace {

// Warps per block and blocks per SM.  FP64: one block of 12 warps (164
// registers, no spills) took 138 us at 122,880 atoms, two of 8 (128
// registers, spilling) 149 us.  FP32 pairs: 169 us and 157 us.
template <bool F32> constexpr int kWarps = F32 ? 8 : 12;
template <bool F32> constexpr int kBlocks = F32 ? 2 : 1;
constexpr int kMaxWarps = 12;
constexpr int kAtomUnroll = 4;             // entries per lane in flight of rows of atoms
// Slices per trip: saves the feed's register moves.  1 / 2 / 4, walk in us: FP64
// 30,000 atoms 37.8 / 37.9 / 37.2, 122,880 atoms 141 / 141 / 136.5, 16 replicas of
// 215,000 in all (a step) 500 / 492 / 462; FP32 pairs 44.8 / 42.9 / 43.8.
template <bool F32> constexpr int kClusUnroll = F32 ? 2 : 4;
constexpr int kMaskBit = 22, kCodeBit = 27;
constexpr unsigned kAtomBits = (1u << kMaskBit) - 1u;
static_assert(kClusG <= kCodeBit - kMaskBit, "mask bits of a row entry");
static_assert(kClusMaxAtoms == 1 << kMaskBit, "partner bits of a row entry");

constexpr int kCandBatch = 64, kCandMax = kCandBatch + 64;

struct ClusShared {
    double sm[32 * kNV];
    double hh[18];
    double shift[32][4];                       // image offsets of each code; from 27: far away
    int perm[64 + kClusG];                     // LJClus::perm (molecules of up to 64 atoms)
    double part[kMaxWarps][3 * kClusG];       // force sums of a row split over warps
    unsigned cand[kMaxWarps][kCandMax];        // candidates of the row being built
};

// What an evaluation is of (the kernel's parameter; of a batch, in shared memory).
struct ClusArgs {
    LJClus c;
    LJPruneOut po;
    LJP p;
    const double *pos, *hh;
    double *F, *Facc, *part;
    int na, nrec, mode;
};

// The cluster's atoms (-1: none) and their positions: the first absolute, the
// others from it (nearest image).
struct Cluster {
    int id[kClusG];
    double x0, y0, z0;
    double x[kClusG], y[kClusG], z[kClusG];
};

__device__ __forceinline__ void cluster_ids(const LJClus& c, int k, const int* perm, Cluster& q) {
    const int m = k / c.cpm, kk = k - m * c.cpm;
#pragma unroll
    for (int g = 0; g < kClusG; g++) {
        const int a = perm[kk * kClusG + g];
        q.id[g] = a < 0 ? -1 : m * c.S + a;
    }
}

// With the images of the last build (img: 5 bits per atom after the first).
__device__ __forceinline__ Cluster load_cluster(const LJClus& c, int k, int img, const double* __restrict__ x,
                                                const ClusShared& s) {
    Cluster q;
    cluster_ids(c, k, s.perm, q);
    const int i0 = q.id[0];
    q.x0 = x[3 * i0]; q.y0 = x[3 * i0 + 1]; q.z0 = x[3 * i0 + 2];
    q.x[0] = q.y[0] = q.z[0] = 0.0;
#pragma unroll
    for (int g = 1; g < kClusG; g++) {
        const int i = q.id[g] < 0 ? i0 : q.id[g];
        const double* sh = s.shift[(img >> (5 * (g - 1))) & 31];
        q.x[g] = (x[3 * i] - sh[0]) - q.x0;
        q.y[g] = (x[3 * i + 1] - sh[1]) - q.y0;
        q.z[g] = (x[3 * i + 2] - sh[2]) - q.z0;
    }
    return q;
}

__device__ __forceinline__ unsigned image_code(double kx, double ky, double kz) {
    return (unsigned)((int)kx + 1 + 3 * ((int)ky + 1) + 9 * ((int)kz + 1)) & 31u;
}

// Idle entries from out to the end of its slice; returns that end.
constexpr unsigned kIdle = 27u << kCodeBit;
__device__ __forceinline__ int fill_slice(int* row, int out, int stride, int lane) {
    const int end = (out + 31) & ~31;
    if (out + lane < end && out + lane < stride) row[out + lane] = (int)kIdle;
    return end;
}

// The row being built by a warp: candidates (partner and list bits) gather in
// buf and are tested kCandBatch at a time, so that the lanes of a test are
// full and each has two positions in flight.
struct RowBuild {
    const Cluster& q;
    const double* pos;
    const double* hh;
    double r2;
    bool one;                                  // one image of a partner serves the cluster
    unsigned* buf;
    int* row;
    int stride, lane;
    int nbuf = 0, out = 0;
    unsigned per[(kClusG + 1) / 2];            // kept entries per atom, two 16-bit counts a word (lane sums)
    unsigned inc[(kClusG + 1) / 2];            // candidates of lower molecules per atom, likewise

    // Candidates buf[0 .. n), n <= kCandBatch: those within the radius go to the row.
    __device__ __forceinline__ void test(int n) {
        __syncwarp();
        const double* hi = hh + 9;
        unsigned c[2];
        double px[2], py[2], pz[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            c[u] = lane + 32 * u < n ? buf[lane + 32 * u] : 0u;
            const double* p = pos + 3 * (size_t)(c[u] & kAtomBits);
            px[u] = p[0]; py[u] = p[1]; pz[u] = p[2];
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const double rx = px[u] - q.x0, ry = py[u] - q.y0, rz = pz[u] - q.z0;
            double kx = rint(rx * hi[0]), ky = rint(ry * hi[4]), kz = rint(rz * hi[8]);
            double dx = fma(-hh[0], kx, rx), dy = fma(-hh[4], ky, ry), dz = fma(-hh[8], kz, rz);
            unsigned keep = 0u, code[kClusG];
            code[0] = image_code(kx, ky, kz);
#pragma unroll
            for (int g = 0; g < kClusG; g++) {
                if (!one && g) {
                    kx = rint((rx - q.x[g]) * hi[0]); ky = rint((ry - q.y[g]) * hi[4]); kz = rint((rz - q.z[g]) * hi[8]);
                    dx = fma(-hh[0], kx, rx); dy = fma(-hh[4], ky, ry); dz = fma(-hh[8], kz, rz);
                    code[g] = image_code(kx, ky, kz);
                }
                const double ux = dx - q.x[g], uy = dy - q.y[g], uz = dz - q.z[g];
                if (ux * ux + uy * uy + uz * uz <= r2) keep |= 1u << g;
            }
            keep &= c[u] >> kMaskBit;
#pragma unroll
            for (int g = 0; g < kClusG; g++) per[g / 2] += ((keep >> g) & 1u) << (16 * (g & 1));
            do {                               // a second pass only where images differ
                unsigned now = keep, at = code[0];
                if (!one) {
                    now = 0u;
#pragma unroll
                    for (int g = kClusG - 1; g >= 0; g--)
                        if ((keep >> g) & 1u) at = code[g];
#pragma unroll
                    for (int g = 0; g < kClusG; g++)
                        if (((keep >> g) & 1u) && code[g] == at) now |= 1u << g;
                }
                const unsigned b = __ballot_sync(kFull, now != 0u);
                const int o = out + __popc(b & ((1u << lane) - 1u));
                if (now && o < stride) row[o] = (int)((c[u] & kAtomBits) | (now << kMaskBit) | (at << kCodeBit));
                out += __popc(b);
                keep &= ~now;
            } while (!one && __any_sync(kFull, keep != 0u));
        }
        __syncwarp();
    }
    // The lane's candidate j with list bits mk (0: none).
    __device__ __forceinline__ void add(unsigned mk, int j) {
        const unsigned b = __ballot_sync(kFull, mk != 0u);
        if (mk) buf[nbuf + __popc(b & ((1u << lane) - 1u))] = (unsigned)j | (mk << kMaskBit);
        nbuf += __popc(b);
    }
    // Tests a full batch (all: whatever there is).
    __device__ __forceinline__ void flush(bool all) {
        while (nbuf >= kCandBatch || (all && nbuf > 0)) {
            const int n = min(nbuf, kCandBatch);
            test(n);
            nbuf -= n;
            unsigned rest[2];
#pragma unroll
            for (int u = 0; u < 2; u++) rest[u] = lane + 32 * u < nbuf ? buf[n + lane + 32 * u] : 0u;
            __syncwarp();
#pragma unroll
            for (int u = 0; u < 2; u++)
                if (lane + 32 * u < nbuf) buf[lane + 32 * u] = rest[u];
        }
    }
};

// Builds cluster k's row from the candidate bitmaps at positions pos, and
// writes its atoms' pruned-row lengths, fractional and followed positions.
__device__ __forceinline__ void build_row(const LJClus& c, int k, const double* __restrict__ pos, ClusShared& sh,
                                          const LJPruneOut& po, int w, int lane) {
    const int m = k / c.cpm;
    const double* hh = sh.hh;
    const double* hi = hh + 9;
    Cluster q;
    cluster_ids(c, k, sh.perm, q);
    const int i0 = q.id[0];
    q.x0 = pos[3 * i0]; q.y0 = pos[3 * i0 + 1]; q.z0 = pos[3 * i0 + 2];
    q.x[0] = q.y[0] = q.z[0] = 0.0;
    double far2 = 0.0;
    unsigned img = 0u;
#pragma unroll
    for (int g = 1; g < kClusG; g++) {
        const int i = q.id[g] < 0 ? i0 : q.id[g];
        const double ux = pos[3 * i] - q.x0, uy = pos[3 * i + 1] - q.y0, uz = pos[3 * i + 2] - q.z0;
        const double kx = rint(ux * hi[0]), ky = rint(uy * hi[4]), kz = rint(uz * hi[8]);
        q.x[g] = fma(-hh[0], kx, ux); q.y[g] = fma(-hh[4], ky, uy); q.z[g] = fma(-hh[8], kz, uz);
        img |= image_code(kx, ky, kz) << (5 * (g - 1));
        far2 = fmax(far2, q.x[g] * q.x[g] + q.y[g] * q.y[g] + q.z[g] * q.z[g]);
    }
    int a[kClusG];                             // the atoms within the molecule
    bool lo = false, hi2 = false;              // some of them in its first 32, after them
#pragma unroll
    for (int g = 0; g < kClusG; g++) {
        a[g] = q.id[g] < 0 ? -1 : q.id[g] - m * c.S;
        if (a[g] >= 0) { lo |= a[g] < 32; hi2 |= a[g] >= 32; }
    }
    RowBuild r{q, pos, hh, po.r2, fmin(hh[0], fmin(hh[4], hh[8])) > 2.0 * (sqrt(po.r2) + sqrt(far2)) + 0.1,
               sh.cand[w], c.rows + (size_t)k * c.stride, c.stride, lane};
#pragma unroll
    for (int g = 0; g < (kClusG + 1) / 2; g++) r.per[g] = r.inc[g] = 0u;
    const int np = c.npart[m];
    const int* pa = c.part + (size_t)m * c.pmax;
    const int* rv = c.rev + (size_t)m * c.pmax;
    int nlow = 0;
    for (int q0 = 0; q0 < np; q0 += 32) {
        const int B = q0 + lane < np ? pa[q0 + lane] : 0x7fffffff;
        nlow += __popc(__ballot_sync(kFull, B < m));
    }
    // One step per partner, higher molecules first.  For those lane 2 p + h
    // holds the cluster's words for half h of the p-th of 16 partners (the
    // atoms of that half in each cluster atom's row); for a lower molecule
    // the lanes hold the words of its atoms, loaded one partner ahead.
    const int nup = np - nlow;
    int nown = 0;
    unsigned own[kClusG], some = 0u;
    int j0 = 0;
    unsigned nw[2][2] = {{0u, 0u}, {0u, 0u}};
    int nB = 0;
    auto load_lower = [&](int s) {
        nB = pa[s];
        const unsigned* bw = c.bm + ((size_t)nB * 2 * c.pmax + 2 * rv[s]) * c.S;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int b = 32 * h + lane;
            nw[h][0] = lo && b < c.S ? bw[b] : 0u;
            nw[h][1] = hi2 && b < c.S ? bw[c.S + b] : 0u;
        }
    };
    if (nlow > 0) load_lower(0);
#pragma unroll
    for (int g = 0; g < kClusG; g++) own[g] = 0u;
#pragma unroll 1
    for (int t = 0; t < np; t++) {
        unsigned mk[2] = {0u, 0u};
        int j = 0;
        if (t < nup) {
            if ((t & 15) == 0) {
                const int p = t + (lane >> 1), h = lane & 1;
                unsigned any = 0u;
                const unsigned* bw = c.bm + ((size_t)m * 2 * c.pmax + 2 * p + h) * c.S;
                j0 = p < nup ? pa[nlow + p] * c.S : 0;
#pragma unroll
                for (int g = 0; g < kClusG; g++) {
                    own[g] = p < nup && a[g] >= 0 ? bw[a[g]] : 0u;
                    any |= own[g];
                }
                some = __ballot_sync(kFull, any != 0u);
            }
            const int src = 2 * (t & 15);
            if ((some >> src) & 3u) {
#pragma unroll
                for (int h = 0; h < 2; h++)
#pragma unroll
                    for (int g = 0; g < kClusG; g++)
                        mk[h] |= ((__shfl_sync(kFull, own[g], src + h) >> lane) & 1u) << g;
                j = __shfl_sync(kFull, j0, src);
            }
        } else {
            const int s = t - nup;
            j = nB * c.S;
#pragma unroll
            for (int h = 0; h < 2; h++)
#pragma unroll
                for (int g = 0; g < kClusG; g++) {
                    const unsigned wd = a[g] >= 32 ? nw[h][1] : nw[h][0];
                    mk[h] |= a[g] >= 0 ? ((wd >> (a[g] & 31)) & 1u) << g : 0u;
                }
            if (s + 1 < nlow) load_lower(s + 1);
#pragma unroll
            for (int g = 0; g < kClusG; g++)
                r.inc[g / 2] += (((mk[0] >> g) & 1u) + ((mk[1] >> g) & 1u)) << (16 * (g & 1));
        }
        const bool last = t == nup - 1 || t == np - 1;
        if (__any_sync(kFull, (mk[0] | mk[1]) != 0u)) {
            r.add(mk[0], j + lane);
            r.add(mk[1], j + 32 + lane);
        }
        r.flush(last);
        if (t == nup - 1) nown = r.out = fill_slice(r.row, r.out, c.stride, lane);
    }
    if (lane == 0) {
        // the atoms' rows fit together unless one of them overflowed (reported by the list build)
        if (r.out > c.stride && atomicCAS(&c.err->code, FMD_OK, FMD_ERR_CAPACITY) == FMD_OK) {
            c.err->where = K_LJ; c.err->index = q.id[0]; c.err->value = r.out;
        }
        c.cnt[k] = make_int4(min(nown, c.stride & ~31), min(r.out, c.stride), (int)img, 0);
    }
    unsigned per[(kClusG + 1) / 2];
#pragma unroll
    for (int g = 0; g < (kClusG + 1) / 2; g++) per[g] = __reduce_add_sync(kFull, r.per[g]);
    unsigned inc[(kClusG + 1) / 2];
#pragma unroll
    for (int g = 0; g < (kClusG + 1) / 2; g++) inc[g] = __reduce_add_sync(kFull, r.inc[g]);
#pragma unroll
    for (int g = 0; g < kClusG; g++) {
        const int i = q.id[g];
        if (lane == g && i >= 0) {
            const double px = pos[3 * i], py = pos[3 * i + 1], pz = pos[3 * i + 2];
            po.cnt[i] = (int)((per[g / 2] >> (16 * (g & 1))) & 0xffffu);
            // more than a full row holds: an error, as where the full rows are built
            const int in = (int)((inc[g / 2] >> (16 * (g & 1))) & 0xffffu);
            if (in > c.full_cap - c.half_cap && atomicCAS(&c.err->code, FMD_OK, FMD_ERR_CAPACITY) == FMD_OK) {
                c.err->where = K_TRANSPOSE; c.err->index = i; c.err->value = in;
            }
            po.sb[3 * i] = hi[0] * px; po.sb[3 * i + 1] = hi[4] * py; po.sb[3 * i + 2] = hi[8] * pz;
            c.upos[3 * i] = px; c.upos[3 * i + 1] = py; c.upos[3 * i + 2] = pz;
        }
    }
}

// A pair's force over its distance, zero where the pair is out (in), without
// the factor 24 eps sigma^6 in FP64.  COUNT: its energy (without 4 eps sigma^6
// and the shift in FP64) and number, with SOME only where count says so.  No
// branches, so that the pairs of a lane are independent chains.
struct ClusConst {
    double s6, two_s6;                         // sigma^6, twice
};
template <bool F32, bool COUNT, bool SOME>
__device__ __forceinline__ double pair_term(double r2, bool in, bool count, const LJP& p, const LJF& pf,
                                            const ClusConst& cc, double& e, int& np) {
    // r^2 < 1/4 by its high word: exact, and not on the FP64 pipe
    const int rh = __double2hiint(r2);
    const bool close = rh < 0x3fd00000;
    r2 = __hiloint2double(close ? 0x3fd00000 : rh, close ? 0 : __double2loint(r2));
    if (F32) {
        // the FP32 pair algebra of lj_pair, operation for operation
        const float ri2 = rcp_f32((float)r2);
        const float s2 = fmaf(pf.sig2, ri2, pf.sig2_lo * ri2), s6 = s2 * s2 * s2, s12 = s6 * s6;
        if (COUNT && (SOME ? count : in)) e += (double)(pf.c4 * (s12 - s6)) - p.vshift;
        return in ? (double)(pf.c24 * (2.f * s12 - s6) * ri2) : 0.0;
    }
    // 1/r^2 as in lj_pair, zero where the pair is out (by the approximation's
    // high word)
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(r2));
    y = __hiloint2double(in ? __double2hiint(y) : 0, 0);
    const double e0 = fma(-r2, y, 1.0), e1 = fma(e0, e0, e0), i2 = fma(y, e1, y);
    const double i6 = i2 * i2 * i2;
    if (COUNT) {
        const double c6 = SOME ? __hiloint2double(count ? __double2hiint(i6) : 0, count ? __double2loint(i6) : 0) : i6;
        e = fma(c6, fma(cc.s6, i6, -1.0), e);
        np += SOME ? count : in;
    }
    return (i6 * i2) * fma(cc.two_s6, i6, -1.0);
}

// Pair sums of a lane: fm d per atom of the cluster, and on the counting side
// the virial's first part, the energy and the number of pairs.
struct ClusSum {
    double fx[kClusG], fy[kClusG], fz[kClusG];
    double w[6];                               // xx xy xz yy yz zz
    double e;
    int np;
};

// The entry in flight and the next one's index: an entry's position is
// loaded one slice and its index two slices before its pair terms.
struct ClusFeed {
    const int* row;
    int k, end;                                // index of the entry after e2, entries of the row
    unsigned e1, e2;
    double x, y, z;                            // position of e1
    __device__ __forceinline__ unsigned entry() const { return k < end ? (unsigned)row[k] : kIdle; }
    __device__ __forceinline__ void load(const double* __restrict__ pos) {
        const double* p = pos + 3 * (size_t)(e1 & kAtomBits);
        x = p[0]; y = p[1]; z = p[2];
    }
};

// n slices, step entries apart, of the row in f.
template <bool FV, bool F32, bool OWN>
__device__ __forceinline__ void clus_slices(const double* __restrict__ pos, int n, int step, ClusFeed& f,
                                            const Cluster& q, const double (*shift)[4], const LJP& p, const LJF& pf,
                                            const ClusConst& cc, ClusSum& s) {
    constexpr int unroll = kClusUnroll<F32>;
#pragma unroll unroll
    for (int t = 0; t < n; t++) {
        const unsigned ec = f.e1;
        const double cx = f.x, cy = f.y, cz = f.z;
        f.e1 = f.e2;
        f.load(pos);
        f.k += step;
        f.e2 = f.entry();
        const double* sh = shift[ec >> kCodeBit];
        const double2 sxy = *reinterpret_cast<const double2*>(sh);
        const double d0x = (cx - sxy.x) - q.x0, d0y = (cy - sxy.y) - q.y0, d0z = (cz - sh[2]) - q.z0;
        double gx = 0.0, gy = 0.0, gz = 0.0;
#pragma unroll
        for (int g = 0; g < kClusG; g++) {
            const double dx = g ? d0x - q.x[g] : d0x, dy = g ? d0y - q.y[g] : d0y, dz = g ? d0z - q.z[g] : d0z;
            const double r2 = fma(dx, dx, fma(dy, dy, dz * dz));
            const bool in = ((ec >> (kMaskBit + g)) & 1u) && !(r2 > p.rc2);
            const double fm = pair_term<F32, OWN, false>(r2, in, in, p, pf, cc, s.e, s.np);
            s.fx[g] = fma(fm, dx, s.fx[g]);
            s.fy[g] = fma(fm, dy, s.fy[g]);
            s.fz[g] = fma(fm, dz, s.fz[g]);
            if (OWN) { gx = fma(fm, dx, gx); gy = fma(fm, dy, gy); gz = fma(fm, dz, gz); }
        }
        if (OWN) {
            s.w[0] = fma(d0x, gx, s.w[0]);
            if (FV) { s.w[1] = fma(d0x, gy, s.w[1]); s.w[2] = fma(d0x, gz, s.w[2]); }
            s.w[3] = fma(d0y, gy, s.w[3]);
            if (FV) s.w[4] = fma(d0y, gz, s.w[4]);
            s.w[5] = fma(d0z, gz, s.w[5]);
        }
    }
}

// Sums the cluster's force over the warp: the lanes first split the atoms among
// themselves, so lanes 8 g hold atom g's sum.
static_assert(kClusG == 4, "lanes of an atom's sum");
constexpr int kOwnerStep = 32 / kClusG;
__device__ __forceinline__ int owner_atom(int lane) { return lane % kOwnerStep == 0 ? lane / kOwnerStep : -1; }
__device__ __forceinline__ void swap_add(double& keep, double other, bool hi, int o) {
    const double send = hi ? keep : other;
    keep = (hi ? other : keep) + __shfl_xor_sync(kFull, send, o);
}
__device__ __forceinline__ void clus_reduce(ClusSum& s, int lane, double& fx, double& fy, double& fz) {
    int o = 16;
#pragma unroll
    for (int half = kClusG / 2; half > 0; half >>= 1, o >>= 1) {
        const bool hi = lane & o;
#pragma unroll
        for (int g = 0; g < half; g++) {
            swap_add(s.fx[g], s.fx[g + half], hi, o);
            swap_add(s.fy[g], s.fy[g + half], hi, o);
            swap_add(s.fz[g], s.fz[g + half], hi, o);
        }
    }
    fx = s.fx[0]; fy = s.fy[0]; fz = s.fz[0];
#pragma unroll
    for (; o > 0; o >>= 1) {
        fx += __shfl_xor_sync(kFull, fx, o);
        fy += __shfl_xor_sync(kFull, fy, o);
        fz += __shfl_xor_sync(kFull, fz, o);
    }
}

// Atom i's full row, by a warp, from the candidate bitmaps: the row that
// k_mol_incoming (molnlist.cu) builds.
__device__ __noinline__ void build_full_row(const LJClus& c, int i, int lane) {
    const int B = i / c.S, jb = i - B * c.S, lim = c.full_cap - c.half_cap;
    const unsigned below = (1u << lane) - 1u;
    int* row = c.full_list + (size_t)i * c.full_cap;
    const int* pa = c.part + (size_t)B * c.pmax;
    const int* rv = c.rev + (size_t)B * c.pmax;
    const int np = c.npart[B];
    int n = 0;
    for (int q = 0; q < np && pa[q] < B; q++) {            // ascending: the lower partners come first
        const int A = pa[q];
        const unsigned* bw = c.bm + ((size_t)A * 2 * c.pmax + 2 * rv[q] + (jb >> 5)) * c.S;
        for (int a0 = 0; a0 < c.S; a0 += 32) {
            const bool in = a0 + lane < c.S && (bw[a0 + lane] >> (jb & 31) & 1u);
            const unsigned m = __ballot_sync(kFull, in);
            const int k = n + __popc(m & below);
            if (in && k < lim) row[k] = A * c.S + a0 + lane;
            n += __popc(m);
        }
    }
    if (lane == 0 && n > lim && atomicCAS(&c.err->code, FMD_OK, FMD_ERR_CAPACITY) == FMD_OK) {
        c.err->where = K_TRANSPOSE; c.err->index = i; c.err->value = n;
    }
    n = min(n, lim);
    const int own = c.half_cnt[i];
    for (int k = lane; k < own; k += 32) row[n + k] = c.half_list[(size_t)i * c.half_cap + k];
    if (lane == 0) c.full_cnt[i] = n + own;
    __syncwarp();                                          // the row, before the warp's lanes read it
}

// The block's atoms i0 .. i1 - 1 over rows of their own, as the row gather
// (airebo.cu): over the full rows, which it builds first where the list build
// left them out, writing the pruned ones (ATOMS_PRUNE) or not (ATOMS_FULL), or
// over those of the last prune.  Rounds of one atom per warp, then the remaining
// atoms with their rows split over the warps where no row is written.  F, and
// {E, W} into the block's record.  All of the block's work, called with nothing
// left to do: values kept across the call would cost the cluster walk registers
// (2 % of its time).
template <bool FV, bool F32>
__device__ __noinline__ void atom_rows(const ClusArgs& a, int blk, int nblk, int mode, ClusShared& sh) {
    const LJClus& c = a.c;
    const LJP p = a.p;
    const double* __restrict__ pos = a.pos;
    double *F = a.F, *Facc = a.Facc;
    const int i0 = (int)((long long)blk * a.na / nblk), i1 = (int)((long long)(blk + 1) * a.na / nblk);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const double* h = sh.hh;
    const double* hi = sh.hh + 9;
    double (*part)[3 * kClusG] = sh.part;
    const bool diag = h[1] == 0.0 && h[2] == 0.0 && h[3] == 0.0 && h[5] == 0.0 && h[6] == 0.0 && h[7] == 0.0 &&
                      hi[1] == 0.0 && hi[2] == 0.0 && hi[3] == 0.0 && hi[5] == 0.0 && hi[6] == 0.0 && hi[7] == 0.0;
    const bool wide = diag && 0.25 * fmin(h[0] * h[0], fmin(h[4] * h[4], h[8] * h[8])) > p.rc2 * (1.0 + 1e-9);
    const LJF pf{(float)p.sig2, (float)(p.sig2 - (double)(float)p.sig2), (float)p.c4, (float)p.c24};
    const ClusConst cc{p.sig2 * p.sig2 * p.sig2, 2.0 * (p.sig2 * p.sig2 * p.sig2)};
    const double fs = F32 ? 1.0 : p.c24 * cc.s6;
    double acc[kNV], e = 0.0, vir[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    int np = 0;
#pragma unroll
    for (int k = 0; k < kNV; k++) acc[k] = 0.0;
    constexpr int U = kAtomUnroll;
    LJPruneOut po = a.po;
    po.list = c.rows;
    const int* cnt = mode == ATOMS_WALK ? po.cnt : c.full_cnt;
    const int* list = mode == ATOMS_WALK ? c.rows : c.full_list;
    if (mode != ATOMS_PRUNE) po.cnt = nullptr;
    const bool build = mode == ATOMS_PRUNE && c.flag[2] != 0;
    constexpr int W = kWarps<F32>;
    const int whole = (i1 - i0) / W * W, rest = i1 - i0 - whole;
    const int split = mode != ATOMS_PRUNE && rest > 0 ? W / rest : 1;
    for (int r = 0; r <= whole; r += W) {
        const bool tail = r == whole;
        if (tail && rest == 0) break;
        const int sp = tail ? split : 1, kk = w / sp, first = w - kk * sp;
        const bool mine = !tail || kk < rest;
        const int i = mine ? i0 + r + kk : i0;
        if (build && mine) build_full_row(c, i, lane);
        const double px = pos[3 * i], py = pos[3 * i + 1], pz = pos[3 * i + 2];
        const LJAcc fa = lj_acc_load(Facc, i, lane);
        double fx = 0.0, fy = 0.0, fz = 0.0, sx = 0.0, sy = 0.0, sz = 0.0;
        const int tot = mine ? min(cnt[i], c.full_cap) : 0;
        const int* row = list + (size_t)i * c.full_cap;
        int* prow = c.rows + (size_t)i * c.full_cap;
        int pc = 0;
        int jj[U];                                         // indices one chunk ahead
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int k = 32 * (U * first + u) + lane;
            jj[u] = k < tot ? row[k] : -1;
        }
        for (int b0 = 32 * U * first; b0 < tot; b0 += 32 * U * sp) {
            int jc[U];
            double cx[U], cy[U], cz[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int j = jj[u] < 0 ? i : jj[u];
                jc[u] = jj[u];
                cx[u] = pos[3 * j]; cy[u] = pos[3 * j + 1]; cz[u] = pos[3 * j + 2];
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int k = b0 + 32 * (U * sp + u) + lane;
                jj[u] = k < tot ? row[k] : -1;
            }
            if (!wide) {
                lj_chunk<FV, F32, U>(jc, cx, cy, cz, i, px, py, pz, h, hi, diag, wide, p, pf, fx, fy, fz, acc, po, prow,
                                     pc, lane);
                continue;
            }
            bool keep[U];
            auto chunk = [&](auto count_tag) {
                constexpr bool COUNT = decltype(count_tag)::value;
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const double dx = mimg1_rint(__dsub_rn(cx[u], px), h[0], hi[0]),
                                 dy = mimg1_rint(__dsub_rn(cy[u], py), h[4], hi[4]),
                                 dz = mimg1_rint(__dsub_rn(cz[u], pz), h[8], hi[8]);
                    const double r2 = norm2_rn(dx, dy, dz);
                    const bool in = jc[u] >= 0 && !(r2 > p.rc2), own = jc[u] > i;
                    keep[u] = jc[u] >= 0 && r2 <= po.r2;
                    const double fm = pair_term<F32, COUNT, true>(r2, in, in && own, p, pf, cc, e, np);
                    const double gx = fm * dx, gy = fm * dy, gz = fm * dz;
                    sx += gx; sy += gy; sz += gz;
                    if (COUNT) {
                        const double ox = own ? gx : 0.0, oy = own ? gy : 0.0, oz = own ? gz : 0.0;
                        vir[0] = fma(dx, ox, vir[0]);
                        if (FV) { vir[1] = fma(dx, oy, vir[1]); vir[2] = fma(dx, oz, vir[2]); }
                        vir[3] = fma(dy, oy, vir[3]);
                        if (FV) vir[4] = fma(dy, oz, vir[4]);
                        vir[5] = fma(dz, oz, vir[5]);
                    }
                }
            };
            bool own = false;
#pragma unroll
            for (int u = 0; u < U; u++) own = own || jc[u] > i;
            if (__any_sync(kFull, own)) chunk(std::true_type{});
            else chunk(std::false_type{});
            if (po.cnt) {
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const unsigned m = __ballot_sync(kFull, keep[u]);
                    if (keep[u]) prow[pc + __popc(m & ((1u << lane) - 1u))] = jc[u];
                    pc += __popc(m);
                }
            }
        }
        fx -= fs * sx; fy -= fs * sy; fz -= fs * sz;
        if (sp == 1) {
            if (mine) lj_atom_done(i, fx, fy, fz, px, py, pz, hi, F, Facc, po, pc, lane, fa);
            continue;
        }
        fx = warp_sum(fx); fy = warp_sum(fy); fz = warp_sum(fz);
        if (lane == 0) { part[w][0] = fx; part[w][1] = fy; part[w][2] = fz; }
        __syncthreads();                                   // once: the tail is the last round
        if (mine && first == 0 && lane == 0) {
            for (int t = 1; t < sp; t++) { fx += part[w + t][0]; fy += part[w + t][1]; fz += part[w + t][2]; }
            F[3 * i] = fa.x + fx; F[3 * i + 1] = fa.y + fy; F[3 * i + 2] = fa.z + fz;
            if (Facc != F) { Facc[3 * i] = 0.0; Facc[3 * i + 1] = 0.0; Facc[3 * i + 2] = 0.0; }
        }
    }
    acc[0] += F32 ? e : p.c4 * cc.s6 * e - p.vshift * np;
    acc[1] += fs * vir[0]; acc[5] += fs * vir[3]; acc[9] += fs * vir[5];
    acc[2] += fs * vir[1]; acc[3] += fs * vir[2]; acc[6] += fs * vir[4];
    lj_virial_mirror<FV>(acc);
    block_sum_fields<kNV>(acc, sh.sm, a.part + (size_t)blk * kNV);
}

// Block blk of nblk: its run of clusters.  Rounds of one cluster per warp,
// then the remaining clusters with their rows split over the warps, so that
// no warp idles through a whole row (7,500 clusters are 3.2 per warp at
// 30,000 atoms; a system of 1,920 has fewer clusters than the GPU has
// schedulers).
template <bool FV, bool F32>
__device__ __forceinline__ void lj_clus_body(const ClusArgs& a, const LJP& p, int blk, int nblk, ClusShared& sh) {
    const LJClus& c = a.c;
    const LJPruneOut& po = a.po;
    const double* __restrict__ pos = a.pos;
    const double* __restrict__ hh = a.hh;
    double* __restrict__ F = a.F;
    double* __restrict__ Facc = a.Facc;
    int mode = a.mode;
    constexpr int kClusWarps = kWarps<F32>, kClusThreads = 32 * kClusWarps;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x < 18) sh.hh[threadIdx.x] = hh[threadIdx.x];
    __syncthreads();
    if (mode < 0) mode = lj_clus_mode(c, po.words, sh.hh, po.hb, po.delta, po.rc);
    if (lj_clus_kind(mode) == kRowsAtoms) {
        atom_rows<FV, F32>(a, blk, nblk, mode, sh);
        return;
    }
    if (threadIdx.x < 32) {
        const int t = threadIdx.x;
        sh.shift[t][0] = sh.hh[0] * (t < 27 ? t % 3 - 1 : 4);
        sh.shift[t][1] = sh.hh[4] * (t < 27 ? t / 3 % 3 - 1 : 4);
        sh.shift[t][2] = sh.hh[8] * (t < 27 ? t / 9 - 1 : 4);
    }
    for (int t = threadIdx.x; t < c.cpm * kClusG; t += kClusThreads) sh.perm[t] = c.perm[t];
    const int c0 = (int)((long long)blk * c.nclus / nblk), c1 = (int)((long long)(blk + 1) * c.nclus / nblk);
    ClusSum s;
    s.e = 0.0;
    s.np = 0;
#pragma unroll
    for (int k = 0; k < 6; k++) s.w[k] = 0.0;
    __syncthreads();                       // image offsets, clusters
    if (mode == CLUS_PRUNE)
        for (int k = c0 + w; k < c1; k += kClusWarps) build_row(c, k, pos, sh, po, w, lane);
    __syncthreads();                       // rows of this block
    const double* x = mode == CLUS_PRUNE ? pos : c.upos;
    const LJF pf{(float)p.sig2, (float)(p.sig2 - (double)(float)p.sig2), (float)p.c4, (float)p.c24};
    const ClusConst cc{p.sig2 * p.sig2 * p.sig2, 2.0 * (p.sig2 * p.sig2 * p.sig2)};
    const double fs = F32 ? 1.0 : p.c24 * cc.s6;
    const int whole = (c1 - c0) / kClusWarps * kClusWarps, rest = c1 - c0 - whole;
    const int split = rest > 0 ? kClusWarps / rest : 1;
    for (int r = 0; r <= whole; r += kClusWarps) {
        const bool tail = r == whole;
        if (tail && rest == 0) break;
        const int sp = tail ? split : 1;
        const int kk = w / sp, first = w % sp;
        const int k = c0 + r + kk;
        const bool mine = !tail || kk < rest;
        const int own = owner_atom(lane);
        double fx = 0.0, fy = 0.0, fz = 0.0;
        int io = -1;                       // atom this lane writes
        LJAcc fa;
        if (mine) {
            const int4 n = c.cnt[k];
            const Cluster q = load_cluster(c, k, n.z, x, sh);
#pragma unroll
            for (int g = 0; g < kClusG; g++)
                if (own == g) io = q.id[g];
            if (io >= 0 && first == 0) { fa.x = Facc[3 * io]; fa.y = Facc[3 * io + 1]; fa.z = Facc[3 * io + 2]; }
#pragma unroll
            for (int g = 0; g < kClusG; g++) s.fx[g] = s.fy[g] = s.fz[g] = 0.0;
            // slices first, first + sp, ...: the counting ones, then the others
            const int nsl = (n.y + 31) >> 5, nown = n.x >> 5;
            const int mine_all = nsl > first ? (nsl - first + sp - 1) / sp : 0;
            const int mine_own = nown > first ? (nown - first + sp - 1) / sp : 0;
            ClusFeed f;
            f.row = c.rows + (size_t)k * c.stride;
            f.end = n.y;
            f.k = 32 * first + lane;
            f.e1 = f.entry();
            f.load(x);
            f.k += 32 * sp;
            f.e2 = f.entry();
            clus_slices<FV, F32, true>(x, mine_own, 32 * sp, f, q, sh.shift, p, pf, cc, s);
#pragma unroll
            for (int g = 1; g < kClusG; g++) {     // the virial's second part
                s.w[0] = fma(-q.x[g], s.fx[g], s.w[0]);
                if (FV) { s.w[1] = fma(-q.x[g], s.fy[g], s.w[1]); s.w[2] = fma(-q.x[g], s.fz[g], s.w[2]); }
                s.w[3] = fma(-q.y[g], s.fy[g], s.w[3]);
                if (FV) s.w[4] = fma(-q.y[g], s.fz[g], s.w[4]);
                s.w[5] = fma(-q.z[g], s.fz[g], s.w[5]);
            }
            clus_slices<FV, F32, false>(x, mine_all - mine_own, 32 * sp, f, q, sh.shift, p, pf, cc, s);
            clus_reduce(s, lane, fx, fy, fz);
        }
        if (sp > 1) {
            if (own >= 0) {
                sh.part[w][3 * own] = fx; sh.part[w][3 * own + 1] = fy; sh.part[w][3 * own + 2] = fz;
            }
            __syncthreads();
            if (first == 0 && own >= 0)
                for (int t = 1; t < sp; t++) {
                    fx += sh.part[w + t][3 * own];
                    fy += sh.part[w + t][3 * own + 1];
                    fz += sh.part[w + t][3 * own + 2];
                }
        }
        if (io >= 0 && first == 0) {
            F[3 * io] = fa.x - fs * fx;
            F[3 * io + 1] = fa.y - fs * fy;
            F[3 * io + 2] = fa.z - fs * fz;
            if (Facc != F) { Facc[3 * io] = 0.0; Facc[3 * io + 1] = 0.0; Facc[3 * io + 2] = 0.0; }
        }
    }
    double acc[kNV];
    acc[0] = F32 ? s.e : p.c4 * cc.s6 * s.e - p.vshift * s.np;
    acc[1] = fs * s.w[0]; acc[5] = fs * s.w[3]; acc[9] = fs * s.w[5];
    acc[2] = acc[4] = FV ? fs * s.w[1] : 0.0;
    acc[3] = acc[7] = FV ? fs * s.w[2] : 0.0;
    acc[6] = acc[8] = FV ? fs * s.w[4] : 0.0;
    block_sum_fields<kNV>(acc, sh.sm, a.part + (size_t)blk * kNV);
}

template <bool FV, bool F32>
__global__ void __launch_bounds__(32 * kWarps<F32>, kBlocks<F32>)
k_lj_clus(const __grid_constant__ ClusArgs a) {
    FMD_PDL_WAIT();
    __shared__ ClusShared sh;
    lj_clus_body<FV, F32>(a, a.p, blockIdx.x, gridDim.x, sh);
    if (threadIdx.x < kNV)
        for (int r = gridDim.x + blockIdx.x; r < a.nrec; r += gridDim.x) a.part[(size_t)r * kNV + threadIdx.x] = 0.0;
}

// Replica batch (MM): block b serves replica r as its local block b - off[r].
template <bool F32>
__global__ void __launch_bounds__(32 * kWarps<F32>, kBlocks<F32>)
k_b_lj_clus(const StepArrays* __restrict__ As, const int* __restrict__ off, int R) {
    __shared__ ClusShared sh;
    __shared__ ClusArgs args;
    const int r = batch_rep(off, R, blockIdx.x);
    const LJP p = lj_params_dev(FMD_FF_MM);
    if (threadIdx.x == 0) {
        const StepArrays& a = As[r];
        const double rp = a.prune_rc + a.prune_delta;
        LJPruneOut po;
        po.cnt = a.prune_cnt;
        po.sb = const_cast<double*>(a.prune_sb);
        po.r2 = rp * rp;
        po.words = a.prune_umax;
        po.hb = a.prune_hb;
        po.delta = a.prune_delta;
        po.rc = a.prune_rc;
        args = ClusArgs{a.clus, po, p, a.pos, a.S->h, a.F, a.Facc, a.part_f2, a.n, 0, -1};
    }
    __syncthreads();
    lj_clus_body<false, F32>(args, p, blockIdx.x - off[r], off[r + 1] - off[r], sh);
}

template <bool FV, bool F32>
int clus_grid() {
    static int grid = 0;
    if (grid == 0) {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_lj_clus<FV, F32>, 32 * kWarps<F32>, 0) != cudaSuccess || b < 1)
            b = 1;
        grid = std::min(kLJMaxBlocks, b * kSMs);
    }
    return grid;
}

}  // namespace

int lj_clus_threads(int precision) { return 32 * (precision == FMD_PREC_FP32_PAIR ? kWarps<true> : kWarps<false>); }

int lj_clus_blocks(int ff, int precision) {
    const bool f32 = precision == FMD_PREC_FP32_PAIR;
    if (ff == FMD_FF_AIREBO) return f32 ? clus_grid<true, true>() : clus_grid<true, false>();
    return f32 ? clus_grid<false, true>() : clus_grid<false, false>();
}

cudaError_t lj_clus_launch(int ff, const LJClus& c, const double* pos, const double* hh, int na, double* F,
                           double* Facc, double* part, cudaStream_t st, int precision, const LJPruneOut& po, int nrec,
                           int mode) {
    const LJP p = lj_params_dev(ff);
    const bool f32 = precision == FMD_PREC_FP32_PAIR;
    const dim3 grid(lj_clus_blocks(ff, precision)), block(lj_clus_threads(precision));
#define FMD_CLUS(FV, F32)                                                                                            \
    launch_pdl(k_lj_clus<FV, F32>, grid, block, 0, st, ClusArgs{c, po, p, pos, hh, F, Facc, part, na, nrec, mode})
    if (ff == FMD_FF_AIREBO) return f32 ? FMD_CLUS(true, true) : FMD_CLUS(true, false);
    return f32 ? FMD_CLUS(false, true) : FMD_CLUS(false, false);
#undef FMD_CLUS
}

cudaError_t batch_lj_clus_launch(const StepArrays* As, const int* off, int R, int nblocks, int precision,
                                 cudaStream_t st) {
    if (precision == FMD_PREC_FP32_PAIR) k_b_lj_clus<true><<<nblocks, 32 * kWarps<true>, 0, st>>>(As, off, R);
    else k_b_lj_clus<false><<<nblocks, 32 * kWarps<false>, 0, st>>>(As, off, R);
    return cudaGetLastError();
}

// Clusters by greedy growth (each takes the free atom nearest to its atoms
// so far), then exchanges of atoms between clusters while one lowers the sum
// of squared distances within clusters; the atom with the least largest
// distance to the others goes first.
std::vector<int> lj_clus_assign(const double* x, int S) {
    constexpr int G = kClusG;
    const int nc = (S + G - 1) / G;
    std::vector<double> d2((size_t)S * S);
    for (int a = 0; a < S; a++)
        for (int b = 0; b < S; b++) {
            const double u = x[3 * a] - x[3 * b], v = x[3 * a + 1] - x[3 * b + 1], w = x[3 * a + 2] - x[3 * b + 2];
            d2[(size_t)a * S + b] = u * u + v * v + w * w;
        }
    std::vector<int> perm((size_t)nc * G, -1);
    std::vector<char> used(S, 0);
    for (int c = 0; c < nc; c++) {
        int* q = &perm[(size_t)c * G];
        for (int g = 0; g < G; g++) {
            int best = -1;
            double bd = std::numeric_limits<double>::infinity();
            for (int a = 0; a < S; a++) {
                if (used[a]) continue;
                double t = 0.0;
                for (int k = 0; k < g; k++) t += d2[(size_t)a * S + q[k]];
                if (best < 0 || t < bd) { best = a; bd = t; }
            }
            if (best < 0) break;
            used[best] = 1;
            q[g] = best;
        }
    }
    // sum[c * S + a]: squared distances of atom a to the atoms of cluster c
    std::vector<double> sum((size_t)nc * S, 0.0);
    auto add = [&](int c, int b, double sign) {
        if (b < 0) return;
        double* t = &sum[(size_t)c * S];
        const double* r = &d2[(size_t)b * S];
        for (int a = 0; a < S; a++) t[a] += sign * r[a];
    };
    for (int u = 0; u < nc * G; u++) add(u / G, perm[u], 1.0);
    for (int pass = 0; pass < 8; pass++) {
        bool any = false;
        for (int u = 0; u < nc * G; u++)
            for (int v = (u / G + 1) * G; v < nc * G; v++) {
                const int a = perm[u], b = perm[v], c = u / G, e = v / G;
                if (a < 0 || b < 0) continue;
                const double ab = d2[(size_t)a * S + b];
                const double now = sum[(size_t)c * S + a] + sum[(size_t)e * S + b];
                const double then = sum[(size_t)c * S + b] + sum[(size_t)e * S + a] - 2.0 * ab;
                if (then < now - 1e-9) {
                    add(c, a, -1.0); add(c, b, 1.0);
                    add(e, b, -1.0); add(e, a, 1.0);
                    std::swap(perm[u], perm[v]);
                    any = true;
                }
            }
        if (!any) break;
    }
    for (int c = 0; c < nc; c++) {
        int* q = &perm[(size_t)c * G];
        int best = 0;
        double bd = std::numeric_limits<double>::infinity();
        for (int g = 0; g < G && q[g] >= 0; g++) {
            double t = 0.0;
            for (int k = 0; k < G; k++)
                if (q[k] >= 0) t = std::max(t, d2[(size_t)q[g] * S + q[k]]);
            if (t < bd) { bd = t; best = g; }
        }
        std::swap(q[0], q[best]);
    }
    return perm;
}

}  // namespace fmd
