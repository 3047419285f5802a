// step.cu -- NPT velocity-Verlet on the device (a17 rigid LJ:434-538,
// a18 atomistic AI:518-590 / MM:811-890) and the driver's per-step schedule
// (a19: LJ:847-897, AI:871-912, MM:1192-1236).
//
// The reference keeps xi, Vg and h on the host and synchronises several
// times per step.  Here they live in a device struct (SysScal) updated on the
// device, so a whole step -- and a list rebuild -- is
// a fixed sequence of launches with no host round trip, which is what lets
// the step be replayed as a CUDA graph:
//
//   k_begin_kick  schedule (Tt ramp, cold resets), thermostat/barostat
//               first half, scaling factors, cell update and its inverse
//               (every block on its own copy of the scalars), then the first
//               half-kick, drift in fractional coordinates, wrap, back to
//               Cartesian with the new cell (+ quaternion update)
//   forces      (airebo.cu / rigid.cu / mm.cu)
//   k_kick2_end second half-kick with per-block kinetic partials; the last
//               block to finish: force/kinetic reductions (fixed order),
//               thermostat/barostat second half, observables, rescale
//               decision, averages
//   k_rescale / k_rescale_end   cold/warm phases only
//
// Scalar arithmetic follows the reference expressions; this file is built
// with -fmad=false so they round like the reference's host code.
#include <algorithm>
#include <cmath>
#include "step.h"
#include "ljprune.h"
#include "mmmol.h"
#include "ljprune.cuh"
#include "ljclus.cuh"
#include "geom.cuh"
#include "sg_host.h"
#include "pdl.cuh"
#include "rigidpair.cuh"

namespace fmd {
namespace {

constexpr int kPB = 256;   // threads of per-particle kernels
constexpr int kRedThreads = 512;   // the one-block reductions of the partial records
constexpr double kMC = 12.011;

__device__ __forceinline__ double clampd(double x, double lo, double hi) {
    return x < lo ? lo : (x > hi ? hi : x);
}
__device__ __forceinline__ double inst_T(double ke, int nf) { return 2 * ke / (nf * kKB); }
__device__ __forceinline__ double inst_P(const double* W, double ke, double V) {
    return (2 * ke + W[0] + W[4] + W[8]) / (3 * V) * kEV2GPa;
}

// Thermostat + barostat half update (LJ:448-455, AI:524-530).
__device__ void npt_half(fmd_npt& s, double hdt, double ke, double ke_p, const double* W, double V,
                         double xi_lim, double vg_lim) {
    s.xi += hdt * (2 * ke - s.Nf * kKB * s.Tt) / s.Q;
    s.xi = clampd(s.xi, -xi_lim, xi_lim);
    const double dP = inst_P(W, ke_p, V) - s.Pe;
    for (int a = 0; a < 3; a++) s.Vg[a * 4] += hdt * V * dP / (s.W * kEV2GPa);
    for (int a = 0; a < 3; a++) s.Vg[a * 4] = clampd(s.Vg[a * 4], -vg_lim, vg_lim);
}

}  // namespace

__device__ void begin_body(SysScal* S, int kind, const StepParams& p) {
    fmd_npt& npt = S->npt;
    if (p.schedule) {
        const int g = ++S->gstep;
        // Tt schedule and resets (LJ:851-857)
        if (g <= p.coldstart) npt.Tt = p.T_cold;
        else if (g <= p.coldstart + p.warmup)
            npt.Tt = p.T_cold + (p.T - p.T_cold) * double(g - p.coldstart) / double(p.warmup);
        else npt.Tt = p.T;
        if (p.coldstart > 0 && g == p.coldstart + 1) {
            npt.xi = 0;
            for (int k = 0; k < 9; k++) npt.Vg[k] = 0;
        }
        if (g <= p.coldstart)
            for (int k = 0; k < 9; k++) npt.Vg[k] = 0;
    }
    const double hdt = 0.5 * p.dt;
    const bool rigid = kind == FMD_SYS_RIGID;
    if (rigid) inv9(S->h, S->hi);                                  // LJ:442
    const double V = fabs(det9(S->h));
    if (rigid) npt_half(npt, hdt, S->kt + S->kr, S->kt, S->W9, V, 0.1, 0.01);
    else npt_half(npt, hdt, S->KE, S->KE, S->W9, V, 0.05, 0.005);
    const double eps = npt.Vg[0] * S->hi[0] + npt.Vg[4] * S->hi[4] + npt.Vg[8] * S->hi[8];
    const double sc_nh = exp(-hdt * npt.xi), sc_pr = exp(-hdt * eps / 3.0);
    S->sc_nh = sc_nh;
    S->sc_v = sc_nh * sc_pr;
    for (int k = 0; k < 9; k++) S->hi_old[k] = S->hi[k];
    for (int k = 0; k < 9; k++) S->h[k] += p.dt * npt.Vg[k];          // LJ:484
    inv9(S->h, S->hi);                                                // LJ:509, AI:555
    const double eps2 = npt.Vg[0] * S->hi[0] + npt.Vg[4] * S->hi[4] + npt.Vg[8] * S->hi[8];
    S->sc_v2 = sc_nh * exp(-hdt * eps2 / 3.0);
}

namespace {

// LJ:166-174.  The reference multiplies q by the rotation increment on the
// right (q dq), which applies the lab-frame angular velocity as a body-frame
// one; left (dq q, FMD_PHYS_QUAT) rotates the lab-frame sites about the lab
// axis w, which is what the lab-frame torque update of w describes.
template <bool LEFT>
__device__ __forceinline__ void quat_step(double* q, double wx, double wy, double wz, double dt) {
    double dq[4];
    const double wm = sqrt(wx * wx + wy * wy + wz * wz), th = wm * dt * 0.5;
    if (th < 1e-14) { dq[0] = 1.0; dq[1] = 0.5 * dt * wx; dq[2] = 0.5 * dt * wy; dq[3] = 0.5 * dt * wz; }
    else { const double s = sin(th) / wm; dq[0] = cos(th); dq[1] = s * wx; dq[2] = s * wy; dq[3] = s * wz; }
    double o[4];
    if (LEFT) {
        o[0] = dq[0] * q[0] - dq[1] * q[1] - dq[2] * q[2] - dq[3] * q[3];
        o[1] = dq[0] * q[1] + dq[1] * q[0] + dq[2] * q[3] - dq[3] * q[2];
        o[2] = dq[0] * q[2] - dq[1] * q[3] + dq[2] * q[0] + dq[3] * q[1];
        o[3] = dq[0] * q[3] + dq[1] * q[2] - dq[2] * q[1] + dq[3] * q[0];
    } else {
        o[0] = q[0] * dq[0] - q[1] * dq[1] - q[2] * dq[2] - q[3] * dq[3];
        o[1] = q[0] * dq[1] + q[1] * dq[0] + q[2] * dq[3] - q[3] * dq[2];
        o[2] = q[0] * dq[2] - q[1] * dq[3] + q[2] * dq[0] + q[3] * dq[1];
        o[3] = q[0] * dq[3] + q[1] * dq[2] - q[2] * dq[1] + q[3] * dq[0];
    }
    const double nrm = sqrt(o[0] * o[0] + o[1] * o[1] + o[2] * o[2] + o[3] * o[3]), inv = 1.0 / nrm;
    for (int k = 0; k < 4; k++) q[k] = o[k] * inv;
}

}  // namespace

// What the first kick reads of particle i.
struct KickIn {
    double v[3], F[3], p[3], m, sb[3];
};
__device__ __forceinline__ KickIn kick_load(const StepArrays& a, int i) {
    KickIn k;
    k.m = a.mass != nullptr ? a.mass[i] : 0.0;
#pragma unroll
    for (int c = 0; c < 3; c++) {
        k.v[c] = a.vel[3 * i + c]; k.F[c] = a.F[3 * i + c]; k.p[c] = a.pos[3 * i + c];
        k.sb[c] = a.prune_sb ? a.prune_sb[3 * i + c] : 0.0;
    }
    return k;
}

// in: the thread's first particle, already loaded.
__device__ void kick_body(const StepArrays& a, double dt, int blk, int nblk, const SysScal* sc = nullptr,
                          const KickIn* in = nullptr) {
    const SysScal* S = sc ? sc : a.S;
    const double hdt = 0.5 * dt, sc_v = S->sc_v, sc_nh = S->sc_nh;
    const double* hi = S->hi_old;
    const double* h = S->h;
    const bool rigid = a.kind == FMD_SYS_RIGID;
    const double cF = rigid ? kConv / a.Mmol : kConv / kMC, cT = rigid ? kConv / a.I0 : 0.0;
    double u2 = 0.0;   // largest squared displacement since the last LJ prune
    for (int i = blk * blockDim.x + threadIdx.x; i < a.n; i += nblk * blockDim.x) {
        KickIn k;
        if (in) k = *in;
        else k = kick_load(a, i);
        in = nullptr;
        const double mi = (a.mass != nullptr) ? kConv / k.m : cF;
        double v[3];
        const double* p = k.p;
        for (int c = 0; c < 3; c++) {
            v[c] = k.v[c] * sc_v + hdt * k.F[c] * mi;
            a.vel[3 * i + c] = v[c];
        }
        double sx = hi[0] * p[0] + hi[1] * p[1] + hi[2] * p[2];
        double sy = hi[3] * p[0] + hi[4] * p[1] + hi[5] * p[2];
        double sz = hi[6] * p[0] + hi[7] * p[1] + hi[8] * p[2];
        const double vx = hi[0] * v[0] + hi[1] * v[1] + hi[2] * v[2];
        const double vy = hi[3] * v[0] + hi[4] * v[1] + hi[5] * v[2];
        const double vz = hi[6] * v[0] + hi[7] * v[1] + hi[8] * v[2];
        sx += dt * vx; sy += dt * vy; sz += dt * vz;
        sx -= floor(sx); sy -= floor(sy); sz -= floor(sz);
        a.pos[3 * i] = h[0] * sx + h[1] * sy + h[2] * sz;
        a.pos[3 * i + 1] = h[3] * sx + h[4] * sy + h[5] * sz;
        a.pos[3 * i + 2] = h[6] * sx + h[7] * sy + h[8] * sz;
        if (a.prune_sb) {
            // nearest-image fractional displacement, measured in the new cell
            double ex = sx - k.sb[0], ey = sy - k.sb[1], ez = sz - k.sb[2];
            const double kx = rint(ex), ky = rint(ey), kz = rint(ez);
            ex -= kx; ey -= ky; ez -= kz;
            if (a.clus.on) {
                // the position followed from the last prune without wrapping
                const double wx = sx - kx, wy = sy - ky, wz = sz - kz;
                a.clus.upos[3 * i] = h[0] * wx + h[1] * wy + h[2] * wz;
                a.clus.upos[3 * i + 1] = h[3] * wx + h[4] * wy + h[5] * wz;
                a.clus.upos[3 * i + 2] = h[6] * wx + h[7] * wy + h[8] * wz;
            }
            const double ux = h[0] * ex + h[1] * ey + h[2] * ez, uy = h[3] * ex + h[4] * ey + h[5] * ez,
                         uz = h[6] * ex + h[7] * ey + h[8] * ez;
            u2 = fmax(u2, ux * ux + uy * uy + uz * uz);
        }
        if (rigid) {
            double w[3];
            for (int c = 0; c < 3; c++) {
                w[c] = a.omg[3 * i + c] * sc_nh + hdt * a.T[3 * i + c] * cT;
                a.omg[3 * i + c] = w[c];
            }
            if (a.quat_left) quat_step<true>(a.qv + 4 * i, w[0], w[1], w[2], dt);
            else quat_step<false>(a.qv + 4 * i, w[0], w[1], w[2], dt);     // LJ:503-508
        }
    }
    if (a.prune_sb) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) u2 = fmax(u2, __shfl_xor_sync(kFull, u2, o));
        if ((threadIdx.x & 31) == 0 && u2 > 0.0)
            atomicMax(a.prune_umax, (unsigned long long)__double_as_longlong(sqrt(u2) * (1.0 + 1e-12)));
    }
}

// Second half-kick with per-block sums of m v^2 (atomistic) or v^2 and w^2
// (rigid) into part_ke[2 * blk]; sm holds 64 doubles.
__device__ void kick2_body(const StepArrays& a, double dt, int blk, int nblk, double* sm) {
    const SysScal* S = a.S;
    const double hdt = 0.5 * dt, sc_v2 = S->sc_v2, sc_nh = S->sc_nh;
    const bool rigid = a.kind == FMD_SYS_RIGID;
    const double cF = rigid ? kConv / a.Mmol : kConv / kMC, cT = rigid ? kConv / a.I0 : 0.0;
    double acc[2] = {0.0, 0.0};
    for (int i = blk * blockDim.x + threadIdx.x; i < a.n; i += nblk * blockDim.x) {
        const double mi = (a.mass != nullptr) ? kConv / a.mass[i] : cF;
        double vv = 0;
        for (int c = 0; c < 3; c++) {
            const double v = (a.vel[3 * i + c] + hdt * a.F[3 * i + c] * mi) * sc_v2;
            a.vel[3 * i + c] = v;
            vv += v * v;
        }
        if (rigid) {
            double ww = 0;
            for (int c = 0; c < 3; c++) {
                const double w = (a.omg[3 * i + c] + hdt * a.T[3 * i + c] * cT) * sc_nh;
                a.omg[3 * i + c] = w;
                ww += w * w;
            }
            acc[0] += vv;
            acc[1] += ww;
        } else {
            acc[0] += (a.mass != nullptr ? a.mass[i] : kMC) * vv;
        }
    }
    block_sum_store<2>(acc, sm, a.part_ke + 2 * blk);
}

namespace {

// The start of a step and the first half-kick with drift in one launch: every
// block copies the step scalars into shared memory and runs the thermostat,
// barostat and cell update on its copy (the same arithmetic on the same
// inputs, so every copy is the same), kicks and drifts its particles with
// them and takes a ticket; the last block, once every block has read the old
// scalars, writes its copy back and so resets the ticket.
__global__ void __launch_bounds__(kPB) k_begin_kick(StepArrays a, StepParams p) {
    FMD_PDL_WAIT();
    __shared__ SysScal sS;
    __shared__ bool last;
    static_assert(sizeof(SysScal) % sizeof(int) == 0, "SysScal copied as words");
    constexpr int kWords = sizeof(SysScal) / sizeof(int);
    const int* src = reinterpret_cast<const int*>(a.S);
    int* dst = reinterpret_cast<int*>(&sS);
    for (int k = threadIdx.x; k < kWords; k += blockDim.x) dst[k] = src[k];
    __syncthreads();
    // the particles' loads wait beside thread 0's scalars
    const int i0 = blockIdx.x * blockDim.x + threadIdx.x;
    KickIn in;
    if (i0 < a.n) in = kick_load(a, i0);
    if (threadIdx.x == 0) {
        begin_body(&sS, a.kind, p);
        sS.kick_done = 0u;                     // a block that starts late has copied other blocks' tickets
    }
    __syncthreads();
    kick_body(a, p.dt, blockIdx.x, gridDim.x, &sS, &in);
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&a.S->kick_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    int* out = reinterpret_cast<int*>(a.S);
    for (int k = threadIdx.x; k < kWords; k += blockDim.x) out[k] = dst[k];
}

__global__ void __launch_bounds__(kPB) k_ke_partial(StepArrays a) {
    __shared__ double sm[32 * 2];
    const bool rigid = a.kind == FMD_SYS_RIGID;
    double acc[2] = {0.0, 0.0};
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
        const double vv = a.vel[3 * i] * a.vel[3 * i] + a.vel[3 * i + 1] * a.vel[3 * i + 1] +
                          a.vel[3 * i + 2] * a.vel[3 * i + 2];
        if (rigid) {
            acc[0] += vv;
            acc[1] += a.omg[3 * i] * a.omg[3 * i] + a.omg[3 * i + 1] * a.omg[3 * i + 1] +
                      a.omg[3 * i + 2] * a.omg[3 * i + 2];
        } else {
            acc[0] += (a.mass != nullptr ? a.mass[i] : kMC) * vv;
        }
    }
    block_sum_store<2>(acc, sm, a.part_ke + 2 * blockIdx.x);
}

}  // namespace

__device__ void rescale_body(const StepArrays& a, int blk, int nblk, double* sm) {
    const SysScal* S = a.S;
    const bool rigid = a.kind == FMD_SYS_RIGID;
    const bool doit = S->do_rescale != 0;
    const double sc = S->scale;
    double acc[2] = {0.0, 0.0};
    for (int i = blk * blockDim.x + threadIdx.x; i < a.n; i += nblk * blockDim.x) {
        double vv = 0, ww = 0;
        for (int c = 0; c < 3; c++) {
            double v = a.vel[3 * i + c];
            if (doit) { v *= sc; a.vel[3 * i + c] = v; }
            vv += v * v;
            if (rigid) {
                double w = a.omg[3 * i + c];
                if (doit) { w *= sc; a.omg[3 * i + c] = w; }
                ww += w * w;
            }
        }
        if (rigid) { acc[0] += vv; acc[1] += ww; }
        else acc[0] += (a.mass != nullptr ? a.mass[i] : kMC) * vv;
    }
    block_sum_store<2>(acc, sm, a.part_ke + 2 * blk);
}

namespace {

__global__ void __launch_bounds__(kPB) k_rescale(StepArrays a) {
    FMD_PDL_WAIT();
    __shared__ double sm[32 * 2];
    rescale_body(a, blockIdx.x, gridDim.x, sm);
}

// Sums of the partial records, t[]: [0,10) part_f1 fields, [10,20) part_f2
// fields, [20] part_f3, [21,23) kinetic; valid in every thread.  The record
// arrays are read as they lie, element by element across the threads (a thread
// stride that is a multiple of the record width keeps a thread on one field),
// the first loads of all arrays before any is used; then a warp sums the
// threads of a field.  Fixed order.  The step's end is one block's latency, so
// code and waits are kept short: k_kick2_end takes 7.6 us at 1,920 atoms and
// 9.5 us at 30,000, against 12.0 and 13.2 us when a thread walked whole records
// 80 bytes from its neighbour's, 23 fields were summed over the block one
// after the other and one thread did all scalar work.
constexpr int kRedFields = 23;
constexpr int kRedShared = 4 * kRedThreads + kRedFields + 1;

// Threads that read an array of this record width.
__device__ __forceinline__ int red_stride(int width) {
    const bool half = blockDim.x == 256;
    return width == 10 ? (half ? 250 : 510) : (width == 7 ? (half ? 252 : 511) : (int)blockDim.x);
}

// One array's sum by threads: NU loads, then the rest NU at a time.
template <int NU>
struct FlatSum {
    const double* part;
    int stride, n, e;
    double v[NU];
    __device__ __forceinline__ FlatSum(const double* p, int nrec, int width)
        : part(p), stride(red_stride(width)), n((int)threadIdx.x < stride ? nrec * width : 0), e(threadIdx.x) {
        load();
    }
    __device__ __forceinline__ void load() {               // L2: other blocks of the launch wrote them
#pragma unroll
        for (int u = 0; u < NU; u++) v[u] = e + u * stride < n ? __ldcg(part + e + u * stride) : 0.0;
        e += NU * stride;
    }
    __device__ __forceinline__ double sum() {
        double acc = 0.0;
        for (;;) {
#pragma unroll
            for (int u = 0; u < NU; u++) acc += v[u];
            if (e >= n) return acc;
            load();
        }
    }
};

__device__ void reduce_all(const StepArrays& a, int nblk_f1, int nblk_ke, bool forces, bool kinetic, double* sm,
                           const double*& t, int nblk_f2) {
    const int nt = blockDim.x, w1 = a.kind == FMD_SYS_MM ? kMMNV : kNV;
    {
        FlatSum<2> k(a.part_ke, kinetic ? nblk_ke : 0, 2);
        FlatSum<8> f1(a.part_f1, forces ? nblk_f1 : 0, w1), f2(a.part_f2, forces && a.kind != FMD_SYS_RIGID ? nblk_f2 : 0, kNV);
        sm[3 * nt + threadIdx.x] = k.sum();
        sm[threadIdx.x] = f1.sum();
        double v2 = f2.sum(), v3 = 0.0;
        if (forces && a.kind == FMD_SYS_MM && a.has_charge) v3 = FlatSum<2>(a.part_f3, kForceBlocks, 1).sum();
        // the switched-LJ correction belongs to the LJ term
        if (forces && a.kind == FMD_SYS_AIREBO && (a.rebo2_flags & FMD_REBO2_LJ_SWITCH))
            v2 += FlatSum<8>(a.part_sw, kForceBlocks, kNV).sum();
        sm[nt + threadIdx.x] = v2;
        sm[2 * nt + threadIdx.x] = v3;
    }
    __syncthreads();
    double* out = sm + 4 * kRedThreads;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    constexpr int kRounds = 3;                             // of 8 (16) warps
    double x[kRounds];
#pragma unroll
    for (int r = 0; r < kRounds; r++) {
        const int f = w + r * (nt >> 5);
        const int arr = f < 10 ? 0 : (f < 20 ? 1 : (f < 21 ? 2 : 3));
        const int width = arr == 0 ? w1 : (arr == 1 ? kNV : (arr == 2 ? 1 : 2));
        const int k = f < 20 ? f - 10 * arr : (f < 21 ? 0 : f - 21), end = red_stride(width);
        x[r] = 0.0;
        if (f < kRedFields && k < width)
            for (int q = lane * width + k; q < end; q += 32 * width) x[r] += sm[arr * nt + q];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int r = 0; r < kRounds; r++) x[r] += __shfl_xor_sync(kFull, x[r], o);
    if (lane == 0)
#pragma unroll
        for (int r = 0; r < kRounds; r++)
            if (w + r * (nt >> 5) < kRedFields) out[w + r * (nt >> 5)] = x[r];
    __syncthreads();
    t = out;
}

// Thread 0: kinetic energies from the reduced sums into S (a.S or a copy).
__device__ void kinetic_from_sums(SysScal* S, const StepArrays& a, const double* t) {
    if (a.kind == FMD_SYS_RIGID) {
        S->kt = 0.5 * a.Mmol * t[21] / kConv;     // LJ:411
        S->kr = 0.5 * a.I0 * t[22] / kConv;       // LJ:420
        S->KE = S->kt + S->kr;
    } else {
        S->KE = 0.5 * t[21] / kConv;              // AI:506, MM:799
    }
}

// Virial entry q and energy q (program grouping) from the reduced sums.
__device__ __forceinline__ double virial_of(int kind, const double* t, int q) {
    if (kind == FMD_SYS_RIGID) return t[1 + q];
    if (kind == FMD_SYS_AIREBO) return t[1 + q] + t[11 + q];
    return q % 4 == 0 ? t[4 + q / 4] + t[11 + q] : 0.0;
}
__device__ __forceinline__ double energy_of(const StepArrays& a, const double* t, int q) {
    if (a.kind == FMD_SYS_RIGID) return q == 0 ? t[0] : 0.0;
    if (a.kind == FMD_SYS_AIREBO) return q == 0 ? t[0] + t[10] : (q == 1 ? t[0] : (q == 2 ? t[10] : 0.0));
    const double ec = a.has_charge ? t[20] : 0.0;
    return q < 4 ? t[q] : (q == 4 ? t[10] : (q == 5 ? ec : (q == 6 ? t[0] + t[1] + t[2] + t[3] + t[10] + ec : 0.0)));
}

// Threads 32.. of the block: virial and energies into S (a.S or a copy).
__device__ __forceinline__ void forces_from_sums(SysScal* S, const StepArrays& a, const double* t) {
    const int q = (int)threadIdx.x - 32;
    if (q >= 0 && q < 9) S->W9[q] = virial_of(a.kind, t, q);
    if (q >= 32 && q < 40) S->E[q - 32] = energy_of(a, t, q - 32);
}

// Observables, averages and the monitor record (LJ:874-897, AI:896-912,
// MM:1215-1236), by threads of one block on S: thread 0 temperature, pressure,
// lattice constant and kinetic energy, eight threads from first the energies,
// each its own (e: energy q, d: the energy of the q-th average).
__device__ __forceinline__ void record_state(SysScal* S, const StepParams& p) {
    const int g = S->gstep;
    const double an = S->h[0] / p.nc;
    S->an = an;
    if (g >= p.gavg_from && g <= p.gavg_to) {
        fmd_avg& A = S->avg;
        A.sT += S->Tn; A.sP += S->Pn; A.sa += an;
        A.n++;
    }
    fmd_obs& o = S->obs;
    o.step = g; o.T = S->Tn; o.P = S->Pn; o.a = an; o.KE = S->KE;
}
// The energy of the program's q-th average: rigid {Ep}; AIREBO {REBO, LJ,
// total}; MM {bond, angle, dihedral + improper, LJ, total}.
__device__ __forceinline__ double average_energy(int kind, const double* E, int q) {
    if (kind == FMD_SYS_RIGID) return E[0];
    if (kind == FMD_SYS_AIREBO) return E[q == 2 ? 0 : q + 1];
    return q == 2 ? E[2] + E[3] : E[q < 2 ? q : (q == 3 ? 4 : 6)];
}
__device__ __forceinline__ void record_energy(SysScal* S, int kind, const StepParams& p, const double* E, int q) {
    const int g = S->gstep;
    if (g >= p.gavg_from && g <= p.gavg_to && q < (kind == FMD_SYS_RIGID ? 1 : (kind == FMD_SYS_AIREBO ? 3 : 5)))
        S->avg.sE[q] += average_energy(kind, E, q) / p.nmol;
    S->obs.E[q] = E[q];
}

}  // namespace

// After the LJ gather of a force evaluation (thread 0 of its reduction): when
// that gather pruned (the same decision on the same inputs), the displacement
// bound restarts from this step's positions and cell hh; counts evaluations
// and prunes.
__device__ void lj_prune_commit(const StepArrays& a, const double* hh) {
    if (!a.prune_hb || !(a.prune_delta > 0.0)) return;
    if (!a.prune_walk) {
        atomicAdd(&a.prune_stats[0], 1ull);
        return;
    }
    const int mode = a.clus.on ? lj_clus_mode(a.clus, a.prune_umax, hh, a.prune_hb, a.prune_delta, a.prune_rc)
                     : lj_prune_needed(a.prune_umax, hh, a.prune_hb, a.prune_delta, a.prune_rc, kRowsAtoms)
                         ? ATOMS_PRUNE
                         : ATOMS_WALK;
    if (a.clus.on && mode == ATOMS_PRUNE) a.clus.flag[2] = 0;          // the gather has built the full rows
    if (lj_clus_prunes(mode)) {
        a.prune_umax[0] = 0ull;
        a.prune_umax[1] = lj_rows_tag(lj_clus_kind(mode), a.prune_delta);
        for (int q = 0; q < 9; q++) a.prune_hb[q] = hh[q];
        atomicAdd(&a.prune_stats[1], 1ull);
    }
    atomicAdd(&a.prune_stats[0], 1ull);
    atomicAdd(&a.prune_stats[4 + mode], 1ull);
}

// The scalar end of a step on the copy S, by the block's threads: thread 0 the
// kinetic energy, the thermostat/barostat second half and the driver's
// temperature and pressure; others the virial and the energies with their
// averages meanwhile.
__device__ void end_scalars(const StepArrays& a, const StepParams& p, const double* t, SysScal* S) {
    const bool rigid = a.kind == FMD_SYS_RIGID;
    const int g = S->gstep;
    const bool phase = g <= p.coldstart || g <= p.coldstart + p.warmup;
    const bool rec = p.schedule && !phase;
    if (threadIdx.x != 0) {
        forces_from_sums(S, a, t);
        const int q = (int)threadIdx.x - 64;
        if (rec && q >= 0 && q < 8) {
            double E[8];
#pragma unroll
            for (int k = 0; k < 8; k++) E[k] = energy_of(a, t, k);
            record_energy(S, a.kind, p, E, q);
        }
        return;
    }
    double W[9];
#pragma unroll
    for (int q = 0; q < 9; q += 4) W[q] = virial_of(a.kind, t, q);
    kinetic_from_sums(S, a, t);
    const double hdt = 0.5 * p.dt;
    const double V = fabs(det9(S->h));
    if (rigid) npt_half(S->npt, hdt, S->KE, S->kt, W, V, 0.1, 0.01);
    else npt_half(S->npt, hdt, S->KE, S->KE, W, V, 0.05, 0.005);
    if (!p.schedule) return;
    // Driver observables after step_npt (LJ:874-876, AI:896, MM:1215-1219).
    S->Tn = inst_T(S->KE, S->npt.Nf);
    S->Pn = inst_P(W, rigid ? S->kt : S->KE, V);
    S->do_rescale = 0;
    if (phase && S->Tn > 0.1) {                                      // LJ:879-894
        const double tgt = (g <= p.coldstart) ? p.T_cold : S->npt.Tt;
        S->scale = sqrt(fmax(tgt, 0.1) / S->Tn);
        S->do_rescale = 1;
    }
    if (rec) record_state(S, p);
}

// The end of a step in one block: the block copies the step scalars into
// shared memory (sS) and reduces the partial records, thread 0 runs the
// scalar end on that copy (shared-memory latency on its serial chain instead
// of global), and the block writes the copy back with the block ticket
// kick2_done reset.  No other block reads the scalars meanwhile.
__device__ void end_body(const StepArrays& a, const StepParams& p, int nblk_f1, int nblk_ke, int nblk_f2,
                         double* sm, SysScal* sS) {
    static_assert(sizeof(SysScal) % sizeof(int) == 0, "SysScal copied as words");
    constexpr int kWords = sizeof(SysScal) / sizeof(int);
    int* gS = reinterpret_cast<int*>(a.S);
    int* cS = reinterpret_cast<int*>(sS);
    for (int k = threadIdx.x; k < kWords; k += blockDim.x) cS[k] = __ldcg(gS + k);
    // the prune bookkeeping reads only the cell: beside the reduction
    if (threadIdx.x == blockDim.x - 32) lj_prune_commit(a, a.S->h);
    const double* t;
    reduce_all(a, nblk_f1, nblk_ke, true, true, sm, t, nblk_f2);
    end_scalars(a, p, t, sS);
    if (threadIdx.x == 0) sS->kick2_done = 0u;
    __syncthreads();
    for (int k = threadIdx.x; k < kWords; k += blockDim.x) gS[k] = cS[k];
}

__device__ void rescale_end_body(const StepArrays& a, const StepParams& p, int nblk_ke, double* sm) {
    SysScal* S = a.S;
    const bool doit = S->do_rescale != 0;
    const double* t;
    if (doit) reduce_all(a, 0, nblk_ke, false, true, sm, t, 0);
    if (threadIdx.x == 0) {
        if (doit) {
            kinetic_from_sums(S, a, t);
            S->Tn = inst_T(S->KE, S->npt.Nf);
            S->npt.xi = 0;
            if (S->gstep <= p.coldstart)
                for (int k = 0; k < 9; k++) S->npt.Vg[k] = 0;
        }
        record_state(S, p);
    }
    const int q = (int)threadIdx.x - 64;
    if (q >= 0 && q < 8) {
        double E[8];
        for (int k = 0; k < 8; k++) E[k] = S->E[k];
        record_energy(S, a.kind, p, E, q);
    }
}

namespace {

// The second half-kick and the end of the step in one launch: every block
// writes its kinetic partial and takes a ticket; the last block to finish
// runs end_body (the same fixed-order reduction of all partial records, so
// the result does not depend on which block is last) and resets the ticket.
__global__ void __launch_bounds__(kPB) k_kick2_end(StepArrays a, StepParams p, int nblk_f1) {
    FMD_PDL_WAIT();
    __shared__ double sm[kRedShared];
    __shared__ SysScal sS;
    __shared__ bool last;
    kick2_body(a, p.dt, blockIdx.x, gridDim.x, sm);
    __threadfence();                      // this block's partial before its ticket
    if (threadIdx.x == 0) last = atomicAdd(&a.S->kick2_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    end_body(a, p, nblk_f1, gridDim.x, a.lj_blocks, sm, &sS);   // resets kick2_done
}

// The same for the rigid pair kernel (rigidpair.cu), a warp per molecule: its
// force and torque are summed here, kept for the next step's first kick and
// applied by the warp's first lane.  Each block writes one force and one
// kinetic record.
__global__ void __launch_bounds__(kPB) k_rigid_kick2_end(StepArrays a, StepParams p) {
    FMD_PDL_WAIT();
    __shared__ double sm[kRedShared];
    __shared__ SysScal sS;
    __shared__ bool last;
    const int lane = threadIdx.x & 31;
    const double hdt = 0.5 * p.dt, sc_v2 = a.S->sc_v2, sc_nh = a.S->sc_nh, cF = kConv / a.Mmol, cT = kConv / a.I0;
    double tot[kNV], vv = 0.0, ww = 0.0, acc[kNV + 2];
#pragma unroll
    for (int k = 0; k < kNV; k++) tot[k] = 0.0;
    for (int i = blockIdx.x * (kPB / 32) + (threadIdx.x >> 5); i < a.n; i += gridDim.x * (kPB / 32)) {
        double v[6];
        rigid_pair_sum(a.rigid_pair, a.cnt_a, a.list_a, a.cap_a, i, lane, v, tot);
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < 3; c++) {
                a.F[3 * i + c] = v[c];
                a.T[3 * i + c] = v[3 + c];
                const double x = (a.vel[3 * i + c] + hdt * v[c] * cF) * sc_v2;
                a.vel[3 * i + c] = x;
                vv += x * x;
                const double w = (a.omg[3 * i + c] + hdt * v[3 + c] * cT) * sc_nh;
                a.omg[3 * i + c] = w;
                ww += w * w;
            }
    }
#pragma unroll
    for (int k = 0; k < kNV; k++) acc[k] = tot[k];
    acc[kNV] = vv;
    acc[kNV + 1] = ww;
    __shared__ double rec[kNV + 2];
    block_sum_fields<kNV + 2>(acc, sm, rec);
    if (threadIdx.x < kNV) a.part_f1[(size_t)blockIdx.x * kNV + threadIdx.x] = rec[threadIdx.x];
    else if (threadIdx.x < kNV + 2) a.part_ke[2 * blockIdx.x + threadIdx.x - kNV] = rec[threadIdx.x];
    __threadfence();                      // this block's records before its ticket
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&a.S->kick2_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    end_body(a, p, gridDim.x, gridDim.x, 0, sm, &sS);   // resets kick2_done
}

__global__ void __launch_bounds__(kRedThreads) k_rescale_end(StepArrays a, StepParams p, int nblk_ke) {
    FMD_PDL_WAIT();
    __shared__ double sm[kRedShared];
    rescale_end_body(a, p, nblk_ke, sm);
}

__global__ void __launch_bounds__(kRedThreads) k_ke_final(StepArrays a, int nblk_ke) {
    __shared__ double sm[kRedShared];
    const double* t;
    reduce_all(a, 0, nblk_ke, false, true, sm, t, 0);
    if (threadIdx.x == 0) kinetic_from_sums(a.S, a, t);
}

// ---- replica batch: each single-system kernel once over all replicas ----
__global__ void k_b_begin(BatchDev b) {
    if (threadIdx.x != 0) return;
    const StepArrays& a = b.A[blockIdx.x];
    begin_body(a.S, a.kind, b.P[blockIdx.x]);
}

__global__ void __launch_bounds__(kPB) k_b_kick(BatchDev b) {
    const int r = batch_rep(b.off_atom, b.R, blockIdx.x);
    kick_body(b.A[r], b.P[r].dt, blockIdx.x - b.off_atom[r], b.off_atom[r + 1] - b.off_atom[r]);
}

__global__ void __launch_bounds__(kPB) k_b_kick2(BatchDev b) {
    __shared__ double sm[32 * 2];
    const int r = batch_rep(b.off_atom, b.R, blockIdx.x);
    kick2_body(b.A[r], b.P[r].dt, blockIdx.x - b.off_atom[r], b.off_atom[r + 1] - b.off_atom[r], sm);
}

__global__ void __launch_bounds__(kPB) k_b_rescale(BatchDev b) {
    __shared__ double sm[32 * 2];
    const int r = batch_rep(b.off_atom, b.R, blockIdx.x);
    rescale_body(b.A[r], blockIdx.x - b.off_atom[r], b.off_atom[r + 1] - b.off_atom[r], sm);
}

__global__ void __launch_bounds__(256) k_b_end(BatchDev b) {
    __shared__ double sm[kRedShared];
    __shared__ SysScal sS;
    const int r = blockIdx.x;
    end_body(b.A[r], b.P[r], b.off_f1[r + 1] - b.off_f1[r], b.off_atom[r + 1] - b.off_atom[r],
             b.off_lj[r + 1] - b.off_lj[r], sm, &sS);
}

__global__ void __launch_bounds__(256) k_b_rescale_end(BatchDev b) {
    __shared__ double sm[kRedShared];
    const int r = blockIdx.x;
    rescale_end_body(b.A[r], b.P[r], b.off_atom[r + 1] - b.off_atom[r], sm);
}

__global__ void __launch_bounds__(kRedThreads) k_force_final(StepArrays a, int nblk_f1) {
    __shared__ double sm[kRedShared];
    const double* t;
    reduce_all(a, nblk_f1, 0, true, false, sm, t, a.lj_blocks);
    forces_from_sums(a.S, a, t);
    if (threadIdx.x == 0) lj_prune_commit(a, a.S->h);
}

}  // namespace

int force_partial_blocks(const StepArrays& a) {
    if (a.kind == FMD_SYS_RIGID && a.rigid_pair.on) return rigid_pair_records(a.n);
    return a.kind == FMD_SYS_RIGID ? rigid_grid(a.n) : (a.kind == FMD_SYS_AIREBO ? a.rebo_blocks : mm_bonded_blocks(a.topo));
}

// LJ term of an atomistic system: the gather over the full rows, or with
// pruned rows the gather that decides per evaluation between pruning the full
// rows and walking the pruned ones.
cudaError_t enqueue_lj(const StepArrays& a, int ff, cudaStream_t st) {
    const double* hh = a.S->h;
    if (!a.prune || a.prune->delta <= 0.0)
        return lj_gather_launch(ff, a.pos, hh, a.cnt_a, a.list_a, a.cap_a, a.in_cnt, a.in_list, a.in_cap, a.n, a.F,
                                a.Facc, a.part_f2, st, a.precision, a.lj_shape, a.err, LJPruneOut{}, a.lj_blocks);
    if (a.clus.on)
        return lj_clus_launch(ff, a.clus, a.pos, hh, a.n, a.F, a.Facc, a.part_f2, st, a.precision,
                              lj_prune_out(*a.prune), a.lj_blocks);
    // one launch: each block decides whether this evaluation prunes (full
    // rows, pruned rows written) or walks the pruned rows; the step's
    // reduction then restarts the displacement bound (lj_prune_commit)
    return lj_gather_launch(ff, a.pos, hh, a.cnt_a, a.list_a, a.cap_a, a.in_cnt, a.in_list, a.in_cap, a.n, a.F,
                            a.Facc, a.part_f2, st, a.precision, a.lj_shape_p, a.err, lj_prune_out(*a.prune),
                            a.lj_blocks);
}

cudaError_t enqueue_rigid(const StepArrays& a, cudaStream_t st, bool reduce) {
    const double* hh = a.S->h;
    if (a.rigid_pair.on) {
        const cudaError_t e = rigid_pair_launch(a.rigid_pair, a.precision, a.pos, a.qv, a.body, hh, a.cnt_a, a.list_a,
                                                a.cap_a, a.n, a.natom, a.rmcut2, st);
        if (e != cudaSuccess || !reduce) return e;
        return rigid_pair_reduce(a.rigid_pair, a.cnt_a, a.list_a, a.cap_a, a.n, a.F, a.T, a.part_f1, st);
    }
    return rigid_launch(a.precision, a.pos, a.qv, a.body, hh, a.cnt_a, a.list_a, a.cap_a, a.n, a.natom, a.rmcut2, a.F,
                        a.T, a.part_f1, st, a.rigid_lab);
}

cudaError_t enqueue_forces(const StepArrays& a, cudaStream_t st, bool judge, bool reduce) {
    cudaError_t e = cudaSuccess;
    const double* hh = a.S->h;
    if (a.kind == FMD_SYS_RIGID) {
        e = enqueue_rigid(a, st, reduce);
    } else if (a.kind == FMD_SYS_AIREBO) {
        if (a.rebo2_flags & FMD_REBO2_BOND_ORDER)
            e = rebo2_launch(a.rebo2, a.pos, hh, a.cnt_b, a.list_b, a.cap_b, a.n, a.Facc, a.part_f1, a.rebo_blocks,
                             st);
        else if (a.sg) e = sg_enqueue_rebo(*a.sg, a, judge, st);
        else if (a.rebo_slots || a.rebo_mol.M)
            e = rebo_slots_launch(a.pos, hh, a.cnt_b, a.list_b, a.cap_b, a.n, a.rebo_slots, a.Facc, a.part_f1,
                                  a.rebo_blocks, nullptr, 0, st, a.rebo_ids, a.rebo_phys != 0, a.rebo_mol);
        else e = rebo_launch(a.pos, hh, a.cnt_b, a.list_b, a.cap_b, a.n, a.Facc, a.part_f1, st);
        if (e != cudaSuccess) return e;
        e = enqueue_lj(a, FMD_FF_AIREBO, st);
        // the switched LJ: its correction adds into the finished F
        if (e == cudaSuccess && (a.rebo2_flags & FMD_REBO2_LJ_SWITCH))
            e = lj_switch_launch(a.rebo2, a.pos, hh, a.cnt_b, a.list_b, a.cap_b, a.cnt_a, a.list_a, a.cap_a, a.n,
                                 a.F, a.part_sw, kForceBlocks, (a.rebo2_flags & FMD_REBO2_BOND_ORDER) != 0, st);
    } else {
        if ((e = mm_bonded_launch(a.topo, a.pos, hh, a.Facc, a.part_f1, st)) != cudaSuccess) return e;
        if (a.has_charge)
            if ((e = mm_coulomb_launch(a.pos, hh, a.charge, a.mol_id, a.n, a.Facc, a.part_f3, st)) != cudaSuccess) return e;
        e = enqueue_lj(a, FMD_FF_MM, st);
    }
    return e;
}

cudaError_t enqueue_force_reduce(const StepArrays& a, cudaStream_t st) {
    k_force_final<<<1, kRedThreads, 0, st>>>(a, force_partial_blocks(a));
    return cudaGetLastError();
}

cudaError_t enqueue_ke(const StepArrays& a, cudaStream_t st) {
    k_ke_partial<<<kForceBlocks, kPB, 0, st>>>(a);
    k_ke_final<<<1, kRedThreads, 0, st>>>(a, kForceBlocks);
    return cudaGetLastError();
}

cudaError_t enqueue_step(const StepArrays& a, const StepParams& p, bool rescale_phase, cudaStream_t st,
                         bool judge) {
    cudaError_t e;
    // programmatic dependent launches: each kernel's launch overlaps the
    // previous one's tail (pdl.cuh)
    // per-particle kernels: one thread per particle (grid-stride beyond kForceBlocks)
    const int pblocks = std::max(1, std::min(kForceBlocks, (a.n + kPB - 1) / kPB));
    if ((e = launch_pdl(k_begin_kick, dim3(pblocks), dim3(kPB), 0, st, a, p)) != cudaSuccess) return e;
    const bool pairs = a.kind == FMD_SYS_RIGID && a.rigid_pair.on;
    if ((e = enqueue_forces(a, st, judge, !pairs)) != cudaSuccess) return e;
    if (pairs) {
        const int blocks = force_partial_blocks(a);
        if ((e = launch_pdl(k_rigid_kick2_end, dim3(blocks), dim3(kPB), 0, st, a, p)) != cudaSuccess) return e;
    } else if ((e = launch_pdl(k_kick2_end, dim3(pblocks), dim3(kPB), 0, st, a, p, force_partial_blocks(a))) != cudaSuccess)
        return e;
    if (rescale_phase && p.schedule) {
        if ((e = launch_pdl(k_rescale, dim3(kForceBlocks), dim3(kPB), 0, st, a)) != cudaSuccess) return e;
        if ((e = launch_pdl(k_rescale_end, dim3(1), dim3(kRedThreads), 0, st, a, p, kForceBlocks)) != cudaSuccess)
            return e;
    }
    return cudaGetLastError();
}

cudaError_t enqueue_batch_step(const BatchDev& b, bool rescale_phase, cudaStream_t st) {
    cudaError_t e;
    k_b_begin<<<b.R, 32, 0, st>>>(b);
    k_b_kick<<<b.nblk_atom, kPB, 0, st>>>(b);
    if (b.mol_smem) {
        if ((e = batch_mm_mol_launch(b.A, b.off_f1, b.R, b.nblk_f1, b.mol_smem, st)) != cudaSuccess) return e;
    } else if (b.kind == FMD_SYS_MM)
        if ((e = batch_mm_bonded_launch(b.A, b.off_f1, b.R, b.nblk_f1, b.f1_threads, st)) != cudaSuccess) return e;
    if (b.lj_clus) {
        if ((e = batch_lj_clus_launch(b.A, b.off_lj, b.R, b.nblk_lj, b.precision, st)) != cudaSuccess) return e;
    } else if ((e = batch_lj_launch(b.A, b.off_lj, b.R, b.nblk_lj, b.ff, b.precision, b.lj_threads, b.lj_unroll, st,
                             b.lj_staged_in_cap)) != cudaSuccess)
        return e;
    k_b_kick2<<<b.nblk_atom, kPB, 0, st>>>(b);
    k_b_end<<<b.R, 256, 0, st>>>(b);
    if (rescale_phase) {
        k_b_rescale<<<b.nblk_atom, kPB, 0, st>>>(b);
        k_b_rescale_end<<<b.R, 256, 0, st>>>(b);
    }
    return cudaGetLastError();
}

}  // namespace fmd
