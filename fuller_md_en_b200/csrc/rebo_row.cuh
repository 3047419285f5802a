// rebo_row.cuh -- REBO bonds of one list row straight from positions
// (airebo.cu), and the functions that every REBO kernel shares (airebo.cu,
// rebomol.cu).
#pragma once
#include "rebo_fn.cuh"

namespace fmd {
namespace rebo {

__device__ __forceinline__ void ang_g_dg(double x, double& g, double& dg) {
    const double c2 = G_C0 * G_C0, d2 = G_D0 * G_D0, hh = 1.0 + x, inv = 1.0 / (d2 + hh * hh);
    g = G_A0 * (1.0 + c2 / d2 - c2 * inv);
    dg = G_A0 * 2.0 * c2 * hh * inv * inv;
}

__device__ __forceinline__ void rebo_pair_fn(double r, double rinv, double& vr, double& dvr, double& va,
                                             double& dva) {
    const double ea = A_CC * exp(-ALPHA_CC * r);
    const double qr = Q_CC * rinv;
    vr = (1.0 + qr) * ea;
    dvr = (-qr * rinv) * ea + (1.0 + qr) * (-ALPHA_CC) * ea;
    const double e1 = exp(-BETA1_CC * r), e2 = exp(-BETA2_CC * r), e3 = exp(-BETA3_CC * r);
    va = B1_CC * e1 + B2_CC * e2 + B3_CC * e3;
    dva = -BETA1_CC * B1_CC * e1 - BETA2_CC * B2_CC * e2 - BETA3_CC * B3_CC * e3;
}

// Three-body coefficient of centre c for a bond with f_c and V_A.
__device__ __forceinline__ double three_body_coeff(double gs, double b, double fcut, double va) {
    if (!(fabs(gs) > 1e-20 && va > 1e-20)) return 0.0;
    const double dbp = -BO_DELTA * b / (1.0 + gs);
    return -(0.5 * fcut * va) * dbp;
}

// Sum over the centre's other neighbours of fc * G(cos theta) (AI:301-309).
__device__ __forceinline__ double bo_sum(const double* __restrict__ pos, const int* __restrict__ cnt,
                         const int* __restrict__ list, int cap, const double* h, const double* hi,
                         int c, int skip, double bx, double by, double bz, double rb) {
    double gs = 0.0;
    const int m = cnt[c];
    for (int kn = 0; kn < m; kn++) {
        const int k = list[(size_t)c * cap + kn];
        if (k == skip) continue;
        double kx, ky, kz;
        bond_vec(pos, c, k, h, hi, kx, ky, kz);
        const double rk = sqrt(norm2_rn(kx, ky, kz));
        if (rk > DMAX_CC) continue;
        const double fk = sw_fc(rk);
        if (fk < 1e-15) continue;
        const double ct = clamp1((bx * kx + by * ky + bz * kz) / (rb * rk));
        gs += fk * ang_g(ct);
    }
    return gs;
}

// Three-body forces on the neighbours of centre c (AI:361-419).  PHYS: the
// gradient of the bond-order term instead of the reference's (opposite sign on
// the neighbours, and the term on the bond partner `skip`).
// b = (1+gs)^-1/2 is passed in, so db/dgs = -1/2 (1+gs)^-3/2 = -b / (2 (1+gs)).
template <bool PHYS>
__device__ __forceinline__ void bo_three_body(double* __restrict__ F, const double* __restrict__ pos,
                              const int* __restrict__ cnt, const int* __restrict__ list, int cap,
                              const double* h, const double* hi, int c, int skip, double bx, double by,
                              double bz, double rb, double ux, double uy, double uz, double gs, double b,
                              double fcut, double va) {
    if (!(fabs(gs) > 1e-20 && va > 1e-20)) return;
    const double dbp = -BO_DELTA * b / (1.0 + gs);
    const double vh = 0.5 * fcut * va;
    const double coeff = -vh * dbp;
    const int m = cnt[c];
    double fcx = 0.0, fcy = 0.0, fcz = 0.0;
    double fbx = 0.0, fby = 0.0, fbz = 0.0;
    for (int kn = 0; kn < m; kn++) {
        const int k = list[(size_t)c * cap + kn];
        if (k == skip) continue;
        double kx, ky, kz;
        bond_vec(pos, c, k, h, hi, kx, ky, kz);
        const double rk = sqrt(norm2_rn(kx, ky, kz));
        if (rk > DMAX_CC) continue;
        const double fck = sw_fc(rk);
        if (fck < 1e-15) continue;
        const double dfck = sw_dfc(rk);
        const double rki = 1.0 / rk;
        const double rx = kx * rki, ry = ky * rki, rz = kz * rki;
        const double ct = clamp1((bx * kx + by * ky + bz * kz) / (rb * rk));
        const double gv = ang_g(ct), dgv = ang_dg(ct);
        const double a1 = PHYS ? -(coeff * dfck * gv) : coeff * dfck * gv;
        const double a2 = PHYS ? -(coeff * fck * dgv) : coeff * fck * dgv;
        const double fx = a1 * rx + a2 * ((ux - ct * rx) * rki);
        const double fy = a1 * ry + a2 * ((uy - ct * ry) * rki);
        const double fz = a1 * rz + a2 * ((uz - ct * rz) * rki);
        atomic_add3(F, k, fx, fy, fz);
        fcx -= fx; fcy -= fy; fcz -= fz;
        if (PHYS) {
            const double a3 = a2 / rb;
            fbx += a3 * (rx - ct * ux); fby += a3 * (ry - ct * uy); fbz += a3 * (rz - ct * uz);
        }
    }
    if (PHYS) {
        atomic_add3(F, skip, fbx, fby, fbz);
        fcx -= fbx; fcy -= fby; fcz -= fbz;
    }
    atomic_add3(F, c, fcx, fcy, fcz);
}

// The bonds j > i of row i in slots lane, lane + step, ...: forces by atomics
// into F, {E, W9} added to acc.
template <bool PHYS>
__device__ __forceinline__ void rebo_row(const double* __restrict__ pos, const double* h, const double* hi,
                                         const int* __restrict__ cnt, const int* __restrict__ list, int cap, int i,
                                         int lane, int step, double* __restrict__ F, double (&acc)[kNV]) {
    const int m = cnt[i];
    double fix = 0.0, fiy = 0.0, fiz = 0.0;
    for (int jn = lane; jn < m; jn += step) {
        const int j = list[(size_t)i * cap + jn];
        if (j <= i) continue;
        double dx, dy, dz;
        bond_vec(pos, i, j, h, hi, dx, dy, dz);
        const double rij = sqrt(norm2_rn(dx, dy, dz));
        if (rij > DMAX_CC) continue;
        const double fcut = sw_fc(rij), dfcut = sw_dfc(rij);
        if (fcut < 1e-15 && dfcut == 0) continue;
        // V_R, V_A and derivatives (AI:173-183)
        const double ea = A_CC * exp(-ALPHA_CC * rij);
        const double vr = (1.0 + Q_CC / rij) * ea;
        const double dvr = (-Q_CC / (rij * rij)) * ea + (1.0 + Q_CC / rij) * (-ALPHA_CC) * ea;
        const double e1 = exp(-BETA1_CC * rij), e2 = exp(-BETA2_CC * rij), e3 = exp(-BETA3_CC * rij);
        const double va = B1_CC * e1 + B2_CC * e2 + B3_CC * e3;
        const double dva = -BETA1_CC * B1_CC * e1 - BETA2_CC * B2_CC * e2 - BETA3_CC * B3_CC * e3;
        const double rinv = 1.0 / rij;
        const double ux = dx * rinv, uy = dy * rinv, uz = dz * rinv;
        const double gij = bo_sum(pos, cnt, list, cap, h, hi, i, j, dx, dy, dz, rij);
        const double gji = bo_sum(pos, cnt, list, cap, h, hi, j, i, -dx, -dy, -dz, rij);
        // (1+g)^-1/2 (AI:310, 323) as a reciprocal square root
        const double bij = 1.0 / sqrt(1.0 + gij), bji = 1.0 / sqrt(1.0 + gji);
        const double bbar = 0.5 * (bij + bji);
        acc[0] += fcut * (vr - bbar * va);
        const double fpair = (dfcut * (vr - bbar * va) + fcut * (dvr - bbar * dva)) * rinv;
        fix += fpair * dx; fiy += fpair * dy; fiz += fpair * dz;
        atomic_add3(F, j, -fpair * dx, -fpair * dy, -fpair * dz);
        const double d[3] = {dx, dy, dz};
#pragma unroll
        for (int a = 0; a < 3; a++)
#pragma unroll
            for (int b = 0; b < 3; b++) acc[1 + a * 3 + b] -= d[a] * fpair * d[b];
        bo_three_body<PHYS>(F, pos, cnt, list, cap, h, hi, i, j, dx, dy, dz, rij, ux, uy, uz, gij, bij, fcut, va);
        bo_three_body<PHYS>(F, pos, cnt, list, cap, h, hi, j, i, -dx, -dy, -dz, rij, -ux, -uy, -uz, gji, bji, fcut,
                      va);
    }
    if (fix != 0.0 || fiy != 0.0 || fiz != 0.0) atomic_add3(F, i, fix, fiy, fiz);
}

}  // namespace rebo
}  // namespace fmd
