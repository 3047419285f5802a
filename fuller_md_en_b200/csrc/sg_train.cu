// sg_train.cu -- training of the learned bond-order potential on the GPU.
//
// One step on a snapshot with reference REBO energy, forces and virial:
//   inference path (surrogate.cu)            b, db/dx, E, F, W
//   k_sg_lambda                              dL/dF per atom, sum dF^2
//   k_sg_adjoint                             per row dL/db and dL/d(db/dx)
//   k_sg_chain  (tcgen05, 10 GEMMs / tile)   double backpropagation through
//                                            the network; writes the BF16
//                                            operand tiles of the weight
//                                            gradients, sums dL/dw4
//   k_sg_wgrad  (tcgen05)                    dW_l = sum over rows, reduced in
//                                            TMEM per CTA
//   k_sg_adam                                FP64 master weights, then repack
// The loss is  wF mean(dF^2) + wE (dE/na)^2 + wW mean((dW/na)^2)  with dF over
// the REBO forces; every step restates oracle/sg_oracle.py:mlp_backward with
// the same BF16 rounding points.
#include <cuda_bf16.h>

#include "kernels.h"
#include "pdl.cuh"
#include "sg_dev.cuh"
#include "sg_train.cuh"
#include "umma.cuh"

namespace fmd {
namespace sg {
namespace {

using namespace dev;

// ------------------------------------------------------------- adjoints
__global__ void __launch_bounds__(256)
k_sg_lambda(const double* __restrict__ F, const double* __restrict__ Fref, int na, double wF,
            double* __restrict__ lamF, double* __restrict__ part) {
    FMD_PDL_WAIT();
    __shared__ double sm[32];
    double acc[1] = {0.0};
    const double k = 2.0 * wF / (3.0 * na);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < 3 * na; e += gridDim.x * blockDim.x) {
        const double d = F[e] - Fref[e];
        lamF[e] = k * d;
        acc[0] += d * d;
    }
    block_sum_store<1>(acc, sm, part + blockIdx.x);
}

// sc: {E, W9} of the prediction; ref: {E, W9} of the reference.
__global__ void k_sg_loss(const double* __restrict__ sc, const double* __restrict__ ref,
                          const double* __restrict__ sumdf2, int na, double wE, double wF, double wW,
                          double* __restrict__ lam, double* __restrict__ loss_acc) {
    FMD_PDL_WAIT();
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const double n2 = (double)na * na;
    const double dE = sc[0] - ref[0];
    double lw = 0.0;
    lam[0] = 2.0 * wE * dE / n2;
    for (int a = 0; a < 9; a++) {
        const double dW = sc[1 + a] - ref[1 + a];
        lam[1 + a] = 2.0 * wW * dW / (9.0 * n2);
        lw += dW * dW;
    }
    loss_acc[0] += wF * sumdf2[0] / (3.0 * na) + wE * dE * dE / n2 + wW * lw / (9.0 * n2);
    loss_acc[1] += sumdf2[0] / (3.0 * na);          // mean dF^2 (for the force RMSE)
}

// One thread per row: beta = dL/db, and the U tile row = dL/d(db/dxn).
__global__ void __launch_bounds__(128)
k_sg_adjoint(const double* __restrict__ pos, const double* __restrict__ hh, const int* __restrict__ cnt,
             const int* __restrict__ list, int cap, int na, const int* __restrict__ aoff,
             const int* __restrict__ row_i, const int* __restrict__ row_s, const float* __restrict__ vec,
             const double* __restrict__ lamF, const double* __restrict__ lam, int r_cap,
             float* __restrict__ beta, uint16_t* __restrict__ U) {
    FMD_PDL_WAIT();
    double h[9], hi[9];
    load_cell(hh, h, hi);
    const int R = aoff[na];
    const int Rpad = (R + TILE - 1) / TILE * TILE;
    const double lE = lam[0];
    double LW[9];
#pragma unroll
    for (int a = 0; a < 9; a++) LW[a] = lam[1 + a];
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < Rpad && r < r_cap; r += gridDim.x * blockDim.x) {
        float u[D];
#pragma unroll
        for (int f = 0; f < D; f++) u[f] = 0.f;
        float bt = 0.f;
        if (r < R) {
            const int i = row_i[r], j = list[(size_t)i * cap + row_s[r]];
            double dx, dy, dz;
            bond_vec(pos, i, j, h, hi, dx, dy, dz);
            const double rij = sqrt(norm2_rn(dx, dy, dz));
            const double fcut = sw_fc(rij), dfcut = sw_dfc(rij);
            const double e1 = exp(-BETA1_CC * rij), e2 = exp(-BETA2_CC * rij), e3 = exp(-BETA3_CC * rij);
            const double va = B1_CC * e1 + B2_CC * e2 + B3_CC * e3;
            const double dva = -BETA1_CC * B1_CC * e1 - BETA2_CC * B2_CC * e2 - BETA3_CC * B3_CC * e3;
            // dL/dfpair through F_i, F_j (pair force) and W (pair virial)
            const double d[3] = {dx, dy, dz};
            double dfp = 0.0, dWd = 0.0;
#pragma unroll
            for (int a = 0; a < 3; a++) {
                dfp += (lamF[3 * i + a] - lamF[3 * j + a]) * d[a];
#pragma unroll
                for (int c = 0; c < 3; c++) dWd += d[a] * LW[3 * a + c] * d[c];
            }
            dfp -= dWd;
            const double phi = -(dfcut * va + fcut * dva) / rij;     // d fpair / d b_bar
            bt = (float)(-0.5 * fcut * va * lE + 0.5 * phi * dfp);
            // dL/d(db/dxn): three-body forces F_k += w db/dr_k, F_i -= the same
            const double w = -0.5 * fcut * va;
            const double rinv = 1.0 / rij;
            const double ux = dx * rinv, uy = dy * rinv, uz = dz * rinv;
            for (int kn = 0; kn < cnt[i]; kn++) {
                const int k = list[(size_t)i * cap + kn];
                if (k == j) continue;
                double kx, ky, kz;
                bond_vec(pos, i, k, h, hi, kx, ky, kz);
                const double rk = sqrt(norm2_rn(kx, ky, kz));
                if (rk > DMAX_CC) continue;
                const double fk = sw_fc(rk);
                if (fk < 1e-15) continue;
                const double dfk = sw_dfc(rk);
                const double ct = clamp1((dx * kx + dy * ky + dz * kz) / (rij * rk));
                const double rki = 1.0 / rk;
                const double rx = kx * rki, ry = ky * rki, rz = kz * rki;
                const double lx = lamF[3 * k] - lamF[3 * i], ly = lamF[3 * k + 1] - lamF[3 * i + 1],
                             lz = lamF[3 * k + 2] - lamF[3 * i + 2];
                const float p1 = (float)(w * (lx * rx + ly * ry + lz * rz));                 // w dl . rhat_k
                const float p2 = (float)(w * (lx * (ux - ct * rx) + ly * (uy - ct * ry) + lz * (uz - ct * rz)) * rki);
                float Tr[NR], dTr[NR], Ta[NA], dTa[NA];
                cheb<NR>((float)((rk - RHO_C) / RHO_W), Tr, dTr);
                cheb<NA>((float)ct, Ta, dTa);
#pragma unroll
                for (int a = 0; a < NR; a++) {
                    const float phi_a = (float)fk * Tr[a];
                    const float dphi_a = (float)dfk * Tr[a] + (float)fk * dTr[a] * (float)(1.0 / RHO_W);
#pragma unroll
                    for (int b = 0; b < NA; b++) u[a * NA + b] += dphi_a * Ta[b] * p1 + phi_a * dTa[b] * p2;
                }
            }
#pragma unroll
            for (int f = 0; f < D - 1; f++) u[f] *= vec[V_SINV + f];
            u[D - 1] = 0.f;
        }
        beta[r] = bt;
        unsigned char* tile = reinterpret_cast<unsigned char*>(U) + (size_t)(r / TILE) * TILE * D * 2;
        const int q = r % TILE;
#pragma unroll
        for (int c8 = 0; c8 < D / 8; c8++) {
            uint4 v;
            v.x = umma::pack_bf16(u[8 * c8 + 0], u[8 * c8 + 1]);
            v.y = umma::pack_bf16(u[8 * c8 + 2], u[8 * c8 + 3]);
            v.z = umma::pack_bf16(u[8 * c8 + 4], u[8 * c8 + 5]);
            v.w = umma::pack_bf16(u[8 * c8 + 6], u[8 * c8 + 7]);
            *reinterpret_cast<uint4*>(tile + umma::il_off(q, 8 * c8, D)) = v;
        }
    }
}

// ------------------------------------------------------------- chain
// 16 warps: four per TMEM lane quadrant, each owning 32 of the 128 columns.
// The sigmoid of z1 and z2 is evaluated twice per element: in the forward
// pass, and where SiLU' and SiLU'' are first needed together; there SiLU'(z)
// replaces z in TMEM for the later stages.  The kernel is bound
// by the serial chain of ten GEMMs and epilogues of a tile (21 us; its special
// functions alone, six sigmoids an element, take 7).  90,000 rows: 102 us; 243
// us with 8 warps, ten sigmoids an element and 160 shuffles per 32 columns of
// dL/dw4.
constexpr int kThreads = 512;
constexpr int kCols = TILE * H / kThreads;   // columns per thread
static_assert(kCols == 32, "two slices of 16 columns per thread");
constexpr int C_W1 = 0, C_W2 = C_W1 + H * D * 2, C_W3 = C_W2 + H * H * 2, C_X = C_W3 + H * H * 2,
              C_U = C_X + TILE * D * 2, C_ACT = C_U + TILE * D * 2, C_E1 = C_ACT + TILE * H * 2,
              C_E2 = C_E1 + TILE * H * 2, C_W4 = C_E2 + TILE * H * 2, C_DW4 = C_W4 + H * 4,
              C_TOTAL = C_DW4 + H * 4;
constexpr uint32_t T_Z1 = 0, T_Z2 = 128, T_Z3 = 256, T_T = 384;

__device__ __forceinline__ unsigned char* gtile(uint16_t* buf, int tile) {
    return reinterpret_cast<unsigned char*>(buf) + (size_t)tile * TILE * H * 2;
}

// The thread's part of a tile: row q, columns c0 .. c0 + 31, its warp's TMEM lanes at tl.
struct ChainThread {
    uint32_t tl;
    int q, c0;
};

// Sums 32 columns over the warp's rows (one per lane) and adds column k's to
// acc[k]: each exchange hands half of the columns over, so lane l ends with
// column l (31 shuffles instead of 160).
__device__ __forceinline__ void add_columns(float (&v)[kCols], float* acc, int lane) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const bool hi = lane & o;
#pragma unroll
        for (int k = 0; k < o; k++) {
            const float send = hi ? v[k] : v[k + o];
            v[k] = (hi ? v[k + o] : v[k]) + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
    atomicAdd(&acc[lane], v[0]);
}

// h = SiLU(z) (column 127: 1) to the operand tile and to out.
__device__ __forceinline__ void chain_forward(const ChainThread& c, uint32_t tz, unsigned char* act, unsigned char* out) {
#pragma unroll 1
    for (int cc = c.c0; cc < c.c0 + kCols; cc += 16) {
        float z[16];
        umma::tmem_ld16(c.tl + tz + cc, z);
#pragma unroll
        for (int e = 0; e < 16; e++) z[e] *= sigm(z[e]);
        if (cc + 16 == H) z[15] = 1.f;
        st_tile16(act, c.q, cc, z);
        st_tile16(out, c.q, cc, z);
    }
}

// g = t SiLU'(z) to out (and to the operand tile, if any), t SiLU''(z) to E; SiLU'(z) replaces z.
__device__ __forceinline__ void chain_gradient(const ChainThread& c, uint32_t tz, unsigned char* act, unsigned char* out,
                                               unsigned char* E) {
#pragma unroll 1
    for (int cc = c.c0; cc < c.c0 + kCols; cc += 16) {
        float t[16], z[16], e2[16];
        umma::tmem_ld16x2(c.tl + T_T + cc, c.tl + tz + cc, t, z);
#pragma unroll
        for (int e = 0; e < 16; e++) {
            const float s = sigm(z[e]), d = dsilu(z[e], s);
            e2[e] = t[e] * d2silu(z[e], s);
            t[e] *= d;
            z[e] = d;
        }
        if (cc + 16 == H) e2[15] = t[15] = 0.f;
        umma::tmem_st16(c.tl + tz + cc, z);
        if (act != nullptr) st_tile16(act, c.q, cc, t);
        st_tile16(out, c.q, cc, t);
        st_tile16(E, c.q, cc, e2);
    }
    umma::tmem_wait_st();
}

// t = gb SiLU'(z) to the operand tile and to out; E := gb E.
__device__ __forceinline__ void chain_adjoint(const ChainThread& c, uint32_t td, unsigned char* act, unsigned char* out,
                                              unsigned char* E) {
#pragma unroll 1
    for (int cc = c.c0; cc < c.c0 + kCols; cc += 16) {
        float gb[16], d[16], e2[16];
        umma::tmem_ld16x2(c.tl + T_T + cc, c.tl + td + cc, gb, d);
        ld_tile16(E, c.q, cc, e2);
#pragma unroll
        for (int e = 0; e < 16; e++) {
            d[e] *= gb[e];
            e2[e] *= gb[e];
        }
        if (cc + 16 == H) d[15] = e2[15] = 0.f;
        st_tile16(act, c.q, cc, d);
        st_tile16(out, c.q, cc, d);
        st_tile16(E, c.q, cc, e2);
    }
}

// z = E + hb SiLU'(z) to out (and to the operand tile, if any).
__device__ __forceinline__ void chain_backward(const ChainThread& c, uint32_t td, unsigned char* act, unsigned char* out,
                                               const unsigned char* E) {
#pragma unroll 1
    for (int cc = c.c0; cc < c.c0 + kCols; cc += 16) {
        float hb[16], d[16], e2[16];
        umma::tmem_ld16x2(c.tl + T_T + cc, c.tl + td + cc, hb, d);
        ld_tile16(E, c.q, cc, e2);
#pragma unroll
        for (int e = 0; e < 16; e++) d[e] = e2[e] + hb[e] * d[e];
        if (cc + 16 == H) d[15] = 0.f;
        if (act != nullptr) st_tile16(act, c.q, cc, d);
        st_tile16(out, c.q, cc, d);
    }
}

__global__ void __launch_bounds__(kThreads, 1)
k_sg_chain(const uint16_t* __restrict__ img, const float* __restrict__ vec, const int* __restrict__ nrows,
           const uint16_t* __restrict__ X, const uint16_t* __restrict__ Ut, const float* __restrict__ beta,
           OperandTiles out, float* __restrict__ dw4_glob, int* __restrict__ err) {
    FMD_PDL_WAIT();
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tbase;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int R = *nrows;
    const int ntiles = (R + TILE - 1) / TILE;
    if ((int)blockIdx.x >= ntiles) return;
    {
        const uint4* src = reinterpret_cast<const uint4*>(img);
        uint4* dst = reinterpret_cast<uint4*>(sm + C_W1);
        for (int e = t; e < IMG_N * 2 / 16; e += kThreads) dst[e] = src[e];
        float* w4 = reinterpret_cast<float*>(sm + C_W4);
        float* dw4 = reinterpret_cast<float*>(sm + C_DW4);
        for (int e = t; e < H; e += kThreads) { w4[e] = vec[V_W4 + e]; dw4[e] = 0.f; }
    }
    if (w == 0) {
        umma::tmem_alloc(&tbase, 512);
        umma::tmem_relinquish();
    }
    if (t == 0) umma::mbar_init(&mbar, 1);
    to_mma();
    const uint32_t tm = tbase;
    const ChainThread c{tm + ((uint32_t)(32 * (w & 3)) << 16), 32 * (w & 3) + lane, kCols * (w >> 2)};
    const uint32_t sW1 = umma::smem_u32(sm + C_W1), sW2 = umma::smem_u32(sm + C_W2), sW3 = umma::smem_u32(sm + C_W3),
                   sX = umma::smem_u32(sm + C_X), sU = umma::smem_u32(sm + C_U), sA = umma::smem_u32(sm + C_ACT);
    unsigned char* act = sm + C_ACT;
    unsigned char* E1 = sm + C_E1;
    unsigned char* E2 = sm + C_E2;
    const float* w4 = reinterpret_cast<const float*>(sm + C_W4);
    const float bs = vec[V_BS];
    float* dw4 = reinterpret_cast<float*>(sm + C_DW4);
    float dw[kCols];                       // a stage's part of dL/dw4, this row
    uint32_t ph = 0;
    bool ok = true;

    // The next tile's operands, one 16-byte piece each per thread, wait in registers.
    static_assert(TILE * D * 2 / 16 == kThreads, "one 16-byte piece of an operand tile per thread");
    uint4 xnext = reinterpret_cast<const uint4*>(X + (size_t)blockIdx.x * TILE * D)[t];
    uint4 unext = reinterpret_cast<const uint4*>(Ut + (size_t)blockIdx.x * TILE * D)[t];
    float bnext = beta[(size_t)blockIdx.x * TILE + c.q];

    // Wait for the MMAs of this step, then (after the epilogue) hand the new
    // operand tile to the issuing thread; a wait that ran out ends every
    // thread at the next hand-off.
#define SG_WAIT()                                                     \
    do {                                                              \
        if (ok) {                                                     \
            ok = umma::mbar_wait(&mbar, ph);                          \
            if (ok) ph ^= 1u;                                         \
        }                                                             \
        umma::fence_after();                                          \
    } while (0)
#define SG_HANDOFF()                                                  \
    do {                                                              \
        if (!to_mma_and(ok)) { ok = false; goto done; }               \
    } while (0)

    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const float ybar = bnext * bs;
        reinterpret_cast<uint4*>(sm + C_X)[t] = xnext;
        reinterpret_cast<uint4*>(sm + C_U)[t] = unext;
        SG_HANDOFF();
        // ---- forward
        if (t == 0) issue(tm + T_Z1, sX, D, false, sW1, D, false, H, D / 16, &mbar);
        SG_WAIT();
        if (tile + (int)gridDim.x < ntiles) {
            const size_t next = (size_t)(tile + gridDim.x) * TILE;
            xnext = reinterpret_cast<const uint4*>(X + next * D)[t];
            unext = reinterpret_cast<const uint4*>(Ut + next * D)[t];
            bnext = beta[next + c.q];
        }
        chain_forward(c, T_Z1, act, gtile(out.h1, tile));
        SG_HANDOFF();
        if (t == 0) issue(tm + T_Z2, sA, H, false, sW2, H, false, H, H / 16, &mbar);
        SG_WAIT();
        chain_forward(c, T_Z2, act, gtile(out.h2, tile));
        SG_HANDOFF();
        if (t == 0) issue(tm + T_Z3, sA, H, false, sW3, H, false, H, H / 16, &mbar);
        SG_WAIT();
#pragma unroll
        for (int k = 0; k < kCols; k += 16) {   // g3 = bs w4 SiLU'(z3); dw4 += ybar h3
            const int cc = c.c0 + k;
            float z[16];
            umma::tmem_ld16(c.tl + T_Z3 + cc, z);
#pragma unroll
            for (int e = 0; e < 16; e++) {
                const bool last = e == 15 && cc + 16 == H;
                const float s = sigm(z[e]);
                dw[k + e] = ybar * (last ? 1.f : z[e] * s);
                z[e] = last ? 0.f : bs * w4[cc + e] * dsilu(z[e], s);
            }
            st_tile16(act, c.q, cc, z);
            st_tile16(gtile(out.g3, tile), c.q, cc, z);
        }
        add_columns(dw, dw4 + c.c0, lane);
        // ---- gradient network
        SG_HANDOFF();
        if (t == 0) issue(tm + T_T, sA, H, false, sW3, H, true, H, H / 16, &mbar);        // t2 = g3 W3^T
        SG_WAIT();
        chain_gradient(c, T_Z2, act, gtile(out.g2, tile), E2);
        SG_HANDOFF();
        if (t == 0) issue(tm + T_T, sA, H, false, sW2, H, true, H, H / 16, &mbar);        // t1 = g2 W2^T
        SG_WAIT();
        chain_gradient(c, T_Z1, nullptr, gtile(out.g1, tile), E1);
        // ---- adjoint of the gradient network
        SG_HANDOFF();
        if (t == 0) issue(tm + T_T, sU, D, false, sW1, D, false, H, D / 16, &mbar);        // gb1 = u W1
        SG_WAIT();
        chain_adjoint(c, T_Z1, act, gtile(out.tb1, tile), E1);
        SG_HANDOFF();
        if (t == 0) issue(tm + T_T, sA, H, false, sW2, H, false, H, H / 16, &mbar);       // gb2 = tb1 W2
        SG_WAIT();
        chain_adjoint(c, T_Z2, act, gtile(out.tb2, tile), E2);
        SG_HANDOFF();
        if (t == 0) issue(tm + T_T, sA, H, false, sW3, H, false, H, H / 16, &mbar);       // gb3 = tb2 W3
        SG_WAIT();
#pragma unroll
        for (int k = 0; k < kCols; k += 16) {   // dw4 += bs gb3 SiLU'(z3); zb3
            const int cc = c.c0 + k;
            float gb[16], z[16];
            umma::tmem_ld16x2(c.tl + T_T + cc, c.tl + T_Z3 + cc, gb, z);
#pragma unroll
            for (int e = 0; e < 16; e++) {
                const bool last = e == 15 && cc + 16 == H;
                const float s = sigm(z[e]), d = dsilu(z[e], s);
                dw[k + e] = last ? 0.f : bs * gb[e] * d;
                z[e] = last ? 0.f : gb[e] * bs * w4[cc + e] * d2silu(z[e], s) + ybar * w4[cc + e] * d;
            }
            st_tile16(act, c.q, cc, z);
            st_tile16(gtile(out.z3, tile), c.q, cc, z);
        }
        add_columns(dw, dw4 + c.c0, lane);
        // ---- adjoint of the forward network
        SG_HANDOFF();
        if (t == 0) issue(tm + T_T, sA, H, false, sW3, H, true, H, H / 16, &mbar);        // hb2 = zb3 W3^T
        SG_WAIT();
        chain_backward(c, T_Z2, act, gtile(out.z2, tile), E2);
        SG_HANDOFF();
        if (t == 0) issue(tm + T_T, sA, H, false, sW2, H, true, H, H / 16, &mbar);        // hb1 = zb2 W2^T
        SG_WAIT();
        chain_backward(c, T_Z1, nullptr, gtile(out.z1, tile), E1);
        umma::fence_before();
        // the next tile's first hand-off orders these TMEM reads before its MMAs
    }
done:
    if (!ok) {
        if (t == 0) atomicCAS(err + 2, 0, 1);
        // a thread whose own wait ran out gives the MMA in flight a bounded
        // chance to land before TMEM is released
        umma::mbar_wait(&mbar, ph);
    }
    umma::fence_before();
    __syncthreads();
    if (ok)
        for (int e = t; e < H; e += kThreads) atomicAdd(&dw4_glob[e], dw4[e]);
    if (w == 0) umma::tmem_dealloc(tm, 512);
#undef SG_WAIT
#undef SG_HANDOFF
}

// ------------------------------------------------------------- weight gradients
// Six products per tile of 128 rows, each over a pair of operand tiles as the
// chain wrote them (dW1^T = z1^T x + g1^T u, dW2^T = z2^T h1 + g2^T tb1,
// dW3^T = z3^T h2 + g3^T tb2), summed in TMEM over the CTA's tiles.  One
// thread copies the pairs into a ring of stages, one issues the MMAs as they
// arrive.  It is bound by the reading of the operand tiles (336 KB a tile).
// 90,000 rows: 58 us, 225 MB (34 us from memory); 160 us with loads by all
// threads, then MMAs, in turn.  From the last tile back, with the chain's newest
// still in L2, it takes 49 us, but the sums would be added in another order.
constexpr int kGThreads = 256, kGStages = 3;
constexpr int G_A = 0, G_B = TILE * H * 2, G_STAGE = 2 * TILE * H * 2, G_TOTAL = kGStages * G_STAGE;
constexpr uint32_t T_D1 = 0, T_D2 = 128, T_D3 = 256;

struct GradPair {
    const uint16_t *a, *b;                 // [tiles][128][128], [tiles][128][bcols]
    int bcols;
    uint32_t dcol;                         // TMEM column of the sum
};
__device__ __forceinline__ GradPair grad_pair(const OperandTiles& in, const uint16_t* X, const uint16_t* Ut, int p) {
    switch (p) {
        case 0: return {in.z1, X, D, T_D1};
        case 1: return {in.g1, Ut, D, T_D1};
        case 2: return {in.z2, in.h1, H, T_D2};
        case 3: return {in.g2, in.tb1, H, T_D2};
        case 4: return {in.z3, in.h2, H, T_D3};
        default: return {in.g3, in.tb2, H, T_D3};
    }
}

// Four floats at p += v.
__device__ __forceinline__ void red_add4(float* p, const float* v) {
    asm volatile("red.relaxed.gpu.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
                 "f"(v[3])
                 : "memory");
}

__global__ void __launch_bounds__(kGThreads, 1)
k_sg_wgrad(const int* __restrict__ nrows, const uint16_t* __restrict__ X, const uint16_t* __restrict__ Ut,
           OperandTiles in, float* __restrict__ grad, int* __restrict__ err) {
    FMD_PDL_WAIT();
    extern __shared__ __align__(1024) unsigned char sm[];
    __shared__ uint64_t full[kGStages], empty[kGStages], fin;
    __shared__ uint32_t tbase;
    __shared__ int bad;
    const int t = threadIdx.x, w = t >> 5, lane = t & 31;
    const int R = *nrows;
    const int ntiles = (R + TILE - 1) / TILE;
    if ((int)blockIdx.x >= ntiles) return;
    const int mine = (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1, steps = 6 * mine;
    if (w == 0) {
        umma::tmem_alloc(&tbase, 512);
        umma::tmem_relinquish();
    }
    if (t == 0) {
        for (int s = 0; s < kGStages; s++) { umma::mbar_init(&full[s], 1); umma::mbar_init(&empty[s], 1); }
        umma::mbar_init(&fin, 1);
        bad = 0;
    }
    to_mma();
    const uint32_t tm = tbase;
    if (t == 0) {                          // copies
        int it = 0;
        for (; it < steps; it++) {
            const int s = it % kGStages, tile = (int)blockIdx.x + it / 6 * (int)gridDim.x;
            if (it >= kGStages && !umma::mbar_wait(&empty[s], (uint32_t)(it / kGStages - 1) & 1u)) { bad = 1; break; }
            const GradPair p = grad_pair(in, X, Ut, it % 6);
            const uint32_t base = umma::smem_u32(sm) + s * G_STAGE, bb = TILE * p.bcols * 2;
            umma::mbar_expect(&full[s], TILE * H * 2 + bb);
            umma::bulk_load(base + G_A, p.a + (size_t)tile * TILE * H, TILE * H * 2, &full[s]);
            umma::bulk_load(base + G_B, p.b + (size_t)tile * TILE * p.bcols, bb, &full[s]);
        }
        // the copies in flight land before the block ends
        for (int k = max(0, it - kGStages); k < it; k++)
            umma::mbar_wait(&full[k % kGStages], (uint32_t)(k / kGStages) & 1u);
    } else if (t == 32) {                  // products
        for (int it = 0; it < steps; it++) {
            const int s = it % kGStages;
            if (!umma::mbar_wait(&full[s], (uint32_t)(it / kGStages) & 1u)) { bad = 1; break; }
            umma::fence_after();
            const GradPair p = grad_pair(in, X, Ut, it % 6);
            const uint32_t a = umma::smem_u32(sm) + s * G_STAGE + G_A, b = umma::smem_u32(sm) + s * G_STAGE + G_B;
            const uint32_t id = umma::idesc_bf16(128, p.bcols, true, true);
            const bool fresh = it < 6 && it % 2 == 0;
            for (int k = 0; k < TILE / 16; k++)
                umma::mma_bf16(tm + p.dcol, umma::desc_mn(a, H, k), umma::desc_mn(b, p.bcols, k), id, !(fresh && k == 0));
            umma::commit(&empty[s]);
        }
        umma::commit(&fin);
        if (!umma::mbar_wait(&fin, 0u)) bad = 1;
    }
    __syncwarp();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    if (bad == 0) {   // this CTA's sums -> global (row = output unit, columns = input unit)
        const uint32_t tl = tm + ((uint32_t)(32 * (w & 3)) << 16);
        const int row = 32 * (w & 3) + lane;
        if (w < 4) {
            for (int c = 0; c < D; c += 16) {
                float v[16];
                umma::tmem_ld16(tl + T_D1 + c, v);
                for (int e = 0; e < 16; e += 4) red_add4(&grad[row * D + c + e], v + e);
            }
        }
        const int half = 64 * (w >> 2);
        for (int l = 0; l < 2; l++) {
            float* G = grad + H * D + l * H * H;
            for (int c = half; c < half + 64; c += 16) {
                float v[16];
                umma::tmem_ld16(tl + (l == 0 ? T_D2 : T_D3) + c, v);
                for (int e = 0; e < 16; e += 4) red_add4(&G[row * H + c + e], v + e);
            }
        }
    } else if (t == 0) {
        atomicCAS(err + 3, 0, 1);
    }
    umma::fence_before();
    __syncthreads();
    if (w == 0) umma::tmem_dealloc(tm, 512);
}

// Gradient in the master layout (W[in][out]); only the network weights train.
__device__ __forceinline__ double grad_of(const float* g, int p) {
    if (p < OW2) {
        const int d = p / H, h = p % H;
        return g[h * D + d];
    }
    if (p < OW4) {
        const int l = p < OW3 ? 0 : 1;
        const int e = p - (l == 0 ? OW2 : OW3);
        const int k = e / H, o = e % H;
        return g[H * D + l * H * H + o * H + k];
    }
    return g[H * D + 2 * H * H + (p - OW4)];
}

__global__ void k_sg_adam(double* __restrict__ P, double* __restrict__ m, double* __restrict__ v,
                          const float* __restrict__ g, AdamArgs a) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < OM; p += gridDim.x * blockDim.x) {
        double gr = grad_of(g, p) * a.scale;
        if (a.clip > 0.0) gr = fmin(fmax(gr, -a.clip), a.clip);
        const double mm = a.b1 * m[p] + (1.0 - a.b1) * gr;
        const double vv = a.b2 * v[p] + (1.0 - a.b2) * gr * gr;
        m[p] = mm;
        v[p] = vv;
        P[p] -= a.lr * (mm / a.bc1) / (sqrt(vv / a.bc2) + a.eps);
    }
}

// mean over 3na of (F - Fref)^2 added to out[0] (block partials, then one block)
__global__ void __launch_bounds__(256)
k_sg_mse_part(const double* __restrict__ F, const double* __restrict__ Fref, int n3, double* __restrict__ part) {
    __shared__ double sm[32];
    double acc[1] = {0.0};
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n3; e += gridDim.x * blockDim.x) {
        const double d = F[e] - Fref[e];
        acc[0] += d * d;
    }
    block_sum_store<1>(acc, sm, part + blockIdx.x);
}
__global__ void __launch_bounds__(256)
k_sg_mse_final(const double* __restrict__ part, int nblk, int n3, double* __restrict__ out) {
    __shared__ double sm[32];
    double acc[1] = {0.0};
    for (int b = threadIdx.x; b < nblk; b += blockDim.x) acc[0] += part[b];
    double tot[1];
    block_sum_store<1>(acc, sm, tot);
    if (threadIdx.x == 0) out[0] += tot[0] / n3;
}

// Per-feature sums of the (raw) descriptors of rows [0, R): acc[2f] += x,
// acc[2f+1] += x^2.
__global__ void __launch_bounds__(256)
k_sg_xstats(const uint16_t* __restrict__ X, const int* __restrict__ nrows, double* __restrict__ acc) {
    __shared__ double sm[2 * D];
    for (int e = threadIdx.x; e < 2 * D; e += blockDim.x) sm[e] = 0.0;
    __syncthreads();
    const int R = *nrows;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < R; r += gridDim.x * blockDim.x) {
        const unsigned char* tile = reinterpret_cast<const unsigned char*>(X) + (size_t)(r / TILE) * TILE * D * 2;
        for (int f = 0; f < D; f++) {
            const uint16_t bits = *reinterpret_cast<const uint16_t*>(tile + umma::il_off(r % TILE, f, D));
            const double x = (double)__uint_as_float((uint32_t)bits << 16);
            atomicAdd(&sm[2 * f], x);
            atomicAdd(&sm[2 * f + 1], x * x);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 2 * D; e += blockDim.x) atomicAdd(&acc[e], sm[e]);
}

__global__ void k_sg_grad_out(const float* __restrict__ g, double scale, double* __restrict__ out) {
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < NPARAM; p += gridDim.x * blockDim.x)
        out[p] = p < OM ? grad_of(g, p) * scale : 0.0;
}

}  // namespace

cudaError_t train_alloc(TrainWork& tw, const Work& w) {
    if (tw.r_cap >= w.r_cap && tw.na_cap >= w.na_cap) return cudaSuccess;
    train_free(tw);
    cudaError_t e = cudaSuccess;
    auto A = [&](void** p, size_t bytes) {
        if (e == cudaSuccess) e = cudaMalloc(p, bytes);
    };
    const size_t tb = sizeof(uint16_t) * (size_t)w.r_cap * H;
    uint16_t** bufs[10] = {&tw.t.h1, &tw.t.h2, &tw.t.g1, &tw.t.g2, &tw.t.g3, &tw.t.tb1, &tw.t.tb2,
                           &tw.t.z1, &tw.t.z2, &tw.t.z3};
    for (auto b : bufs) A((void**)b, tb);
    A((void**)&tw.U, sizeof(uint16_t) * (size_t)w.r_cap * D);
    A((void**)&tw.beta, sizeof(float) * (size_t)w.r_cap);
    A((void**)&tw.lamF, sizeof(double) * 3 * (size_t)w.na_cap);
    A((void**)&tw.part, sizeof(double) * kRowBlocks);
    A((void**)&tw.sc, sizeof(double) * 32);
    if (e != cudaSuccess) {
        train_free(tw);
        return e;
    }
    tw.r_cap = w.r_cap;
    tw.na_cap = w.na_cap;
    return cudaSuccess;
}

void train_free(TrainWork& tw) {
    uint16_t* bufs[10] = {tw.t.h1, tw.t.h2, tw.t.g1, tw.t.g2, tw.t.g3, tw.t.tb1, tw.t.tb2, tw.t.z1, tw.t.z2, tw.t.z3};
    for (auto b : bufs) cudaFree(b);
    cudaFree(tw.U); cudaFree(tw.beta); cudaFree(tw.lamF); cudaFree(tw.part); cudaFree(tw.sc);
    tw = TrainWork{};
}

cudaError_t accumulate_grad(Work& w, TrainWork& tw, const uint16_t* img, const float* vec, const double* pos,
                            const double* hh, const int* cnt, const int* list, int cap, int na, const double* Fref,
                            const double* ref10, double wE, double wF, double wW, double* F, double* loss_acc,
                            float* grad, cudaStream_t st) {
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(k_sg_chain, cudaFuncAttributeMaxDynamicSharedMemorySize, C_TOTAL);
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k_sg_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, G_TOTAL);
        if (e != cudaSuccess) return e;
        attr = true;
    }
    cudaError_t e = cudaMemsetAsync(F, 0, sizeof(double) * 3 * (size_t)na, st);
    if (e == cudaSuccess) e = rebo_forces(w, img, vec, pos, hh, cnt, list, cap, na, F, w.part, st);
    if (e == cudaSuccess) e = reduce_partials(w.part, kRowBlocks, kNV, tw.sc, st);           // sc[0..9] = E, W
    if (e != cudaSuccess) return e;
    if ((e = launch_pdl(k_sg_lambda, dim3(kRowBlocks), dim3(256), 0, st, F, Fref, na, wF, tw.lamF,
                        tw.part)) != cudaSuccess)
        return e;
    e = reduce_partials(tw.part, kRowBlocks, 1, tw.sc + 10, st);                              // sc[10] = sum dF^2
    if (e != cudaSuccess) return e;
    if ((e = launch_pdl(k_sg_loss, dim3(1), dim3(32), 0, st, tw.sc, ref10, tw.sc + 10, na, wE, wF, wW, tw.sc + 12,
                        loss_acc)) != cudaSuccess)
        return e;   // sc[12..21] = lambdas
    if ((e = launch_pdl(k_sg_adjoint, dim3(kRowBlocks), dim3(128), 0, st, pos, hh, cnt, list, cap, na, w.aoff,
                        w.row_i, w.row_s, vec, tw.lamF, tw.sc + 12, w.r_cap, tw.beta, tw.U)) != cudaSuccess)
        return e;
    const int* nrows = w.aoff + w.na_used;
    if ((e = launch_pdl(k_sg_chain, dim3(kSMs), dim3(kThreads), C_TOTAL, st, img, vec, nrows, w.X, tw.U, tw.beta,
                        tw.t, grad + H * D + 2 * H * H, w.err)) != cudaSuccess)
        return e;
    if ((e = launch_pdl(k_sg_wgrad, dim3(kSMs), dim3(kGThreads), G_TOTAL, st, nrows, w.X, tw.U, tw.t, grad,
                        w.err)) != cudaSuccess)
        return e;
    return cudaGetLastError();
}

cudaError_t adam_step(double* P, double* m, double* v, const float* grad, const AdamArgs& a, uint16_t* img,
                      float* vec, cudaStream_t st) {
    k_sg_adam<<<64, 256, 0, st>>>(P, m, v, grad, a);
    return pack_params(P, img, vec, st);
}

cudaError_t force_mse(const double* F, const double* Fref, int na, double* part, double* out, cudaStream_t st) {
    k_sg_mse_part<<<kRowBlocks, 256, 0, st>>>(F, Fref, 3 * na, part);
    k_sg_mse_final<<<1, 256, 0, st>>>(part, kRowBlocks, 3 * na, out);
    return cudaGetLastError();
}

cudaError_t feature_sums(const Work& w, double* acc, cudaStream_t st) {
    k_sg_xstats<<<kSMs * 2, 256, 0, st>>>(w.X, w.aoff + w.na_used, acc);
    return cudaGetLastError();
}

cudaError_t grad_to_params(const float* grad, double scale, double* out, cudaStream_t st) {
    k_sg_grad_out<<<64, 256, 0, st>>>(grad, scale, out);
    return cudaGetLastError();
}

}  // namespace sg
}  // namespace fmd
