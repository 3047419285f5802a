// rigidpair.cu -- rigid-body site-site LJ of a device-resident system, each
// molecule pair evaluated once (LJ:271-400).
//
// The directed kernel (rigid.cu) evaluates every molecule pair from both
// sides because a molecule owns its sums.  Here one of the two owns the pair
// (rigid_owner(): alternating, so that every molecule owns half of its pairs) and
// leaves the other's force and torque in a record:
//   k_rigid_prep   warp per molecule: lab-frame sites, and its own pairs
//                  within rmcut with their image vectors, costliest first
//   k_rigid_pairs  warp per molecule and part of its pairs: site pairs of each
//   rigid_pair_sum warp per molecule: its parts plus the records of the pairs
//                  others own, in list order (deterministic, no atomics): at
//                  the step's second kick, or in k_rigid_sum
// Force evaluation, directed kernel -> this one (B200, C60, FP32 / FP64): 613
// -> 216 us / 996 -> 327 us at 4,000 molecules, 49 -> 27 / 70 -> 31 at 108.
// The site kernel is bound by FP32 (FP64) issue (59 % of the slots, the FMA
// pipe as busy), the light pairs' set-up and sums about half of it.  With d = m + r_b - r_a and
// the site force g parallel to d, the torques of a pair about the two centres
// differ by m x F (m the image vector), so the partner's torque costs nothing
// in the site loop.
//
// FP32 pairs: lengths in units of sigma (no factor on 1/r^2), sites rounded
// once from the pair's midpoint, where the sites that meet are, and the
// lane's two sites packed as f32x2, so that subtractions, products and FMAs
// take one instruction for both.  A pair outside the cutoff is masked, not branched
// around: in the nearest shell, where the work is, some lane is always inside.
//
// A list entry whose reverse is missing (a row cut at the list width) is
// evaluated one-sided by its row, energy and virial halved, as the directed
// kernel does with every entry.
#include <algorithm>
#include <cmath>

#include "geom.cuh"
#include "kernels.h"
#include "rigidpair.cuh"

namespace fmd {
namespace {

constexpr double kSig = 3.431, kEps = 2.635e-3;   // LJ:103
constexpr int kSites = 64;                         // sites per molecule of this path
constexpr int kPairWarps = 4;                      // warps per block of the pair kernel
// Blocks per SM asked of the compiler.  FP32: 6 (80 registers) took 216 us at
// 4,000 C60 (forces of one evaluation), 5 221, 4 243; FP64: 4 (128 registers)
// 327, with more of the loop unrolled and 3 blocks 341.
constexpr int kPairBlocks32 = 6, kPairBlocks64 = 4;

struct __align__(32) Vec {
    double x, y, z, pad;
};
static_assert(sizeof(Vec) == sizeof(double) * kRigidLabDoubles, "the sites of rigid.cu fit in");

// R(q) (LJ:155-159) with reference rounding.
__device__ __forceinline__ void rotation(const double* q, double* R) {
    const double w = q[0], x = q[1], y = q[2], z = q[3];
    R[0] = __dsub_rn(1.0, __dmul_rn(2.0, __dadd_rn(__dmul_rn(y, y), __dmul_rn(z, z))));
    R[1] = __dmul_rn(2.0, __dsub_rn(__dmul_rn(x, y), __dmul_rn(w, z)));
    R[2] = __dmul_rn(2.0, __dadd_rn(__dmul_rn(x, z), __dmul_rn(w, y)));
    R[3] = __dmul_rn(2.0, __dadd_rn(__dmul_rn(x, y), __dmul_rn(w, z)));
    R[4] = __dsub_rn(1.0, __dmul_rn(2.0, __dadd_rn(__dmul_rn(x, x), __dmul_rn(z, z))));
    R[5] = __dmul_rn(2.0, __dsub_rn(__dmul_rn(y, z), __dmul_rn(w, x)));
    R[6] = __dmul_rn(2.0, __dsub_rn(__dmul_rn(x, z), __dmul_rn(w, y)));
    R[7] = __dmul_rn(2.0, __dadd_rn(__dmul_rn(y, z), __dmul_rn(w, x)));
    R[8] = __dsub_rn(1.0, __dmul_rn(2.0, __dadd_rn(__dmul_rn(x, x), __dmul_rn(y, y))));
}

// A pair of molecule i's own: partner, image vector, list position (< 0: one-sided).
struct __align__(32) OwnPair {
    double mx, my, mz;
    int j, k;
};

// Position of i in the row of each of its partners, -1 where it is missing.
__global__ void __launch_bounds__(256)
k_rigid_back(const int* __restrict__ cnt, const int* __restrict__ list, int cap, int n, int* __restrict__ back) {
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (w >= n) return;
    for (int k = lane; k < cnt[w]; k += 32) {
        const int j = list[(size_t)w * cap + k];
        const int* row = list + (size_t)j * cap;
        int lo = 0, hi = cnt[j];
        while (lo < hi) {                                  // rows are ascending
            const int mid = (lo + hi) >> 1;
            if (row[mid] < w) lo = mid + 1; else hi = mid;
        }
        back[(size_t)w * cap + k] = lo < cnt[j] && row[lo] == w ? lo : -1;
    }
}

__global__ void __launch_bounds__(128)
k_rigid_prep(const double* __restrict__ pos, const double* __restrict__ qv, const double* __restrict__ body,
             const double* __restrict__ hh, const int* __restrict__ cnt, const int* __restrict__ list,
             const int* __restrict__ back, int cap, int n, int natom, double rmcut2, int chunks, Vec* __restrict__ lab,
             OwnPair* __restrict__ own, int* __restrict__ nown, double* __restrict__ rec) {
    __shared__ float s_cost[4][kRigidListMax];
    __shared__ OwnPair s_pair[4][kRigidListMax];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int i = blockIdx.x * 4 + w;
    if (i >= n) return;                                    // whole warps; no block barrier below
    double h[9], hi[9], R[9];
#pragma unroll
    for (int k = 0; k < 9; k++) { h[k] = hh[k]; hi[k] = hh[9 + k]; }
    rotation(qv + 4 * i, R);
    double r2 = 0.0;
    for (int a = lane; a < natom; a += 32) {
        const double bx = body[3 * a], by = body[3 * a + 1], bz = body[3 * a + 2];
        const double x = dot3_rn(R[0], R[1], R[2], bx, by, bz), y = dot3_rn(R[3], R[4], R[5], bx, by, bz),
                     z = dot3_rn(R[6], R[7], R[8], bx, by, bz);
        r2 = fmax(r2, x * x + y * y + z * z);
        lab[(size_t)i * natom + a] = Vec{x, y, z, 0.0};
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) r2 = fmax(r2, __shfl_xor_sync(kFull, r2, o));
    const float r = sqrtf((float)r2), S = (float)(3.0 * kSig) + r;
    const double pix = pos[3 * i], piy = pos[3 * i + 1], piz = pos[3 * i + 2];
    const int nn = cnt[i];
    int m = 0;
    for (int k0 = 0; k0 < nn; k0 += 32) {
        const int k = k0 + lane;
        bool mine = false;
        OwnPair q;
        float cost = 0.f;
        if (k < nn) {
            const size_t t = (size_t)i * cap + k;
            q.j = list[t];
            const bool lone = back[t] < 0;
            q.k = lone ? -1 - k : k;
            if (lone || rigid_owner(i, q.j) == i) {
                q.mx = __dsub_rn(pos[3 * q.j], pix);
                q.my = __dsub_rn(pos[3 * q.j + 1], piy);
                q.mz = __dsub_rn(pos[3 * q.j + 2], piz);
                mimg(q.mx, q.my, q.mz, hi, h);
                const double d2 = norm2_rn(q.mx, q.my, q.mz);
                mine = !(d2 > rmcut2);                     // LJ:320
                if (!mine) {                               // the partner sums this record
                    double* o = rec + t * chunks * 6;
                    for (int c = 0; c < 6 * chunks; c++) o[c] = 0.0;
                }
                // sites of a sphere of radius R at distance d within reach of
                // i's: (S^2 - (d - R)^2) / (4 d R) of them
                const float d = sqrtf((float)d2);
                const float f = d + r <= S ? 1.f : (d - r >= S ? 0.f : (S * S - (d - r) * (d - r)) / (4.f * d * r));
                cost = 0.1f + fminf(1.f, fmaxf(0.f, f));
            }
        }
        const unsigned b = __ballot_sync(kFull, mine);
        const int at = m + __popc(b & ((1u << lane) - 1u));
        if (mine) { s_cost[w][at] = cost; s_pair[w][at] = q; }
        m += __popc(b);
    }
    __syncwarp();
    for (int k = lane; k < m; k += 32) {                   // rank by cost, ties by list position
        const float c = s_cost[w][k];
        int rank = 0;
        for (int u = 0; u < m; u++) rank += s_cost[w][u] > c || (s_cost[w][u] == c && u < k);
        own[(size_t)i * cap + rank] = s_pair[w][k];
    }
    if (lane == 0) nown[i] = m;
}

// ---- packed FP32 pairs ------------------------------------------------------
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ double sum2(f2 v) {
    float a, b;
    unpack2(v, a, b);
    return (double)(a + b);
}
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// j's kept sites: FP64 from i's centre; FP32 from the pair's midpoint, each
// component twice, ready as a packed operand.
template <class P> struct SiteBuf;
template <> struct SiteBuf<double> {
    double x[kSites], y[kSites], z[kSites];
    __device__ __forceinline__ void put(int k, double a, double b, double c) { x[k] = a; y[k] = b; z[k] = c; }
};
template <> struct SiteBuf<float> {
    float4 xy[kSites];
    float2 z[kSites];
    __device__ __forceinline__ void put(int k, double a, double b, double c) {
        const float u = (float)a, v = (float)b, t = (float)c;
        xy[k] = make_float4(u, u, v, v);
        z[k] = make_float2(t, t);
    }
};

// Sums of one molecule pair over a lane's sites: the forces on its two sites
// of i (f), energy and virial (xx xy xz yy yz zz).  The pair loops return
// whether the lane has a pair inside the cutoff.
struct PairSum {
    double f[2][3], w[6], e;
};

// FP64: the reference's distances and cutoff test (LJ:330-336); pair terms in
// the factored form of ljpair.cuh without their constant factors.
__device__ __forceinline__ bool site_pairs(const SiteBuf<double>& b, int k0, int k1, const double (&r)[2][3], bool v0,
                                           bool v1, const double (&)[3], bool dense, PairSum& s) {
    constexpr double rc2 = (3.0 * kSig) * (3.0 * kSig), sig2 = kSig * kSig, s6c = sig2 * sig2 * sig2;
    constexpr double sr2 = (1.0 / 3.0) * (1.0 / 3.0), sr6 = sr2 * sr2 * sr2;
    double e = 0.0;
    int np = 0;
#pragma unroll 1
    for (int k = k0; k < k1; k++) {
        const double bx = b.x[k], by = b.y[k], bz = b.z[k];
        double dx[2], dy[2], dz[2], r2[2];
        bool in[2];
#pragma unroll
        for (int t = 0; t < 2; t++) {
            dx[t] = __dsub_rn(bx, r[t][0]); dy[t] = __dsub_rn(by, r[t][1]); dz[t] = __dsub_rn(bz, r[t][2]);
            r2[t] = norm2_rn(dx[t], dy[t], dz[t]);
            in[t] = (t ? v1 : v0) && r2[t] < rc2;
        }
        if (!dense && !__any_sync(kFull, in[0] || in[1])) continue;
        double gx = 0.0, gy = 0.0, gz = 0.0;
#pragma unroll
        for (int t = 0; t < 2; t++) {
            // r^2 < 1/4 by its high word
            const int rh = __double2hiint(r2[t]);
            const bool close = rh < 0x3fd00000;
            const double q = __hiloint2double(close ? 0x3fd00000 : rh, close ? 0 : __double2loint(r2[t]));
            double y;
            asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(q));
            y = __hiloint2double(in[t] ? __double2hiint(y) : 0, 0);
            const double e0 = fma(-q, y, 1.0), e1 = fma(e0, e0, e0), i2 = fma(y, e1, y), i6 = i2 * i2 * i2;
            const double fm = (i6 * i2) * fma(2.0 * s6c, i6, -1.0);
            e = fma(i6, fma(s6c, i6, -1.0), e);
            np += in[t];
            gx = fma(fm, dx[t], gx); gy = fma(fm, dy[t], gy); gz = fma(fm, dz[t], gz);
            s.f[t][0] = fma(-fm, dx[t], s.f[t][0]);
            s.f[t][1] = fma(-fm, dy[t], s.f[t][1]);
            s.f[t][2] = fma(-fm, dz[t], s.f[t][2]);
        }
        // virial: sum over the lane's sites of (b - a) (x) g = (b - a0) (x) sum g - (a1 - a0) (x) g1
        s.w[0] = fma(dx[0], gx, s.w[0]); s.w[1] = fma(dx[0], gy, s.w[1]); s.w[2] = fma(dx[0], gz, s.w[2]);
        s.w[3] = fma(dy[0], gy, s.w[3]); s.w[4] = fma(dy[0], gz, s.w[4]); s.w[5] = fma(dz[0], gz, s.w[5]);
    }
    {
        const double ux = r[1][0] - r[0][0], uy = r[1][1] - r[0][1], uz = r[1][2] - r[0][2];
        const double* f = s.f[1];                          // -sum g1
        s.w[0] = fma(ux, f[0], s.w[0]); s.w[1] = fma(ux, f[1], s.w[1]); s.w[2] = fma(ux, f[2], s.w[2]);
        s.w[3] = fma(uy, f[1], s.w[3]); s.w[4] = fma(uy, f[2], s.w[4]); s.w[5] = fma(uz, f[2], s.w[5]);
    }
    constexpr double c24 = 24.0 * kEps * s6c, c4 = 4.0 * kEps * s6c, vshift = 4.0 * kEps * (sr6 * sr6 - sr6);
#pragma unroll
    for (int c = 0; c < 3; c++) { s.f[0][c] *= c24; s.f[1][c] *= c24; }
#pragma unroll
    for (int c = 0; c < 6; c++) s.w[c] *= c24;
    s.e = c4 * e - vshift * np;
    return np > 0;
}

// FP32, lengths in sigma: r2 < 9, s6 = r^-6, force 24 eps / sigma^2 times
// s6 (2 s6 - 1) / r^2 d, energy 4 eps (s6^2 - s6) - shift.
__device__ __forceinline__ bool site_pairs(const SiteBuf<float>& b, int k0, int k1, const double (&r)[2][3], bool v0,
                                           bool v1, const double (&mid)[3], bool dense, PairSum& s) {
    // the lane's sites from the midpoint, negated; a lane without one stands far away
    f2 a[3];
#pragma unroll
    for (int c = 0; c < 3; c++)
        a[c] = pack2(v0 ? (float)(mid[c] - r[0][c] * (1.0 / kSig)) : 1e4f, v1 ? (float)(mid[c] - r[1][c] * (1.0 / kSig)) : 1e4f);
    const f2 ax = a[0], ay = a[1], az = a[2];
    const f2 one = pack2(1.f, 1.f), mone = pack2(-1.f, -1.f), two = pack2(2.f, 2.f);
    constexpr float close = (float)(0.25 / (kSig * kSig));
    f2 fx = 0, fy = 0, fz = 0, wxx = 0, wxy = 0, wxz = 0, wyy = 0, wyz = 0, wzz = 0, e2 = 0, e1 = 0;
    int np = 0;
#pragma unroll 4
    for (int k = k0; k < k1; k++) {
        const ulonglong2 xy = *reinterpret_cast<const ulonglong2*>(&b.xy[k]);
        const f2 dx = add2(xy.x, ax), dy = add2(xy.y, ay),
                 dz = add2(*reinterpret_cast<const f2*>(&b.z[k]), az);
        const f2 rr = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        float q0, q1;
        unpack2(rr, q0, q1);
        const bool i0 = q0 < 9.f, i1 = q1 < 9.f;
        if (!dense && !__any_sync(kFull, i0 || i1)) continue;
        q0 = fmaxf(q0, close); q1 = fmaxf(q1, close);
        // 1/r^2: the approximation and one Newton step
        const f2 y = pack2(rcp_approx(q0), rcp_approx(q1)), q = pack2(q0, q1);
        const f2 i2 = fma2(fma2(q, mul2(y, mone), one), y, y);
        f2 s6 = mul2(mul2(i2, i2), i2);
        unpack2(s6, q0, q1);
        s6 = pack2(i0 ? q0 : 0.f, i1 ? q1 : 0.f);
        np += i0;
        np += i1;
        const f2 t = fma2(two, s6, mone), fm = mul2(mul2(s6, i2), t);
        e2 = fma2(s6, t, e2);                              // sum (2 s6^2 - s6)
        e1 = add2(s6, e1);
        const f2 gx = mul2(fm, dx), gy = mul2(fm, dy), gz = mul2(fm, dz);
        fx = add2(fx, gx); fy = add2(fy, gy); fz = add2(fz, gz);
        wxx = fma2(dx, gx, wxx); wxy = fma2(dx, gy, wxy); wxz = fma2(dx, gz, wxz);
        wyy = fma2(dy, gy, wyy); wyz = fma2(dy, gz, wyz); wzz = fma2(dz, gz, wzz);
    }
    constexpr double sr2 = (1.0 / 3.0) * (1.0 / 3.0), sr6 = sr2 * sr2 * sr2;
    constexpr double cf = 24.0 * kEps / kSig, cw = 24.0 * kEps, vshift = 4.0 * kEps * (sr6 * sr6 - sr6);
    if (!__any_sync(kFull, np > 0)) return false;
    float u, v;
    unpack2(fx, u, v); s.f[0][0] = -cf * u; s.f[1][0] = -cf * v;
    unpack2(fy, u, v); s.f[0][1] = -cf * u; s.f[1][1] = -cf * v;
    unpack2(fz, u, v); s.f[0][2] = -cf * u; s.f[1][2] = -cf * v;
    s.w[0] = cw * sum2(wxx); s.w[1] = cw * sum2(wxy); s.w[2] = cw * sum2(wxz);
    s.w[3] = cw * sum2(wyy); s.w[4] = cw * sum2(wyz); s.w[5] = cw * sum2(wzz);
    s.e = 2.0 * kEps * sum2(fma2(mone, e1, e2)) - vshift * np;
    return np > 0;
}

// Warp (i, part): units part, then in snake order, of molecule i; a unit is a
// chunk of an own pair's site loop (chunks > 1 spreads the few heavy pairs of
// a small system over the GPU).
template <class P>
__global__ void __launch_bounds__(32 * kPairWarps, sizeof(P) == 4 ? kPairBlocks32 : kPairBlocks64)
k_rigid_pairs(const Vec* __restrict__ lab, const OwnPair* __restrict__ own, const int* __restrict__ nown, int cap,
              int n, int natom, int parts, int chunks, double* __restrict__ rec, double* __restrict__ out) {
    __shared__ SiteBuf<P> s_buf[kPairWarps];
    constexpr bool F32 = sizeof(P) == 4;
    constexpr double u = F32 ? 1.0 / kSig : 1.0;           // to the pair loop's lengths
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long task = (long long)blockIdx.x * kPairWarps + w;
    if (task >= (long long)n * parts) return;
    // costly parts of all molecules first
    const int part = (int)(task / n), i = (int)(task - (long long)part * n);
    const int units = nown[i] * chunks;
    SiteBuf<P>& buf = s_buf[w];
    const bool v0 = lane < natom, v1 = lane + 32 < natom;
    double r[2][3] = {{0.0, 0.0, 0.0}, {0.0, 0.0, 0.0}};
#pragma unroll
    for (int t = 0; t < 2; t++)
        if (t ? v1 : v0) {
            const Vec a = lab[(size_t)i * natom + lane + 32 * t];
            r[t][0] = a.x; r[t][1] = a.y; r[t][2] = a.z;
        }
    // Only j's sites within the cutoff + R of i's centre can meet one of i's
    // (R the largest site radius, one body for all molecules); the margin is
    // far above the rounding of either precision.
    double rad2 = fmax(r[0][0] * r[0][0] + r[0][1] * r[0][1] + r[0][2] * r[0][2],
                       r[1][0] * r[1][0] + r[1][1] * r[1][1] + r[1][2] * r[1][2]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rad2 = fmax(rad2, __shfl_xor_sync(kFull, rad2, o));
    const double reach = 3.0 * kSig + 1e-2, screen = reach + sqrt(rad2), screen2 = screen * screen;
    double ft[3] = {0.0, 0.0, 0.0};                        // lanes 0-15: force, 16-31: torque
    double we[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};    // virial, energy
    for (int round = 0; round * parts < units; round++) {
        const int unit = round * parts + ((round & 1) ? parts - 1 - part : part);
        if (unit >= units) continue;
        const int rank = unit / chunks, chunk = unit - rank * chunks;
        const OwnPair q = own[(size_t)i * cap + rank];
        const double mid[3] = {0.5 * u * q.mx, 0.5 * u * q.my, 0.5 * u * q.mz};
        __syncwarp();
        int nb = 0;
#pragma unroll
        for (int t = 0; t < 2; t++) {
            double x = 0.0, y = 0.0, z = 0.0;
            bool keep = false;
            if (t ? v1 : v0) {
                const Vec s = lab[(size_t)q.j * natom + lane + 32 * t];
                x = __dadd_rn(q.mx, s.x); y = __dadd_rn(q.my, s.y); z = __dadd_rn(q.mz, s.z);
                keep = x * x + y * y + z * z < screen2;
            }
            const unsigned bal = __ballot_sync(kFull, keep);
            if (keep) {
                const int at = nb + __popc(bal & ((1u << lane) - 1u));
                if (F32) buf.put(at, u * x - mid[0], u * y - mid[1], u * z - mid[2]);
                else buf.put(at, x, y, z);
            }
            nb += __popc(bal);
        }
        __syncwarp();
        double* o = rec + (((size_t)i * cap + (q.k < 0 ? 0 : q.k)) * chunks + chunk) * 6;
        if (nb == 0) {                                     // most pairs of the third shell reach nobody
            if (q.k >= 0 && lane < 6) o[lane] = 0.0;
            continue;
        }
        PairSum s;
#pragma unroll
        for (int c = 0; c < 3; c++) s.f[0][c] = s.f[1][c] = 0.0;
#pragma unroll
        for (int c = 0; c < 6; c++) s.w[c] = 0.0;
        s.e = 0.0;
        const bool dense = q.mx * q.mx + q.my * q.my + q.mz * q.mz < reach * reach;
        if (!__any_sync(kFull, site_pairs(buf, nb * chunk / chunks, nb * (chunk + 1) / chunks, r, v0, v1, mid, dense, s))) {
            if (q.k >= 0 && lane < 6) o[lane] = 0.0;
            continue;
        }
        // force and torque on i (LJ:337): T = sum r_a x f_a
        double F[3], T[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const int c1 = (c + 1) % 3, c2 = (c + 2) % 3;
            F[c] = s.f[0][c] + s.f[1][c];
            T[c] = r[0][c1] * s.f[0][c2] - r[0][c2] * s.f[0][c1] + (r[1][c1] * s.f[1][c2] - r[1][c2] * s.f[1][c1]);
        }
        const bool lone = q.k < 0;
        const double half = lone ? 0.5 : 1.0;              // LJ:339-341, both sides or one
#pragma unroll
        for (int c = 0; c < 6; c++) we[c] += half * s.w[c];
        we[6] += half * s.e;
        // lanes 0-15 sum F, lanes 16-31 T
        const bool upper = lane & 16;
#pragma unroll
        for (int c = 0; c < 3; c++) {
            const double send = upper ? F[c] : T[c];
            F[c] = (upper ? T[c] : F[c]) + __shfl_xor_sync(kFull, send, 16);
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < 3; c++) F[c] += __shfl_xor_sync(kFull, F[c], o);
#pragma unroll
        for (int c = 0; c < 3; c++) ft[c] += F[c];
        if (lone) continue;
        // the partner's force -F and torque m x F - T
        const double fx = __shfl_sync(kFull, F[0], 0), fy = __shfl_sync(kFull, F[1], 0), fz = __shfl_sync(kFull, F[2], 0);
        if (lane == 0) { o[0] = -fx; o[1] = -fy; o[2] = -fz; }
        if (lane == 16) {
            o[3] = (q.my * fz - q.mz * fy) - F[0];
            o[4] = (q.mz * fx - q.mx * fz) - F[1];
            o[5] = (q.mx * fy - q.my * fx) - F[2];
        }
    }
    double* o = out + ((size_t)i * parts + part) * kRigidRec;
    if ((lane & 15) == 0) {
#pragma unroll
        for (int c = 0; c < 3; c++) o[3 * (lane >> 4) + c] = ft[c];
    }
#pragma unroll
    for (int k = 0; k < 7; k++) {
        const double t = warp_sum(we[k]);
        if (lane == 0) o[6 + k] = t;
    }
}

constexpr int kSumWarps = 8;

__global__ void __launch_bounds__(32 * kSumWarps)
k_rigid_sum(RigidPair rp, const int* __restrict__ cnt, const int* __restrict__ list, int cap, int n,
            double* __restrict__ F, double* __restrict__ T, double* __restrict__ part) {
    __shared__ double sm[32 * kNV];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    double tot[kNV];
#pragma unroll
    for (int k = 0; k < kNV; k++) tot[k] = 0.0;
    for (int i = blockIdx.x * kSumWarps + w; i < n; i += gridDim.x * kSumWarps) {
        double v[6];
        rigid_pair_sum(rp, cnt, list, cap, i, lane, v, tot);
        if (lane == 0) {
            F[3 * i] = v[0]; F[3 * i + 1] = v[1]; F[3 * i + 2] = v[2];
            T[3 * i] = v[3]; T[3 * i + 1] = v[4]; T[3 * i + 2] = v[5];
        }
    }
    block_sum_fields<kNV>(tot, sm, part + (size_t)blockIdx.x * kNV);
}

// Warps per molecule: about one own pair each (21) at 108 molecules, four at
// 4,000 (313 us against 343 us with 21, whose set-up and sums come once per
// warp).  Splitting the site loops only pays where there are fewer nearest
// pairs than schedulers (32 molecules: 20.6 us against 22.7).
int pair_chunks(int n) { return n <= 64 ? 2 : 1; }
int pair_parts(int n) { return std::max(4, std::min(24, kSMs * 96 / n)); }

}  // namespace

bool rigid_pair_fits(int natom, int cap) { return natom <= kSites && cap <= kRigidListMax; }

size_t rigid_pair_bytes(int n, int natom, int cap) {
    return sizeof(Vec) * (size_t)n * natom + sizeof(OwnPair) * (size_t)n * cap +
           sizeof(double) * (6 * (size_t)n * cap * pair_chunks(n) + (size_t)n * pair_parts(n) * kRigidRec) +
           sizeof(int) * ((size_t)n * cap + n);
}

RigidPair rigid_pair_layout(void* mem, int n, int natom, int cap) {
    RigidPair r;
    r.parts = pair_parts(n);
    r.chunks = pair_chunks(n);
    char* p = static_cast<char*>(mem);
    r.own = p; p += sizeof(OwnPair) * (size_t)n * cap;
    r.lab = p; p += sizeof(Vec) * (size_t)n * natom;
    r.rec = reinterpret_cast<double*>(p); p += sizeof(double) * 6 * (size_t)n * cap * r.chunks;
    r.out = reinterpret_cast<double*>(p); p += sizeof(double) * (size_t)n * r.parts * kRigidRec;
    r.back = reinterpret_cast<int*>(p); p += sizeof(int) * (size_t)n * cap;
    r.nown = reinterpret_cast<int*>(p);
    r.on = 1;
    return r;
}

int rigid_pair_records(int n) { return std::max(1, std::min(2 * kSMs, (n + kSumWarps - 1) / kSumWarps)); }

cudaError_t rigid_pair_lists(const RigidPair& r, const int* cnt, const int* list, int cap, int n, cudaStream_t st) {
    k_rigid_back<<<(n * 32 + 255) / 256, 256, 0, st>>>(cnt, list, cap, n, r.back);
    return cudaGetLastError();
}

cudaError_t rigid_pair_launch(const RigidPair& r, int precision, const double* pos, const double* qv,
                              const double* body, const double* hh, const int* cnt, const int* list, int cap, int n,
                              int natom, double rmcut2, cudaStream_t st) {
    OwnPair* own = static_cast<OwnPair*>(r.own);
    Vec* lab = static_cast<Vec*>(r.lab);
    const int blocks = (int)(((long long)n * r.parts + kPairWarps - 1) / kPairWarps);
    k_rigid_prep<<<(n + 3) / 4, 128, 0, st>>>(pos, qv, body, hh, cnt, list, r.back, cap, n, natom, rmcut2, r.chunks,
                                              lab, own, r.nown, r.rec);
    if (precision == FMD_PREC_FP32_PAIR)
        k_rigid_pairs<float><<<blocks, 32 * kPairWarps, 0, st>>>(lab, own, r.nown, cap, n, natom, r.parts, r.chunks,
                                                                 r.rec, r.out);
    else
        k_rigid_pairs<double><<<blocks, 32 * kPairWarps, 0, st>>>(lab, own, r.nown, cap, n, natom, r.parts, r.chunks,
                                                                  r.rec, r.out);
    return cudaGetLastError();
}

cudaError_t rigid_pair_reduce(const RigidPair& r, const int* cnt, const int* list, int cap, int n, double* F,
                              double* T, double* part, cudaStream_t st) {
    k_rigid_sum<<<rigid_pair_records(n), 32 * kSumWarps, 0, st>>>(r, cnt, list, cap, n, F, T, part);
    return cudaGetLastError();
}

}  // namespace fmd
