// wcns_dev.cuh -- device data model and arithmetic shared by all WCNS kernels.
//
// Every per-point field lives in the reference's ghosted index space
// (-2:n+3 in each direction, i fastest) so that index arithmetic is the same
// for prim (which has real ghosts) and interior-only fields.  All blocks of a
// field are concatenated in one allocation; DevBlock::off is the block base.
//
// Arithmetic restates the reference operation by operation.  The library is
// compiled with -fmad=false so that no multiply-add is fused: with IEEE
// division and square root (the CUDA defaults for double) each expression
// then rounds exactly as gfortran -O2 does on x86-64.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace wcns {

constexpr double SMALL = 1.0e-38;     // Globalvar.f90:215
constexpr double SML_SSS = 1.0e-30;   // Globalvar.f90:218
constexpr double PMIN_LIMIT = 1.0e-8; // Globalvar.f90:223
constexpr double PMAX_LIMIT = 1.0e+3;
constexpr double RMIN_LIMIT = 1.0e-8;
constexpr double RMAX_LIMIT = 1.0e+3;
constexpr double TMIN_LIMIT = 1.0e-8;
constexpr int NIJK2D = 4;   // Main.f90:20
constexpr int NIJK2ND = 4;  // Main.f90:21

enum Field : int {
    F_R = 0, F_U, F_V, F_W, F_P, F_T,
    F_DQ1, F_DQ2, F_DQ3, F_DQ4, F_DQ5,
    F_DTDT, F_SRA, F_SRB, F_SRC, F_SRVA, F_SRVB, F_SRVC,
    F_KCX, F_KCY, F_KCZ, F_ETX, F_ETY, F_ETZ, F_CTX, F_CTY, F_CTZ, F_VOL,
    F_C, F_VISL, F_Q1, F_Q2, F_Q3, F_Q4, F_Q5,
    F_NPUBLIC,
    // internal work arrays
    F_RHS1 = F_NPUBLIC, F_RHS2, F_RHS3, F_RHS4, F_RHS5,
    F_COED,
    F_OLD1, F_OLD2, F_OLD3, F_OLD4, F_OLD5,
    F_DUV0,  // 12 node derivatives of (u,v,w,T): F_DUV0 .. F_DUV0+11
    F_MU = F_DUV0 + 12,  // viscosity and heat conductivity at the interior points, for the viscous residual
    F_NPOOL = F_MU + 2,  // fields of the pool
    // the SA model's eddy viscosity (its own allocation; null while the
    // model is not set up, which the kernels read as vist = 0)
    F_VIST = F_NPOOL,
    F_NALL
};

struct DevParams {
    double gama, g1;  // g1 = gama/(gama-1)
    double moo, moo2, moocp;
    double reynolds, re, visc;
    double cp_prl, cp_prt, cc23;
    double cfl, timedt_rate, efix, csrv;
    double roo, uoo, voo, woo, poo, coo;
    double twall_nd;
    int nvis, nscheme, nflux, adiabatic;
};

struct DevBlock {
    int ni, nj, nk;
    int gx, gy, gz;
    long long off;   // base offset of this block in every field
    long long npts;  // ni*nj*nk
    long long pmoff; // base offset in the plane-major sweep arrays
    // the free stream's Mach-dependent constants of init_inflow
    // (PreProcess.f90:968-1113) for this block: the context's by default,
    // a case's own when independent cases of different Mach numbers share
    // one context (wcns_set_block_freestream)
    double moo2, moocp, poo, coo, cp_prl, cp_prt;
};

// Plane-major layout for the LU-SGS sweeps.  Cell (i,j,k) of a block lives
// in plane p = i+j+k at column slot c(j,k); the cells of one hyperplane are
// contiguous.  Columns are grouped in j-chunks, one chunk per CTA of the
// block's sweep cluster: chunk q covers j-1 in [q*nj/C, (q+1)*nj/C) for all
// k, and slot = j0(q)*nk + (k-1)*width(q) + (j-1-j0(q)).
__host__ __device__ inline int chunk_j0(int q, int nj, int C) { return q * nj / C; }  // q <= C <= 16: no overflow
__host__ __device__ inline int chunk_of(int jj, int nj, int C) {  // jj = j-1
    int q = (int)(((long long)jj * C) / nj);
    if (q > C - 1) q = C - 1;
    while (q > 0 && chunk_j0(q, nj, C) > jj) q--;
    while (q < C - 1 && chunk_j0(q + 1, nj, C) <= jj) q++;
    return q;
}
__host__ __device__ inline int col_slot(int j, int k, int nj, int nk, int C) {
    int jj = j - 1, q = chunk_of(jj, nj, C);
    int j0 = chunk_j0(q, nj, C), w = chunk_j0(q + 1, nj, C) - j0;
    return j0 * nk + (k - 1) * w + (jj - j0);
}

// static per-cell record of the sweeps (written once per step by k_lhs_prep)
enum StatRec : int {
    SR_COED = 0, SR_RHS = 1,              // coed, rhs(5)
    SR_U = 6,                             // u, v, w, H
    SR_G = 10,                            // the nine metrics, direction by direction
    SR_RAD = 19,                          // inviscid radii
    SR_RADS = 22,                         // inviscid plus viscous radii
    SR_N = 26                             // record length (16-byte multiple)
};
constexpr int DYN_N = 16;                 // dynamic per-cell record: dq of lusgs_l, or old-side terms 5*d + m

struct PmFields {
    double *dq[5];   // SoA dq in plane-major order (result of gs_pr_u, the last sweep)
    long long dq_stride;  // dq[m] = dq[0] + m * dq_stride
    double *stat;    // [cell][SR_N]
    double *dyn;     // [cell][DYN_N] dq of lusgs_l, read by lusgs_u
    double *gs[2];   // [cell][DYN_N] old-side terms along i, j, k: written by lusgs_u for gs_pr_l (gs[0])
                     // and by gs_pr_l for gs_pr_u (gs[1]); zero where the neighbour is outside the block
    int csize;       // CTAs per block cluster (defines the column slots)
};

__host__ __device__ inline long long pmidx(const DevBlock &b, int p, int slot) {
    return b.pmoff + (long long)(p - 3) * ((long long)b.nj * b.nk) + slot;
}

struct DevFields {
    double *f[F_NALL];
};

__host__ __device__ inline long long gidx(const DevBlock &b, int i, int j, int k) {
    return b.off + (long long)(i + 2) + (long long)b.gx * ((long long)(j + 2) + (long long)b.gy * (long long)(k + 2));
}

// Division by a divisor that is the same for the whole kernel: one high
// multiply instead of a division sequence.  Exact for 0 <= n, d and
// n * d < 2^32 (m = ceil(2^32 / d); the error n * (m - 2^32/d) / 2^32 < n / 2^32
// stays below 1/d).
struct FastDiv {
    unsigned d, m;
};
__host__ __device__ inline FastDiv fast_div_init(int d) {
    FastDiv f;
    f.d = (unsigned)d;
    f.m = d <= 1 ? 0u : 0xFFFFFFFFu / (unsigned)d + 1u;
    return f;
}
__device__ __forceinline__ int fdiv(int n, FastDiv f) { return f.d <= 1 ? n : (int)__umulhi((unsigned)n, f.m); }

// interior point index p = (i-1) + ni*((j-1) + nj*(k-1)) -> (i, j, k); 32-bit
// divisions whenever p fits (every realistic block)
__device__ __forceinline__ void decode_point(const DevBlock &B, long long p, int &i, int &j, int &k) {
    if (p < 0x7fffffffLL) {
        const int q = (int)p, r = q / B.ni;
        i = q - r * B.ni + 1;
        j = r % B.nj + 1;
        k = r / B.nj + 1;
    } else {
        i = (int)(p % B.ni) + 1;
        j = (int)((p / B.ni) % B.nj) + 1;
        k = (int)(p / ((long long)B.ni * B.nj)) + 1;
    }
}

__host__ __device__ inline int dimof(const DevBlock &b, int d) { return d == 0 ? b.ni : (d == 1 ? b.nj : b.nk); }

// stride (in elements) along direction d
__host__ __device__ inline long long dstride(const DevBlock &b, int d) {
    return d == 0 ? 1LL : (d == 1 ? (long long)b.gx : (long long)b.gx * b.gy);
}

// ---------------------------------------------------------------------------
// Line operators evaluated at one position.  `Acc` maps a 1-based point index
// to a value.
// ---------------------------------------------------------------------------

// VALUE_HALF_NODE (WCNSE5.f90:799-852) at half node h in 0..n
template <class Acc>
__device__ __forceinline__ double value_half_node_at(const Acc &q, int n, int h) {
    if (n <= NIJK2ND) {
        if (h == 0) {
            int i2 = n < 2 ? n : 2, i3 = n < 3 ? n : 3;
            return (15.0 * q(1) - 10.0 * q(i2) + 3.0 * q(i3)) / 8.0;
        }
        if (h == n) {
            int j1 = n - 1 > 1 ? n - 1 : 1, j2 = n - 2 > 1 ? n - 2 : 1;
            return (15.0 * q(n) - 10.0 * q(j1) + 3.0 * q(j2)) / 8.0;
        }
        return 0.5 * (q(h) + q(h + 1));
    }
    if (h == 0) return (35.0 * q(1) - 35.0 * q(2) + 21.0 * q(3) - 5.0 * q(4)) / 16.0;
    if (h == n) return (35.0 * q(n) - 35.0 * q(n - 1) + 21.0 * q(n - 2) - 5.0 * q(n - 3)) / 16.0;
    if (h == 1) return (5.0 * q(1) + 15.0 * q(2) + -5.0 * q(3) + 1.0 * q(4)) / 16.0;
    if (h == n - 1) return (5.0 * q(n) + 15.0 * q(n - 1) + -5.0 * q(n - 2) + 1.0 * q(n - 3)) / 16.0;
    return (9.0 * (q(h) + q(h + 1)) + -1.0 * (q(h + 2) + q(h - 1))) / 16.0;
}

// VALUE_HALF_NODE_IJK (newvis.f90:421-554) for one component at half node h
template <class Acc>
__device__ __forceinline__ double value_half_node_ijk_at(const Acc &q, int n, int h) {
    if (n <= NIJK2ND) {
        if (h == 0) return 1.5 * q(1) - 0.5 * q(n < 2 ? n : 2);
        if (h == n) return 1.5 * q(n) - 0.5 * q(n - 1 > 1 ? n - 1 : 1);
        return 0.5 * (q(h) + q(h + 1));
    }
    if (h == 0) return (35.0 * q(1) - 35.0 * q(2) + 21.0 * q(3) - 5.0 * q(4)) / 16.0;
    if (h == n) return (35.0 * q(n) - 35.0 * q(n - 1) + 21.0 * q(n - 2) - 5.0 * q(n - 3)) / 16.0;
    if (h == 1) return (5.0 * q(1) + 15.0 * q(2) + -5.0 * q(3) + 1.0 * q(4)) / 16.0;
    if (h == n - 1) return (5.0 * q(n) + 15.0 * q(n - 1) + -5.0 * q(n - 2) + 1.0 * q(n - 3)) / 16.0;
    return (9.0 * (q(h) + q(h + 1)) + -1.0 * (q(h + 2) + q(h - 1))) / 16.0;
}

// FLUX_DXYZ (WCNSE5.f90:209-254) at point l in 1..n; f(h) for h in 0..n
template <class Acc>
__device__ __forceinline__ double flux_dxyz_at(const Acc &f, int n, int l) {
    if (n <= NIJK2ND) return f(l) - f(l - 1);
    if (l == 1) return (-23.0 * f(0) + 21.0 * f(1) + 3.0 * f(2) - f(3)) / 24.0;
    if (l == n) return -(-23.0 * f(n) + 21.0 * f(n - 1) + 3.0 * f(n - 2) - f(n - 3)) / 24.0;
    if (l == 2) return (f(0) - 27.0 * f(1) + 27.0 * f(2) - f(3)) / 24.0;
    if (l == n - 1) return -(f(n) - 27.0 * f(n - 1) + 27.0 * f(n - 2) - f(n - 3)) / 24.0;
    return (2250.0 * (f(l) - f(l - 1)) - 125.0 * (f(l + 1) - f(l - 2)) + 9.0 * (f(l + 2) - f(l - 3))) / 1920.0;
}

// ---------------------------------------------------------------------------
// Numerical fluxes
// ---------------------------------------------------------------------------

// flux_SW_pn (flux.f90:17-77); gethmgm_ns (GasModel.f90:385-399)
__device__ __forceinline__ void flux_sw_pn(const DevParams &P, const double *prim, double nx, double ny, double nz,
                                           double nt, double *f, int npn) {
    const double gama = P.gama;
    double rm = prim[0], um = prim[1], vm = prim[2], wm = prim[3], pm = prim[4];
    double u2 = 0.5 * (um * um + vm * vm + wm * wm);
    double hint = P.g1 * pm / rm;
    double eint = hint - pm / rm;
    double em = eint + u2;
    double cm = sqrt(gama * pm / rm);
    double ct = nx * um + ny * vm + nz * wm + nt;
    double cgm = sqrt(nx * nx + ny * ny + nz * nz);
    cgm = fmax(cgm, SML_SSS);
    double l1 = ct, l4 = ct + cm * cgm, l5 = ct - cm * cgm;
    double eps = P.efix * P.efix * cgm * cgm;
    double dn = (double)npn;
    l1 = 0.5 * (l1 + dn * sqrt(l1 * l1 + eps));
    l4 = 0.5 * (l4 + dn * sqrt(l4 * l4 + eps));
    l5 = 0.5 * (l5 + dn * sqrt(l5 * l5 + eps));
    double cgm1 = 1.0 / cgm;
    double nxa = nx * cgm1, nya = ny * cgm1, nza = nz * cgm1;
    double cta = (ct - nt) * cgm1;
    double c2r = cm * cm / gama;
    double x1 = c2r * (2.0 * l1 - l4 - l5) / (2.0 * cm * cm);
    double x2 = c2r * (l4 - l5) / (2.0 * cm);
    double hm = em + pm / rm;
    f[0] = (l1 - x1) * rm;
    f[1] = (l1 * um - x1 * um + nxa * x2) * rm;
    f[2] = (l1 * vm - x1 * vm + nya * x2) * rm;
    f[3] = (l1 * wm - x1 * wm + nza * x2) * rm;
    f[4] = (l1 * em - x1 * hm + cta * x2) * rm;
}

// flux_vanleer_pn (flux.f90:410-501), gethmgm -> gethmgm_ns
// (GasModel.f90:376-399).  Returns 1 when c^2 < 0 (the reference stops).
// (b +- 1)**2 is a product, as gfortran evaluates an integer exponent 2.
__device__ __forceinline__ int flux_vl_pn(const DevParams &P, const double *prim, double nx, double ny, double nz,
                                          double nt, double *f, int npn) {
    const double gama = P.gama;
    double rm = prim[0], um = prim[1], vm = prim[2], wm = prim[3], pm = prim[4];
    double u2 = 0.5 * (um * um + vm * vm + wm * wm);
    double hint = P.g1 * pm / rm;
    double hm = hint + u2;
    double c2 = gama * pm / rm;
    const int bad = c2 < 0.0 ? 1 : 0;
    double cm = sqrt(c2);
    double ct = nx * um + ny * vm + nz * wm + nt;
    double cgm = sqrt(nx * nx + ny * ny + nz * nz) + SML_SSS;
    double cgm1 = 1.0 / cgm;
    double nxa = nx * cgm1, nya = ny * cgm1, nza = nz * cgm1;
    double cta = ct * cgm1;
    double bmvl = cta / cm;
#pragma unroll
    for (int m = 0; m < 5; m++) f[m] = 0.0;
    if (fabs(bmvl) < 1.0) {
        double ctcm, b;
        if (npn == 1) {
            ctcm = (-cta + 2.0 * cm) / gama;
            b = (bmvl + 1.0) * (bmvl + 1.0);
            f[0] = 0.25 * cgm * rm * cm * b;
        } else {
            ctcm = (-cta - 2.0 * cm) / gama;
            b = (bmvl - 1.0) * (bmvl - 1.0);
            f[0] = -(0.25 * cgm * rm * cm * b);
        }
        f[1] = f[0] * (um + nxa * ctcm);
        f[2] = f[0] * (vm + nya * ctcm);
        f[3] = f[0] * (wm + nza * ctcm);
        f[4] = f[0] * hm;
    } else if (npn == 1 ? bmvl >= 1.0 : bmvl <= -1.0) {
        double rmct = rm * cta;
        f[0] = cgm * rmct;
        f[1] = cgm * (rmct * um + pm * nxa);
        f[2] = cgm * (rmct * vm + pm * nya);
        f[3] = cgm * (rmct * wm + pm * nza);
        f[4] = cgm * rmct * hm;
    }
    return bad;
}

// a / b from r = 1 / b: the quotient of the two rounded values corrected by
// its remainder (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990): the rounded quotient for every sample of
// tests/test_device_arithmetic.py.  For b and 1 / b normal and a far from the subnormal
// numbers; where a, b or r is zero or infinite the correction is NaN and the first
// quotient is what a division gives (-0 / b gives +0).  A division costs a dozen
// instructions and a branch, this six; without the last step the residual phases take
// 1.3 % less (channel: viscous 1345 for 1364 us, inviscid 1136 for 1148) and turn an
// infinite derivative into an undefined one.
__device__ __forceinline__ double div_by(double a, double b, double r) {
    const double q = a * r, c = fma(fma(-q, b, a), r, q);
    return c == c ? c : q;
}

// 1 / b and 1 / sqrt(x) of normal numbers from the hardware's approximation
// (relative error below 2^-19.9) by one step of the iteration of third order
// (Householder), to 0.51 and 1.02 ulp: where the last bit does not matter.  Zero, an
// infinity or a subnormal number gives NaN or an infinity, where 1 / b may give zero.
__device__ __forceinline__ double recip(double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    const double e = fma(-b, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double recip_sqrt(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y, e * fma(e, 0.375, 0.5), y);
}

// flux_Roe (flux.f90:116-244) with its operations in their order, for the half nodes
// that flux_roe leaves.  l, r: the left and the right state.  Returns 1 when c^2 <= 0.
__device__ __forceinline__ int flux_roe_div(double gama, double efix, double nx, double ny, double nz, const double *l, const double *r, double *f) {
    const double gama1 = gama - 1.0, gama2 = gama / gama1, nt = 0.0;
    double dq[5], fs[5], h[2];
#pragma unroll
    for (int s = 0; s < 2; s++) {  // flux (Convect.f90:1245-1272) with getem (GasModel.f90:358-374), of the right state first
        const double *p = s ? l : r;
        const double v2 = p[1] * p[1] + p[2] * p[2] + p[3] * p[3], em = p[4] / gama1 + 0.5 * p[0] * v2;
        const double cit = nx * p[1] + ny * p[2] + nz * p[3] + nt, ms = p[0] * cit;
        const double g[5] = {ms, ms * p[1] + nx * p[4], ms * p[2] + ny * p[4], ms * p[3] + nz * p[4], (em + p[4]) * cit - p[4] * nt};
#pragma unroll
        for (int m = 0; m < 5; m++) fs[m] = s ? fs[m] + g[m] : g[m];
        h[s] = gama2 * p[4] / p[0] + 0.5 * v2;
    }
#pragma unroll
    for (int m = 0; m < 5; m++) dq[m] = r[m] - l[m];
    const double rm = sqrt(l[0] * r[0]), rrl = sqrt(r[0] / l[0]), w = rrl + 1.0;
    const double um = (l[1] + r[1] * rrl) / w, vm = (l[2] + r[2] * rrl) / w, wm = (l[3] + r[3] * rrl) / w, hm = (h[1] + h[0] * rrl) / w;
    const double c2 = (hm - 0.5 * (um * um + vm * vm + wm * wm)) * gama1, c = sqrt(c2);
    const double cta = um * nx + vm * ny + wm * nz + nt;
    const double cgm = fmax(sqrt(nx * nx + ny * ny + nz * nz), SML_SSS), cgm1 = 1.0 / cgm;
    nx = nx * cgm1;
    ny = ny * cgm1;
    nz = nz * cgm1;
    const double ccgm = c * cgm, det = efix * cgm, det2 = det * det;
    auto root = [det2](double x) { return sqrt(x * x + det2); };
    const double l1 = root(fabs(cta - ccgm)), l4 = root(fabs(cta)), l5 = root(fabs(cta + ccgm));
    const double rodcta = rm * (dq[1] * nx + dq[2] * ny + dq[3] * nz), cta1 = cta * cgm1;
    const double dp_c2 = dq[4] / c2, rodctac = rodcta / c;
    const double a1 = l4 * (dq[0] - dp_c2), a2 = l5 * (dp_c2 + rodctac) * 0.5, a3 = l1 * (dp_c2 - rodctac) * 0.5;
    const double a4 = a1 + a2 + a3, a5 = c * (a2 - a3);
    const double a6 = l4 * (rm * dq[1] - nx * rodcta), a7 = l4 * (rm * dq[2] - ny * rodcta), a8 = l4 * (rm * dq[3] - nz * rodcta);
    f[0] = 0.5 * (fs[0] - a4);
    f[1] = 0.5 * (fs[1] - (um * a4 + nx * a5 + a6));
    f[2] = 0.5 * (fs[2] - (vm * a4 + ny * a5 + a7));
    f[3] = 0.5 * (fs[3] - (wm * a4 + nz * a5 + a8));
    f[4] = 0.5 * (fs[4] - (hm * a4 + cta1 * a5 + um * a6 + vm * a7 + wm * a8 - c2 * a1 / gama1));
    return c2 <= 0.0 ? 1 : 0;
}

// flux_Roe for the FP64 residual: the central part with the operations of the reference
// and in their order; what the jump multiplies with short reciprocals and roots, and
// sqrt(rl rr) as rl sqrt(rr / rl).
// gama1_1 = 1 / (gama - 1); same: ql equals qr, which leaves the central part.
// Returns false, and no flux, where it is not finite or c^2 is not well above the
// round-off of the enthalpy that it is the rest of: flux_roe_div.
__device__ __forceinline__ bool flux_roe(const DevParams &P, double gama1_1, const double *ql, const double *qr, double nx,
                                             double ny, double nz, double nt, bool same, double *f) {
    const double gama = P.gama, gama1 = gama - 1.0, gama2 = gama / gama1;
    const double v2l = ql[1] * ql[1] + ql[2] * ql[2] + ql[3] * ql[3], v2r = qr[1] * qr[1] + qr[2] * qr[2] + qr[3] * qr[3];
    double s[5];  // fr + fl
    {
        // flux (Convect.f90:1245-1272) with getem (GasModel.f90:358-374)
        const double el = div_by(ql[4], gama1, gama1_1) + 0.5 * ql[0] * v2l, er = div_by(qr[4], gama1, gama1_1) + 0.5 * qr[0] * v2r;
        const double cl = nx * ql[1] + ny * ql[2] + nz * ql[3] + nt, cr = nx * qr[1] + ny * qr[2] + nz * qr[3] + nt;
        const double ml = ql[0] * cl, mr = qr[0] * cr;
        s[0] = mr + ml;
        s[1] = (mr * qr[1] + nx * qr[4]) + (ml * ql[1] + nx * ql[4]);
        s[2] = (mr * qr[2] + ny * qr[4]) + (ml * ql[2] + ny * ql[4]);
        s[3] = (mr * qr[3] + nz * qr[4]) + (ml * ql[3] + nz * ql[4]);
        s[4] = ((er + qr[4]) * cr - qr[4] * nt) + ((el + ql[4]) * cl - ql[4] * nt);
    }
    // what is not finite reaches the energy flux, by each of the other terms
    auto finite = [](double x) { return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000; };
    const double rl1 = recip(ql[0]);
    if (same) {
#pragma unroll
        for (int m = 0; m < 5; m++) f[m] = 0.5 * s[m];
        const double pr = ql[4] * rl1;
        return pr > 1.0e-10 * fma(gama2, pr, 0.5 * v2l) && finite(f[4]);
    }
    const double hl = fma(gama2, ql[4] * rl1, 0.5 * v2l), hr = fma(gama2, qr[4] * recip(qr[0]), 0.5 * v2r);
    const double rr = qr[0] * rl1, rrl = rr * recip_sqrt(rr), w = recip(rrl + 1.0), rm = ql[0] * rrl;
    const double um = fma(qr[1], rrl, ql[1]) * w, vm = fma(qr[2], rrl, ql[2]) * w, wm = fma(qr[3], rrl, ql[3]) * w,
                 hm = fma(hr, rrl, hl) * w;
    const double c2 = (hm - 0.5 * fma(um, um, fma(vm, vm, wm * wm))) * gama1;
    const double c_1 = recip_sqrt(c2), c = c2 * c_1;
    const double cta = fma(um, nx, fma(vm, ny, wm * nz)) + nt;
    const double k2 = fmax(fma(nx, nx, fma(ny, ny, nz * nz)), SML_SSS * SML_SSS), cgm1 = recip_sqrt(k2), cgm = k2 * cgm1;
    nx = nx * cgm1;
    ny = ny * cgm1;
    nz = nz * cgm1;
    const double ccgm = c * cgm, deti = P.efix * cgm, det2 = deti * deti, lm = cta - ccgm, lp = cta + ccgm;
    // the floor stands for a zero root (no entropy fix and a zero eigenvalue)
    auto root = [](double x) { x = fmax(x, 1.0e-290); return x * recip_sqrt(x); };
    const double l1 = root(fma(lm, lm, det2)), l4 = root(fma(cta, cta, det2)), l5 = root(fma(lp, lp, det2));
    const double d0 = qr[0] - ql[0], d1 = qr[1] - ql[1], d2 = qr[2] - ql[2], d3 = qr[3] - ql[3], d4 = qr[4] - ql[4];
    const double rodcta = rm * fma(d1, nx, fma(d2, ny, d3 * nz));
    const double dp_c2 = d4 * c_1 * c_1, rodctac = rodcta * c_1;
    const double a1 = l4 * (d0 - dp_c2), a2 = 0.5 * l5 * (dp_c2 + rodctac), a3 = 0.5 * l1 * (dp_c2 - rodctac);
    const double a4 = a1 + a2 + a3, a5 = c * (a2 - a3);
    const double a6 = l4 * fma(rm, d1, -nx * rodcta), a7 = l4 * fma(rm, d2, -ny * rodcta), a8 = l4 * fma(rm, d3, -nz * rodcta);
    f[0] = 0.5 * (s[0] - a4);
    f[1] = 0.5 * (s[1] - fma(um, a4, fma(nx, a5, a6)));
    f[2] = 0.5 * (s[2] - fma(vm, a4, fma(ny, a5, a7)));
    f[3] = 0.5 * (s[3] - fma(wm, a4, fma(nz, a5, a8)));
    f[4] = 0.5 * (s[4] - (fma(hm, a4, cta * cgm1 * a5) + fma(um, a6, fma(vm, a7, wm * a8)) - c2 * a1 * gama1_1));
    return c2 > 1.0e-10 * hm && finite(f[4]);
}

// the flux-vector splittings chosen by nflux (Convect.f90:12-46): 1
// Steger-Warming, 2 Van Leer.  Returns the number of c^2 failures.
template <int NFLUX>
__device__ __forceinline__ int flux_split(const DevParams &P, const double *ql, const double *qr, double nx, double ny, double nz,
                                          double nt, double *f) {
    double fl[5], fr[5];
    int bad = 0;
    if (NFLUX == 2) {
        bad = flux_vl_pn(P, ql, nx, ny, nz, nt, fl, 1);
        bad += flux_vl_pn(P, qr, nx, ny, nz, nt, fr, -1);
    } else {
        flux_sw_pn(P, ql, nx, ny, nz, nt, fl, 1);
        flux_sw_pn(P, qr, nx, ny, nz, nt, fr, -1);
    }
#pragma unroll
    for (int m = 0; m < 5; m++) f[m] = fl[m] + fr[m];
    return bad;
}

// Sutherland viscosity, compute_visl_ns (GasModel.f90:219-235)
__device__ __forceinline__ double sutherland(const DevParams &P, double tm) {
    return tm * sqrt(tm) * (1.0 + P.visc) / (tm + P.visc);
}

// error counters
enum ErrSlot : int { ERR_ROE = 0, ERR_UPDATE_BLOCKS = 1, ERR_BADLIST_OVERFLOW = 2, ERR_TIMEOUT = 3, ERR_NSLOTS = 4 };

}  // namespace wcns
