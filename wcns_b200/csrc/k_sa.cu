// k_sa.cu -- Spalart-Allmaras turbulence model: turbulence(nb) ->
// differential_model_turbulence (turblence.f90:15-103) with nlamtur=1,
// nameturb='SA', ncmpcor<=9, ndes=0, ntrans=0, nwtmax=0 and method=1
// (finite differences), for all blocks at once.
//
// Per step:
//   k_sa_point<SA_DMU>    derivatives of qke at points 1..n (dfidxyz_center)
//   k_sa_point<SA_RHS>    per interior point: SA source, diffusion, spectral
//                         radius and first-order upwind convection, in the
//                         reference's order of accumulation into dqke/spec
//   k_sa_lusgs            scalar LU-SGS, forward and backward hyperplane
//                         wavefronts, one CTA per block
//   k_sa_point<SA_UPDATE> qke update, vist, kmaxlim clamp
// Set-up: k_sa_wall_dist (calc_wall_dists_parallel) and k_sa_init (init_SA).
#include "wcns_launch.h"

namespace wcns {

namespace {

constexpr double SA_CB1 = 0.1355, SA_CB2 = 0.622, SA_EPS = 1.0e-20;  // turblence.f90:2508-2513
constexpr double SA_CGA = 2. / 3.0;
constexpr double SA_CW2 = 0.3;
constexpr double SA_MUOO = 1.0e-1;    // inflow_turbulence, turblence.f90:3174
constexpr double SA_MINLIM = 1.0e-20; // update_turbulence, turblence.f90:589

enum SaPhase { SA_DMU = 0, SA_RHS = 1, SA_UPDATE = 2 };

__device__ __forceinline__ double dmax(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double dmin(double a, double b) { return a < b ? a : b; }

// dfidxyz_center, turblence.f90:753-849 (finite-difference branch)
__device__ __forceinline__ void center_deriv(const DevFields &F, const DevBlock &B, const double *fi, long long id,
                                             double *d) {
    const long long sj = B.gx, sk = (long long)B.gx * B.gy;
    double dkc = fi[id + 1] - fi[id - 1];
    double det = fi[id + sj] - fi[id - sj];
    double dct = fi[id + sk] - fi[id - sk];
    double ddx = dkc * F.f[F_KCX][id] + det * F.f[F_ETX][id] + dct * F.f[F_CTX][id];
    double ddy = dkc * F.f[F_KCY][id] + det * F.f[F_ETY][id] + dct * F.f[F_CTY][id];
    double ddz = dkc * F.f[F_KCZ][id] + det * F.f[F_ETZ][id] + dct * F.f[F_CTZ][id];
    double vol2 = 0.5 / F.f[F_VOL][id];
    d[0] = ddx * vol2;
    d[1] = ddy * vol2;
    d[2] = ddz * vol2;
}

__device__ __forceinline__ double cube(double x) { return x * x * x; }

// flux_turbulence, turblence.f90:437-459, of the state u, v, w, qke, r with the
// half-point normal nx, ny, nz: positive (SIGN 1) or negative (-1) part
template <int SIGN>
__device__ __forceinline__ double conv_flux(double u, double v, double w, double q, double r, double nx, double ny, double nz) {
    double l1 = nx * u + ny * v + nz * w;
    l1 = 0.5 * (l1 + SIGN * fabs(l1));
    return l1 * q * r;
}

// One point's right-hand side: 90 loads, 450 FP64 operations (2650 and 950 before).
// Bound by the neighbours' way from L2 now, by its instructions then.  Every
// neighbour's value is loaded once and serves the gradients, the diffusion and the
// convection; the viscosity it needs there is a field (viseq, written with the
// derivatives of qke), not a division per half point; the powers are products, and the
// sixth root a cube root of a square root.  The terms add up in the reference's order.
// Channel (4.2 M points) with the derivatives: 574 us before, 461 now; 64 small blocks
// (0.9 M points) 143 and 120 us.  Three CTAs of 256 per SM; two 504 us, four 475.
__device__ void sa_rhs_point(const DevFields &F, const SaFields &S, const SaParams &P, const DevBlock &B, int id) {
    const double uc = __ldg(F.f[F_U] + id), vc = __ldg(F.f[F_V] + id), wc = __ldg(F.f[F_W] + id), ro = __ldg(F.f[F_R] + id);
    const double vtbar = S.qke[id], visc = __ldg(S.vis + id);
    const double dmc[3] = {__ldg(S.dmu[0] + id), __ldg(S.dmu[1] + id), __ldg(S.dmu[2] + id)};
    double du[3][3];            // differences of u, v, w along each direction
    double dif[3], conv[3];     // cal_rhs_viscous_turbulence_dif_r (turblence.f90:1022-1185) and NND_turbulence (291-435) per direction
    double kc[3][3];            // the point's metrics
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const int st = d == 0 ? 1 : d == 1 ? B.gx : B.gx * B.gy;
        const double *mx = F.f[F_KCX + 3 * d], *my = F.f[F_KCY + 3 * d], *mz = F.f[F_KCZ + 3 * d];
        kc[d][0] = __ldg(mx + id);
        kc[d][1] = __ldg(my + id);
        kc[d][2] = __ldg(mz + id);
        double un[2], vn[2], wn[2], fvl[2], fc[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {  // the half points below and above
            const int q = h ? id + st : id - st;
            const double nx = 0.5 * (__ldg(mx + q) + kc[d][0]), ny = 0.5 * (__ldg(my + q) + kc[d][1]), nz = 0.5 * (__ldg(mz + q) + kc[d][2]);
            un[h] = __ldg(F.f[F_U] + q);
            vn[h] = __ldg(F.f[F_V] + q);
            wn[h] = __ldg(F.f[F_W] + q);
            const double rn = __ldg(F.f[F_R] + q), qn = S.qke[q];
            const double dmudx = __ldg(S.dmu[0] + q) + dmc[0], dmudy = __ldg(S.dmu[1] + q) + dmc[1], dmudz = __ldg(S.dmu[2] + q) + dmc[2];
            fvl[h] = (dmudx * nx + dmudy * ny + dmudz * nz) * (__ldg(S.vis + q) + visc) * 0.25;
            // xk = xb = 0 (never assigned in the reference), so the minmod slopes
            // are zeros and the half-point states are the neighbouring points'
            // values exactly: fc(l) = f+(q(l-1)) + f-(q(l)).
            if (h == 0) fc[0] = conv_flux<1>(un[0], vn[0], wn[0], qn, rn, nx, ny, nz) + conv_flux<-1>(uc, vc, wc, vtbar, ro, nx, ny, nz);
            else fc[1] = conv_flux<1>(uc, vc, wc, vtbar, ro, nx, ny, nz) + conv_flux<-1>(un[1], vn[1], wn[1], qn, rn, nx, ny, nz);
        }
        du[d][0] = un[1] - un[0];
        du[d][1] = vn[1] - vn[0];
        du[d][2] = wn[1] - wn[0];
        dif[d] = fvl[1] - fvl[0];
        conv[d] = fc[1] - fc[0];
    }
    // cal_rhs_source_SA, turblence.f90:2567-2686; the gradient as in center_deriv
    const double volume = __ldg(F.f[F_VOL] + id), vsl = __ldg(F.f[F_VISL] + id);
    const double vol2 = 0.5 / volume;
    auto grad = [&](int m, int x) { return (du[0][m] * kc[0][x] + du[1][m] * kc[1][x] + du[2][m] * kc[2][x]) * vol2; };
    const double romu = ro * vtbar;
    const double ds = __ldg(S.dist + id);
    const double dn = ds > P.re ? ds : P.re;
    const double dn2 = dn * dn;
    const double reki2dn2 = P.reynolds * P.ki2 * dn2;
    const double kafan = romu / vsl;
    const double kf3 = cube(kafan);
    const double fv1 = kf3 / (kf3 + P.cv13);
    const double fv2 = 1.0 - kafan / (1.0 + kafan * fv1);
    const double a = grad(0, 1) - grad(1, 0), b = grad(1, 2) - grad(2, 1), c = grad(2, 0) - grad(0, 2);
    const double omg = sqrt(a * a + b * b + c * c);
    double sbar = omg + vtbar / reki2dn2 * fv2;
    sbar = sbar > SA_EPS ? sbar : SA_EPS;
    double rbar = vtbar / (sbar * reki2dn2);
    rbar = rbar < 10.0 ? rbar : 10.0;
    const double rbar2 = rbar * rbar, rbar5 = rbar2 * rbar2 * rbar;
    const double gbar = rbar + SA_CW2 * rbar * (rbar5 - 1.0);
    const double gbar6 = cube(gbar * gbar);
    const double fw = gbar * cbrt(sqrt((1.0 + P.cw36) / (gbar6 + P.cw36)));
    const double cpmu = SA_CB1 * sbar;  // ft2 = 0
    const double cdmu = P.cw1 * fw * vtbar / dn2 / P.reynolds;
    const double sp = cpmu * vtbar, sd = cdmu * vtbar;
    const double dbar = SA_CB2 / SA_CGA * (dmc[0] * dmc[0] + dmc[1] * dmc[1] + dmc[2] * dmc[2]) * P.re;
    double dq = 0.0 - ro * (sp - sd + dbar) * volume;
    const double sm = cpmu - 2.0 * cdmu;
    double spec = 0.0 - (sm < 0.0 ? sm : 0.0) * volume;
    const double rre = P.re * ro;
#pragma unroll
    for (int d = 0; d < 3; d++) dq = dq - rre * dif[d];
#pragma unroll
    for (int d = 0; d < 3; d++) dq = dq + conv[d];
    // cal_spec_turbulence_r, turblence.f90:218-259
    double un[3], nn[3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
        un[d] = uc * kc[d][0] + vc * kc[d][1] + wc * kc[d][2];
        nn[d] = kc[d][0] * kc[d][0] + kc[d][1] * kc[d][1] + kc[d][2] * kc[d][2];
    }
    spec = spec + fabs(un[0]) + fabs(un[1]) + fabs(un[2]) + 1.0 / (__ldg(F.f[F_DTDT] + id) * P.timedt_turb);
    spec = spec + P.re * 2.0 * (visc / volume) * (nn[0] + nn[1] + nn[2]);
    S.dqke[id] = dq;
    S.spec[id] = 1.0 / spec;  // the sweeps multiply: a division would be 124 cycles of every plane's chain
}

// cal_vist_SA (turblence.f90:2735-2760) at one point
__device__ __forceinline__ double vist_of(double r, double qke, double visl, double cv13) {
    double romu = r * qke;
    double kafan = romu / visl;
    double kf3 = cube(kafan);
    double fv1 = kf3 / (kf3 + cv13);
    return romu * fv1;
}

// One kernel for the point-wise phases.  lo: first index of the range in
// every direction (1 for SA_DMU, 2 for SA_RHS, 0 for SA_UPDATE); the range
// ends at n - (lo == 2 ? 1 : 0).  Fields are indexed with 32 bits (HBM would hold
// fields of 4e8 points).
template <int PHASE>
__global__ void __launch_bounds__(256, PHASE == SA_RHS ? 3 : 0) k_sa_point(DevFields F, SaFields S, SaParams P, const DevBlock *__restrict__ blocks) {
    const DevBlock B = blocks[blockIdx.y];
    const int lo = PHASE == SA_DMU ? 1 : PHASE == SA_RHS ? 2 : 0;
    const int hi_off = PHASE == SA_RHS ? 1 : 0;
    const int mi = B.ni - hi_off - lo + 1, mj = B.nj - hi_off - lo + 1, mk = B.nk - hi_off - lo + 1;
    if (mi <= 0 || mj <= 0 || mk <= 0) return;
    const long long np = (long long)mi * mj * mk;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < np; q += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        {
            const int q32 = (int)q, r = q32 / mi;
            i = q32 - r * mi + lo;
            j = r % mj + lo;
            k = r / mj + lo;
        }
        const int id = (int)gidx(B, i, j, k);
        if (PHASE == SA_DMU) {
            double d[3];
            center_deriv(F, B, S.qke, id, d);
            S.dmu[0][id] = d[0];
            S.dmu[1][id] = d[1];
            S.dmu[2][id] = d[2];
            // viscosity_equivalent_SA_r, turblence.f90:2785-2808
            S.vis[id] = 1.5 * (F.f[F_VISL][id] / F.f[F_R][id] + S.qke[id]);
        } else if (PHASE == SA_RHS) {
            sa_rhs_point(F, S, P, B, id);
        } else {
            const bool in1 = i >= 1 && j >= 1 && k >= 1;
            const bool in2 = i >= 2 && j >= 2 && k >= 2 && i <= B.ni - 1 && j <= B.nj - 1 && k <= B.nk - 1;
            double vt = S.vist[id];
            if (in1) {
                double qk = S.qke[id];
                const double r = F.f[F_R][id];
                if (in2) {  // update_turbulence, turblence.f90:606-615
                    double qn = qk + S.dqke[id] / r, lim = SA_MINLIM * SA_MUOO;
                    qk = dmax(qn, lim);
                    S.qke[id] = qk;
                }
                vt = vist_of(r, qk, F.f[F_VISL][id], P.cv13);
            }
            if (P.kmaxlim > 1.0e-15) vt = dmin(vt, P.kmaxlim * F.f[F_VISL][id]);  // max_control_turbulence
            S.vist[id] = vt;
        }
    }
}

// lusgs_turbulence, turblence.f90:477-558.  The lexicographic forward sweep
// reads the already updated lower neighbours (i-1, j-1, k-1) and the
// backward sweep the upper ones, so every hyperplane i+j+k = p can be
// updated at once after the previous one; one CTA per block walks the
// planes with a barrier in between (dqke stays in global memory, which the
// barrier makes visible to the whole CTA).
__device__ __forceinline__ double mxdq(const DevFields &F, long long nid, long long mid, int d, double dq, double npn) {
    // mxdq_std_turbulence (turblence.f90:560-583) with the neighbour's
    // velocity and the metrics of getrkec_mml at the neighbour (mid: the
    // neighbour with indices 0 and n+1 clamped to the block)
    double l1 = F.f[F_KCX + 3 * d][mid] * F.f[F_U][nid] + F.f[F_KCY + 3 * d][mid] * F.f[F_V][nid] +
                F.f[F_KCZ + 3 * d][mid] * F.f[F_W][nid];
    l1 = 0.5 * (l1 + npn * fabs(l1));
    return l1 * dq;
}

__global__ void __launch_bounds__(1024) k_sa_lusgs(DevFields F, SaFields S, const DevBlock *__restrict__ blocks) {
    const DevBlock B = blocks[blockIdx.x];
    const int ni = B.ni, nj = B.nj, nk = B.nk;
    if (ni < 3 || nj < 3 || nk < 3) return;
    const int wj = nj - 2, ncol = (nj - 2) * (nk - 2);
    const long long st[3] = {1, B.gx, (long long)B.gx * B.gy};
    const int n3[3] = {ni, nj, nk};
    double *dqke = S.dqke;
    for (int pass = 0; pass < 2; pass++) {
        const int np = (ni - 1) + (nj - 1) + (nk - 1) - 6 + 1;  // planes 6 .. (ni-1)+(nj-1)+(nk-1)
        for (int pp = 0; pp < np; pp++) {
            const int p = pass == 0 ? 6 + pp : (ni - 1) + (nj - 1) + (nk - 1) - pp;
            for (int t = threadIdx.x; t < ncol; t += blockDim.x) {
                const int j = 2 + t % wj, k = 2 + t / wj, i = p - j - k;
                if (i < 2 || i > ni - 1) continue;
                const long long id = gidx(B, i, j, k);
                const int c[3] = {i, j, k};
                double tt[3];
#pragma unroll
                for (int d = 0; d < 3; d++) {
                    const long long nid = pass == 0 ? id - st[d] : id + st[d];
                    const int cn = pass == 0 ? c[d] - 1 : c[d] + 1;
                    // getrkec_mml clamps 0 -> 1 and n+1 -> n; neighbours of
                    // interior points stay within 1..n, so mid == nid
                    const long long mid = (cn == 0) ? nid + st[d] : (cn == n3[d] + 1) ? nid - st[d] : nid;
                    tt[d] = mxdq(F, nid, mid, d, dqke[nid], pass == 0 ? 1.0 : -1.0);
                }
                const double rhs0 = tt[0] + tt[1] + tt[2];
                if (pass == 0) dqke[id] = (rhs0 - dqke[id]) * S.spec[id];
                else dqke[id] = dqke[id] - rhs0 * S.spec[id];
            }
            __syncthreads();
        }
    }
}

// calc_wall_dists_parallel, parallel.f90:4313-4470: the squared distance to
// the nearest wall point (exact minimum, so the order of the wall list does
// not matter), then sqrt + small, at points 1..n.
constexpr int WD_TILE = 512;
// The wall points a block measures to are those of its own set of blocks
// joined through interfaces (wall_range[2b] .. wall_range[2b+1]): one case,
// also when independent cases share a context.
__global__ void __launch_bounds__(256) k_sa_wall_dist(SaFields S, const double *__restrict__ xyz, long long total,
                                                      const double *__restrict__ wall, const int *__restrict__ wall_range,
                                                      const DevBlock *__restrict__ blocks) {
    __shared__ double sw[3 * WD_TILE];
    const DevBlock B = blocks[blockIdx.y];
    const int wbeg = wall_range[2 * blockIdx.y], nwall = wall_range[2 * blockIdx.y + 1];
    const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const bool act = q < B.npts;
    long long id = 0;
    double xc = 0.0, yc = 0.0, zc = 0.0, dmn = 1.0e30;
    if (act) {
        int i, j, k;
        decode_point(B, q, i, j, k);
        id = gidx(B, i, j, k);
        xc = xyz[id];
        yc = xyz[total + id];
        zc = xyz[2 * total + id];
    }
    for (int w0 = wbeg; w0 < nwall; w0 += WD_TILE) {
        const int nt = nwall - w0 < WD_TILE ? nwall - w0 : WD_TILE;
        __syncthreads();
        for (int e = threadIdx.x; e < 3 * nt; e += blockDim.x) sw[e] = wall[3 * (long long)w0 + e];
        __syncthreads();
        if (act)
            for (int w = 0; w < nt; w++) {
                double dx = xc - sw[3 * w], dy = yc - sw[3 * w + 1], dz = zc - sw[3 * w + 2];
                double dist = dx * dx + dy * dy + dz * dz;
                dmn = dist < dmn ? dist : dmn;
            }
    }
    if (act) S.dist[id] = sqrt(dmn) + SMALL;
}

// init_SA, turblence.f90:2701-2733: qke = muoo, vist = vt over -1..n+1
__global__ void k_sa_init(SaFields S, double vt, const DevBlock *__restrict__ blocks) {
    const DevBlock B = blocks[blockIdx.y];
    const int mi = B.ni + 3, mj = B.nj + 3, mk = B.nk + 3;
    const long long np = (long long)mi * mj * mk;
    for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < np; q += (long long)gridDim.x * blockDim.x) {
        const long long r = q / mi;
        const int i = (int)(q - r * mi) - 1, j = (int)(r % mj) - 1, k = (int)(r / mj) - 1;
        const long long id = gidx(B, i, j, k);
        S.qke[id] = SA_MUOO;
        S.vist[id] = vt;
    }
}

long long max_points(const LaunchCtx &c, int extra) {
    long long m = 0;
    for (int b = 0; b < c.nblocks; b++) {
        const DevBlock &B = c.hblocks[b];
        long long n = (long long)(B.ni + extra) * (B.nj + extra) * (B.nk + extra);
        m = n > m ? n : m;
    }
    return m;
}

unsigned grid_for(long long n) {
    long long g = (n + 255) / 256;
    return (unsigned)(g < 1 ? 1 : (g > 4096 ? 4096 : g));
}

}  // namespace

void launch_sa_setup(const LaunchCtx &c, const double *xyz, const double *wall, const int *wall_range, double vt) {
    k_sa_init<<<dim3(grid_for(max_points(c, 3)), c.nblocks), 256, 0, c.stream>>>(*c.SA, vt, c.blocks);
    k_sa_wall_dist<<<dim3((unsigned)((max_points(c, 0) + 255) / 256), c.nblocks), 256, 0, c.stream>>>(
        *c.SA, xyz, c.total, wall, wall_range, c.blocks);
}

int launch_turbulence(const LaunchCtx &c) {
    k_sa_point<SA_DMU><<<dim3(grid_for(max_points(c, 0)), c.nblocks), 256, 0, c.stream>>>(*c.F, *c.SA, *c.SAP, c.blocks);
    k_sa_point<SA_RHS><<<dim3(grid_for(max_points(c, 0)), c.nblocks), 256, 0, c.stream>>>(*c.F, *c.SA, *c.SAP, c.blocks);
    prof_mark(c, "sa_rhs");
    // large blocks: the scalar sweeps on the wide chunks of the mean-flow sweeps
    const int nl = (c.wide && c.wide->A.sa) ? launch_sa_lusgs_wide(c) : 1;
    if (nl == 1) k_sa_lusgs<<<c.nblocks, 1024, 0, c.stream>>>(*c.F, *c.SA, c.blocks);
    prof_mark(c, "sa_lusgs");
    k_sa_point<SA_UPDATE><<<dim3(grid_for(max_points(c, 1)), c.nblocks), 256, 0, c.stream>>>(*c.F, *c.SA, *c.SAP, c.blocks);
    prof_mark(c, "sa_update");
    return 3 + nl;
}

}  // namespace wcns
