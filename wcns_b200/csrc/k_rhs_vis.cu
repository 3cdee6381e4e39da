// k_rhs_vis.cu -- laminar viscous residual.
//
// Restates r_h_s_vis (RHS.f90:2-30) -> WCNSE5_VIS_virtual
// (sub_tgh.f90:1511-1810):
//   * node derivatives of (u,v,w,T) along each index direction
//     (UVWT_DER_4th_virtual sub_tgh.f90:1909-2029 with
//     DUVWT_NODE_LINE_virtual 2217-2272) -> 12 fields, one kernel;
//   * per line and half node: VALUE_line_half_virtual (2335-2387),
//     VALUE_HALF_NODE_IJK (newvis.f90:421-554), half-node derivatives
//     (DUVWT_half_line_virtual 2277-2330), metric/volume/viscosity
//     interpolation (VALUE_HALF_NODE WCNSE5.f90:799-852), Cartesian
//     gradients (DUVWT_DXYZ WCNSE5.f90:854-890), stress and heat flux
//     (FLUX_VIS_LINE_new newvis.f90:283-349);
//   * per point: FLUX_DXYZ and dq -= re*dFv.
// The boundary flag of a line is the reference's uvwt(4,-2) test: -1 when the
// third ghost density is negative, otherwise the ghost temperature.
#include <algorithm>

#include "wcns_dev.cuh"
#include "wcns_launch.h"

namespace wcns {

// ---------------------------------------------------------------------------
// node derivatives and the molecular viscosity: one thread per interior point
// ---------------------------------------------------------------------------
// Bound by the instructions around its 48 loads: fields are indexed with 32 bits
// (a field has far fewer points than that: HBM would hold 4e8), and the one-sided
// formulas run only where an end has a boundary, not wherever a line ends.
// The viscosity goes to memory here, so that the three line kernels read 8 bytes
// where each would evaluate a root and a division per point.
__global__ void __launch_bounds__(256, 5) k_node_deriv(DevParams P, DevFields F, const DevBlock *__restrict__ blocks, int nblocks) {
    int bi = blockIdx.y;
    if (bi >= nblocks) return;
    const DevBlock B = blocks[bi];
    long long np = B.npts;
    for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < np; p += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        decode_point(B, p, i, j, k);
        const int id = (int)gidx(B, i, j, k);
        // viscosities at the point, as the reference's visl/vist arrays:
        // mu + vist and mu*cp_prl + vist*cp_prt (vist = 0 when laminar)
        const double mu = sutherland(P, __ldg(F.f[F_T] + id));
        const double vt = F.f[F_VIST] ? __ldg(F.f[F_VIST] + id) : 0.0;
        F.f[F_MU][id] = mu + vt;
        F.f[F_MU + 1][id] = mu * B.cp_prl + vt * B.cp_prt;
#pragma unroll 1
        for (int d = 0; d < 3; d++) {
            const int n = dimof(B, d);
            const int l = d == 0 ? i : (d == 1 ? j : k);
            const int st = (int)dstride(B, d);
            bool fl = false, fr = false;
            const int l0 = id - l * st;  // index of position 0 on the line
            if (n > NIJK2ND) {
                if (l <= 2) fl = __ldg(F.f[F_R] + l0 - 2 * st) < 0.0 ? true : (__ldg(F.f[F_T] + l0 - 2 * st) < 0.0);
                else if (l >= n - 1) fr = __ldg(F.f[F_R] + l0 + (n + 3) * st) < 0.0 ? true : (__ldg(F.f[F_T] + l0 + (n + 3) * st) < 0.0);
            }
            if (n <= NIJK2ND) {
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    const double *u = F.f[m == 3 ? F_T : F_U + m] + id;
                    F.f[F_DUV0 + m + 4 * d][id] = 0.5 * (__ldg(u + st) - __ldg(u - st));
                }
            } else if (!fl && !fr) {  // the interior formula
                double v[4][4];
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    const double *u = F.f[m == 3 ? F_T : F_U + m] + id;
                    v[m][0] = __ldg(u - 2 * st);
                    v[m][1] = __ldg(u - st);
                    v[m][2] = __ldg(u + st);
                    v[m][3] = __ldg(u + 2 * st);
                }
#pragma unroll
                for (int m = 0; m < 4; m++)
                    F.f[F_DUV0 + m + 4 * d][id] = div_by(8.0 * (v[m][2] - v[m][1]) + -1.0 * (v[m][3] - v[m][0]), 12.0, 1.0 / 12.0);
            } else {  // one-sided at the first and second point from the end
                const int e = l0 + (fl ? st : n * st), s1 = fl ? st : -st;
                const bool end = l == 1 || l == n;
                const double c0 = end ? -11. : -3.0, c1 = end ? 18. : -10.0, c2 = end ? -9. : 18.0, c3 = end ? 2. : -6.0;
                const double den = end ? 6.0 : 12.0, rden = end ? 1.0 / 6.0 : 1.0 / 12.0;
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    const double *u = F.f[m == 3 ? F_T : F_U + m] + e;
                    double du = c0 * __ldg(u) + c1 * __ldg(u + s1) + c2 * __ldg(u + 2 * s1) + c3 * __ldg(u + 3 * s1);
                    const double u4 = __ldg(u + 4 * s1);
                    if (!end) du = du + u4;
                    F.f[F_DUV0 + m + 4 * d][id] = div_by(fl ? du : -du, den, rden);
                }
            }
        }
    }
}

void launch_node_derivatives(const LaunchCtx &c) {
    if (c.mixed) return launch_node_derivatives_mx(c);
    long long maxp = 0;
    for (int b = 0; b < c.nblocks; b++) maxp = c.hblocks[b].npts > maxp ? c.hblocks[b].npts : maxp;
    int gx = (int)((maxp + 255) / 256);
    dim3 grid(gx, c.nblocks);
    k_node_deriv<<<grid, 256, 0, c.stream>>>(*c.P, *c.F, c.blocks, c.nblocks);
}

// ---------------------------------------------------------------------------
// viscous line flux
// ---------------------------------------------------------------------------
// One CTA marches along NL lines, C half nodes at a time: thread (c, ln) forms the
// viscous flux at half node h0 + c of line ln, then the flux difference at a point.
// VIS_NF quantities of the points h0-1 .. h0+C+1 are in a ring in shared memory:
// u, v, w, T, the 8 node derivatives along the two other directions, the 9 metrics
// in the order kcx,etx,ctx,kcy,ety,cty,kcz,etz,ctz, vol and the two viscosities;
// the next C points replace the oldest while the differences are formed.
//
// What bounds it: latency, of loads above all (staging and storing alone were 82 %
// of the kernel that staged whole lines; FP64 pipe 13-16 % busy, DRAM 20 %).  So
//   - a chunk of C = 8 half nodes (cmax) leaves room for 16 lines in a CTA: 128 contiguous
//     bytes per load across the lines, where 3 to 5 whole lines were 24 to 40 (the
//     sectors read from L2 were four times the bytes used in the j direction);
//   - the copies are asynchronous and need no registers, four CTAs of 128 registers
//     fit an SM, and the old residual is read ahead of the barrier;
//   - a point's quantities lie together, so a thread reaches all of them, 16 bytes at
//     a time, from one address; the pitch is 2 mod 4: eight lanes' 16 bytes never
//     share a bank;
//   - formulas of the ends run in their own threads, not for a warp's every line.
// Measured with the node derivatives, per step: channel (24 blocks, 4.2 M points)
// 3110 us before, 1365 now; 64 small blocks (0.9 M points) 872 and 389 us; the plate
// (8 blocks, 0.23 M points) 217 and 119 us.  Other splits over the channel: C = 10
// 1437 us, C = 16 with 256 threads 1541, 64 threads 1804, 96 registers with spills
// 1948; a ring that prefetches one chunk more (and holds fewer warps) 1861.
constexpr int VIS_NF = 24, VIS_PITCH = 26, VIS_FP = 4;
constexpr int VIS_THREADS = 128, VIS_CTAS = 4;
constexpr int VIS_MAX_LINES = 32;  // lines per CTA
enum : int { VS_U = 0, VS_DN = 4, VS_MET = 12, VS_VOL = 21, VS_V1 = 22, VS_V2 = 23 };

// A line of n points has n+1 half nodes in nch chunks of C; the first one takes the
// remainder, so that the half nodes near the right end have a full chunk of points.
__host__ __device__ inline int vis_chunk(int n, int cmax) {
    const int H = n + 1, nch = (H + cmax - 1) / cmax;
    return (H + nch - 1) / nch;
}
__host__ __device__ inline int vis_ring(int n, int cmax) {  // points in the ring
    const int w = vis_chunk(n, cmax) + 3;
    return w < n + 4 ? w : n + 4;
}
// lanes of a row of the ring: odd for i-lines, whose loads walk along a line
__host__ __device__ inline int vis_row(int dir, int nl) { return dir == 0 ? nl | 1 : nl; }

__device__ __forceinline__ void copy8_async(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// out == nullptr: dq -= re*dFv in place; otherwise re*dFv is stored in
// out[m*stride + point] for an ordered combine (k_combine_dq).
template <int dir>
__global__ void __launch_bounds__(VIS_THREADS, VIS_CTAS) k_rhs_vis(DevParams P, DevFields F, const DevBlock *__restrict__ blocks,
                                                    const LineGroup *__restrict__ groups, int cmax, double *out, long long stride) {
    extern __shared__ __align__(16) double smem[];
    const LineGroup G = groups[blockIdx.x];
    const DevBlock B = blocks[G.blk];
    const int n = dimof(B, dir), NL = G.nl, NLP = vis_row(dir, NL);
    const int H = n + 1, C = vis_chunk(n, cmax), RP = vis_ring(n, cmax), FR = C + 5;
    double *fv = smem + RP * NLP * VIS_PITCH;  // the last FR half nodes' fluxes
    __shared__ int flags[VIS_MAX_LINES];       // bit 0: the left end has a boundary, bit 1: the right end
    constexpr int a1 = dir == 0 ? 1 : 0, a2 = dir == 2 ? 1 : 2;
    const int st = (int)dstride(B, dir);
    int o[3];
    o[a1] = G.a0;
    o[a2] = G.b;
    o[dir] = 0;
    const int base = (int)gidx(B, o[0], o[1], o[2]);          // position 0 of the first line
    const int lstep = (int)dstride(B, a1);                    // to the next line
    if ((int)threadIdx.x < NL) {
        const int gl = base + threadIdx.x * lstep - 2 * st, gr = gl + (n + 5) * st;
        const double rl = F.f[F_R][gl], tl = F.f[F_T][gl], rr = F.f[F_R][gr], tr = F.f[F_T][gr];
        flags[threadIdx.x] = (rl < 0.0 || tl < 0.0 ? 1 : 0) | (rr < 0.0 || tr < 0.0 ? 2 : 0);
    }
    // this thread's half node and line; its point and line in the loads and stores,
    // which walk along the line for i-lines and across the lines otherwise
    const int c = threadIdx.x / NL, ln = threadIdx.x - c * NL;
    const int pc = dir == 0 ? threadIdx.x % C : c, pl = dir == 0 ? threadIdx.x / C : ln;
    const bool work = c < C, mover = dir == 0 ? pl < NL : c < C;
    const int pbase = base + pl * lstep;
    auto wrap = [](int x, int m) { return x >= m ? x - m : x; };
    auto load = [&](int lo, int hi, int slo) {  // points lo..hi into the ring, from slot slo on
        if (mover)
            for (int p = lo + pc; p <= hi; p += C) {
                constexpr int g0 = dir == 0 ? 1 : 0, g1 = dir == 2 ? 1 : 2;  // the two other directions
                const int gi = pbase + p * st;
                double *S = smem + (wrap(slo + p - lo, RP) * NLP + pl) * VIS_PITCH;
#pragma unroll
                for (int m = 0; m < 4; m++) copy8_async(S + VS_U + m, F.f[m == 3 ? F_T : F_U + m] + gi);
                if (p >= 1 && p <= n) {
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        copy8_async(S + VS_DN + m, F.f[F_DUV0 + m + 4 * g0] + gi);
                        copy8_async(S + VS_DN + 4 + m, F.f[F_DUV0 + m + 4 * g1] + gi);
                    }
#pragma unroll
                    for (int q = 0; q < 9; q++)  // kcx,etx,ctx,kcy,... = F_KCX + 3*(q%3) + q/3
                        copy8_async(S + VS_MET + q, F.f[F_KCX + 3 * (q % 3) + q / 3] + gi);
                    copy8_async(S + VS_VOL, F.f[F_VOL] + gi);
                    copy8_async(S + VS_V1, F.f[F_MU] + gi);
                    copy8_async(S + VS_V2, F.f[F_MU + 1] + gi);
                }
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int h0 = 0, len = H - (H - 1) / C * C;       // this chunk's half nodes h0 .. h0+len-1
    int have = len + 1 < 5 ? 5 : len + 1;        // the last point loaded: the left end's formulas reach point 5
    if (have > n + 2) have = n + 2;
    int hs = 0, fs = 0;                          // slots of point h0-1 and of half node h0
    int done = 0;                                // the last point whose difference is out
    load(-1, have, 0);
    for (;;) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const int lhi = h0 + len == H ? n : h0 + len - 3;  // differences this chunk completes: done+1 .. lhi
        // the old residual of this thread's point, ahead of the barrier
        double old[4];
        const int l1 = done + 1 + pc, gi1 = pbase + l1 * st;
        const bool out1 = mover && l1 <= lhi;
        if (out1 && !out) {
#pragma unroll
            for (int m = 0; m < 4; m++) old[m] = F.f[F_DQ2 + m][gi1];
        }
        if (work && c < len) {
            const int h = h0 + c;
            // at the half node: (u,v,w,T) by VALUE_line_half_virtual, the derivatives
            // along the own direction by DUVWT_half_line_virtual and along the two
            // others interpolated from node derivatives, the metrics
            // (kcx,etx,ctx,kcy,ety,cty,kcz,etz,ctz), volume and viscosities
            double uh[4], dh[12], kh[9], volh, v1h, v2h;
            auto set = [&](int f, double v) {  // staged quantity f (a constant): its value at the half node
                if (f < VS_DN) uh[f] = v;
                else if (f < VS_MET) {
                    const int g = (f - VS_DN) / 4, gd = g < dir ? g : g + 1;
                    dh[(f - VS_DN) % 4 + 4 * gd] = v;
                } else if (f < VS_VOL) kh[f - VS_MET] = v;
                else if (f == VS_VOL) volh = v;
                else if (f == VS_V1) v1h = v;
                else v2h = v;
            };
            auto at = [&](int p) { return smem + (wrap(hs + p + 1 - h0, RP) * NLP + ln) * VIS_PITCH; };
            auto at2 = [&](int p) { return (const double2 *)at(p); };
            if (n <= NIJK2ND) {
                double t[VIS_NF];
#pragma unroll 1
                for (int f = 0; f < VIS_NF; f++) {
                    auto Q = [&](int p) { return at(p)[f]; };
                    t[f] = f >= VS_MET ? value_half_node_at(Q, n, h) : f >= VS_DN ? value_half_node_ijk_at(Q, n, h) : 0.5 * (Q(h) + Q(h + 1));
                }
#pragma unroll
                for (int f = 0; f < VIS_NF; f++) set(f, t[f]);
#pragma unroll
                for (int m = 0; m < 4; m++) dh[m + 4 * dir] = at(h + 1)[m] - at(h)[m];
            } else {
                const bool left = h <= 1, near = left || h >= n - 1, end = h == 0 || h == n;
                const bool flag = near && (flags[ln] & (left ? 1 : 2));
                if (!flag) {  // u, v, w, T with the points around the half node
                    const double2 *qa = at2(h - 1), *qb = at2(h), *qc = at2(h + 1), *qd = at2(h + 2);
#pragma unroll
                    for (int q = 0; q < VS_DN / 2; q++) {
                        const double2 va = qa[q], vb = qb[q], vc = qc[q], vd = qd[q];
                        set(2 * q, (9.0 * (vb.x + vc.x) + -1.0 * (vd.x + va.x)) / 16.0);
                        set(2 * q + 1, (9.0 * (vb.y + vc.y) + -1.0 * (vd.y + va.y)) / 16.0);
                        dh[2 * q + 4 * dir] = div_by(27.0 * (vc.x - vb.x) + -1.0 * (vd.x - va.x), 24.0, 1.0 / 24.0);
                        dh[2 * q + 1 + 4 * dir] = div_by(27.0 * (vc.y - vb.y) + -1.0 * (vd.y - va.y), 24.0, 1.0 / 24.0);
                    }
                }
                if (!near) {
                    const double2 *qa = at2(h - 1), *qb = at2(h), *qc = at2(h + 1), *qd = at2(h + 2);
#pragma unroll
                    for (int q = VS_DN / 2; q < VIS_NF / 2; q++) {
                        const double2 va = qa[q], vb = qb[q], vc = qc[q], vd = qd[q];
                        set(2 * q, (9.0 * (vb.x + vc.x) + -1.0 * (vd.x + va.x)) / 16.0);
                        set(2 * q + 1, (9.0 * (vb.y + vc.y) + -1.0 * (vd.y + va.y)) / 16.0);
                    }
                } else {  // the other quantities have no ghost values: one-sided from the end's four points
                    const int e = left ? 1 : n, s1 = left ? 1 : -1;
                    const double *qa = at(e), *qb = at(e + s1), *qc = at(e + 2 * s1), *qd = at(e + 3 * s1);
                    const double ca = end ? 35.0 : 5.0, cb = end ? -35.0 : 15.0, cc = end ? 21.0 : -5.0, cd = end ? -5.0 : 1.0;
#pragma unroll
                    for (int f = VS_DN; f < VIS_NF; f++) set(f, (ca * qa[f] + cb * qb[f] + cc * qc[f] + cd * qd[f]) / 16.0);
                    if (flag) {
                        const double *qe = at(e + 4 * s1);
                        const double da = end ? -71.0 : -22.0, db = end ? 141.0 : 17.0, dc = end ? -93.0 : 9.0, dd = end ? 23.0 : -5.0;
#pragma unroll
                        for (int f = 0; f < VS_DN; f++) {
                            set(f, (ca * qa[f] + cb * qb[f] + cc * qc[f] + cd * qd[f]) / 16.0);
                            double d = da * qa[f] + db * qb[f] + dc * qc[f] + dd * qd[f];
                            if (!end) d = d + qe[f];
                            dh[f + 4 * dir] = div_by(left ? d : -d, 24.0, 1.0 / 24.0);
                        }
                    }
                }
            }
            // DUVWT_DXYZ
            const double rvol = 1.0 / volh;
            double dx[12];
#pragma unroll
            for (int m = 1; m <= 3; m++) {
                int m1 = m + m + m - 2, m2 = m1 + 1, m3 = m2 + 1;
                dx[m - 1] = div_by(kh[m1 - 1] * dh[0] + kh[m2 - 1] * dh[4] + kh[m3 - 1] * dh[8], volh, rvol);
                dx[m + 2] = div_by(kh[m1 - 1] * dh[1] + kh[m2 - 1] * dh[5] + kh[m3 - 1] * dh[9], volh, rvol);
                dx[m + 5] = div_by(kh[m1 - 1] * dh[2] + kh[m2 - 1] * dh[6] + kh[m3 - 1] * dh[10], volh, rvol);
                dx[m + 8] = div_by(kh[m1 - 1] * dh[3] + kh[m2 - 1] * dh[7] + kh[m3 - 1] * dh[11], volh, rvol);
            }
            // FLUX_VIS_LINE_new
            double vs = v1h;
            double vscc = vs * P.cc23;
            double dudx = dx[0], dudy = dx[1], dudz = dx[2];
            double dvdx = dx[3], dvdy = dx[4], dvdz = dx[5];
            double dwdx = dx[6], dwdy = dx[7], dwdz = dx[8];
            double t1 = vscc * (2.0 * dudx - dvdy - dwdz);
            double t5 = vscc * (2.0 * dvdy - dwdz - dudx);
            double t9 = vscc * (2.0 * dwdz - dudx - dvdy);
            double t2 = vs * (dudy + dvdx);
            double t3 = vs * (dudz + dwdx);
            double t6 = vs * (dvdz + dwdy);
            double kcp = v2h;
            const double nx = dir == 0 ? kh[0] : dir == 1 ? kh[1] : kh[2];
            const double ny = dir == 0 ? kh[3] : dir == 1 ? kh[4] : kh[5];
            const double nz = dir == 0 ? kh[6] : dir == 1 ? kh[7] : kh[8];
            double f1 = t1 * nx + t2 * ny + t3 * nz;
            double f2 = t2 * nx + t5 * ny + t6 * nz;
            double f3 = t3 * nx + t6 * ny + t9 * nz;
            double f4 = uh[0] * f1 + uh[1] * f2 + uh[2] * f3 + kcp * (dx[9] * nx + dx[10] * ny + dx[11] * nz);
            double2 *w = (double2 *)(fv + (wrap(fs + c, FR) * NLP + ln) * VIS_FP);
            w[0] = make_double2(f1, f2);  // the mass flux is zero
            w[1] = make_double2(f3, f4);
        }
        __syncthreads();
        if (have < n + 2) {
            int hi = h0 + len + C + 1;
            if (hi > n + 2) hi = n + 2;
            load(have + 1, hi, wrap(hs + have + 2 - h0, RP));
            have = hi;
        }
        // FLUX_DXYZ and dq -= re*dfv
        auto fslot = [&](int h) { return wrap(fs + h - h0 < 0 ? fs + h - h0 + FR : fs + h - h0, FR); };
        if (mover)
            for (int l = l1; l <= lhi; l += C) {
                const int gi = pbase + l * st;
                if (n > NIJK2ND && l > 2 && l < n - 1) {
                    double f[6][4];
#pragma unroll
                    for (int q = 0; q < 6; q++) {
                        const double2 *a = (const double2 *)(fv + (fslot(l - 3 + q) * NLP + pl) * VIS_FP);
                        const double2 x = a[0], y = a[1];
                        f[q][0] = x.x; f[q][1] = x.y; f[q][2] = y.x; f[q][3] = y.y;
                    }
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        const double dfv = div_by(2250.0 * (f[3][m] - f[2][m]) - 125.0 * (f[4][m] - f[1][m]) + 9.0 * (f[5][m] - f[0][m]),
                                                  1920.0, 1.0 / 1920.0);
                        if (out) out[(m + 1) * stride + gi] = P.re * dfv;
                        else F.f[F_DQ2 + m][gi] = (l == l1 ? old[m] : F.f[F_DQ2 + m][gi]) - P.re * dfv;
                    }
                } else {
#pragma unroll 1
                    for (int m = 0; m < 4; m++) {
                        const double *f = fv + pl * VIS_FP + m;
                        auto fa = [&](int hh) { return f[fslot(hh) * NLP * VIS_FP]; };
                        const double dfv = flux_dxyz_at(fa, n, l);
                        if (out) out[(m + 1) * stride + gi] = P.re * dfv;
                        else F.f[F_DQ2 + m][gi] = F.f[F_DQ2 + m][gi] - P.re * dfv;
                    }
                }
            }
        if (lhi == n) break;
        if (lhi > done) done = lhi;
        h0 += len;
        hs = wrap(hs + len, RP);
        fs = wrap(fs + len, FR);
        len = C;
    }
}

size_t rhs_vis_line_bytes(int dir, int n, int nl, int cmax) {
    return sizeof(double) * (size_t)vis_row(dir, nl) * (vis_ring(n, cmax) * VIS_PITCH + VIS_FP * (vis_chunk(n, cmax) + 5));
}
int rhs_vis_lines(int n, int cmax) { return std::min(VIS_MAX_LINES, VIS_THREADS / vis_chunk(n, cmax)); }
int rhs_vis_chunks(int n, int cmax) { return (n + vis_chunk(n, cmax)) / vis_chunk(n, cmax); }

void launch_rhs_vis(const LaunchCtx &c, int dir, cudaStream_t st, double *out) {
    if (c.mixed) return launch_rhs_vis_mx(c, dir, st, out);
    const DirTable &T = c.vis[dir];
    if (T.ngroups == 0) return;
    const long long stride = c.total;
    if (dir == 0) k_rhs_vis<0><<<T.ngroups, VIS_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, T.cmax, out, stride);
    else if (dir == 1) k_rhs_vis<1><<<T.ngroups, VIS_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, T.cmax, out, stride);
    else k_rhs_vis<2><<<T.ngroups, VIS_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, T.cmax, out, stride);
}

void setup_rhs_vis_attrs() {
    allow_all_smem(k_rhs_vis<0>);
    allow_all_smem(k_rhs_vis<1>);
    allow_all_smem(k_rhs_vis<2>);
}

}  // namespace wcns
