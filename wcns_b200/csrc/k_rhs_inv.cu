// k_rhs_inv.cu -- inviscid residual along one index direction.
//
// Restates r_h_s_invis (RHS.f90:35-72) -> invcode -> inviscd3d
// (Convect.f90:2-56, 58-649) with the WCNS-E-5 line scheme WCNS_E_5
// (WCNSE5.f90:2-206, nscheme=4), WCNS_E_5_41 (WCNSE5.f90:2087-2759,
// nscheme=41) or WCNS_E_5_42 (WCNSE5.f90:2766-3438, nscheme=42, the 41
// sections with second-order end states), Steger-Warming (flux.f90:2-77),
// Van Leer (flux.f90:395-501) or Roe (flux.f90:116-244) fluxes, and
// FLUX_DXYZ (WCNSE5.f90:209-254).  dq += dF.
//
// One CTA owns a group of NL lines of one block, staged in shared memory.  The
// reference's sequential line loop is split into two parallel phases:
//   A  per half node: the left state (weights centred at point h) and the right
//      state (point h+1), boundary closures, positivity fallback, numerical
//      flux; plus the 26 independent fluxes of the nscheme=41/42 boundary
//      sections, in lines that have one;
//   B  per point: sixth-order flux difference (or the boundary-section
//      difference where the reference overrides it) accumulated into dq.
//
// What bounds it: the FP64 operations of phase A and, before anything, their
// divisions (124 cycles each, a dozen instructions).  So
//   - the nonlinear weights are formed over a common denominator: with
//     E = (eps + IS)^2, w_k = C_k / E_k / sum(C / E) = C_k prod_{j != k} E_j / S,
//     one division per state instead of six.  E is between eps^2 = 1e-12 and
//     q^4, so the products stay far inside the exponent range;
//   - a half node's two states are formed by the thread that evaluates its
//     flux: the smoothness indicators are computed twice, but nothing of them
//     goes through shared memory and one barrier less separates the phases;
//   - a reciprocal whose last bit does not matter takes five instructions
//     (recip), a quotient that does, by a constant, three (div_by);
//   - the code of the few half nodes near a flagged end is kept out of the way
//     and in one copy for the five variables: unrolled it was as long as the
//     rest, and a quarter of the warps' time went into instruction fetches.
// Before, with a thread's states unrolled for every closure and six divisions
// each, the FP64 pipe was busy 25-37 % and the warps waited 5.4 cycles per
// instruction for code.  Measured per step, before and now: channel 3540 and
// 1500 us, 64 small blocks 1543 and 535 us, one block of 121x75x51 points (Roe)
// 347 and 190 us, the plate 265 and 148 us, one vortex 73 and 57 us.
// The central part of the fluxes and the differences keep the reference's
// operations and their order: where the flow is uniform they cancel to
// round-off, which is compared.  The weights, and in the Roe flux all that is
// multiplied by the jump, are free of that.
#include "wcns_dev.cuh"
#include "wcns_launch.h"

namespace wcns {

struct InvLine {
    const double *sq;  // shared-memory copy of the prim line: sq[m*(n+6) + l+2], l = -2..n+3
    const double *sk;  // shared-memory copy of the metrics (kx,ky,kz) of the line: sk[c*n + l-1], l = 1..n
    long long stride;
    long long dqbase;  // field index of point l=0 on the line (point l at dqbase + l*stride)
    int n, ist, ied;
};

__device__ __forceinline__ double qv(const InvLine &L, int m, int l) { return L.sq[m * (L.n + 6) + l + 2]; }

// 80 registers and 72 KB of staged lines per CTA, 24 warps per SM.  Against four
// CTAs of 256 threads at 64 registers: 1500 instead of 1544 us per step over the
// channel (24 blocks, 4.2 M points, Roe, nscheme 41), 535 instead of 513 us over
// 64 small blocks (0.9 M points), 57 instead of 63 us over a vortex of 65x33x17.
constexpr int INV_THREADS = 256, INV_CTAS = 3;
constexpr int INV_MAX_LINES = 32;  // lines per CTA (short lines are grouped many to a CTA)

// doubles of shared memory per line: prim 5 x (n+6), metrics 3 x n, f 5 x (n+1)
// and, with boundary sections, their 26 fluxes; padded to 2 mod 16 so that the
// lines of a group fall on different banks
__host__ __device__ inline int inv_line_stride(int n, bool sections) {
    int raw = 5 * (n + 6) + 3 * n + 5 * (n + 1) + (sections ? 130 : 0);
    return (raw + 13) / 16 * 16 + 2;
}

// The state at a half node from the five points around `c0` (WCNSE5.f90:2-206):
// left states from point h, right states from point h+1.
template <bool LEFT>
__device__ __forceinline__ double wcns_state(double m2, double m1, double c0, double p1, double p2) {
    const double EPS = 1.0e-6;
    const double g0 = 0.5 * (m2 - 4.0 * m1 + 3.0 * c0), g1 = 0.5 * (p1 - m1), g2 = 0.5 * (-3.0 * c0 + 4.0 * p1 - p2);
    const double s0 = m2 - 2.0 * m1 + c0, s1 = m1 - 2.0 * c0 + p1, s2 = c0 - 2.0 * p1 + p2;
    const double t0 = EPS + fma(g0, g0, s0 * s0), t1 = EPS + fma(g1, g1, s1 * s1), t2 = EPS + fma(g2, g2, s2 * s2);
    const double e0 = t0 * t0, e1 = t1 * t1, e2 = t2 * t2;
    const double four = LEFT ? 4.0 : -4.0;
    const double a0 = fma(four, g0, s0), a1 = fma(four, g1, s1), a2 = fma(four, g2, s2);
    // weights 1/16, 10/16, 5/16 (left), 5/16, 10/16, 1/16 (right)
    const double w0 = LEFT ? e1 * e2 : 5.0 * (e1 * e2), w1 = 10.0 * (e0 * e2), w2 = LEFT ? 5.0 * (e0 * e1) : e0 * e1;
    return c0 + 0.125 * (fma(w2, a2, fma(w1, a1, w0 * a0)) * recip(w0 + w1 + w2));
}

// Boundary-section states (left WCNSE5.f90:2284-2459, right 2524-2705, which
// count down from n with the same coefficients): four coefficients on the
// points 1..4 (or n..n-3), the divisor and its reciprocal.  nscheme=42 has
// second-order states at the first four half nodes (2967-2986, 3207-3226).
enum : int { SEC_S1 = 0, SEC_S1_42 = 4, SEC_S2 = 8, SEC_S2R2 = 13, SEC_S3L2 = 14, SEC_C = 15, SEC_ROWS = 18, SEC_W = 6 };
#define SEC_ROW(a, b, c, d, den) a, b, c, d, den, 1.0 / (den)
__constant__ double sec_table[SEC_ROWS * SEC_W] = {
    // s1 at half nodes 0..3, nscheme 41
    SEC_ROW(3.0, -1.0, 0.0, 0.0, 2.0), SEC_ROW(19.0, 25.0, -2.0, 0.0, 42.0), SEC_ROW(4.0, 3.0, 9.0, 2.0, 18.0), SEC_ROW(-2.0, 3.0, 3.0, 2.0, 6.0),
    // the same, nscheme 42
    SEC_ROW(677.0, -421.0, 99.0, 13.0, 368.0), SEC_ROW(5.0, 15.0, -5.0, 1.0, 16.0), SEC_ROW(-1.0, 9.0, 9.0, -1.0, 16.0), SEC_ROW(1.0, -5.0, 15.0, 5.0, 16.0),
    // s2 at half nodes 1..5 (left states at the left end, right ones at the right end)
    SEC_ROW(3.0, 6.0, -1.0, 0.0, 8.0), SEC_ROW(-30.0, 145.0, 29.0, -8.0, 136.0), SEC_ROW(0.0, -1.0, 6.0, 3.0, 8.0), SEC_ROW(0.0, 1.0, 2.0, 5.0, 8.0), SEC_ROW(0.0, 1.0, 1.0, 6.0, 8.0),
    // the other side's state of s2 at half node 2; s3 at half node 2
    SEC_ROW(2.0, 49.0, 125.0, -40.0, 136.0), SEC_ROW(-29.0, 170.0, 63.0, 12.0, 216.0),
    // the nscheme=4 closures at half nodes 0..2 of a flagged end (WCNSE5.f90:2-206)
    SEC_ROW(35.0, -35.0, 21.0, -5.0, 16.0), SEC_ROW(5.0, 15.0, -5.0, 1.0, 16.0), SEC_ROW(-1.0, 9.0, 9.0, -1.0, 16.0)};
#undef SEC_ROW

// state of variable m from a row: points 1..4, or n..n-3 for the right end
__device__ __forceinline__ double sec_state(const double *row, const double *q, int m, int n, bool right) {
    const double *x = q + m * (n + 6) + (right ? n + 2 : 3);
    const int d = right ? -1 : 1;
    return div_by(row[0] * x[0] + row[1] * x[d] + row[2] * x[2 * d] + row[3] * x[3 * d], row[4], row[5]);
}

// Where a half node's left state comes from near a flagged end: the row of its
// closure, -1 where the interior scheme stands (end: the end it counts from)
__device__ __forceinline__ int closure_left(const InvLine &L, int h, bool &end) {
    end = false;
    if (L.ist > 1 && h <= 2) return SEC_C + h;
    end = true;
    return L.ied < L.n && h >= L.n - 1 ? SEC_C + L.n - h : -1;
}
__device__ __forceinline__ int closure_right(const InvLine &L, int h, bool &end) {
    end = false;
    if (L.ist > 1 && h <= 1) return SEC_C + h;
    end = true;
    return L.ied < L.n && h >= L.n - 2 ? SEC_C + L.n - h : -1;
}

// dq += dF in place.
template <int dir, int NFLUX>
__global__ void __launch_bounds__(INV_THREADS, INV_CTAS) k_rhs_invis(DevParams P, DevFields F, const DevBlock *__restrict__ blocks,
                                                       const LineGroup *__restrict__ groups, int *err) {
    extern __shared__ double smem[];
    const LineGroup G = groups[blockIdx.x];
    const DevBlock B = blocks[G.blk];
    const int n = dimof(B, dir);
    const int H = n + 1, W = n + 6;
    const int NL = G.nl;
    const bool scheme4x = P.nscheme == 41 || P.nscheme == 42;
    const int LS = inv_line_stride(n, scheme4x);
    const int wf = 5 * W + 3 * n, wsec = wf + 5 * H;  // flux, section fluxes within a line
    __shared__ InvLine lines[INV_MAX_LINES];
    __shared__ int flagged;  // a line of the group has a boundary section
    __shared__ double sec[SEC_ROWS * SEC_W];
    if (threadIdx.x == 0) flagged = 0;
    if (threadIdx.x < SEC_ROWS * SEC_W) sec[threadIdx.x] = sec_table[threadIdx.x];
    __syncthreads();
    const int a1 = dir == 0 ? 1 : 0, a2 = dir == 2 ? 1 : 2;
    if (threadIdx.x < NL) {
        int c[3];
        c[a1] = G.a0 + threadIdx.x;
        c[a2] = G.b;
        c[dir] = -2;
        long long base = gidx(B, c[0], c[1], c[2]);
        InvLine L;
        L.sq = smem + (size_t)threadIdx.x * LS;
        L.sk = L.sq + (size_t)5 * W;
        L.stride = dstride(B, dir);
        L.dqbase = base + 2 * L.stride;
        L.n = n;
        L.ist = __ldg(F.f[F_R] + base) < SMALL ? 2 : 0;
        L.ied = __ldg(F.f[F_R] + base + (long long)(n + 5) * L.stride) < SMALL ? n - 2 : n;
        lines[threadIdx.x] = L;
        if (scheme4x && (L.ist > 1 || L.ied < n)) flagged = 1;
    }
    __syncthreads();
    constexpr bool posmajor = (dir == 0);
    const FastDiv dNL = fast_div_init(NL), dW = fast_div_init(W), dn = fast_div_init(n);
    // ---- stage the prim line (l = -2..n+3) and the metrics of this
    // direction (l = 1..n): one thread per (line, point), coalesced along the
    // line for i-lines and across the group's neighbouring lines otherwise
    for (int e = threadIdx.x; e < NL * W; e += blockDim.x) {
        const int qq = posmajor ? fdiv(e, dW) : fdiv(e, dNL);
        const int ln = posmajor ? qq : e - qq * NL;
        const int p = posmajor ? e - qq * W : qq;
        const long long gi = lines[ln].dqbase + (long long)(p - 2) * lines[ln].stride;
        double v[8];
#pragma unroll
        for (int m = 0; m < 5; m++) v[m] = __ldg(F.f[F_R + m] + gi);
        const bool inner = p >= 3 && p <= n + 2;
#pragma unroll
        for (int c = 0; c < 3; c++) v[5 + c] = inner ? __ldg(F.f[F_KCX + 3 * dir + c] + gi) : 0.0;
        double *sq = smem + (size_t)ln * LS;
#pragma unroll
        for (int m = 0; m < 5; m++) sq[m * W + p] = v[m];
        if (inner) {
#pragma unroll
            for (int c = 0; c < 3; c++) sq[5 * W + c * n + p - 3] = v[5 + c];
        }
    }
    __syncthreads();
    // Phase A walks the items line-fastest in every direction: the lanes of a
    // warp take the same position on neighbouring lines and follow one control
    // path, and items without work (boundary sections of a line that has none)
    // gather into whole warps that skip them.
    {
        const int NT = H + (flagged ? 26 : 0);
        const double gama1 = P.gama - 1.0, gama1_1 = 1.0 / gama1;
        int nbad = 0;
        for (int idx = threadIdx.x; idx < NL * NT; idx += blockDim.x) {
            const int t = fdiv(idx, dNL);
            const int ln = idx - t * NL;
            const InvLine &L = lines[ln];
            double ql[5], qr[5], fl[5];
            // Where the two states come from: a row of the table (and the end it
            // counts from) or, -1, the interior scheme.  Sections 0..25: at the
            // left end s1 at half nodes 0..3, s2 at 1..5, s3 at 1..4; at the right
            // end s4, s5, s6 likewise, counting down from n.
            int h = t, rowl = -1, rowr = -1;
            bool endl = false, endr = false;
            if (t >= H) {
                int sidx = t - H;
                const bool right = sidx >= 13;
                if (right ? L.ied >= n : L.ist <= 1) continue;
                if (right) sidx -= 13;
                const int s1 = P.nscheme == 42 ? SEC_S1_42 : SEC_S1;
                int o;  // half nodes from the end
                if (sidx < 4) {
                    o = sidx;
                    rowl = rowr = s1 + o;
                } else if (sidx < 9) {
                    o = sidx - 3;
                    rowl = SEC_S2 + o - 1;
                    rowr = o == 2 ? SEC_S2R2 : rowl;
                } else {
                    o = sidx - 8;
                    rowl = o == 2 ? SEC_S3L2 : SEC_S2 + o - 1;
                }
                h = o;
                if (right) {
                    h = n - o;
                    const int x = rowl;
                    rowl = rowr;
                    rowr = x;
                    endl = endr = true;
                    // s6: the left state as the left sections left it where they
                    // ran (h <= 5), otherwise the interior scheme's
                    if (sidx >= 9 && L.ist > 1 && h <= 5) {
                        endl = false;
                        rowl = h == 0 ? s1 : h == 2 ? SEC_S3L2 : SEC_S2 + h - 1;
                    }
                }
            }
            if (rowl < 0) rowl = closure_left(L, h, endl);
            if (rowr < 0) rowr = closure_right(L, h, endr);
            if (rowl < 0 && rowr < 0) {
#pragma unroll
                for (int m = 0; m < 5; m++) {
                    const double *q = L.sq + m * W + h + 2;
                    const double q0 = q[-2], q1 = q[-1], q2 = q[0], q3 = q[1], q4 = q[2], q5 = q[3];
                    ql[m] = wcns_state<true>(q0, q1, q2, q3, q4);
                    qr[m] = wcns_state<false>(q1, q2, q3, q4, q5);
                }
            } else {  // few items: one copy of the code for all variables
                double tl[5], tr[5];
#pragma unroll 1
                for (int m = 0; m < 5; m++) {
                    const double *q = L.sq + m * W + h + 2;
                    tl[m] = rowl < 0 ? wcns_state<true>(q[-2], q[-1], q[0], q[1], q[2]) : sec_state(sec + rowl * SEC_W, L.sq, m, n, endl);
                    tr[m] = rowr < 0 ? wcns_state<false>(q[-1], q[0], q[1], q[2], q[3]) : sec_state(sec + rowr * SEC_W, L.sq, m, n, endr);
                }
#pragma unroll
                for (int m = 0; m < 5; m++) { ql[m] = tl[m]; qr[m] = tr[m]; }
            }
            // positivity fallback: the neighbouring point; in s1 and s4 means
            const bool badl = ql[0] <= RMIN_LIMIT || ql[4] <= PMIN_LIMIT, badr = qr[0] <= RMIN_LIMIT || qr[4] <= PMIN_LIMIT;
            const bool same = t >= H && rowl == rowr && rowl < SEC_S2;
            if (badl || badr) {
                const int ia = h > 1 ? h : 1, ib = h + 1 < n ? h + 1 : n;
                // points of the means; of the neighbours
                const int la = same && endl ? 1 : ia, lb = same ? (endl ? h : h + 1) : ia, ra = same ? la : ib, rb = same ? lb : ib;
#pragma unroll
                for (int m = 0; m < 5; m++) {
                    if (badl) ql[m] = (qv(L, m, la) + qv(L, m, lb)) / 2.0;
                    if (badr) qr[m] = (qv(L, m, ra) + qv(L, m, rb)) / 2.0;
                }
            }
            // half-node metrics: VALUE_HALF_NODE of (kx,ky,kz) along the line
            auto ax = [&](int l) { return L.sk[l - 1]; };
            auto ay = [&](int l) { return L.sk[n + l - 1]; };
            auto az = [&](int l) { return L.sk[2 * n + l - 1]; };
            double kx = value_half_node_at(ax, n, h), ky = value_half_node_at(ay, n, h), kz = value_half_node_at(az, n, h);
            const double kt = 0.0;  // kct=0, so every half-node value of kt is +0
            if (NFLUX == 3) nbad += flux_roe(P, gama1_1, ql, qr, kx, ky, kz, kt, same, fl);
            else nbad += flux_split<NFLUX>(P, ql, qr, kx, ky, kz, kt, fl);
            double *f_ = smem + (size_t)ln * LS;
            if (t < H) {
                f_ += wf + h;
#pragma unroll
                for (int m = 0; m < 5; m++) f_[m * H] = fl[m];
            } else {
                f_ += wsec + (t - H) * 5;
#pragma unroll
                for (int m = 0; m < 5; m++) f_[m] = fl[m];
            }
        }
        if (nbad) atomicAdd(&err[ERR_ROE], nbad);
    }
    __syncthreads();
    // ---- phase B: flux difference and accumulation into dq, per (line, point),
    // in the order of memory: along the line for i-lines, across the
    // neighbouring lines otherwise
    for (int idx = threadIdx.x; idx < NL * n; idx += blockDim.x) {
        const int qq = posmajor ? fdiv(idx, dn) : fdiv(idx, dNL);
        const int ln = posmajor ? qq : idx - qq * NL;
        const int l = 1 + (posmajor ? idx - qq * n : qq);
        const InvLine &L = lines[ln];
        const long long gi = L.dqbase + (long long)l * L.stride;
        const double *f_ = smem + (size_t)ln * LS + wf;
        const double *sc = smem + (size_t)ln * LS + wsec;
        const bool right = scheme4x && L.ied < n && l >= n - 2, left = scheme4x && L.ist > 1 && l <= 3;
        if (!right && !left && l > 2 && l < n - 1) {
            double old[5];
#pragma unroll
            for (int m = 0; m < 5; m++) old[m] = F.f[F_DQ1 + m][gi];
#pragma unroll
            for (int m = 0; m < 5; m++) {
                const double *f = f_ + m * H + l;
                F.f[F_DQ1 + m][gi] = old[m] + div_by(2250.0 * (f[0] - f[-1]) - 125.0 * (f[1] - f[-2]) + 9.0 * (f[2] - f[-3]), 1920.0, 1.0 / 1920.0);
            }
            continue;
        }
#pragma unroll 1
        for (int m = 0; m < 5; m++) {
            double df;
            if (right) {
                const double *s4 = sc + 13 * 5 + m, *s5 = sc + 17 * 5 + m, *s6 = sc + 22 * 5 + m;
                // section fluxes f(ni-h): s4[k] holds f(k), s5[k] and s6[k] hold f(k+1)
                if (l == n) df = -(-23.0 * s4[0] + 21.0 * s4[5] + 3.0 * s4[10] - 1.0 * s4[15]) / 24.0;
                else if (l == n - 1) df = -(-22.0 * s5[0] + 17.0 * s5[5] + 9.0 * s5[10] - 5.0 * s5[15] + s5[20]) / 24.0;
                else df = -(s6[0] - 27.0 * s6[5] + 27.0 * s6[10] - s6[15]) / 24.0;
            } else if (left) {
                const double *s1 = sc + m, *s2 = sc + 4 * 5 + m, *s3 = sc + 9 * 5 + m;
                if (l == 1) df = (-23.0 * s1[0] + 21.0 * s1[5] + 3.0 * s1[10] - 1.0 * s1[15]) / 24.0;
                else if (l == 2) df = (-22.0 * s2[0] + 17.0 * s2[5] + 9.0 * s2[10] - 5.0 * s2[15] + s2[20]) / 24.0;
                else df = (s3[0] - 27.0 * s3[5] + 27.0 * s3[10] - s3[15]) / 24.0;
            } else {
                auto fa = [&](int hh) { return f_[m * H + hh]; };
                df = flux_dxyz_at(fa, n, l);
            }
            F.f[F_DQ1 + m][gi] = F.f[F_DQ1 + m][gi] + df;
        }
    }
}

template <int NFLUX>
static void launch_invis(const LaunchCtx &c, int dir, cudaStream_t st) {
    const DirTable &T = c.inv[dir];
    if (dir == 0) k_rhs_invis<0, NFLUX><<<T.ngroups, INV_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, c.err);
    else if (dir == 1) k_rhs_invis<1, NFLUX><<<T.ngroups, INV_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, c.err);
    else k_rhs_invis<2, NFLUX><<<T.ngroups, INV_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, c.err);
}

void launch_rhs_invis(const LaunchCtx &c, int dir, cudaStream_t st, double *out) {
    if (c.mixed) return launch_rhs_invis_mx(c, dir, st, out);
    if (c.inv[dir].ngroups == 0) return;
    if (c.P->nflux == 1) launch_invis<1>(c, dir, st);
    else if (c.P->nflux == 2) launch_invis<2>(c, dir, st);
    else launch_invis<3>(c, dir, st);
}

template <int NFLUX>
static void set_invis_attrs(int max_smem) {
    cudaFuncSetAttribute(k_rhs_invis<0, NFLUX>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
    cudaFuncSetAttribute(k_rhs_invis<1, NFLUX>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
    cudaFuncSetAttribute(k_rhs_invis<2, NFLUX>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem);
}

void setup_rhs_invis_attrs(size_t max_smem, int nflux) {
    if (nflux == 1) set_invis_attrs<1>((int)max_smem);
    else if (nflux == 2) set_invis_attrs<2>((int)max_smem);
    else set_invis_attrs<3>((int)max_smem);
}

size_t rhs_invis_line_bytes(int n, bool sections) { return (size_t)inv_line_stride(n, sections) * 8; }
int rhs_invis_threads() { return INV_THREADS; }
size_t rhs_invis_smem() { return (size_t)(216 * 1024 / INV_CTAS); }
int rhs_invis_max_lines() { return INV_MAX_LINES; }

}  // namespace wcns
