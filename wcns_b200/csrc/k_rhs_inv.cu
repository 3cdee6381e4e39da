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
// One CTA marches along a group of NL lines of one block, C half nodes at a time
// (cmax in wcns_launch.h), over a ring of points in shared memory.  Per chunk:
//   A  per half node: the left state (weights centred at point h) and the right
//      state (point h+1), boundary closures, positivity fallback, numerical
//      flux; at a flagged end also the 13 independent fluxes of the
//      nscheme=41/42 boundary sections;
//   B  per point: sixth-order flux difference (or the boundary-section
//      difference where the reference overrides it) accumulated into dq, while
//      the next points arrive (asynchronous copies).
//
// What bounds it: the FP64 operations of phase A (the pipe is busy half of the
// time), and the latency around them.  So
//   - the nonlinear weights are formed over a common denominator: with
//     E = (eps + IS)^2, w_k = C_k / E_k / sum(C / E) = C_k prod_{j != k} E_j / S,
//     one division per state instead of six (124 cycles each, a dozen
//     instructions).  E is between eps^2 = 1e-12 and q^4, so the products stay inside
//     the exponent range while q is below 1e37 (beyond, see the end);
//   - a half node's two states are formed by the thread that evaluates its
//     flux: the smoothness indicators are computed twice, but nothing of them
//     goes through shared memory;
//   - a reciprocal whose last bit does not matter takes five instructions
//     (recip), a quotient that does, by a constant, six (div_by);
//   - the code of the few half nodes near a flagged end is kept out of the way
//     and in one copy for the five variables: unrolled it was as long as the
//     rest, and a quarter of the warps' time went into instruction fetches;
//   - whole lines in shared memory leave room for three to seven of them, loads
//     across the lines then fetch twice the bytes they use, and staging,
//     arithmetic and stores follow one another; a ring of a chunk and its halo
//     leaves room for 16 lines.
// Measured per step, with the closures unrolled and whole lines; the code above on
// whole lines; now, chunk lengths as build_line_tables picks them: channel (24 blocks,
// 4.2 M points, Roe, nscheme 41) 3540, 1511, 1152 us; 64 small blocks (0.9 M points)
// 1543, 539, 472; one block of 121x75x51 points (nscheme 4) 347, 190, 171; the plate
// (0.23 M points) 265, 148, 118; one vortex of 65x33x17 73, 57, 46.  Three, five, six
// CTAs per SM over the channel, where four took 1135: 1228, 1216, 1323 us; two of 256
// threads with C = 16 1300.
// The central part of the fluxes and the differences keep the reference's
// operations and their order: where the flow is uniform they cancel to
// round-off, which is compared.  The weights, and in the Roe flux all that is
// multiplied by the jump, are free of that.  Where a sum of weights, a sound speed or a
// Roe flux leaves the range of the short forms, the CTA ends its march and does the rest
// of its lines with the reference's divisions (inv_rest), so that special values reach
// the residual as they do in the reference.  The checks take 0.5 % (channel 1148 to
// 1154 us); a branch to the divisions in the loop took 6 % there and 9 % on 64 small
// blocks, a call for the chunk 17 %, by the registers they hold.  A state that is
// undefined everywhere takes 1.5 ms where the channel of 0.5 M points takes 0.24.
#include <algorithm>

#include "wcns_dev.cuh"
#include "wcns_launch.h"

namespace wcns {

// The ring: the five variables of the points h0-2 .. h0+C+2 and, at 1..n, the
// metrics of this direction, one point's eight values after the other.
constexpr int INV_PITCH = 10, INV_FP = 6;
constexpr int INV_THREADS = 128, INV_CTAS = 4;
constexpr int INV_MAX_LINES = 32;  // lines per CTA

// A line of n points has n+1 half nodes in nch chunks of C; the first one takes the
// remainder, so that all that the right end's formulas reach lies in the last chunk's
// points.  Short lines are one chunk: both ends' sections reach the other end there.
__host__ __device__ inline int inv_chunk(int n, int cmax) {
    const int H = n + 1;
    if (H <= 13) return H;
    const int nch = (H + cmax - 1) / cmax;
    return (H + nch - 1) / nch;
}
// lanes of a row of the ring: odd for i-lines, whose loads walk along a line
__host__ __device__ inline int inv_row(int dir, int nl) { return dir == 0 ? nl | 1 : nl; }

struct InvLine {  // one line's view of the ring
    const double *ring;  // point p at slot wrap(s0 + p - p0), NLP * INV_PITCH apart
    int p0, s0, RP, step;
    int n, ist, ied;
    __device__ __forceinline__ const double *at(int p) const {
        int s = s0 + p - p0;
        if (s >= RP) s -= RP;
        return ring + s * step;
    }
};

// The state at a half node from the five points around `c0` (WCNSE5.f90:2-206):
// left states from point h, right states from point h+1.  top: the largest sum of
// weights so far (its high word; NaN above all numbers).  From TOP_WEIGHT, 1e300, on
// the products and the reciprocal may leave the range.
constexpr unsigned TOP_WEIGHT = 0x7e37e43cu;
template <bool LEFT>
__device__ __forceinline__ double wcns_state(double m2, double m1, double c0, double p1, double p2, unsigned &top) {
    const double EPS = 1.0e-6;
    const double g0 = 0.5 * (m2 - 4.0 * m1 + 3.0 * c0), g1 = 0.5 * (p1 - m1), g2 = 0.5 * (-3.0 * c0 + 4.0 * p1 - p2);
    const double s0 = m2 - 2.0 * m1 + c0, s1 = m1 - 2.0 * c0 + p1, s2 = c0 - 2.0 * p1 + p2;
    const double t0 = EPS + fma(g0, g0, s0 * s0), t1 = EPS + fma(g1, g1, s1 * s1), t2 = EPS + fma(g2, g2, s2 * s2);
    const double e0 = t0 * t0, e1 = t1 * t1, e2 = t2 * t2;
    const double four = LEFT ? 4.0 : -4.0;
    const double a0 = fma(four, g0, s0), a1 = fma(four, g1, s1), a2 = fma(four, g2, s2);
    // weights 1/16, 10/16, 5/16 (left), 5/16, 10/16, 1/16 (right)
    const double w0 = LEFT ? e1 * e2 : 5.0 * (e1 * e2), w1 = 10.0 * (e0 * e2), w2 = LEFT ? 5.0 * (e0 * e1) : e0 * e1;
    const double sum = w0 + w1 + w2;
    top = max(top, (unsigned)__double2hiint(sum));
    return c0 + 0.125 * (fma(w2, a2, fma(w1, a1, w0 * a0)) * recip(sum));
}
// The same with the reference's divisions, which overflow at far larger values and
// pass infinities on.
template <bool LEFT>
__device__ __forceinline__ double wcns_state_div(double m2, double m1, double c0, double p1, double p2) {
    const double g[3] = {0.5 * (m2 - 4.0 * m1 + 3.0 * c0), 0.5 * (p1 - m1), 0.5 * (-3.0 * c0 + 4.0 * p1 - p2)};
    const double s[3] = {m2 - 2.0 * m1 + c0, m1 - 2.0 * c0 + p1, c0 - 2.0 * p1 + p2};
    const double cl[3] = {1.0 / 16.0, 10.0 / 16.0, 5.0 / 16.0}, four = LEFT ? 4.0 : -4.0;
    double b[3], a = 0.0;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double t = 1.0e-6 + (g[k] * g[k] + s[k] * s[k]);
        b[k] = cl[LEFT ? k : 2 - k] / (t * t);
    }
    const double sum = b[0] + b[1] + b[2];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const double x = b[k] / sum * (s[k] + four * g[k]);
        a = k ? a + x : x;
    }
    return c0 + 0.125 * a;
}

// Boundary-section states (left WCNSE5.f90:2284-2459, right 2524-2705, which
// count down from n with the same coefficients): four coefficients on the
// points 1..4 (or n..n-3), the divisor and its reciprocal.  nscheme=42 has
// second-order states at the first four half nodes (2967-2986, 3207-3226).
enum : int { SEC_S1 = 0, SEC_S1_42 = 4, SEC_S2 = 8, SEC_S2R2 = 13, SEC_S3L2 = 14, SEC_C = 15, SEC_ROWS = 18, SEC_W = 6 };
// A coefficient 0.0 stands for a point that the reference's formula has not, -0.0 for
// its explicit product with zero.
#define SEC_ROW(a, b, c, d, den) a, b, c, d, den, 1.0 / (den)
__constant__ double sec_table[SEC_ROWS * SEC_W] = {
    // s1 at half nodes 0..3, nscheme 41
    SEC_ROW(3.0, -1.0, -0.0, 0.0, 2.0), SEC_ROW(19.0, 25.0, -2.0, 0.0, 42.0), SEC_ROW(4.0, 3.0, 9.0, 2.0, 18.0), SEC_ROW(-2.0, 3.0, 3.0, 2.0, 6.0),
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
__device__ __forceinline__ double sec_state(const double *row, const InvLine &L, int m, bool right) {
    const int e = right ? L.n : 1, d = right ? -1 : 1;
    return div_by(row[0] * L.at(e)[m] + row[1] * L.at(e + d)[m] + row[2] * L.at(e + 2 * d)[m] + row[3] * L.at(e + 3 * d)[m], row[4], row[5]);
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

// Where an item's two states come from: a row of the table and the end it counts from
// or, -1, the interior scheme and its closures.  Item: a half node (sec < 0), or a flux
// of the ends' sections.  Sections 0..25: at the left end s1 at half nodes 0..3, s2 at
// 1..5, s3 at 1..4; at the right end s4, s5, s6 likewise, counting down from n.
struct InvItem {
    int h, isec, rowl, rowr;
    bool endl, endr;
    // false: the line has no section there
    __device__ __forceinline__ bool set(int nscheme, const InvLine &L, int half, int sec) {
        h = half;
        isec = sec;
        rowl = rowr = -1;
        endl = endr = false;
        if (sec < 0) return true;
        const bool right = sec >= 13;
        if (right ? L.ied >= L.n : L.ist <= 1) return false;
        const int q = right ? sec - 13 : sec, s1 = nscheme == 42 ? SEC_S1_42 : SEC_S1;
        int o;  // half nodes from the end
        if (q < 4) {
            o = q;
            rowl = rowr = s1 + o;
        } else if (q < 9) {
            o = q - 3;
            rowl = SEC_S2 + o - 1;
            rowr = o == 2 ? SEC_S2R2 : rowl;
        } else {
            o = q - 8;
            rowl = o == 2 ? SEC_S3L2 : SEC_S2 + o - 1;
        }
        h = o;
        if (right) {
            h = L.n - o;
            const int x = rowl;
            rowl = rowr;
            rowr = x;
            endl = endr = true;
            // s6: the left state as the left sections left it where they
            // ran (h <= 5), otherwise the interior scheme's
            if (q >= 9 && L.ist > 1 && h <= 5) {
                endl = false;
                rowl = h == 0 ? s1 : h == 2 ? SEC_S3L2 : SEC_S2 + h - 1;
            }
        }
        return true;
    }
};

__device__ __forceinline__ void inv_copy8(double *dst, const double *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

// The difference at the o-th point from a flagged end, of one component of the line's
// section fluxes.  s1, s4 hold f(k) and s2, s3, s5, s6 f(k + 1), k half nodes from the end.
__device__ __forceinline__ double section_difference(const double *s, bool right, int o) {
    if (right) s += 13 * 5;
    const double *a = s, *b = s + 4 * 5, *c = s + 9 * 5;
    const double d = o == 0 ? -23.0 * a[0] + 21.0 * a[5] + 3.0 * a[10] - 1.0 * a[15]
                   : o == 1 ? -22.0 * b[0] + 17.0 * b[5] + 9.0 * b[10] - 5.0 * b[15] + b[20] : c[0] - 27.0 * c[5] + 27.0 * c[10] - c[15];
    return (right ? -d : d) / 24.0;
}

// The points done+1..n of a group's lines with the reference's divisions, from memory: C
// points at a time, their half nodes' fluxes in `fr` (C + 5 per line), the sections'
// in `secf`.  Called by all threads of the CTA when nothing of the march is needed any
// more, so that it costs the march no registers.  Returns the thread's c^2 failures at
// the half nodes from h0 on (and the sections after it), each counted once.
template <int dir, int NFLUX>
__device__ __noinline__ int inv_rest(const DevParams *P, const DevFields *F, const DevBlock *B, const LineGroup *G, int done, int h0, int C, double *fr,
                                     double *secf, const double *sec) {
    const int n = dimof(*B, dir), NL = G->nl, st = (int)dstride(*B, dir);
    constexpr int a1 = dir == 0 ? 1 : 0, a2 = dir == 2 ? 1 : 2;
    const int lstep = (int)dstride(*B, a1);
    int o3[3];
    o3[a1] = G->a0;
    o3[a2] = G->b;
    o3[dir] = 0;
    const int base = (int)gidx(*B, o3[0], o3[1], o3[2]);
    const bool scheme4x = P->nscheme == 41 || P->nscheme == 42;
    int bad = 0, hc = h0;  // half nodes below hc have been counted
    auto line = [&](int ln) {
        InvLine L;
        L.n = n;
        const double *rho = F->f[F_R] + base + ln * lstep;
        L.ist = rho[-2 * st] < SMALL ? 2 : 0;
        L.ied = rho[(n + 3) * st] < SMALL ? n - 2 : n;
        return L;
    };
    // one item's flux
    auto item = [&](int ln, int half, int isec, double *f) {
        const InvLine L = line(ln);
        InvItem I;
        if (!I.set(P->nscheme, L, half, isec)) return;
        const int h = I.h, g = base + ln * lstep;
        auto q = [&](int m, int p) { return F->f[F_R + m][g + p * st]; };
        if (I.rowl < 0) I.rowl = closure_left(L, h, I.endl);
        if (I.rowr < 0) I.rowr = closure_right(L, h, I.endr);
        auto row = [&](int rw, int m, bool right) {  // a row's state, of the points that its formula has
            const double *c = sec + rw * SEC_W;
            double a = -0.0;
            for (int k = 0; k < 4; k++)
                if (__double_as_longlong(c[k]) != 0) a = a + c[k] * q(m, right ? n - k : 1 + k);
            return a / c[4];
        };
        double ql[5], qr[5], fl[5];
#pragma unroll
        for (int m = 0; m < 5; m++) {
            ql[m] = I.rowl >= 0 ? row(I.rowl, m, I.endl) : wcns_state_div<true>(q(m, h - 2), q(m, h - 1), q(m, h), q(m, h + 1), q(m, h + 2));
            qr[m] = I.rowr >= 0 ? row(I.rowr, m, I.endr) : wcns_state_div<false>(q(m, h - 1), q(m, h), q(m, h + 1), q(m, h + 2), q(m, h + 3));
        }
        const bool badl = ql[0] <= RMIN_LIMIT || ql[4] <= PMIN_LIMIT, badr = qr[0] <= RMIN_LIMIT || qr[4] <= PMIN_LIMIT;
        const bool same = isec >= 0 && I.rowl == I.rowr && I.rowl < SEC_S2;
        const int ia = h > 1 ? h : 1, ib = h + 1 < n ? h + 1 : n;
        const int la = same && I.endl ? 1 : ia, lb = same ? (I.endl ? h : h + 1) : ia, ra = same ? la : ib, rb = same ? lb : ib;
#pragma unroll
        for (int m = 0; m < 5; m++) {
            if (badl) ql[m] = (q(m, la) + q(m, lb)) / 2.0;
            if (badr) qr[m] = (q(m, ra) + q(m, rb)) / 2.0;
        }
        double k[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            auto a = [&](int p) { return F->f[F_KCX + 3 * dir + d][g + p * st]; };
            k[d] = value_half_node_at(a, n, h);
        }
        const int b = NFLUX == 3 ? flux_roe_div(P->gama, P->efix, k[0], k[1], k[2], ql, qr, fl)
                                 : flux_split<NFLUX>(*P, ql, qr, k[0], k[1], k[2], 0.0, fl);
        if (isec < 0 ? h >= hc : isec >= 13 || h0 == 0) bad += b;
#pragma unroll
        for (int m = 0; m < 5; m++) f[m] = fl[m];
    };
    __syncthreads();
    if (scheme4x)
        for (int e = threadIdx.x; e < 26 * NL; e += INV_THREADS) item(e % NL, 0, e / NL, secf + (e % NL * 26 + e / NL) * 5);
    for (int l0 = done + 1; l0 <= n; l0 += C) {
        const int l1 = l0 + C - 1 < n ? l0 + C - 1 : n;
        // the half nodes of these points' differences: l-3..l+2, 0..4 and n-4..n at the ends
        const int ha = max(0, min(l0 - 3, n - 4)), hb = min(n, max(l1 + 2, 4));
        __syncthreads();
        for (int e = threadIdx.x; e < (hb - ha + 1) * NL; e += INV_THREADS) item(e % NL, ha + e / NL, -1, fr + e * 5);
        hc = max(hc, hb + 1);
        __syncthreads();
        for (int e = threadIdx.x; e < (l1 - l0 + 1) * NL; e += INV_THREADS) {
            const int ln = e % NL, l = l0 + e / NL, gi = base + ln * lstep + l * st;
            const InvLine L = line(ln);
            const int end = !scheme4x ? 0 : L.ied < n && l >= n - 2 ? 2 : L.ist > 1 && l <= 3 ? 1 : 0;
            for (int m = 0; m < 5; m++) {
                auto fa = [&](int hh) { return fr[((hh - ha) * NL + ln) * 5 + m]; };
                const double v = end ? section_difference(secf + ln * 130 + m, end == 2, end == 2 ? n - l : l - 1) : flux_dxyz_at(fa, n, l);
                F->f[F_DQ1 + m][gi] = F->f[F_DQ1 + m][gi] + v;
            }
        }
    }
    return bad;
}

// dq += dF in place.
template <int dir, int NFLUX>
__global__ void __launch_bounds__(INV_THREADS, INV_CTAS) k_rhs_invis(const __grid_constant__ DevParams P, const __grid_constant__ DevFields F, const DevBlock *__restrict__ blocks,
                                                       const LineGroup *__restrict__ groups, int cmax, int *err) {
    extern __shared__ __align__(16) double smem[];
    const LineGroup G = groups[blockIdx.x];
    const DevBlock B = blocks[G.blk];
    const int n = dimof(B, dir), NL = G.nl, NLP = inv_row(dir, NL);
    const int H = n + 1, C = inv_chunk(n, cmax), RP = C + 5, FR = C + 5;
    const bool scheme4x = P.nscheme == 41 || P.nscheme == 42;
    double *fr = smem + RP * NLP * INV_PITCH;   // the last FR half nodes' fluxes
    double *secf = fr + FR * NLP * INV_FP;      // 26 section fluxes per line
    __shared__ int flags[INV_MAX_LINES];        // bit 0: the left end has a boundary, bit 1: the right end
    __shared__ double sec[SEC_ROWS * SEC_W];
    if (threadIdx.x < SEC_ROWS * SEC_W) sec[threadIdx.x] = sec_table[threadIdx.x];
    static_assert(SEC_ROWS * SEC_W <= INV_THREADS, "the table is copied in one go");
    constexpr int a1 = dir == 0 ? 1 : 0, a2 = dir == 2 ? 1 : 2;
    const int st = (int)dstride(B, dir), lstep = (int)dstride(B, a1);
    int o3[3];
    o3[a1] = G.a0;
    o3[a2] = G.b;
    o3[dir] = 0;
    const int base = (int)gidx(B, o3[0], o3[1], o3[2]);  // position 0 of the first line
    // this thread's half node and line; its point and line in the loads and stores,
    // which walk along the line for i-lines and across the lines otherwise
    const int TC = INV_THREADS / NL, c = threadIdx.x / NL, ln = threadIdx.x - c * NL;
    const int pc = dir == 0 ? threadIdx.x % C : c, pl = dir == 0 ? threadIdx.x / C : ln;
    const bool mover = dir == 0 ? pl < NL : c < C;
    const int pbase = base + pl * lstep;
    auto wrap = [](int x, int m) { return x >= m ? x - m : x; };
    auto load = [&](int lo, int hi, int slo) {  // points lo..hi into the ring, from slot slo on
        if (mover)
            for (int p = lo + pc; p <= hi; p += C) {
                const int gi = pbase + p * st;
                double *S = smem + (wrap(slo + p - lo, RP) * NLP + pl) * INV_PITCH;
#pragma unroll
                for (int m = 0; m < 5; m++) inv_copy8(S + m, F.f[F_R + m] + gi);
                if (p >= 1 && p <= n) {
#pragma unroll
                    for (int q = 0; q < 3; q++) inv_copy8(S + 5 + q, F.f[F_KCX + 3 * dir + q] + gi);
                }
            }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    int h0 = 0, len = H - (H - 1) / C * C;  // this chunk's half nodes h0 .. h0+len-1
    int have = len + 2 < 7 ? 7 : len + 2;   // the last point loaded: the left end's sections reach point 7
    if (have > n + 3) have = n + 3;
    int hs = 0, fs = 0;                     // slots of point h0-2 and of half node h0
    int done = 0;                           // the last point whose difference is out
    load(-2, have, 0);
    int anyl = 0, anyr = 0;                 // a line has a boundary section at its left, right end
    if ((int)threadIdx.x < NL) {
        const int g = base + threadIdx.x * lstep;
        anyl = __ldg(F.f[F_R] + g - 2 * st) < SMALL;
        anyr = __ldg(F.f[F_R] + g + (n + 3) * st) < SMALL;
        flags[threadIdx.x] = anyl | anyr << 1;
    }
    anyl = __syncthreads_or(scheme4x && anyl);
    anyr = __syncthreads_or(scheme4x && anyr);
    const double gama1 = P.gama - 1.0, gama1_1 = 1.0 / gama1;
    int nbad = 0;
    bool rest = false;
    InvLine L;
    L.ring = smem + ln * INV_PITCH;
    L.RP = RP;
    L.step = NLP * INV_PITCH;
    L.n = n;
    L.ist = flags[ln] & 1 ? 2 : 0;
    L.ied = flags[ln] & 2 ? n - 2 : n;
    for (;;) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        const bool last = h0 + len == H;
        const int lhi = last ? n : h0 + len - 3;  // differences this chunk completes: done+1 .. lhi
        // the old residual of this thread's point, ahead of the barrier
        double old[5];
        const int l1 = done + 1 + pc, gi1 = pbase + l1 * st;
        if (mover && l1 <= lhi) {
#pragma unroll
            for (int m = 0; m < 5; m++) old[m] = F.f[F_DQ1 + m][gi1];
        }
        L.p0 = h0 - 2;
        L.s0 = hs;
        // the half nodes, then the sections of the ends in the chunk: items
        // line-fastest, the lanes of a warp take the same position on neighbouring
        // lines and follow one control path
        const int nl13 = h0 == 0 && anyl ? 13 : 0, T = len + nl13 + (last && anyr ? 13 : 0);
        bool odd = false;  // an item left the range of the short forms
        int bad = 0;
        for (int t = c; t < T && c < TC; t += TC) {
            double ql[5], qr[5], fl[5];
            InvItem I;
            if (!I.set(P.nscheme, L, h0 + t, t < len ? -1 : t - len + (nl13 ? 0 : 13))) continue;
            const int h = I.h, isec = I.isec;
            int rowl = I.rowl, rowr = I.rowr;
            bool endl = I.endl, endr = I.endr;
            if (rowl < 0) rowl = closure_left(L, h, endl);
            if (rowr < 0) rowr = closure_right(L, h, endr);
            const double *x0 = L.at(h - 2), *x1 = L.at(h - 1), *x2 = L.at(h), *x3 = L.at(h + 1), *x4 = L.at(h + 2), *x5 = L.at(h + 3);
            unsigned top = 0;
            if (rowl < 0 && rowr < 0) {
#pragma unroll
                for (int m = 0; m < 5; m++) {
                    ql[m] = wcns_state<true>(x0[m], x1[m], x2[m], x3[m], x4[m], top);
                    qr[m] = wcns_state<false>(x1[m], x2[m], x3[m], x4[m], x5[m], top);
                }
            } else {  // few items: one copy of the code for all variables
                double tl[5], tr[5];
#pragma unroll 1
                for (int m = 0; m < 5; m++) {
                    tl[m] = rowl < 0 ? wcns_state<true>(x0[m], x1[m], x2[m], x3[m], x4[m], top) : sec_state(sec + rowl * SEC_W, L, m, endl);
                    tr[m] = rowr < 0 ? wcns_state<false>(x1[m], x2[m], x3[m], x4[m], x5[m], top) : sec_state(sec + rowr * SEC_W, L, m, endr);
                    top = max(top, max((unsigned)__double2hiint(tl[m]) & 0x7fffffffu, (unsigned)__double2hiint(tr[m]) & 0x7fffffffu));
                }
#pragma unroll
                for (int m = 0; m < 5; m++) { ql[m] = tl[m]; qr[m] = tr[m]; }
            }
            odd = odd || top >= TOP_WEIGHT;
            // positivity fallback: the neighbouring point; in s1 and s4 means
            const bool badl = ql[0] <= RMIN_LIMIT || ql[4] <= PMIN_LIMIT, badr = qr[0] <= RMIN_LIMIT || qr[4] <= PMIN_LIMIT;
            const bool same = isec >= 0 && rowl == rowr && rowl < SEC_S2;
            if (badl || badr) {
                const int ia = h > 1 ? h : 1, ib = h + 1 < n ? h + 1 : n;
                // points of the means; of the neighbours
                const int la = same && endl ? 1 : ia, lb = same ? (endl ? h : h + 1) : ia, ra = same ? la : ib, rb = same ? lb : ib;
#pragma unroll
                for (int m = 0; m < 5; m++) {  // from memory: a mean may reach the line's first point
                    const double *q = F.f[F_R + m] + base + ln * lstep;
                    if (badl) ql[m] = (q[la * st] + q[lb * st]) / 2.0;
                    if (badr) qr[m] = (q[ra * st] + q[rb * st]) / 2.0;
                }
            }
            // half-node metrics: VALUE_HALF_NODE of (kx,ky,kz) along the line
            double kx, ky, kz;
            if (h > 1 && h < n - 1) {
                kx = (9.0 * (x2[5] + x3[5]) + -1.0 * (x4[5] + x1[5])) / 16.0;
                ky = (9.0 * (x2[6] + x3[6]) + -1.0 * (x4[6] + x1[6])) / 16.0;
                kz = (9.0 * (x2[7] + x3[7]) + -1.0 * (x4[7] + x1[7])) / 16.0;
            } else {  // from the end's four points
                const bool right = h >= n - 1, end = h == 0 || h == n;
                const int e = right ? n : 1, d = right ? -1 : 1;
                const double *ka = L.at(e), *kb = L.at(e + d), *kc = L.at(e + 2 * d), *kd = L.at(e + 3 * d);
                const double ca = end ? 35.0 : 5.0, cb = end ? -35.0 : 15.0, cc = end ? 21.0 : -5.0, cd = end ? -5.0 : 1.0;
                kx = (ca * ka[5] + cb * kb[5] + cc * kc[5] + cd * kd[5]) / 16.0;
                ky = (ca * ka[6] + cb * kb[6] + cc * kc[6] + cd * kd[6]) / 16.0;
                kz = (ca * ka[7] + cb * kb[7] + cc * kc[7] + cd * kd[7]) / 16.0;
            }
            const double kt = 0.0;  // kct=0, so every half-node value of kt is +0
            if (NFLUX == 3) odd = !flux_roe(P, gama1_1, ql, qr, kx, ky, kz, kt, same, fl) || odd;
            else bad += flux_split<NFLUX>(P, ql, qr, kx, ky, kz, kt, fl);
            double *f_ = isec < 0 ? fr + (wrap(fs + h - h0, FR) * NLP + ln) * INV_FP : secf + (ln * 26 + isec) * 5;
#pragma unroll
            for (int m = 0; m < 5; m++) f_[m] = fl[m];
        }
        if (__syncthreads_or(odd)) {
            rest = true;
            break;
        }
        nbad += bad;
        if (have < n + 3) {  // the next chunk's points, in place of the oldest
            int hi = h0 + len + C + 2;
            if (hi > n + 3) hi = n + 3;
            load(have + 1, hi, wrap(hs + have + 3 - h0, RP));
            have = hi;
        }
        // flux difference and accumulation into dq, in the order of memory: along
        // the line for i-lines, across the neighbouring lines otherwise
        auto fslot = [&](int h) { return wrap(fs + h - h0 < 0 ? fs + h - h0 + FR : fs + h - h0, FR); };
        if (mover) {
            const int fl = flags[pl];
            for (int l = l1; l <= lhi; l += C) {
                const int gi = pbase + l * st;
                const bool right = scheme4x && (fl & 2) && l >= n - 2, left = scheme4x && (fl & 1) && l <= 3;
                if (l != l1) {
#pragma unroll
                    for (int m = 0; m < 5; m++) old[m] = F.f[F_DQ1 + m][gi];
                }
                if (!right && !left && l > 2 && l < n - 1) {
                    const double *q[6];
#pragma unroll
                    for (int x = 0; x < 6; x++) q[x] = fr + (fslot(l - 3 + x) * NLP + pl) * INV_FP;
#pragma unroll
                    for (int m = 0; m < 5; m++)
                        F.f[F_DQ1 + m][gi] = old[m] + div_by(2250.0 * (q[3][m] - q[2][m]) - 125.0 * (q[4][m] - q[1][m]) + 9.0 * (q[5][m] - q[0][m]),
                                                             1920.0, 1.0 / 1920.0);
                    continue;
                }
                const double *sc = secf + pl * 130;
                double df[5];
#pragma unroll 1
                for (int m = 0; m < 5; m++) {
                    double v;
                    if (right || left) {
                        v = section_difference(sc + m, right, right ? n - l : l - 1);
                    } else {
                        auto fa = [&](int hh) { return fr[(fslot(hh) * NLP + pl) * INV_FP + m]; };
                        v = flux_dxyz_at(fa, n, l);
                    }
                    df[m] = v;
                }
#pragma unroll
                for (int m = 0; m < 5; m++) F.f[F_DQ1 + m][gi] = old[m] + df[m];
            }
        }
        if (last) break;
        if (lhi > done) done = lhi;
        h0 += len;
        hs = wrap(hs + len, RP);
        fs = wrap(fs + len, FR);
        len = C;
    }
    if (rest) nbad += inv_rest<dir, NFLUX>(&P, &F, &blocks[G.blk], groups + blockIdx.x, done, h0, C, smem, secf, sec);
    if (nbad) atomicAdd(&err[ERR_ROE], nbad);
}

template <int NFLUX>
static void launch_invis(const LaunchCtx &c, int dir, cudaStream_t st) {
    const DirTable &T = c.inv[dir];
    if (dir == 0) k_rhs_invis<0, NFLUX><<<T.ngroups, INV_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, T.cmax, c.err);
    else if (dir == 1) k_rhs_invis<1, NFLUX><<<T.ngroups, INV_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, T.cmax, c.err);
    else k_rhs_invis<2, NFLUX><<<T.ngroups, INV_THREADS, T.smem, st>>>(*c.P, *c.F, c.blocks, T.groups, T.cmax, c.err);
}

void launch_rhs_invis(const LaunchCtx &c, int dir, cudaStream_t st, double *out) {
    if (c.mixed) return launch_rhs_invis_mx(c, dir, st, out);
    if (c.inv[dir].ngroups == 0) return;
    if (c.P->nflux == 1) launch_invis<1>(c, dir, st);
    else if (c.P->nflux == 2) launch_invis<2>(c, dir, st);
    else launch_invis<3>(c, dir, st);
}

template <int NFLUX>
static void set_invis_attrs() {
    allow_all_smem(k_rhs_invis<0, NFLUX>);
    allow_all_smem(k_rhs_invis<1, NFLUX>);
    allow_all_smem(k_rhs_invis<2, NFLUX>);
}

void setup_rhs_invis_attrs(int nflux) {
    if (nflux == 1) set_invis_attrs<1>();
    else if (nflux == 2) set_invis_attrs<2>();
    else set_invis_attrs<3>();
}

size_t rhs_invis_line_bytes(int dir, int n, int nl, int cmax, bool sections) {
    const int C = inv_chunk(n, cmax);
    return sizeof(double) * ((size_t)inv_row(dir, nl) * (C + 5) * (INV_PITCH + INV_FP) + (sections ? (size_t)nl * 130 : 0));
}
int rhs_invis_lines(int n, int cmax) { return std::min(INV_MAX_LINES, INV_THREADS / inv_chunk(n, cmax)); }
int rhs_invis_chunks(int n, int cmax) { return (n + inv_chunk(n, cmax)) / inv_chunk(n, cmax); }

}  // namespace wcns
