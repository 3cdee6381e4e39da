// wcns_sweep.cuh -- the arithmetic of the LU-SGS sweeps, shared by the
// clustered and the wide kernels so that a cell's values are the same bits in
// either (the file that includes it is compiled without contraction; every
// fused multiply-add is written out).
//
// The neighbour term mxdq_std (LHS.f90:756-828) is the split Jacobian
// 0.5 (A + s r I) dq of the neighbour along one direction, with s = +1 for a
// lower and -1 for an upper neighbour, r its inviscid spectral radius, and A
// the flux Jacobian for its metrics g.  The routine reaches it through the
// three eigenvalues l1, l4, l5 and the normalised metrics; with the one
// radius r for all three eigenvalues the routine's
// x1 = (2 l1 - l4 - l5) / (2 c^2) is zero up to round-off and
// x2 = (l4 - l5) / (2 c) is |g| / 2, so the same map is, with
// theta = g.V, D = theta dq0 - g.(dq1, dq2, dq3) and
// dh = (gama - 1) (V^2/2 dq0 - V.(dq1, dq2, dq3) + dq4),
//     f0   = l dq0 - D/2
//     f123 = l dq123 + (g dh - V D)/2        l = (theta + s r)/2
//     f4   = l dq4 + (theta dh - H D)/2.
// It needs neither the sound speed nor a normalisation: 16 words per cell
// (u, v, w, H, nine metrics, three radii) for both signs instead of the 36 of
// the eigenvalue form, and about 80 operations for the three directions
// instead of 230.
//
// The viscous part of lusgs_l / lusgs_u, +-0.5 srv dq, has the same form as
// the radius: it goes into l as r + srv.
#pragma once
#include <cuda_runtime.h>

namespace wcns {

// The velocity as the terms take it.  The routine divides by the sound speed and its
// square: where c^2 is not a positive number all its terms are undefined, and so they
// are here, by way of theta.  hint = c^2 / (gama - 1)
__device__ __forceinline__ double sw_velocity(double u, double hint) {
    return hint > 0.0 && hint <= 1.7976931348623157e308 ? u : __longlong_as_double(0x7ff8000000000000LL);
}

// theta = g.V
__device__ __forceinline__ double sw_theta(double gx, double gy, double gz, double u, double v, double w) {
    return fma(gz, w, fma(gy, v, gx * u));
}
// dh / 2, the same for the three directions; aeh = 0.5 * (gama - 1)
__device__ __forceinline__ double sw_half_dh(double aeh, double u, double v, double w, const double *dq) {
    const double q = 0.5 * fma(w, w, fma(v, v, u * u));
    return aeh * (fma(q, dq[0], dq[4]) - fma(w, dq[3], fma(v, dq[2], u * dq[1])));
}
// D / 2
__device__ __forceinline__ double sw_half_d(double gx, double gy, double gz, double th, const double *dq) {
    return 0.5 * fma(th, dq[0], -fma(gz, dq[3], fma(gy, dq[2], gx * dq[1])));
}
// l for the radius r and the sign s
template <bool FWD>
__device__ __forceinline__ double sw_l(double th, double r) {
    return FWD ? 0.5 * (th + r) : 0.5 * (th - r);
}
// the part of component m that does not depend on the radius; a: g_m (theta
// for m = 4), b: V_m (H for m = 4)
__device__ __forceinline__ double sw_t0(double d2) { return -d2; }
__device__ __forceinline__ double sw_tm(double a, double b, double e, double d2) { return fma(a, e, -(b * d2)); }

// the five terms t along one direction
__device__ __forceinline__ void sw_terms(double gx, double gy, double gz, double th, double u, double v, double w, double h,
                                         double e, const double *dq, double *t) {
    const double d2 = sw_half_d(gx, gy, gz, th, dq);
    t[0] = sw_t0(d2);
    t[1] = sw_tm(gx, u, e, d2);
    t[2] = sw_tm(gy, v, e, d2);
    t[3] = sw_tm(gz, w, e, d2);
    t[4] = sw_tm(th, h, e, d2);
}

// new dq of a component from the sum of its received terms:
//   MODE 0 lusgs_l   base = rhs
//   MODE 1 lusgs_u   base = dq of lusgs_l
//   MODE 2 gs_pr_l   sum: lower terms, old: upper terms, base = rhs
//   MODE 3 gs_pr_u   sum: upper terms, base = lower terms - rhs
template <int MODE>
__device__ __forceinline__ double sw_new(double sum, double old, double base, double coed) {
    if (MODE == 0) return (sum - base) * coed;
    if (MODE == 1) return fma(-sum, coed, base);
    if (MODE == 2) return ((sum - old) - base) * coed;
    return fma(-sum, coed, base * coed);
}

}  // namespace wcns
