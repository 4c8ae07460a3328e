// physics.cuh -- FP64 point physics shared by the stage kernels and the point
// entry points.  Each function states the reference routine it computes; the algebra
// is regrouped to spend fewer FP64 instructions (one reciprocal of rho per point,
// contravariant fluxes formed directly, viscous and AV fluxes fused), so results
// agree with the reference to rounding, not bit for bit.
#pragma once
#include <cuda_runtime.h>

namespace chorus {

constexpr double kLambda = -2.0 / 3.0;  // setup2d.f90:70
constexpr double kPrandt = 0.72;        // setup2d.f90:71

// 1/x for the positive, normal densities of the path: the hardware approximation
// r (PTX rcp.approx.ftz.f64, relative error e = 1 - x r below 2^-19.9 over 2^28 sampled
// normal x) refined by one third-order step of the series 1/x = r/(1 - e) =
// r(1 + e + e^2 + ...): r <- r + r(e + e^2), leaving a relative error of about e^3
// (2^-60) below the rounding of the last FMA.  Measured on the same sample: within one
// ulp of the IEEE quotient 1.0/x (0.03% of values one ulp off), in 3 FP64 FMAs against
// the longer IEEE-rounded division sequence.
__host__ __device__ __forceinline__ double rcp_pos(double x) {
#ifdef __CUDA_ARCH__
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
#else
  return 1.0 / x;
#endif
}

// x/2 without an FP64 instruction (a multiplication for the rare values would be predicated
// and take its time for all): the exponent field less one for normal results; zeros and
// results below the normal range shift the significand, rounded to nearest even as the
// multiplication does; infinities and NaNs stay.  0.5*a + 0.5*b == half(a + b) bit for bit for
// normal operands.
__host__ __device__ __forceinline__ double half(double x) {
#ifdef __CUDA_ARCH__
  const unsigned long long b = (unsigned long long)__double_as_longlong(x), m = b & 0x7fffffffffffffffULL;
  const int ex = (int)(m >> 52);
  const unsigned long long tiny = (m >> 1) + (m & (m >> 1) & 1);
  const unsigned long long r = ex > 1 ? (ex < 0x7FF ? m - (1ULL << 52) : m) : tiny;
  return __longlong_as_double((long long)(r | (b & 0x8000000000000000ULL)));
#else
  return 0.5 * x;
#endif
}

// -x as a sign-bit flip: a negation that no add or multiply absorbs would otherwise
// take an FP64 instruction
__host__ __device__ __forceinline__ double negate(double x) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(__double_as_longlong(x) ^ (long long)0x8000000000000000ULL);
#else
  return -x;
#endif
}

// x * s for s = +-1 as a sign-bit flip (integer pipe, exact)
__host__ __device__ __forceinline__ double times_sign(double x, double s) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(__double_as_longlong(x) ^ (__double_as_longlong(s) & (long long)0x8000000000000000ULL));
#else
  return x * s;
#endif
}

// Contravariant ideal-MHD flux F*sx + G*sy of getIfluxvectors (getrusanov.f90:111-153)
// as used by inviscid_flux_interior (compflux.f90:77-78, 96-97).  Written in the
// momenta: with m = (ru, rv, rw), the mass flux m.s, the normal velocity (m.s)/rho and
// the normal field over rho, Bn/rho, give every term without forming u, v, w
// (u*Bn = ru*(Bn/rho), u.B = (m.B)/rho, rho|u|^2 = |m|^2/rho), 40 FP64 operations.
__host__ __device__ __forceinline__ void iflux_contra(const double* q, double sx, double sy, double gm1,
                                                      double* F) {
  const double rho = q[0], ru = q[1], rv = q[2], rw = q[3], E = q[4], Bx = q[5], By = q[6], Bz = q[7];
  const double ri = rcp_pos(rho);
  const double F0 = ru * sx + rv * sy;  // rho * Un
  const double Un = F0 * ri;
  const double Bn = Bx * sx + By * sy;
  const double bn = Bn * ri;            // Bn / rho
  const double B2 = Bx * Bx + By * By + Bz * Bz;
  const double m2 = ru * ru + rv * rv + rw * rw;
  const double hB2 = half(B2);
  const double pg = gm1 * (E - half(m2) * ri - hB2);
  const double pt = pg + hB2;
  const double mB = ru * Bx + rv * By + rw * Bz;
  F[0] = F0;
  F[1] = ru * Un + pt * sx - Bx * Bn;
  F[2] = rv * Un + pt * sy - By * Bn;
  F[3] = rw * Un - Bz * Bn;
  F[4] = (E + pt) * Un - mB * bn;
  F[5] = Bx * Un - ru * bn;
  F[6] = By * Un - rv * bn;
  F[7] = Bz * Un - rw * bn;
}

// Rusanov flux of getrusanovflux (getrusanov.f90:1-109) along the unit normal (ux,uy),
// times `scale`: Fh = scale*(Fl + Fr - eigv*(qr - ql)); with scale = magnorm*sign_l/2
// this is the reference's Fnl in the left cell's computational frame (:90-93).  Returns
// the left normal velocity (for the A_z upwinding, :99-103) and the wave-speed bound
// eigv (:87).
__host__ __device__ __forceinline__ void rusanov_core(const double* ql, const double* qr, double ux, double uy,
                                                      double gam, double scale, double* Fh, double& vnl,
                                                      double& eigv) {
  const double gm1 = gam - 1.0;
  double Fl[8], Fr[8], pgl, pgr, vn[2];
  const double* qs[2] = {ql, qr};
  double* Fs[2] = {Fl, Fr};
  double* pg[2] = {&pgl, &pgr};
#pragma unroll
  for (int side = 0; side < 2; side++) {
    const double* q = qs[side];
    double* F = Fs[side];
    const double ri = rcp_pos(q[0]);
    const double u = ri * q[1], v = ri * q[2], w = ri * q[3];
    const double Bx = q[5], By = q[6], Bz = q[7];
    const double B2 = Bx * Bx + By * By + Bz * Bz;
    const double p = gm1 * (q[4] - 0.5 * q[0] * (u * u + v * v + w * w) - B2 * 0.5);
    const double pt = p + 0.5 * B2;
    const double Vn = u * ux + v * uy;
    const double Bn = Bx * ux + By * uy;
    F[0] = q[0] * Vn;
    F[1] = q[1] * Vn + pt * ux - Bx * Bn;
    F[2] = q[2] * Vn + pt * uy - By * Bn;
    F[3] = q[3] * Vn - Bz * Bn;
    F[4] = (q[4] + pt) * Vn - Bn * (u * Bx + v * By + w * Bz);
    F[5] = (v * Bx - u * By) * uy;
    F[6] = (u * By - v * Bx) * ux;
    F[7] = Bz * Vn - w * Bn;
    *pg[side] = p;
    vn[side] = Vn;
  }
  const double Bx = 0.5 * (ql[5] + qr[5]), By = 0.5 * (ql[6] + qr[6]), Bz = 0.5 * (ql[7] + qr[7]);
  const double irs = rcp_pos(ql[0] + qr[0]);
  const double ca = gam * (pgl + pgr) * irs;
  const double cd = (Bx * Bx + By * By + Bz * Bz) * (2.0 * irs);
  const double bn = Bx * ux + By * uy;
  const double cn = bn * bn * (2.0 * irs);
  const double cad = ca + cd;
  const double ctmp = sqrt(cad * cad - 4.0 * ca * cn);
  const double cf = sqrt(0.5 * (cad + ctmp));
  eigv = 0.5 * fabs(vn[0] + vn[1]) + cf;
#pragma unroll
  for (int k = 0; k < 8; k++) Fh[k] = scale * fma(-eigv, qr[k] - ql[k], Fl[k] + Fr[k]);
  vnl = vn[0];
}

// Contravariant viscous + resistive + artificial-viscosity flux at one flux point:
// getVfluxvectors (getrusanov.f90:157-249) with (mu, eta0) plus getVfluxvectors_AV
// (:251-360) with (mu_art, 0), summed (the hydrodynamic terms are linear in the
// viscosity) and contracted with the metric row (sx, sy) as in comp_viscous_flux
// (compflux.f90:216-225, 241-250).  g is nablaQ(9,2) in Fortran order; only
// components 1..7 of the result are nonzero (Fv(1) = Fv(9) = 0).
//
// With w_c = rho grad u_c = grad m_c - u_c grad rho and everything contracted with S as early
// as it can be, the stress row is (mu / rho) c, c_i = w_i.S + (d_i w).S - 2/3 div S_i, the energy
// flux u.F + (mu gamma / (Pr rho)) H with H = rho^2 grad e / rho . S, and the resistive
// part adds B.F_B: 75 FP64 operations against 115 of the vectors contracted at the end.
// (vflux_int is the integer form of the same steps.)
__host__ __device__ __forceinline__ void vflux_contra(const double* q, const double* g, double mut, double eta0,
                                                      double gam, double sx, double sy, double* Fc) {
  const double rho = q[0], Bx = q[5], By = q[6], Bz = q[7];
  const double ri = rcp_pos(rho);
  const double u = q[1] * ri, v = q[2] * ri, w = q[3] * ri;
  const double hNU = half(u * u + v * v + w * w);
  const double B2 = Bx * Bx + By * By + Bz * Bz;
  const double inte = q[4] * ri - hNU - half(B2) * ri;
  const double* gy = g + 9;
  const double rx = g[0], ry = gy[0], rS = rx * sx + ry * sy;
  // rho times the velocity gradients of the plane
  const double ux = g[1] - rx * u, uy = gy[1] - ry * u, vx = g[2] - rx * v, vy = gy[2] - ry * v;
  const double ld = kLambda * (ux + vy);
  const double c1 = ux * sx + uy * sy + (ux * sx + vx * sy) + ld * sx;
  const double c2 = vx * sx + vy * sy + (uy * sx + vy * sy) + ld * sy;
  const double mzS = g[3] * sx + gy[3] * sy, c3 = mzS - rS * w;
  const double bzS = g[7] * sx + gy[7] * sy;
  double H = g[4] * sx + gy[4] * sy;
  H -= u * (g[1] * sx + gy[1] * sy) + v * (g[2] * sx + gy[2] * sy) + w * mzS;
  H -= Bx * (g[5] * sx + gy[5] * sy) + By * (g[6] * sx + gy[6] * sy) + Bz * bzS;
  H += (hNU - inte) * rS;
  const double M = mut * ri;
  Fc[0] = 0.0;
  Fc[1] = M * c1;
  Fc[2] = M * c2;
  Fc[3] = M * c3;
  Fc[4] = M * (u * c1 + v * c2 + w * c3 + (gam / kPrandt) * H);
  Fc[5] = 0.0;
  Fc[6] = 0.0;
  Fc[7] = 0.0;
  if (eta0 != 0.0) {  // resistive terms (the AV form has eta_art = 0)
    const double eJz = eta0 * (g[6] - gy[5]);
    Fc[5] = negate(eJz) * sy;
    Fc[6] = eJz * sx;
    Fc[7] = eta0 * bzS;
    Fc[4] += Bx * Fc[5] + By * Fc[6] + Bz * Fc[7];
  }
}

// muAV of variable 1 (AV.f90:157-172 with se_low=-6, se_high=-1) from the sensor sum
// ssum = sum ((Qsm-rho)/rho)^2 of a cell, Se = log10(ssum): zero below 1e-6, epsilon0
// above 0.1 (the ramp is continuous at both ends), the sine ramp in between.
// muAV = epsilon0 / 2 * av_ramp.
__host__ __device__ __forceinline__ double av_ramp(double ssum) {
  if (ssum < 1e-6) return 0.0;
  if (ssum > 0.1) return 2.0;
  const double se = log10(ssum);
  const double s0 = -3.5, kr = 2.5, pi = 3.14159265358979323846;
  return 1.0 + sin(pi * (se - s0) / 2.0 / kr);
}

__host__ __device__ __forceinline__ double av_mu(double ssum, double eps0) { return eps0 / 2.0 * av_ramp(ssum); }

}  // namespace chorus
