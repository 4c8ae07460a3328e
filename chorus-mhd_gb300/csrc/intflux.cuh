// intflux.cuh -- the ideal-MHD point fluxes in integer arithmetic.
//
// GB300 executes FP64 at 2 lane-operations per clock per SM (a warp instruction occupies
// its scheduler's FP64 unit for 64 clocks), the integer pipes take 64 each.  The nonlinear
// fluxes are products and sums of few variables, so they are evaluated in integers: a value is
// v 2^e with a 64-bit integer v and an exponent e of its own, products keep the upper part of the
// 128-bit product of two such integers, sums align to the largest of their terms, and each
// result is rounded once into a double.
//
//   * A product takes the operands as limbs v = h 2^31 + l (|l| < 2^31):
//     (a b) >> 62 = ha hb + ((ha lb + la hb) >> 31) in three 32x32->64 multiply-adds; the
//     product of the low limbs is below one unit and left out.
//   * A product of two operands of full length (2^60 .. 2^61) is off by two units of at least 2^58;
//     operands that have lost length, to a cancellation or over several products, are shifted up
//     again (ix_up).  Each term of a component is then off by less than 2^-54 of itself, and the
//     component, with its rounding, by less than 2^-52 of the sum of its terms' magnitudes (the
//     viscous flux 2^-51).  Over states with components of all sizes the rms error is at or below
//     that of the FP64 forms, component by component, typically half of it.
//
// The integer form takes finite states with a normal positive density and magnitudes within
// a wide window (2^-200 .. 2^200, the viscous flux 2^-120 .. 2^120; zero and smaller values of all but
// the density, energy and metric as well), so that no result leaves the range of a double;
// everything else (infinities, NaNs, zero or negative density, a negative pressure, a density ratio
// above 8 across a face, a negative discriminant) is left to the FP64 form, whose results on
// such states the caller keeps.
#pragma once
#include <cstdint>

#include "fixdot.cuh"

namespace chorus {

struct Limbs {
  int h, l;
};

FIX_HD Limbs ix_limbs(int64_t v) { return Limbs{(int)(v >> 31), (int)(v & 0x7fffffff)}; }

// v >> d for d >= 0, the sign for d > 63
FIX_HD int64_t ix_shr(int64_t v, int d) {
#ifdef __CUDA_ARCH__
  int64_t r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(d));  // clamps the amount
  return r;
#else
  return v >> (d < 63 ? d : 63);
#endif
}
FIX_HD int64_t ix_shl(int64_t v, int n) { return (int64_t)((uint64_t)v << n); }

// (a b) >> 62
FIX_HD int64_t ix_mul(Limbs a, Limbs b) {
  const int64_t t = fix_mad(a.l, b.h, fix_mad(a.h, b.l, 0));
  return fix_mad(a.h, b.h, t >> 31);
}
FIX_HD int64_t ix_mul(int64_t a, Limbs b) { return ix_mul(ix_limbs(a), b); }

FIX_HD uint32_t ix_abs_word(double x) { return (uint32_t)(fix_bits(x) >> 32) & 0x7fffffffu; }
FIX_HD uint32_t ix_max(uint32_t a, uint32_t b) { return a > b ? a : b; }
FIX_HD int ix_max(int a, int b) { return a > b ? a : b; }

// x as an integer aligned to the exponent of the magnitude word m >= that of x: a value of
// that exponent has its leading bit at bit 63 - SH, i.e. v = x 2^(63 - SH + 1023 - (m >> 20))
// truncated (a zero, which has no hidden bit, is shifted out: m is that of a group that
// has a nonzero value, above 2^-900, or the group is all zero and not used)
template <int SH>
FIX_HD int64_t ix_align(double x, uint32_t m) {
  const uint64_t u = fix_bits(x);
  const uint32_t a = (uint32_t)(u >> 32) & 0x7fffffffu;
  const int d = (int)(((m | 0xfffffu) + ((uint32_t)SH << 20) - a) >> 20);
  const int64_t v = (int64_t)fix_shru((u << 11) | 0x8000000000000000ull, d);
  return (int64_t)u < 0 ? -v : v;
}
// the exponent e of v 2^e for ix_align<SH>
template <int SH>
FIX_HD int ix_exp(uint32_t m) {
  return (int)(m >> 20) - 1023 - (63 - SH);
}

// v 2^e as a double, rounded to nearest; results below the normal range are flushed to zero
FIX_HD double ix_double(int64_t v, int e) { return fix_cvt_v<true>(v, e + 1); }

// 2^122 / d for d in [2^61, 2^62): in (2^60, 2^61], within a few units.  The hardware
// approximation r0 (relative error below 2^-19.9) refined by 1/D = r0 (1 + e + e^2 + ...),
// e = 1 - D r0, to e^3 < 2^-59.
FIX_HD int64_t ix_rcp(int64_t d) {
  const uint32_t hi = (uint32_t)(d >> 41) & 0xfffffu;  // the 20 bits below the leading one
#ifdef __CUDA_ARCH__
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(__hiloint2double((int)(hi | 0x3ff00000u), (int)((uint32_t)(d >> 9)))));
  const int r0 = (int)(((uint32_t)__double2hiint(r) - (1021u << 20)) << 9);  // 2^30 / D
#else
  const int r0 = (int)((uint32_t)(1073741824.0 / (1.0 + hi * 0x1p-20 + 0x1p-21)) & ~511u);
#endif
  const Limbs D = ix_limbs(d);  // D 2^61
  const int64_t P = fix_mad(D.h, r0, fix_mad(D.l, r0, 0) >> 31);  // D r0, 60 fraction bits
  const int64_t e = ((int64_t)1 << 60) - P;                           // |e| < 2^40.2
  const int eh = (int)(e >> 10);
  const int64_t s = e + (fix_mad(eh, eh, 0) >> 40);  // e + e^2
  const int sh = (int)(s >> 10), sl = (int)(s & 1023);
  return ((int64_t)r0 << 31) + (fix_mad(r0, sh, fix_mad(r0, sl, 0) >> 10) >> 19);
}

// sqrt(v 2^e) for v > 0 as s 2^es, s in [2^60, 2^61]: y0 = 1/sqrt by the hardware
// approximation (relative error below 2^-22), a = x y0, f = 1 - x y0^2,
// sqrt x = a (1 - f)^(-1/2) = a (1 + f/2 + 3 f^2 / 8 + ...), the cubic term is below 2^-64
FIX_HD int64_t ix_sqrt(int64_t v, int e, int& es) {
#ifdef __CUDA_ARCH__
  int lz = __clzll(v);
#else
  int lz = __builtin_clzll((uint64_t)v);
#endif
  // x = v << n in [2^60, 2^62) with e - n even
  int n = lz - 2;
  n -= (n ^ e) & 1;
  int64_t x = n >= 0 ? (int64_t)((uint64_t)v << n) : v >> 1;
  const int er = e - n;  // even: v 2^e = x 2^er
  // X = x 2^-62 in [1/4, 1): y0 ~ X^-1/2 in (1, 2], 29 fraction bits
  const float xf = (float)(uint32_t)(x >> 30);  // 2^32 X
#ifdef __CUDA_ARCH__
  float yf;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(yf) : "f"(xf));
#else
  const float yf = 1.0f / __builtin_sqrtf(xf);
#endif
  const int y0 = (int)(yf * 0x1p45f);  // 2^16 2^29 / sqrt(2^32 X)
  const Limbs L = ix_limbs(x);
  const int64_t a = fix_mad(L.h, y0, fix_mad(L.l, y0, 0) >> 31);  // X y0: 60 fraction bits (62 + 29 - 31)
  const Limbs La = ix_limbs(a);
  const int64_t b = fix_mad(La.h, y0, fix_mad(La.l, y0, 0) >> 31);  // X y0^2: 58 fraction bits
  const int64_t f = ((int64_t)1 << 58) - b;                               // |f| < 2^-20: below 2^38
  const int fh = (int)(f >> 8);                                            // 50 fraction bits
  const int64_t c = (f >> 1) + ((3 * (fix_mad(fh, fh, 0) >> 20)) >> 25);  // f/2 + 3 f^2/8, 58 fraction bits
  const int c1 = (int)(c >> 7), c0 = (int)(c & 127);                       // 51 and 58 fraction bits
  es = er / 2 + 31 - 61;
  // 2 a (1 + c), a = h 2^-29 + l 2^-60
  return a + a + (fix_mad(La.h, c1, (fix_mad(La.l, c1, 0) >> 31) + (fix_mad(La.h, c0, 0) >> 7)) >> 19);
}

// leading zeros of |v| among the upper 32 bits, less `keep`: a left shift by that many bits
// (at least 0) leaves |v| <= 2^(64 - keep)
FIX_HD int ix_room(int64_t v, int keep) {
  const int hi = (int)(v >> 32);
  const uint32_t a = (uint32_t)(hi ^ (hi >> 31));
#ifdef __CUDA_ARCH__
  return ix_max(__clz((int)a) - keep, 0);
#else
  return ix_max((a ? __builtin_clz(a) : 32) - keep, 0);
#endif
}

// ---------------------------------------------------------------------------
// Values with an exponent of their own.  Every variable of a state, every component of a normal
// and every product carries one, so that a small component beside a large one keeps all its bits
// as it does in FP64 (with one exponent for the components of the plane a transverse flux of
// 10^-8 of the main one was left with 29 bits); only the terms of a sum are aligned, to the
// largest of them.  [b] in the comments means a magnitude of at most 2^b.
// ---------------------------------------------------------------------------
struct IxF {  // an operand: m 2^e, [61]
  Limbs m;
  int e;
};
struct IxV {  // a product or a sum: v 2^e
  int64_t v;
  int e;
};

constexpr uint32_t kIxLow = 823u << 20, kIxHigh = 1223u << 20;  // 2^-200 .. 2^200
constexpr uint32_t kIxVLow = 903u << 20, kIxVHigh = 1143u << 20;  // 2^-120 .. 2^120: the viscous flux
constexpr uint32_t kIxZero = 66u << 20;  // magnitude words below: a zero

// x without rounding, 2^60 <= |m| < 2^61; both limbs carry the sign.  A zero gets the exponent of
// kIxZero, which no sum aligns to
FIX_HD IxF ix_load(double x) {
  const uint64_t u = fix_bits(x);
  const uint32_t hi = (uint32_t)(u >> 32), lo = (uint32_t)u, a = hi & 0x7fffffffu;
  const int s = a < kIxZero ? 0 : (int)hi < 0 ? -1 : 1;
  const int h = (int)((((hi << 9) | (lo >> 23)) & 0x3fffffffu) | 0x20000000u), l = (int)((lo << 8) & 0x7fffffffu);
  return IxF{Limbs{h * s, l * s}, (int)(ix_max(a, kIxZero) >> 20) - 1083};
}
// 1/x of a positive normal x
FIX_HD IxF ix_inverse(double x) {
  const uint64_t u = fix_bits(x);
  return IxF{ix_limbs(ix_rcp((int64_t)(((u << 11) | 0x8000000000000000ull) >> 2))), 962 - (int)(u >> 52)};
}
FIX_HD IxV ix_whole(IxF a) { return IxV{(int64_t)a.m.h * ((int64_t)1 << 31) + a.m.l, a.e}; }
FIX_HD IxF ix_split(IxV a) { return IxF{ix_limbs(a.v), a.e}; }          // of [61.6] at most
FIX_HD IxV ix_times(IxF a, IxF b) { return IxV{ix_mul(a.m, b.m), a.e + b.e + 62}; }  // [60], off by two units
FIX_HD IxV ix_square(IxF a) {                                          // [60]
  return IxV{fix_mad(a.m.h, a.m.h, fix_mad(a.m.h, a.m.l, 0) >> 30), 2 * a.e + 62};
}
FIX_HD int64_t ix_at(IxV a, int K) { return ix_shr(a.v, K - a.e); }  // a in units of 2^K, K >= a.e
FIX_HD IxV ix_plus(IxV a, IxV b) {
  const int K = ix_max(a.e, b.e);
  return IxV{ix_at(a, K) + ix_at(b, K), K};
}
FIX_HD IxV ix_minus(IxV a, IxV b) {
  const int K = ix_max(a.e, b.e);
  return IxV{ix_at(a, K) - ix_at(b, K), K};
}
FIX_HD IxV ix_halved(IxV a) { return IxV{a.v >> 1, a.e + 1}; }  // the same value in one bit less
// an operand of full length (up to 29 leading zeros are shifted out)
FIX_HD IxF ix_up(IxV a) {
  const int n = ix_room(a.v, 3);
  return IxF{ix_limbs(ix_shl(a.v, n)), a.e - n};
}
FIX_HD double ix_double(IxV a) { return ix_double(a.v, a.e); }

// the products q(r) s(r) of a line as integers X_r, |X_r| < 2^58, aligned to the largest of them;
// returns their exponent, or a number above kIxNoLine / 2 where an operand has the exponent
// kIxNoLine (a value that the integer form leaves out)
constexpr int kIxNoLine = 1 << 24;
template <int NI, class Q, class S>
FIX_HD int ix_line_products(Q&& q, S&& s, int64_t (&X)[NI]) {
  int e[NI], K = -kIxNoLine;
#pragma unroll
  for (int r = 0; r < NI; r++) {
    const IxV p = ix_times(q(r), s(r));
    X[r] = p.v;
    e[r] = p.e;
    K = ix_max(K, p.e);
  }
#pragma unroll
  for (int r = 0; r < NI; r++) X[r] = ix_shr(X[r], K - e[r] + 2);
  return K + 2;
}

// constants of a solve, prepared once (host or device): half of gamma - 1, gamma, gamma / Pr
struct IxGas {
  IxF g, gam, kap;
};
FIX_HD IxGas ix_gas(double gamma) { return IxGas{ix_load(0.5 * (gamma - 1.0)), ix_load(gamma), ix_load(gamma / 0.72)}; }

// Contravariant ideal-MHD flux F sx + G sy (iflux_contra); q(k) reads variable k, out(j, a, b)
// takes components 2 j and 2 j + 1.  Returns false, without output, where the integer form does
// not apply.  Every term of a component's sum is off by less than 2^-54 of itself (three products
// of operands of full length in a row).
template <class Q, class Out>
FIX_HD bool iflux_int(Q&& q, double sx, double sy, const IxGas& gas, Out&& out) {
  const uint32_t r = (uint32_t)(fix_bits(q(0)) >> 32), me = ix_abs_word(q(4));  // r: huge if the sign is set
  const uint32_t mz = ix_max(ix_abs_word(q(3)), ix_abs_word(q(7)));
  const uint32_t mp = ix_max(ix_max(ix_abs_word(q(1)), ix_abs_word(q(2))), ix_max(ix_abs_word(q(5)), ix_abs_word(q(6))));
  const uint32_t ms = ix_max(ix_abs_word(sx), ix_abs_word(sy));
  if (ix_max(ix_max(ix_max(r, me), ix_max(mp, mz)), ms) >= kIxHigh || r < kIxLow || me < kIxLow || ms < kIxLow) return false;
  const bool hasz = mz >= kIxZero;
  const IxF nx = ix_load(sx), ny = ix_load(sy), mx = ix_load(q(1)), my = ix_load(q(2));
  const IxF bx = ix_load(q(5)), by = ix_load(q(6)), ri = ix_inverse(q(0));
  // mass flux, normal velocity (normal field the same), v Bx - u By
  const IxV f0 = ix_plus(ix_times(mx, nx), ix_times(my, ny));  // [61]
  const double F0 = ix_double(f0);
  const IxF V = ix_up(ix_times(ix_split(f0), ri));
  const IxF Bn = ix_up(ix_plus(ix_times(bx, nx), ix_times(by, ny))), bnl = ix_split(ix_times(Bn, ri));
  const IxF W = ix_up(ix_times(ix_split(ix_minus(ix_times(my, bx), ix_times(mx, by))), ri));
  IxV k2 = ix_plus(ix_square(mx), ix_square(my)), b2 = ix_plus(ix_square(bx), ix_square(by));  // [61]
  IxV mB = ix_plus(ix_times(mx, bx), ix_times(my, by));
  double F3 = 0.0, F7 = 0.0;
  if (hasz) {
    const IxF w = ix_load(q(3)), bz = ix_load(q(7));
    k2 = ix_plus(k2, ix_square(w));  // [61.6]
    b2 = ix_plus(b2, ix_square(bz));
    mB = ix_plus(mB, ix_times(w, bz));
    F3 = ix_double(ix_minus(ix_times(w, V), ix_times(bz, Bn)));
    F7 = ix_double(ix_minus(ix_times(bz, V), ix_times(w, bnl)));
  }
  // 2 p / (gamma - 1) = 2 E - m^2/rho - B^2, the total pressure, E + pt
  const IxF E = ix_load(q(4));
  const IxV kr = ix_times(ix_split(k2), ri);
  const int KS = ix_max(ix_max(E.e + 1, kr.e), b2.e);
  const int64_t S = ix_shr(ix_whole(E).v, KS - E.e - 1) - ix_at(kr, KS) - ix_at(b2, KS);
  if (S < 0) return false;
  const IxF P = ix_up(ix_halved(ix_plus(ix_times(IxF{ix_limbs(S), KS}, gas.g), IxV{b2.v, b2.e - 1})));
  const IxF Ep = ix_split(ix_halved(ix_plus(ix_whole(E), ix_whole(P))));
  auto component = [&](IxF m, IxF b, IxF n) {  // m V - b Bn + pt n
    const IxV a = ix_times(m, V), c = ix_times(b, Bn), d = ix_times(P, n);
    const int K = ix_max(ix_max(a.e, c.e), d.e);
    return ix_double(ix_at(a, K) - ix_at(c, K) + ix_at(d, K), K);
  };
  out(0, F0, component(mx, bx, nx));
  out(1, component(my, by, ny), F3);
  out(2, ix_double(ix_minus(ix_times(Ep, V), ix_times(ix_up(ix_halved(mB)), bnl))), ix_double(ix_times(W, ny)));
  const IxV f6 = ix_times(W, nx);
  out(3, ix_double(-f6.v, f6.e), F7);
  return true;
}

// Contravariant viscous, resistive and artificial-viscosity flux (vflux_contra, whose formulas
// these are): q(k) the state, g(d, k) its gradient, mut and eta the viscosity and resistivity.
// out(k, value) takes components 1..7; false, without output, where the integer form does not
// apply.  The first output comes after the last use of q, which may therefore lie in the outputs'
// place.  Magnitudes of up to 2^120 (and a density down to 2^-120) are taken: the largest product,
// the viscosity times the squared velocity times the velocity gradient, stays below 2^1000.
template <class Q, class G, class Out>
FIX_HD bool vflux_int(Q&& q, G&& g, double mut, double eta, double sx, double sy, const IxGas& gas, Out&& out) {
  auto w1 = [&](int k) { return ix_abs_word(q(k)); };
  auto w2 = [&](int k) { return ix_max(ix_abs_word(g(0, k)), ix_abs_word(g(1, k))); };
  const uint32_t r = (uint32_t)(fix_bits(q(0)) >> 32);  // huge if the sign is set
  const uint32_t mz = ix_max(ix_max(w1(3), w1(7)), ix_max(w2(3), w2(7)));
  const uint32_t mq = ix_max(ix_max(ix_max(w1(1), w1(2)), ix_max(w1(5), w1(6))), ix_max(w1(4), r));
  const uint32_t mg = ix_max(ix_max(ix_max(w2(0), w2(1)), ix_max(w2(2), w2(4))), ix_max(w2(5), w2(6)));
  const uint32_t ms = ix_max(ix_abs_word(sx), ix_abs_word(sy)), mc = ix_max(ix_abs_word(mut), ix_abs_word(eta));
  if (ix_max(ix_max(ix_max(mq, mg), ix_max(mz, ms)), mc) >= kIxVHigh || r < kIxVLow || ms < kIxVLow) return false;
  const bool hasz = mz >= kIxZero;
  const IxF nx = ix_load(sx), ny = ix_load(sy), ri = ix_inverse(q(0));
  const IxF M = ix_up(ix_times(ix_load(mut), ri));  // mu / rho
  auto along = [&](IxF a, IxF b) { return ix_plus(ix_times(a, nx), ix_times(b, ny)); };  // a sx + b sy: [61]
  // velocities; X = |u|^2 + B^2/(2 rho) - E/rho
  const IxF mx = ix_load(q(1)), my = ix_load(q(2)), bx = ix_load(q(5)), by = ix_load(q(6));
  const IxF u = ix_up(ix_times(mx, ri)), v = ix_up(ix_times(my, ri));
  IxF w{Limbs{0, 0}, 0}, bz{Limbs{0, 0}, 0};
  IxF X;
  {
    IxV k2 = ix_plus(ix_square(mx), ix_square(my)), b2 = ix_plus(ix_square(bx), ix_square(by));  // [61]
    if (hasz) {
      const IxF mw = ix_load(q(3));
      bz = ix_load(q(7));
      w = ix_up(ix_times(mw, ri));
      k2 = ix_plus(k2, ix_square(mw));  // [61.6]
      b2 = ix_plus(b2, ix_square(bz));
    }
    const IxV kr = ix_times(ix_split(k2), ri), E = ix_whole(ix_load(q(4)));
    const int K = ix_max(ix_max(kr.e, b2.e - 1), E.e) + 1;
    X = ix_up(ix_times(ix_split(IxV{ix_at(kr, K) + ix_shr(b2.v, K - b2.e + 1) - ix_at(E, K), K}), ri));
  }
  const IxF rx = ix_load(g(0, 0)), ry = ix_load(g(1, 0)), rS = ix_up(along(rx, ry));
  // rho times the velocity gradients of the plane; with a third of the divergence D, the rows
  // c1 = 2 (ux - D) sx + (uy + vx) sy, c2 = (uy + vx) sx + 2 (vy - D) sy of the stress
  IxF c1, c2;
  IxV t2;  // u.(grad m . S) of the plane
  {
    const IxF ax = ix_load(g(0, 1)), ay = ix_load(g(1, 1)), cx = ix_load(g(0, 2)), cy = ix_load(g(1, 2));
    t2 = ix_plus(ix_times(ix_up(along(ax, ay)), u), ix_times(ix_up(along(cx, cy)), v));  // [61]
    auto rel = [&](IxF a, IxF r_, IxF u_) { return ix_minus(ix_halved(ix_whole(a)), ix_times(r_, u_)); };  // [61]
    const IxV ux = rel(ax, rx, u), uy = rel(ay, ry, u), vx = rel(cx, rx, v), vy = rel(cy, ry, v);
    const IxF third{ix_limbs(1537228672809129301LL), -62};  // 2^62 / 3
    const IxV D = ix_times(ix_split(ix_halved(ix_plus(ux, vy))), third);
    const IxF a = ix_up(ix_halved(ix_minus(ux, D))), b = ix_up(ix_halved(ix_plus(uy, vx))), d = ix_up(ix_halved(ix_minus(vy, D)));
    auto twice = [](IxV t) { return IxV{t.v, t.e + 1}; };
    c1 = ix_up(ix_plus(twice(ix_times(a, nx)), ix_times(b, ny)));
    c2 = ix_up(ix_plus(ix_times(b, nx), twice(ix_times(d, ny))));
  }
  out(1, ix_double(ix_times(c1, M)));
  out(2, ix_double(ix_times(c2, M)));
  // energy: M (u.c + gamma/Pr H), H = grad E.S - u.(grad m.S) - B.(grad B.S) + X grad rho.S
  const IxF yx = ix_load(g(0, 6)), xy = ix_load(g(1, 5));
  IxV H = ix_minus(ix_plus(along(ix_load(g(0, 4)), ix_load(g(1, 4))), ix_times(X, rS)), t2);  // [62.6]
  H = ix_minus(H, ix_plus(ix_times(ix_up(along(ix_load(g(0, 5)), xy)), bx), ix_times(ix_up(along(yx, ix_load(g(1, 6)))), by)));  // [63 - ]
  IxV uc = ix_plus(ix_times(c1, u), ix_times(c2, v));  // [61]
  double F3 = 0.0;
  IxF bzS{Limbs{0, 0}, 0};
  if (hasz) {
    const IxF mzS = ix_up(along(ix_load(g(0, 3)), ix_load(g(1, 3))));
    bzS = ix_up(along(ix_load(g(0, 7)), ix_load(g(1, 7))));
    const IxF c3 = ix_up(ix_minus(ix_halved(ix_whole(mzS)), ix_times(rS, w)));
    F3 = ix_double(ix_times(c3, M));
    H = ix_minus(ix_halved(H), ix_plus(ix_times(mzS, w), ix_times(bzS, bz)));
    uc = ix_plus(uc, ix_times(c3, w));  // [61.6]
  }
  out(3, F3);
  IxV F4 = ix_times(ix_up(ix_halved(ix_plus(uc, ix_times(ix_up(ix_halved(H)), gas.kap)))), M);  // [60]
  double F5 = 0.0, F6 = 0.0, F7 = 0.0;
  if (eta != 0.0) {  // resistive terms: F_B = eta (-Jz sy, Jz sx, grad Bz.S), the energy takes B.F_B
    const IxF et = ix_load(eta);
    const IxF J = ix_up(ix_times(ix_up(ix_halved(ix_minus(ix_whole(yx), ix_whole(xy)))), et));
    const IxV jy = ix_times(J, ny);
    F5 = ix_double(-jy.v, jy.e);
    F6 = ix_double(ix_times(J, nx));
    IxV R = ix_times(J, ix_up(ix_minus(ix_times(by, nx), ix_times(bx, ny))));
    if (hasz) {
      const IxF f7 = ix_up(ix_times(bzS, et));
      F7 = ix_double(ix_whole(f7));
      R = ix_plus(R, ix_times(f7, bz));
    }
    F4 = ix_plus(F4, R);
  }
  out(4, ix_double(F4));
  out(5, F5);
  out(6, F6);
  out(7, F7);
  return true;
}

// Rusanov flux along the unit normal (ux, uy) times `scale` (rusanov_core): Fh = scale
// (Fl + Fr - eigv (qr - ql)).  q(side, k) reads variable k of the left (0) or right (1)
// state, out(j, a, b) takes components 2 j and 2 j + 1.  Returns false, without output, where
// the integer form does not apply (a density ratio above 8 among them).
//
// The two sides stream through sums (of the flux components without the pressure, of the
// pressures, of the field), so that no component of the states lives longer than its side; each
// term keeps its own exponent until its sum is formed, whichever side it comes from.
template <class Q, class Out>
FIX_HD bool rusanov_int(Q&& q, double ux, double uy, const IxGas& gas, double scale, double& eigv, Out&& out) {
  // ---- range of the states
  auto word = [&](int k) { return ix_max(ix_abs_word(q(0, k)), ix_abs_word(q(1, k))); };
  const uint32_t mr = word(0), ms = ix_abs_word(scale), el = ix_abs_word(q(0, 4)), er = ix_abs_word(q(1, 4));
  const uint32_t mz = ix_max(word(3), word(7)), mp = ix_max(ix_max(word(1), word(2)), ix_max(word(5), word(6)));
  const uint32_t rl = (uint32_t)(fix_bits(q(0, 0)) >> 32), rr = (uint32_t)(fix_bits(q(1, 0)) >> 32);  // sign set: huge
  const uint32_t rmin = rl < rr ? rl : rr, rmax = rl < rr ? rr : rl;
  if (ix_max(ix_max(ix_max(rmax, ix_max(el, er)), ix_max(mp, mz)), ms) >= kIxHigh || rmin < kIxLow ||
      ix_max(el, er) < kIxLow || ms < kIxLow || rmax - rmin >= (3u << 20))
    return false;
  const bool hasz = mz >= kIxZero;
  const IxF nx = ix_load(ux), ny = ix_load(uy);
  // ---- the sums over the sides
  IxV F0, W, Gx, Gy, Gz{0, 0}, G7{0, 0}, GE, va, P, ps, sx, sy, sz{0, 0};
  bool ok = true;
#pragma unroll
  for (int s = 0; s < 2; s++) {
    const IxF ri = ix_inverse(q(s, 0)), mx = ix_load(q(s, 1)), my = ix_load(q(s, 2));
    const IxF bx = ix_load(q(s, 5)), by = ix_load(q(s, 6));
    const IxV f = ix_plus(ix_times(mx, nx), ix_times(my, ny));  // [61]
    const IxF V = ix_up(ix_times(ix_split(f), ri));
    const IxF Bn = ix_up(ix_plus(ix_times(bx, nx), ix_times(by, ny))), bnl = ix_split(ix_times(Bn, ri));
    const IxV w = ix_times(ix_split(ix_minus(ix_times(my, bx), ix_times(mx, by))), ri);  // v Bx - u By: [60]
    const IxV gx = ix_minus(ix_times(mx, V), ix_times(bx, Bn)), gy = ix_minus(ix_times(my, V), ix_times(by, Bn));  // [61]
    IxV k2 = ix_plus(ix_square(mx), ix_square(my)), b2 = ix_plus(ix_square(bx), ix_square(by));
    IxV mB = ix_plus(ix_times(mx, bx), ix_times(my, by));
    if (hasz) {
      const IxF mw = ix_load(q(s, 3)), bz = ix_load(q(s, 7));
      k2 = ix_plus(k2, ix_square(mw));  // [61.6]
      b2 = ix_plus(b2, ix_square(bz));
      mB = ix_plus(mB, ix_times(mw, bz));
      const IxV gz = ix_minus(ix_times(mw, V), ix_times(bz, Bn)), g7 = ix_minus(ix_times(bz, V), ix_times(mw, bnl));
      Gz = s ? ix_plus(Gz, gz) : gz;  // [62]
      G7 = s ? ix_plus(G7, g7) : g7;
      sz = s ? ix_plus(sz, ix_whole(bz)) : ix_whole(bz);
    }
    // 2 p / (gamma - 1) = 2 E - m^2/rho - B^2, the total pressure, E + pt
    const IxF E = ix_load(q(s, 4));
    const IxV kr = ix_times(ix_split(k2), ri);
    const int KS = ix_max(ix_max(E.e + 1, kr.e), b2.e);
    const int64_t S = ix_shr(ix_whole(E).v, KS - E.e - 1) - ix_at(kr, KS) - ix_at(b2, KS);
    ok = ok && S >= 0;
    const IxV p = ix_times(IxF{ix_limbs(S & ~(S >> 63)), KS}, gas.g);  // [60]
    const IxF pt = ix_up(ix_halved(ix_plus(p, IxV{b2.v, b2.e - 1})));
    const IxF Ep = ix_split(ix_halved(ix_plus(ix_whole(E), ix_whole(pt))));
    const IxV ge = ix_minus(ix_times(Ep, V), ix_times(ix_up(ix_halved(mB)), bnl));  // [61]
    F0 = s ? ix_plus(F0, f) : f;  // [62]
    W = s ? ix_plus(W, w) : w;    // [61]
    Gx = s ? ix_plus(Gx, gx) : gx;
    Gy = s ? ix_plus(Gy, gy) : gy;
    GE = s ? ix_plus(GE, ge) : ge;
    va = s ? ix_plus(va, ix_whole(V)) : ix_whole(V);  // [62]
    P = s ? ix_plus(P, p) : p;  // [61]
    ps = s ? ix_plus(ps, ix_whole(pt)) : ix_whole(pt);  // [62]
    sx = s ? ix_plus(sx, ix_whole(bx)) : ix_whole(bx);
    sy = s ? ix_plus(sy, ix_whole(by)) : ix_whole(by);
  }
  // ---- wave speed: with P = gamma (pl + pr), B twice the averaged field, T = P + |B|^2 / 2 and
  // rs = rho_l + rho_r, cf^2 = (T + sqrt(T^2 - 2 P bn^2)) / (2 rs).  Operands are shifted up to full
  // length before they are multiplied on: a field that reverses across the face leaves B far below
  // either side's (with its leading zeros the speed lost up to 2^-26 of itself at a beta of 1e-8)
  P = ix_times(ix_split(P), gas.gam);
  if (!ok || P.v <= 0) return false;
  IxF eig;  // -eigv
  {
    const IxF Pl = ix_up(P), Bx = ix_up(ix_halved(sx)), By = ix_up(ix_halved(sy));
    IxV D = ix_plus(ix_square(Bx), ix_square(By));
    if (hasz) D = ix_plus(D, ix_square(ix_up(ix_halved(sz))));  // [61.6]
    const IxF bn = ix_up(ix_plus(ix_times(Bx, nx), ix_times(By, ny)));
    const IxF T = ix_up(ix_halved(ix_plus(ix_whole(Pl), IxV{D.v, D.e - 1})));
    IxV N = ix_times(Pl, ix_up(ix_square(bn)));
    N.e++;
    const IxV disc = ix_minus(ix_square(T), N);
    if (disc.v < 0) return false;
    IxV U = ix_halved(ix_whole(T));  // [60]
    if (disc.v > 0) {
      IxV sq;
      sq.v = ix_sqrt(disc.v, disc.e, sq.e);  // at most T
      U.v += ix_shr(sq.v, U.e - sq.e);       // [61]
    }
    const int64_t rs = ix_align<3>(q(0, 0), mr) + ix_align<3>(q(1, 0), mr);  // 2^60 < rs < 2^62
    const int up = rs < ((int64_t)1 << 61) ? 1 : 0;
    const IxF irs{ix_limbs(ix_rcp(ix_shl(rs, up))), up - 122 - ix_exp<3>(mr)};
    const IxV cf2 = ix_times(ix_split(U), irs);
    IxV cf;
    cf.v = ix_sqrt(cf2.v, cf2.e - 1, cf.e);  // [61]
    va.v = va.v < 0 ? -va.v : va.v;
    const int K = ix_max(va.e - 1, cf.e) + 1;
    const int64_t ev = ix_shr(va.v, K - va.e + 1) + ix_at(cf, K);  // [61.6]
    eig = IxF{ix_limbs(-ev), K};
    eigv = ix_double(ev, K);
  }
  const IxF sc = ix_load(scale);
  // - eigv (qr - ql) of variable k: one FP64 subtraction (the pipe has room), so that small
  // differences keep their bits
  auto jump = [&](int k) { return ix_times(ix_load(q(1, k) - q(0, k)), eig); };  // [60.6]
  auto scaled = [&](IxV a, IxV b) { return ix_double(ix_times(ix_up(ix_halved(ix_plus(a, b))), sc)); };  // a + b: [62.6]
  double f0 = scaled(F0, jump(0)), f1;
  {
    const IxF pt = ix_up(ix_halved(ps));
    f1 = scaled(ix_plus(Gx, ix_times(pt, nx)), jump(1));
    out(0, f0, f1);
    f0 = scaled(ix_plus(Gy, ix_times(pt, ny)), jump(2));
  }
  out(1, f0, hasz ? scaled(Gz, jump(3)) : 0.0);
  f0 = scaled(GE, jump(4));
  {  // induction: (v Bx - u By) (uy, -ux) in the plane
    const IxF w = ix_up(W);
    f1 = scaled(ix_times(w, ny), jump(5));
    out(2, f0, f1);
    IxV d = ix_times(w, nx);
    d.v = -d.v;
    f0 = scaled(d, jump(6));
  }
  out(3, f0, hasz ? scaled(G7, jump(7)) : 0.0);
  return true;
}

}  // namespace chorus
