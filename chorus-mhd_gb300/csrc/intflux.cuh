// intflux.cuh -- the ideal-MHD point fluxes in integer arithmetic.
//
// GB300 executes FP64 at 2 lane-operations per clock per SM (a warp instruction occupies
// its scheduler's FP64 unit for 64 clocks), the integer pipes take 64 each.  The nonlinear
// fluxes are products and sums of few variables, so they are evaluated as block fixed-point
// numbers: a value is v 2^e with a 64-bit integer v and an exponent e that a group of
// quantities shares, products keep the upper part of the 128-bit product of two such
// integers, sums align to the larger exponent, and each result is rounded once into a
// double.
//
//   * Groups: the x and y components of the momentum (of both sides of a face), their z
//     components, the same for B, the energies, the densities.  The z components have
//     exponents of their own because they can be small and decoupled from the plane.
//   * A product takes the operands as limbs v = h 2^31 + l (0 <= l < 2^31):
//     (a b) >> 62 = ha hb + ((ha lb + la hb) >> 31) in three 32x32->64 multiply-adds; the
//     product of the low limbs is below one unit and left out.
//   * Values keep 57 to 61 significant bits relative to the largest term of their sum, so
//     the errors before the final rounding stay below those of the FP64 chain, which
//     rounds every intermediate to 53 bits.
//
// The integer form takes finite states with a normal positive density and exponents within
// a wide window (2^-200 .. 2^200; zero and smaller values of momentum and B as well); everything else (infinities, NaNs, zero or negative
// density, a density ratio above 8 across a face, a negative discriminant) is left to the
// FP64 form, whose results on such states the caller keeps.
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

// a sum of products, >> 62 at the end
struct IxSum {
  int64_t A = 0, T = 0;
  FIX_HD void add(Limbs a, Limbs b) {
    T = fix_mad(a.h, b.l, T);
    T = fix_mad(a.l, b.h, T);
    A = fix_mad(a.h, b.h, A);
  }
  FIX_HD void square(Limbs a) {  // half of the cross terms: value() with shift 30
    T = fix_mad(a.h, a.l, T);
    A = fix_mad(a.h, a.h, A);
  }
  FIX_HD int64_t value() const { return A + (T >> 31); }
  FIX_HD int64_t value2() const { return ix_shl(A, 1) + (T >> 30); }  // >> 61
  FIX_HD int64_t value4() const { return ix_shl(A, 2) + (T >> 29); }  // >> 60
  FIX_HD int64_t value4_squares() const { return ix_shl(A, 2) + (T >> 28); }
};

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

// v >> d, or v << -d (where the caller knows that it fits)
FIX_HD int64_t ix_shift(int64_t v, int d) { return d >= 0 ? ix_shr(v, d) : ix_shl(v, -d); }

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

// limbs of v shifted up to [60] where it is below that, with its exponent; and of a pair
FIX_HD Limbs ix_up(int64_t v, int& e) {
  const int n = ix_room(v, 3);
  e -= n;
  return ix_limbs(ix_shl(v, n));
}
FIX_HD void ix_up2(int64_t a, int64_t b, int& e, Limbs& la, Limbs& lb) {
  const int n = ix_room((a ^ (a >> 63)) | (b ^ (b >> 63)), 3);
  e -= n;
  la = ix_limbs(ix_shl(a, n));
  lb = ix_limbs(ix_shl(b, n));
}

// constants of a solve, prepared once (host or device): half of gamma - 1, gamma, as limbs
// of normalised integers in [2^60, 2^61) with their exponents
struct IxGas {
  Limbs g, gam;
  int eg, egam;
  Limbs kap;  // gamma / Pr
  int ekap;
  int eh;  // E + p + B^2/2 <= (1 + gamma) E, as p >= 0 and B^2/2 <= E: below 2^(eh + 0.7) E
};
FIX_HD IxGas ix_gas(double gamma) {
  IxGas c;
  const double gm = 0.5 * (gamma - 1.0);
  c.g = ix_limbs(ix_align<3>(gm, ix_abs_word(gm)));
  c.eg = ix_exp<3>(ix_abs_word(gm));
  c.gam = ix_limbs(ix_align<3>(gamma, ix_abs_word(gamma)));
  c.egam = ix_exp<3>(ix_abs_word(gamma));
  const double kp = gamma / 0.72;
  c.kap = ix_limbs(ix_align<3>(kp, ix_abs_word(kp)));
  c.ekap = ix_exp<3>(ix_abs_word(kp));
  for (c.eh = 1; c.eh < 60 && 1.0 + gamma > 1.62 * (double)(1LL << c.eh); c.eh++) {
  }
  return c;
}


// a product as an increment of a sum: (a b) >> 61
FIX_HD int64_t ix_prod(Limbs a, Limbs b) {
  IxSum p;
  p.add(a, b);
  return p.value2();
}

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
  const IxF P = ix_up(ix_halved(ix_plus(ix_times(IxF{ix_limbs(S), KS}, IxF{gas.g, gas.eg}), IxV{b2.v, b2.e - 1})));
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
// place.  [b] in the comments means a magnitude below 2^b.
template <class Q, class G, class Out>
FIX_HD bool vflux_int(Q&& q, G&& g, double mut, double eta, double sx, double sy, const IxGas& gas, Out&& out) {
  const uint32_t zero = 66u << 20;  // a group of zeros: zeros are shifted out at this exponent
  auto w1 = [&](int k) { return ix_max(zero, ix_abs_word(q(k))); };
  auto w2 = [&](int k) { return ix_max(zero, ix_max(ix_abs_word(g(0, k)), ix_abs_word(g(1, k)))); };
  const uint32_t r = (uint32_t)(fix_bits(q(0)) >> 32);  // huge if the sign is set
  const uint32_t mm = ix_max(w1(1), w1(2)), mz = w1(3), me = w1(4), mb = ix_max(w1(5), w1(6)), mw = w1(7);
  const uint32_t gr = w2(0), gm = ix_max(w2(1), w2(2)), gz = w2(3), ge = w2(4), gb = ix_max(w2(5), w2(6)), gw = w2(7);
  const uint32_t ms = ix_max(ix_abs_word(sx), ix_abs_word(sy));
  const uint32_t mu = ix_max(zero, ix_abs_word(mut)), mt = ix_max(zero, ix_abs_word(eta));
  const uint32_t top = ix_max(ix_max(ix_max(ix_max(r, mm), ix_max(mz, me)), ix_max(ix_max(mb, mw), ix_max(ms, mu))),
                              ix_max(ix_max(ix_max(gr, gm), ix_max(gz, ge)), ix_max(ix_max(gb, gw), mt)));
  if (top >= kIxHigh || r < kIxLow || ms < kIxLow) return false;
  const bool hasz = ix_max(ix_max(mz, mw), ix_max(gz, gw)) != zero;
  const int em = ix_exp<4>(mm), eB = ix_exp<4>(mb), eS = ix_exp<4>(ms), e_ri = -122 - ix_exp<2>(r);
  const int egr = ix_exp<4>(gr), egm = ix_exp<4>(gm), egB = ix_exp<4>(gb);
  const Limbs nx = ix_limbs(ix_align<4>(sx, ms)), ny = ix_limbs(ix_align<4>(sy, ms));  // [60]
  const Limbs ri = ix_limbs(ix_rcp(ix_align<2>(q(0), r)));                             // [61]
  int eM = ix_exp<3>(mu) + e_ri + 62;
  const Limbs M = ix_up(ix_mul(ix_align<3>(mut, mu), ri), eM);                         // [60] mu / rho
  auto contracted = [&](Limbs a, Limbs b) {  // a sx + b sy: [60.5], exponent of a + eS + 60
    IxSum t;
    t.add(a, nx); t.add(b, ny);
    return t.value4();
  };
  // velocities, m^2 + ... of the internal energy: X = |u|^2 + B^2/(2 rho) - E/rho
  const Limbs mx = ix_limbs(ix_align<4>(q(1), mm)), my = ix_limbs(ix_align<4>(q(2), mm));  // [60]
  int eu = em + e_ri + 61;
  Limbs u, v;  // [60]
  ix_up2(ix_prod(mx, ri), ix_prod(my, ri), eu, u, v);
  const Limbs bx = ix_limbs(ix_align<4>(q(5), mb)), by = ix_limbs(ix_align<4>(q(6), mb));
  IxSum k2, b2;
  k2.square(mx); k2.square(my);
  b2.square(bx); b2.square(by);
  int64_t kv = k2.value4_squares(), bv = b2.value4_squares();  // [61]
  int ek = 2 * em + 60, eB2 = 2 * eB + 60;
  Limbs w{0, 0}, bz{0, 0};
  int ew = 0, eBz = 0;
  if (hasz) {
    const int emz = ix_exp<4>(mz);
    eBz = ix_exp<4>(mw);
    const int km = ix_max(em, emz), kb = ix_max(eB, eBz);
    const Limbs mzl = ix_limbs(ix_align<4>(q(3), mz));
    bz = ix_limbs(ix_align<4>(q(7), mw));
    IxSum a, b;
    a.square(mzl); b.square(bz);
    kv = ix_shr(kv, 2 * (km - em)) + ix_shr(a.value4_squares(), 2 * (km - emz));  // [61.6]
    bv = ix_shr(bv, 2 * (kb - eB)) + ix_shr(b.value4_squares(), 2 * (kb - eBz));
    ek = 2 * km + 60;
    eB2 = 2 * kb + 60;
    ew = emz + e_ri + 61;
    w = ix_up(ix_prod(mzl, ri), ew);
  }
  ek += e_ri + 62;
  const int eE = ix_exp<3>(me), KY = ix_max(ix_max(ek, eB2 - 1), eE) + 1;
  int eX = KY + e_ri + 62;
  const Limbs X = ix_up(ix_mul(ix_shr(ix_mul(kv, ri), KY - ek) + ix_shr(bv, KY - eB2 + 1) - ix_shr(ix_align<3>(q(4), me), KY - eE), ri), eX);  // [60]
  // gradients of the density, and rho times those of the plane's velocity
  const Limbs rx = ix_limbs(ix_align<4>(g(0, 0), gr)), ry = ix_limbs(ix_align<4>(g(1, 0), gr));
  int erS = egr + eS + 60;
  const Limbs rS = ix_up(contracted(rx, ry), erS);  // [60]
  const int ep = egr + eu + 61, Kw = ix_max(egm, ep) + 1;
  Limbs c1, c2;
  int64_t t2;  // u.(grad m . S) of the plane
  int ec = Kw + eS + 61, e2 = egm + eS + 60;
  {
    const int64_t ax = ix_align<4>(g(0, 1), gm), ay = ix_align<4>(g(1, 1), gm);
    const int64_t bx_ = ix_align<4>(g(0, 2), gm), by_ = ix_align<4>(g(1, 2), gm);
    Limbs mxS, myS;
    ix_up2(contracted(ix_limbs(ax), ix_limbs(ay)), contracted(ix_limbs(bx_), ix_limbs(by_)), e2, mxS, myS);
    t2 = ix_prod(mxS, u) + ix_prod(myS, v);  // [60]
    e2 += eu + 61;
    auto rel = [&](int64_t a, Limbs r_, Limbs u_) { return ix_shr(a, Kw - egm) - ix_shr(ix_prod(r_, u_), Kw - ep); };  // [60]
    const int64_t ux = rel(ax, rx, u), uy = rel(ay, ry, u), vx = rel(bx_, rx, v), vy = rel(by_, ry, v);
    const Limbs two3{(int)(1537228672809129301LL >> 31), (int)(1537228672809129301LL & 0x7fffffff)};  // 2^62 / 3
    const int64_t ld = ix_prod(ix_limbs(ux + vy), two3);  // 2/3 of the divergence: [60.5]
    const Limbs a = ix_limbs(ux + ux - ld), b = ix_limbs(uy + vx), d = ix_limbs(vy + vy - ld);  // [61.7]
    ix_up2(ix_prod(a, nx) + ix_prod(b, ny), ix_prod(b, nx) + ix_prod(d, ny), ec, c1, c2);  // [61.4], [60] if shifted
  }
  out(1, ix_double(ix_mul(c1, M), ec + eM + 62));
  out(2, ix_double(ix_mul(c2, M), ec + eM + 62));
  // energy: M (u.c + gamma/Pr H), H = grad E.S - u.(grad m.S) - B.(grad B.S) + X grad rho.S
  const uint32_t gE = ge;
  const int e1 = ix_exp<4>(gE) + eS + 60, e4 = eX + erS + 61;
  int e3 = egB + eS + 60;
  const int64_t t1 = contracted(ix_limbs(ix_align<4>(g(0, 4), gE)), ix_limbs(ix_align<4>(g(1, 4), gE)));
  const int64_t yx = ix_align<4>(g(0, 6), gb), xy = ix_align<4>(g(1, 5), gb);
  Limbs bxS, byS;
  ix_up2(contracted(ix_limbs(ix_align<4>(g(0, 5), gb)), ix_limbs(xy)), contracted(ix_limbs(yx), ix_limbs(ix_align<4>(g(1, 6), gb))), e3,
         bxS, byS);
  const int64_t t3 = ix_prod(bxS, bx) + ix_prod(byS, by);
  e3 += eB + 61;
  const int64_t t4 = ix_prod(X, rS);
  int KH = ix_max(ix_max(e1, e2), ix_max(e3, e4)) + 2;
  int64_t H, uc = ix_prod(c1, u) + ix_prod(c2, v);  // [61.4]
  int euc = ec + eu + 61;
  double F3 = 0.0;
  int64_t bzS = 0;
  int ebz = 0;
  if (hasz) {
    const int egz = ix_exp<4>(gz), ez = egz + eS + 60;
    ebz = ix_exp<4>(gw) + eS + 60;
    const int64_t mzS = contracted(ix_limbs(ix_align<4>(g(0, 3), gz)), ix_limbs(ix_align<4>(g(1, 3), gz)));
    bzS = contracted(ix_limbs(ix_align<4>(g(0, 7), gw)), ix_limbs(ix_align<4>(g(1, 7), gw)));
    const int er = erS + ew + 61, K3 = ix_max(ez, er) + 1;
    const int64_t c3 = ix_shr(mzS, K3 - ez) - ix_shr(ix_prod(rS, w), K3 - er);  // [60.5]
    F3 = ix_double(ix_mul(c3, M), K3 + eM + 62);
    const int e5 = ez + ew + 61, e6 = ebz + eBz + 61;
    KH = ix_max(KH, ix_max(e5, e6) + 2);
    H = -ix_shr(ix_prod(ix_limbs(mzS), w), KH - e5) - ix_shr(ix_prod(ix_limbs(bzS), bz), KH - e6);
    const int e7 = K3 + ew + 61, K = ix_max(euc, e7) + 1;
    uc = ix_shr(uc, K - euc) + ix_shr(ix_prod(ix_limbs(c3), w), K - e7);
    euc = K;
  } else {
    H = 0;
  }
  out(3, F3);
  H += ix_shr(t1, KH - e1) - ix_shr(t2, KH - e2) - ix_shr(t3, KH - e3) + ix_shr(t4, KH - e4);  // [61.1]
  const Limbs Hl = ix_up(H, KH);
  const int eH = KH + gas.ekap + 61, K4 = ix_max(euc, eH) + 1;
  int64_t F4 = ix_mul(ix_shr(uc, K4 - euc) + ix_shr(ix_prod(Hl, gas.kap), K4 - eH), M);  // [60]
  int eF4 = K4 + eM + 62;
  double F5 = 0.0, F6 = 0.0, F7 = 0.0;
  if (eta != 0.0) {  // resistive terms: F_B = eta (-Jz sy, Jz sx, grad Bz.S), the energy takes B.F_B
    const Limbs et = ix_limbs(ix_align<3>(eta, mt));
    const int eet = ix_exp<3>(mt);
    int eJ = egB + eet + 62, eR = eB + eS + 60;
    const int64_t j = ix_mul(yx - xy, et);  // [60]
    Limbs jl, jn;
    ix_up2(j, -j, eJ, jl, jn);
    F5 = ix_double(ix_prod(jn, ny), eJ + eS + 61);
    F6 = ix_double(ix_prod(jl, nx), eJ + eS + 61);
    IxSum t;  // By sx - Bx sy
    t.add(by, nx);
    IxSum t_;
    t_.add(bx, ny);
    const Limbs Rl = ix_up(t.value4() - t_.value4(), eR);
    int64_t R = ix_prod(jl, Rl);  // [60.5]
    eR += eJ + 61;
    if (hasz) {
      const int64_t f7 = ix_mul(bzS, et);  // [59.5]
      const int e7 = ebz + eet + 62, e8 = e7 + eBz + 61, K = ix_max(eR, e8) + 1;
      F7 = ix_double(f7, e7);
      R = ix_shr(R, K - eR) + ix_shr(ix_prod(ix_limbs(f7), bz), K - e8);
      eR = K;
    }
    const int K = ix_max(eF4, eR) + 1;
    F4 = ix_shr(F4, K - eF4) + ix_shr(R, K - eR);
    eF4 = K;
  }
  out(4, ix_double(F4, eF4));
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
    const IxV p = ix_times(IxF{ix_limbs(S & ~(S >> 63)), KS}, IxF{gas.g, gas.eg});  // [60]
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
  P = ix_times(ix_split(P), IxF{gas.gam, gas.egam});
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
