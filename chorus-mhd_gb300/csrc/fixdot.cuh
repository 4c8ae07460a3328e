// fixdot.cuh -- the fixed line operators (Lmat interpolation, Mmat differentiation)
// applied in integer arithmetic.
//
// GB300 executes FP64 at 2 operations per clock per SM, while its integer pipes take
// 64 lane-operations per clock each and sat nearly idle while these passes were in FP64.  A
// line operator y_k = sum_j C_kj x_j with fixed coefficients is therefore cheaper as an
// integer dot product:
//   * the inputs of one line are aligned to the largest exponent among them and held as
//     58-bit signed integers (5 guard bits below the 53-bit significand of the largest input;
//     smaller inputs lose only bits below 2^-58 of the largest, by truncation),
//   * the coefficients as 59-bit signed integers c = round(C * 2^S), S per operator,
//   * both split into signed limbs h 2^29 + l, |l| <= 2^28; the products of two low limbs are left
//     out, so a term is three 32x32->64 multiply-adds into two 64-bit accumulators,
//   * the sum, rounded to a multiple of 2^58 in the units of the products, is rounded once, to
//     nearest-even, into a double.
// The error stays below one unit in the last place of the line's largest term, as with a
// chain of FP64 fused multiply-adds, whose rounding errors are of that size too.
//
// The stage kernels apply the operators in this form through the mirror symmetry
// (fix_mirror_line, fix_mirror_sums): the solution and flux points are symmetric about the cell
// centre, so the operators satisfy C(NO-1-k, NI-1-j) = sigma C(k, j) (sigma = +1 for the
// interpolation Lmat, -1 for the derivative Mmat) up to the rounding of their construction
// (1e-16 to 2e-15 of the largest coefficient for N = 2..8).  With E_j = X_j + X_{NI-1-j} and
// O_j = X_j - X_{NI-1-j} (exact integers) each pair of mirror outputs k, NO-1-k shares one sum over
// the NI/2 input pairs, U + W and sigma (U - W), so a line takes half the multiply-adds.  The
// coefficients are those of the operator averaged with its mirror image, each within one
// unit of 2^-S of both rows, and the error bound above holds for that operator.  The
// caller keeps the FP64 form for lines with NaN, infinite, huge (above 2^876) or tiny (below
// 2^-957, not zero) inputs, so non-finite states propagate as before.  Zero results are +0;
// results below the normal range are flushed to zero.
//
// fix_dot and what it calls (fix_align, fix_mac, fix_round, fix_split_coef) are the plain form for
// any operator: 57-bit inputs rounded with kFixG = 4 guard bits, unsigned low limbs, four
// multiply-adds a term, the sum truncated to a multiple of 2^58.  No kernel calls it, nor
// fix_apply_mirror, the mirror form for lines of any finite size: they are what the host tests
// compare with exact sums and hold the mirror form against.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FIX_HD __host__ __device__ __forceinline__
#else
#define FIX_HD inline
#endif

namespace chorus {

constexpr int kFixG = 4;       // guard bits of the aligned inputs of the plain form (and of the scale k of all forms)
constexpr int kFixSplit = 29;  // limb split of inputs and coefficients
constexpr int kFixEmaxFast = 1900;  // largest biased input exponent of the integer form

FIX_HD uint64_t fix_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  __builtin_memcpy(&u, &x, 8);
  return u;
#endif
}

FIX_HD double fix_double(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  __builtin_memcpy(&x, &u, 8);
  return x;
#endif
}

FIX_HD int fix_clz64(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)u);
#else
  return u ? __builtin_clzll(u) : 64;
#endif
}

// acc + a b, 32x32->64 signed.  Written as mad.lo.cc / madc.hi because the compiler makes one
// multiply-add instruction of the pair, and a multiplication and two additions of
// `acc += (int64_t)a * b` or of mad.wide (counted: 4 against 12 instructions for a chain of
// four).
FIX_HD int64_t fix_mad(int a, int b, int64_t acc) {
#ifdef __CUDA_ARCH__
  uint32_t lo = (uint32_t)acc, hi = (uint32_t)((uint64_t)acc >> 32);
  // (the low word is written before the factors are read again: early clobber)
  asm("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.s32 %1, %2, %3, %1;" : "+&r"(lo), "+r"(hi) : "r"(a), "r"(b));
  return (int64_t)(((uint64_t)hi << 32) | lo);
#else
  return acc + (int64_t)a * b;
#endif
}

// v >> d, zero for d > 63
FIX_HD uint64_t fix_shru(uint64_t v, int d) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(d));  // clamps the amount
  return r;
#else
  return d < 64 ? v >> d : 0;
#endif
}

// biased exponent field of x
FIX_HD int fix_exp(double x) { return (int)((fix_bits(x) >> 52) & 0x7ff); }

// the largest biased exponent over a line of NI values (at least 1, the exponent of
// the subnormals)
template <int NI>
FIX_HD int fix_emax(const double (&v)[NI]) {
  int e = 1;
#pragma unroll
  for (int j = 0; j < NI; j++) {
    const int ej = fix_exp(v[j]);
    e = ej > e ? ej : e;
  }
  return e;
}

// aligned integers of a line: X_j = x_j 2^(1075 + G - emax), rounded to the nearest
// integer (ties away from zero in magnitude); |X_j| < 2^57
template <int NI>
FIX_HD void fix_align_x(const double (&v)[NI], int emax, int64_t (&X)[NI]) {
#pragma unroll
  for (int j = 0; j < NI; j++) {
    const uint64_t u = fix_bits(v[j]);
    const int e = (int)((u >> 52) & 0x7ff);
    int d = emax - (e ? e : 1);  // zeros and subnormals have exponent 1, no hidden bit
    d = d < 63 ? d : 63;         // inputs 2^-59 below the largest vanish
    const uint64_t m = ((u & 0xfffffffffffffull) | (e ? 0x10000000000000ull : 0ull)) << kFixG;
    const int64_t x = (int64_t)((m + ((1ull << d) >> 1)) >> d);  // rounded to the nearest unit
    X[j] = (u >> 63) ? -x : x;
  }
}

// limbs x = h 2^29 + l, 0 <= l < 2^29 (h keeps the sign)
FIX_HD void fix_split(int64_t x, int& h, int& l) {
  h = (int)(x >> kFixSplit);
  l = (int)(x & ((1 << kFixSplit) - 1));
}

// aligned limbs of a line: X_j = h_j 2^29 + l_j
template <int NI>
FIX_HD void fix_align(const double (&v)[NI], int emax, int (&h)[NI], int (&l)[NI]) {
  int64_t X[NI];
  fix_align_x(v, emax, X);
#pragma unroll
  for (int j = 0; j < NI; j++) fix_split(X[j], h[j], l[j]);
}

// one term of a dot product in limbs: 2^58 h ch + 2^29 (h cl + l ch) + l cl
FIX_HD void fix_mac(int h, int l, int ch, int cl, int64_t& A, int64_t& B, int64_t& D) {
  A += (int64_t)h * ch;
  B += (int64_t)h * cl;
  B += (int64_t)l * ch;
  D += (int64_t)l * cl;
}

// the sum A 2^58 + B 2^29 + D rounded into a double scaled by 2^k (k = emax - 1017 - G - S:
// the sum is V 2^58 in units of 2^(emax - 1075 - G - S)); the shifts are arithmetic, so D
// may be negative (a difference of two sums)
FIX_HD double fix_round(int64_t A, int64_t B, int64_t D, int k) {
  B += D >> kFixSplit;
  const int64_t V = A + (B >> kFixSplit);  // floor(sum c X / 2^58)
  const uint64_t sgn = (uint64_t)V & 0x8000000000000000ull;
  const uint64_t u = V < 0 ? (uint64_t)(-V) : (uint64_t)V;
  if (u == 0) return 0.0;
  const int lz = fix_clz64(u);
  const uint64_t top = u << lz;
  uint64_t mant = top >> 11;
  const uint64_t rem = top & 0x7ff;
  mant += (rem > 0x400 || (rem == 0x400 && (mant & 1))) ? 1 : 0;
  const int E = k + 1086 - lz;  // biased exponent of mant * 2^(11 - lz + k)
  if (E < 1) return fix_double(sgn);  // below the normal range: flushed to zero
  return fix_double(sgn | (((uint64_t)(E - 1) << 52) + mant));
}

// sum of ch, cl against the aligned limbs, rounded into a double scaled by 2^k
template <int NI>
FIX_HD double fix_dot(const int (&h)[NI], const int (&l)[NI], const int* ch, const int* cl, int k) {
  int64_t A = 0, B = 0, D = 0;  // |A| < 2^61.2, |B| < 2^62.5, 0 <= D < 2^61.2 for NI <= 9
#pragma unroll
  for (int j = 0; j < NI; j++) fix_mac(h[j], l[j], ch[j], cl[j], A, B, D);
  return fix_round(A, B, D, k);
}

// the line's largest magnitude word: the high 31 bits of the largest |x| (0 for a line of
// zeros and of values below 2^-1042)
template <int NI>
FIX_HD uint32_t fix_amax(const double (&v)[NI]) {
  uint32_t a = 0;
#pragma unroll
  for (int j = 0; j < NI; j++) {
    const uint32_t aj = (uint32_t)(fix_bits(v[j]) >> 32) & 0x7fffffffu;
    a = aj > a ? aj : a;
  }
  return a;
}

// Does fix_mirror_line take a line whose largest magnitude word is a?  Lines of zeros and
// those whose largest exponent lies between kFixEmaxMin and kFixEmaxFast: below, results
// could leave the normal range, above, infinities and NaNs have to propagate.
constexpr int kFixEmaxMin = 66;
FIX_HD bool fix_line_ok(uint32_t a) {
  return a == 0 || a - ((uint32_t)kFixEmaxMin << 20) < ((uint32_t)(kFixEmaxFast + 1 - kFixEmaxMin) << 20);
}

// V 2^k' (|V| < 2^63) rounded to nearest, k' = k - 1 with k as in fix_round; CHECK: results
// below the normal range are flushed to zero (otherwise the caller knows that there are
// none); ties up in magnitude, or (EVEN) to even as the conversion instruction rounds them
template <bool CHECK, bool EVEN = false>
FIX_HD double fix_round_v(int64_t V, int k) {
  const int64_t s = V >> 63;
  const uint64_t u = (uint64_t)((V ^ s) - s);
  uint32_t uh = (uint32_t)(u >> 32), ul = (uint32_t)u;
  int e = k + 1084;  // biased exponent of a value whose leading bit is bit 63, less one
  if (uh == 0) {     // at most 32 bits are left
    uh = ul >> 1;
    ul <<= 31;
    e -= 31;
  }
#ifdef __CUDA_ARCH__
  const int lz = __clz((int)uh);
#else
  const int lz = uh ? __builtin_clz(uh) : 32;
#endif
  const uint64_t top = (((uint64_t)uh << 32) | ul) << (lz - 1);                      // leading bit 62 (lz >= 1)
  const uint64_t mant = (top + (EVEN ? 0x1ff + ((top >> 10) & 1) : 0x200)) >> 10;  // 2^52 .. 2^53
  const int E = e - lz;
  uint32_t h = (uint32_t)(mant >> 32) + ((uint32_t)E << 20);
  uint32_t l = (uint32_t)mant;
  if (uh == 0 && ul == 0) h = 0;  // (l is 0 too)
  if (CHECK && E < 0) h = l = 0;
  h |= (uint32_t)(s >> 32) & 0x80000000u;
  return fix_double(((uint64_t)h << 32) | l);
}

// the same through the conversion instruction (nearest, ties to even), which takes the FP64
// unit of its scheduler for 64 clocks but saves some 20 instructions.  The exponent is added to the
// bits, here as there, so a result past the largest double would come out as some other number:
// the callers' windows keep |V 2^k'| below 2^1023.
template <bool CHECK>
FIX_HD double fix_cvt_v(int64_t V, int k) {
#ifdef __CUDA_ARCH__
  const uint64_t d = (uint64_t)__double_as_longlong(__ll2double_rn(V));
#else
  const uint64_t d = fix_bits((double)V);
#endif
  const uint32_t hi = (uint32_t)(d >> 32);
  if (CHECK && (int)((hi >> 20) & 0x7ff) + k - 1 < 1) return 0.0;
  const uint32_t h = hi == 0 ? 0 : hi + ((uint32_t)(k - 1) << 20);
  return fix_double(((uint64_t)h << 32) | (uint32_t)d);
}
// y = C v for C (NO x NI) in mirror form (fix_mirror_coefs: per row r < (NO+1)/2 the
// coefficients [P(0..NI/2) | Q(0..NI/2) | R]), scaled by 2^k as fix_dot.  With
// E_j = X_j + X_{NI-1-j}, O_j = X_j - X_{NI-1-j}, U = sum P E (+ R X_m for odd NI) and
// W = sum Q O: y_r = U + W, y_{NO-1-r} = sigma (U - W).  The middle row of an odd NO has
// only U (sigma = +1) or only W (sigma = -1): the other half is exactly zero.
//
// What bounds the passes that call this is the number of integer instructions, most of
// them the alignment of the inputs and the rounding of the outputs, so:
//  - X = |x| 2^(1080 - emax), 58 bits truncated (5 guard bits): the significand is placed
//    at the top of 64 bits, with its hidden bit whatever the exponent (an input that has
//    none is below the line's largest by more than 64 bits and is shifted out), and
//    shifted right once; the truncation error equals that of rounding with 4 guard bits;
//  - the limbs of E, O and of the coefficients are h 2^29 + l with |l| <= 2^28 (signed), so
//    that the products of two low limbs can be left out: at most NI / 4 units of 2^-58 of
//    the largest term, of either sign, against the one unit, always downwards, that
//    truncating the sum used to take; three multiply-adds a term instead of four;
//  - the sum is rounded to a multiple of 2^58 (2^28 in the start value of B).
// A derivative line of six inputs and five outputs went from about 635 to 350 instructions;
// 512x512 cells, N = 5 (GB300): E3 1.361 -> 1.150 ms per stage, the step 18.2 -> 17.2 ms.
// Bounds for NI <= 9 with |P +- Q| < 2^59, |X| < 2^58: |A| < 9 2^59, and the partial sums
// over U or W alone < 4 2^60 + 2^59; |B| < 9 (2^58 + 2^58) + 2^28: all below 2^63.
//
// fix_mirror_sums hands out the sums V of the rows as they are formed, put(row, V): y =
// V 2^(k-1) with k as in fix_dot, |V| at most the row's sum of |c|, below 2^62.2;
// fix_mirror_core the same from aligned integers X of exponent e: y = V 2^(e + 58 - S).
template <int NO, int NI, int SIGMA, class Put>
FIX_HD void fix_mirror_core(const int64_t (&X)[NI], const int* ch, const int* cl, Put&& put) {  // |X| < 2^58
  constexpr int NP = NI / 2;
  constexpr int64_t kHalfL = (int64_t)1 << (kFixSplit - 1);
  auto split = [](int64_t x, int& h, int& l) {  // x offset by half a limb
    h = (int)(x >> kFixSplit);
    l = (int)(x & ((1 << kFixSplit) - 1)) - (1 << (kFixSplit - 1));
  };
  // limbs of -x are those of x negated (half a limb is rounded away from zero), so that the products
  // left out are too: a mirrored line, whose O change sign, has the mirrored sums to the bit
  auto split_odd = [](int64_t x, int& h, int& l) {
    h = (int)((x + kHalfL + (x >> 63)) >> kFixSplit);
    l = (int)((uint32_t)x - ((uint32_t)h << kFixSplit));
  };
  int eh[NP > 0 ? NP : 1], el[NP > 0 ? NP : 1], oh[NP > 0 ? NP : 1], ol[NP > 0 ? NP : 1];
#pragma unroll
  for (int j = 0; j < NP; j++) {
    split(X[j] + X[NI - 1 - j] + kHalfL, eh[j], el[j]);
    split_odd(X[j] - X[NI - 1 - j], oh[j], ol[j]);
  }
  int mh = 0, ml = 0;
  if (NI & 1) split(X[NP] + kHalfL, mh, ml);
#pragma unroll
  for (int r = 0; r < (NO + 1) / 2; r++) {
    const int* rh = ch + r * NI;
    const int* rl = cl + r * NI;
    const bool mid = (NO & 1) && r == NO / 2;
    int64_t Au = 0, Bu = kHalfL, Aw = 0, Bw = 0;
    if (!mid || SIGMA > 0) {
#pragma unroll
      for (int j = 0; j < NP; j++) {
        Au = fix_mad(eh[j], rh[j], Au);
        Bu = fix_mad(eh[j], rl[j], Bu);
        Bu = fix_mad(el[j], rh[j], Bu);
      }
      if (NI & 1) {
        Au = fix_mad(mh, rh[2 * NP], Au);
        Bu = fix_mad(mh, rl[2 * NP], Bu);
        Bu = fix_mad(ml, rh[2 * NP], Bu);
      }
    }
    if (!mid || SIGMA < 0) {
#pragma unroll
      for (int j = 0; j < NP; j++) {
        Aw = fix_mad(oh[j], rh[NP + j], Aw);
        Bw = fix_mad(oh[j], rl[NP + j], Bw);
        Bw = fix_mad(ol[j], rh[NP + j], Bw);
      }
    }
    put(r, Au + Aw + ((Bu + Bw) >> kFixSplit));
    if (!mid) {
      const int64_t V = Au - Aw + ((Bu - Bw) >> kFixSplit);
      put(NO - 1 - r, SIGMA > 0 ? V : -V);
    }
  }
}

template <int NO, int NI, int SIGMA, class Put>
FIX_HD void fix_mirror_sums(const double (&v)[NI], int emax, const int* ch, const int* cl, Put&& put) {
  int64_t X[NI];
  const uint32_t eb = ((uint32_t)emax << 20) | 0xfffffu;
#pragma unroll
  for (int j = 0; j < NI; j++) {
    const uint64_t u = fix_bits(v[j]);
    const uint32_t a = (uint32_t)(u >> 32) & 0x7fffffffu;
    const uint32_t d = (eb + (6u << 20) - a) >> 20;  // emax - exponent + 6
    const uint64_t t = (u << 11) | 0x8000000000000000ull;
    const int64_t x = (int64_t)fix_shru(t, (int)d);
    X[j] = (int64_t)u < 0 ? -x : x;
  }
  fix_mirror_core<NO, NI, SIGMA>(X, ch, cl, put);
}

template <int NO, int NI, int SIGMA, bool CHECK>
FIX_HD void fix_mirror_line(const double (&v)[NI], int emax, const int* ch, const int* cl, int k, double (&y)[NO]) {
  fix_mirror_sums<NO, NI, SIGMA>(v, emax, ch, cl, [&](int r, int64_t V) { y[r] = r < NO / 2 ? fix_cvt_v<CHECK>(V, k) : fix_round_v<CHECK, true>(V, k); });
}

// the same for any finite line with emax <= kFixEmaxFast: lines below kFixEmaxMin are scaled
// up by 2^200 (exact) and their results back
template <int NO, int NI, int SIGMA>
FIX_HD void fix_apply_mirror(const double (&v)[NI], int emax, const int* ch, const int* cl, int k, double (&y)[NO]) {
  if (emax >= kFixEmaxMin) {
    fix_mirror_line<NO, NI, SIGMA, true>(v, emax, ch, cl, k, y);
    return;
  }
  double w[NI];
#pragma unroll
  for (int j = 0; j < NI; j++) w[j] = v[j] * 0x1p200;
  const int ew = fix_emax(w);
  const int em = ew > kFixEmaxMin ? ew : kFixEmaxMin;  // (a line of zeros)
  fix_mirror_line<NO, NI, SIGMA, true>(w, em, ch, cl, k - emax + em - 200, y);
}

// integer form of coefficients (host side): c = round(C 2^S), S the largest shift that
// keeps every |c| below 2^59 (S = 59 - e for max |C| in [2^(e-1), 2^e))
inline int fix_shift_for(const double* C, int n) {
  double mx = 0.0;
  for (int i = 0; i < n; i++) mx = C[i] > mx ? C[i] : (-C[i] > mx ? -C[i] : mx);
  if (mx == 0.0) return 59;
  int e;
  __builtin_frexp(mx, &e);
  return 59 - e;
}

// round(C 2^S) (ties away from zero), exact: |C 2^S| < 2^59
inline int64_t fix_coef(double C, int S) {
  double t = C;
  for (int i = 0; i < S; i++) t *= 2.0;  // exact scaling by 2^S
  const double r = t < 0 ? -__builtin_floor(-t + 0.5) : __builtin_floor(t + 0.5);
  return (int64_t)r;
}

// split c = ch 2^29 + cl with 0 <= cl < 2^29
inline void fix_split_coef(double C, int S, int* ch, int* cl) {
  const int64_t c = fix_coef(C, S);
  *ch = (int)(c >> kFixSplit);
  *cl = (int)(c & ((1 << kFixSplit) - 1));
}

// c = ch 2^29 + cl with -2^28 <= cl < 2^28
inline void fix_split_signed(int64_t c, int* ch, int* cl) {
  const int64_t half = (int64_t)1 << (kFixSplit - 1);
  *ch = (int)((c + half) >> kFixSplit);
  *cl = (int)((c + half) & ((1 << kFixSplit) - 1)) - (int)half;
}

// the mirror form of C (NO x NI, row-major C[k NI + j], C(NO-1-k, NI-1-j) = sigma C(k, j)
// up to rounding) for fix_apply_mirror: for each row k < (NO+1)/2, k' = NO-1-k, and input
// pair j < NI/2, j' = NI-1-j, from the integers c = round(C 2^S),
//   P(k,j) = (c(k,j) + c(k,j') + sigma c(k',j') + sigma c(k',j)) / 4
//   Q(k,j) = (c(k,j) - c(k,j') + sigma c(k',j') - sigma c(k',j)) / 4
//   R(k)   = (c(k,m) + sigma c(k',m)) / 2          (middle input m of an odd NI)
// each an exact 64-bit sum rounded once (half up), stored in limbs per row as
// [P(0..NI/2) | Q(0..NI/2) | R].  P + Q and P - Q, the coefficients of inputs j and j' in
// row k, lie within one unit of the average of row k and the mirror image of row k'.
inline void fix_mirror_coefs(const double* C, int NO, int NI, int sigma, int S, int* ch, int* cl) {
  const int NP = NI / 2;
  for (int k = 0; k < (NO + 1) / 2; k++) {
    const int kk = NO - 1 - k;
    auto c = [&](int row, int j) { return fix_coef(C[row * NI + j], S); };
    for (int j = 0; j < NP; j++) {
      const int jj = NI - 1 - j;
      const int64_t p = (c(k, j) + c(k, jj) + sigma * (c(kk, jj) + c(kk, j)) + 2) >> 2;
      const int64_t q = (c(k, j) - c(k, jj) + sigma * (c(kk, jj) - c(kk, j)) + 2) >> 2;
      fix_split_signed(p, &ch[k * NI + j], &cl[k * NI + j]);
      fix_split_signed(q, &ch[k * NI + NP + j], &cl[k * NI + NP + j]);
    }
    if (NI & 1) {
      const int64_t r = (c(k, NP) + sigma * c(kk, NP) + 1) >> 1;
      fix_split_signed(r, &ch[k * NI + 2 * NP], &cl[k * NI + 2 * NP]);
    }
  }
}

}  // namespace chorus
