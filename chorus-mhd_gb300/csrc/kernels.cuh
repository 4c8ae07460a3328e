// kernels.cuh -- stage kernels of the residual-and-time-step path, templated on N.
//
// One RK stage (compresid.f90:1-67 + the stage update of iterations.f90:162-217) is
// four launches (five on large meshes), one per grid-wide dependency level of the reference's
// compflux:
//   E1  cell pass  Q -> flux-point values (all 2N(N+1) points), interior inviscid
//                  flux, interior A_z, AV sensor and ramp  inviscid_flux_interior,
//                                                          comp_artificial_viscosity
//   F1  face pass  Rusanov flux on every face point, upwinded A_z, max wave speed,
//                  list of the cells with viscous work     interfaceflux, CYCLOCFLUX,
//                                                          BCFLUX, getrusanovflux
//   E2  cell pass  grad Q (vars 1-8) at the solution and flux points of the listed cells
//                  and their neighbours                    nablaQsp, nablaQ_interior_FP
//   V   cell pass  face AV viscosities, viscous + AV flux of the listed cells with the
//                  face-averaged traces                    compAVflux, interfaceVISflux,
//                                                          comp_viscous_flux
//   E3  cell pass  (V's work on small meshes,) divergence, grad A_z, A_z advection, RK
//                  update                                  nablaAsp, compresid, RK_S5P3
// (k_f2 stores the face-averaged grad Q traces only when they are downloaded.)
// Cell passes stage a block of `epb` cells in shared memory; face passes run one
// thread per face point.  Values are IEEE doubles throughout; the fixed line operators
// (Lmat interpolation, Mmat differentiation, which carry no data-dependent
// coefficients) run as integer dot products on the integer pipes (fixdot.cuh), the
// point fluxes in integers with an exponent per value there too (intflux.cuh), all other
// arithmetic is FP64.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "chorus_internal.h"
#include "fixdot.cuh"
#include "intflux.cuh"
#include "physics.cuh"

namespace chorus {

constexpr int kHalfF = kMaxN / 2 + 1;  // flux points up to the middle of a line
constexpr int kHalfS = kMaxN / 2;      // mirrored pairs of solution points

// wait for the predecessor grid of a programmatic (PDL) launch: its completion and its
// memory; a no-op for a launch without the attribute
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch with programmatic stream serialization: the kernel waits (griddepcontrol.wait, at its
// entry) for the predecessor's completion and memory before touching any of its data; the wait
// is hardware-managed.  No pass releases its dependents before it ends, so what overlaps is the
// scheduling of the next pass with the flush of the last one's memory after its last CTA has
// exited: 0.430 -> 0.407 ms a step of 64x64 cells.
template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kern)(KArgs...), int grid, int block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}


struct OpsN {
  double L[(kMaxN + 1) * kMaxN];  // Lmat(N+1,N) column-major
  double M[(kMaxN + 1) * kMaxN];  // Mmat(N+1,N)
  double A[kMaxN * kMaxN];        // AV smoothing operator A[i*N+m] (projection to N-1 points and back)
  double Ar[kMaxN], Al[kMaxN];    // A = 1 - Ar Al^T: the projection drops one polynomial
  double Xf[kMaxN + 1];
  double Xs[kMaxN];
  // Lmat split by the mirror symmetry of the points (Xs and Xf symmetric about 1/2):
  // for flux point f <= N/2 and solution pair (j, N-1-j),
  //   CE[f][j] = (L(f,j) + L(f,N-1-j))/2,  CO[f][j] = (L(f,j) - L(f,N-1-j))/2,
  // LMID[f] = L(f,(N-1)/2) for odd N; then with e_j = q_j + q_{N-1-j},
  // o_j = q_j - q_{N-1-j}: Qf(f) = E + O and Qf(N-f) = E - O,
  // E = sum CE e + LMID q_mid, O = sum CO o.
  double CE[kHalfF * kHalfS];
  double CO[kHalfF * kHalfS];
  double LMID[kHalfF];
  // the integer form of Lmat (fixdot.cuh) in mirror form (fix_mirror_coefs, sigma = +1,
  // C(f, j) = L(f, j): rows f <= N/2 of N limbs) at scale 2^LS
  int LH[(kMaxN + 1) * kMaxN];
  int LL[(kMaxN + 1) * kMaxN];
  int LS;
  // and of Mmat (sigma = -1, C(i, r) = M(r, i), the weight of flux point r in the
  // derivative at solution point i: rows i < (N+1)/2 of N+1 limbs) at scale 2^MS
  int MH[(kMaxN + 1) * kMaxN];
  int ML[(kMaxN + 1) * kMaxN];
  int MS;
  int MV;  // right shift that keeps the sum of two derivative sums (fix_mirror_sums) below 2^62
};

// one copy per translation unit; upload_ops_n<N>() fills it
static __constant__ OpsN c_ops;

// operator accessors: the per-N kernels read their translation unit's single table,
// the multi-solve kernels one table per N
struct OpsTU {
  __device__ static const OpsN& ops() { return c_ops; }
};

template <int N>
struct D {
  static constexpr int NS = N * N;
  static constexpr int NF1 = (N + 1) * N;
  static constexpr int NFP = 2 * NF1;
};

// element-local flux-point index of face point nfp (0-based) of local face lf (1..4),
// from face2fpconnec (initsetup.f90:343-379)
template <int N>
__device__ __forceinline__ int face_fp(int lf, int nfp) {
  constexpr int NF1 = D<N>::NF1;
  switch (lf) {
    case 1: return NF1 + nfp;                   // family 2, ifp = nfp,     jfp = 1
    case 2: return nfp * (N + 1) + N;           // family 1, ifp = N+1,     jfp = nfp
    case 3: return NF1 + N * N + (N - 1 - nfp); // family 2, ifp = N-nfp+1, jfp = N+1
    default: return (N - 1 - nfp) * (N + 1);    // family 1, ifp = 1,       jfp = N-nfp+1
  }
}

// the inverse of face_fp: the local face (1..4) of element flux point fp and its
// position nfp along that face; 0 for an interior flux point
template <int N>
__device__ __forceinline__ int fp_face(int fp, int& nfp) {
  constexpr int NF1 = D<N>::NF1;
  if (fp < NF1) {
    const int ifp = fp % (N + 1), jfp = fp / (N + 1);
    if (ifp == 0) { nfp = N - 1 - jfp; return 4; }
    if (ifp == N) { nfp = jfp; return 2; }
    return 0;
  }
  const int r = fp - NF1, ifp = r % N, jfp = r / N;
  if (jfp == 0) { nfp = ifp; return 1; }
  if (jfp == N) { nfp = N - 1 - ifp; return 3; }
  return 0;
}

__device__ __forceinline__ unsigned long long ev_bits(double ev, unsigned int* err) {
  if (!(ev >= 0.0) || ev > 1.0e300) {  // NaN or inf wave speed: non-physical state
    atomicOr(err, 1u);
    return 0ull;
  }
  return (unsigned long long)__double_as_longlong(ev);
}

__device__ __forceinline__ void block_max_ull(unsigned long long v, unsigned long long* out) {
  __shared__ unsigned long long red[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
    v = w > v ? w : v;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = v;
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    v = lane < nw ? red[lane] : 0ull;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long w = __shfl_xor_sync(0xffffffffu, v, o);
      v = w > v ? w : v;
    }
    if (lane == 0 && v) atomicMax(out, v);
  }
}

// ---------------------------------------------------------------------------
// E1: flux-point values, interior inviscid flux, AV sensor
// ---------------------------------------------------------------------------
// sum of v over the lanes of a warp (all lanes must call)
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// dst[0..n) = src[0..n) by the whole CTA, in 16-byte pieces when both are 16-byte
// aligned (the branch is uniform over the CTA)
__device__ __forceinline__ void block_copy(double* dst, const double* src, int n) {
  if (((reinterpret_cast<uintptr_t>(dst) | reinterpret_cast<uintptr_t>(src)) & 15) == 0) {
    const double2* s2 = reinterpret_cast<const double2*>(src);
    double2* d2 = reinterpret_cast<double2*>(dst);
#pragma unroll 4
    for (int i = threadIdx.x; i < (n >> 1); i += blockDim.x) d2[i] = s2[i];
    if ((n & 1) && threadIdx.x == 0) dst[n - 1] = src[n - 1];
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = src[i];
  }
}

// asynchronous copies into shared memory
__device__ __forceinline__ void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// dst[0..n) = src[0..n) by the whole CTA, asynchronously; dst is 16-byte aligned, src is as its
// place in the array has it (pieces of 16 bytes where it is too)
__device__ __forceinline__ void block_copy_async(double* dst, const double* src, int n) {
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    for (int i = threadIdx.x; i < (n >> 1); i += blockDim.x) cp_async16(dst + 2 * i, src + 2 * i);
    if ((n & 1) && threadIdx.x == 0) cp_async8(dst + n - 1, src + n - 1);
  } else {
    for (int i = threadIdx.x; i < n; i += blockDim.x) cp_async8(dst + i, src + i);
  }
}

// dst[0..n) = src[0..n) by the whole CTA, src in shared memory, in 16-byte stores from the first
// 16-byte boundary of dst on
__device__ __forceinline__ void block_copy_out(double* dst, const double* src, int n) {
  const int head = (int)((reinterpret_cast<uintptr_t>(dst) >> 3) & 1);
  double2* d2 = reinterpret_cast<double2*>(dst + head);
  const int pairs = (n - head) >> 1;
#pragma unroll 4
  for (int i = threadIdx.x; i < pairs; i += blockDim.x) d2[i] = make_double2(src[head + 2 * i], src[head + 2 * i + 1]);
  if (threadIdx.x == 0 && head) dst[0] = src[0];
  if (threadIdx.x == 0 && head + 2 * pairs < n) dst[n - 1] = src[n - 1];
}

// element-local flux-point index of the i-th interior flux point (i < 2N(N-1)):
// family 1 with ifp = 1..N-1, then family 2 with jfp = 1..N-1
template <int N>
__device__ __forceinline__ int interior_fp(int i) {
  constexpr int H = N * (N - 1);
  if (i < H) {
    const int jfp = i / (N - 1), ifp = 1 + i % (N - 1);
    return jfp * (N + 1) + ifp;
  }
  const int r = i - H, jfp = 1 + r / N, ifp = r % N;
  return D<N>::NF1 + jfp * N + ifp;
}

// interpolation along one line from the N solution values to the N+1 flux points,
// y_f = sum_j L(f,j) v_j: the integer form (fixdot.cuh), or FP64 for a line with
// non-finite, huge or tiny values, where the mirror symmetry of the points halves the
// multiplications (see OpsN::CE)
template <int N, class O>
__device__ __forceinline__ void interp_line(const double (&v)[N], double (&y)[N + 1]) {
  const uint32_t am = fix_amax(v);
  if (fix_line_ok(am)) {
    const int emax = max((int)(am >> 20), kFixEmaxMin);
    fix_mirror_line<N + 1, N, 1, false>(v, emax, O::ops().LH, O::ops().LL, emax - 1017 - kFixG - O::ops().LS, y);
    return;
  }
  double ev[N / 2 > 0 ? N / 2 : 1], od[N / 2 > 0 ? N / 2 : 1];
#pragma unroll
  for (int j = 0; j < N / 2; j++) {
    ev[j] = v[j] + v[N - 1 - j];
    od[j] = v[j] - v[N - 1 - j];
  }
#pragma unroll
  for (int f = 0; f <= N / 2; f++) {
    double E = (N & 1) ? O::ops().LMID[f] * v[(N - 1) / 2] : 0.0;
    double Od = 0.0;
#pragma unroll
    for (int j = 0; j < N / 2; j++) {
      E += O::ops().CE[f * kHalfS + j] * ev[j];
      Od += O::ops().CO[f * kHalfS + j] * od[j];
    }
    y[f] = E + Od;
    if (f != N - f) y[N - f] = E - Od;
  }
}

// the derivative along one line, y_i = sum_r M(r,i) x_r (i < N) from the N+1 flux values
// x_r = x[r*xs]: the integer form (fixdot.cuh), or FP64 for a line with non-finite,
// huge or tiny values
template <int N, class O>
__device__ __forceinline__ void deriv_line(const double* x, int xs, double (&y)[N]) {
  double v[N + 1];
#pragma unroll
  for (int r = 0; r <= N; r++) v[r] = x[r * xs];
  const uint32_t am = fix_amax(v);
  if (fix_line_ok(am)) {
    const int emax = max((int)(am >> 20), kFixEmaxMin);
    fix_mirror_line<N, N + 1, -1, false>(v, emax, O::ops().MH, O::ops().ML, emax - 1017 - kFixG - O::ops().MS, y);
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) {
      double a = 0.0;
#pragma unroll
      for (int r = 0; r <= N; r++) a += O::ops().M[r + (N + 1) * i] * v[r];
      y[i] = a;
    }
  }
}

// the FP64 form of an interior point's flux, in the place of its state, for the states that the
// integer form leaves out: a call, so that it takes no registers from the other points
static __device__ __noinline__ void iflux_fp64(double* q, double sx, double sy, double gam) {
  double F[8];
  iflux_contra(q, sx, sy, gam - 1.0, F);
#pragma unroll
  for (int k = 0; k < 8; k++) q[k] = F[k];
}

template <int N, class O>
__device__ __forceinline__ void e1_body(const SolveDev& s, int e0, int cnt, int epb, int sensor, double* sm) {
  constexpr int NS = D<N>::NS, NF1 = D<N>::NF1, NFP = D<N>::NFP, NINT = 2 * N * (N - 1);
  double* sQ = sm;                    // [epb][NS][9]   cell states (16-byte aligned)
  double* sT = sQ + epb * NS * 9;     // [epb][NS]      sensor scratch
  double* sU = sT + epb * NS;         // [epb][NS]
  double* sV = sU + epb * NS;         // [epb][NFP][9]  flux-point values
  double* sA = sV + epb * NFP * 9;    // [N] Ar; for variable 6 the AV smoothing operator (N, N)
  // all global traffic of the pass is contiguous block copies (coalesced)
  block_copy(sQ, s.Q + (size_t)e0 * NS * 9, cnt * NS * 9);
  for (int i = threadIdx.x; i < N; i += blockDim.x) sA[i] = O::ops().Ar[i];
  __syncthreads();
  // interpolation to every flux point, one (cell, line, variable) per thread so that
  // every lane of every warp does work; the line operator runs on the integer pipes,
  // which the FP64 work of the pass leaves idle
  for (int t = threadIdx.x; t < cnt * 2 * N * 9; t += blockDim.x) {
    const int k = t % 9, el = t / 9, e = el / (2 * N), line = el - e * 2 * N;
    const double* q = sQ + e * NS * 9 + k;
    const bool fam1 = line < N;
    const int ln = fam1 ? line : line - N;
    // solution values along the line and where the line's flux values go
    const double* qb = fam1 ? q + ln * N * 9 : q + ln * 9;
    const int qs = fam1 ? 9 : N * 9;
    double* ob = sV + (e * NFP + (fam1 ? ln * (N + 1) : NF1 + ln)) * 9 + k;
    const int os = fam1 ? 9 : N * 9;
    double v[N], y[N + 1];
#pragma unroll
    for (int sp = 0; sp < N; sp++) v[sp] = qb[sp * qs];
    interp_line<N, O>(v, y);
#pragma unroll
    for (int f = 0; f <= N; f++) ob[f * os] = y[f];
  }
  __syncthreads();
  // the flux-point values go out before the fluxes take their place
  block_copy(s.Qvf + (size_t)e0 * NFP * 9, sV, cnt * NFP * 9);
  __syncthreads();
  // contravariant inviscid flux at the interior flux points only (face points of Fc and
  // Azf belong to the face pass), one point per thread, in the place of the point's state
  // 512x512 cells, N = 5 (GB300): the pass took 1.14 ms a stage with 40 FP64 operations a point
  // (84% of that pipe), 0.86 ms with integer instructions (issue slots 62% busy, the
  // FP64 pipe 45% with conversions and sensor).  A quarter of the points left in FP64 form beside them:
  // 0.92 ms (part-filled warps in two loops).  64 registers (32 warps per SM): 0.95 ms at 80,
  // 1.06 at 96 without the spill of 28 bytes.
  for (int t = threadIdx.x; t < cnt * NINT; t += blockDim.x) {
    const int e = t / NINT, fp = interior_fp<N>(t - e * NINT);
    volatile double* q = sV + (e * NFP + fp) * 9;
    const double2 m = reinterpret_cast<const double2*>(s.met)[(size_t)(e0 + e) * NFP + fp];  // 16-byte metric pair
    auto put = [&](int j, double a, double b) {
      q[2 * j] = a;
      q[2 * j + 1] = b;
    };
    if (!iflux_int([&](int k) { return q[k]; }, m.x, m.y, s.gas, put)) iflux_fp64(sV + (e * NFP + fp) * 9, m.x, m.y, s.gam);
  }
  __syncthreads();
  // the flux records, four threads to a record: consecutive points of a line adjoin
  for (int t = threadIdx.x; t < cnt * NINT * 4; t += blockDim.x) {
    const int i = t >> 2, j = t & 3, e = i / NINT, fp = interior_fp<N>(i - e * NINT);
    const double* F = sV + (e * NFP + fp) * 9;
    const size_t g = (size_t)(e0 + e) * NFP + fp;
    reinterpret_cast<double2*>(s.Fc + g * 8)[j] = make_double2(F[2 * j], F[2 * j + 1]);
    if (j == 0) s.Azf[g] = F[8];
  }
  if (!sensor) {
    if (s.skip)
      for (int e = threadIdx.x; e < cnt; e += blockDim.x) {
        s.act[e0 + e] = 0;
        s.nv[e0 + e] = 0;
        s.gr[e0 + e] = 0;
      }
    return;
  }
  // AV sensor of variable 1 (AV.f90:15-82): Qsm = A rho A^T, sum ((Qsm-rho)/rho)^2.
  // Se = log10(sum) is compared with -6 and -1 only; the sum itself is kept (Se < -6
  // exactly when sum < 1e-6) and the logarithm is taken where the ramp needs it.
  // With A = 1 - r l^T, Qsm - rho = -(r_i t_j + r_j u_i - r_i r_j w): t and u are the sums of
  // l rho along the two families of lines and w that of l t, so a point takes 3 FP64
  // operations where the products with A take 10 and a subtraction that cancels.  A few lanes of
  // one warp sum a cell, so that a warp's FP64 instruction, which takes its time however many
  // lanes are on, serves several cells.  The pass with the products and a warp per cell -> like
  // this (ms a stage; GB300): 301x277 cells, N = 3 0.120 -> 0.104; 256x256, N = 4 0.143 -> 0.136;
  // 512x512, N = 5 0.847 -> 0.836.
  for (int t = threadIdx.x; t < cnt * 2 * N; t += blockDim.x) {
    const int e = t / (2 * N), j = t - e * 2 * N;
    const double* q = sQ + e * NS * 9 + (j < N ? j * N * 9 : (j - N) * 9);
    const int qs = j < N ? 9 : N * 9;
    double a = 0.0;
#pragma unroll
    for (int m = 0; m < N; m++) a += O::ops().Al[m] * q[m * qs];
    sT[t] = a;  // [e][2N]: t, u
  }
  __syncthreads();
  constexpr int LPC = N <= 2 ? 2 : N == 3 ? 4 : N <= 6 ? 8 : 16;  // lanes per cell
  const int lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  for (int t = threadIdx.x; t < cnt * LPC; t += blockDim.x) {
    const int e = t / LPC, l = t - e * LPC;
    const double* q = sQ + e * NS * 9;
    const double* T = sT + e * 2 * N;
    double w = 0.0;
#pragma unroll
    for (int n = 0; n < N; n++) w += O::ops().Al[n] * T[n];
    double acc = 0.0;
#pragma unroll 1
    for (int p = l; p < NS; p += LPC) {
      const int i = p % N, j = p / N;
      const double d = (sA[i] * T[j] + sA[j] * (T[N + i] - sA[i] * w)) * rcp_pos(q[p * 9]);
      acc += d * d;
    }
    const unsigned group = (LPC == 32 ? 0xffffffffu : (1u << LPC) - 1) << (lane & ~(LPC - 1));
#pragma unroll
    for (int o = LPC / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(group, acc, o);
    if (l == 0) {
      s.Se[e0 + e] = acc;
      if (s.skip) {
        s.act[e0 + e] = (acc < 1e-6) ? 0 : 1;  // NaN counts as active
        s.nv[e0 + e] = 0;  // F1 marks the active cells and their face neighbours
        s.gr[e0 + e] = 0;
      }
      // the AV ramp (log10 and sin) once per cell: in the pass that reads it for a cell and its
      // four neighbours it took 14 us of a small mesh's stage
      s.Sw[e0 + e] = av_ramp(acc);
    }
  }
  if (!(sensor & 2)) return;
  // the same sensor of variable 6 (B_x), whose muAV(6) only the plot output reads
  // (tecplotter.f90:39 from AV.f90:60-73); in the reference's division form, so a zero
  // B_x gives the reference's inf or NaN
  __syncthreads();
  for (int i = threadIdx.x; i < N * N; i += blockDim.x) sA[i] = O::ops().A[i];
  __syncthreads();
  for (int t = threadIdx.x; t < cnt * NS; t += blockDim.x) {
    const int e = t / NS, p = t - e * NS, is = p % N, n = p / N;
    const double* q = sQ + e * NS * 9 + 5;
    double a = 0.0;
#pragma unroll
    for (int m = 0; m < N; m++) a += sA[is * N + m] * q[(n * N + m) * 9];
    sT[e * NS + p] = a;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < cnt * NS; t += blockDim.x) {
    const int e = t / NS, p = t - e * NS, is = p % N, js = p / N;
    double a = 0.0;
#pragma unroll
    for (int n = 0; n < N; n++) a += sA[js * N + n] * sT[e * NS + n * N + is];
    const double b = sQ[(e * NS + p) * 9 + 5];
    sU[e * NS + p] = ((a - b) * (a - b)) / (b * b);
  }
  __syncthreads();
  for (int e = threadIdx.x >> 5; e < cnt; e += nwarp) {
    double acc = 0.0;
    for (int p = lane; p < NS; p += 32) acc += sU[e * NS + p];
    acc = warp_sum(acc);
    if (lane == 0) s.Se6[e0 + e] = acc;
  }
}

// registers per thread of the pass (101x90 cells, N = 8: 98 us at 64, 94 us at 80)
constexpr int e1_regs(int N) { return N > 6 ? 80 : 64; }

// cells [c0, c1) of the solve, epb per CTA
template <int N>
__global__ void __maxnreg__(e1_regs(N)) k_e1(const __grid_constant__ SolveDev s, int epb, int sensor, int c0, int c1) {
  extern __shared__ __align__(16) double sm[];
  pdl_wait();
  // bit 4: the first pass of a stage, which starts the stage's wave-speed maximum and list
  if ((sensor & 4) && c0 == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
    *s.eig = 0ull;
    *s.vcount = 0;
  }
  sensor &= 3;
  const int e0 = c0 + blockIdx.x * epb;
  const int cnt = min(epb, c1 - e0);
  if (cnt <= 0) return;
  if ((sensor & 2) && !*s.plot_flag) sensor &= 1;  // the plot's sensor only when asked for
  e1_body<N, OpsTU>(s, e0, cnt, epb, sensor, sm);
}

// cells of this CTA with a viscous flux, compacted into a shared list; returns the count
__device__ __forceinline__ int active_cells(const SolveDev& s, int e0, int cnt, int* list) {
  // the first warp tests 32 cells at a time (their flag loads in flight together) and
  // compacts them in cell order with a ballot
  __shared__ int n_act;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    int n = 0;
    for (int base = 0; base < cnt; base += 32) {
      const int e = base + lane;
      const bool need = e < cnt && (!s.skip || s.nv[e0 + e]);
      const unsigned m = __ballot_sync(0xffffffffu, need);
      if (need) list[n + __popc(m & ((1u << lane) - 1u))] = e;
      n += __popc(m);
    }
    if (lane == 0) n_act = n;
  }
  __syncthreads();
  return n_act;
}

// ---------------------------------------------------------------------------
// F1: Rusanov flux on every face point (interfaceflux / CYCLOCFLUX / BCFLUX)
// ---------------------------------------------------------------------------
// the FP64 form of a face point's flux, for the states that the integer form leaves out, and the
// left side's normal velocity: a call, so that it takes no registers from the points that do not
// need it
static __device__ __noinline__ double rusanov_fp64(const double* pl, const double* pr, const FaceNorm* fn, double gam,
                                            double* Fh, double& vnl) {
  double ql[9], qr[9], ev;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    ql[k] = pl[k];
    qr[k] = pr[k];
  }
  rusanov_core(ql, qr, fn->ux, fn->uy, gam, fn->msl, Fh, vnl, ev);
  return ev;
}

// shared memory of one warp of the face pass, for 32 points: two buffers of their traces
// (left and right) and face normals, their flux records, the places of the traces, and the
// face records of three rounds
struct F1Warp {
  double q[2][2][32 * 9];  // [buffer][side][point][variable]
  double2 fn[2][32][2];    // [buffer][point] FaceNorm
  double F[32 * 9];        // [point][component], a stride of 9 against bank conflicts
  long long g[2][2][32];   // [buffer][side][point] flux-point index; right: -1 on a FREE face
  int4 rec[3][32];
};
constexpr int kF1Threads = 160;
constexpr size_t f1_smem(int threads) { return (size_t)(threads / 32) * sizeof(F1Warp); }

// put cell c on the list of the cells with viscous flux, the first time
__device__ __forceinline__ void mark_viscous(const SolveDev& s, int c) {
  if (atomicExch(&s.nv[c], 1) == 0) s.vlist[atomicAdd(s.vcount, 1)] = c;
}

// Face points first .. first + 31, then on by step, ... < n of a warp (first and step are the
// warp's, the same for its lanes); map(i) is the point's number among the solve's two-sided
// (t < nface2*N) then FREE face points.  Returns the bit pattern of the lane's largest wave
// speed.
//
// A point is one lane's work, some 2500 instructions at 168 registers, so ten warps share an SM:
// too few to hide the two dependent loads (face record, traces) behind
// other warps.  The warp therefore copies the next 32 points' traces and the face records of
// the 32 after them while it computes a round.  The 72-byte traces and 64-byte flux records
// are moved by the warp together, consecutive lanes taking consecutive words of a record:
// one lane per record would touch every 32-byte sector of the L2 four times.
// 512x512 cells, N = 5 (GB300): 0.867 ms a stage in FP64 (80% of that pipe), 0.62 ms in integer
// form with one thread's own loads and the averaged traces stored, 0.42 ms in this form (0.36 with
// one exponent for several components, which cost small ones their bits), of
// which the 5.1 kB per cell that it moves take 0.2 ms at the copy rate.  Ten warps at 168
// registers: at 128 registers (16 warps) the spills go past an L1 that the traces fill, 0.73 ms.
template <int N, class Map>
__device__ __forceinline__ unsigned long long f1_points(const SolveDev& s, int first, int step, int n, F1Warp* warps, Map&& map) {
  constexpr int NFP = D<N>::NFP;
  const int n2 = s.nface2 * N, lane = threadIdx.x & 31;
  F1Warp& w = warps[threadIdx.x >> 5];
  auto fetch_rec = [&](int i, int slot) {
    if (i >= n) return;
    const int t = map(i);
    if (t < n2) cp_async16(&w.rec[slot][lane], s.face2 + t / N);
    else cp_async8(&w.rec[slot][lane], s.face1 + (t - n2) / N);
  };
  auto normal = [&](int t) { return t < n2 ? s.fn2 + t : s.fn1 + (t - n2); };
  // the round whose lane has point i: where its traces are, and their copies
  auto fetch_data = [&](int i, int slot, int buf) {
    long long gl = -1, gr = -1;
    if (i < n) {
      const int t = map(i);
      const int4 fc = w.rec[slot][lane];
      const int nfp = t < n2 ? t % N : (t - n2) % N;
      gl = (long long)fc.x * NFP + face_fp<N>(fc.y, nfp);
      if (t < n2) gr = (long long)fc.z * NFP + face_fp<N>(fc.w, N - 1 - nfp);
      const double2* pn = reinterpret_cast<const double2*>(normal(t));
      cp_async16(&w.fn[buf][lane][0], pn);
      cp_async16(&w.fn[buf][lane][1], pn + 1);
    }
    w.g[buf][0][lane] = gl;
    w.g[buf][1][lane] = gr;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < 9; r++) {
      const int j = r * 32 + lane, p = j / 9, k = j - 9 * p;
      const long long pl = w.g[buf][0][p], pr = w.g[buf][1][p];
      if (pl >= 0) {
        cp_async8(&w.q[buf][0][j], s.Qvf + pl * 9 + k);
        cp_async8(&w.q[buf][1][j], s.Qvf + (pr >= 0 ? pr : pl) * 9 + k);  // a FREE face has its own state on both sides
      }
    }
  };
  fetch_rec(first + lane, 0);
  fetch_rec(first + step + lane, 1);
  cp_async_commit();
  pdl_wait();  // (the face records do not depend on the pass before)
  cp_async_wait();
  fetch_data(first + lane, 0, 0);
  cp_async_commit();
  unsigned long long evb = 0ull;
  int buf = 0, slot = 0;
#pragma unroll 1
  for (int i0 = first; i0 < n; i0 += step) {
    const int next = slot == 2 ? 0 : slot + 1, i = i0 + lane;
    cp_async_wait();  // this turn's traces, the next turn's records
    __syncwarp();
    fetch_data(i + step, next, buf ^ 1);
    fetch_rec(i + 2 * step, next == 2 ? 0 : next + 1);
    cp_async_commit();
    if (i < n) {
      const int t = map(i);
      const bool nfp0 = (t < n2 ? t : t - n2) % N == 0;
      const long long gl = w.g[buf][0][lane], gr = w.g[buf][1][lane];
      const double2 nrm = w.fn[buf][lane][0];
      // (the states are read from shared memory where they are used, not kept)
      const volatile double* ql = w.q[buf][0] + 9 * lane;
      const volatile double* qr = w.q[buf][1] + 9 * lane;
      double* F = w.F + 9 * lane;
      auto put = [&](int j, double a, double b) {
        F[2 * j] = a;
        F[2 * j + 1] = b;
      };
      double ev, vn = fma(ql[1], nrm.x, ql[2] * nrm.y);  // m.n, of the sign of u.n
      if (!rusanov_int([&](int side, int k) { return side ? qr[k] : ql[k]; }, nrm.x, nrm.y, s.gas, w.fn[buf][lane][1].x, ev, put)) {
        double Fd[8];
        ev = rusanov_fp64(w.q[buf][0] + 9 * lane, w.q[buf][1] + 9 * lane, normal(t), s.gam, Fd, vn);  // (a negative density among them)
#pragma unroll
        for (int j = 0; j < 4; j++) put(j, Fd[2 * j], Fd[2 * j + 1]);
      }
      const unsigned long long e = ev_bits(ev, s.err);
      evb = e > evb ? e : evb;
      // A_z from the upwind side (getrusanov.f90:99-103)
      const double az = vn > 0.0 ? ql[8] : qr[8];
      s.Azf[gl] = az;
      if (gr >= 0) {
        s.Azf[gr] = az;
      }
      if (s.skip && nfp0) {  // once per face: AV-active cells and their neighbours carry viscous flux
        const int4 fc = w.rec[slot][lane];
        if (s.act[fc.x] || (gr >= 0 && s.act[fc.z])) {
          mark_viscous(s, fc.x);
          if (gr >= 0) mark_viscous(s, fc.z);
        }
      }
    }
    __syncwarp();
    // the flux records, four lanes to a record
#pragma unroll
    for (int r = 0; r < 4; r++) {
      const int p = r * 8 + (lane >> 2), j = lane & 3;
      const long long pl = w.g[buf][0][p], pr = w.g[buf][1][p];
      if (pl < 0) continue;
      const double a = w.F[9 * p + 2 * j], b = w.F[9 * p + 2 * j + 1];
      reinterpret_cast<double2*>(s.Fc + pl * 8)[j] = make_double2(a, b);
      if (pr >= 0) {
        const double ss = w.fn[buf][p][1].y;
        reinterpret_cast<double2*>(s.Fc + pr * 8)[j] = make_double2(times_sign(a, ss), times_sign(b, ss));
      }
    }
    __syncwarp();
    buf ^= 1;
    slot = next;
  }
  return evb;
}

// face points [t2, t2 + n2) of the two-sided list, then [t1, t1 + n - n2) of the FREE list
// (f1_points numbering: the FREE faces follow the two-sided ones)
template <int N>
__global__ void __launch_bounds__(kF1Threads, 2) k_f1(SolveDev s, int t2, int n2, int t1, int n) {
  extern __shared__ __align__(16) double sm[];
  const int nw = blockDim.x >> 5;
  const unsigned long long evb = f1_points<N>(s, (blockIdx.x * nw + (threadIdx.x >> 5)) * 32, gridDim.x * nw * 32, n,
                                              reinterpret_cast<F1Warp*>(sm),
                                              [&](int i) { return i < n2 ? t2 + i : t1 + (i - n2); });
  block_max_ull(evb, s.eig);
}

// the traces of the two-sided faces replaced by their mean (interfaceflux /
// CYCLOCFLUX, interfaceflux_all.f90:79-91).  A stage takes the mean where it reads the traces
// (E2, E3: few cells as a rule); this pass makes the stored traces equal to the reference's
// Qvfi/Qvfj where they are downloaded or differentiated.  (A second run changes nothing.)
template <int N>
__global__ void __launch_bounds__(256) k_qavg(SolveDev s) {
  constexpr int NFP = D<N>::NFP;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= s.nface2 * N) return;
  const int f = t / N, nfp = t - f * N;
  const int4 fc = s.face2[f];
  double* a = s.Qvf + ((size_t)fc.x * NFP + face_fp<N>(fc.y, nfp)) * 9;
  double* b = s.Qvf + ((size_t)fc.z * NFP + face_fp<N>(fc.w, N - 1 - nfp)) * 9;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double v = half(a[k] + b[k]);
    a[k] = v;
    b[k] = v;
  }
}

// the flux point across the face from point fp of cell c: its index among all flux points, or
// -1 for an interior point and on a FREE face
template <int N>
__device__ __forceinline__ long long across(const SolveDev& s, int c, int fp) {
  int nfp = 0;
  const int lf = fp_face<N>(fp, nfp);
  const int o = lf ? (&s.nbr[c].x)[lf - 1] : -1;
  if (o < 0) return -1;
  return (long long)o * D<N>::NFP + face_fp<N>((&s.nbrlf[c].x)[lf - 1], N - 1 - nfp);
}

// ---------------------------------------------------------------------------
// E2: gradients at solution points and their values at every flux point
// ---------------------------------------------------------------------------
// the AV viscosity on local face lf of cell c (compAVflux / interfaceAVflux / cyclocAVflux,
// AV.f90:199-303, 494-564): the mean of the two cells' muAV(1) on a two-sided face (the same
// bits from either side: the sum commutes), the cell's own on a FREE face; muAV(1) from the
// stage's sensor and epsilon0 = eigvmax h/(N-1) (AV.f90:147)
template <int N>
__device__ __forceinline__ double face_mu(const SolveDev& s, int c, int lf) {
  const int o = (&s.nbr[c].x)[lf - 1];
  const double rc = s.Sw[c], ro = o >= 0 ? s.Sw[o] : 0.0;
  const long long eig = (long long)*s.eig;
  // (no ramp and a finite wave speed: leave before the FP64 operations, which a warp's few lanes
  // that come here do not share)
  if (((__double_as_longlong(rc) | __double_as_longlong(ro)) << 1) == 0 && (unsigned)(eig >> 52) < 0x7ffu) return 0.0;
  const double eps0 = __longlong_as_double(eig) * s.hmsh / (double)(N - 1) * 1.0, h0 = eps0 / 2.0;
  const double mc = h0 * rc;
  return o >= 0 ? half(mc + h0 * ro) : mc;
}

template <int N>
__device__ __forceinline__ void cell_face_mu(const SolveDev& s, int c) {
#pragma unroll
  for (int k = 0; k < 4; k++) s.muf[4 * c + k] = s.artiv ? face_mu<N>(s, c, k + 1) : 0.0;
}

constexpr int kE3Fp64 = -(1 << 28);  // in place of an exponent: the value is a double

// 1/J (sum of the two families' derivatives) where one of the three is not in integer form: a
// call, because a branch of few FP64 instructions would be predicated, and an FP64 instruction
// occupies its pipe whether its lanes are on or off.  k0, k1: exponents of the sums V0, V1 or
// kE3Fp64 for doubles.
static __device__ __noinline__ double e3_fp64(int64_t V0, int k0, int64_t V1, int k1, double j) {
  const double y0 = k0 != kE3Fp64 ? ix_double(V0, k0) : __longlong_as_double(V0);
  const double y1 = k1 != kE3Fp64 ? ix_double(V1, k1) : __longlong_as_double(V1);
  return (y0 + y1) * j;
}

// shared memory of the pass for epb cells (e2_cells)
constexpr size_t e2_smem(int N, int epb) {
  return (size_t)epb * ((size_t)2 * (N + 1) * N * (72 + 16 + 8) + (size_t)N * N * (128 + 8 + 4) + (size_t)N * 16 * 4) + 64;
}

template <int N, class O>
__device__ __forceinline__ void e2_cells(const SolveDev& s, const int* cells, int n, int keep, double* sm) {
  // gradients of the n (<= epb) listed cells; grad A_z (nablaAsp) is computed with the
  // divergence in the last pass.  nablaQsp (compflux.f90:107-157) in its conservative
  // form: grad_x Q = (1/J) [d/dxi (S1(1,1) Q) + d/deta (S2(2,1) Q)], grad_y the same with
  // the second metric entries, i.e. the divergence of the products of the face-averaged
  // flux-point states with the metric terms, differentiated along the lines on the integer
  // pipes as in E3.  The products are integers too (ix_line_products), each from operands with
  // their own exponents and aligned to the line's largest product, so that a metric entry that is
  // small beside the other one (flat cells) or along a part of the line keeps its bits.
  constexpr int NS = D<N>::NS, NF1 = D<N>::NF1, NFP = D<N>::NFP;
  double* sQ = sm;                                              // [n][NFP][9] Q
  Limbs* sS = reinterpret_cast<Limbs*>(sQ + n * NFP * 9);       // [n][NFP][2] metric entries (ix_load)
  double* sG = reinterpret_cast<double*>(sS + n * NFP * 2);     // [n][NS][16] grad Q (d*8 + k)
  int64_t* sJ = reinterpret_cast<int64_t*>(sG + n * NS * 16);   // [n][NS] 1/J as an integer
  int* sE = reinterpret_cast<int*>(sJ + n * NS);                // [n][NS] and its exponent
  int* sK = sE + n * NS;                                        // [n][N][8][2] exponents of the xi-line sums
  int* sX = sK + n * N * 16;                                    // [n][NFP][2] exponents of the metric entries
  for (int le = 0; le < n; le++)
    block_copy_async(sQ + le * NFP * 9, s.Qvf + (size_t)cells[le] * NFP * 9, NFP * 9);
  cp_async_commit();
  for (int i = threadIdx.x; i < n * NS; i += blockDim.x) {
    const int le = i / NS;
    const double j = s.invJ[(size_t)cells[le] * NS + i - le * NS];
    const uint32_t m = ix_abs_word(j);
    sJ[i] = ix_align<2>(j, m);
    sE[i] = m >= kIxLow && m < kIxHigh ? ix_exp<2>(m) : kE3Fp64;
  }
  for (int i = threadIdx.x; i < n * NFP * 2; i += blockDim.x) {
    const int le = i / (NFP * 2);
    const double m = s.met[(size_t)cells[le] * NFP * 2 + i - le * NFP * 2];
    const IxF a = ix_load(m);
    sS[i] = a.m;
    sX[i] = ix_abs_word(m) < kIxHigh ? a.e : kIxNoLine;
  }
  cp_async_wait();
  __syncthreads();
  // face traces enter as the mean of both sides
  for (int i = threadIdx.x; i < n * 4 * N * 8; i += blockDim.x) {
    const int k = i & 7, r = i >> 3, le = r / (4 * N), f = r - le * 4 * N, lf = f / N + 1, nfp = f - (lf - 1) * N;
    const int c = cells[le], o = (&s.nbr[c].x)[lf - 1];
    if (o < 0) continue;
    double* q = sQ + (le * NFP + face_fp<N>(lf, nfp)) * 9 + k;
    *q = half(*q + s.Qvf[((size_t)o * NFP + face_fp<N>((&s.nbrlf[c].x)[lf - 1], N - 1 - nfp)) * 9 + k]);
  }
  __syncthreads();
  // grad Q (variables 1-8) at the solution points: one (cell, line, variable) per thread,
  // the xi lines first, then the eta lines adding to them and multiplying by 1/J
#pragma unroll 1
  for (int fam = 0; fam < 2; fam++) {
    for (int t = threadIdx.x; t < n * N * 8; t += blockDim.x) {
      const int k = t & 7, el = t >> 3, le = el / N, ln = el - le * N;
      const int fp0 = le * NFP + (fam ? NF1 + ln : ln * (N + 1)), fps = fam ? N : 1;
      uint32_t m = 0;
#pragma unroll
      for (int r = 0; r <= N; r++) m = ix_max(m, ix_abs_word(sQ[(fp0 + r * fps) * 9 + k]));
#pragma unroll 1
      for (int d = 0; d < 2; d++) {
        double* g = sG + le * NS * 16 + d * 8 + k;
        int64_t X[N + 1];
        const int eX = ix_line_products<N + 1>([&](int r) { return ix_load(sQ[(fp0 + r * fps) * 9 + k]); },
                                               [&](int r) { const int i = (fp0 + r * fps) * 2 + d; return IxF{sS[i], sX[i]}; }, X);
        const bool ok = m < kIxHigh && eX < kIxNoLine / 2;
        const int kv = ok ? eX + 58 - O::ops().MS : kE3Fp64;
        if (!fam) sK[2 * t + d] = kv;
        auto finish = [&](int i, int64_t V) {
          if (!fam) {
            g[(ln * N + i) * 16] = __longlong_as_double(V);
            return;
          }
          const int p = i * N + ln, ps = le * NS + p, eJ = sE[ps], k0 = sK[((le * N + i) * 8 + k) * 2 + d];
          const int64_t V0 = __double_as_longlong(g[p * 16]);
          double a;
          if (ok && k0 != kE3Fp64 && eJ != kE3Fp64) {
            const int K = max(k0, kv);
            const int64_t sum = ix_shr(V0, K - k0 + O::ops().MV) + ix_shr(V, K - kv + O::ops().MV);
            a = ix_double(ix_mul(sum, ix_limbs(sJ[ps])), K + O::ops().MV + eJ + 62);
          } else {
            a = e3_fp64(V0, k0, V, kv, s.invJ[(size_t)cells[le] * NS + p]);
          }
          g[p * 16] = a;
          // (only the evaluation whose arrays can be downloaded stores them)
          if (keep) s.nQs[((size_t)cells[le] * NS + p) * 18 + 9 * d + k] = a;
        };
        if (ok) {
          fix_mirror_core<N, N + 1, -1>(X, O::ops().MH, O::ops().ML, finish);
        } else {
          const double* met = s.met + (size_t)cells[le] * NFP * 2 + d;
#pragma unroll 1
          for (int i = 0; i < N; i++) {
            double a = 0.0;
#pragma unroll 1
            for (int r = 0; r <= N; r++) {
              const int fp = fp0 + r * fps;
              a += O::ops().M[r + (N + 1) * i] * (sQ[fp * 9 + k] * met[2 * (fp - le * NFP)]);
            }
            finish(i, __double_as_longlong(a));
          }
        }
      }
    }
    __syncthreads();
  }
  // grad Q at every flux point (nablaQ_interior_FP + face traces): one (cell, line,
  // component) per thread, the line operator on the integer pipes as in E1
  for (int t = threadIdx.x; t < n * 2 * N * 16; t += blockDim.x) {
    const int c = t & 15, el = t >> 4, le = el / (2 * N), line = el - le * 2 * N;
    const bool fam1 = line < N;
    const int ln = fam1 ? line : line - N;
    const double* gb = sG + (le * NS + (fam1 ? ln * N : ln)) * 16 + c;
    const int gs = fam1 ? 16 : N * 16;
    const int f0 = fam1 ? ln * (N + 1) : NF1 + ln, fs = fam1 ? 1 : N;
    double* ob = s.nQvf + ((size_t)cells[le] * NFP + f0) * 18 + (c < 8 ? c : c + 1);
    double v[N], y[N + 1];
#pragma unroll
    for (int sp = 0; sp < N; sp++) v[sp] = gb[sp * gs];
    interp_line<N, O>(v, y);
#pragma unroll
    for (int f = 0; f <= N; f++) ob[(size_t)f * fs * 18] = y[f];
  }
}

// E2 by a CTA that is number `first` of `stride`.  Every cell (skip = 0): groups of epb cells.
// Otherwise the listed cells with a viscous flux and their face neighbours: a CTA takes epb
// list entries at a time and those of their neighbours that are not listed and that no other
// CTA has claimed (a cell's gradients do not depend on who computes them), in groups.  The
// work is spread evenly however the active cells lie: with one CTA per range of cells E2 and V
// took 0.235 ms a stage for the 2% of active cells of a rotor (256x256, N = 4), 0.060 ms like this.
// keep: also every cell's face viscosities, which can be downloaded.
template <int N, class O>
__device__ __forceinline__ void e2_all(const SolveDev& s, int first, int stride, int epb, int keep, double* sm) {
  __shared__ int list[5 * 64];
  __shared__ int taken;
  if (keep)
    for (int c = first * blockDim.x + threadIdx.x; c < s.NC; c += stride * blockDim.x) cell_face_mu<N>(s, c);
  const int total = s.skip ? *s.vcount : s.NC;
  for (int base = first * epb; base < total; base += stride * epb) {
    const int m = min(epb, total - base);
    if (threadIdx.x == 0) taken = s.skip ? 0 : m;
    __syncthreads();
    for (int t = threadIdx.x; t < (s.skip ? 5 * m : m); t += blockDim.x) {
      if (!s.skip) {
        list[t] = base + t;
        continue;
      }
      const int v = s.vlist[base + t / 5], k = t % 5, c = k == 4 ? v : (&s.nbr[v].x)[k];
      if (k == 4 || (c >= 0 && !s.nv[c] && atomicExch(&s.gr[c], 1) == 0)) list[atomicAdd(&taken, 1)] = c;
    }
    __syncthreads();
    const int n = taken;
    for (int g = 0; g < n; g += epb) {
      e2_cells<N, O>(s, list + g, min(epb, n - g), keep, sm);
      __syncthreads();
    }
  }
}

template <int N>
__global__ void __launch_bounds__(512, 2) k_e2(const __grid_constant__ SolveDev s, int epb, int keep) {
  extern __shared__ __align__(16) double sm[];
  pdl_wait();
  e2_all<N, OpsTU>(s, blockIdx.x, gridDim.x, epb, keep, sm);
}

// ---------------------------------------------------------------------------
// V: the total flux Ft = Fc - viscous, resistive and AV flux of the cells that carry one, in
// Fc's place or (where the inviscid flux stays downloadable) beside it (interfaceVISflux /
// BCVISFLUX / CYCLOCVISFLUX, comp_viscous_flux).  One flux point per thread with the integer
// form of the flux; the FP64 form inside E3 kept that pass at 0.37 ms over its inviscid time
// (128x128 cells, N = 5, every cell viscous), V takes 0.153 ms.  Bound by latency with the integer
// issue (51%), the FP64 pipe (52%: averages, conversions) and the loads of Q and grad Q (292 MB,
// 1.9 TB/s) all about half used: 27 doubles of shared memory a point (the flux in the place of
// the state) and 64 registers for eight CTAs per SM, against 0.171 ms with 36 and 72 for six.
// ---------------------------------------------------------------------------
// cells per group and threads per CTA: one flux point per thread
constexpr int v_epb(int N) { return N >= 6 ? 1 : 128 / (2 * (N + 1) * N); }
constexpr int v_threads(int N) { return (v_epb(N) * 2 * (N + 1) * N + 31) / 32 * 32; }
constexpr size_t v_smem(int N) { return (size_t)v_epb(N) * 2 * (N + 1) * N * 27 * 8; }

// the viscosity of flux point fp of a cell with AV viscosities mf[4] on its local faces 1..4:
// mu + the AV viscosity, linear between the faces
template <int N, class O>
__device__ __forceinline__ double point_mu(const SolveDev& s, const double* mf, int fp) {
  constexpr int NF1 = D<N>::NF1;
  if (!s.artiv) return s.mu;
  const double x = O::ops().Xf[fp < NF1 ? fp % (N + 1) : (fp - NF1) / N];
  const double a = fp < NF1 ? mf[3] : mf[0], b = fp < NF1 ? mf[1] : mf[2];
  if (((__double_as_longlong(a) | __double_as_longlong(b)) << 1) == 0) return s.mu;
  return s.mu + (a * (1.0 - x) + b * x);
}

// the FP64 form of a point's flux, for the states that the integer form leaves out (a call, so
// that it takes no registers from the other points)
static __device__ __noinline__ void vflux_fp64(const double* q, const double* g, double mut, double eta, double gam,
                                               double sx, double sy, double* F) {
  double Fv[8];
  vflux_contra(q, g, mut, eta, gam, sx, sy, Fv);
#pragma unroll
  for (int k = 1; k < 8; k++) F[k] = Fv[k];
}

template <int N, class O>
__device__ __forceinline__ void v_cells(const SolveDev& s, const int* cells, int n, double* Ft, double* sm) {
  constexpr int NFP = D<N>::NFP;
  double* sG = sm;                // [n][NFP][18] grad Q
  double* sQ = sG + n * NFP * 18;  // [n][NFP][9] Q, then the viscous flux (components 1..7)
  for (int le = 0; le < n; le++) {
    block_copy_async(sG + le * NFP * 18, s.nQvf + (size_t)cells[le] * NFP * 18, NFP * 18);
    block_copy_async(sQ + le * NFP * 9, s.Qvf + (size_t)cells[le] * NFP * 9, NFP * 9);
  }
  cp_async_commit();
  __shared__ double smu[v_epb(N)][4];
  if (s.artiv && (int)threadIdx.x < 4 * n) smu[threadIdx.x >> 2][threadIdx.x & 3] = face_mu<N>(s, cells[threadIdx.x >> 2], (threadIdx.x & 3) + 1);
  cp_async_wait();
  __syncthreads();
  // on a two-sided face the traces of Q and of grad Q are the means of both sides'
  // (interfaceflux_all.f90:79-91, 118-199, cyclocflux_all.f90:118-208); a FREE face keeps its
  // own (BCVISFLUX): 24 values of each of a cell's 4 N face points
  for (int i = threadIdx.x; i < n * 4 * N * 24; i += blockDim.x) {
    const int j = i % 24, r = i / 24, le = r / (4 * N), k = r - le * 4 * N, lf = k / N + 1, nfp = k - (lf - 1) * N;
    const int c = cells[le], o = (&s.nbr[c].x)[lf - 1];
    if (o < 0) continue;
    const size_t go = (size_t)o * NFP + face_fp<N>((&s.nbrlf[c].x)[lf - 1], N - 1 - nfp);
    const int at = le * NFP + face_fp<N>(lf, nfp);
    if (j < 16) {
      const int m = j < 8 ? j : j + 1;
      sG[at * 18 + m] = half(sG[at * 18 + m] + s.nQvf[go * 18 + m]);
    } else {
      sQ[at * 9 + j - 16] = half(sQ[at * 9 + j - 16] + s.Qvf[go * 9 + j - 16]);
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < n * NFP; t += blockDim.x) {
    const int le = t / NFP, fp = t - le * NFP, c = cells[le];
    const double2 m = reinterpret_cast<const double2*>(s.met)[(size_t)c * NFP + fp];
    const double mut = point_mu<N, O>(s, smu[le], fp);
    volatile double* q = sQ + 9 * t;
    const volatile double* gr = sG + 18 * t;
    if (((__double_as_longlong(mut) | __double_as_longlong(s.eta0)) << 1) == 0) {
      // no flux, whatever the gradient is: 0 times an infinity of a neighbour is not let in
#pragma unroll
      for (int k = 1; k < 8; k++) q[k] = 0.0;
      continue;
    }
    // (the flux takes the place of the point's state, which vflux_int has read by its first output)
    if (!vflux_int([&](int k) { return q[k]; }, [&](int d, int k) { return gr[9 * d + k]; }, mut, s.eta0, m.x, m.y, s.gas,
                   [&](int k, double f) { q[k] = f; }))
      vflux_fp64(sQ + 9 * t, sG + 18 * t, mut, s.eta0, s.gam, m.x, m.y, sQ + 9 * t);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n * NFP * 4; i += blockDim.x) {
    const int t = i >> 2, j = i & 3, le = t / NFP;
    const size_t g = ((size_t)cells[le] * NFP + (t - le * NFP)) * 8 + 2 * j;
    const double2 a = *reinterpret_cast<const double2*>(s.Fc + g);
    *reinterpret_cast<double2*>(Ft + g) = make_double2(j ? a.x - sQ[9 * t + 2 * j] : a.x, a.y - sQ[9 * t + 2 * j + 1]);
  }
}

// V by a CTA that is number `first` of `stride`
template <int N, class O>
__device__ __forceinline__ void v_all(const SolveDev& s, int first, int stride, double* Ft, double* sm) {
  __shared__ int list[v_epb(N)];
  const int total = s.skip ? *s.vcount : s.NC;
  for (int base = first * v_epb(N); base < total; base += stride * v_epb(N)) {
    const int m = min(v_epb(N), total - base);
    if ((int)threadIdx.x < m) list[threadIdx.x] = s.skip ? s.vlist[base + threadIdx.x] : base + threadIdx.x;
    __syncthreads();
    v_cells<N, O>(s, list, m, Ft, sm);
    __syncthreads();
  }
}

template <int N>
__global__ void __maxnreg__(64) k_v(const __grid_constant__ SolveDev s, double* Ft) {
  extern __shared__ __align__(16) double sm[];
  pdl_wait();
  v_all<N, OpsTU>(s, blockIdx.x, gridDim.x, Ft, sm);
}

// ---------------------------------------------------------------------------
// F2: face-averaged gradients and face AV viscosity
// ---------------------------------------------------------------------------
// face averages of the grad Q traces in place (interfaceVISflux, CYCLOCVISFLUX).  The
// stage itself averages them where the viscous flux reads them (V, E3); this pass makes the
// stored traces equal to the reference's nablaQvfi/nablaQvfj when they are downloaded.
template <int N>
__device__ __forceinline__ void f2_point(const SolveDev& s, int t) {
  constexpr int NFP = D<N>::NFP;
  if (t >= s.nface2 * N) return;
  const int f = t / N, nfp = t - f * N;
  const int4 fc = s.face2[f];
  double* a = s.nQvf + ((size_t)fc.x * NFP + face_fp<N>(fc.y, nfp)) * 18;
  double* b = s.nQvf + ((size_t)fc.z * NFP + face_fp<N>(fc.w, N - 1 - nfp)) * 18;
#pragma unroll
  for (int d = 0; d < 2; d++)
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const double v = half(a[9 * d + k] + b[9 * d + k]);
      a[9 * d + k] = v;
      b[9 * d + k] = v;
    }
}

template <int N>
__global__ void __launch_bounds__(256) k_f2(SolveDev s) {
  f2_point<N>(s, blockIdx.x * blockDim.x + threadIdx.x);
}

// the viscous, resistive and AV flux of the nact listed cells of the block, subtracted from
// their total flux in shared memory: a call, so that the registers it needs are not those of
// the whole pass
template <int N, class O>
static __device__ __noinline__ void e3_viscous(const SolveDev& s, int e0, int nact, const int* list, double* sF, double* smu) {
  constexpr int NFP = D<N>::NFP;
  if (s.artiv)
    for (int i = threadIdx.x; i < 4 * nact; i += blockDim.x) smu[i] = face_mu<N>(s, e0 + list[i >> 2], (i & 3) + 1);
  __syncthreads();
  for (int t = threadIdx.x; t < nact * NFP; t += blockDim.x) {
    const int le = t / NFP, fp = t - le * NFP, e = list[le], c = e0 + e;
    const size_t g = (size_t)c * NFP + fp;
    const double mut = point_mu<N, O>(s, smu + 4 * le, fp);
    if (mut != 0.0 || s.eta0 != 0.0) {
      double q[9], gq[18], Fv[8];
      const double* pq = s.Qvf + g * 9;
      const double* pg = s.nQvf + g * 18;
      // on a two-sided face the traces of Q and of grad Q are the means of both sides'
      // (interfaceflux_all.f90:79-91, 118-199, cyclocflux_all.f90:118-208); a FREE face keeps
      // its own (BCVISFLUX)
      const long long o = across<N>(s, c, fp);
      if (o >= 0) {
        const double* qo = s.Qvf + o * 9;
        const double* po = s.nQvf + o * 18;
#pragma unroll
        for (int k = 0; k < 8; k++) {
          q[k] = half(pq[k] + qo[k]);
          gq[k] = half(pg[k] + po[k]);
          gq[9 + k] = half(pg[9 + k] + po[9 + k]);
        }
      } else {
#pragma unroll
        for (int k = 0; k < 8; k++) {
          q[k] = pq[k];
          gq[k] = pg[k];
          gq[9 + k] = pg[9 + k];
        }
      }
      q[8] = 0.0;
      gq[8] = 0.0;
      gq[17] = 0.0;
      vflux_contra(q, gq, mut, s.eta0, s.gam, s.met[2 * g], s.met[2 * g + 1], Fv);
      double* d = sF + (e * NFP + fp) * 8;
#pragma unroll
      for (int k = 1; k < 8; k++) d[k] -= Fv[k];
    }
  }
}

// shared memory of the pass for epb cells (e3_body)
constexpr size_t e3_smem(int N, int epb) {
  return (size_t)epb * ((size_t)2 * (N + 1) * N * 10 * 8 + (size_t)N * N * (72 + 16 + 8 + 4) + (size_t)N * 10 * 4) + 16;
}

// The most of it that a launch may ask for: 200 kB, or what as many cells take as fitted into 200 kB
// while a cell's exponents were not kept (42 of N = 4 want 1.7% more).
constexpr int e3_smem_limit(int N) {
  const int cells = 200 * 1024 / (8 * (20 * (N + 1) * N + 13 * N * N));
  const size_t need = e3_smem(N, cells < 64 ? cells : 64);
  return need > 200 * 1024 ? (int)need : 200 * 1024;
}

constexpr long long kVPassPoints = 49152;

// Does the viscous flux get its own pass?  On meshes large enough for the extra launch to be
// small beside a stage; E3 then runs without the registers, the shared memory and the uneven
// load that the flux needs.  (By the size alone: the two forms round differently, and skipping
// work that is exactly zero must not change a result.)
// A step without the pass -> with it (us; GB300), every cell viscous: 8,000 points 207 -> 237 at
// N = 3, 229 -> 244 at N = 5; 16,000 256 -> 260, 286 -> 276; 32,000 362 -> 329, 376 -> 338; 49,000 516 -> 424,
// 513 -> 418; 200,000 1641 -> 1400, 1574 -> 1235.  With AV in a few fronts: 16,000 332 -> 339, 383 -> 364; 49,000
// 513 -> 434, 508 -> 466; 200,000 954 -> 874, 915 -> 848.  Without any active cell its launches
// cost some 7 us a step.  So the pass pays from some 20,000 points on where it has work, and the
// line keeps smaller solves, for which the launch counts most, free of it.
__host__ __device__ inline bool v_pass(const SolveDev& s) { return (long long)s.NC * s.N * s.N >= kVPassPoints; }

// Can a solve have a viscous flux at all?
__host__ __device__ inline bool viscous(const SolveDev& s) { return s.artiv || s.mu != 0.0 || s.eta0 != 0.0; }

// what E3 does about the viscous flux (e3_body): keep = the inviscid flux stays downloadable
__host__ __device__ inline int e3_visc(const SolveDev& s, bool keep) {
  return !viscous(s) ? 0 : !v_pass(s) ? 1 : keep ? 2 : 0;
}

// does a stage only need its increment cR * resid, so that cR is folded into 1/J?
__host__ __device__ inline bool e3_pre(const RKStage& rk, int update) {
  return update && !rk.write_resid && !rk.save_R && !rk.diag;
}

// PRE = e3_pre(rk, update): two bodies, since FP64 instructions that a stage does not need
// would be predicated and still take their time
template <int N, class O, bool PRE>
__device__ __forceinline__ void e3_body(const SolveDev& s, int e0, int cnt, int epb, const RKStage& rk, int update, int visc, double* sm) {
  constexpr int NS = D<N>::NS, NF1 = D<N>::NF1, NFP = D<N>::NFP;
  constexpr int NQ = 10;  // line quantities: eight flux components, two of A_z S

  double* sF = sm;                                          // [epb][NFP][8] total flux, then the residual
  double* sZ = sF + epb * NFP * 8;                          // [epb][NFP][2] A_z * (S_x, S_y), then grad A_z
  double* sQ = sZ + epb * NFP * 2;                          // [epb][NS][9] state (16-byte aligned: NFP is even)
  double* sU = sQ + ((epb * NS * 9 + 1) & ~1);              // [epb][NS][2] u, v; then the residual of A_z
  int64_t* sJ = reinterpret_cast<int64_t*>(sU + epb * NS * 2);  // [epb][NS] 1/J as an integer
  double* sD = sU + epb * NS * 2;                           // [epb][NS] diagnostic sums, in its place
  int* sE = reinterpret_cast<int*>(sJ + epb * NS);          // [epb][NS] and its exponent
  int* sK = sE + epb * NS;                                  // [epb][N][NQ] exponents of the xi-line sums
  __shared__ int list[64];
  // the residual of solution point p = (is, js) of a cell stands in the slot of family-1 flux
  // point js (N+1) + is, which its xi line has consumed
  auto slot = [](int e, int p) { return e * NFP + p + p / N; };
  // the block's fluxes and state, copied while the rest of the inputs is read
  block_copy_async(sF, (visc == 2 && !s.skip ? s.Ft : s.Fc) + (size_t)e0 * NFP * 8, cnt * NFP * 8);
  block_copy_async(sQ, s.Q + (size_t)e0 * NS * 9, cnt * NS * 9);
  cp_async_commit();
  {
    for (int i = threadIdx.x; i < cnt * NS; i += blockDim.x) {
      double j = s.invJ[(size_t)e0 * NS + i];
      if (PRE) j *= rk.cR;
      const uint32_t m = ix_abs_word(j);
      sJ[i] = ix_align<2>(j, m);
      sE[i] = m >= kIxLow && m < kIxHigh ? ix_exp<2>(m) : kE3Fp64;
    }
    const double2* met2 = reinterpret_cast<const double2*>(s.met);
    for (int i = threadIdx.x; i < cnt * NFP; i += blockDim.x) {
      const size_t g = (size_t)e0 * NFP + i;
      const double z = s.Azf[g];
      const double2 m = met2[g];
      sZ[2 * i] = z * m.x;
      sZ[2 * i + 1] = z * m.y;
    }
  }
  cp_async_wait();
  // the viscous flux: visc = 0 nothing left to do, 1 evaluated here, 2 by pass V, whose total
  // fluxes replace those of the cells that have one
  int nact = 0;
  if (visc == 1 || (visc == 2 && s.skip)) nact = active_cells(s, e0, cnt, list);  // (ends with a barrier)
  else __syncthreads();
  if (nact) {
    if (visc == 1) {
      e3_viscous<N, O>(s, e0, nact, list, sF, sU);  // (sU: free until the velocities)
    } else {
      for (int i = 0; i < nact; i++)
        block_copy_async(sF + list[i] * NFP * 8, s.Ft + (size_t)(e0 + list[i]) * NFP * 8, NFP * 8);
      cp_async_commit();
      cp_async_wait();
    }
    __syncthreads();
  }
  // divergence of the total flux and grad A_z in the conservative form of nablaAsp
  // (magnetic_potential.f90:1-42), (1/J) sum_r Mmat (A_z S): ten line quantities per cell,
  // each differentiated along its lines on the integer pipes, one (cell, line, quantity) per
  // thread; first the family-1 lines (xi), whose sums stay integers with one exponent per
  // line, then the family-2 lines (eta), which add theirs, multiply by 1/J and round once.
  // In integers these two operations cost about 20 instructions a value on pipes that the
  // FP64 work of the pass leaves idle, against 2 FP64 operations of 64 clocks a warp, and the
  // xi sums are not rounded in between.
  // 512x512 cells, N = 5 (GB300), a stage without terms of earlier states: 1.15 ms with the two
  // operations in FP64, the state read from global memory where it is used and predicated FP64
  // instructions (see PRE), 0.72 ms in this form; 9.2 kB per cell take 0.36 ms at the copy rate.
  // (the stage update takes the state's place as the residual appears: what else reads the old
  // state does so here)
  if (update && rk.save_old) block_copy_out(rk.save_old + (size_t)e0 * NS * 9, sQ, cnt * NS * 9);
  for (int t = threadIdx.x; t < cnt * NS; t += blockDim.x) {
    const double* q = sQ + 9 * t;
    const double ri = rcp_pos(q[0]);
    sU[2 * t] = q[1] * ri;
    sU[2 * t + 1] = q[2] * ri;
  }
#pragma unroll 1
  for (int fam = 0; fam < 2; fam++) {
    for (int t = threadIdx.x; t < cnt * N * NQ; t += blockDim.x) {
      const int k = t % NQ, el = t / NQ, e = el / N, ln = el - e * N;
      const bool fl = k < 8;
      // flux point r of line ln: family 1 at ln*(N+1) + r, family 2 at NF1 + r*N + ln
      const int fp0 = e * NFP + (fam ? NF1 + ln : ln * (N + 1)), fps = fam ? N : 1;
      double* base = fl ? sF + k : sZ + (k - 8);
      const int w = fl ? 8 : 2;
      double v[N + 1];
#pragma unroll
      for (int r = 0; r <= N; r++) v[r] = base[(fp0 + r * fps) * w];
      const uint32_t am = fix_amax(v);
      const bool ok = fix_line_ok(am) && am < kIxHigh;
      const int emax = max((int)(am >> 20), kFixEmaxMin), kv = ok ? emax - 1022 - O::ops().MS : kE3Fp64;
      auto fp64_row = [&](int i) {
        double a = 0.0;
#pragma unroll
        for (int r = 0; r <= N; r++) a += O::ops().M[r + (N + 1) * i] * v[r];
        return a;
      };
      if (!fam) {
        sK[t] = kv;
        if (ok) {
          fix_mirror_sums<N, N + 1, -1>(v, emax, O::ops().MH, O::ops().ML, [&](int i, int64_t V) {
            base[(fp0 + i) * w] = __longlong_as_double(V);
          });
        } else {
#pragma unroll
          for (int i = 0; i < N; i++) base[(fp0 + i) * w] = fp64_row(i);
        }
      } else {
        // row i is the solution point p = i N + ln
        auto finish = [&](int i, int64_t V) {
          const int p = i * N + ln, ps = e * NS + p, eJ = sE[ps], k0 = sK[(e * N + i) * NQ + k];
          double* at = base + slot(e, p) * w;
          const int64_t V0 = __double_as_longlong(*at);
          double a;
          if (ok && k0 != kE3Fp64 && eJ != kE3Fp64) {
            const int K = max(k0, kv);
            const int64_t sum = ix_shr(V0, K - k0 + O::ops().MV) + ix_shr(V, K - kv + O::ops().MV);
            a = fix_round_v<true>(ix_mul(fl ? -sum : sum, ix_limbs(sJ[ps])), K + O::ops().MV + eJ + 63);
          } else {
            double j = s.invJ[(size_t)e0 * NS + ps];
            if (PRE) j *= rk.cR;
            a = e3_fp64(V0, k0, V, kv, fl ? negate(j) : j);
          }
          *at = a;
          if (fl && (PRE || update)) {  // RK_S5P3 / FiveStageRk, but for the terms of earlier states
            double* q = sQ + 9 * ps + k;
            *q = PRE ? fma(rk.cQ, *q, a) : rk.cQ * *q + rk.cR * a;
          }
        };
        if (ok) {
          fix_mirror_sums<N, N + 1, -1>(v, emax, O::ops().MH, O::ops().ML, finish);
        } else {
#pragma unroll 1
          for (int i = 0; i < N; i++) finish(i, __double_as_longlong(fp64_row(i)));
        }
      }
    }
    __syncthreads();
  }
  // an earlier state's values go where the cells' family-2 fluxes were (8 NF1 >= 9 NS)
  static_assert(8 * (N + 1) * N >= 9 * N * N, "a cell's state fits its family-2 fluxes");
  auto src_slot = [&](int e) { return sF + (e * NFP + NF1) * 8; };
  if (update && rk.nsrc > 0) {
    for (int i = threadIdx.x; i < cnt * NS * 9; i += blockDim.x) {
      const int e = i / (NS * 9);
      cp_async8(src_slot(e) + (i - e * NS * 9), rk.src[0] + (size_t)e0 * NS * 9 + i);
    }
    cp_async_commit();
  }
  // A_z advection (resid(9), compresid.f90:45-47) at every solution point
  const bool b0 = s.B0x != 0.0 || s.B0y != 0.0;
  for (int t = threadIdx.x; t < cnt * NS; t += blockDim.x) {
    const int e = t / NS;
    const double* z = sZ + 2 * slot(e, t - e * NS);
    double ax = z[0], ay = z[1];
    if (!PRE && rk.write_resid) {  // kept for download; the last evaluation of a step writes it
      s.nAs[((size_t)e0 * NS + t) * 2] = ax;
      s.nAs[((size_t)e0 * NS + t) * 2 + 1] = ay;
    }
    if (b0) {  // (with cR folded in, the background gradient takes it too)
      ax -= PRE ? rk.cR * s.B0y : s.B0y;
      ay += PRE ? rk.cR * s.B0x : s.B0x;
    }
    const double r = negate(sU[2 * t] * ax + sU[2 * t + 1] * ay);
    sU[2 * t] = r;
    if (PRE || update) {
      double* q = sQ + 9 * t + 8;
      *q = PRE ? fma(rk.cQ, *q, r) : rk.cQ * *q + rk.cR * r;
    }
  }
  cp_async_wait();
  __syncthreads();
  const size_t g0 = (size_t)e0 * NS * 9;
  const int n = cnt * NS * 9;
  if (update) {
    if (rk.nsrc == 0 && !rk.R0) {
      block_copy_out(s.Q + g0, sQ, n);
      if (rk.save_new) block_copy_out(rk.save_new + g0, sQ, n);
    } else if (rk.nsrc == 1 && !rk.R0 && !rk.save_new) {
      const double c0 = rk.c[0];
#pragma unroll 4
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int e = i / (NS * 9);
        s.Q[g0 + i] = fma(c0, src_slot(e)[i - e * NS * 9], sQ[i]);
      }
    } else {
      // the terms of earlier states, elementwise over the block's contiguous state
#pragma unroll 4
      for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const size_t g = g0 + i;
        const int e = i / (NS * 9);
        double qn = sQ[i];
        if (rk.nsrc > 0) qn += rk.c[0] * src_slot(e)[i - e * NS * 9];
#pragma unroll
        for (int j = 1; j < 3; j++)
          if (j < rk.nsrc) qn += rk.c[j] * rk.src[j][g];
        if (rk.R0) qn += rk.cR0 * rk.R0[g];
        s.Q[g] = qn;
        if (rk.save_new) rk.save_new[g] = qn;
      }
    }
  }
  if (!PRE && (rk.write_resid || rk.save_R)) {
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int pt = i / 9, k = i - 9 * pt, e = pt / NS;
      const double r = k < 8 ? sF[8 * slot(e, pt - e * NS) + k] : sU[2 * pt];
      if (rk.write_resid) s.resid[g0 + i] = r;
      if (rk.save_R) rk.save_R[g0 + i] = r;
    }
  }
  if (!PRE && rk.diag) {
    for (int t = threadIdx.x; t < cnt * NS; t += blockDim.x) {
      const int e = t / NS;
      const double* r = sF + 8 * slot(e, t - e * NS);
      double acc = sU[2 * t] * sU[2 * t];
#pragma unroll
      for (int k = 0; k < 8; k++) acc += r[k] * r[k];
      sD[t] = acc;
    }
    __syncthreads();
  }
  if (!PRE && rk.diag) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    for (int e = warp; e < cnt; e += nwarp) {
      double acc = 0.0;
      for (int p = lane; p < NS; p += 32) acc += sD[e * NS + p];
      acc = warp_sum(acc);
      if (lane == 0) s.diag[2 * (e0 + e)] = acc;
    }
  }
}

// registers per thread of the pass: the line sums spill at 64, more cost resident CTAs.  A step of
// 800,000 points at 72 -> 80 (us; GB300): N = 3 1679 -> 1702, N = 4 1549 -> 1581, N = 5 1666 -> 1575,
// N = 6 1625 -> 1615, N = 7 1591 -> 1656, N = 8 1513 -> 1548.
constexpr int e3_regs(int N) { return N == 5 ? 80 : 72; }

template <int N, bool PRE>
__global__ void __maxnreg__(e3_regs(N)) k_e3(const __grid_constant__ SolveDev s, const __grid_constant__ RKStage rk, int epb, int update, int visc, int c0, int c1) {
  extern __shared__ __align__(16) double sm[];
  pdl_wait();
  const int e0 = c0 + blockIdx.x * epb;
  const int cnt = min(epb, c1 - e0);
  if (cnt <= 0) return;
  e3_body<N, OpsTU, PRE>(s, e0, cnt, epb, rk, update, visc, sm);
}

// ---------------------------------------------------------------------------
// CT projection (correct_B_via_curl_Az, setinitialcond.f90:82-91)
//   mode 0: A_z at every flux point (into Qvf variable 9)
//   mode 2: grad A_z from the face-averaged values, B <- B0 + curl A_z
// (mode 1, the face average, is k_ctface)
// ---------------------------------------------------------------------------
template <int N, class O>
__device__ __forceinline__ void ct_elem_body(const SolveDev& s, int e0, int cnt, int epb, int mode, double* sm) {
  constexpr int NS = D<N>::NS, NF1 = D<N>::NF1, NFP = D<N>::NFP;
  // the A_z traces go to Azf only, which the gradient below reads coalesced; the
  // reference's Qvfi(9)/Qvfj(9) are filled from Azf where they are read (downloads,
  // nablaQsp(9,9)), so the pass makes no strided writes into Qvf
  if (mode == 0) {
    double* sA = sm;  // [epb][NS] A_z at the solution points
    for (int i = threadIdx.x; i < cnt * NS; i += blockDim.x) sA[i] = s.Q[((size_t)e0 * NS + i) * 9 + 8];
    __syncthreads();
    // one (cell, line) per thread, the line operator on the integer pipes as in E1
    for (int t = threadIdx.x; t < cnt * 2 * N; t += blockDim.x) {
      const int e = t / (2 * N), line = t - e * 2 * N;
      const bool fam1 = line < N;
      const int ln = fam1 ? line : line - N;
      const double* qb = sA + e * NS + (fam1 ? ln * N : ln);
      const int qs = fam1 ? 1 : N;
      const int f0 = fam1 ? ln * (N + 1) : NF1 + ln, fs = fam1 ? 1 : N;
      double v[N], y[N + 1];
#pragma unroll
      for (int sp = 0; sp < N; sp++) v[sp] = qb[sp * qs];
      interp_line<N, O>(v, y);
      double* az = s.Azf + (size_t)(e0 + e) * NFP + f0;
#pragma unroll
      for (int f = 0; f <= N; f++) az[f * fs] = y[f];
    }
  } else {
    // nablaQsp(9,9) (compflux.f90:107-157): (1/J) sum_r Mmat (A_z S) over both line
    // families, each component differentiated along its lines on the integer pipes, one
    // (cell, line, component) per thread, the xi lines first; then update_B
    // (magnetic_potential.f90:44-67): B = B0 + curl A_z
    double* sZ = sm;                  // [epb][NFP][2] A_z * (S_x, S_y)
    double* sP = sZ + epb * NFP * 2;  // [epb][NS][2]  the xi-line part of the gradient
    for (int i = threadIdx.x; i < cnt * NFP; i += blockDim.x) {
      const size_t g = (size_t)e0 * NFP + i;
      const double z = s.Azf[g];
      const double2 m = reinterpret_cast<const double2*>(s.met)[g];
      sZ[2 * i] = z * m.x;
      sZ[2 * i + 1] = z * m.y;
    }
    __syncthreads();
#pragma unroll 1
    for (int fam = 0; fam < 2; fam++) {
      for (int t = threadIdx.x; t < cnt * N * 2; t += blockDim.x) {
        const int c = t & 1, el = t >> 1, e = el / N, ln = el - e * N;
        const int fp0 = fam ? NF1 + ln : ln * (N + 1), fps = fam ? N : 1;
        double y[N];
        deriv_line<N, O>(sZ + (e * NFP + fp0) * 2 + c, fps * 2, y);
        const int p0 = e * NS + (fam ? ln : ln * N), ps = fam ? N : 1;
        if (!fam) {
#pragma unroll
          for (int i = 0; i < N; i++) sP[(p0 + i * ps) * 2 + c] = y[i];
        } else {
#pragma unroll
          for (int i = 0; i < N; i++) {
            const size_t gs = (size_t)e0 * NS + p0 + i * ps;
            const double a = (sP[(p0 + i * ps) * 2 + c] + y[i]) * s.invJ[gs];
            s.nQs9[gs * 2 + c] = a;
            if (c) s.Q[gs * 9 + 5] = a + s.B0x;  // Bx = dA/dy
            else s.Q[gs * 9 + 6] = s.B0y - a;    // By = -dA/dx
          }
        }
      }
      __syncthreads();
    }
  }
}

template <int N>
__global__ void __launch_bounds__(256) k_ct_elem(SolveDev s, int epb, int mode, int c0, int c1) {
  extern __shared__ __align__(16) double sm[];
  pdl_wait();
  const int e0 = c0 + blockIdx.x * epb;
  const int cnt = min(epb, c1 - e0);
  if (cnt <= 0) return;
  ct_elem_body<N, OpsTU>(s, e0, cnt, epb, mode, sm);
}

template <int N>
__device__ __forceinline__ void ctface_point(const SolveDev& s, int t) {
  constexpr int NFP = D<N>::NFP;
  if (t >= s.nface2 * N) return;
  const int f = t / N, nfp = t - f * N;
  const int4 fc = s.face2[f];
  const size_t gl = (size_t)fc.x * NFP + face_fp<N>(fc.y, nfp);
  const size_t gr = (size_t)fc.z * NFP + face_fp<N>(fc.w, N - 1 - nfp);
  const double v = half(s.Azf[gl] + s.Azf[gr]);
  s.Azf[gl] = v;
  s.Azf[gr] = v;
}

// the points of two-sided faces [f0, f1)
template <int N>
__global__ void __launch_bounds__(256) k_ct_face(SolveDev s, int f0, int f1) {
  pdl_wait();
  const int t = f0 * N + blockIdx.x * blockDim.x + threadIdx.x;
  if (t < f1 * N) ctface_point<N>(s, t);
}

// The diagnostic of iterations.f90:35-36 (comp_inviscid_flux, then nablaQsp(6,7) for
// div B) reads only B_x and B_y at the flux points: interpolate those two variables of
// the CT-corrected state (mode 0, one (cell, line, variable) per thread, the mirror
// symmetry of the points as in E1) and average them across the two-sided faces (the face
// pass below), as interfaceflux/CYCLOCFLUX do (interfaceflux_all.f90:79-91); a FREE face
// keeps its interior trace (bcflux.f90).
template <int N, class O>
__device__ __forceinline__ void diag_interp_body(const SolveDev& s, int e0, int cnt, double* sm) {
  constexpr int NS = D<N>::NS, NF1 = D<N>::NF1, NFP = D<N>::NFP;
  double* sB = sm;  // [cnt][NS][2] B_x, B_y
  for (int i = threadIdx.x; i < cnt * NS * 2; i += blockDim.x)
    sB[i] = s.Q[((size_t)e0 * NS + (i >> 1)) * 9 + 5 + (i & 1)];
  __syncthreads();
  for (int t = threadIdx.x; t < cnt * 2 * N * 2; t += blockDim.x) {
    const int v = t & 1, el = t >> 1, e = el / (2 * N), line = el - e * 2 * N;
    const bool fam1 = line < N;
    const int ln = fam1 ? line : line - N;
    const double* qb = sB + (e * NS + (fam1 ? ln * N : ln)) * 2 + v;
    const int qs = fam1 ? 2 : 2 * N;
    const int f0 = fam1 ? ln * (N + 1) : NF1 + ln, fs = fam1 ? 1 : N;
    double* ob = s.Qvf + ((size_t)(e0 + e) * NFP + f0) * 9 + 5 + v;
    double w[N], y[N + 1];
#pragma unroll
    for (int sp = 0; sp < N; sp++) w[sp] = qb[sp * qs];
    interp_line<N, O>(w, y);
#pragma unroll
    for (int f = 0; f <= N; f++) ob[(size_t)f * fs * 9] = y[f];
  }
}

template <int N>
__global__ void __launch_bounds__(256) k_diag_interp(SolveDev s, int epb) {
  extern __shared__ __align__(16) double sm[];
  const int e0 = blockIdx.x * epb;
  const int cnt = min(epb, s.NC - e0);
  if (cnt <= 0) return;
  diag_interp_body<N, OpsTU>(s, e0, cnt, sm);
}

template <int N>
__global__ void __launch_bounds__(256) k_diag_face(SolveDev s) {
  constexpr int NFP = D<N>::NFP;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= s.nface2 * N) return;
  const int f = t / N, nfp = t - f * N;
  const int4 fc = s.face2[f];
  double* a = s.Qvf + ((size_t)fc.x * NFP + face_fp<N>(fc.y, nfp)) * 9 + 5;
  double* b = s.Qvf + ((size_t)fc.z * NFP + face_fp<N>(fc.w, N - 1 - nfp)) * 9 + 5;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const double v = half(a[k] + b[k]);
    a[k] = v;
    b[k] = v;
  }
}

// nablaQsp(v0..v1) (compflux.f90:107-157) from the current Qvf, 0-based variables, for
// cells [e0, e0+cnt): the conservative form of E2 (metric-state products differentiated
// along the lines on the integer pipes), 2 (v1-v0+1) line quantities per cell
template <int N, class O>
__device__ __forceinline__ void nqsp_cells(const SolveDev& s, int e0, int cnt, int v0, int v1, double* sm) {
  constexpr int NS = D<N>::NS, NF1 = D<N>::NF1, NFP = D<N>::NFP;
  const int nv = v1 - v0 + 1, NQ = 2 * nv;
  double* sP = sm;                  // [cnt][NFP][NQ] Q_k * S_x (k < nv), Q_k * S_y
  double* sG = sP + cnt * NFP * NQ;  // [cnt][NS][NQ] the xi-line part
  for (int i = threadIdx.x; i < cnt * NFP * nv; i += blockDim.x) {
    const int kk = i % nv, lf = i / nv;
    const size_t g = (size_t)e0 * NFP + lf;
    const double q = s.Qvf[g * 9 + v0 + kk];
    sP[lf * NQ + kk] = q * s.met[2 * g];
    sP[lf * NQ + nv + kk] = q * s.met[2 * g + 1];
  }
  __syncthreads();
#pragma unroll 1
  for (int fam = 0; fam < 2; fam++) {
    for (int t = threadIdx.x; t < cnt * N * NQ; t += blockDim.x) {
      const int c = t % NQ, el = t / NQ, le = el / N, ln = el - le * N;
      const int fp0 = fam ? NF1 + ln : ln * (N + 1), fps = fam ? N : 1;
      double y[N];
      deriv_line<N, O>(sP + (le * NFP + fp0) * NQ + c, fps * NQ, y);
      const int p0 = fam ? ln : ln * N, ps = fam ? N : 1;
      double* g = sG + (le * NS + p0) * NQ + c;
      if (!fam) {
#pragma unroll
        for (int i = 0; i < N; i++) g[i * ps * NQ] = y[i];
      } else {
        const int k = v0 + c % nv, d = c / nv;
#pragma unroll
        for (int i = 0; i < N; i++) {
          const size_t gs = (size_t)(e0 + le) * NS + p0 + i * ps;
          const double a = (g[i * ps * NQ] + y[i]) * s.invJ[gs];
          if (k < 8) s.nQs[gs * 18 + 9 * d + k] = a;
          else s.nQs9[gs * 2 + d] = a;  // variable 9 is kept in its own array
        }
      }
    }
    __syncthreads();
  }
}

template <int N>
__global__ void __launch_bounds__(256) k_nqsp(SolveDev s, int epb, int v0, int v1) {
  extern __shared__ __align__(16) double sm[];
  const int e0 = blockIdx.x * epb;
  const int cnt = min(epb, s.NC - e0);
  if (cnt <= 0) return;
  nqsp_cells<N, OpsTU>(s, e0, cnt, v0, v1, sm);
}

// per-cell sum of (dBx/dx + dBy/dy)^2 (iterations.f90:48) into diag[e][1]
template <int N>
__global__ void __launch_bounds__(256) k_divb(SolveDev s) {
  constexpr int NS = D<N>::NS;
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= s.NC) return;
  double acc = 0.0;
  for (int p = 0; p < NS; p++) {
    const double* g = s.nQs + ((size_t)c * NS + p) * 18;
    const double d = g[5] + g[9 + 6];
    acc += d * d;
  }
  s.diag[2 * c + 1] = acc;
}

}  // namespace chorus
