// kernels_inst.cuh -- explicit instantiation of the stage kernels for N = CHORUS_N.
// Each translation unit holds its own constant-memory copy of the N-point operators.
#include <algorithm>

#include "kernels.cuh"

#ifndef CHORUS_N
#error "define CHORUS_N before including kernels_inst.cuh"
#endif
#define CHORUS_CAT2(a, b) a##b
#define CHORUS_CAT(a, b) CHORUS_CAT2(a, b)

namespace chorus {

namespace {
constexpr int kN = CHORUS_N;
inline size_t smem_e1(int epb) {
  return sizeof(double) * ((size_t)epb * (D<kN>::NS * 9 + 2 * D<kN>::NS + D<kN>::NFP * 9) + kN * kN);
}
inline size_t smem_ct(int epb) { return sizeof(double) * epb * (D<kN>::NFP * 2 + D<kN>::NS * 2); }
inline int grid_cells(int nc, int epb) { return (nc + epb - 1) / epb; }

// threads per CTA of a face-point pass: 256, or 64 when that leaves fewer than about
// eight CTAs per SM (small meshes), so that the points spread over every SM
inline int face_threads(int n) { return n >= 152 * 8 * 256 ? 256 : 64; }

// SMs of the current device, looked up once
int sm_count() {
  static int nsm_of[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return 152;
  if (!nsm_of[dev] && (cudaDeviceGetAttribute(&nsm_of[dev], cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
                       nsm_of[dev] <= 0))
    nsm_of[dev] = 152;
  return nsm_of[dev];
}

// Cells per CTA of a launch over n cells: the tuned number, or fewer where that leaves an SM
// fewer than four CTAs, since the pass then lasts as long as one CTA takes for its cells.  A step
// of all passes and the CT projection, tuned -> spread (us a step; GB300, without AV): N = 3,
// 1024 cells 116 -> 96; N = 4, 784 cells 117 -> 103; N = 5, 576 cells 134 -> 107; N = 6, 256 cells
// 140 -> 109; N = 8, 324 cells 150 -> 132; N = 5, 2304 cells 183 -> 175; N = 2, 10000 cells 161.
// A line at six CTAs: N = 6, 1600 cells 177 instead of 191, but N = 8, 784 cells 184 against 168.
// From four CTAs per SM on the tuned number is as good or better.
inline int spread(int n, int epb) {
  const int ctas = 4 * sm_count();
  return std::max(1, std::min(epb, (n + ctas - 1) / ctas));
}

// The same for E3, whose loops are over the 10 N line quantities of a cell and family: on a
// launch of few CTAs, down to half as many cells, the number whose lines fill the threads best,
// since little covers a CTA's part-filled last turn there.
// Tuned -> this (us a step; GB300): N = 6, 3969 cells 338 -> 321, 1600 cells 185 -> 179; N = 3, 8100
// cells 197 -> 189; N = 2, 10000 cells 162 -> 158.  From some 12 CTAs per SM on the bigger CTAs
// are as good or better: N = 3, 19600 cells (16 per SM) 400 -> 403; N = 2, 32400 cells (13) 345 -> 348.
inline int e3_cells(int n, const Launch& L) {
  const int epb = spread(n, L.epb), lines = 10 * kN;
  if (grid_cells(n, epb) >= 12 * sm_count()) return epb;
  auto idle = [&](int e) { return (e * lines + L.threads - 1) / L.threads * L.threads / (double)(e * lines); };
  int best = epb;
  for (int e = epb - 1; 2 * e > epb; e--)
    if (idle(e) < idle(best)) best = e;
  return best;
}

void set_smem_limits() {
  static bool done[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && done[dev]) return;
  const int lim = 200 * 1024;
  cudaFuncSetAttribute(k_e1<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  cudaFuncSetAttribute(k_e2<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  cudaFuncSetAttribute(k_v<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  cudaFuncSetAttribute(k_f1<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  cudaFuncSetAttribute(k_e3<kN, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, e3_smem_limit(kN));
  cudaFuncSetAttribute(k_e3<kN, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, e3_smem_limit(kN));
  cudaFuncSetAttribute(k_ct_elem<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  cudaFuncSetAttribute(k_diag_interp<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  cudaFuncSetAttribute(k_nqsp<kN>, cudaFuncAttributeMaxDynamicSharedMemorySize, lim);
  if (dev < 64) done[dev] = true;
}
}  // namespace

void CHORUS_CAT(upload_ops_n, CHORUS_N)(const OpsN& o) {
  set_smem_limits();
  cudaMemcpyToSymbol(c_ops, &o, sizeof(OpsN));
}

template <>
void launch_e1<kN>(const SolveDev& s, const Launch& L, cudaStream_t st, int plot, int c0, int c1) {
  const int sensor = (s.artiv ? (plot ? 3 : 1) : 0) | 4;  // 4: also reset the stage's wave speed
  if (c1 < 0) c1 = s.NC;
  const int epb = spread(c1 - c0, L.epb);
  if (c1 > c0) launch_pdl(k_e1<kN>, grid_cells(c1 - c0, epb), L.threads, smem_e1(epb), st, s, epb, sensor, c0, c1);
}
void CHORUS_CAT(launch_e1_nosensor_n, CHORUS_N)(const SolveDev& s, const Launch& L, cudaStream_t st) {
  launch_pdl(k_e1<kN>, grid_cells(s.NC, L.epb), L.threads, smem_e1(L.epb), st, s, L.epb, 0, 0, s.NC);
}
template <>
void launch_f1<kN>(const SolveDev& s, cudaStream_t st, int a2, int b2, int a1, int b1) {
  if (b2 < 0) b2 = s.nface2;
  if (b1 < 0) b1 = s.nface1;
  const int n2 = (b2 - a2) * kN, n = n2 + (b1 - a1) * kN;
  // two resident CTAs of kF1Threads per SM walk the points; fewer points than that go one
  // to a thread, in CTAs of 64 so that they spread over every SM
  const int thr = n >= 2 * kF1Threads * sm_count() ? kF1Threads : 64;
  const int grid = std::min((n + thr - 1) / thr, thr == kF1Threads ? 2 * sm_count() : n);
  if (n > 0)
    launch_pdl(k_f1<kN>, grid, thr, f1_smem(thr), st, s, a2 * kN, n2, (s.nface2 + a1) * kN, n);
}
template <>
void launch_e2<kN>(const SolveDev& s, const Launch& L, cudaStream_t st, bool keep) {
  // every cell: a CTA per group; a list of unknown length: eight CTAs per SM walk it
  const int nsm = sm_count();
  const int all2 = grid_cells(s.NC, L.epb);
  launch_pdl(k_e2<kN>, s.skip ? std::min(all2, 8 * nsm) : all2, L.threads, e2_smem(kN, L.epb), st, s, L.epb, (int)keep);
  if (v_pass(s) && viscous(s)) {
    const int allv = grid_cells(s.NC, v_epb(kN));
    launch_pdl(k_v<kN>, s.skip ? std::min(allv, 8 * nsm) : allv, v_threads(kN), v_smem(kN), st, s, keep ? s.Ft : s.Fc);
  }
}
template <>
void launch_qavg<kN>(const SolveDev& s, cudaStream_t st) {
  const int n = s.nface2 * kN;
  if (n > 0) k_qavg<kN><<<(n + face_threads(n) - 1) / face_threads(n), face_threads(n), 0, st>>>(s);
}
template <>
void launch_f2<kN>(const SolveDev& s, cudaStream_t st) {
  const int n = (s.nface2 + s.nface1) * kN;
  if (n > 0) k_f2<kN><<<(n + face_threads(n) - 1) / face_threads(n), face_threads(n), 0, st>>>(s);
}
template <>
void launch_e3<kN>(const SolveDev& s, const RKStage& rk, const Launch& L, cudaStream_t st, int c0, int c1) {
  const int update = (rk.cQ != 0.0 || rk.cR != 0.0 || rk.nsrc > 0) ? 1 : 0;
  if (c1 < 0) c1 = s.NC;
  const int epb = e3_cells(c1 - c0, L);
  if (c1 > c0)
    launch_pdl(e3_pre(rk, update) ? k_e3<kN, true> : k_e3<kN, false>, grid_cells(c1 - c0, epb), L.threads,
               e3_smem(kN, epb), st, s, rk, epb, update, e3_visc(s, rk.write_resid), c0, c1);
}
template <>
void launch_ct<kN>(const SolveDev& s, const Launch& L, cudaStream_t st, int mode, int c0, int c1) {
  if (mode == 1) {
    if (c1 < 0) c1 = s.nface2;
    const int n = (c1 - c0) * kN;
    if (n > 0)
      launch_pdl(k_ct_face<kN>, (n + face_threads(n) - 1) / face_threads(n), face_threads(n), 0, st, s, c0, c1);
  } else {
    if (c1 < 0) c1 = s.NC;
    const int epb = spread(c1 - c0, L.epb);
    if (c1 > c0) launch_pdl(k_ct_elem<kN>, grid_cells(c1 - c0, epb), L.threads, smem_ct(epb), st, s, epb, mode, c0, c1);
  }
}
template <>
void launch_diag<kN>(const SolveDev& s, const Launch& L, cudaStream_t st, int mode) {
  if (mode == 0) {
    k_diag_interp<kN><<<grid_cells(s.NC, L.epb), L.threads, sizeof(double) * L.epb * D<kN>::NS * 2, st>>>(s, L.epb);
  } else {
    const int n = s.nface2 * kN;
    if (n > 0) k_diag_face<kN><<<(n + face_threads(n) - 1) / face_threads(n), face_threads(n), 0, st>>>(s);
  }
}
template <>
void launch_nqsp<kN>(const SolveDev& s, int v0, int v1, cudaStream_t st) {
  // 4 cells per 128 threads; 12 kB of shared memory per cell for all nine variables
  const int epb = 4, nq = 2 * (v1 - v0 + 1);
  const size_t smem = sizeof(double) * epb * (size_t)(D<kN>::NFP + D<kN>::NS) * nq;
  k_nqsp<kN><<<grid_cells(s.NC, epb), 128, smem, st>>>(s, epb, v0, v1);
}
template <>
void launch_divb<kN>(const SolveDev& s, cudaStream_t st) {
  k_divb<kN><<<(s.NC + 255) / 256, 256, 0, st>>>(s);
}

}  // namespace chorus
