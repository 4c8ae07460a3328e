// intflux_driver in out: evaluates the integer point fluxes of intflux.cuh on the host.
// Input: int kind (0 Rusanov, 1 interior, 2 viscous), int n, then n records of doubles:
//   kind 0: ql[8], qr[8], ux, uy, scale, gamma;  kind 1: q[8], sx, sy, gamma;
//   kind 2: q[8], dq/dx[8], dq/dy[8], viscosity, resistivity, sx, sy, gamma
// Output: n records of doubles: 1 if the integer form took the point, F[8], the wave speed
// (kind 0 only).
#include <cstdio>
#include <vector>

#include "intflux.cuh"

using namespace chorus;

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  FILE* f = std::fopen(argv[1], "rb");
  int hdr[2];
  if (!f || std::fread(hdr, sizeof(int), 2, f) != 2) return 2;
  const int kind = hdr[0], n = hdr[1], w = kind == 2 ? 29 : kind ? 11 : 20, wo = kind ? 9 : 10;
  std::vector<double> in((size_t)n * w), out((size_t)n * wo, 0.0);
  if (std::fread(in.data(), sizeof(double), in.size(), f) != in.size()) return 2;
  std::fclose(f);
  for (int i = 0; i < n; i++) {
    const double* a = &in[(size_t)i * w];
    double* o = &out[(size_t)i * wo];
    auto put = [&](int j, double x, double y) {
      o[1 + 2 * j] = x;
      o[2 + 2 * j] = y;
    };
    if (kind == 0)
      o[0] = rusanov_int([&](int side, int k) { return a[8 * side + k]; }, a[16], a[17], ix_gas(a[19]), a[18], o[9], put);
    else if (kind == 2)
      o[0] = vflux_int([&](int k) { return a[k]; }, [&](int d, int k) { return a[8 + 8 * d + k]; }, a[24], a[25], a[26],
                       a[27], ix_gas(a[28]), [&](int k, double x) { o[1 + k] = x; });
    else
      o[0] = iflux_int([&](int k) { return a[k]; }, a[8], a[9], ix_gas(a[10]), put);
  }
  FILE* g = std::fopen(argv[2], "wb");
  if (!g) return 2;
  std::fwrite(out.data(), sizeof(double), out.size(), g);
  std::fclose(g);
  return 0;
}
