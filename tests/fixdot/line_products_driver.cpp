// Host driver of the products of a line's states and metric entries (ix_line_products,
// chorus-mhd_gb300/csrc/intflux.cuh): reads  int n; double q[n][6], s[n][6]  from argv[1], writes
// n records of doubles to argv[2]: the exponent, then the upper and lower parts of the six
// integers (X = upper 2^30 + lower).
#include <cstdio>
#include <vector>

#include "intflux.cuh"

using namespace chorus;

int main(int argc, char** argv) {
  if (argc != 3) return 2;
  FILE* f = std::fopen(argv[1], "rb");
  int n;
  if (!f || std::fread(&n, sizeof(int), 1, f) != 1 || n < 0) return 2;
  std::vector<double> q((size_t)n * 6), s((size_t)n * 6), out((size_t)n * 13);
  if (std::fread(q.data(), sizeof(double), q.size(), f) != q.size()) return 2;
  if (std::fread(s.data(), sizeof(double), s.size(), f) != s.size()) return 2;
  std::fclose(f);
  for (int i = 0; i < n; i++) {
    int64_t X[6];
    double* o = &out[(size_t)i * 13];
    o[0] = ix_line_products<6>([&](int r) { return ix_load(q[6 * i + r]); }, [&](int r) { return ix_load(s[6 * i + r]); }, X);
    for (int r = 0; r < 6; r++) {
      o[1 + 2 * r] = (double)(X[r] >> 30);
      o[2 + 2 * r] = (double)(X[r] & ((1 << 30) - 1));
    }
  }
  FILE* g = std::fopen(argv[2], "wb");
  if (!g) return 2;
  std::fwrite(out.data(), sizeof(double), out.size(), g);
  std::fclose(g);
  return 0;
}
