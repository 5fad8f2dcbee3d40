// Every geometry of the streaming GEMV over a range of devices and sizes has a form of the kernel that serves it: more than two
// parts of K only for one token through strips of two boxes, all of the matrix's columns covered, no part of K empty.
#include <cstdio>

#include "kernels.h"

int main() {
  using namespace mld;
  // one token on 148 SMs: K cut into more than two parts only where it pays
  const int parts[][4] = {{4, 8192, 4608, 2}, {8, 3072, 4608, 2}, {8, 4096, 6144, 2}, {4, 4584, 8704, 2},  // bits, N, K, parts
                          {4, 5120, 6144, 4}, {4, 5120, 10240, 5}, {4, 4096, 14336, 7}, {4, 4608, 16384, 7}};
  for (const auto& c : parts) {
    const StripGeometry g = strip_geometry(c[0], c[1], c[2], 1, 8, MLD_SCALE_BLOCK, 148, true, 0, false, true);
    if (g.ksplit != c[3]) {
      printf("bits %d N %d K %d: %d parts\n", c[0], c[1], c[2], g.ksplit);
      return 1;
    }
  }
  long n = 0;
  for (int sms : {1, 2, 3, 4, 6, 8, 9, 16, 74, 147, 148})
    for (int bits : {4, 8})
      for (int N = 8; N < 300000; N = N * 5 / 4 / 8 * 8 + 8)  // (others take the general kernel)
        for (int K = 64; K <= 16384; K = K * 4 / 3 / 4 * 4 + 64)
          for (int m : {1, 2, 8, 12, 32})
            for (int zp = 0; zp < 2; ++zp, ++n) {
              const StripGeometry g = strip_geometry(bits, N, K, m, 8, MLD_SCALE_BLOCK, sms, true, 0, zp != 0, true);
              const bool cut = g.ksplit <= 2 || (m == 1 && g.w == 2);
              const int rows = (K + 3) / 4, chunks = (N + 3) / 4 * (bits == 4 ? 8 : 16) / 16;
              const bool parts = g.ksplit == 1 || (g.ksplit - 1) * g.rows_per_split < rows;
              const bool whole = g.grid == g.strips * g.ksplit && g.strips >= 1 && g.ksplit * g.rows_per_split >= rows;
              // (an average strip's share of the boxes that it fetches: no more than all)
              if (!cut || !parts || !whole || (chunks >= g.strips && g.fill > 100)) {
                printf("sms %d bits %d N %d K %d tokens %d zp %d: %d parts, %d boxes, %d strips, fill %d\n", sms, bits, N, K, m, zp,
                       g.ksplit, g.w, g.strips, g.fill);
                return 1;
              }
            }
  printf("%ld geometries\n", n);
  return 0;
}
