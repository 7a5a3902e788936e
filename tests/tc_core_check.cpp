// Checks on the CPU that the Toeplitz buffer of a launch (tc_core_matrices in
// tc_schedule.h, the core matrices the builder warps write) holds everything
// the MMA windows read: for every case "Wl Wr tf32" on standard input prints
// "ok" or "FAIL <core matrices> <largest read + 1> of <buffer>".
#include <algorithm>
#include <cstdio>

#include "tc_schedule.h"

using namespace xc;

int main() {
  int Wl, Wr, tf;
  while (std::scanf("%d %d %d", &Wl, &Wr, &tf) == 3) {
    const int Sx = Wl + Wr - 1;
    const TcParts t = tc_parts(Sx, Wr, tf != 0);
    // one group of eight shifts is one core matrix (BF16) or two (TF32), one
    // K-step two
    const int group = tf ? 2 : 1;
    // two halves per part, and (at most 256 shifts) one range of whole windows
    for (int one = 0; one <= (Sx <= kHalfCols ? 1 : 0); ++one) {
    const int width = one ? (Sx + 15) / 16 * 16 : t.half_w, halves = one ? 1 : 2;
    const int nq = tc_core_matrices(halves * width, Wr, tf != 0);
    int most = 0;
    for (int xp = 0; xp < t.n_xparts; ++xp)
      for (int kp = 0; kp < t.n_kparts; ++kp)
        for (int h = 0; h < halves; ++h)
          for (int j = -1; j < 256 / t.kstep; ++j) {
            const int kbase = 256 * kp, k0 = kbase + std::max(0, j) * t.kstep;
            const uint32_t e = window_of(Sx, Wl, Wr, width, t.kstep, 512 * xp, kbase, h, k0, j < 0);
            if (!((e >> 14) & 1u)) continue;
            const int n = (int)((e >> 9) & 31u) * 16;
            most = std::max(most, (int)(e >> 16) + (n / 8 - 1) * group + 1 + 1);
          }
    const int kq = one ? (tf ? 128 : 64) : tf ? kTQTf32 : kTQBf16;
    if (most > nq || nq > kq) {
      std::printf("FAIL %d %d of %d\n", nq, most, kq);
      return 0;
    }
    }
    std::printf("ok\n");
  }
  return 0;
}
