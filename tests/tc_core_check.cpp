// Checks on the CPU that the Toeplitz buffer of a launch (tc_core_matrices in
// tc_schedule.h, the core matrices the builder warps write) holds everything
// the MMA windows read: for every case "Wl Wr tf32" on standard input prints
// "ok" or "FAIL <core matrices> <largest read + 1> of <buffer>".  Three forms
// of a launch's shifts: x-parts of 512, one range (at most 256 shifts), and
// even x-parts, whose windows are also checked to cover every shift that meets
// the left row ("FAIL shift ...").
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
    for (int form = 0; form < 3; ++form) {
    const bool one = form == 1, even = form == 2;
    if ((one && Sx > kHalfCols) || (even && t.n_xparts == 1)) continue;
    const int width = one ? (Sx + 15) / 16 * 16 : even ? tc_even_half(Sx, t.n_xparts) : t.half_w;
    const int halves = one ? 1 : 2, part = even ? 2 * width : 512;
    if (even && (width > kHalfCols || part * t.n_xparts < Sx)) {
      std::printf("FAIL parts of %d\n", part);
      return 0;
    }
    const int nq = tc_core_matrices(halves * width, Wr, tf != 0);
    int most = 0;
    for (int xp = 0; xp < t.n_xparts; ++xp)
      for (int kp = 0; kp < t.n_kparts; ++kp)
        for (int h = 0; h < halves; ++h)
          for (int j = -1; j < 256 / t.kstep; ++j) {
            const int kbase = 256 * kp, k0 = kbase + std::max(0, j) * t.kstep;
            const uint32_t e = window_of(Sx, Wl, Wr, width, t.kstep, part * xp, kbase, h, k0, j < 0);
            const int H0 = part * xp + h * width, w0 = H0 + (int)(e & 511u) - h * kHalfCols;
            const int w1 = (e >> 14) & 1u ? w0 + (int)((e >> 9) & 31u) * 16 : w0;
            for (int sx = H0; even && j >= 0 && sx < std::min(Sx, H0 + width); ++sx) {
              bool meets = false;
              for (int k = k0; k < std::min(Wr, k0 + t.kstep); ++k) meets = meets || (sx + k - (Wr - 1) >= 0 && sx + k - (Wr - 1) < Wl);
              if (meets && (sx < w0 || sx >= w1)) {
                std::printf("FAIL shift %d\n", sx);
                return 0;
              }
            }
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
