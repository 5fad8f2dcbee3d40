// Decode attention's split of its heads over a range of devices, heads and cache lengths: no part without a round of tokens for
// its warps, and a launch whose clusters and CTAs are resident at once wherever it has more than one CTA to a head.
#include <cstdio>

#include "kernels.h"

int main() {
  using namespace mld;
  long n = 0;
  for (int sms : {1, 2, 8, 16, 74, 132, 147, 148})
    for (int heads = 1; heads <= 5000; heads = heads < 700 ? heads + 1 : heads * 2)
      for (int tokens = 1; tokens <= 40000; tokens += 1 + tokens / 9)
        for (int by16 : {0, sms / 10, sms / 8}) {
          ++n;
          const AttnShape s = attn_shape(heads, tokens, sms, by16);
          const int ctas = heads * s.parts, warps = ctas * s.warps, round = s.warps * 16;
          const bool form = (s.warps == 4 || s.warps == 8) && s.parts >= 1 && s.parts <= 16 && (s.warps == 8 || s.parts <= 9);
          // an SM holds sixteen warps; clusters of three to nine CTAs find places for seven eighths of that, larger ones for seven
          // tenths or as many as the device says
          const bool resident = s.parts == 1   ? s.warps == 4 || warps <= 16 * sms
                                : s.parts == 2 ? warps <= 16 * sms
                                : s.parts < 9 || s.warps == 4 ? warps <= 14 * sms
                                : s.parts < 16 ? 5 * ctas <= 7 * sms
                                               : heads <= by16;
          if (!form || !resident || (s.parts - 1) * round >= tokens) {
            printf("%d SMs, %d heads of %d tokens: %d parts of %d warps\n", sms, heads, tokens, s.parts, s.warps);
            return 1;
          }
        }
  printf("%ld shapes\n", n);
  return 0;
}
