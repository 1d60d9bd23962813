// Every pair of neighbouring blocks with up to 6 groups each, up to 9 groups apart:
// what one sends is what the other waits for, group by group, in both sweeps.
#include <cstdio>
#include <set>

#include "../../xfluid_b200/csrc/xfp_edges.h"

using namespace xfp;

int main() {
  long checked = 0;
  for (int rev = 0; rev < 2; ++rev)
    for (int p_ng = 0; p_ng <= 6; ++p_ng)
      for (int c_ng = 0; c_ng <= 6; ++c_ng)
        for (int apart = -9; apart <= 9; ++apart) {
          // a block without groups is all zeros in the table
          const int p_g0 = p_ng ? 5 : 0, c_g0 = c_ng ? 5 + apart : 0;
          const int shift = edge_shift(rev, p_g0, p_ng, c_g0, c_ng);
          // the global group of a block's q-th group in sweep order
          auto global = [&](int g0, int ng, int q) { return rev ? g0 + ng - 1 - q : g0 + q; };
          std::set<int> wanted, sent, range;
          if (c_ng > 0)
            for (int u = 0; u <= c_ng; ++u) {
              if (edge_comes(u, shift, p_ng)) wanted.insert(u);
              // the producer's group is the consumer's group u - 1
              if (edge_comes(u, shift, p_ng) && global(p_g0, p_ng, u + shift) != global(c_g0, c_ng, u - 1)) return 1;
            }
          if (p_ng > 0)
            for (int q = 0; q < p_ng; ++q)
              if (q >= shift && q <= last_sent(shift, p_ng, c_ng)) sent.insert(q - shift);
          if (c_ng > 0)
            for (int u = first_edge(shift); u <= last_edge(shift, p_ng, c_ng); ++u) range.insert(u);
          if (wanted != sent || wanted != range) {
            std::fprintf(stderr, "rev %d, producer %d groups, consumer %d, %d apart\n", rev, p_ng, c_ng, apart);
            return 1;
          }
          checked += (long)wanted.size();
        }
  std::printf("%ld\n", checked);
  return checked > 1000 ? 0 : 2;
}
