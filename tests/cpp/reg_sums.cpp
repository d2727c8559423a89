// Host model of the phases in which k_reg_solve exchanges its partial sums of
// Dif^2 (reg_sums.h): in phase 2 of iteration it every CTA reads all blocks' sums
// of it - 1, then stores its own of it; a barrier follows.  The sums lie where the
// header puts them.  Every CTA in turn is the late one: it reads after all others
// have stored.  Exit status 0: nobody ever read another iteration's sum.
#include <cstdio>
#include <vector>

#include "reg_sums.h"

int main() {
  for (int blocks : {1, 2, 3, 7, 25, 400}) {
    for (int late = 0; late < blocks; ++late) {
      std::vector<int> part(gbn::reg_dif_floats(size_t(blocks)), -1);  // the iteration each stored sum is of
      for (int it = 1; it <= 7; ++it) {
        auto read = [&]() {
          if (it < 2) return true;
          for (int b = 0; b < blocks; ++b)
            if (part[gbn::reg_dif_at(it - 1, blocks) + size_t(b)] != it - 1) return false;
          return true;
        };
        auto store = [&](int b) { part[gbn::reg_dif_at(it, blocks) + size_t(b)] = it; };
        bool ok = read();  // the CTAs in time
        for (int b = 0; b < blocks; ++b)
          if (b != late) store(b);
        ok = ok && read();  // the late one
        store(late);
        if (!ok) {
          std::printf("blocks %d, iteration %d, CTA %d late: it adds sums of another iteration\n", blocks, it, late);
          return 1;
        }
      }
    }
  }
  return 0;
}
