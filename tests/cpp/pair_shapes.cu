// Host-side check of the column-pair iteration's per-length shapes (rowpair.cuh): for
// every length that runs it one line "H PA PB NP bytes min_ctas tmem_cols rcap" on stdout.
// Built with nvcc and run on the host only (no kernel is launched).
#include <cstdio>

#include "rowpair.cuh"

using namespace gbn;

template <int H>
void line() {
  if constexpr (fft_size_ok(H) && iter_pair_ok(H)) {
    using P = PairShape<H>;
    std::printf("%d %d %d %d %d %d %d %d\n", H, P::PA, P::PB, P::NP, P::BYTES, iter_pair_min_blocks(H),
                P::ACC_TM ? int(P::TCOLS) : 0, P::RCAP);
  }
}

int main() {
  sfor<1, 65>([](auto i) { line<8 * decltype(i)::value>(); });
  return 0;
}
