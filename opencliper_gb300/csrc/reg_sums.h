// Where k_reg_solve (registration.cu) keeps an iteration's partial sums of Dif^2.
//
// In phase 2 of iteration `it` every CTA adds up the sums of it - 1 and then
// stores its own blocks' sums of it, with no barrier in between: a CTA that is
// late reads while others already store.  Two sets in turn keep the two apart,
// and a set is stored again only two phases of barriers later.
#pragma once

#include <cstddef>

#ifdef __CUDACC__
#define GBN_HD __host__ __device__
#else
#define GBN_HD
#endif

namespace gbn {

// floats that `blocks` blocks' sums take
constexpr size_t reg_dif_floats(size_t blocks) { return 2 * blocks; }
// the first of iteration `it`'s
GBN_HD constexpr size_t reg_dif_at(int it, int blocks) { return size_t(it & 1) * size_t(blocks); }

}  // namespace gbn
