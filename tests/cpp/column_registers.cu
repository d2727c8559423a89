// Instantiations whose registers tests/test_column_registers.py reads.
#include "inst.cuh"

namespace gbn {
#define ADJ(L)                                                                                                       \
  template __global__ void k_adj_cols<L, false>(const float2*, const float2* __restrict__, float2* __restrict__, int, \
                                                int, float, const float2* __restrict__);
#define INV(L)                                                                                              \
  template __global__ void k_inv_cols<L, false>(const FusedArgs* __restrict__, const __grid_constant__ BatchMap, int); \
  template __global__ void k_inv_cols<L, true>(const FusedArgs* __restrict__, const __grid_constant__ BatchMap, int);
INV(168)
INV(288)
INV(360)
INV(392)
ADJ(384)
ADJ(504)
ADJ(512)
}  // namespace gbn
