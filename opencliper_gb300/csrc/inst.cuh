// Host launchers for the templated kernels of one transform length.
#pragma once

#include "nesta_kernels.cuh"
#include "pdl.cuh"
#include "registry.h"
#include "rowlocal.cuh"
#include "rowpair.cuh"

namespace gbn {

template <int L>
struct Launchers {
  static void fwd_cols(const FusedArgs* tab, const BatchMap& bm, int it, int cpb, dim3 grid, cudaStream_t s) {
    static OptedIn ok;
    allow_smem(k_fwd_cols<L>, FwdColsSmem<L>::BYTES, ok);
    launch_chain(it == 0, k_fwd_cols<L>, grid, kColNT, FwdColsSmem<L>::BYTES, s, tab, bm, it, cpb);
  }
  // resident CTAs per SM of the row kernel (queried once)
  static int rows_occupancy(bool resid) {
    static int occ1 = 0, occ0 = 0;
    int& o = resid ? occ1 : occ0;
    if (o == 0) {
      static OptedIn ok1, ok0;
      int nb = 0;
      if (resid) {
        allow_smem(k_rows<L, true>, RowsSmem<L, true>::BYTES, ok1);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_rows<L, true>, kRowNT, RowsSmem<L, true>::BYTES);
      } else {
        allow_smem(k_rows<L, false>, RowsSmem<L, false>::BYTES, ok0);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_rows<L, false>, kRowNT, RowsSmem<L, false>::BYTES);
      }
      o = nb > 0 ? nb : 1;
    }
    return o;
  }
  static void rows(const FusedArgs* tab, const BatchMap& bm, int it, bool resid, int grid, cudaStream_t s) {
    static OptedIn ok1, ok0;
    if (resid) {
      allow_smem(k_rows<L, true>, RowsSmem<L, true>::BYTES, ok1);
      launch_pdl(k_rows<L, true>, dim3(grid), kRowNT, RowsSmem<L, true>::BYTES, s, tab, bm, it);
    } else {
      allow_smem(k_rows<L, false>, RowsSmem<L, false>::BYTES, ok0);
      launch_chain(true, k_rows<L, false>, dim3(grid), kRowNT, RowsSmem<L, false>::BYTES, s, tab, bm, it);
    }
  }
  template <bool UPDATE, bool PREF>
  static void inv_cols_of(const FusedArgs* tab, const BatchMap& bm, int it, dim3 grid, cudaStream_t s) {
    static OptedIn ok;
    allow_smem(k_inv_cols<L, UPDATE, PREF>, InvColsSmem<L>::BYTES, ok);
    launch_pdl(k_inv_cols<L, UPDATE, PREF>, grid, kColNT, InvColsSmem<L>::BYTES, s, tab, bm, it);
  }
  static void inv_cols(const FusedArgs* tab, const BatchMap& bm, int it, bool update, dim3 grid, cudaStream_t s) {
    constexpr bool pref = inv_prefetch(L), other = pref != inv_two_forms<L>();
    const bool plain = inv_two_forms<L>() && inv_fewer_waves((long long)grid.x * grid.y * grid.z, device_sms());
    if (update)
      plain ? inv_cols_of<true, other>(tab, bm, it, grid, s) : inv_cols_of<true, pref>(tab, bm, it, grid, s);
    else
      plain ? inv_cols_of<false, other>(tab, bm, it, grid, s) : inv_cols_of<false, pref>(tab, bm, it, grid, s);
  }
  static void iter_cols(const FusedArgs* tab, const BatchMap& bm, int it, bool motion, dim3 grid, cudaStream_t s) {
    if constexpr (iter_pair_ok(L)) {
      using P = PairShape<L>;
      static OptedIn ok0, ok1;
      const int ncg = int(grid.x) * kWB / P::COLS, frames = int(grid.z);
      if (motion) {
        allow_smem(k_iter_pair<L, true>, P::BYTES, ok1);
        launch_pdl(k_iter_pair<L, true>, dim3(ncg, frames), kPairNT, P::BYTES, s, tab, bm, it, 0);
      } else {
        allow_smem(k_iter_pair<L, false>, P::BYTES, ok0);
        launch_chain(it == 0, k_iter_pair<L, false>, dim3(ncg, frames + cdiv(bm.n, ncg)), kPairNT, P::BYTES, s, tab, bm,
                     it, 0);
      }
    } else if constexpr (iter_cols_ok(L)) {
      static OptedIn ok0, ok1;
      if (motion) {
        allow_smem(k_iter_cols<L, true>, IterColsSmem<L>::BYTES, ok1);
        launch_pdl(k_iter_cols<L, true>, grid, IterColsSmem<L>::NT, IterColsSmem<L>::BYTES, s, tab, bm, it);
      } else {
        allow_smem(k_iter_cols<L, false>, IterColsSmem<L>::BYTES, ok0);
        launch_chain(it == 0, k_iter_cols<L, false>, grid, IterColsSmem<L>::NT, IterColsSmem<L>::BYTES, s, tab, bm, it);
      }
    }
  }
  static void iter_finish(const FusedArgs* tab, const BatchMap& bm, int it, dim3 grid, cudaStream_t s) {
    if constexpr (iter_pair_ok(L)) {
      using P = PairShape<L>;
      static OptedIn ok;
      allow_smem(k_iter_pair<L, false>, P::BYTES, ok);
      const int ncg = int(grid.x) * kWB / P::COLS;
      launch_pdl(k_iter_pair<L, false>, dim3(ncg, cdiv(bm.n, ncg)), kPairNT, P::BYTES, s, tab, bm, it, int(grid.z));
    }
  }
  static void fft_rows(const float2* in, float2* out, int nrows, int inv, float scale, const float2* tw,
                       const uint8_t* mask, int C, int H, int grid, bool first, cudaStream_t s) {
    launch_chain(first, mask ? k_fft_rows_dense<L, true> : k_fft_rows_dense<L, false>, dim3(grid), kRowNT, 0, s, in, out,
                 nrows, inv, scale, tw, mask, C, H);
  }
  static void fft_cols(const float2* in, float2* out, int W, int nimg, int inv, float scale, const float2* tw, int nsm,
                       cudaStream_t s) {
    constexpr bool two = cols_dense_two_forms(L);
    const bool few = two && cols_dense_few((long long)(W / kWB) * nimg, nsm);
    launch_pdl(few ? k_fft_cols_dense<L, two> : k_fft_cols_dense<L, false>, dim3(W / kWB, nimg), kColNT, 0, s, in, out,
               W, inv, scale, tw);
  }
  static void enc_cols(const float2* x, const float2* S, float2* out, int W, int C, int F, const float2* tw,
                       cudaStream_t s) {
    k_enc_cols<L><<<dim3(W / kWB, cdiv(C, kEncCoils), F), kColNT, 0, s>>>(x, S, out, W, C, tw);
  }
  template <bool RSS>
  static void adj_cols_of(const float2* T, const float2* S, float2* x, int W, int C, int F, float scale,
                          const float2* tw, int cs, cudaStream_t s) {
    static OptedIn ok;
    constexpr int bytes = AdjColsShape<L, RSS>::BYTES;
    allow_smem(k_adj_cols<L, RSS>, bytes, ok);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(W / kWB, cs, F);
    cfg.blockDim = dim3(AdjColsShape<L, RSS>::NT);
    cfg.dynamicSmemBytes = bytes;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = unsigned(cs);
    at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, k_adj_cols<L, RSS>, T, S, x, W, C, scale, tw);
  }
  static void adj_cols(const float2* T, const float2* S, float2* x, int W, int C, int F, float scale,
                       const float2* tw, int cs, cudaStream_t s) {
    if (S)
      adj_cols_of<false>(T, S, x, W, C, F, scale, tw, cs, s);
    else
      adj_cols_of<true>(T, S, x, W, C, F, scale, tw, cs, s);
  }
  static SizeKernels entry() {
    static_assert(fft_size_ok(L), "unsupported transform length");
    return SizeKernels{L, &fwd_cols, &rows, &inv_cols, &fft_rows, &fft_cols, &enc_cols, &adj_cols,
                       iter_cols_ok(L) ? &iter_cols : nullptr, &iter_finish, iter_pair_ok(L) ? pair_cols(L) : 0,
                       {AdjColsShape<L, false>::MINB, AdjColsShape<L, true>::MINB}, RowCfg<L>::RPC, &rows_occupancy};
  }
};

}  // namespace gbn

// Defines gbn::register_sizes_<TAG>(SizeKernels* out) returning the count.
#define GBN_SIZE_TU(TAG, ...)                                              \
  namespace gbn {                                                          \
  int register_sizes_##TAG(SizeKernels* out) {                             \
    const SizeKernels e[] = {__VA_ARGS__};                                 \
    const int n = int(sizeof(e) / sizeof(e[0]));                           \
    for (int i = 0; i < n; ++i) out[i] = e[i];                             \
    return n;                                                              \
  }                                                                        \
  }
#define GBN_L(L) gbn::Launchers<L>::entry()
