// gbn_problem_fit_rows on the host (fake_cudart.cpp): whichever of its allocations
// fails, the problem keeps the buffers it had and stays usable; a later call that gets
// its memory succeeds, and nothing is lost or freed twice.
#include <cstdio>

#include "fake_cudart.h"
#include "nesta_host.cu"

namespace gbn {
void prof_begin(gbn_ctx*, int, cudaEvent_t*) {}
void prof_end(gbn_ctx*, int, cudaEvent_t) {}
void tuning_for(gbn_ctx*, int, int, int, int, int*, int*) {}
int cuda_status(cudaError_t e, const char*) { return e == cudaSuccess ? GBN_OK : GBN_ERR_CUDA; }
int set_error(int code, const std::string&) { return code; }
void motion_free(gbn_problem*) {}
const float2* ctx_twiddles(gbn_ctx*, int) { return nullptr; }
int nesta_run_mc(gbn_ctx*, gbn_problem*, const gbn_nesta_params*, float2*) { return GBN_OK; }
const SizeKernels* find_size(int L) {
  static SizeKernels k{};
  k.L = L;
  k.pair_cols = pair_split_ok(L) ? pair_cols(L) : 0;
  k.rows_per_cta = 1;
  return &k;
}
}  // namespace gbn

#define CHECK(c)                                        \
  do {                                                  \
    if (!(c)) {                                         \
      std::printf("line %d: %s\n", __LINE__, #c);       \
      return 1;                                         \
    }                                                   \
  } while (0)

int main() {
  using namespace gbn;
  for (int H : {64, 280}) {                     // with and without a column-pair form
    for (int kept : {1, 40, 64 * 4}) {
      gbn_ctx ctx{};
      gbn_problem P{};
      P.ctx = &ctx;
      P.W = 32;
      P.H = H;
      P.F = 4;
      P.C = 3;
      CHECK(problem_alloc(&P) == GBN_OK);
      P.rowoff[P.F] = kept;                     // what the row analysis finds
      int failures = 0;
      for (int k = 1;; ++k) {
        float2* const T = P.T;
        float4* const Tt = P.Tt;
        const size_t rows = P.T_rows, trows = P.Tt_rows, blocks = fake::live_blocks();
        fake::fail_in(k);
        int got = -1;
        const int rc = problem_fit_rows(&P, 0, &got);
        fake::fail_in(0);
        if (rc == GBN_OK) break;                // fewer than k allocations: all of them had their turn
        ++failures;
        CHECK(rc == GBN_ERR_NOMEM);
        CHECK(P.T == T && P.T_rows == rows && fake::live(P.T));
        CHECK(P.Tt == Tt && P.Tt_rows == trows && (!P.Tt || fake::live(P.Tt)));
        CHECK(fake::live_blocks() == blocks);
      }
      CHECK(failures >= 1 || kept == P.F * H);    // every row kept: nothing to resize
      CHECK(P.T_rows == size_t(kept) && fake::live(P.T) && (!P.Tt || fake::live(P.Tt)));
      int got = -1;
      P.rowoff[P.F] = 2 * kept <= P.F * H ? 2 * kept : kept;
      CHECK(problem_fit_rows(&P, 3, &got) == GBN_OK && got == P.rowoff[P.F]);
      CHECK(P.T_rows == std::min<size_t>(size_t(P.F) * H, size_t(got) + 3));
      problem_free(&P);
      CHECK(fake::live_blocks() == 0 && fake::bad_frees == 0);
    }
  }
  return 0;
}
