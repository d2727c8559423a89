// The memory of the column-pair row-local iteration on the host (fake_cudart.cpp): a
// problem without it takes what it took before that iteration existed; the first run
// that wants it allocates it; a run that cannot have it runs the three-pass iteration,
// and a later one that can, the row-local one.
#include <cstdio>

#include "fake_cudart.h"
#include "nesta_host.cu"

static int n_iter = 0, n_fwd = 0;

namespace gbn {
void prof_begin(gbn_ctx*, int, cudaEvent_t*) {}
void prof_end(gbn_ctx*, int, cudaEvent_t) {}
void tuning_for(gbn_ctx*, int, int, int, int, int* a, int* b) { *a = *b = 1; }
int cuda_status(cudaError_t e, const char*) { return e == cudaSuccess ? GBN_OK : GBN_ERR_CUDA; }
int set_error(int code, const std::string&) { return code; }
void motion_free(gbn_problem*) {}
const float2* ctx_twiddles(gbn_ctx*, int) { return nullptr; }
int nesta_run_mc(gbn_ctx*, gbn_problem*, const gbn_nesta_params*, float2*) { return GBN_OK; }
const SizeKernels* find_size(int L) {
  static SizeKernels t[65];
  SizeKernels& k = t[L / 8];
  k.L = L;
  k.pair_cols = pair_split_ok(L) ? pair_cols(L) : 0;
  k.rows_per_cta = 1;
  k.rows_occupancy = [](bool) { return 1; };
  k.fwd_cols = [](const FusedArgs*, const BatchMap&, int, int, dim3, cudaStream_t) { ++n_fwd; };
  k.rows = [](const FusedArgs*, const BatchMap&, int, bool, int, cudaStream_t) {};
  k.inv_cols = [](const FusedArgs*, const BatchMap&, int, bool, dim3, cudaStream_t) {};
  k.iter_cols = [](const FusedArgs*, const BatchMap&, int, bool, dim3, cudaStream_t) { ++n_iter; };
  k.iter_finish = [](const FusedArgs*, const BatchMap&, int, dim3, cudaStream_t) {};
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
  gbn_ctx ctx{};
  ctx.nsm = 152;
  gbn_problem P{};
  P.ctx = &ctx;
  P.W = 48;
  P.H = 64;
  P.F = 4;
  P.C = 8;
  const size_t image = size_t(P.W) * P.H * P.F * sizeof(float2), k = image * P.C, maps = k / P.F;
  CHECK(problem_alloc(&P) == GBN_OK);
  CHECK(fake::live_bytes() < k + 4 * image + 64 * 1024);  // k-space rows, x and w twice, tables

  gbn_nesta_params prm{};
  prm.maxIntIter = 1;
  prm.maxIter = 3;
  float2* const x = static_cast<float2*>(std::malloc(image));
  auto run = [&]() {
    n_iter = n_fwd = 0;
    return nesta_run(&ctx, &P, &prm, x, nullptr);
  };
  ctx.row_local = 0;
  CHECK(run() == GBN_OK && n_fwd == 3 && n_iter == 0);     // the run's own small buffers
  const size_t small = fake::live_bytes();
  CHECK(run() == GBN_OK && fake::live_bytes() == small);
  P.st->partial_rows = 5;                                  // pixel masks
  ctx.row_local = 1;
  CHECK(run() == GBN_OK && n_fwd == 3 && n_iter == 0 && fake::live_bytes() == small);
  P.st->partial_rows = 0;                                  // row masks, but no memory
  fake::fail_in(1);
  CHECK(run() == GBN_OK && n_fwd == 3 && n_iter == 0 && fake::live_bytes() == small);
  fake::fail_in(0);
  CHECK(!P.St && !P.Tt && !P.xt && !P.xk2 && !P.wacc2 && P.Tt_rows == 0);
  CHECK(run() == GBN_OK && n_fwd == 0 && n_iter == 3);
  const size_t all = fake::live_bytes();
  CHECK(all > small && all <= small + maps + 3 * image + k / 2 + 4096);  // 32 of 64 rows at this length
  CHECK(run() == GBN_OK && n_iter == 3 && fake::live_bytes() == all);
  CHECK(P.Tt_rows == size_t(P.F) * 32);

  // a fitted row buffer: the tiles go, and come back fitted
  P.rowoff[P.F] = 10;
  int kept = 0;
  CHECK(problem_fit_rows(&P, 0, &kept) == GBN_OK && kept == 10);
  CHECK(!P.St && !P.xk2 && fake::live_bytes() < small);
  CHECK(run() == GBN_OK && n_iter == 3 && P.Tt_rows == 10);
  problem_free(&P);

  // the motion-compensated form first, which does without the third buffers
  gbn_problem Q{};
  Q.ctx = &ctx;
  Q.W = 48;
  Q.H = 64;
  Q.F = 4;
  Q.C = 8;
  CHECK(problem_alloc(&Q) == GBN_OK);
  bool fresh = false;
  CHECK(problem_tiles(&Q, false, &fresh) == GBN_OK && fresh && Q.St && Q.Tt && Q.xt && !Q.xk2 && !Q.wacc2);
  CHECK(problem_tiles(&Q, false, &fresh) == GBN_OK && !fresh);
  fake::fail_in(1);
  CHECK(problem_tiles(&Q, true, &fresh) == GBN_ERR_NOMEM && Q.St && !Q.xk2);
  fake::fail_in(0);
  float4* const St = Q.St;
  CHECK(problem_tiles(&Q, true, &fresh) == GBN_OK && fresh && Q.xk2 && Q.wacc2 && Q.St == St);
  problem_free(&Q);
  CHECK(fake::live_blocks() == 0 && fake::bad_frees == 0);
  std::free(x);
  return 0;
}
