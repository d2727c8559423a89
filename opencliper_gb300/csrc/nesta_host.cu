// tTV-NESTA solver: launch sequence of NestaUp::launch
// (src/processes/nesta/NestaUp.cpp:442-910) on one CUDA stream with all scalar
// bookkeeping kept on the device, plus the non-templated kernels (kept-row
// analysis, initial maxima, power-method norm estimate, scalar setup).
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <string>

#include "ctx.h"
#include "nesta_kernels.cuh"
#include "rowlocal.cuh"
#include "solver.h"

namespace gbn {

constexpr int kNeIters = 100;  // myNormest maxiter (NestaUp.cpp:294)
constexpr int kNeNT = 256;

// ---------------------------------------------------------------------------
// drand48 jump-ahead (host and device)
// ---------------------------------------------------------------------------
constexpr uint64_t kMask48 = (1ULL << 48) - 1;
constexpr uint64_t kRandA = 0x5DEECE66DULL, kRandC = 0xBULL;

__host__ __device__ inline Lcg48 lcg_compose(Lcg48 first, Lcg48 second) {
  // x -> second(first(x)) = sa*(fa*x + fc) + sc
  return Lcg48{(second.a * first.a) & kMask48, (second.a * first.c + second.c) & kMask48};
}
__host__ __device__ inline Lcg48 lcg_jump_k(uint64_t k) {
  Lcg48 r{1, 0}, b{kRandA, kRandC};
  while (k) {
    if (k & 1) r = lcg_compose(r, b);
    b = lcg_compose(b, b);
    k >>= 1;
  }
  return r;
}
Lcg48 lcg48_jump(uint64_t k) { return lcg_jump_k(k); }
uint64_t lcg48_apply(const Lcg48& j, uint64_t x) { return (j.a * x + j.c) & kMask48; }

// ---------------------------------------------------------------------------
// Kept k-space rows: a row (f, h) is carried by the solver when its mask row
// has any sampled pixel or any coil holds a nonzero datum there.  Rows that are
// neither contribute exactly zero to E^H(Ex - y) and to ||Ex - y||^2.
// flags: 0 not kept, 1 kept with sampled pixels, 2 kept for its data only;
// full: every pixel of the mask row sampled.  grid = (H, F)
// ---------------------------------------------------------------------------
// One CTA per row; the rows without samples are read whole (their data decide),
// a coil per warp and step, so that a CTA keeps 8 x 4 loads of 512 bytes in
// flight: bound by memory (256 x 256 x 20 x 12, R = 8, 110 MB: 32 -> 19 us
// against a coil at a time with a CTA barrier after each).
constexpr int kFlagNT = 256;
__global__ void __launch_bounds__(kFlagNT) k_rowflags(const float2* __restrict__ y, const uint8_t* __restrict__ mask,
                                                      int W, int H, int F, int C, int* __restrict__ flags,
                                                      int* __restrict__ full) {
  const int h = blockIdx.x, f = blockIdx.y, t = threadIdx.x, lane = t & 31;
  const uint8_t* m = mask + (size_t(f) * H + h) * W;
  int any = 0, all = 1;
  for (int w = t; w < W; w += kFlagNT) {
    const int nz = m[w] != 0;
    any |= nz;
    all &= nz;
  }
  any = __syncthreads_or(any);
  all = __syncthreads_and(all);
  const int sampled = any;
  if (!any) {
    const int WQ = W / 2;
    const size_t coil = size_t(H) * WQ;
    const float4* row = reinterpret_cast<const float4*>(y) + (size_t(f) * C * H + h) * WQ;
    int nz = 0;
    for (int c = t >> 5; c < C; c += kFlagNT / 32) {
      const float4* yr = row + c * coil;
      for (int q = lane; q < WQ; q += 4 * 32) {
        float4 v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = (q + 32 * u < WQ) ? yr[q + 32 * u] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < 4; ++u) nz |= (v[u].x != 0.f) | (v[u].y != 0.f) | (v[u].z != 0.f) | (v[u].w != 0.f);
      }
    }
    any = __syncthreads_or(nz);
  }
  if (t == 0) {
    flags[f * H + h] = sampled ? 1 : (any ? 2 : 0);
    full[f * H + h] = all;
  }
}

constexpr int kStatusRowsOverflow = 6;  // NestaDevState::status: kept rows beyond the row buffer were dropped

// One CTA of 512 threads per frame (H <= 512): prefix numbering of the frame's
// kept rows, after those of the frames before it (which every CTA counts for
// itself: at most 64 x 512 flags); rows beyond the row buffer's capacity `cap`
// are dropped (rowmap -1) and reported in *status; *partial counts what keeps a
// problem off the row-local iteration: kept rows whose mask row is sampled in
// part, and frames with more kept rows than that iteration stages
// (iter_cols_rcap).  ptab (column pairs, rowpair.cuh; PA <= 32, PB <= 16): the
// kept rows of every second-pass item k1 (rows k1 + PA*k2) and their staged
// slots in (k1, k2) order.  ctl: the control block of a group of this one
// instance.  (One CTA for all frames took 28 us at 20 frames, 41 at 30.)
struct RowScan {
  const int* flags;
  const int* full;
  int H, F, C, cap;
  int *rowmap, *rowoff, *rows_h, *rows_f, *row_full, *status, *partial;
  uint4* ptab;
  int* rowslot;
  int PA, PB;
  ClassCtl* ctl;
  int rpc;
};
__device__ void group_init_one(ClassCtl* ctl, int items, int rpc) {
  ctl->step_base[0] = 0;
  ctl->nitems[0] = items;
  ctl->step_base[1] = (items + rpc - 1) / rpc;
  ctl->row_next = 0;
  ctl->ticket = 0;
}
__global__ void __launch_bounds__(512) k_rowscan(RowScan a) {
  __shared__ int wsum[16], wbase[16], srow[512];
  __shared__ unsigned char sfull[512];
  const int f = blockIdx.x, t = threadIdx.x, lane = t & 31, wid = t >> 5, H = a.H;
  int before = 0;
  for (int i = t; i < f * H; i += 512) before += a.flags[i] != 0;
  const int fl = (t < H) ? a.flags[f * H + t] : 0, fu = (t < H) ? a.full[f * H + t] : 0;
  before = __reduce_add_sync(0xffffffffu, before);
  const unsigned bal = __ballot_sync(0xffffffffu, fl);
  const int pre = __popc(bal & ((1u << lane) - 1u));
  if (lane == 0) {
    wsum[wid] = __popc(bal);
    wbase[wid] = before;
  }
  const int npart = __syncthreads_count(t < H && fl == 1 && !fu);
  int woff = 0, tot = 0, base = 0;
  for (int i = 0; i < 16; ++i) {
    if (i < wid) woff += wsum[i];
    tot += wsum[i];
    base += wbase[i];
  }
  base = min(base, a.cap);
  const int room = a.cap - base, j = (fl && woff + pre < room) ? woff + pre : -1;
  if (t < H) {
    a.rowmap[f * H + t] = j;
    if (j >= 0) {
      a.rows_h[base + j] = t;
      a.rows_f[base + j] = f;
      a.row_full[base + j] = fu;
    }
  }
  srow[t] = j;
  sfull[t] = fu != 0;
  if (t == 0) {
    a.rowoff[f] = base;
    const int mine = npart + (tot > iter_cols_rcap(H));
    if (mine) atomicAdd(a.partial, mine);
    if (tot > room) atomicExch(a.status, kStatusRowsOverflow);
    if (f == a.F - 1) {
      const int g = base + min(tot, room);
      a.rowoff[a.F] = g;
      if (a.ctl) group_init_one(a.ctl, g * a.C, a.rpc);
    }
  }
  if (a.ctl && f == a.F - 1 && t < kMaxBatch) a.ctl->done[t] = 0;
  __syncthreads();
  if (a.ptab && wid == 0) {
    unsigned mk = 0, ms = 0;
    int n = 0;
    if (lane < a.PA) {
      for (int k2 = 0; k2 < a.PB; ++k2) {
        const int h = lane + a.PA * k2;
        if (srow[h] >= 0) {
          mk |= 1u << k2;
          ms |= unsigned(sfull[h]) << k2;
        }
      }
      n = __popc(mk);
    }
    int end = n;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += v;
    }
    if (lane < a.PA) {
      int q = end - n;
      a.ptab[f * a.PA + lane] = make_uint4(mk, ms, unsigned(q), 0u);
      for (int k2 = 0; k2 < a.PB; ++k2) {
        const int jj = srow[lane + a.PA * k2];
        if (jj >= 0) a.rowslot[base + jj] = q++;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Instance tables of a launch group.  k_store_args writes one entry from its
// by-value parameter (no host buffer has to outlive the call); k_group_init
// numbers the row-pass steps of every instance from its kept-row count and
// clears the group's counters.
// ---------------------------------------------------------------------------
__global__ void k_store_args(FusedArgs* __restrict__ dst, FusedArgs v) { *dst = v; }
__global__ void k_set_u64(unsigned long long* dst, unsigned long long v) { *dst = v; }

__global__ void k_group_init(const FusedArgs* __restrict__ tab, int n, int rpc, ClassCtl* __restrict__ ctl) {
  if (threadIdx.x == 0) {
    int base = 0;
    for (int i = 0; i < n; ++i) {
      const FusedArgs& a = tab[i];
      const int items = a.rowoff[a.F] * a.C;
      ctl->step_base[i] = base;
      ctl->nitems[i] = items;
      base += (items + rpc - 1) / rpc;
    }
    ctl->step_base[n] = base;
    ctl->row_next = 0;
    ctl->ticket = 0;
  }
  for (int i = threadIdx.x; i < kMaxBatch; i += blockDim.x) ctl->done[i] = 0;
}

// ---------------------------------------------------------------------------
// State initialisation from the launch parameters, and the instance's table
// entry if given (one thread).
// ---------------------------------------------------------------------------
__global__ void k_state_init(NestaDevState* st, gbn_nesta_params p, FusedArgs* dst, FusedArgs args) {
  NestaDevState s;
  memset(&s, 0, sizeof(s));
  s.lambda_i = p.lambda_i;
  s.mu_f = p.mu_f;
  s.La = p.La;
  s.tolVar_in = p.tolVar;
  s.maxIntIter = int(p.maxIntIter);
  s.maxIter = int(p.maxIter);
  s.stoptest = int(p.stoptest);
  s.miniter = int(p.miniter);
  s.last_iter = -1;
  *st = s;
  if (dst) *dst = args;
}

// ---------------------------------------------------------------------------
// max|x0| and max|U x0| (NestaUp.cpp:521-568: ComplexAbs + host loop).  Values
// are non-negative, so float order equals unsigned order of their bits.
// ---------------------------------------------------------------------------
// xu: the image the sparsity operator is applied to (x itself, or M x with
// motion compensation)
__global__ void __launch_bounds__(256) k_maxima(const float2* __restrict__ x, const float2* __restrict__ xu, int N,
                                                int F, NestaDevState* st) {
  __shared__ float s1[8], s2[8];
  float m1 = 0.f, m2 = 0.f;
  const int f = blockIdx.y;
  const float2* xf = x + size_t(f) * N;
  const float2* uf = xu + size_t(f) * N;
  const float2* um = xu + size_t((f + F - 1) % F) * N;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) {
    const float2 a = xf[p];
    const float2 d = csub(uf[p], um[p]);
    m1 = fmaxf(m1, sqrtf(a.x * a.x + a.y * a.y));
    m2 = fmaxf(m2, sqrtf(d.x * d.x + d.y * d.y));
  }
  m1 = warp_max(m1);
  m2 = warp_max(m2);
  if ((threadIdx.x & 31) == 0) {
    s1[threadIdx.x >> 5] = m1;
    s2[threadIdx.x >> 5] = m2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int i = 1; i < 8; ++i) {
      m1 = fmaxf(m1, s1[i]);
      m2 = fmaxf(m2, s2[i]);
    }
    atomicMax(&st->maxX_bits, __float_as_uint(m1));
    atomicMax(&st->maxUX_bits, __float_as_uint(m2));
  }
}

// ---------------------------------------------------------------------------
// Power method for ||U|| (myNormest, NestaUp.cpp:291-439).
//
// The start vector is all ones, so U x = 0 exactly and the reference always
// restarts from r = (drand48(), 0) drawn in [frame][row][col] order
// (NestaUp.cpp:369-385).  From there e_1 = ||r|| and, for m >= 1,
// e_{m+1} = ||D b_m|| / ||b_m|| with b_1 = D^T r and b_{m+1} = D^T D b_m
// (the reference's per-iteration normalisations and the sign of its adjoint
// kernel cancel in these ratios).  D acts along frames only, so every pixel's
// frame vector evolves independently: one thread per pixel advances it in
// registers (scaled by 1/4 per step, exact in binary floating point, to stay
// in range) and per-step sums of ||b_m||^2 and ||D b_m||^2 are reduced per
// block.  Steps run in chunks; the last CTA of each chunk replays the
// reference's stopping rule on the sums available so far (normest_check) and,
// once it has stopped, later chunks return immediately; the last chunk ends
// with the derived constants (derive_constants).
// part layout: [block][step - m_begin (+1 for the first chunk)][2]; in the
// first chunk slot 0 holds ||r||^2.
// ---------------------------------------------------------------------------
constexpr int kNeChunks = 3;
constexpr int kNeBounds[kNeChunks + 1] = {1, 17, 49, kNeIters};
constexpr int kNeMaxSlots = 52;  // largest chunk (51 steps) + ||r||^2 slot

// one CTA of kNeNT threads: reduce the chunk's per-block sums (two threads per
// sum, blocks in order) and continue the reference's convergence loop
// (NestaUp.cpp:325-431).  tot holds 2 * kNeSums doubles.
constexpr int kNeSums = 128;
static_assert(2 * kNeMaxSlots <= kNeSums && 2 * kNeSums == kNeNT, "two threads per sum");
__device__ void normest_check(const double* __restrict__ part, int nblk, int m_begin, int m_end, int N, int F,
                              NestaDevState* st, double* tot) {
  const int slot0 = (m_begin == 1) ? 1 : 0;
  const int nsum = (slot0 + m_end - m_begin) * 2;
  const int i = threadIdx.x % kNeSums, half = threadIdx.x / kNeSums;
  double s = 0.0;
  if (i < nsum) {
    constexpr int U = 8;
    for (int b0 = half; b0 < nblk; b0 += 2 * U) {
      double v[U];
#pragma unroll
      for (int u = 0; u < U; ++u)
        v[u] = (b0 + 2 * u < nblk) ? __ldcg(part + size_t(b0 + 2 * u) * kNeMaxSlots * 2 + i) : 0.0;
#pragma unroll
      for (int u = 0; u < U; ++u) s += v[u];
    }
  }
  tot[threadIdx.x] = s;
  __syncthreads();
  if (half == 0) tot[i] += tot[i + kNeSums];
  __syncthreads();
  if (threadIdx.x == 0) {
    const float tol = 1e-3f;
    float e, e0;
    int cnt;
    if (m_begin == 1) {
      e = sqrtf(float(unsigned(N) * unsigned(F)));  // ||ones||
      e0 = 0.f;
      cnt = 0;
    } else {
      e = st->ne_e;
      e0 = st->ne_e0;
      cnt = st->ne_cnt;
    }
    bool stopped = false;
    for (;;) {
      if (!(fabsf(e - e0) > tol * e && cnt < kNeIters)) {
        stopped = true;
        break;
      }
      if (cnt > 0 && cnt >= m_end) break;  // needs steps of a later chunk
      const float en = (cnt == 0) ? float(sqrt(tot[0]))
                                  : float(sqrt(tot[2 * (slot0 + cnt - m_begin) + 1] / tot[2 * (slot0 + cnt - m_begin)]));
      e0 = e;
      e = en;
      ++cnt;
    }
    st->ne_e = e;
    st->ne_e0 = e0;
    st->ne_cnt = cnt;
    if (stopped) {
      st->normU = e;
      st->normest_iters = cnt;
      st->ne_done = 1;
    }
  }
}

// ---------------------------------------------------------------------------
// Derived constants (NestaUp.cpp:570-583), by the first warp of a CTA: gamma and
// gammat, each a pow in double, on a lane of its own (and none with one outer
// loop, where both are the bases themselves).
// ---------------------------------------------------------------------------
__device__ void derive_constants(NestaDevState* st) {
  NestaDevState& s = *st;
  const int lane = threadIdx.x;
  const float maxX = __uint_as_float(s.maxX_bits), maxUX = __uint_as_float(s.maxUX_bits);
  const float lambda = s.lambda_i * maxX, muf = s.mu_f * maxX;
  float mu0 = float(0.9 * double(maxUX));
  const float muL = lambda / s.La;
  if (muL > mu0) mu0 = muL;
  double g = (lane == 0) ? double(muf / mu0) : double(s.tolVar_in) / 0.1;
  if (s.maxIntIter != 1 && lane < 2) g = pow(g, 1.0 / double(unsigned(s.maxIntIter)));
  const float gamma = float(g), gammat = __shfl_sync(0xffffffffu, float(g), 1);
  if (lane == 0) {
    s.maxX = maxX;
    s.maxUX = maxUX;
    s.lambda = lambda;
    s.muf = muf;
    s.mu0 = mu0;
    s.gamma = gamma;
    s.mu = mu0;
    s.gammat = gammat;
    s.tolVar = 0.1f;
  }
}
__global__ void k_setup(NestaDevState* st) { derive_constants(st); }

template <int FMAX>
__global__ void __launch_bounds__(kNeNT) k_normest_chunk(int N, int F, RandStart rs,
                                                         unsigned long long jumpN_a, unsigned long long jumpN_c,
                                                         int m_begin, int m_end, float* __restrict__ bstore,
                                                         double* __restrict__ part, NestaDevState* st) {
  __shared__ float sw[kNeNT / 32][kNeMaxSlots][2];
  __shared__ double tot[2 * kNeSums];
  __shared__ bool s_last;
  if (st->ne_done) {
    if (m_end == kNeIters && blockIdx.x == 0 && threadIdx.x < 32) derive_constants(st);
    return;
  }
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  const int p = blockIdx.x * kNeNT + t;
  const bool act = p < N;
  const int slot0 = (m_begin == 1) ? 1 : 0;
  float b[FMAX], d[FMAX];
  if (m_begin == 1) {
    const unsigned long long x0 = rs.p ? ((rs.ja * *rs.p + rs.jc) & kMask48) : rs.x0;
    // element (f, p) is draw number f*N + p + 1 after the state x0
    const Lcg48 jp = lcg_jump_k(uint64_t(act ? p : 0) + 1);
    uint64_t X = (jp.a * x0 + jp.c) & kMask48;
#pragma unroll
    for (int f = 0; f < FMAX; ++f) {
      if (f < F && act) {
        d[f] = __double2float_rn(double(X) * 0x1p-48);
        X = (jumpN_a * X + jumpN_c) & kMask48;
      } else {
        d[f] = 0.f;
      }
    }
    float s0 = 0.f;
#pragma unroll
    for (int f = 0; f < FMAX; ++f) s0 = fmaf(d[f], d[f], s0);
    // b_1 = D^T r: (D^T v)_f = v_f - v_{f+1 mod F}
#pragma unroll
    for (int f = 0; f < FMAX; ++f) {
      const float nx = (f + 1 < FMAX && f + 1 < F) ? d[(f + 1) % FMAX] : d[0];
      b[f] = (f < F) ? d[f] - nx : 0.f;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s0 += __shfl_down_sync(0xffffffffu, s0, o);
    if (lane == 0) {
      sw[wid][0][0] = s0;
      sw[wid][0][1] = 0.f;
    }
  } else {
#pragma unroll
    for (int f = 0; f < FMAX; ++f) b[f] = (f < F && act) ? bstore[size_t(f) * N + p] : 0.f;
  }
  for (int m = m_begin; m < m_end; ++m) {
    float last = b[0];
#pragma unroll
    for (int f = 1; f < FMAX; ++f)
      if (f == F - 1) last = b[f];
    float sb = 0.f, sd = 0.f;
#pragma unroll
    for (int f = 0; f < FMAX; ++f) {
      const float pv = (f == 0) ? last : b[(f + FMAX - 1) % FMAX];
      d[f] = (f < F) ? b[f] - pv : 0.f;
      sb = fmaf(b[f], b[f], sb);
      sd = fmaf(d[f], d[f], sd);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sb += __shfl_down_sync(0xffffffffu, sb, o);
      sd += __shfl_down_sync(0xffffffffu, sd, o);
    }
    if (lane == 0) {
      sw[wid][slot0 + m - m_begin][0] = sb;
      sw[wid][slot0 + m - m_begin][1] = sd;
    }
#pragma unroll
    for (int f = 0; f < FMAX; ++f) {
      const float nx = (f + 1 < FMAX && f + 1 < F) ? d[(f + 1) % FMAX] : d[0];
      b[f] = (f < F) ? (d[f] - nx) * 0.25f : 0.f;
    }
  }
  if (m_end < kNeIters && act) {
#pragma unroll
    for (int f = 0; f < FMAX; ++f)
      if (f < F) bstore[size_t(f) * N + p] = b[f];
  }
  __syncthreads();
  const int nslots = slot0 + m_end - m_begin;
  for (int i = t; i < nslots * 2; i += kNeNT) {
    double s = 0.0;
    for (int w = 0; w < kNeNT / 32; ++w) s += double(sw[w][i >> 1][i & 1]);
    part[size_t(blockIdx.x) * kNeMaxSlots * 2 + i] = s;
  }
  // the chunk's last CTA replays the stopping rule
  __threadfence();
  __syncthreads();
  if (t == 0) {
    s_last = atomicAdd(&st->ne_arrived, 1u) == gridDim.x - 1;
    if (s_last) st->ne_arrived = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  normest_check(part, gridDim.x, m_begin, m_end, N, F, st, tot);
  if (m_end == kNeIters) {
    __syncthreads();
    if (t < 32) derive_constants(st);
  }
}

__device__ void outer_begin_state(NestaDevState* st, int nl, float* fmean) {
  NestaDevState& s = *st;
  s.outer_active = 1;
  s.nl = nl;
  s.mu = s.mu * s.gamma;
  s.tolVar = s.tolVar * s.gammat;
  s.Ak = 0.0f;
  float Lmu = s.normU / s.mu;
  if (s.miniter > 0) fmean[s.miniter - 1] = float(LONG_MAX);
  Lmu = s.lambda * Lmu + s.La;
  s.Lmu = Lmu;
  s.Lmu1 = 1.0f / Lmu;
  s.qpDone = 0;
  s.fixup = 0;
  s.last_iter = s.maxIter - 1;
}

// Start of an outer (continuation) loop (NestaUp.cpp:604-648):
// mu and tolVar updates, Lmu, w = 0, x_k = x_ref.
__global__ void k_outer_begin(NestaDevState* st, int nl, float* fmean, const float2* __restrict__ xref,
                              float2* __restrict__ xk0, float2* __restrict__ wacc, size_t n) {
  if (nl > st->maxIntIter) {
    // this instance has run all its outer loops (a batch runs the largest count)
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->outer_active = 0;
      st->last_iter = -1;
    }
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) outer_begin_state(st, nl, fmean);
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) {
    xk0[i] = xref[i];
    wacc[i] = make_float2(0.f, 0.f);
  }
}

// ---------------------------------------------------------------------------
// Tiles of the column-pair row-local iteration (rowpair.cuh).  A tile holds the
// columns [cg*2NP, (cg+1)*2NP) as [row][pair], each pair of adjacent columns
// planar: (re0, re1, im0, im1).
// ---------------------------------------------------------------------------
__device__ __forceinline__ float4 planar_pair(const float2* src) {
  const float2 u = src[0], v = src[1];  // the caller's images are 8-byte aligned
  return make_float4(u.x, v.x, u.y, v.y);
}

// Start of an outer loop: x_ref into tiles and the scalar state as k_outer_begin
// leaves it; before the first loop (St given) also S and the kept rows'
// IDFT_W(y), which T holds since x0 = E^H y.  A warp per row of W/2 pairs.  The
// data tiles are skipped when the rows do not suit the row-local iteration: they
// may then exceed Tt (the run or replay reports it).
__global__ void __launch_bounds__(256) k_outer_begin_pair(const FusedArgs* __restrict__ tab, int nl,
                                                          const float2* __restrict__ xref, float4* __restrict__ xt,
                                                          float4* __restrict__ St, float4* __restrict__ Tt,
                                                          const int* __restrict__ rowslot, int NP) {
  const FusedArgs& a = *tab;
  NestaDevState* st = a.st;
  if (nl > st->maxIntIter) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      st->outer_active = 0;
      st->last_iter = -1;
    }
    return;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) outer_begin_state(st, nl, a.fmean);
  const int W = a.W, H = a.H, F = a.F, C = a.C, WQ = W / 2, NCG = WQ / NP, lane = threadIdx.x & 31;
  const int nX = F * H, nS = St && !st->partial_rows ? C * H : 0;
  const long long rows = nX + nS + (nS ? (long long)a.rowoff[F] * C : 0);
  for (long long r = (long long)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (long long)gridDim.x * 8) {
    const float2* src;
    float4* dst;
    size_t step;  // from one column group to the next
    if (r < nX + nS) {
      const int k = int(r < nX ? r : r - nX), img = k / H, row = k % H;  // img: frame, or coil
      src = (r < nX ? xref : a.S) + size_t(k) * W;
      step = size_t(H) * NP;
      dst = (r < nX ? xt : St) + size_t(img) * NCG * step + row * NP;
    } else {
      const long long k = r - nX - nS;
      const int g = int(k / C), c = int(k % C), f = a.rows_f[g];
      const size_t nr = a.rowoff[f + 1] - a.rowoff[f];
      src = a.T + size_t(k) * W;
      step = size_t(C) * nr * NP;
      dst = Tt + size_t(a.rowoff[f]) * C * WQ + (size_t(c) * nr + rowslot[g]) * NP;
    }
    for (int q = lane; q < WQ; q += 32) dst[(q / NP) * step + q % NP] = planar_pair(src + 2 * q);
  }
}

// End of an outer loop from tiles: x_ref = x_k (nothing ran: x_ref stays)
__global__ void __launch_bounds__(256) k_outer_end_pair(const NestaDevState* st, const float4* __restrict__ xk0,
                                                        const float4* __restrict__ xk1, const float4* __restrict__ xk2,
                                                        float2* __restrict__ xref, int W, int H, int rows, int NP) {
  if (!st->outer_active || st->last_iter < 0) return;
  const int k3 = (st->last_iter + 1) % 3;
  const float4* src = k3 == 0 ? xk0 : k3 == 1 ? xk1 : xk2;
  const int WQ = W / 2, lane = threadIdx.x & 31, step = H * NP;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8) {  // a warp per row
    const float4* from = src + size_t(r / H) * (WQ / NP) * step + (r % H) * NP;
    float2* to = xref + size_t(r) * W;
    for (int q = lane; q < WQ; q += 32) {
      const float4 v = from[size_t(q / NP) * step + q % NP];
      to[2 * q] = make_float2(v.x, v.z);
      to[2 * q + 1] = make_float2(v.y, v.w);
    }
  }
}

// End of an outer loop: x_ref = x_k (NestaUp.cpp:889).
__global__ void k_outer_end(const NestaDevState* st, const float2* __restrict__ xk0, const float2* __restrict__ xk1,
                            float2* __restrict__ xref, size_t n) {
  if (!st->outer_active) return;
  const float2* src = ((st->last_iter + 1) & 1) ? xk1 : xk0;
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x)
    xref[i] = src[i];
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
namespace {

template <typename T>
int grow(T*& p, int& cap, int need) {
  if (need <= cap) return GBN_OK;
  if (p) cudaFree(p);
  p = nullptr;
  cap = 0;
  if (cudaMalloc(&p, sizeof(T) * size_t(need)) != cudaSuccess) {
    cudaGetLastError();
    return set_error(GBN_ERR_NOMEM, "workspace allocation failed");
  }
  cap = need;
  return GBN_OK;
}

int normest_fmax(int F) {
  for (int m : {8, 16, 24, 32, 40, 48, 64})
    if (F <= m) return m;
  return 0;
}

void launch_normest_chunk(int fmax, int nblk, cudaStream_t s, int N, int F, const RandStart& x0, const Lcg48& jN, int mb,
                          int me, float* bstore, double* part, NestaDevState* st) {
#define GBN_NE_CASE(M)                                                                                  \
  case M:                                                                                               \
    k_normest_chunk<M><<<nblk, kNeNT, 0, s>>>(N, F, x0, jN.a, jN.c, mb, me, bstore, part, st); \
    break;
  switch (fmax) {
    GBN_NE_CASE(8)
    GBN_NE_CASE(16)
    GBN_NE_CASE(24)
    GBN_NE_CASE(32)
    GBN_NE_CASE(40)
    GBN_NE_CASE(48)
    default:
      k_normest_chunk<64><<<nblk, kNeNT, 0, s>>>(N, F, x0, jN.a, jN.c, mb, me, bstore, part, st);
  }
#undef GBN_NE_CASE
}

}  // namespace

// a buffer to carve from a block
struct Part {
  void** p;
  size_t bytes;
};
// One allocation for all of them, each 256-byte aligned; on failure none is touched.
static cudaError_t alloc_parts(void** block, const Part* parts, int n) {
  auto up = [](size_t v) { return (v + 255) / 256 * 256; };
  size_t total = 0;
  for (int k = 0; k < n; ++k) total += up(parts[k].bytes);
  const cudaError_t e = cudaMalloc(block, total);
  if (e != cudaSuccess) {
    *block = nullptr;
    return e;
  }
  unsigned char* b = static_cast<unsigned char*>(*block);
  for (int k = 0; k < n; b += up(parts[k].bytes), ++k) *parts[k].p = b;
  return cudaSuccess;
}

int problem_alloc(gbn_problem* P) {
  const size_t FH = size_t(P->F) * P->H;
  const size_t X = size_t(P->F) * P->H * P->W;
  const size_t K = X * P->C;
  const SizeKernels* kh = find_size(P->H);
  const bool pair = kh && kh->pair_cols;
  // one allocation for everything but the row buffer, which fit_rows resizes, and the
  // tiles, which only row-local runs of column-pair lengths need
  const Part parts[] = {{(void**)&P->flags, FH * sizeof(int)},
                        {(void**)&P->full_fh, FH * sizeof(int)},
                        {(void**)&P->rowmap, FH * sizeof(int)},
                        {(void**)&P->rowoff, (P->F + 1) * sizeof(int)},
                        {(void**)&P->rows_h, FH * sizeof(int)},
                        {(void**)&P->rows_f, FH * sizeof(int)},
                        {(void**)&P->row_full, FH * sizeof(int)},
                        {(void**)&P->xk0, X * sizeof(float2)},
                        {(void**)&P->xk1, X * sizeof(float2)},
                        {(void**)&P->wacc, X * sizeof(float2)},
                        {(void**)&P->wacc1, X * sizeof(float2)},
                        {(void**)&P->st, sizeof(NestaDevState)},
                        {(void**)&P->d_args, sizeof(FusedArgs)},
                        {(void**)&P->ctl, sizeof(ClassCtl)},
                        // column pairs only
                        {(void**)&P->ptab, size_t(P->F) * pair_a(P->H) * sizeof(uint4)},
                        {(void**)&P->rowslot, FH * sizeof(int)}};
  const int nparts = int(sizeof(parts) / sizeof(parts[0])) - (pair ? 0 : 2);
  cudaError_t e = alloc_parts(&P->block, parts, nparts);
  if (e == cudaSuccess) {
    e = cudaMalloc(&P->T, K * sizeof(float2));
    P->T_rows = FH;
  }
  if (e != cudaSuccess) {
    cudaGetLastError();
    return set_error(GBN_ERR_NOMEM, std::string("problem workspace allocation failed: ") + cudaGetErrorString(e));
  }
  return GBN_OK;
}

int problem_tiles(gbn_problem* P, bool plain, bool* fresh) {
  const size_t X = size_t(P->F) * P->H * P->W;
  Part parts[5];
  int n = 0;
  size_t trows = P->Tt_rows;
  if (!P->St) {
    trows = std::min<size_t>(P->T_rows, size_t(P->F) * std::min(P->H, iter_cols_rcap(P->H)));
    parts[n++] = {(void**)&P->Tt, std::max<size_t>(trows, 1) * P->C * P->W * sizeof(float2)};
    parts[n++] = {(void**)&P->St, size_t(P->C) * P->H * P->W * sizeof(float2)};
    parts[n++] = {(void**)&P->xt, X * sizeof(float2)};
  }
  if (plain && !P->xk2) {
    parts[n++] = {(void**)&P->xk2, X * sizeof(float2)};
    parts[n++] = {(void**)&P->wacc2, X * sizeof(float2)};
  }
  *fresh = n > 0;
  if (n == 0) return GBN_OK;
  if (alloc_parts(&P->tiles[P->tiles[0] ? 1 : 0], parts, n) != cudaSuccess) {
    cudaGetLastError();
    return GBN_ERR_NOMEM;
  }
  P->Tt_rows = trows;
  return GBN_OK;
}

static void tiles_free(gbn_problem* P) {
  for (void*& b : P->tiles) {
    if (b) cudaFree(b);
    b = nullptr;
  }
  P->St = P->Tt = P->xt = nullptr;
  P->xk2 = P->wacc2 = nullptr;
  P->Tt_rows = 0;
}

void launch_row_analysis(gbn_problem* P, ClassCtl* ctl, cudaStream_t s);

// Shrinks (or grows) the row buffer T to the rows the current y and mask keep
// plus `headroom` (at most every row); returns the kept rows in *kept.
int problem_fit_rows(gbn_problem* P, int headroom, int* kept) {
  if (headroom < 0) return set_error(GBN_ERR_INVALID, "headroom must be >= 0");
  if (P->in_batches > 0)
    return set_error(GBN_ERR_INVALID, "fit rows: the problem belongs to a live batch (destroy it first)");
  cudaStream_t s = P->ctx->stream;
  cudaError_t e = cudaMemsetAsync(&P->st->status, 0, sizeof(int), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(&P->st->partial_rows, 0, sizeof(int), s);
  const size_t saved = P->T_rows;
  P->T_rows = size_t(P->F) * P->H;  // count every kept row
  if (e == cudaSuccess) {
    launch_row_analysis(P, nullptr, s);
    int g = 0;
    if ((e = cudaMemcpyAsync(&g, P->rowoff + P->F, sizeof(int), cudaMemcpyDeviceToHost, s)) == cudaSuccess &&
        (e = cudaStreamSynchronize(s)) == cudaSuccess) {
      const size_t want = std::min<size_t>(size_t(P->F) * P->H, size_t(g) + size_t(headroom));
      // the new buffer before the old one is given back: a failure leaves the problem as it was
      float2* nt = nullptr;
      if (want == saved || (e = cudaMalloc(&nt, std::max<size_t>(want, 1) * P->C * P->W * sizeof(float2))) == cudaSuccess) {
        if (nt) {
          cudaFree(P->T);
          P->T = nt;
          tiles_free(P);  // sized for the rows before; the next run that takes them allocates them
        }
        P->T_rows = want;
        if (kept) *kept = g;
        return GBN_OK;
      }
    }
  }
  P->T_rows = saved;
  cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? set_error(GBN_ERR_NOMEM, "row buffer allocation failed")
                                        : cuda_status(e, "fit rows");
}

void motion_free(gbn_problem* P);

void problem_free(gbn_problem* P) {
  tiles_free(P);
  void* ptrs[] = {P->block,   P->T,    P->fmean,  P->part_tv, P->part_r, P->part_ne,
                  P->ne_b, P->fk, P->colmax, P->smax,    P->fa};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  motion_free(P);
}

// Kept-row analysis for the current contents of y and mask (device only).
void launch_row_analysis(gbn_problem* P, ClassCtl* ctl, cudaStream_t s) {
  k_rowflags<<<dim3(P->H, P->F), kFlagNT, 0, s>>>(P->y, P->mask, P->W, P->H, P->F, P->C, P->flags, P->full_fh);
  RowScan r{};
  r.flags = P->flags;
  r.full = P->full_fh;
  r.H = P->H;
  r.F = P->F;
  r.C = P->C;
  r.cap = int(P->T_rows);
  r.rowmap = P->rowmap;
  r.rowoff = P->rowoff;
  r.rows_h = P->rows_h;
  r.rows_f = P->rows_f;
  r.row_full = P->row_full;
  r.status = &P->st->status;
  r.partial = &P->st->partial_rows;
  if (P->ptab) {
    r.ptab = P->ptab;
    r.rowslot = P->rowslot;
    r.PA = pair_a(P->H);
    r.PB = pair_b(P->H);
  }
  r.ctl = ctl;
  r.rpc = find_size(P->W)->rows_per_cta;
  k_rowscan<<<P->F, 512, 0, s>>>(r);
}

FusedArgs make_args(gbn_problem* P, float2* xref) {
  gbn_ctx* ctx = P->ctx;
  FusedArgs a;
  memset(&a, 0, sizeof(a));
  a.W = P->W;
  a.H = P->H;
  a.F = P->F;
  a.C = P->C;
  a.N = P->W * P->H;
  a.y = P->y;
  a.S = P->S;
  a.mask = P->mask;
  a.rowmap = P->rowmap;
  a.rowoff = P->rowoff;
  a.rows_h = P->rows_h;
  a.rows_f = P->rows_f;
  a.row_full = P->row_full;
  a.T = P->T;
  a.xk0 = P->xk0;
  a.xk1 = P->xk1;
  a.xref = xref;
  a.wacc = P->wacc;
  a.wacc1 = P->wacc1;
  a.st = P->st;
  a.fmean = P->fmean;
  a.part_tv = P->part_tv;
  a.part_r = P->part_r;
  a.twH = ctx_twiddles(ctx, P->H);
  a.twW = ctx_twiddles(ctx, P->W);
  const unsigned N = unsigned(P->W) * unsigned(P->H);
  a.s_fwd = float(1.0 / std::sqrt(double(N)));               // NestaUp.cpp:712: 1/(sqrt(cols*rows*slices))
  a.s_adj = std::sqrt(float(N)) * (1.0f / float(N));        // NestaUp.cpp:749 sqrt(float(N)) times clFFT 1/N
  a.s_row = float(double(P->W) * double(a.s_fwd));
  a.ntv = P->F * (P->W / kWB);
  a.St = P->St;
  a.Tt = P->Tt;
  a.xt = P->xt;
  float2* const px[3] = {P->xk0, P->xk1, P->xk2};
  float2* const pw[3] = {P->wacc, P->wacc1, P->wacc2};
  for (int b = 0; b < 3; ++b) {
    a.px[b] = reinterpret_cast<float4*>(px[b]);
    a.pw[b] = reinterpret_cast<float4*>(pw[b]);
  }
  a.ptab = P->ptab;
  return a;
}

BatchMap single_map(int F, ClassCtl* ctl) {
  BatchMap bm;
  memset(&bm, 0, sizeof(bm));
  bm.n = 1;
  bm.fbase[0] = 0;
  bm.fbase[1] = F;
  bm.ctl = ctl;
  return bm;
}

int validate_problem_dims(int W, int H, int F, int C) {
  if (W <= 0 || H <= 0 || F <= 0 || C <= 0) return set_error(GBN_ERR_INVALID, "dimensions must be positive");
  if (W % 8 != 0) return set_error(GBN_ERR_INVALID, "NDArray dimension 0 (width) is not multiple of 8");
  if (!find_size(W) || !find_size(H))
    return set_error(GBN_ERR_UNSUPPORTED,
                     "FFT lengths must be 7-smooth multiples of 8 in [8, 512] (got W=" + std::to_string(W) +
                         ", H=" + std::to_string(H) + ")");
  return GBN_OK;
}

int run_prepare(gbn_ctx* ctx, gbn_problem* P, const gbn_nesta_params* prm) {
  if (!ctx || !P || !prm) return set_error(GBN_ERR_INVALID, "null argument");
  if (P->F < 2) return set_error(GBN_ERR_INVALID, "temporal TV needs at least 2 frames (F=1 makes ||U|| undefined)");
  if (prm->stoptest == 1 && prm->miniter == 0) return set_error(GBN_ERR_INVALID, "miniter must be >= 1 when stoptest == 1");
  if (!normest_fmax(P->F)) return set_error(GBN_ERR_UNSUPPORTED, "more than 64 frames is not supported");
  const SizeKernels* kh = find_size(P->H);
  const SizeKernels* kw = find_size(P->W);
  if (!kh || !kw) return set_error(GBN_ERR_UNSUPPORTED, "unsupported FFT length");
  const int W = P->W, H = P->H, F = P->F, C = P->C, N = W * H;
  const long long steps_max = ((long long)F * H * C + kw->rows_per_cta - 1) / kw->rows_per_cta;
  const int nblk_ne = (N + kNeNT - 1) / kNeNT;
  int rc;
  if ((rc = grow(P->fmean, P->fmean_cap, std::max<int>(1, int(prm->miniter)))) != GBN_OK) return rc;
  // one (|u|^2, Re<u,d>) pair per (frame, 8-column tile) and coil half (row-local iteration)
  // (two sets for the column pairs, which sum one iteration while the next runs)
  if ((rc = grow(P->part_tv, P->part_tv_cap, (kh->pair_cols ? 8 : 4) * F * (W / kWB))) != GBN_OK) return rc;
  if ((rc = grow(P->part_r, P->part_r_cap, std::max(int(steps_max) * kRowWarps, 4 * F * (W / kWB)))) != GBN_OK)
    return rc;
  if ((rc = grow(P->part_ne, P->part_ne_cap, nblk_ne * kNeMaxSlots * 2)) != GBN_OK) return rc;
  if ((rc = grow(P->ne_b, P->ne_b_cap, N * F)) != GBN_OK) return rc;
  return GBN_OK;
}

int row_grid(gbn_ctx* ctx, const SizeKernels* kw, bool resid, long long steps, int k2_per_sm) {
  const int per_sm = std::max(1, std::min(k2_per_sm, kw->rows_occupancy(resid)));
  return int(std::max<long long>(1, std::min<long long>(steps, (long long)ctx->nsm * per_sm)));
}

int launch_store_args(FusedArgs* dst, const FusedArgs& a, cudaStream_t s) {
  k_store_args<<<1, 1, 0, s>>>(dst, a);
  return 1;
}

int launch_group_init(const FusedArgs* tab, int n, int rows_per_cta, ClassCtl* ctl, cudaStream_t s) {
  k_group_init<<<1, 64, 0, s>>>(tab, n, rows_per_cta, ctl);
  return 1;
}

int launch_set_rand(unsigned long long* dst, unsigned long long v, cudaStream_t s) {
  k_set_u64<<<1, 1, 0, s>>>(dst, v);
  return 1;
}

int launch_pre(gbn_problem* P, const gbn_nesta_params& prm, cudaStream_t s, FusedArgs* tab, const FusedArgs* args,
               ClassCtl* ctl) {
  k_state_init<<<1, 1, 0, s>>>(P->st, prm, tab, args ? *args : FusedArgs{});
  launch_row_analysis(P, ctl, s);
  return 3;
}

namespace {
int elementwise_grid(gbn_ctx* ctx, size_t n) { return int(std::min<size_t>((n + 255) / 256, size_t(ctx->nsm) * 8)); }
}  // namespace

int launch_constants(gbn_ctx* ctx, gbn_problem* P, const float2* xref, const RandStart& rs, cudaStream_t s) {
  const int N = P->W * P->H, F = P->F;
  const int nblk_ne = (N + kNeNT - 1) / kNeNT;
  // maxima, norm estimate, constants (NestaUp.cpp:521-583)
  launch_maxima(ctx, P, xref, xref, s);
  const Lcg48 jN = lcg_jump_k(uint64_t(N));
  for (int ch = 0; ch < kNeChunks; ++ch)
    launch_normest_chunk(normest_fmax(F), nblk_ne, s, N, F, rs, jN, kNeBounds[ch], kNeBounds[ch + 1], P->ne_b,
                         P->part_ne, P->st);
  return 1 + kNeChunks;
}

int launch_maxima(gbn_ctx* ctx, gbn_problem* P, const float2* x0, const float2* xu, cudaStream_t s) {
  const int N = P->W * P->H;
  const dim3 g(std::min((N + 511) / 512, std::max(1, ctx->nsm * 8 / P->F)), P->F);
  k_maxima<<<g, 256, 0, s>>>(x0, xu, N, P->F, P->st);
  return 1;
}

int launch_setup(gbn_problem* P, cudaStream_t s) {
  k_setup<<<1, 32, 0, s>>>(P->st);
  return 1;
}

int launch_outer_begin_pair(gbn_ctx* ctx, gbn_problem* P, int nl, const float2* xref, const FusedArgs* tab,
                            cudaStream_t s) {
  const bool first = nl == 1;
  const long long rows = (long long)P->F * P->H + (first ? (long long)P->C * P->H + (long long)P->Tt_rows * P->C : 0);
  const int grid = int(std::min<long long>((rows + 7) / 8, (long long)ctx->nsm * 8));
  k_outer_begin_pair<<<grid, 256, 0, s>>>(tab, nl, xref, P->xt, first ? P->St : nullptr, P->Tt, P->rowslot,
                                          pair_np(P->H));
  return 1;
}

int launch_outer_end_pair(gbn_ctx* ctx, gbn_problem* P, float2* xref, cudaStream_t s) {
  const int rows = P->F * P->H;
  k_outer_end_pair<<<std::min((rows + 7) / 8, ctx->nsm * 8), 256, 0, s>>>(
      P->st, reinterpret_cast<const float4*>(P->xk0), reinterpret_cast<const float4*>(P->xk1),
      reinterpret_cast<const float4*>(P->xk2), xref, P->W, P->H, rows, pair_np(P->H));
  return 1;
}

int launch_outer_begin(gbn_ctx* ctx, gbn_problem* P, int nl, const float2* xref, cudaStream_t s) {
  const size_t X = size_t(P->W) * P->H * P->F;
  k_outer_begin<<<elementwise_grid(ctx, X), 256, 0, s>>>(P->st, nl, P->fmean, xref, P->xk0, P->wacc, X);
  return 1;
}

int launch_outer_end(gbn_ctx* ctx, gbn_problem* P, float2* xref, cudaStream_t s) {
  const size_t X = size_t(P->W) * P->H * P->F;
  k_outer_end<<<elementwise_grid(ctx, X), 256, 0, s>>>(P->st, P->xk0, P->xk1, xref, X);
  return 1;
}

int read_stats(gbn_problem* P, cudaStream_t s, gbn_nesta_stats* stats) {
  NestaDevState h;
  int G = 0;
  cudaError_t e;
  if ((e = cudaMemcpyAsync(&h, P->st, sizeof(h), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return cuda_status(e, "stats copy");
  if ((e = cudaMemcpyAsync(&G, P->rowoff + P->F, sizeof(int), cudaMemcpyDeviceToHost, s)) != cudaSuccess)
    return cuda_status(e, "stats copy");
  if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_status(e, "nesta run");
  stats->normU = h.normU;
  stats->maxX = h.maxX;
  stats->maxUX = h.maxUX;
  stats->lambda = h.lambda;
  stats->muf = h.muf;
  stats->mu0 = h.mu0;
  stats->mu_final = h.mu;
  stats->tolVar_final = h.tolVar;
  stats->fx_final = h.fx;
  stats->qp_final = h.qp;
  stats->inner_iters = h.iters_total;
  stats->normest_iters = h.normest_iters;
  stats->kept_rows = G;
  stats->status = h.status;
  return GBN_OK;
}

int nesta_run_mc(gbn_ctx* ctx, gbn_problem* P, const gbn_nesta_params* prm, float2* x_out);

// pinned read-back slot and event of the per-run row-structure check (first use)
int partial_flag_ready(gbn_ctx* ctx) {
  if (ctx->host_partial) return GBN_OK;
  cudaError_t e = cudaHostAlloc(&ctx->host_partial, sizeof(int), cudaHostAllocDefault);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ctx->ev_partial, cudaEventDisableTiming);
  return cuda_status(e, "pinned row-structure flag");
}

int nesta_run(gbn_ctx* ctx, gbn_problem* P, const gbn_nesta_params* prm, float2* x_out, gbn_nesta_stats* stats) {
  if (!x_out) return set_error(GBN_ERR_INVALID, "null argument");
  int rc = run_prepare(ctx, P, prm);
  if (rc != GBN_OK) return rc;
  if (P->mc_on) {
    if ((rc = nesta_run_mc(ctx, P, prm, x_out)) != GBN_OK) return rc;
    return stats ? read_stats(P, ctx->stream, stats) : GBN_OK;
  }
  const SizeKernels* kh = find_size(P->H);
  const SizeKernels* kw = find_size(P->W);
  const int W = P->W, H = P->H, F = P->F, C = P->C;
  cudaStream_t s = ctx->stream;
  int cpb, k2;
  tuning_for(ctx, W, H, F, C, &cpb, &k2);
  cpb = std::max(1, std::min(cpb, C));
  const dim3 g1(W / kWB, (C + cpb - 1) / cpb, F);
  const long long steps = ((long long)F * H * C + kw->rows_per_cta - 1) / kw->rows_per_cta;
  const int g2 = row_grid(ctx, kw, true, steps, k2), g2a = row_grid(ctx, kw, false, steps, k2);
  const dim3 g3(W / kWB, 2, F);  // clusters of 2 along y
  const FusedArgs a = make_args(P, x_out);
  const FusedArgs* tab = P->d_args;
  const BatchMap bm = single_map(F, P->ctl);

  // the row-local iteration needs every kept row fully sampled or unsampled:
  // the row analysis's count of partly sampled rows comes back to pinned
  // host memory while the setup below is queued, and is read before the
  // iterations are
  const bool check_rows = ctx->row_local && kh->iter_cols;
  int rc2 = check_rows ? partial_flag_ready(ctx) : GBN_OK;
  if (rc2 != GBN_OK) return rc2;
  cudaError_t ef = cudaSuccess;
  int n_setup = 0;
  GBN_LAUNCH(ctx, GBN_PROF_SETUP, n_setup, {
    n_setup += launch_pre(P, *prm, s, P->d_args, &a, P->ctl);
    if (check_rows) {
      ef = cudaMemcpyAsync(ctx->host_partial, &P->st->partial_rows, sizeof(int), cudaMemcpyDeviceToHost, s);
      if (ef == cudaSuccess) ef = cudaEventRecord(ctx->ev_partial, s);
    }
    // x0 = E^H y (NestaUp.cpp:465-486); T keeps IDFT_W(y) of the kept rows
    kw->rows(tab, bm, 0, false, g2a, s);
    kh->inv_cols(tab, bm, 0, false, g3, s);
    n_setup += 2;
    n_setup += launch_constants(ctx, P, x_out, RandStart{ctx->rand48, nullptr, 1, 0}, s);
    ctx->rand48 = lcg48_apply(lcg_jump_k(uint64_t(W) * uint64_t(H) * uint64_t(F)), ctx->rand48);
  });
  if (ef != cudaSuccess) return cuda_status(ef, "row structure read-back");
  bool row_local = false;
  if (ctx->row_local && kh->iter_cols) {
    if ((ef = cudaEventSynchronize(ctx->ev_partial)) != cudaSuccess) return cuda_status(ef, "row structure read-back");
    row_local = *ctx->host_partial == 0;
  }
  if (row_local && kh->pair_cols) {  // the setup is still running while the tiles are allocated
    bool fresh = false;
    row_local = problem_tiles(P, true, &fresh) == GBN_OK;
    if (row_local && fresh) ctx->launches += launch_store_args(P->d_args, make_args(P, x_out), s);
  }
  // stopping test on: the launches that recompute the last update if the rule
  // stops the loop (row-local iteration only; the column pairs run one iteration
  // ahead of the test)
  const bool pair = row_local && kh->pair_cols;
  const unsigned n_iter_launch = prm->maxIter + ((row_local && prm->stoptest == 1) ? (pair ? 2u : 1u) : 0u);

  for (unsigned nl = 1; nl <= prm->maxIntIter; ++nl) {
    GBN_LAUNCH(ctx, GBN_PROF_OUTER, 1,
               pair ? launch_outer_begin_pair(ctx, P, int(nl), x_out, tab, s)
                    : launch_outer_begin(ctx, P, int(nl), x_out, s));
    if (row_local) {
      for (unsigned it = 0; it < n_iter_launch; ++it)
        GBN_LAUNCH(ctx, GBN_PROF_ITER, 1, kh->iter_cols(tab, bm, int(it), false, g3, s));
      if (pair && prm->stoptest != 1) GBN_LAUNCH(ctx, GBN_PROF_OUTER, 1, kh->iter_finish(tab, bm, int(prm->maxIter), g3, s));
    } else {
      for (unsigned it = 0; it < prm->maxIter; ++it) {
        GBN_LAUNCH(ctx, GBN_PROF_FWD_COLS, 1, kh->fwd_cols(tab, bm, int(it), cpb, g1, s));
        GBN_LAUNCH(ctx, GBN_PROF_ROWS, 1, kw->rows(tab, bm, int(it), true, g2, s));
        GBN_LAUNCH(ctx, GBN_PROF_INV_COLS, 1, kh->inv_cols(tab, bm, int(it), true, g3, s));
      }
    }
    GBN_LAUNCH(ctx, GBN_PROF_OUTER, 1,
               pair ? launch_outer_end_pair(ctx, P, x_out, s) : launch_outer_end(ctx, P, x_out, s));
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e, "nesta launch");
  if (stats) return read_stats(P, s, stats);
  return GBN_OK;
}

}  // namespace gbn
