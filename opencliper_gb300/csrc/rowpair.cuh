// Row-local tTV-NESTA iteration on column pairs (the algorithm of
// rowlocal.cuh: one fused kernel per inner iteration for problems whose kept
// k-space rows are each fully sampled or not sampled at all).
//
// k_iter_pair<H, MOTION>: grid (W / COLS, frames), 128 threads.  A CTA owns
// one frame and COLS = 2*NP adjacent columns, and each of its four warps a
// quarter of the coils (coil c on warp c % 4).  A lane works on two adjacent
// columns at a time in planar pairs (pairdft.cuh), and a warp holds whole
// columns: NP pairs times PB lanes = 32.  So per coil
//   F1  lane (s, w): S_c x_f at rows PB*n1 + s, DFT_PA, twiddles -> exchange
//   F2  item (k1, w): DFT_PB over s (rows k1 + PA*k2), residual on the kept rows,
//   I1  the same item: DFT_PB of the conjugate, twiddles -> the slots it read
//   I2  lane (k1', w): DFT_PA, conj(S_c) accumulation at rows k1' + PB*k2
// the exchange is private to the warp, F2/I1 run in place, and the loop over
// coils has warp barriers only (k_iter_cols: four CTA barriers per coil).  The
// coil accumulators live in the lane's tensor memory (PA > kPairAccReg) or in
// registers; the image tile sits in shared memory for all four warps, and the
// kept rows' IDFT_W(y) is copied one coil ahead.
//
// Every operand is read in tiles that a setup kernel lays out once per solve
// (k_outer_begin_pair; the kept rows' tables are k_rowscan's): planar pairs, [row][pair] of one column group
// contiguous, so that a warp's 16-byte loads are 512 contiguous bytes.  Read in
// the natural order, a tile's rows are 32-byte pieces W apart, and the sixteen
// cache lines a load touches made this kernel no faster than k_iter_cols
// (100.8 against 99.7 us under ncu at 256 x 256 x 20 frames x 12 coils).
//
// After the coil loop the four accumulators are summed in warp order and each
// thread finishes its pixels: tTV gradient, Nesterov update and, where a
// stopping test or the run's statistics will read it, the objective's partial
// sums (without the test only the last iteration's objective is ever read).
// The plain form reduces them in the next launch, in CTAs of their own beside
// that iteration, which therefore runs one ahead of the stopping test: when the
// rule fires at iteration s, launch s + 1 has already run in vain, and launch
// s + 2 recomputes the update of s with the rule's weights from x_s and w_s,
// which the third buffer has kept.  Counting the CTAs with a fence and an atomic
// and reducing in the last one, as k_iter_cols and the motion-compensated form
// do, put 7 us on every iteration (us per iteration with the test, before ->
// now: 64 x 64 x 6 x 4 11.2 -> 6.3, 256 x 256 x 20 x 12 70.5 -> 60.1).
//
// Bound by FP32 issue in the coil loop (about 0.58 of the FMA pipe at 48 coils,
// 12 warps per SM) and by the latency around it (a CTA's first loads, the update's).
// One GB300, us per iteration, R = 8, k_iter_cols -> now: 256 x 256 x 20 frames x
// 12 coils 90 -> 58, 128 x 128 x 10 x 8 19.7 -> 12.2, 64 x 64 x 6 x 4 12.9 -> 3.8;
// 384 x 384 x 30 x 16 460 -> 305.  Tried and not kept: a persistent grid with the next
//   task's operands copied ahead (68.9 against 69.7 at H = 256, 46.9 against 40.5
//   at H = 128, both with the objective every iteration), four CTAs per SM at 128
//   registers (72.7 against 69.7).
#pragma once

#include "pairdft.cuh"
#include "rowlocal.cuh"

namespace gbn {

constexpr int kPairNT = 128;
constexpr int kPairWarps = 4;
// Largest PA whose accumulators stay in registers: past it they and the
// transform spill much at 168 registers (H = 192: 46.6 us with tensor memory, 50.3
// with registers; H = 64, PA = 8: 11.3 and 9.8).  Most lengths still spill 16 to 100
// bytes a thread (256: 72).
constexpr int kPairAccReg = 8;
// S is used by F1 and again, at the same rows of the same lane, by I2.  With
// four pairs per warp (PB = 8) it stays in registers in between; with two the
// transforms leave no room and reading it again is faster (H = 256: 69.7
// against 78.6 us, H = 128 with four pairs: 42.1 against 40.5).
constexpr bool pair_sreg(int H) { return pair_a(H) <= 16 && pair_b(H) == 8; }

constexpr bool iter_pair_ok(int H) { return iter_cols_ok(H) && pair_split_ok(H); }

__device__ __forceinline__ PairC pc_of(const float4& e) {
  return PairC{make_float2(e.x, e.y), make_float2(e.z, e.w)};
}
__device__ __forceinline__ float4 f4_of(const PairC& v) { return make_float4(v.re.x, v.re.y, v.im.x, v.im.y); }
// two adjacent complex values <-> their planar pair
__device__ __forceinline__ float4 planar(const float4& v) { return make_float4(v.x, v.z, v.y, v.w); }

template <int H>
struct PairShape {
  static constexpr int PB = pair_b(H), PA = pair_a(H), NP = pair_np(H), COLS = pair_cols(H);
  static constexpr int KS = 32 + NP;         // exchange stride between k1 groups (16-byte units): F2's 8 lanes of a
                                             // 16-byte phase fall into different banks
  static constexpr int TS = pair_ts(H);
  static constexpr int RCAP = iter_cols_rcap(H);
  static constexpr bool ACC_TM = PA > kPairAccReg;
  static constexpr bool SREG = pair_sreg(H);
  static constexpr int NI2 = cdiv(PA * NP, 32);            // F2/I1 rounds
  static constexpr int NU = cdiv(H * NP, kPairNT);         // update units (two pixels) per thread
  static constexpr uint32_t TCOLS = 4 * PA <= 32 ? 32u : 4 * PA <= 64 ? 64u : 128u;
  // shared memory in 16-byte units
  static constexpr int EX_OFF = 0;                                  // float4 [warps][PA*KS]
  static constexpr int X_OFF = EX_OFF + kPairWarps * PA * KS;       // float4 [H][NP]
  static constexpr int TW_OFF = X_OFF + H * NP;                     // float4 [PB][TS]: (c, c, s, s)
  static constexpr int Y_OFF = TW_OFF + PB * TS;                    // float4 [warps][RCAP][NP]
  static constexpr int F4_END = Y_OFF + kPairWarps * RCAP * NP;
  static constexpr int BYTES = F4_END * 16 + 3 * kPairWarps * 8 + kFmeanCopy * 4;
  static_assert(4 * PA <= 128, "accumulators fit 128 tensor-memory columns");
};

// CTAs per SM the registers are for: 168 a thread, or 255 past PA = 16, where
// the transform alone holds 4*PA (four CTAs at PA <= 8, 128 registers, spill: H =
// 64 13.1 against 9.8 us)
constexpr int iter_pair_min_blocks(int H) { return pair_a(H) <= 16 ? 3 : 2; }

// a load that is issued where it stands
__device__ __forceinline__ int ld_now(const int* p) {
  int v;
  asm volatile("ld.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p));
  return v;
}

// Sums of three doubles over the CTA's 128 threads in a fixed order: *ra and, if
// given, rbc[0] and rbc[1] (all written by warp 0).  FP64 adds are the cost (two
// per cycle and SM): the first two shuffle rounds leave each value to its own
// lanes, 6 adds a lane instead of 15, and one warp adds the four warps' sums of
// all three at once.  sred holds 3 * kPairWarps doubles.
__device__ __forceinline__ void pair_block_sum3(double a, double b, double c, double* sred, double* ra, double* rbc) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const bool hi = lane & 16, mid = lane & 8;
  const double x = __shfl_xor_sync(0xffffffffu, hi ? a : c, 16), y = __shfl_xor_sync(0xffffffffu, b, 16);
  const double p = (hi ? c : a) + x, q = b + y;  // lanes 0-15: a and b, lanes 16-31: c
  const double z = __shfl_xor_sync(0xffffffffu, (hi || mid) ? p : q, 8);
  double r = ((mid && !hi) ? q : p) + z;         // lanes 0-7: a, 8-15: b, 16-31: c
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r += __shfl_xor_sync(0xffffffffu, r, o);
  if (lane % 8 == 0 && lane < 24) sred[(lane / 8) * kPairWarps + wid] = r;
  __syncthreads();
  if (wid == 0) {
    r = lane < 3 * kPairWarps ? sred[lane] : 0.0;
    r += __shfl_xor_sync(0xffffffffu, r, 1);
    r += __shfl_xor_sync(0xffffffffu, r, 2);
    if (lane == 0) *ra = r;
    if (rbc && (lane == kPairWarps || lane == 2 * kPairWarps)) rbc[lane / kPairWarps - 1] = r;
  }
}

template <int H, bool MOTION>
__global__ void __launch_bounds__(kPairNT, iter_pair_min_blocks(H))
    k_iter_pair(const FusedArgs* __restrict__ tab, const __grid_constant__ BatchMap bm, int it, int z0) {
  using L = PairShape<H>;
  constexpr int PA = L::PA, PB = L::PB, NP = L::NP, KS = L::KS, TS = L::TS, RCAP = L::RCAP, NU = L::NU;
  __shared__ uint32_t tslot;
  extern __shared__ float4 smem4[];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  float4* const ex = smem4 + L::EX_OFF + wid * PA * KS;
  float4* const xs = smem4 + L::X_OFF;
  float4* const tw = smem4 + L::TW_OFF;
  float4* const Yw = smem4 + L::Y_OFF + wid * RCAP * NP;
  double* sred = reinterpret_cast<double*>(smem4 + L::F4_END);
  float* fm = reinterpret_cast<float*>(sred + 3 * kPairWarps);

  // the plain form's last rows of CTAs, one CTA per instance, sum the objective of
  // the iteration before and run its scalar step while the others compute this one
  // (z0 = frames: those alone)
  const int frames = bm.fbase[bm.n], ncg = gridDim.x, z = int(blockIdx.y) + z0;
  if (!MOTION && z >= frames) {
    const int inst = (z - frames) * ncg + int(blockIdx.x), k = it - 1;
    if (inst >= bm.n) return;
    const FusedArgs& a = tab[inst];
    NestaDevState* const st = a.st;
    grid_dep_wait();
    grid_dep_release();
    if (k < 0 || st->partial_rows || !st->outer_active || k >= st->maxIter || st->last_iter < k) return;
    const int nblk = a.F * ncg;
    if (st->stoptest == 1 || k == st->maxIter - 1)
      rowlocal_finish<kPairNT>(a, st, bm.ctl, inst, k, 0.5f * (float(k) + 1.0f), a.part_tv + (k & 1) * 2 * nblk, nblk,
                               a.part_r + (k & 1) * nblk, nblk, sred, fm, st->stoptest == 1 ? 0 : k);
    return;
  }
  const int inst = find_inst(bm, z);
  const FusedArgs& a = tab[inst];
  NestaDevState* st = a.st;
  const int f = z - bm.fbase[inst], cg = blockIdx.x;
  const int W = a.W, C = a.C, F = a.F;
  const int rowbase = a.rowoff[f];
  // at most RCAP kept rows (a frame with more is counted in partial_rows, checked below)
  const int nrows = min(a.rowoff[f + 1] - rowbase, RCAP);
  constexpr int TU = H * NP;  // 16-byte units of a tile: [row][pair]

  // S of the warp's first coil: an input of the whole solve, requested first
  const float4* const s_src = a.St + size_t(cg) * TU + lane;
  const size_t s_coil = size_t(ncg) * TU;
  float4 sv[L::SREG ? PA : 1];
  if constexpr (L::SREG) {
    if (wid < C) {
#pragma unroll
      for (int n1 = 0; n1 < PA; ++n1) sv[n1] = __ldg(s_src + size_t(wid) * s_coil + 32 * n1);
    }
  }
  const float4* const y_src = a.Tt + (size_t(rowbase) * C * W) / 2 + size_t(cg) * C * nrows * NP;
  auto issue_Y = [&](int c) {
    const float4* src = y_src + size_t(c) * nrows * NP;
    for (int q = lane; q < nrows * NP; q += 32) cp_async16(Yw + q, src + q);
  };
  if (wid < C) issue_Y(wid);
  for (int d = t; d < PB * TS; d += kPairNT) cp_async16(tw + d, reinterpret_cast<const float4*>(a.twH + 2 * H) + d);
  cp_async_commit();
  // kept rows of this lane's F2 items: bit k2 of x for row k1 + PA*k2 (y: the
  // sampled ones among them), z: the first one's staged slot
  uint4 kept[L::NI2];
#pragma unroll
  for (int r = 0; r < L::NI2; ++r) {
    const int k1 = min((lane + 32 * r) / NP, PA - 1);
    kept[r] = __ldg(a.ptab + f * PA + k1);
  }
  // x_k, w_k and the scalar state come from the previous launch; in the
  // motion-compensated form from three launches back (see k_iter_cols)
  if constexpr (!MOTION) grid_dep_wait();
  grid_dep_release();

  // x_k and w_k in tiles (frame, column group, row, pair), except x_k of the
  // motion-compensated form, which its gathers read in the natural order; the
  // first iteration of an outer loop starts from x_ref with w = 0.  The image
  // tile is requested before the state says how this launch runs
  auto tile = [&](int fr) { return (size_t(fr) * ncg + cg) * TU; };
  auto natural = [&](int u) { return (size_t(f) * a.N + size_t(u / NP) * W + cg * L::COLS) / 2 + u % NP; };
  const size_t off0 = tile(f), offm = tile((f + F - 1) % F), offp = tile((f + 1) % F);
  // (buffers in turn: two, and three in the plain form, which runs one iteration
  // ahead of the stopping test and may have to recompute the one before last)
  constexpr int NB = MOTION ? 2 : 3;
  auto x_of = [&](int k) -> const float4* { return (k == 0 && !MOTION) ? a.xt : a.px[k % NB]; };
  auto issue_x = [&](const float4* src) {
    for (int u = t; u < TU; u += kPairNT) cp_async16(xs + u, MOTION ? src + natural(u) : src + off0 + u);
    cp_async_commit();
  };
  issue_x(x_of(it));

  // Which update this launch computes.  Plain form: the test of iteration it - 1
  // runs beside this launch and may set last_iter = it - 1 meanwhile; what it
  // decides holds from the next launch on, so both values read as "run".
  // (the state's words are requested together: read one by one between the
  // branches they cost a round trip each, 1.5 us on small problems)
  const int last = ld_now(&st->last_iter), partial = ld_now(&st->partial_rows), active = ld_now(&st->outer_active),
            max_it = ld_now(&st->maxIter), fixup = ld_now(&st->fixup), stoptest = ld_now(&st->stoptest);
  bool fix = false;
  int itx = it;
  if (partial) {  // the data changed under a captured row-local solve
    if (t == 0 && cg == 0 && f == 0 && it == 0) st->status = kStatusRowStructure;
    cp_async_wait<0>();
    return;
  }
  const bool runs = MOTION ? it <= last : (active && it < max_it && last >= it - 1);
  if (!runs) {
    cp_async_wait<0>();
    if (!(fixup && (MOTION || active) && it == last + (MOTION ? 1 : 2))) return;
    fix = true;
    itx = last;
    issue_x(x_of(itx));  // each thread over its own copies
  }
  // the objective is read by the stopping test of every iteration, or, without
  // the test, by the statistics of the last one
  const bool want = !fix && (stoptest == 1 || it == max_it - 1);
  const float4* const xr = a.xt;
  const float4* const xk = x_of(itx);
  float4* const xn = a.px[(itx + 1) % NB];
  const float4* const wk = a.pw[itx % NB];
  float4* const wn = a.pw[(itx + 1) % NB];
  const float inv_mu = 1.0f / st->mu;
  // operands of the update: requested before the coil loop where they are few
  // (short columns), else before the other warps are waited for
  constexpr bool EARLY = NU <= 2;
  float4 pm[NU], pp[MOTION ? 1 : NU], pw[NU], pr[NU];
  auto request = [&]() {
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      const int u = t + i * kPairNT;
      if (TU % kPairNT == 0 || u < TU) {
        if constexpr (!MOTION) {
          pm[i] = xk[offm + u];
          pp[i] = xk[offp + u];
        }
        pw[i] = itx == 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : wk[off0 + u];
        pr[i] = xr[off0 + u];
      }
    }
  };
  if constexpr (EARLY) request();
  uint32_t tl = 0;  // this lane's tensor memory
  if constexpr (L::ACC_TM) {
    if (t < 32) {
      tc::tmem_alloc(&tslot, L::TCOLS);
      tc::tmem_relinquish();
    }
    tc::fence_before_sync();
  }
  cp_async_wait<0>();
  if constexpr (MOTION) {
    for (int u = t; u < TU; u += kPairNT) xs[u] = planar(xs[u]);  // this thread's own copies
  }
  __syncthreads();
  PairC acc[L::ACC_TM ? 1 : PA];
  if constexpr (L::ACC_TM) {
    tc::fence_after_sync();
    tl = tslot + (uint32_t(32 * wid) << 16);
    float z[16] = {};
    tmem_pieces<4 * PA>([&](auto oc, auto nc) { tmem_st_n<decltype(nc)::value>(tl + decltype(oc)::value, z); });
    tc::tmem_wait_st();
  } else {
#pragma unroll
    for (int k2 = 0; k2 < PA; ++k2) acc[k2] = PairC{};
  }
  const float s_row = a.s_row;
  float2 racc = make_float2(0.f, 0.f);

  for (int c = wid; c < C; c += kPairWarps) {
    PairC v[PA];
    auto s_at = [&](int n1) {
      if constexpr (L::SREG) return sv[n1];
      else return __ldg(s_src + size_t(c) * s_coil + 32 * n1);
    };
    // F1: S_c x_f, DFT_PA, twiddles
#pragma unroll
    for (int n1 = 0; n1 < PA; ++n1) {
      const float4 s = s_at(n1);
      v[n1] = pc_mul(pc_of(xs[32 * n1 + lane]), make_float2(s.x, s.y), make_float2(s.z, s.w));
    }
    pair_dft<PA>(v);
#pragma unroll
    for (int k1 = 0; k1 < PA; ++k1) {
      if (k1 > 0) {
        const float4 w = tw[(lane / NP) * TS + k1];
        v[k1] = pc_mul(v[k1], make_float2(w.x, w.y), make_float2(w.z, w.w));
      }
      ex[k1 * KS + lane] = f4_of(v[k1]);
    }
    cp_async_wait<0>();
    __syncwarp();  // exchange written, the coil's IDFT_W(y) staged
    // F2, residual, I1
#pragma unroll
    for (int r = 0; r < L::NI2; ++r) {
      const int i = lane + 32 * r;
      if (PA * NP % 32 == 0 || i < PA * NP) {
        const int k1 = i / NP, w = i % NP;
        float4* const slot = ex + k1 * KS + w;
        PairC u[PB];
#pragma unroll
        for (int s = 0; s < PB; ++s) u[s] = pc_of(slot[s * NP]);
        pair_dft<PB>(u);
        const float4* yp = Yw + kept[r].z * NP + w;
#pragma unroll
        for (int k2 = 0; k2 < PB; ++k2) {
          PairC q{};
          if (kept[r].x & (1u << k2)) {
            const PairC y = pc_of(*yp);
            yp += NP;
            const float2 sc = p2((kept[r].y & (1u << k2)) ? s_row : 0.f);  // data only: -y
            q.re = __ffma2_rn(u[k2].re, sc, p2neg(y.re));
            q.im = __ffma2_rn(u[k2].im, sc, p2neg(y.im));
            racc = __ffma2_rn(q.re, q.re, racc);
            racc = __ffma2_rn(q.im, q.im, racc);
          }
          u[k2] = PairC{q.re, p2neg(q.im)};  // the inverse transform runs on the conjugate
        }
        pair_dft<PB>(u);
#pragma unroll
        for (int k1p = 0; k1p < PB; ++k1p) {
          if (k1p > 0) {
            const float4 wv = tw[k1p * TS + k1];
            u[k1p] = pc_mul(u[k1p], make_float2(wv.x, wv.y), make_float2(wv.z, wv.w));
          }
          slot[k1p * NP] = f4_of(u[k1p]);
        }
      }
    }
    __syncwarp();
    if (c + kPairWarps < C) issue_Y(c + kPairWarps);
    cp_async_commit();
    // I2: DFT_PA and conj(S_c) accumulation: conj(v) conj(S) == conj(v S)
#pragma unroll
    for (int s = 0; s < PA; ++s) v[s] = pc_of(ex[s * KS + lane]);
    __syncwarp();  // the exchange is free for the next coil
    pair_dft<PA>(v);
    auto add_term = [&](PairC& d, int k2) {
      const float4 s = s_at(k2);
      const float2 sr = make_float2(s.x, s.y), si = make_float2(s.z, s.w);
      d.re = __ffma2_rn(v[k2].re, sr, __ffma2_rn(p2neg(v[k2].im), si, d.re));
      d.im = __ffma2_rn(p2neg(v[k2].re), si, __ffma2_rn(p2neg(v[k2].im), sr, d.im));
    };
    if constexpr (L::ACC_TM) {
      tc::tmem_wait_st();  // the previous coil's stores
      tmem_pieces<4 * PA>([&](auto oc, auto nc) {
        constexpr int o = decltype(oc)::value, n = decltype(nc)::value;
        float af[n];
        tmem_ld_n<n>(tl + o, af);
#pragma unroll
        for (int e = 0; e < n / 4; ++e) {
          PairC d{make_float2(af[4 * e], af[4 * e + 1]), make_float2(af[4 * e + 2], af[4 * e + 3])};
          add_term(d, o / 4 + e);
          af[4 * e] = d.re.x;
          af[4 * e + 1] = d.re.y;
          af[4 * e + 2] = d.im.x;
          af[4 * e + 3] = d.im.y;
        }
        tmem_st_n<n>(tl + o, af);
      });
    } else {
#pragma unroll
      for (int k2 = 0; k2 < PA; ++k2) add_term(acc[k2], k2);
    }
    if constexpr (L::SREG) {
      if (c + kPairWarps < C) {
#pragma unroll
        for (int n1 = 0; n1 < PA; ++n1) sv[n1] = __ldg(s_src + size_t(c + kPairWarps) * s_coil + 32 * n1);
      }
    }
  }

  // each warp's accumulators to its exchange: unit row*NP + w = k2*32 + lane
  if (wid < C) {
    if constexpr (L::ACC_TM) {
      tc::tmem_wait_st();
      tmem_pieces<4 * PA>([&](auto oc, auto nc) {
        constexpr int o = decltype(oc)::value, n = decltype(nc)::value;
        float af[n];
        tmem_ld_n<n>(tl + o, af);
#pragma unroll
        for (int e = 0; e < n / 4; ++e)
          ex[(o / 4 + e) * 32 + lane] = make_float4(af[4 * e], af[4 * e + 1], af[4 * e + 2], af[4 * e + 3]);
      });
    } else {
#pragma unroll
      for (int k2 = 0; k2 < PA; ++k2)
        ex[k2 * 32 + lane] = f4_of(acc[k2]);
    }
  }
  if constexpr (L::ACC_TM) tc::fence_before_sync();
  if constexpr (!EARLY) request();
  __syncthreads();
  if constexpr (L::ACC_TM) {
    if (t < 32) {
      tc::fence_after_sync();
      tc::tmem_dealloc(tslot, L::TCOLS);
    }
  }
  if constexpr (MOTION) {
    grid_dep_wait();  // M^T(tTVadj u) of x_k
#pragma unroll
    for (int i = 0; i < NU; ++i) {
      const int u = t + i * kPairNT;
      if (TU % kPairNT == 0 || u < TU) pm[i] = planar(reinterpret_cast<const float4*>(a.grad_ext)[natural(u)]);
    }
  }
  const float s_adj = a.s_adj;
  const float lambda = st->lambda, nLmu1 = -st->Lmu1;
  const float apk = fix ? st->apk : 0.5f * (float(itx) + 1.0f);  // nesta_scalar_step's weights for k = itx
  const float tauk = fix ? st->tauk : 2.0f / (float(itx) + 3.0f);
  const float omt = 1.0f - tauk;
  float su2 = 0.f, sud = 0.f;
  const int nw = min(C, kPairWarps);
#pragma unroll
  for (int i = 0; i < NU; ++i) {
    const int u = t + i * kPairNT;
    if (TU % kPairNT == 0 || u < TU) {
      float4 ac = smem4[L::EX_OFF + u];
      for (int g = 1; g < nw; ++g) {
        const float4 o = smem4[L::EX_OFF + g * PA * KS + u];
        ac.x += o.x;
        ac.y += o.y;
        ac.z += o.z;
        ac.w += o.w;
      }
      const float4 xv = xs[u];
      // one pixel: x_k, its neighbours in time (or M^T(tTVadj u)), w_k, x_ref and A^H r
      auto update = [&](float2 xa, float2 xm, float2 xp, float2 wo, float2 xr, float2 accv, float2* wnv, float2* xnv) {
        float2 adj;
        if constexpr (MOTION) {
          adj = xm;
        } else {
          const float2 d = csub(xa, xm);
          const float2 u0 = tv_normalize(d, inv_mu);
          const float2 u1 = tv_normalize(csub(xp, xa), inv_mu);
          su2 = fmaf(u0.x, u0.x, fmaf(u0.y, u0.y, su2));
          sud = fmaf(u0.x, d.x, fmaf(u0.y, d.y, sud));
          adj = csub(u1, u0);
        }
        const float2 ares = cscale(accv, s_adj);
        const float2 df = make_float2(__fadd_rn(__fmul_rn(-adj.x, lambda), ares.x),
                                      __fadd_rn(__fmul_rn(-adj.y, lambda), ares.y));
        const float2 yk = make_float2(fmaf(nLmu1, df.x, xa.x), fmaf(nLmu1, df.y, xa.y));
        *wnv = make_float2(fmaf(apk, df.x, wo.x), fmaf(apk, df.y, wo.y));
        const float2 zk = make_float2(fmaf(nLmu1, wnv->x, xr.x), fmaf(nLmu1, wnv->y, xr.y));
        *xnv = make_float2(fmaf(omt, yk.x, tauk * zk.x), fmaf(omt, yk.y, tauk * zk.y));
      };
      const float4 vm = pm[i], vp = MOTION ? vm : pp[MOTION ? 0 : i], vw = pw[i], vr = pr[i];
      float2 w1, w2, x1, x2;
      auto px0 = [](const float4& q) { return make_float2(q.x, q.z); };
      auto px1 = [](const float4& q) { return make_float2(q.y, q.w); };
      update(px0(xv), px0(vm), px0(vp), px0(vw), px0(vr), px0(ac), &w1, &x1);
      update(px1(xv), px1(vm), px1(vp), px1(vw), px1(vr), px1(ac), &w2, &x2);
      wn[off0 + u] = make_float4(w1.x, w2.x, w1.y, w2.y);
      if constexpr (MOTION)
        xn[natural(u)] = make_float4(x1.x, x1.y, x2.x, x2.y);
      else
        xn[off0 + u] = make_float4(x1.x, x2.x, x1.y, x2.y);
    }
  }
  if (!want) return;

  // fixed-slot partial sums: ||rho||^2 and the tTV terms of this CTA's tile
  const int nblk = F * ncg, blk = f * ncg + cg, set = MOTION ? 0 : it & 1;
  pair_block_sum3(double(racc.x) + double(racc.y), double(su2), double(sud), sred, a.part_r + set * nblk + blk,
                  MOTION ? nullptr : a.part_tv + 2 * (set * nblk + blk));
  if constexpr (MOTION) {  // the tTV sums come from k_mc_tv, in the same buffer
    if (rowlocal_last_cta(bm.ctl, inst, unsigned(nblk)))
      rowlocal_finish<kPairNT>(a, st, bm.ctl, inst, it, apk, a.part_tv, a.ntv, a.part_r, nblk, sred, fm,
                               st->stoptest == 1 ? 0 : it);
  }
}

}  // namespace gbn
