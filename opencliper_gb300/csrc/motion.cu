// Motion-compensated tTV-NESTA (NestaUp with argsMC != nullptr): the sparsity
// operator becomes U x = tTV(M x) and U^T u = M^T tTVadj(u) (NestaUp.cpp:
// 201-278), where M warps every frame by bilinear interpolation on a deformed
// mesh (MotionCompensation.cpp:57-78; optimizer.cl:832-877) and M^T scatters
// back with the same weights (AdjointMotionCompensation.cpp:59-86;
// optimizer.cl:880-937; initialize.cl:55-80).  The solve starts from the image
// already in the output buffer (the reference skips x0 = E^H y with argsMC,
// NestaUp.cpp:483-486).
//
// Both operators run as gathers over tables built from the meshes at the
// start of each run:
//  * inv[p]: the rectangle entry whose warped value lands on pixel p (the
//    last one in the reference's work-item order when several do), or -1:
//    (M x)[f][p] = inv[p] < 0 ? x[f][p] : bilinear x[f] at that entry;
//  * per target pixel and frame, the list of (entry, corner) pairs the
//    scatter would add there, in the reference's work-item order, with each
//    entry's source pixel and fractional position: (M^T g)[q] = (q in the
//    rectangle ? 0 : g[q]) + sum of (g[src] * fa) * fb, each product and sum
//    rounded as the kernel's.
// So M^T is deterministic and equals an in-order scatter bit for bit, where
// the reference's atomic scatter depends on the order of its atomics.
//
// Per inner iteration: k_mc_tv (M x_k for three frames on the fly, D, the
// Huber normalisation, g = D^T u and the objective's partial sums),
// k_mc_adjoint (M^T g), and the data term with the update.  For row masks the
// last is the one-kernel row-local iteration (rowlocal.cuh), launched after
// the two on one stream; its update waits for M^T g, its tTV gradient.
// Otherwise it is the fused forward column and row passes as in the plain form
// (the forward pass skips its tTV sums) and the adjoint column pass, which
// takes M^T g; k_mc_tv and k_mc_adjoint then run on a side stream beside the
// forward column pass, events ordering them after the previous iterate and
// before the row and adjoint column passes.  The power method ||U|| cannot use the plain form's per-pixel
// recurrence (M mixes pixels), so it runs myNormest's loop step for step, in one
// cooperative launch (k_normest).
//
// Bounds: the reference reads the image at the interpolation corners without
// checks; here a corner or target outside the image skips that pixel and sets
// the instance's status (kStatusMotionRange) instead of reading out of range.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ctx.h"
#include "inst.cuh"
#include "solver.h"

namespace gbn {

int op_ttv(gbn_ctx* ctx, int dir, const float2* in, float2* out, int W, int H, int F);
Lcg48 lcg48_jump(uint64_t k);
uint64_t lcg48_apply(const Lcg48& j, uint64_t x);

// tables of one problem's meshes (rebuilt at every run)
struct McTables {
  int* inv = nullptr;         // [H*W] rectangle entry landing on each pixel (then its R1*W + R2), -1 none
  int* cnt = nullptr;         // [F*H*W] contributions per target (then fill cursors)
  int* off = nullptr;         // [F*H*W + 1] exclusive prefix sums of cnt
  int* bsum = nullptr;        // [scan blocks] block totals of the prefix sum
  int* key = nullptr;         // [4 * l1 * l2 * F] contributions grouped by target, sorted by entry * 4 + corner,
                              // then rewritten to (the entry's pixel R1*W + R2) * 4 + corner
  int* srcmap = nullptr;      // [H*W + 1] pixel each entry (by its R1*W + R2) reads in the adjoint; whether any differs
  int* at = nullptr;          // [F][H*W] upper-left pixel of each entry's square in frame f, -1 outside the image
  float2* wts = nullptr;      // [F][H*W] (Whh, Wvv): each entry's fractional position in frame f
  double* tvpart = nullptr;   // [F * pixel blocks][2] partial sums of the fused tTV kernel
  size_t x = 0, entries = 0;  // F*H*W and l1*l2 the buffers were sized for
  int nbp = 0, nscan = 0;
  size_t hw = 0;              // H*W
};

namespace {

constexpr int kStatusMotionRange = 5;  // NestaDevState::status: a mesh point outside the image
constexpr int kNT = 256;
constexpr int kScanItems = 4;                   // prefix-sum elements per thread
constexpr int kScanBlock = kNT * kScanItems;    // per block
constexpr int kTvFrames = 2;                    // frames per thread of the fused tTV kernel

// rows r1b .. r1b+l1-1 and columns r2b .. r2b+l2-1 of the rectangle
// (Interpolator.cpp:63-87: margins H/40 and W/40 in integer division)
struct McRect {
  int r1b, l1, r2b, l2;
};

McRect mc_rect(int W, int H, const int* bb) {
  const int m0 = H / 40, m1 = W / 40;
  McRect r;
  r.l1 = (bb[3] + m0 + 1) - (bb[1] - m0 - 1) + 1;
  r.l2 = (bb[2] + m1 + 1) - (bb[0] - m1 - 1) + 1;
  r.r1b = (bb[1] - m0 - 1) - 1;
  r.r2b = (bb[0] - m1 - 1) - 1;
  return r;
}

bool rect_ok(const McRect& r, int W, int H) {
  return r.l1 > 0 && r.l2 > 0 && r.r1b >= 0 && r.r2b >= 0 && r.r1b + r.l1 <= H && r.r2b + r.l2 <= W;
}

// deformed position of rectangle entry e = i + l1*j in frame k (0-based) and
// its upper-left interpolation corner
struct McPoint {
  float nh, nv;
  int ph, pv;
  bool ok;
};

__device__ __forceinline__ int entry_offset(McRect r, int e, int W) {
  const int i = e % r.l1, j = e / r.l1;
  return (r.r2b + j) + (r.r1b + i) * W;  // (row R1, column R2) in a [H][W] plane
}

__device__ __forceinline__ McPoint mc_point(const float* __restrict__ xn, int xo, int k, int W, int H, int F) {
  const size_t HW = size_t(H) * W;
  const float* const xk = xn + k * HW;
  McPoint q;
  q.nh = __ldg(xk + xo) - 1.f;
  q.nv = __ldg(xk + HW * F + xo) - 1.f;
  q.ph = int(floorf(q.nh));
  q.pv = int(floorf(q.nv));
  q.ok = q.ph >= 0 && q.ph + 1 < W && q.pv >= 0 && q.pv + 1 < H;
  return q;
}

// frame f of a periodic series, -F <= f < 2 F
__device__ __forceinline__ int wrap_frame(int f, int F) { return f < 0 ? f + F : f >= F ? f - F : f; }

// M's points, one per entry (at its pixel R1*W + R2) and frame: the square's upper-left
// pixel (-1: a corner is outside the image, the value stays) and the fractional
// position (Whh, Wvv).  1 - Whh is the interpolator's float(ph + 1) - nh bit for bit:
// past the first pixel both are exact, in it they are the same subtraction.
struct McPoints {
  const int *inv, *at;
  const float2* wts;
};

// the interpolator's value (optimizer.cl:832-877) of frame xf at q, in the
// kernel's order with separately rounded products and sums: with motion
// compensation the power method starts from this interpolation's rounding
// residue on a constant image, so ||U|| depends on these exact bits.  SCALED: of s x,
// each product rounded.  x is read through a plain pointer: other CTAs of the launch
// may have written it before a barrier.
struct McAt {
  int at;
  float2 w;
};
__device__ __forceinline__ McAt mc_at(const McPoints& m, int xo, size_t plane) {
  return {__ldg(m.at + plane + xo), __ldg(m.wts + plane + xo)};
}
// p*u + q*v with both products and the sum rounded separately (the packed products and
// sums fuse)
__device__ __forceinline__ float2 lin2(float p, float2 u, float q, float2 v) {
  return make_float2(__fadd_rn(__fmul_rn(p, u.x), __fmul_rn(q, v.x)), __fadd_rn(__fmul_rn(p, u.y), __fmul_rn(q, v.y)));
}
template <bool SCALED>
__device__ __forceinline__ float2 mc_value(const float2* xf, const McAt& q, int p, int W, float s) {
  auto get = [&](const float2* v) { return SCALED ? make_float2(__fmul_rn(v->x, s), __fmul_rn(v->y, s)) : *v; };
  if (q.at < 0) return get(xf + p);
  const float2 *const c0 = xf + q.at, *const c1 = c0 + W;
  const float2 i1 = get(c0), i2 = get(c0 + 1), i3 = get(c1), i4 = get(c1 + 1);
  const float a = __fsub_rn(1.f, q.w.x), c = __fsub_rn(1.f, q.w.y);
  return lin2(c, lin2(a, i1, q.w.x, i2), q.w.y, lin2(a, i3, q.w.x, i4));
}

// ---- table construction ------------------------------------------------------
// inv[ver*W + hor] = the largest entry e whose original-mesh point is (hor, ver);
// srcmap[R1*W + R2] = that pixel (-1 outside the image); moved: some entry's pixel is
// not its own
__global__ void k_mc_inv(const int* __restrict__ xm, McRect r, int W, int H, int* __restrict__ inv,
                         int* __restrict__ srcmap, int* __restrict__ moved, int* __restrict__ status) {
  const int E = r.l1 * r.l2;
  const size_t HW = size_t(H) * W;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < E; e += gridDim.x * blockDim.x) {
    const int R1 = r.r1b + e % r.l1, R2 = r.r2b + e / r.l1;
    const int hor = xm[R1 + size_t(R2) * H] - 1, ver = xm[R1 + size_t(R2) * H + HW] - 1;
    if (hor < 0 || hor >= W || ver < 0 || ver >= H) {
      srcmap[R1 * W + R2] = -1;
      atomicExch(status, kStatusMotionRange);
      continue;
    }
    srcmap[R1 * W + R2] = ver * W + hor;
    if (hor != R2 || ver != R1) *moved = 1;
    atomicMax(inv + size_t(ver) * W + hor, e);
  }
}

// The (entry, frame) pairs that scatter: target pixel (its original-mesh point) in the
// image, corners too.  Grid y: frames; the threads run along an image row, the meshes'
// and tables' fast axis (entries count down the columns; 256 x 256 x 20: count and fill
// 118 us with the threads along those, 28 now).
struct McEntry {
  int e, xo;  // entry number, pixel R1*W + R2
};
__device__ __forceinline__ McEntry row_entry(McRect r, int t, int W) {
  const int i = t / r.l2, j = t - i * r.l2;
  return {i + r.l1 * j, (r.r1b + i) * W + r.r2b + j};
}

__global__ void __launch_bounds__(kNT) k_mc_count(const float* __restrict__ xn, const int* __restrict__ srcmap, McRect r,
                                                  int W, int H, int F, int* __restrict__ cnt, int* __restrict__ status) {
  const int t = blockIdx.x * kNT + threadIdx.x;
  if (t >= r.l1 * r.l2) return;
  const McEntry m = row_entry(r, t, W);
  const bool in = srcmap[m.xo] >= 0;
  const size_t HW = size_t(H) * W;
  for (int k = blockIdx.y; k < F; k += gridDim.y) {
    const McPoint q = mc_point(xn, m.xo, k, W, H, F);
    if (!(q.ok && in)) {
      atomicExch(status, kStatusMotionRange);
      continue;
    }
    int* c = cnt + k * HW + size_t(q.pv) * W + q.ph;
    atomicAdd(c, 1);
    atomicAdd(c + 1, 1);
    atomicAdd(c + W, 1);
    atomicAdd(c + W + 1, 1);
  }
}

// exclusive prefix sum of n ints in three launches: per-block scan, scan of the
// block totals, add
__device__ __forceinline__ int block_exclusive_scan(int v, int* swarp, int* total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) swarp[wid] = incl;
  __syncthreads();
  if (wid == 0) {
    int w = lane < int(blockDim.x >> 5) ? swarp[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += u;
    }
    if (lane < int(blockDim.x >> 5)) swarp[lane] = wi - w;
    if (lane == int(blockDim.x >> 5) - 1) *total = wi;
  }
  __syncthreads();
  return swarp[wid] + incl - v;
}

__global__ void __launch_bounds__(kNT) k_scan_blocks(const int* __restrict__ in, size_t n, int* __restrict__ out,
                                                      int* __restrict__ bsum) {
  __shared__ int swarp[kNT / 32];
  __shared__ int total;
  const size_t base = size_t(blockIdx.x) * kScanBlock + size_t(threadIdx.x) * kScanItems;
  int v[kScanItems], s = 0;
#pragma unroll
  for (int u = 0; u < kScanItems; ++u) {
    v[u] = base + u < n ? in[base + u] : 0;
    s += v[u];
  }
  int run = block_exclusive_scan(s, swarp, &total);
#pragma unroll
  for (int u = 0; u < kScanItems; ++u) {
    if (base + u < n) out[base + u] = run;
    run += v[u];
  }
  if (threadIdx.x == 0) bsum[blockIdx.x] = total;
}

// one block: exclusive scan of the nb block totals in place; out[n] = the grand total
__global__ void __launch_bounds__(1024) k_scan_totals(int* __restrict__ bsum, int nb, int* __restrict__ out, size_t n) {
  __shared__ int swarp[32];
  __shared__ int total;
  int carry = 0;
  for (int b0 = 0; b0 < nb; b0 += 1024) {
    const int b = b0 + int(threadIdx.x);
    const int v = b < nb ? bsum[b] : 0;
    const int ex = block_exclusive_scan(v, swarp, &total);
    if (b < nb) bsum[b] = carry + ex;
    carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) out[n] = carry;
}

__global__ void k_scan_add(int* __restrict__ out, size_t n, const int* __restrict__ bsum) {
  const size_t i = size_t(blockIdx.x) * kScanBlock + threadIdx.x;
  const int add = bsum[blockIdx.x];
#pragma unroll
  for (int u = 0; u < kScanItems; ++u)
    if (i + size_t(u) * kNT < n) out[i + size_t(u) * kNT] += add;
}

// the contributions of every scattering (entry, frame) to its four corners,
// and the entry's fractional position (Whh, Wvv) the weights derive from
__global__ void __launch_bounds__(kNT) k_mc_fill(const float* __restrict__ xn, const int* __restrict__ srcmap, McRect r,
                                                 int W, int H, int F, const int* __restrict__ off, int* __restrict__ cur,
                                                 int* __restrict__ key, int* __restrict__ at_out,
                                                 float2* __restrict__ wts) {
  const int t = blockIdx.x * kNT + threadIdx.x;
  if (t >= r.l1 * r.l2) return;
  const McEntry m = row_entry(r, t, W);
  const bool in = srcmap[m.xo] >= 0;
  const size_t HW = size_t(H) * W;
  for (int k = blockIdx.y; k < F; k += gridDim.y) {
    const McPoint q = mc_point(xn, m.xo, k, W, H, F);
    at_out[k * HW + m.xo] = q.ok ? q.ph + q.pv * W : -1;
    wts[k * HW + m.xo] = make_float2(q.nh - float(q.ph), q.nv - float(q.pv));
    if (!q.ok || !in) continue;
    const size_t q00 = k * HW + size_t(q.pv) * W + q.ph;
    const size_t tq[4] = {q00, q00 + 1, q00 + W, q00 + W + 1};
    int at[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) at[c] = off[tq[c]] + atomicAdd(cur + tq[c], 1);
#pragma unroll
    for (int c = 0; c < 4; ++c) key[at[c]] = m.e * 4 + c;
  }
}

// Each target's contributions in key order (the reference's work-item order), the
// keys then renumbered to the entry's pixel * 4 + corner, and inv likewise, so that no
// later kernel divides.  Lists are short, four where the mesh is smooth: up to kMcShort
// sort in registers, longer ones in place (one kernel for the sort, one for the
// numbers and one for tables of sources and weights: 97 us; 19 here).
constexpr int kMcShort = 8;
__global__ void __launch_bounds__(kNT) k_mc_lists(const int* __restrict__ off, int* __restrict__ key,
                                                  int* __restrict__ inv, McRect r, int W, int HW, int F) {
  const int p = blockIdx.x * kNT + threadIdx.x;
  if (p >= HW) return;
  if (blockIdx.y == 0) {
    const int e = inv[p];
    if (e >= 0) inv[p] = entry_offset(r, e, W);
  }
  for (int k = blockIdx.y; k < F; k += gridDim.y) {
    const size_t q = size_t(k) * HW + p;
    const int b = off[q], n = off[q + 1] - b;
    auto number = [&](int kc) { return entry_offset(r, kc >> 2, W) * 4 + (kc & 3); };
    if (n <= kMcShort) {
      int v[kMcShort];
#pragma unroll
      for (int u = 0; u < kMcShort; ++u) v[u] = u < n ? key[b + u] : 0x7fffffff;
#pragma unroll
      for (int s = 0; s < kMcShort; ++s)  // odd-even transposition
#pragma unroll
        for (int u = s & 1; u + 1 < kMcShort; u += 2) {
          const int lo = min(v[u], v[u + 1]);
          v[u + 1] = max(v[u], v[u + 1]);
          v[u] = lo;
        }
#pragma unroll
      for (int u = 0; u < kMcShort; ++u)
        if (u < n) key[b + u] = number(v[u]);
    } else {
      for (int i = b + 1; i < b + n; ++i) {
        const int v = key[i];
        int j = i - 1;
        while (j >= b && key[j] > v) {
          key[j + 1] = key[j];
          --j;
        }
        key[j + 1] = v;
      }
      for (int c = b; c < b + n; ++c) key[c] = number(key[c]);
    }
  }
}

// (M^T g) at pixel p of the frame whose plane starts at `plane`: the target's
// contributions in the reference's order, where corner c of an entry's square gets
// (g * fa) * fb with fa = Whh or 1 - Whh (c & 1), fb = Wvv or 1 - Wvv (c & 2), as
// optimizer.cl:880-937 rounds them.  The loads of up to four are issued before any is
// accumulated.  The weights come from the entries' table, which four targets share, and
// the pixel from the key, not from tables per contribution (12 bytes each, 63 MB at 256 x
// 256 x 20).  g is read through a plain pointer: other CTAs of the launch may have
// written it before a barrier.
struct McLists {
  const int *off, *key, *srcmap, *moved;
  const float2* wts;
};
__device__ __forceinline__ float2 mc_adjoint_at(const McLists& l, const float2* g, size_t plane, int p, bool in_rect,
                                                bool moved) {
  const float2 *const gk = g + plane, *const wk = l.wts + plane;
  int c = __ldg(l.off + plane + p);
  const int ce = __ldg(l.off + plane + p + 1);
  float2 acc = in_rect ? make_float2(0.f, 0.f) : gk[p];
  for (; c < ce; c += 4) {
    int k[4];
    float2 w[4], v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) k[u] = c + u < ce ? __ldg(l.key + c + u) : -1;
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k[u] >= 0) {
        const int xo = k[u] >> 2;
        w[u] = __ldg(wk + xo);
        v[u] = gk[moved ? __ldg(l.srcmap + xo) : xo];
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (k[u] >= 0) {
        const float fa = (k[u] & 1) ? w[u].x : __fsub_rn(1.f, w[u].x);
        const float fb = (k[u] & 2) ? w[u].y : __fsub_rn(1.f, w[u].y);
        acc.x = __fadd_rn(acc.x, __fmul_rn(__fmul_rn(v[u].x, fa), fb));
        acc.y = __fadd_rn(acc.y, __fmul_rn(__fmul_rn(v[u].y, fa), fb));
      }
  }
  return acc;
}

// ---- the operators -------------------------------------------------------------
// out = M x (MotionCompensation: copy, then the interpolator), one thread per pixel; grid y: frames
__global__ void __launch_bounds__(kNT) k_mc_warp(const float2* __restrict__ x, float2* __restrict__ out, McPoints m,
                                                 int W, int HW, int F) {
  const int p = blockIdx.x * kNT + threadIdx.x;
  if (p >= HW) return;
  const int xo = m.inv[p];
  for (int k = blockIdx.y; k < F; k += gridDim.y) {
    const size_t o = size_t(k) * HW;
    const McAt q = xo >= 0 ? mc_at(m, xo, o) : McAt{-1, make_float2(0.f, 0.f)};
    out[o + p] = mc_value<false>(x + o, q, p, W, 1.f);
  }
}

// out = M^T g (AdjointMotionCompensation: copy, zero the rectangle, scatter), one
// thread per target (two targets' lists in one thread: 100 us more per solve); grid y: frames
__global__ void __launch_bounds__(kNT) k_mc_adjoint(const float2* g, float2* __restrict__ out, McLists l, McRect r,
                                                     int W, int HW, int F, int pdl) {
  const int p = blockIdx.x * kNT + threadIdx.x;
  if (pdl) {
    grid_dep_wait();  // g comes from the fused tTV kernel two launches back
    grid_dep_release();
  }
  if (p >= HW) return;
  const int row = p / W, col = p - row * W;
  const bool in_rect = row >= r.r1b && row < r.r1b + r.l1 && col >= r.r2b && col < r.r2b + r.l2;
  const bool moved = __ldg(l.moved) != 0;
  for (int k = blockIdx.y; k < F; k += gridDim.y) {
    const size_t o = size_t(k) * HW;
    out[o + p] = mc_adjoint_at(l, g, o, p, in_rect, moved);
  }
}

// g = tTVadj(normalise(D M x)) (temporalTV.cl:78-107 sign: u_{f+1} - u_f) and
// the objective's partial sums of |u|^2 and Re<u, d> per (frame, block of 256
// pixels).  grid (ceil(H*W/256), ceil(F/kTvFrames)); each thread warps its
// pixel for kTvFrames+2 consecutive frames (periodic in f) and slides over them.
// Inner iteration `it` reads x_it from the ping-pong pair (x0, x1); past the
// outer loop's last iteration it does nothing, except in the launch that
// recomputes the last update (row-local iteration, fixup), which reads x_last.
__global__ void __launch_bounds__(kNT) k_mc_tv(const float2* __restrict__ x0, const float2* __restrict__ x1, int it,
                                                McPoints m, const NestaDevState* __restrict__ st,
                                                float2* __restrict__ g, double* __restrict__ part, int W, int H, int F) {
  __shared__ double sred[2 * kTvFrames][kNT / 32];
  const int HW = H * W;
  const int p = blockIdx.x * kNT + threadIdx.x;
  const bool live = p < HW;
  const int xo = live ? __ldg(m.inv + p) : -1;
  const int f0 = blockIdx.y * kTvFrames, f1 = min(F, f0 + kTvFrames);
  grid_dep_wait();  // x_k comes from the previous iteration's update
  grid_dep_release();
  const int last = st->last_iter;
  int itx = it;
  if (it > last) {  // uniform over the grid
    if (!(st->fixup && it == last + 1)) return;
    itx = last;
  }
  const float2* __restrict__ x = (itx & 1) ? x1 : x0;
  const float inv_mu = 1.0f / st->mu;
  float su2[kTvFrames], sud[kTvFrames];
#pragma unroll
  for (int u = 0; u < kTvFrames; ++u) su2[u] = sud[u] = 0.f;
  if (live) {
    // M x_k at this pixel for frames f0-1 .. f1 (periodic): positions, then
    // values, so that the loads of all frames are in flight together
    constexpr int NW = kTvFrames + 2;
    const int nw = f1 - f0 + 2;
    McAt q[NW];
    float2 w[NW];
#pragma unroll
    for (int u = 0; u < NW; ++u) {
      q[u].at = -1;
      if (xo >= 0 && u < nw) q[u] = mc_at(m, xo, size_t(wrap_frame(f0 - 1 + u, F)) * HW);
    }
#pragma unroll
    for (int u = 0; u < NW; ++u)
      if (u < nw) w[u] = mc_value<false>(x + size_t(wrap_frame(f0 - 1 + u, F)) * HW, q[u], p, W, 1.f);
#pragma unroll
    for (int u = 0; u < kTvFrames; ++u) {
      const int f = f0 + u;
      if (f < f1) {
        const float2 d0 = csub(w[u + 1], w[u]);
        const float2 u0 = tv_normalize(d0, inv_mu);
        const float2 u1 = tv_normalize(csub(w[u + 2], w[u + 1]), inv_mu);
        su2[u] = fmaf(u0.x, u0.x, u0.y * u0.y);
        sud[u] = fmaf(u0.x, d0.x, u0.y * d0.y);
        g[size_t(f) * HW + p] = csub(u1, u0);
      }
    }
  }
  // fixed-order reduction: FP32 warp shuffles (32 values), then the warps in
  // order in FP64 (FP64 throughput is a small fraction of FP32's here)
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int u = 0; u < kTvFrames; ++u) {
    float a = su2[u], b = sud[u];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      a += __shfl_down_sync(0xffffffffu, a, o);
      b += __shfl_down_sync(0xffffffffu, b, o);
    }
    if (lane == 0) {
      sred[2 * u][wid] = double(a);
      sred[2 * u + 1][wid] = double(b);
    }
  }
  __syncthreads();
  if (threadIdx.x < 2 * kTvFrames) {
    const int u = threadIdx.x >> 1;
    if (f0 + u < f1) {
      double t = 0.0;
#pragma unroll
      for (int w = 0; w < kNT / 32; ++w) t += sred[threadIdx.x][w];
      part[2 * (size_t(f0 + u) * gridDim.x + blockIdx.x) + (threadIdx.x & 1)] = t;
    }
  }
}

// ---- the power method's vector operations ----------------------------------------
__global__ void k_fill(float2* __restrict__ v, size_t n, float2 value) {
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < n; i += size_t(gridDim.x) * blockDim.x) v[i] = value;
}
int grid1(gbn_ctx* ctx, size_t n) { return int(std::min<size_t>((n + kNT - 1) / kNT, size_t(ctx->nsm) * 8)); }

// ---- the power method ||U|| ---------------------------------------------------------
// myNormest's loop (NestaUp.cpp:291-439) with U = tTV M and U^T = M^T tTVadj, whole in
// one cooperative launch.  A step is two phases with a grid barrier after each:
//   1  a thread warps its pixel for kNeFrames + 2 frames (each value once, where a
//      thread per value would warp two frames for it), and writes g = tTVadj(U x)
//      rather than U x itself; partial sums of |U x|^2
//   2  x = M^T g, the ordered gather; partial sums of |x|^2
// After a barrier every CTA adds the same partials in the same order for itself, so
// that nobody waits for another one's scalars.  U x exactly zero (Scasum == 0,
// NestaUp.cpp:369-385) takes a third phase, which puts the drand48 vector in U x's
// place.  x is stored unscaled; its scale 1/||x|| is applied as each value is read,
// which rounds exactly as a separate scaling pass would.  Bound by the latency of the
// gathers out of L2 and of the barriers: at 256 x 256 x 20, 30 steps, 25 K and 33 K
// cycles in the phases and 18 K at each barrier with its sums and the SMs' unevenness,
// 1.13 ms under ncu (1.9 before with six launches a step; four frames a thread in phase 1
// +70 us, 512 threads +200, 1024 and the next item's loads ahead of this one's: nothing).
constexpr int kNeFrames = 2;     // frames per thread of phase 1
constexpr int kNeNT = 768;        // threads of a CTA, one CTA per SM
constexpr int kNeMaxGrid = 256;
constexpr unsigned kNePolls = 1u << 22;
constexpr float kNeTol = 1e-3f;
constexpr int kNeMax = 100;
struct McNe {
  unsigned bar;             // arrivals at the grid barrier
  int bad;                  // some CTA did not arrive in time
  int nrestart;             // restarts (each consumed F*H*W drand48 draws)
  int pad;
};
struct NeArgs {
  float2 *x, *g;
  double* part;             // [3 phases][kNeMaxGrid][2]: sum of squares, any value not zero
  McNe* ne;
  NestaDevState* st;
  McPoints m;
  McLists l;
  McRect r;
  int W, H, F;
  float e;
  unsigned long long rand, ja, jc;  // drand48 state, and its jump by F*H*W draws
};
constexpr size_t kPartBytes = 3 * 2 * kNeMaxGrid * sizeof(double) + sizeof(McNe);

// All CTAs of the launch; false if some did not arrive in time.
__device__ __forceinline__ bool ne_barrier(McNe* ne, unsigned target) {
  __shared__ bool ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&ne->bar, 1u);
    unsigned seen = 0, polls = 0;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(seen) : "l"(&ne->bar) : "memory");
      if (seen >= target || ++polls >= kNePolls) break;
      __nanosleep(32);
    }
    ok = seen >= target;
    if (!ok) atomicExch(&ne->bad, 1);
  }
  __syncthreads();
  return ok;
}

// A thread's sum of squares, whose number of terms grows with the series (11 items at
// 256 x 256 x 20, 140 at 512 x 512 x 64): with Kahan's compensation, so that its error
// stays that of one FP32 addition.  Four FP32 operations an item; an FP64 addition would
// cost 4 K cycles a phase.
struct NeSum {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    const float y = __fsub_rn(v, c), t = __fadd_rn(s, y);
    c = __fsub_rn(__fsub_rn(t, s), y);
    s = t;
  }
};

// The CTA's partial: FP32 within a thread and a warp, FP64 over the warps.
__device__ __forceinline__ void ne_put(double* part, float s2, bool any) {
  __shared__ float sred[kNeNT / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s2 += __shfl_down_sync(0xffffffffu, s2, o);
  if ((threadIdx.x & 31) == 0) sred[threadIdx.x >> 5] = s2;
  const int some = __syncthreads_or(any);
  if (threadIdx.x == 0) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < kNeNT / 32; ++w) t += double(sred[w]);
    part[2 * blockIdx.x] = t;
    part[2 * blockIdx.x + 1] = some ? 1.0 : 0.0;
  }
}
// The root of the launch's sum of squares, and whether any value was not zero.  FP64 by
// one warp, its rate being a small fraction of FP32's here (the root by every thread:
// 4.5 K cycles a step and phase).
__device__ __forceinline__ float ne_total(const double* part, bool* any) {
  __shared__ float root;
  __shared__ int some;
  constexpr int NL = (kNeMaxGrid + 31) / 32;
  if (threadIdx.x < 32) {
    double2 v[NL];
#pragma unroll
    for (int u = 0; u < NL; ++u) {
      const int b = 32 * u + int(threadIdx.x);
      v[u] = b < int(gridDim.x) ? *reinterpret_cast<const double2*>(part + 2 * b) : make_double2(0.0, 0.0);
    }
    double t = 0.0;
    bool a = false;
#pragma unroll
    for (int u = 0; u < NL; ++u) {
      t += v[u].x;
      a |= v[u].y != 0.0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    a = __any_sync(0xffffffffu, a);
    if (threadIdx.x == 0) {
      root = float(sqrt(t));
      some = a;
    }
  }
  __syncthreads();
  *any = some != 0;
  return root;
}

// draw i + 1 of the drand48 generator in state x0
__device__ __forceinline__ float ne_draw(unsigned long long x0, unsigned long long i) {
  unsigned long long ra = 1, rc = 0, ba = 0x5DEECE66DULL, bc = 0xBULL, k = i + 1;
  const unsigned long long mask = (1ULL << 48) - 1;
  while (k) {
    if (k & 1) {
      rc = (ba * rc + bc) & mask;
      ra = (ba * ra) & mask;
    }
    bc = (ba * bc + bc) & mask;
    ba = (ba * ba) & mask;
    k >>= 1;
  }
  return __double2float_rn(double((ra * x0 + rc) & mask) * 0x1p-48);
}

// a thread's walk over its CTA's share of (pixel p, frame or group of frames f) items
struct NeItems {
  int p, f, left;
  __device__ __forceinline__ void share(long long items, int HW) {
    const long long each = ((items + gridDim.x - 1) / gridDim.x + 31) / 32 * 32;
    const long long i0 = each * blockIdx.x + threadIdx.x, i1 = min(items, each * (blockIdx.x + 1));
    left = int(max(0LL, (i1 - i0 + kNeNT - 1) / kNeNT));
    f = int(i0 / HW);
    p = int(i0 - (long long)f * HW);
  }
  __device__ __forceinline__ void next(int HW) {
    --left;
    for (p += kNeNT; p >= HW; p -= HW) ++f;
  }
};

__global__ void __launch_bounds__(kNeNT, 1) k_normest(NeArgs n) {
  const int W = n.W, H = n.H, F = n.F, HW = H * W;
  const McRect r = n.r;
  const bool moved = __ldg(n.l.moved) != 0;
  // a CTA's share of phase 1's (pixel, kNeFrames frames) and phase 2's (pixel, frame)
  // items: whole warps, so that every SM has the same work
  NeItems it1, it2;
  it1.share((long long)HW * ((F + kNeFrames - 1) / kNeFrames), HW);
  it2.share((long long)HW * F, HW);
  unsigned long long rand = n.rand;
  float e = n.e, e0 = 0.f, sc = 1.0f / n.e;
  int cnt = 0, nrestart = 0;
  unsigned gen = 0;
  bool any;
  while (fabsf(e - e0) > kNeTol * e && cnt < kNeMax) {
    NeSum s2;
    bool nz = false;
    for (NeItems i = it1; i.left > 0; i.next(HW)) {
      constexpr int NW = kNeFrames + 2;
      const int f0 = i.f * kNeFrames, nf = min(kNeFrames, F - f0), xo = __ldg(n.m.inv + i.p);
      McAt q[NW];
      float2 w[NW];
#pragma unroll
      for (int u = 0; u < NW; ++u) {
        q[u].at = -1;
        if (xo >= 0 && u < nf + 2) q[u] = mc_at(n.m, xo, size_t(wrap_frame(f0 - 1 + u, F)) * HW);
      }
#pragma unroll
      for (int u = 0; u < NW; ++u)
        if (u < nf + 2) w[u] = mc_value<true>(n.x + size_t(wrap_frame(f0 - 1 + u, F)) * HW, q[u], i.p, W, sc);
#pragma unroll
      for (int u = 0; u < kNeFrames; ++u) {
        if (u < nf) {
          const float2 d = csub(w[u + 1], w[u]);
          s2.add(fmaf(d.x, d.x, d.y * d.y));
          nz |= fabsf(d.x) + fabsf(d.y) != 0.f;
          n.g[size_t(f0 + u) * HW + i.p] = csub(csub(w[u + 2], w[u + 1]), d);
        }
      }
    }
    double* part = n.part;
    ne_put(part, s2.s, nz);
    if (!ne_barrier(n.ne, (gen += gridDim.x))) return;
    e0 = e;
    float root = ne_total(part, &any);
    if (!any) {  // uniform over the grid
      s2 = NeSum{};
      for (NeItems i = it2; i.left > 0; i.next(HW)) {
        const size_t o = size_t(i.f) * HW;
        const float a = ne_draw(rand, o + i.p);
        s2.add(a * a);
        n.g[o + i.p] =
            make_float2(__fsub_rn(ne_draw(rand, (unsigned long long)wrap_frame(i.f + 1, F) * HW + i.p), a), 0.f);
      }
      part += 2 * kNeMaxGrid;
      ne_put(part, s2.s, false);
      if (!ne_barrier(n.ne, (gen += gridDim.x))) return;
      root = ne_total(part, &any);
      rand = (n.ja * rand + n.jc) & ((1ULL << 48) - 1);
      nrestart += 1;
    }
    e = root;
    s2 = NeSum{};
    for (NeItems i = it2; i.left > 0; i.next(HW)) {
      const int p = i.p, row = p / W, col = p - row * W;
      const bool in_rect = row >= r.r1b && row < r.r1b + r.l1 && col >= r.r2b && col < r.r2b + r.l2;
      const float2 acc = mc_adjoint_at(n.l, n.g, size_t(i.f) * HW, p, in_rect, moved);
      n.x[size_t(i.f) * HW + p] = acc;
      s2.add(fmaf(acc.x, acc.x, acc.y * acc.y));
    }
    part = n.part + 4 * kNeMaxGrid;
    ne_put(part, s2.s, false);
    if (!ne_barrier(n.ne, (gen += gridDim.x))) return;
    sc = 1.0f / ne_total(part, &any);
    cnt += 1;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    n.ne->nrestart = nrestart;
    n.st->normU = e;
    n.st->normest_iters = cnt;
    n.st->ne_done = 1;
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
void tables_free(McTables* t) {
  void* ptrs[] = {t->inv, t->cnt, t->off, t->bsum, t->key, t->srcmap, t->at, t->wts, t->tvpart};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  *t = McTables{};
}

dim3 frame_grid(int HW, int F) { return dim3((HW + kNT - 1) / kNT, std::min(F, 65535)); }
McPoints points_of(const McTables& t) { return {t.inv, t.at, t.wts}; }
McLists lists_of(const McTables& t) { return {t.off, t.key, t.srcmap, t.srcmap + t.hw, t.wts}; }

// buffers for F*H*W pixels and E rectangle entries (kept when large enough)
int tables_alloc(McTables* t, int W, int H, int F, int E) {
  const size_t HW = size_t(H) * W, X = HW * F;
  const int nbp = int((HW + kNT - 1) / kNT);
  if (t->inv && t->x == X && t->hw == HW && size_t(E) <= t->entries) return GBN_OK;
  tables_free(t);
  t->x = X;
  t->hw = HW;
  t->entries = size_t(E);
  t->nbp = nbp;
  t->nscan = int((X + kScanBlock - 1) / kScanBlock);
  cudaError_t e = cudaMalloc(&t->inv, HW * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&t->cnt, X * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&t->off, (X + 1) * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&t->bsum, size_t(t->nscan) * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&t->key, 4 * size_t(E) * F * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&t->srcmap, (HW + 1) * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&t->at, X * sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&t->wts, X * sizeof(float2));
  if (e == cudaSuccess) e = cudaMalloc(&t->tvpart, 2 * size_t(F) * nbp * sizeof(double));
  if (e != cudaSuccess) {
    cudaGetLastError();
    tables_free(t);
    return set_error(GBN_ERR_NOMEM, "motion compensation table allocation failed");
  }
  return GBN_OK;
}

// builds inv and the contribution lists from the meshes (asynchronous on s)
int tables_build(gbn_ctx* ctx, McTables* t, const float* xn, const int* xm, const McRect& r, int W, int H, int F,
                 int* status, cudaStream_t s) {
  const size_t HW = size_t(H) * W, X = HW * F;
  const int E = r.l1 * r.l2;
  cudaError_t e = cudaMemsetAsync(t->inv, 0xFF, HW * sizeof(int), s);  // -1
  if (e == cudaSuccess) e = cudaMemsetAsync(t->srcmap + HW, 0, sizeof(int), s);
  if (e == cudaSuccess) e = cudaMemsetAsync(t->cnt, 0, X * sizeof(int), s);
  if (e != cudaSuccess) return cuda_status(e, "motion compensation tables");
  k_mc_inv<<<grid1(ctx, size_t(E)), kNT, 0, s>>>(xm, r, W, H, t->inv, t->srcmap, t->srcmap + HW, status);
  const dim3 ge((E + kNT - 1) / kNT, std::min(F, 65535)), gx(unsigned((HW + kNT - 1) / kNT), std::min(F, 65535));
  k_mc_count<<<ge, kNT, 0, s>>>(xn, t->srcmap, r, W, H, F, t->cnt, status);
  k_scan_blocks<<<t->nscan, kNT, 0, s>>>(t->cnt, X, t->off, t->bsum);
  k_scan_totals<<<1, 1024, 0, s>>>(t->bsum, t->nscan, t->off, X);
  k_scan_add<<<t->nscan, kNT, 0, s>>>(t->off, X, t->bsum);
  if ((e = cudaMemsetAsync(t->cnt, 0, X * sizeof(int), s)) != cudaSuccess)
    return cuda_status(e, "motion compensation tables");
  k_mc_fill<<<ge, kNT, 0, s>>>(xn, t->srcmap, r, W, H, F, t->off, t->cnt, t->key, t->at, t->wts);
  k_mc_lists<<<gx, kNT, 0, s>>>(t->off, t->key, t->inv, r, W, int(HW), F);
  ctx->launches += 7;
  return GBN_OK;
}

}  // namespace

void motion_free(gbn_problem* P) {
  if (P->mc_tab) {
    tables_free(P->mc_tab);
    delete P->mc_tab;
    P->mc_tab = nullptr;
  }
  void* ptrs[] = {P->mc_xw, P->mc_g, P->mc_gm, P->mc_part};
  for (void* p : ptrs)
    if (p) cudaFree(p);
  P->mc_xw = P->mc_g = P->mc_gm = nullptr;
  P->mc_part = nullptr;
}

int motion_set(gbn_problem* P, const float* xn, const int* xmesh, const int* bb) {
  if (!xn && !xmesh && !bb) {
    P->mc_on = false;
    return GBN_OK;
  }
  if (!xn || !xmesh || !bb) return set_error(GBN_ERR_INVALID, "motion compensation needs xn, the mesh and the bounding box");
  const McRect r = mc_rect(P->W, P->H, bb);
  if (!rect_ok(r, P->W, P->H))
    return set_error(GBN_ERR_INVALID, "motion compensation: bounding box plus margins leaves the image");
  const size_t X = size_t(P->W) * P->H * P->F;
  if (!P->mc_xw) {
    cudaError_t e = cudaMalloc(&P->mc_xw, X * sizeof(float2));
    if (e == cudaSuccess) e = cudaMalloc(&P->mc_g, X * sizeof(float2));
    if (e == cudaSuccess) e = cudaMalloc(&P->mc_gm, X * sizeof(float2));
    if (e == cudaSuccess) e = cudaMalloc(&P->mc_part, kPartBytes);
    if (e != cudaSuccess) {
      cudaGetLastError();
      motion_free(P);
      return set_error(GBN_ERR_NOMEM, "motion compensation workspace allocation failed");
    }
  }
  if (!P->mc_tab) P->mc_tab = new McTables();
  const int rc = tables_alloc(P->mc_tab, P->W, P->H, P->F, r.l1 * r.l2);
  if (rc != GBN_OK) return rc;
  P->mc_xn = xn;
  P->mc_xmesh = xmesh;
  std::memcpy(P->mc_bb, bb, sizeof(P->mc_bb));
  P->mc_on = true;
  return GBN_OK;
}

namespace {

// out = M in
void mc_apply(gbn_ctx* ctx, gbn_problem* P, const float2* in, float2* out, cudaStream_t s) {
  const int HW = P->W * P->H;
  k_mc_warp<<<frame_grid(HW, P->F), kNT, 0, s>>>(in, out, points_of(*P->mc_tab), P->W, HW, P->F);
  ctx->launches += 1;
}

// myNormest (NestaUp.cpp:291-439) with U = tTV M, U^T = M^T tTVadj
int mc_normest(gbn_ctx* ctx, gbn_problem* P, cudaStream_t s) {
  const size_t X = size_t(P->W) * P->H * P->F;
  const McTables* t = P->mc_tab;
  const Lcg48 jX = lcg48_jump(uint64_t(X));
  NeArgs n{};
  n.x = P->mc_gm;
  n.g = P->mc_g;
  n.part = P->mc_part;
  n.ne = reinterpret_cast<McNe*>(P->mc_part + 3 * 2 * kNeMaxGrid);
  n.st = P->st;
  n.m = points_of(*t);
  n.l = lists_of(*t);
  n.r = mc_rect(P->W, P->H, P->mc_bb);
  n.W = P->W;
  n.H = P->H;
  n.F = P->F;
  n.e = float(std::sqrt(double(X)));  // ||ones||
  n.rand = (unsigned long long)ctx->rand48;
  n.ja = (unsigned long long)jX.a;
  n.jc = (unsigned long long)jX.c;
  // every CTA of the launch is resident: one per SM
  const size_t items = size_t(P->W) * P->H * ((P->F + kNeFrames - 1) / kNeFrames);
  const int grid = int(std::min<size_t>(std::min(kNeMaxGrid, ctx->nsm), (items + kNeNT - 1) / kNeNT));
  cudaError_t e = cudaMemsetAsync(n.ne, 0, sizeof(McNe), s);
  if (e != cudaSuccess) return cuda_status(e, "power method");
  k_fill<<<grid1(ctx, X), kNT, 0, s>>>(n.x, X, make_float2(1.f, 0.f));
  void* args[] = {&n};
  e = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_normest), dim3(grid), dim3(kNeNT), args, 0, s);
  ctx->launches += 2;
  McNe h{};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, n.ne, sizeof(h), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, "power method");
  if (h.bad) return set_error(GBN_ERR_CUDA, "power method: the CTAs did not all arrive at a barrier");
  for (int i = 0; i < h.nrestart; ++i) ctx->rand48 = lcg48_apply(jX, ctx->rand48);
  return GBN_OK;
}

}  // namespace

// MotionCompensation (dir = GBN_TTV_FORWARD) or AdjointMotionCompensation
// (GBN_TTV_ADJOINT) of one XData [F][H][W] as a single operator.
int motion_op(gbn_ctx* ctx, int dir, const float2* in, float2* out, const float* xn, const int* xm, const int* bb,
              int W, int H, int F) {
  const McRect r = mc_rect(W, H, bb);
  if (!rect_ok(r, W, H))
    return set_error(GBN_ERR_INVALID, "motion compensation: bounding box plus margins leaves the image");
  if (in == out) return set_error(GBN_ERR_INVALID, "motion compensation: input and output must differ");
  void* scr = nullptr;
  int rc = ctx_scratch(ctx, sizeof(int), &scr);
  if (rc != GBN_OK) return rc;
  int* status = static_cast<int*>(scr);
  cudaStream_t s = ctx->stream;
  McTables t;
  if ((rc = tables_alloc(&t, W, H, F, r.l1 * r.l2)) != GBN_OK) return rc;
  cudaError_t e = cudaMemsetAsync(status, 0, sizeof(int), s);
  if (e != cudaSuccess) rc = cuda_status(e, "motion compensation");
  if (rc == GBN_OK) rc = tables_build(ctx, &t, xn, xm, r, W, H, F, status, s);
  if (rc == GBN_OK) {
    if (dir == GBN_TTV_FORWARD)
      k_mc_warp<<<frame_grid(W * H, F), kNT, 0, s>>>(in, out, points_of(t), W, W * H, F);
    else
      k_mc_adjoint<<<frame_grid(W * H, F), kNT, 0, s>>>(in, out, lists_of(t), r, W, W * H, F, 0);
    ctx->launches += 1;
  }
  int h = 0;
  if (rc == GBN_OK) {
    if ((e = cudaMemcpyAsync(&h, status, sizeof(int), cudaMemcpyDeviceToHost, s)) == cudaSuccess)
      e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) rc = cuda_status(e, "motion compensation");
  } else {
    cudaStreamSynchronize(s);
  }
  tables_free(&t);
  if (rc == GBN_OK && h) return set_error(GBN_ERR_INVALID, "motion compensation: a mesh point interpolates outside the image");
  return rc;
}

// The motion-compensated solve of problem P; x_out holds the starting image.
int nesta_run_mc(gbn_ctx* ctx, gbn_problem* P, const gbn_nesta_params* prm, float2* x_out) {
  const SizeKernels* kh = find_size(P->H);
  const SizeKernels* kw = find_size(P->W);
  const int W = P->W, H = P->H, F = P->F, C = P->C;
  cudaStream_t s = ctx->stream;
  McTables* t = P->mc_tab;
  const McRect r = mc_rect(W, H, P->mc_bb);
  int cpb, k2;
  tuning_for(ctx, W, H, F, C, &cpb, &k2);
  cpb = std::max(1, std::min(cpb, C));
  const dim3 g1(W / kWB, (C + cpb - 1) / cpb, F);
  const long long steps = ((long long)F * H * C + kw->rows_per_cta - 1) / kw->rows_per_cta;
  const int g2 = row_grid(ctx, kw, true, steps, k2);
  const dim3 g3(W / kWB, 2, F);
  const dim3 gtv(t->nbp, (F + kTvFrames - 1) / kTvFrames);
  const dim3 gadj = frame_grid(W * H, F);
  auto entry = [&]() {
    FusedArgs a = make_args(P, x_out);
    a.tv_src = P->mc_xw;  // marks the motion-compensated form: the forward pass skips its tTV sums
    a.grad_ext = P->mc_gm;
    a.part_tv = t->tvpart;
    a.ntv = F * t->nbp;
    return a;
  };
  const FusedArgs a = entry();
  const FusedArgs* tab = P->d_args;
  const BatchMap bm = single_map(F, P->ctl);
  int rc;
  // the row-local iteration (rowlocal.cuh) takes problems whose kept rows are
  // fully sampled or unsampled; the row analysis's result comes back to
  // pinned host memory while the setup is queued
  const bool check_rows = ctx->row_local && kh->iter_cols;
  if (check_rows && (rc = partial_flag_ready(ctx)) != GBN_OK) return rc;
  ctx->launches += launch_pre(P, *prm, s, P->d_args, &a, P->ctl);
  cudaError_t ef = cudaSuccess;
  if (check_rows) {
    ef = cudaMemcpyAsync(ctx->host_partial, &P->st->partial_rows, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (ef == cudaSuccess) ef = cudaEventRecord(ctx->ev_partial, s);
    if (ef != cudaSuccess) return cuda_status(ef, "row structure read-back");
  }
  if ((rc = tables_build(ctx, t, P->mc_xn, P->mc_xmesh, r, W, H, F, &P->st->status, s)) != GBN_OK) return rc;
  if (check_rows) {  // T = IDFT_W(y) of the kept rows, the row-local iteration's data term
    kw->rows(tab, bm, 0, false, row_grid(ctx, kw, false, steps, k2), s);
    ctx->launches += 1;
  }
  // maxima of x0 and of U x0 = tTV(M x0) (NestaUp.cpp:491, 521-568)
  mc_apply(ctx, P, x_out, P->mc_xw, s);
  ctx->launches += launch_maxima(ctx, P, x_out, P->mc_xw, s);
  if ((rc = mc_normest(ctx, P, s)) != GBN_OK) return rc;
  ctx->launches += launch_setup(P, s);
  // k_mc_tv and M^T g run on the side stream beside the forward pass: k_mc_tv
  // waits for the iterate (the previous adjoint column pass), the row pass
  // waits for k_mc_tv's objective sums, the adjoint column pass for M^T g
  cudaError_t se = cudaSuccess;
  if (!ctx->mc_stream) {
    se = cudaStreamCreateWithFlags(&ctx->mc_stream, cudaStreamNonBlocking);
    if (se == cudaSuccess) se = cudaEventCreateWithFlags(&ctx->ev_mc_x, cudaEventDisableTiming);
    if (se == cudaSuccess) se = cudaEventCreateWithFlags(&ctx->ev_mc_tv, cudaEventDisableTiming);
    if (se == cudaSuccess) se = cudaEventCreateWithFlags(&ctx->ev_mc_adj, cudaEventDisableTiming);
    if (se != cudaSuccess) return cuda_status(se, "motion-compensated side stream");
  }
  bool row_local = false;
  if (check_rows) {
    if ((ef = cudaEventSynchronize(ctx->ev_partial)) != cudaSuccess) return cuda_status(ef, "row structure read-back");
    row_local = *ctx->host_partial == 0;
  }
  if (row_local && kh->pair_cols) {
    bool fresh = false;
    row_local = problem_tiles(P, false, &fresh) == GBN_OK;
    if (row_local && fresh) ctx->launches += launch_store_args(P->d_args, entry(), s);
  }
  if (row_local) {
    // per inner iteration, on one stream with programmatic dependent launch:
    // k_mc_tv (M x_k, D, normalisation, tTVadj, objective sums), M^T g, and the
    // one-kernel iteration, whose update waits for M^T g; one more launch per
    // outer loop recomputes the last update if the stopping rule ends the loop
    // (the update gathering M^T g itself, without k_mc_adjoint, measured
    // slower: 20.7 against 16.7 ms per reconstruction at 256x256x20, 12 coils)
    const unsigned n_iter_launch = prm->maxIter + (prm->stoptest == 1 ? 1u : 0u);
    for (unsigned nl = 1; nl <= prm->maxIntIter; ++nl) {
      if (kh->pair_cols) {  // the gathers read x_k in the natural order
        ctx->launches += launch_outer_begin_pair(ctx, P, int(nl), x_out, tab, s);
        cudaMemcpyAsync(P->xk0, x_out, size_t(W) * H * F * sizeof(float2), cudaMemcpyDeviceToDevice, s);
      } else {
        ctx->launches += launch_outer_begin(ctx, P, int(nl), x_out, s);
      }
      for (unsigned it = 0; it < n_iter_launch; ++it) {
        launch_pdl(k_mc_tv, gtv, kNT, 0, s, (const float2*)P->xk0, (const float2*)P->xk1, int(it),
                   points_of(*t), (const NestaDevState*)P->st, P->mc_g, t->tvpart, W, H, F);
        launch_pdl(k_mc_adjoint, gadj, kNT, 0, s, (const float2*)P->mc_g, P->mc_gm, lists_of(*t), r, W, W * H, F, 1);
        GBN_LAUNCH(ctx, GBN_PROF_ITER, 1, kh->iter_cols(tab, bm, int(it), true, g3, s));
        ctx->launches += 2;
      }
      ctx->launches += launch_outer_end(ctx, P, x_out, s);
    }
    const cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? GBN_OK : cuda_status(e, "motion-compensated nesta launch");
  }
  cudaStream_t aux = ctx->mc_stream;
  for (unsigned nl = 1; nl <= prm->maxIntIter; ++nl) {
    ctx->launches += launch_outer_begin(ctx, P, int(nl), x_out, s);
    for (unsigned it = 0; it < prm->maxIter; ++it) {
      cudaEventRecord(ctx->ev_mc_x, s);
      cudaStreamWaitEvent(aux, ctx->ev_mc_x, 0);
      k_mc_tv<<<gtv, kNT, 0, aux>>>(P->xk0, P->xk1, int(it), points_of(*t), P->st, P->mc_g, t->tvpart, W, H, F);
      cudaEventRecord(ctx->ev_mc_tv, aux);
      k_mc_adjoint<<<gadj, kNT, 0, aux>>>(P->mc_g, P->mc_gm, lists_of(*t), r, W, W * H, F, 0);
      cudaEventRecord(ctx->ev_mc_adj, aux);
      kh->fwd_cols(tab, bm, int(it), cpb, g1, s);
      cudaStreamWaitEvent(s, ctx->ev_mc_tv, 0);
      kw->rows(tab, bm, int(it), true, g2, s);
      cudaStreamWaitEvent(s, ctx->ev_mc_adj, 0);
      kh->inv_cols(tab, bm, int(it), true, g3, s);
      ctx->launches += 5;
    }
    ctx->launches += launch_outer_end(ctx, P, x_out, s);
  }
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GBN_OK : cuda_status(e, "motion-compensated nesta launch");
}

}  // namespace gbn
