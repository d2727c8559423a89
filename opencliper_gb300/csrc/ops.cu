// Per-operator kernels: one entry per Process on the NESTA path, operating on
// the reference's dense layouts.  These back the operator-level C ABI and the
// C++ facade's sub-processes; the NESTA solver itself uses the fused kernels.
#include <algorithm>
#include <cmath>
#include <string>

#include "ctx.h"
#include "nesta_kernels.cuh"

namespace gbn {

// Element-wise processes: bound by memory.  In those that write as many values as they
// read a thread takes two adjacent complex values (an image has an even number: W is a
// multiple of 8) in one 16-byte access where every buffer is 16-byte aligned, else in two
// of 8; frames and coils are grid dimensions (strided over, past the grid's limit), so
// that no thread divides (with 8-byte accesses and two 64-bit divisions a value, the eight
// processes of a gradient at 224 x 200 x 16, 10 coils took 117 us; 86 now).
// The normalisation and the sums over coils keep a value per thread: their time is a
// thread's own chain (a root and divisions; a load per coil), which a pair makes longer
// and halves the threads for (us, pairs / values: normalisation of 384 x 384 x 20 11.4 /
// 9.9; coil sum of 128 x 128 x 1, 32 coils 11.3 / 5.1).
namespace {
inline int grid_for(gbn_ctx* ctx, size_t n, int nt = 256) {
  return int(std::max<size_t>(1, std::min<size_t>((n + nt - 1) / nt, size_t(ctx->nsm) * 16)));
}
// CTAs along the pixels of an image, `per` of them a thread, for y x z images
inline dim3 image_grid(gbn_ctx* ctx, int N, int y, int z, int per = 2) {
  y = std::min(y, 65535);
  z = std::min(z, 65535);
  const long long want = std::max<long long>(1, (long long)ctx->nsm * 64 / ((long long)y * z));
  return dim3(unsigned(std::min<long long>((N / per + 255) / 256, want)), unsigned(y), unsigned(z));
}
inline bool aligned16(const void* a, const void* b = nullptr, const void* c = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}
#define GRID_STRIDE(i, n) \
  for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < (n); i += size_t(gridDim.x) * blockDim.x)
#define GRID_PIXELS(i, N) for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (N); i += gridDim.x * blockDim.x)
#define GRID_PAIRS(i, N) for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (N) / 2; i += gridDim.x * blockDim.x)

template <bool V>
__device__ __forceinline__ float4 ld_pair(const float2* p, size_t i) {
  if constexpr (V) return reinterpret_cast<const float4*>(p)[i];
  const float2 a = p[2 * i], b = p[2 * i + 1];
  return make_float4(a.x, a.y, b.x, b.y);
}
template <bool V>
__device__ __forceinline__ void st_pair(float2* p, size_t i, float4 v) {
  if constexpr (V) {
    reinterpret_cast<float4*>(p)[i] = v;
  } else {
    p[2 * i] = make_float2(v.x, v.y);
    p[2 * i + 1] = make_float2(v.z, v.w);
  }
}
}  // namespace

// temporalTV.cl:49-107, grid y: frames
template <bool V>
__global__ void __launch_bounds__(256) k_ttv(const float2* __restrict__ in, float2* __restrict__ out, int N, int F,
                                             int forward) {
  for (int f = blockIdx.y; f < F; f += gridDim.y) {
    const float2* const a = in + size_t(forward ? f : (f + 1) % F) * N;
    const float2* const b = in + size_t(forward ? (f + F - 1) % F : f) * N;
    float2* const o = out + size_t(f) * N;
#pragma unroll 2
    GRID_PAIRS(i, N) {
      const float4 u = ld_pair<V>(a, i), w = ld_pair<V>(b, i);
      st_pair<V>(o, i, make_float4(u.x - w.x, u.y - w.y, u.z - w.z, u.w - w.w));
    }
  }
}

// vectorNormalization.cl:42-56: out = in / fmax(mu, length(in))
__global__ void __launch_bounds__(256) k_normalize(const float2* in, float2* out, size_t n, float mu) {
  GRID_STRIDE(i, n) {
    const float2 v = in[i];
    const float m = fmaxf(mu, sqrtf(fmaf(v.x, v.x, v.y * v.y)));
    out[i] = make_float2(v.x / m, v.y / m);
  }
}

// complexElementProd.cl:42-76: out[f][c][p] = in[f][(c)][p] * (conj?)S[c][p]; grid y: coils, z: frames
template <bool V>
__global__ void __launch_bounds__(256) k_sensmul(const float2* in, int in_has_coils, const float2* __restrict__ S,
                                                 float2* out, int N, int F, int C, int conj) {
  const float sg = conj ? -1.f : 1.f;
  for (int f = blockIdx.z; f < F; f += gridDim.z)
    for (int c = blockIdx.y; c < C; c += gridDim.y) {
      const size_t o = (size_t(f) * C + c) * N;
      const float2* const a0 = in + (in_has_coils ? o : size_t(f) * N);
      const float2* const s0 = S + size_t(c) * N;
      float2* const o0 = out + o;
      GRID_PAIRS(i, N) {
        const float4 a = ld_pair<V>(a0, i);
        float4 s = ld_pair<V>(s0, i);
        s.y *= sg;
        s.w *= sg;
        st_pair<V>(o0, i, make_float4(a.x * s.x - a.y * s.y, a.x * s.y + a.y * s.x, a.z * s.z - a.w * s.w,
                                      a.z * s.w + a.w * s.z));
      }
    }
}

// Pixel i's values of the C coils of a frame (src: coil 0), in order, the loads of
// eight coils (four, one at the end) on their way before the first is used.
template <int U, typename Add>
__device__ __forceinline__ void add_coils(const float2* __restrict__ src, int N, int c, Add&& add) {
  float2 v[U];
#pragma unroll
  for (int u = 0; u < U; ++u) v[u] = src[size_t(c + u) * N];
#pragma unroll
  for (int u = 0; u < U; ++u) add(v[u]);
}
template <typename Add>
__device__ __forceinline__ void over_coils(const float2* __restrict__ src, int N, int C, Add&& add) {
  int c = 0;
  for (; c + 8 <= C; c += 8) add_coils<8>(src, N, c, add);
  if (c + 4 <= C) {
    add_coils<4>(src, N, c, add);
    c += 4;
  }
  for (; c < C; ++c) add_coils<1>(src, N, c, add);
}

// xImageSum.cl:42-61: out[f][p] = sum over coils in order; grid y: frames
__global__ void __launch_bounds__(256) k_coilsum(const float2* __restrict__ in, float2* __restrict__ out, int N, int F,
                                                 int C) {
  for (int f = blockIdx.y; f < F; f += gridDim.y)
    GRID_PIXELS(i, N) {
      float2 acc = make_float2(0.f, 0.f);
      over_coils(in + size_t(f) * C * N + i, N, C, [&](float2 v) { acc = cadd(acc, v); });
      out[size_t(f) * N + i] = acc;
    }
}

// applyMask.cl:5-40; grid y: coils, z: frames.  Only the masked samples are written.
template <bool V>
__global__ void __launch_bounds__(256) k_mask(float2* data, const uint8_t* __restrict__ mask, int N, int F, int C) {
  for (int f = blockIdx.z; f < F; f += gridDim.z)
    for (int c = blockIdx.y; c < C; c += gridDim.y) {
      float2* const d = data + (size_t(f) * C + c) * N;
      const uint8_t* const m = mask + size_t(f) * N;
      GRID_PAIRS(i, N) {
        const bool z0 = m[2 * i] == 0, z1 = m[2 * i + 1] == 0;
        if (z0 && z1) {
          st_pair<V>(d, i, make_float4(0.f, 0.f, 0.f, 0.f));
        } else if (z0 || z1) {
          d[2 * i + (z0 ? 0 : 1)] = make_float2(0.f, 0.f);
        }
      }
    }
}

// SamplingMasksData.cpp:389-441: row value 1 -> 255, 0 -> 0, else error flag
__global__ void k_rowmask(const uint32_t* __restrict__ rm, uint8_t* __restrict__ pm, int W, int H, int F, int* bad) {
  const size_t n = size_t(W) * H * F;
  GRID_STRIDE(i, n) {
    const uint32_t v = rm[i / W];
    if (v > 1u) atomicExch(bad, 1);
    pm[i] = (v == 1u) ? uint8_t(255) : uint8_t(0);
  }
}

// complexAbs.cl:43-70 / complexAbsPow2.cl:43-71
__global__ void k_abs(const float2* in, float2* out, size_t n, int squared) {
  GRID_STRIDE(i, n) {
    const float2 v = in[i];
    const float a2 = v.x * v.x + v.y * v.y;
    out[i] = make_float2(squared ? a2 : sqrtf(a2), 0.f);
  }
}

// ---------------------------------------------------------------------------
int op_ttv(gbn_ctx* ctx, int dir, const float2* in, float2* out, int W, int H, int F) {
  if (in == out) return set_error(GBN_ERR_INVALID, "TemporalTV needs distinct input and output buffers");
  const int N = W * H, fwd = dir == GBN_TTV_FORWARD;
  const dim3 g = image_grid(ctx, N, F, 1);
  if (aligned16(in, out))
    k_ttv<true><<<g, 256, 0, ctx->stream>>>(in, out, N, F, fwd);
  else
    k_ttv<false><<<g, 256, 0, ctx->stream>>>(in, out, N, F, fwd);
  return cuda_status(cudaGetLastError(), "ttv");
}

int op_normalize(gbn_ctx* ctx, const float2* in, float2* out, size_t n, float mu) {
  k_normalize<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(in, out, n, mu);
  return cuda_status(cudaGetLastError(), "normalize");
}

int op_sensmul(gbn_ctx* ctx, int conj, const float2* in, int in_has_coils, const float2* S, float2* out, int W, int H,
               int F, int C) {
  if (!in_has_coils && in == out && C > 1)
    return set_error(GBN_ERR_INVALID, "XData input cannot alias the KData output");
  const int N = W * H;
  const dim3 g = image_grid(ctx, N, C, F);
  if (aligned16(in, S, out))
    k_sensmul<true><<<g, 256, 0, ctx->stream>>>(in, in_has_coils, S, out, N, F, C, conj);
  else
    k_sensmul<false><<<g, 256, 0, ctx->stream>>>(in, in_has_coils, S, out, N, F, C, conj);
  return cuda_status(cudaGetLastError(), "sensmul");
}

int op_coilsum(gbn_ctx* ctx, const float2* in, float2* out, int W, int H, int F, int C) {
  k_coilsum<<<image_grid(ctx, W * H, F, 1, 1), 256, 0, ctx->stream>>>(in, out, W * H, F, C);
  return cuda_status(cudaGetLastError(), "coilsum");
}

int op_mask(gbn_ctx* ctx, float2* data, const uint8_t* mask, int W, int H, int F, int C) {
  const int N = W * H;
  const dim3 g = image_grid(ctx, N, C, F);
  if (aligned16(data))
    k_mask<true><<<g, 256, 0, ctx->stream>>>(data, mask, N, F, C);
  else
    k_mask<false><<<g, 256, 0, ctx->stream>>>(data, mask, N, F, C);
  return cuda_status(cudaGetLastError(), "mask");
}

int op_rowmask(gbn_ctx* ctx, const uint32_t* rm, uint8_t* pm, int W, int H, int F) {
  void* scr = nullptr;
  int rc = ctx_scratch(ctx, sizeof(int), &scr);
  if (rc != GBN_OK) return rc;
  int* bad = static_cast<int*>(scr);
  cudaMemsetAsync(bad, 0, sizeof(int), ctx->stream);
  const size_t n = size_t(W) * H * F;
  k_rowmask<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(rm, pm, W, H, F, bad);
  int hbad = 0;
  cudaError_t e = cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cuda_status(e, "rowmask");
  if (hbad) return set_error(GBN_ERR_INVALID, "sampling mask data element must be 0 or 1");
  return GBN_OK;
}

// rss.cl:43-74 (RSoS): out[f][p] = (sqrt(sum_c |k[f][c][p]|^2), 0), the sum in
// coil order in FP32; grid y: frames
__global__ void __launch_bounds__(256) k_rss(const float2* __restrict__ k, float2* __restrict__ out, int N, int F, int C) {
  for (int f = blockIdx.y; f < F; f += gridDim.y)
    GRID_PIXELS(i, N) {
      float acc = 0.f;
      over_coils(k + size_t(f) * C * N + i, N, C,
                 [&](float2 v) { acc = __fadd_rn(acc, __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y))); });
      out[size_t(f) * N + i] = make_float2(sqrtf(acc), 0.f);
    }
}

int op_rss(gbn_ctx* ctx, const float2* k, float2* out, int W, int H, int F, int C) {
  k_rss<<<image_grid(ctx, W * H, F, 1, 1), 256, 0, ctx->stream>>>(k, out, W * H, F, C);
  ctx->launches += 1;
  return cuda_status(cudaGetLastError(), "rss");
}

int op_abs(gbn_ctx* ctx, const float2* in, float2* out, size_t n, int squared) {
  k_abs<<<grid_for(ctx, n), 256, 0, ctx->stream>>>(in, out, n, squared);
  return cuda_status(cudaGetLastError(), "abs");
}

static int rows_pass(gbn_ctx* ctx, const float2* in, float2* out, int W, int H, long long nrows, int inv, float scale,
                     const uint8_t* mask, int C, bool first = true) {
  if (nrows > 0x7fffffff) return set_error(GBN_ERR_UNSUPPORTED, "too many rows for one transform");
  const SizeKernels* kw = find_size(W);
  const int g = int((nrows + kw->rows_per_cta - 1) / kw->rows_per_cta);
  kw->fft_rows(in, out, int(nrows), inv, scale, ctx_twiddles(ctx, W), mask, C, H, g, first, ctx->stream);
  ctx->launches += 1;
  return GBN_OK;
}

// 2-D FFT of `batch` W x H images: rows along W, then columns along H.
int op_fft2(gbn_ctx* ctx, int direction, const float2* in, float2* out, int W, int H, int batch) {
  const SizeKernels* kw = find_size(W);
  const SizeKernels* kh = find_size(H);
  if (!kw || !kh) return set_error(GBN_ERR_UNSUPPORTED, "unsupported FFT length");
  if (direction != GBN_FFT_FORWARD && direction != GBN_FFT_BACKWARD)
    return set_error(GBN_ERR_INVALID, "FFT direction must be FORWARD or BACKWARD");
  const int inv = direction == GBN_FFT_BACKWARD;
  const float scale = inv ? 1.0f / float(W * H) : 1.0f;
  // (one pass after the other over everything: in chunks whose intermediate stays
  // in L2 the launches' ends cost more than that saves: 384 x 384 x 120 images 247
  // against 230 us there and back)
  const int rc = rows_pass(ctx, in, out, W, H, (long long)batch * H, inv, 1.0f, nullptr, 1);
  if (rc != GBN_OK) return rc;
  kh->fft_cols(out, out, W, batch, inv, scale, ctx_twiddles(ctx, H), ctx->nsm, ctx->stream);
  ctx->launches += 1;
  return cuda_status(cudaGetLastError(), "fft2");
}

// operatorA + 1/sqrt(N): k = mask * FFT2(S x) / sqrt(N): the columns of S_c x_f, then
// the rows with mask and scale
int op_encode(gbn_ctx* ctx, const float2* x, const float2* S, const uint8_t* mask, float2* k, int W, int H, int F,
              int C) {
  const SizeKernels* kh = find_size(H);
  if (!kh || !find_size(W)) return set_error(GBN_ERR_UNSUPPORTED, "unsupported FFT length");
  if (x == k && C > 1) return set_error(GBN_ERR_INVALID, "XData input cannot alias the KData output");
  const float scale = float(1.0 / std::sqrt(double(unsigned(W * H))));
  kh->enc_cols(x, S, k, W, C, F, ctx_twiddles(ctx, H), ctx->stream);
  ctx->launches += 1;
  const int rc = rows_pass(ctx, k, k, W, H, (long long)F * C * H, 0, scale, mask, C, false);
  if (rc != GBN_OK) return rc;
  return cuda_status(cudaGetLastError(), "encode");
}

// Backward rows into `scratch`, then backward columns combined over the coils: E^H
// and SimpleMRIRecon (S given), or SimpleMRIReconSOS.
size_t simple_recon_bytes(int W, int H, int F, int C) { return size_t(F) * C * W * H * sizeof(float2); }
static int adjoint_in(gbn_ctx* ctx, float2* scratch, const float2* k, const float2* S, float2* x, int W, int H, int F,
                      int C, float scale, const float2* twH) {
  const int rc = rows_pass(ctx, k, scratch, W, H, (long long)F * C * H, 1, 1.0f, nullptr, C);
  if (rc != GBN_OK) return rc;
  // CTAs that share a tile's coils: as many as run at once.  A second wave costs more
  // than shorter chains of coils give (E^H in us with 1, 2, 4, 8 CTAs a tile: 512 x 512 x
  // 4 x 8 coils, 256 tiles on 304 places, 54, 100, 116, 155; 72 x 432 x 32 x 4, 288 on 304,
  // 26, 51, 64, 64; 48 x 64 x 40 x 32, 240 on 608, 34, 30, 32, 38; recon of 256 x 256 x 1 x
  // 8, 32 on 456, 19, 16, 12, 10).
  const long long tiles = (long long)(W / kWB) * F, places = (long long)ctx->nsm * find_size(H)->adj_per_sm[S ? 0 : 1];
  int cs = 1;
  while (cs < 8 && 2 * cs <= C && 2 * cs * tiles <= places) cs *= 2;
  find_size(H)->adj_cols(scratch, S, x, W, C, F, scale, twH, cs, ctx->stream);
  ctx->launches += 1;
  return cuda_status(cudaGetLastError(), "adjoint");
}
static int adjoint(gbn_ctx* ctx, const float2* k, const float2* S, float2* x, int W, int H, int F, int C, float scale) {
  if (!find_size(H) || !find_size(W)) return set_error(GBN_ERR_UNSUPPORTED, "unsupported FFT length");
  void* scr = nullptr;
  const int rc = ctx_scratch(ctx, simple_recon_bytes(W, H, F, C), &scr);
  if (rc != GBN_OK) return rc;
  return adjoint_in(ctx, static_cast<float2*>(scr), k, S, x, W, H, F, C, scale, ctx_twiddles(ctx, H));
}

// sqrt(N) pre-scale + operatorAt: x = sum_c conj(S_c) IFFT2(sqrt(N) k_c)
int op_encode_adjoint(gbn_ctx* ctx, const float2* k, const float2* S, float2* x, int W, int H, int F, int C) {
  return adjoint(ctx, k, S, x, W, H, F, C, std::sqrt(float(W * H)) * (1.0f / float(W * H)));
}

__global__ void k_stage_twiddles(const float2* __restrict__ tw, float2* __restrict__ dst, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = tw[i];
}

// SimpleMRIRecon: x = sum_c conj(S_c) ifft2(y_c).  Its column twiddles lie beside
// the intermediates in the scratch, put there by the first call of a shape or
// after another user of the scratch; further calls launch the two passes alone.
// Once a call that uses the scratch has been captured into a graph, what the
// scratch holds is no longer known here (a captured call has not run, a replay
// overwrites it): from then on, and in the captured call itself, the context's
// own table serves.
int simple_recon(gbn_ctx* ctx, const float2* y, const float2* S, float2* x, int W, int H, int F, int C) {
  if (!find_size(H) || !find_size(W)) return set_error(GBN_ERR_UNSUPPORTED, "unsupported FFT length");
  gbn_ctx::SimplePlan& p = ctx->simple_plan;
  const gbn_ctx::SimplePlan had = p;
  void* scr = nullptr;
  const size_t tb = 2 * size_t(H) * sizeof(float2);
  const int rc = ctx_scratch(ctx, tb + simple_recon_bytes(W, H, F, C), &scr);  // forgets the plan
  if (rc != GBN_OK) return rc;
  float2* const tw = static_cast<float2*>(scr);
  const bool keep = !ctx->scratch_in_graph;
  if (keep && (had.ws != scr || had.W != W || had.H != H || had.F != F || had.C != C)) {
    k_stage_twiddles<<<1, 256, 0, ctx->stream>>>(ctx_twiddles(ctx, H), tw, 2 * H);
    ctx->launches += 1;
  }
  const int rc2 = adjoint_in(ctx, tw + 2 * size_t(H), y, S, x, W, H, F, C, 1.0f / float(W * H),
                             keep ? tw : ctx_twiddles(ctx, H));
  if (rc2 == GBN_OK && keep) p = gbn_ctx::SimplePlan{scr, W, H, F, C};
  return rc2;
}
// the same in working memory of simple_recon_bytes that the caller has
int simple_recon_in(gbn_ctx* ctx, void* ws, const float2* y, const float2* S, float2* x, int W, int H, int F, int C) {
  if (!find_size(H) || !find_size(W)) return set_error(GBN_ERR_UNSUPPORTED, "unsupported FFT length");
  return adjoint_in(ctx, static_cast<float2*>(ws), y, S, x, W, H, F, C, 1.0f / float(W * H), ctx_twiddles(ctx, H));
}

// SimpleMRIReconSOS: backward FFT of every coil image (the input stays
// untouched), then the root sum of squares
int simple_recon_sos(gbn_ctx* ctx, const float2* y, float2* x, int W, int H, int F, int C) {
  return adjoint(ctx, y, nullptr, x, W, H, F, C, 1.0f / float(W * H));
}

}  // namespace gbn
