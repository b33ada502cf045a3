// Row-wise kernels of layer stacks:
//   embed_norm      x = scale * E[ids] (+ P[positions] or sinusoids), normed or not;  xn = rmsnorm(x) * w (or x)
//   sandwich_norm   x += rmsnorm(delta) * w_post (or += delta);  xn = rmsnorm(x) * w_next (or x)
//                   delta may have a bias and rows of a second source (a token's experts, weighted or not) added
//   rows_norm       xn[i] = rmsnorm(x[rows[i]]) * w
//   poly_norm       PolyNorm activation: a N(z) + b N(z^2) + c N(z^3) + e, N = division by the row's RMS
// `delta` and `z` arrive as fp32 split-K slabs of the projection in front.  Decode-sized launches spread a
// row over a cluster of eight CTAs (sums exchanged through distributed shared memory), prompt-sized ones
// give a row to one CTA.  All arithmetic is fp32; only what feeds the next product is rounded.
#include "stack_common.cuh"
#include "kernels.h"

namespace bcg {

constexpr int kRowT = 256;          // threads per CTA
constexpr int kRowCluster = 8;
constexpr int kClusterMaxRows = 128;

template <typename T, int V>
__global__ void __launch_bounds__(kRowT)
embed_norm_kernel(const EmbedArgs a, const float* __restrict__ w, float* __restrict__ residual, T* __restrict__ xn, int d,
                  float eps) {
  __shared__ RowSum<kRowT, 1, 1> sh;
  pdl_launch_dependents();
  pdl_wait();
  const long long t = blockIdx.x, row = a.ids[t];
  for (int i = blockIdx.x * kRowT + threadIdx.x; i < a.n_zero; i += gridDim.x * kRowT) a.zero[i] = 0;
  const __nv_bfloat16* pos = nullptr;
  if (a.pos_embed) pos = a.pos_embed + static_cast<long long>(min(a.positions[t], a.n_pos - 1)) * d;
  const double at = a.pos_turns ? a.positions[t] : 0;
  float ss[1] = {0.f};
  for (int v = threadIdx.x * V; v < d; v += kRowT * V) {
    Vec<V> x = load_vec<V>(a.embed + row * d + v);
#pragma unroll
    for (int k = 0; k < V; ++k) x.x[k] *= a.scale;
    if (pos) x.add(load_vec<V>(pos + v));
    if (a.pos_turns) {
      // whole turns are taken off in double precision: the angle is exact at any position
#pragma unroll
      for (int k = 0; k < V; ++k) {
        const double turns = at * a.pos_turns[(v + k) >> 1];
        const float half = static_cast<float>(2.0 * (turns - rint(turns)));
        x.x[k] += ((v + k) & 1) ? cospif(half) : sinpif(half);
      }
    }
    store_vec<V>(residual + t * d + v, x);      // read again below by the same thread
    ss[0] += x.sumsq();
  }
  row_sum<0>(sh, ss);
  float inv = rsqrtf(ss[0] / static_cast<float>(d) + eps);
  if (a.norm) {
    ss[0] = 0.f;
    for (int v = threadIdx.x * V; v < d; v += kRowT * V) {
      Vec<V> x = load_vec<V>(residual + t * d + v);
      const Vec<V> ww = load_vec<V>(a.norm + v);
#pragma unroll
      for (int k = 0; k < V; ++k) x.x[k] *= inv * ww.x[k];
      store_vec<V>(residual + t * d + v, x);
      ss[0] += x.sumsq();
    }
    row_sum<1>(sh, ss);
    inv = rsqrtf(ss[0] / static_cast<float>(d) + eps);
  }
  for (int v = threadIdx.x * V; v < d; v += kRowT * V) {
    Vec<V> x = load_vec<V>(residual + t * d + v);
    if (w) {
      const Vec<V> ww = load_vec<V>(w + v);
#pragma unroll
      for (int k = 0; k < V; ++k) x.x[k] *= inv * ww.x[k];
    }
    store_vec<V>(xn + t * d + v, x);
  }
}

template <typename T, int V, int CL>
__global__ void __launch_bounds__(kRowT)
sandwich_norm_kernel(float* __restrict__ residual, const float* __restrict__ delta, int n_partials,
                     long long partial_stride, const float* __restrict__ w_post, const float* __restrict__ w_next,
                     T* __restrict__ xn, int d, float eps, const NormExtra extra) {
  extern __shared__ float4 stage_raw[];   // this CTA's part of the row
  float* stage = reinterpret_cast<float*>(stage_raw);
  __shared__ RowSum<kRowT, CL, 1> sh;
  pdl_launch_dependents();
  row_sum_begin(sh);
  pdl_wait();
  row_sum_ready<CL>();
  const long long t = CL > 1 ? blockIdx.y : blockIdx.x;
  const int per = (d / V + CL - 1) / CL * V;
  const int v0 = (CL > 1 ? static_cast<int>(blockIdx.x) : 0) * per, v1 = min(d, v0 + per);
  const float inv_d = 1.0f / static_cast<float>(d);
  float ss[1] = {0.f};
  for (int v = v0 + threadIdx.x * V; v < v1; v += kRowT * V) {
    Vec<V> y;
    if (delta) {
      y = slab_sum_vec<V>(delta + t * d + v, n_partials, partial_stride);
    } else {
#pragma unroll
      for (int k = 0; k < V; ++k) y.x[k] = 0.f;
    }
    if (extra.bias) y.add(load_vec<V>(extra.bias + v));
    for (int k = 0; k < extra.per_row; ++k) {
      const Vec<V> row = slab_sum_vec<V>(extra.rows + static_cast<long long>(extra.index[t * extra.per_row + k]) * d + v,
                                         extra.n_partials, extra.partial_stride);
      const float f = extra.weight ? extra.weight[t * extra.per_row + k] : 1.0f;
#pragma unroll
      for (int j = 0; j < V; ++j) y.x[j] = fmaf(f, row.x[j], y.x[j]);
    }
    store_vec<V>(stage + v - v0, y);
    ss[0] += y.sumsq();
  }
  float inv = 1.0f;
  if (w_post) {
    row_sum<0>(sh, ss);
    inv = rsqrtf(ss[0] * inv_d + eps);
  }
  ss[0] = 0.f;
  for (int v = v0 + threadIdx.x * V; v < v1; v += kRowT * V) {
    const Vec<V> y = load_vec<V>(stage + v - v0);
    Vec<V> x = load_vec<V>(residual + t * d + v);
    if (w_post) {
      const Vec<V> ww = load_vec<V>(w_post + v);
#pragma unroll
      for (int k = 0; k < V; ++k) x.x[k] = fmaf(y.x[k], inv * ww.x[k], x.x[k]);
    } else {
#pragma unroll
      for (int k = 0; k < V; ++k) x.x[k] += y.x[k];
    }
    store_vec<V>(residual + t * d + v, x);
    store_vec<V>(stage + v - v0, x);
    if (!w_next && xn) store_vec<V>(xn + t * d + v, x);
    ss[0] += x.sumsq();
  }
  if (w_next) {
    row_sum<1>(sh, ss);
    const float inv2 = rsqrtf(ss[0] * inv_d + eps);
    for (int v = v0 + threadIdx.x * V; v < v1; v += kRowT * V) {
      Vec<V> x = load_vec<V>(stage + v - v0);
      const Vec<V> ww = load_vec<V>(w_next + v);
#pragma unroll
      for (int k = 0; k < V; ++k) x.x[k] *= inv2 * ww.x[k];
      store_vec<V>(xn + t * d + v, x);
    }
  }
}

// A few rows, each spread over a cluster: a thread has one vector of the row from its slabs to its activations, and where the row
// is short GROUPS threads share the vector's slabs and experts.  What counts is how many reads wait for one another: all of a
// thread's are on their way before the first is used, weights even before the predecessor has ended.  In a captured
// decode step of eight rows of 2048 (Bekopel): 6.4 -> 3.9 us, against a cluster whose CTAs had 64 of 256 threads at work and read
// residual and weights behind each sum.
template <typename T, int GROUPS>
__global__ void __launch_bounds__(kRowT)
sandwich_row_kernel(float* residual, const float* delta, int n_partials, long long partial_stride, const float* __restrict__ w_post,
                    const float* __restrict__ w_next, T* xn, int d, float eps, const NormExtra extra) {
  constexpr int CL = kRowCluster, kWidth = kRowT / GROUPS;
  __shared__ RowSum<kRowT, CL, 1> sh;
  __shared__ float4 part[GROUPS > 1 ? GROUPS - 1 : 1][kWidth];
  const int per = (d / 4 + CL - 1) / CL, warps = (per + 31) / 32;
  const int group = threadIdx.x / kWidth, i = threadIdx.x % kWidth, v = static_cast<int>(blockIdx.x) * per + i;
  const bool mine = i < per && v < d / 4;
  const long long t = blockIdx.y;
  pdl_launch_dependents();
  row_sum_begin(sh, warps);
  Vec<4> wp, wn, y;
#pragma unroll
  for (int k = 0; k < 4; ++k) wp.x[k] = wn.x[k] = y.x[k] = 0.f;
  if (mine && group == 0) {
    if (w_post) wp = load_vec<4>(w_post + 4 * v);
    if (w_next) wn = load_vec<4>(w_next + 4 * v);
    if (extra.bias) y = load_vec<4>(extra.bias + 4 * v);
  }
  pdl_wait();
  Vec<4> x = y;
  if (mine) {
    if (group == 0) x = load_vec<4>(residual + t * d + 4 * v);
    if (delta) {
      const int s0 = group * n_partials / GROUPS, s1 = (group + 1) * n_partials / GROUPS;
      if (s1 > s0) y.add(slab_sum_vec<4>(delta + t * d + 4 * v + s0 * partial_stride, s1 - s0, partial_stride));
    }
    for (int k0 = group; k0 < extra.per_row; k0 += 2 * GROUPS) {     // two experts' reads together
      int at[2];
      float f[2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const long long k = t * extra.per_row + min(k0 + j * GROUPS, extra.per_row - 1);
        at[j] = extra.index[k];
        f[j] = k0 + j * GROUPS >= extra.per_row ? 0.f : extra.weight ? extra.weight[k] : 1.0f;
      }
      Vec<4> row[2];
#pragma unroll
      for (int j = 0; j < 2; ++j)
        row[j] = slab_sum_vec<4>(extra.rows + static_cast<long long>(at[j]) * d + 4 * v, extra.n_partials, extra.partial_stride);
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (k0 + j * GROUPS < extra.per_row)
#pragma unroll
          for (int k = 0; k < 4; ++k) y.x[k] = fmaf(f[j], row[j].x[k], y.x[k]);
    }
  }
  if constexpr (GROUPS > 1) {
    if (group) part[group - 1][i] = make_float4(y.x[0], y.x[1], y.x[2], y.x[3]);
    __syncthreads();
  }
  row_sum_ready<CL>();
  if (threadIdx.x >= 32 * warps) return;
  if constexpr (GROUPS > 1) {
#pragma unroll
    for (int g = 0; g < GROUPS - 1; ++g) y.add(load_vec<4>(&part[g][i].x));
  }
  const float inv_d = 1.0f / static_cast<float>(d);
  if (w_post) {
    float ss[1] = {y.sumsq()};
    row_sum<0>(sh, ss, warps);
    const float inv = rsqrtf(ss[0] * inv_d + eps);
#pragma unroll
    for (int k = 0; k < 4; ++k) x.x[k] = fmaf(y.x[k], inv * wp.x[k], x.x[k]);
  } else {
    x.add(y);
  }
  if (!mine) {
#pragma unroll
    for (int k = 0; k < 4; ++k) x.x[k] = 0.f;
  }
  if (mine) store_vec<4>(residual + t * d + 4 * v, x);
  if (w_next) {
    float ss[1] = {x.sumsq()};
    row_sum<1>(sh, ss, warps);
    const float inv = rsqrtf(ss[0] * inv_d + eps);
#pragma unroll
    for (int k = 0; k < 4; ++k) x.x[k] *= inv * wn.x[k];
  }
  if (mine && xn) store_vec<4>(xn + t * d + 4 * v, x);
}

// Prompts: a row per CTA, kept in registers; all reads of a thread are on their way before the first is used.  12,436 rows of 2048:
// 90 -> 76 us (a row staged in shared memory before), 6,378 with eight experts' rows each 150 -> 129.
template <typename T, int THREADS, int NV>
__global__ void __launch_bounds__(THREADS)
sandwich_long_kernel(float* residual, const float* delta, int n_partials, long long partial_stride, const float* __restrict__ w_post,
                     const float* __restrict__ w_next, T* xn, int d, float eps, const NormExtra extra) {
  __shared__ RowSum<THREADS, 1, 1> sh;
  pdl_launch_dependents();
  pdl_wait();
  const long long t = blockIdx.x;
  const int nvec = d / 4;
  Vec<4> x[NV], y[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = static_cast<int>(threadIdx.x) + j * THREADS;
#pragma unroll
    for (int k = 0; k < 4; ++k) x[j].x[k] = y[j].x[k] = 0.f;
    if (v < nvec) {
      if (delta) y[j] = load_vec<4>(delta + t * d + 4 * v);
      x[j] = load_vec<4>(residual + t * d + 4 * v);
    }
  }
  for (int s = 1; s < (delta ? n_partials : 0); ++s) {
    Vec<4> p[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (static_cast<int>(threadIdx.x) + j * THREADS < nvec) p[j] = load_vec<4>(delta + t * d + 4 * (threadIdx.x + j * THREADS) + s * partial_stride);
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (static_cast<int>(threadIdx.x) + j * THREADS < nvec) y[j].add(p[j]);
  }
  if (extra.bias) {
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (static_cast<int>(threadIdx.x) + j * THREADS < nvec) y[j].add(load_vec<4>(extra.bias + 4 * (threadIdx.x + j * THREADS)));
  }
  for (int k = 0; k < extra.per_row; ++k) {
    const float* row = extra.rows + static_cast<long long>(extra.index[t * extra.per_row + k]) * d;
    const float f = extra.weight ? extra.weight[t * extra.per_row + k] : 1.0f;
    Vec<4> p[NV];
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (static_cast<int>(threadIdx.x) + j * THREADS < nvec) p[j] = load_vec<4>(row + 4 * (threadIdx.x + j * THREADS));
    for (int s = 1; s < extra.n_partials; ++s)
#pragma unroll
      for (int j = 0; j < NV; ++j)
        if (static_cast<int>(threadIdx.x) + j * THREADS < nvec)
          p[j].add(load_vec<4>(row + 4 * (threadIdx.x + j * THREADS) + s * extra.partial_stride));
#pragma unroll
    for (int j = 0; j < NV; ++j)
      if (static_cast<int>(threadIdx.x) + j * THREADS < nvec)
#pragma unroll
        for (int i = 0; i < 4; ++i) y[j].x[i] = fmaf(f, p[j].x[i], y[j].x[i]);
  }
  const float inv_d = 1.0f / static_cast<float>(d);
  float ss[1] = {0.f};
  if (w_post) {
#pragma unroll
    for (int j = 0; j < NV; ++j) ss[0] += y[j].sumsq();
    row_sum<0>(sh, ss);
    const float inv = rsqrtf(ss[0] * inv_d + eps);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
      const int v = static_cast<int>(threadIdx.x) + j * THREADS;
      if (v < nvec) {
        const Vec<4> w = load_vec<4>(w_post + 4 * v);
#pragma unroll
        for (int k = 0; k < 4; ++k) x[j].x[k] = fmaf(y[j].x[k], inv * w.x[k], x[j].x[k]);
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < NV; ++j) x[j].add(y[j]);
  }
  float inv = 1.0f;
  if (w_next) {
    ss[0] = 0.f;
#pragma unroll
    for (int j = 0; j < NV; ++j) ss[0] += x[j].sumsq();
    row_sum<1>(sh, ss);
    inv = rsqrtf(ss[0] * inv_d + eps);
  }
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = static_cast<int>(threadIdx.x) + j * THREADS;
    if (v >= nvec) break;
    store_vec<4>(residual + t * d + 4 * v, x[j]);
    if (w_next) {
      const Vec<4> w = load_vec<4>(w_next + 4 * v);
#pragma unroll
      for (int k = 0; k < 4; ++k) x[j].x[k] *= inv * w.x[k];
    }
    if (xn) store_vec<4>(xn + t * d + 4 * v, x[j]);
  }
}

template <typename T, int V>
__global__ void __launch_bounds__(kRowT)
rows_norm_kernel(const float* __restrict__ residual, const int* __restrict__ rows, const float* __restrict__ w,
                 T* __restrict__ xn, int d, float eps) {
  __shared__ RowSum<kRowT, 1, 1> sh;
  pdl_launch_dependents();
  pdl_wait();
  const long long t = blockIdx.x, src = rows[t];
  float ss[1] = {0.f};
  for (int v = threadIdx.x * V; v < d; v += kRowT * V) ss[0] += load_vec<V>(residual + src * d + v).sumsq();
  row_sum<0>(sh, ss);
  const float inv = rsqrtf(ss[0] / static_cast<float>(d) + eps);
  for (int v = threadIdx.x * V; v < d; v += kRowT * V) {
    Vec<V> x = load_vec<V>(residual + src * d + v);
    const Vec<V> ww = load_vec<V>(w + v);
#pragma unroll
    for (int k = 0; k < V; ++k) x.x[k] *= inv * ww.x[k];
    store_vec<V>(xn + t * d + v, x);
  }
}

template <typename T, int V, int CL>
__global__ void __launch_bounds__(kRowT)
poly_norm_kernel(const float* __restrict__ z, int n_partials, long long partial_stride,
                 const float* __restrict__ coef, T* __restrict__ out, int ff, float eps) {
  extern __shared__ float4 stage_raw[];
  float* stage = reinterpret_cast<float*>(stage_raw);
  __shared__ RowSum<kRowT, CL, 3> sh;
  pdl_launch_dependents();
  row_sum_begin(sh);
  pdl_wait();
  row_sum_ready<CL>();
  const long long t = CL > 1 ? blockIdx.y : blockIdx.x;
  const int per = (ff / V + CL - 1) / CL * V;
  const int v0 = (CL > 1 ? static_cast<int>(blockIdx.x) : 0) * per, v1 = min(ff, v0 + per);
  float s[3] = {0.f, 0.f, 0.f};   // sums of z^2, z^4, z^6
  for (int v = v0 + threadIdx.x * V; v < v1; v += kRowT * V) {
    const Vec<V> x = slab_sum_vec<V>(z + t * ff + v, n_partials, partial_stride);
    store_vec<V>(stage + v - v0, x);
#pragma unroll
    for (int k = 0; k < V; ++k) {
      const float x2 = x.x[k] * x.x[k], x4 = x2 * x2;
      s[0] += x2;
      s[1] += x4;
      s[2] = fmaf(x4, x2, s[2]);
    }
  }
  row_sum<0>(sh, s);
  const float inv_f = 1.0f / static_cast<float>(ff);
  const float a = coef[0] * rsqrtf(s[0] * inv_f + eps), b = coef[1] * rsqrtf(s[1] * inv_f + eps),
              c = coef[2] * rsqrtf(s[2] * inv_f + eps), e = coef[3];
  for (int v = v0 + threadIdx.x * V; v < v1; v += kRowT * V) {
    Vec<V> x = load_vec<V>(stage + v - v0);
#pragma unroll
    for (int k = 0; k < V; ++k) x.x[k] = fmaf(x.x[k], fmaf(x.x[k], fmaf(x.x[k], c, b), a), e);
    store_vec<V>(out + t * ff + v, x);
  }
}

// NV vectors per thread, kept in registers between the sums and the polynomial: a few rows over clusters (eight of 7424 in a captured
// step: 7.2 -> 5.4 us), or prompts with a CTA per row (12,436 of 7424: 125 -> 109 us).
template <typename T, int NV, int CL>
__global__ void __launch_bounds__(kRowT)
poly_row_kernel(const float* z, int n_partials, long long partial_stride, const float* __restrict__ coef, T* out, int ff, float eps) {
  __shared__ RowSum<kRowT, CL, 3> sh;
  pdl_launch_dependents();
  row_sum_begin(sh);
  const float c0 = coef[0], c1 = coef[1], c2 = coef[2], e = coef[3];
  const int per = (ff / 4 + CL - 1) / CL, v0 = CL > 1 ? static_cast<int>(blockIdx.x) * per : 0, v1 = min(ff / 4, v0 + per);
  const long long t = CL > 1 ? blockIdx.y : blockIdx.x;
  pdl_wait();
  Vec<4> x[NV];
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = v0 + static_cast<int>(threadIdx.x) + j * kRowT;
    const float* src = z + t * ff + 4 * min(v, ff / 4 - 1);
    if constexpr (CL > 1) x[j] = slab_sum_vec<4>(src, n_partials, partial_stride);
    else x[j] = load_vec<4>(src);
    if (v >= v1)
#pragma unroll
      for (int k = 0; k < 4; ++k) x[j].x[k] = 0.f;
  }
  float s[3] = {0.f, 0.f, 0.f};   // sums of z^2, z^4, z^6
#pragma unroll
  for (int j = 0; j < NV; ++j)
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float x2 = x[j].x[k] * x[j].x[k], x4 = x2 * x2;
      s[0] += x2;
      s[1] += x4;
      s[2] = fmaf(x4, x2, s[2]);
    }
  row_sum_ready<CL>();
  row_sum<0>(sh, s);
  const float inv_f = 1.0f / static_cast<float>(ff);
  const float a = c0 * rsqrtf(s[0] * inv_f + eps), b = c1 * rsqrtf(s[1] * inv_f + eps), c = c2 * rsqrtf(s[2] * inv_f + eps);
#pragma unroll
  for (int j = 0; j < NV; ++j) {
    const int v = v0 + static_cast<int>(threadIdx.x) + j * kRowT;
    if (v >= v1) break;
#pragma unroll
    for (int k = 0; k < 4; ++k) x[j].x[k] = fmaf(x[j].x[k], fmaf(x[j].x[k], fmaf(x[j].x[k], c, b), a), e);
    store_vec<4>(out + t * ff + 4 * v, x[j]);
  }
}

// calls FN<type, vector width>(...) for the activation dtype and the row width
#define BCG_BY_TYPE(FN, WIDTH, DTYPE, ...)                                   \
  do {                                                                       \
    if ((DTYPE) == BCG_DT_F32)                                               \
      return (WIDTH) % 4 ? FN<float, 1>(__VA_ARGS__) : FN<float, 4>(__VA_ARGS__); \
    return (WIDTH) % 4 ? FN<__nv_bfloat16, 1>(__VA_ARGS__) : FN<__nv_bfloat16, 4>(__VA_ARGS__); \
  } while (0)

template <typename T, int V>
static int embed_t(const EmbedArgs& a, const float* w, float* residual, void* xn, int T_rows, int d, float eps,
                   cudaStream_t st) {
  BCG_CUDA_CHECK(launch_k(embed_norm_kernel<T, V>, dim3(T_rows), dim3(kRowT), 0, st, a, w, residual, static_cast<T*>(xn), d,
                          eps));
  return BCG_OK;
}
int embed_norm(const EmbedArgs& a, const float* w, float* residual, void* xn, int act_dtype, int T, int d, float eps,
               cudaStream_t st) {
  BCG_BY_TYPE(embed_t, d, act_dtype, a, w, residual, xn, T, d, eps, st);
}

template <typename T, int V>
static int rows_t(const float* residual, const int* rows, const float* w, void* xn, int n, int d, float eps,
                  cudaStream_t st) {
  BCG_CUDA_CHECK(launch_k(rows_norm_kernel<T, V>, dim3(n), dim3(kRowT), 0, st, residual, rows, w, static_cast<T*>(xn),
                          d, eps));
  return BCG_OK;
}
int rows_norm(const float* residual, const int* rows, const float* w, void* xn, int act_dtype, int n, int d,
              float eps, cudaStream_t st) {
  BCG_BY_TYPE(rows_t, d, act_dtype, residual, rows, w, xn, n, d, eps, st);
}

// One row per cluster (decode) or per CTA; shared memory stages a CTA's part of the row.
static bool row_cluster(int rows, int width) { return rows <= kClusterMaxRows && width >= 1024; }
static size_t row_stage(bool cluster, int width, int v) {
  return static_cast<size_t>(cluster ? (width / v + kRowCluster - 1) / kRowCluster * v : width) * 4;
}

template <typename T, int V>
static int sandwich_t(float* residual, const float* delta, int n_partials, long long stride, const float* w_post,
                      const float* w_next, void* xn, int T_rows, int d, float eps, const NormExtra& extra,
                      cudaStream_t st) {
  const bool cl = row_cluster(T_rows, d);
  const size_t sm = row_stage(cl, d, V);
  T* x = static_cast<T*>(xn);
  const int vecs = (d / 4 + kRowCluster - 1) / kRowCluster;      // of a CTA
  if (cl && V == 4 && vecs <= kRowT) {
    const auto kernel = vecs <= kRowT / 4 ? sandwich_row_kernel<T, 4> : vecs <= kRowT / 2 ? sandwich_row_kernel<T, 2> : sandwich_row_kernel<T, 1>;
    BCG_CUDA_CHECK(launch_cluster(kernel, dim3(kRowCluster, T_rows), dim3(kRowT), kRowCluster, 0, st, residual, delta, n_partials, stride,
                                  w_post, w_next, x, d, eps, extra));
  } else if (cl) {
    BCG_CUDA_CHECK(launch_cluster(sandwich_norm_kernel<T, V, kRowCluster>, dim3(kRowCluster, T_rows), dim3(kRowT),
                                  kRowCluster, sm, st, residual, delta, n_partials, stride, w_post, w_next, x, d, eps, extra));
  } else if (V == 4 && T_rows > kClusterMaxRows && d <= 4096) {
    // wider rows take eight vectors per thread, and staging them is faster: 2,000 rows of 5120 38.9 us staged, 41.0 in registers,
    // 6,000 of 8192 149.5 and 161.8
    const auto kernel = d <= 2048 ? sandwich_long_kernel<T, 128, 4> : sandwich_long_kernel<T, 256, 4>;
    BCG_CUDA_CHECK(launch_k(kernel, dim3(T_rows), dim3(d <= 2048 ? 128 : 256), 0, st, residual, delta, n_partials, stride, w_post, w_next, x,
                            d, eps, extra));
  } else {
    BCG_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(sandwich_norm_kernel<T, V, 1>), 200 * 1024));
    BCG_CUDA_CHECK(launch_k(sandwich_norm_kernel<T, V, 1>, dim3(T_rows), dim3(kRowT), sm, st, residual, delta, n_partials,
                            stride, w_post, w_next, x, d, eps, extra));
  }
  return BCG_OK;
}
int sandwich_norm(float* residual, const float* delta, int n_partials, long long partial_stride,
                  const float* w_post, const float* w_next, void* xn, int act_dtype, int T, int d, float eps,
                  const NormExtra& extra, cudaStream_t st) {
  if (!residual || (!delta && extra.per_row <= 0) || T <= 0 || d <= 0 || d > 51200 || n_partials < 1 || (w_next && !xn)) {
    set_last_error("bcg_sandwich_norm", "bad argument (d <= 51200)");
    return BCG_ERR_ARG;
  }
  BCG_BY_TYPE(sandwich_t, d, act_dtype, residual, delta, n_partials, partial_stride, w_post, w_next, xn, T, d, eps, extra,
              st);
}

template <typename T, int V>
static int poly_t(const float* z, int n_partials, long long stride, const float* coef, void* out, int T_rows, int ff,
                  float eps, cudaStream_t st) {
  const bool cl = row_cluster(T_rows, ff);
  const size_t sm = row_stage(cl, ff, V);
  T* o = static_cast<T*>(out);
  const int vecs = (ff / 4 + kRowCluster - 1) / kRowCluster;     // of a CTA
  if (cl && V == 4 && vecs <= 2 * kRowT) {
    const auto kernel = vecs <= kRowT ? poly_row_kernel<T, 1, kRowCluster> : poly_row_kernel<T, 2, kRowCluster>;
    BCG_CUDA_CHECK(launch_cluster(kernel, dim3(kRowCluster, T_rows), dim3(kRowT), kRowCluster, 0, st, z, n_partials, stride, coef, o, ff, eps));
  } else if (cl) {
    BCG_CUDA_CHECK(launch_cluster(poly_norm_kernel<T, V, kRowCluster>, dim3(kRowCluster, T_rows), dim3(kRowT), kRowCluster,
                                  sm, st, z, n_partials, stride, coef, o, ff, eps));
  } else if (V == 4 && T_rows > kClusterMaxRows && n_partials == 1 && ff <= 16 * 4 * kRowT) {
    const auto kernel = ff <= 4 * 4 * kRowT ? poly_row_kernel<T, 4, 1> : ff <= 8 * 4 * kRowT ? poly_row_kernel<T, 8, 1> : poly_row_kernel<T, 16, 1>;
    BCG_CUDA_CHECK(launch_k(kernel, dim3(T_rows), dim3(kRowT), 0, st, z, n_partials, stride, coef, o, ff, eps));
  } else {
    BCG_TRY(ensure_dynamic_smem(reinterpret_cast<const void*>(poly_norm_kernel<T, V, 1>), 200 * 1024));
    BCG_CUDA_CHECK(launch_k(poly_norm_kernel<T, V, 1>, dim3(T_rows), dim3(kRowT), sm, st, z, n_partials, stride, coef, o,
                            ff, eps));
  }
  return BCG_OK;
}
int poly_norm(const float* z, int n_partials, long long partial_stride, const float* coef, void* out, int act_dtype,
              int T, int ff, float eps, cudaStream_t st) {
  if (!z || !coef || !out || T <= 0 || ff <= 0 || ff > 51200 || n_partials < 1) {
    set_last_error("bcg_poly_norm", "bad argument (ff <= 51200)");
    return BCG_ERR_ARG;
  }
  BCG_BY_TYPE(poly_t, ff, act_dtype, z, n_partials, partial_stride, coef, out, T, ff, eps, st);
}

}  // namespace bcg
