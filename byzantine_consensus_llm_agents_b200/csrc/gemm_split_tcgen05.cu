// out fp32 [M, ldo] = X fp32 [M, ldx] * W bf16 [N, ldw]^T with every product and sum of fp32 quality, on tensor cores.
//
// An fp32 number is the sum of three bf16 ones, cut off its top bits one after another (8 + 8 + 8 bits of mantissa, no rounding),
// and the weights are bf16 already: X = X1 + X2 + X3, three bf16 products give every partial product exactly (where |x| >= 2^-110 or
// x = 0: below, the last parts leave bf16's range, an error of 2^-133 at most).  What is left to rounding are the sums, and tensor cores cut what they add where FMAs round it: so only the 64 inputs of a k-block (smallest
// part first) meet in TMEM, and the blocks are added in registers.
// Relative error against 64 bits (2-norm), one FMA chain per output / here: 8.1e-7 / 1.3e-7 at K = 2048, 1.9e-6 / 2.5e-7 at
// K = 11264.
//
// CUDA cores bounded the product before (64 x 64 tiles, 16 TFLOP/s).  820 x 2048 -> 12288: 1262 -> 205 us, 820 x 11264 -> 2048:
// 1389 -> 205 us, 40 x 2048 -> 12288: 186 -> 35 us.  Per k-block 12 MMAs of 128 x 128 x 16 take 768 clocks and shared memory's
// bandwidth 1280; what bounds the tile now is the conversion of 128 x 64 activations (eight warps, 2200 clocks).
//
// Roles (576 threads): warp 0 = TMA producer of weight tiles, warp 1 = TMEM alloc + MMA issuer, warps 2-9 add what TMEM holds to
// their registers and store, warps 10-17 read, cut and store activations (three 128B-swizzled K-major planes per stage).
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"

namespace bcg {

constexpr int kSpM = 128, kSpK = 64, kSpPlane = kSpM * kSpK * 2, kSpStages = 3, kSpThreads = 576, kSpWarps = 8;
constexpr int split_stage_bytes(int bn) { return 3 * kSpPlane + bn * kSpK * 2; }
constexpr int split_smem(int bn) { return kSpStages * split_stage_bytes(bn) + 1024 + 256; }

struct SplitArgs {
  const float* x;
  const __nv_bfloat16* w;
  float* out;
  int M, N, K, k_blocks, tiles_m;
  long long ldx, ldw, ldo;
  int vec_out;      // output rows start on 16 bytes
};

// Top eight bits of mantissa of two numbers, as bf16
__device__ __forceinline__ uint32_t top_halves(float a, float b) {
  return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
__device__ __forceinline__ float below_top(float a) { return a - __uint_as_float(__float_as_uint(a) & 0xffff0000u); }

// Outputs that came out as NaN, formed again by FMAs, by one warp: with parts, an infinite weight meets parts of x that are zero.  Rows
// with a NaN among their activations keep theirs.  Covers the warp's own 32 rows and `cols` columns.  Looking for them costs nothing
// that shows (820 x 2048 -> 12288: 208 us with and without).
static __device__ __noinline__ void redo_nans(const SplitArgs& a, int m_first, int n_first, int cols) {
  const int lane = threadIdx.x & 31;
  for (int m = m_first; m < min(m_first + 32, a.M); ++m) {
    const float* x = a.x + m * a.ldx;
    bool settled = false;      // the row was looked at
    for (int c0 = 0; c0 < cols; c0 += 32) {
      const int n_lane = n_first + c0 + lane;
      float* o = a.out + m * a.ldo + n_lane;
      uint32_t left = __ballot_sync(0xffffffffu, c0 + lane < cols && n_lane < a.N && *o != *o);
      if (left && !settled) {
        bool nan = false;
        for (int k = lane; k < a.K; k += 32) nan |= x[k] != x[k];
        if (__any_sync(0xffffffffu, nan)) break;
        settled = true;
      }
      for (; left; left &= left - 1) {
        const int at = __ffs(left) - 1;
        const __nv_bfloat16* w = a.w + (n_first + c0 + at) * a.ldw;
        float s = 0.f;
        for (int k = lane; k < a.K; k += 32) s = fmaf(x[k], __bfloat162float(w[k]), s);
        s = warp_sum(s);
        if (lane == at) *o = s;
      }
    }
  }
}

template <int BN>
__global__ void __launch_bounds__(kSpThreads, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ SplitArgs a) {
  constexpr int STAGE = split_stage_bytes(BN), W_BYTES = BN * kSpK * 2, COLS = BN / 2;
  constexpr uint32_t TMEM_COLS = 2 * BN < 32 ? 32 : 2 * BN;
  constexpr uint32_t IDESC = make_idesc_bf16_m128(BN);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + kSpStages * STAGE);
  uint64_t* empty_bar = full_bar + kSpStages;
  uint64_t* acc_full = empty_bar + kSpStages;
  uint64_t* acc_empty = acc_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    for (int s = 0; s < kSpStages; ++s) {
      mbar_init(&full_bar[s], 1 + kSpWarps * 32);     // the weights' copy and every converting thread
      mbar_init(&empty_bar[s], 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(&acc_full[i], 1);
      mbar_init(&acc_empty[i], kSpWarps * 32);
    }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int m0 = (blockIdx.x % a.tiles_m) * kSpM, n0 = (blockIdx.x / a.tiles_m) * BN;

  if (warp == 0) {
    if (elect_one()) {
      for (int kb = 0, stage = 0, phase = 0; kb < a.k_blocks; ++kb) {
        mbar_wait(&empty_bar[stage], phase ^ 1);
        mbar_arrive_expect_tx(&full_bar[stage], W_BYTES);
        tma_load_2d(smem + stage * STAGE + 3 * kSpPlane, &tmap_w, &full_bar[stage], kb * kSpK, n0, kEvictNormal);
        if (++stage == kSpStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint64_t desc0 = make_kmajor_sw128_desc(smem_u32(smem));
      for (int kb = 0, stage = 0, phase = 0; kb < a.k_blocks; ++kb) {
        const int acc = kb & 1;
        mbar_wait(&acc_empty[acc], ((kb >> 1) & 1) ^ 1);
        mbar_wait(&full_bar[stage], phase);
        tc_fence_after();
        const uint64_t dx = desc0 + static_cast<uint64_t>(stage * (STAGE >> 4));
        const uint64_t dw = dx + (3 * kSpPlane >> 4);
        const uint32_t d = tmem_base + static_cast<uint32_t>(acc * BN);
#pragma unroll
        for (int p = 2; p >= 0; --p)
#pragma unroll
          for (int k = 0; k < kSpK / 16; ++k)
            umma_bf16(d, dx + p * (kSpPlane >> 4) + 2 * k, dw + 2 * k, IDESC, (p < 2 || k > 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
        umma_commit(&acc_full[acc]);
        if (++stage == kSpStages) {
          stage = 0;
          phase ^= 1;
        }
      }
    }
  } else if (warp < 2 + kSpWarps) {
    const int q = warp & 3, half = (warp - 2) >> 2;      // TMEM lanes and columns of this warp
    float sum[COLS];
#pragma unroll
    for (int c = 0; c < COLS; ++c) sum[c] = 0.f;
    for (int kb = 0; kb < a.k_blocks; ++kb) {
      const int acc = kb & 1;
      mbar_wait(&acc_full[acc], (kb >> 1) & 1);
      tc_fence_after();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + static_cast<uint32_t>(acc * BN + half * COLS);
#pragma unroll
      for (int c = 0; c < COLS; c += 16) {
        uint32_t v[16];
        tmem_ld_x16(taddr + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[c + j] += __uint_as_float(v[j]);
      }
      tc_fence_before();
      mbar_arrive(&acc_empty[acc]);
    }
    pdl_wait();      // `out` may still be read
    const int m = m0 + q * 32 + lane, n = n0 + half * COLS;
    if (m < a.M) {
      float* o = a.out + m * a.ldo + n;
#pragma unroll
      for (int c = 0; c < COLS; c += 4) {
        if (a.vec_out && n + c + 4 <= a.N) {
          *reinterpret_cast<float4*>(o + c) = make_float4(sum[c], sum[c + 1], sum[c + 2], sum[c + 3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + c + j < a.N) o[c + j] = sum[c + j];
        }
      }
    }
    float odd = 0.f;
#pragma unroll
    for (int c = 0; c < COLS; ++c) odd = fmaf(0.f, sum[c], odd);
    if (__any_sync(0xffffffffu, odd != 0.f && m < a.M)) {
      __syncwarp();
      redo_nans(a, m0 + q * 32, n, COLS);
    }
  } else {
    // eight lanes read 64 columns of a row, a warp four rows at a time
    const int chunk = lane & 7, r0 = (warp - 2 - kSpWarps) * 4 + (lane >> 3);
    // two k-blocks ahead in registers: one ahead, the reads' latency was on the path of every block (223 -> 205 us)
    float buf[2][4][8];
    auto fetch = [&](int kb, float (&f)[4][8]) {
      const int k = kb * kSpK + chunk * 8;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int m = m0 + r0 + 32 * i;
        if (m < a.M && k < a.K) {
          const float4* src = reinterpret_cast<const float4*>(a.x + m * a.ldx + k);
          *reinterpret_cast<float4*>(&f[i][0]) = src[0];
          *reinterpret_cast<float4*>(&f[i][4]) = src[1];
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) f[i][j] = 0.f;
        }
      }
    };
    int stage = 0, phase = 0;
    auto convert = [&](float (&f)[4][8]) {
      mbar_wait(&empty_bar[stage], phase ^ 1);
      uint8_t* sa = smem + stage * STAGE;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = r0 + 32 * i;
        if (m0 + r < a.M) {       // rows beyond M reach only outputs beyond M
          float r1[8], seen = 0.f;
          uint32_t p1[4], p2[4], p3[4];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            r1[j] = below_top(f[i][j]);
            seen += r1[j];
          }
          if (seen != seen) {     // infinities and NaNs stay what they are in the first part, and the others are zero
#pragma unroll
            for (int j = 0; j < 8; ++j)
              if (r1[j] != r1[j]) {
                r1[j] = 0.f;
                if (f[i][j] != f[i][j]) f[i][j] = __uint_as_float(__float_as_uint(f[i][j]) | 0x00400000u);
              }
          }
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            p1[j] = top_halves(f[i][2 * j], f[i][2 * j + 1]);
            p2[j] = top_halves(r1[2 * j], r1[2 * j + 1]);
            p3[j] = top_halves(below_top(r1[2 * j]), below_top(r1[2 * j + 1]));
          }
          uint8_t* dst = sa + r * 128 + ((chunk ^ (r & 7)) << 4);
          *reinterpret_cast<uint4*>(dst) = make_uint4(p1[0], p1[1], p1[2], p1[3]);
          *reinterpret_cast<uint4*>(dst + kSpPlane) = make_uint4(p2[0], p2[1], p2[2], p2[3]);
          *reinterpret_cast<uint4*>(dst + 2 * kSpPlane) = make_uint4(p3[0], p3[1], p3[2], p3[3]);
        }
      }
      fence_proxy_async();
      mbar_arrive(&full_bar[stage]);
      if (++stage == kSpStages) {
        stage = 0;
        phase ^= 1;
      }
    };
    pdl_wait();
    fetch(0, buf[0]);
    fetch(1, buf[1]);
    for (int kb = 0; kb < a.k_blocks; kb += 2) {
      convert(buf[0]);
      fetch(kb + 2, buf[0]);
      if (kb + 1 == a.k_blocks) break;
      convert(buf[1]);
      fetch(kb + 3, buf[1]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// Activations are read with plain loads, here and above: read-only ones may be moved in front of the wait for the predecessor, as
// nothing in the kernel can change what they read (two heads' products behind one another got the first one's rows again).

// A few rows: weights stream through registers, eight output columns per CTA, the inputs split over four warps.  Two rows of
// 2048 -> 12288: 182 -> 22 us (64 x 64 tiles waited for every 16 inputs' reads), of 11264 -> 2048: 771 -> 20 us.
constexpr int kRowCols = 4;      // output columns per warp: what a loaded activation is used for

template <int MR>
__global__ void __launch_bounds__(256)
gemm_rows_kernel(const float* X, const __nv_bfloat16* __restrict__ W, float* out, int M, int N, int K,
                 long long ldx, long long ldw, long long ldo) {
  __shared__ float part[8][kRowCols * MR];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * 2 * kRowCols + (warp >> 2) * kRowCols;
  float acc[MR][kRowCols] = {};
  uint4 w[kRowCols], next[kRowCols];
  auto fetch = [&](int k, uint4 (&v)[kRowCols]) {
#pragma unroll
    for (int c = 0; c < kRowCols; ++c)
      v[c] = (n0 + c < N && k < K) ? ldg_nc_v4(W + (n0 + c) * ldw + k) : make_uint4(0u, 0u, 0u, 0u);
  };
  pdl_launch_dependents();
  const int k_first = ((warp & 3) * 32 + lane) * 8;
  fetch(k_first, w);
  pdl_wait();
  for (int k = k_first; k < K; k += 1024) {
    fetch(k + 1024, next);
    float wf[kRowCols][8];
#pragma unroll
    for (int c = 0; c < kRowCols; ++c) {
      const uint32_t u[4] = {w[c].x, w[c].y, w[c].z, w[c].w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        wf[c][2 * j] = bf16lo(u[j]);
        wf[c][2 * j + 1] = bf16hi(u[j]);
      }
      w[c] = next[c];
    }
#pragma unroll
    for (int m = 0; m < MR; ++m) {
      const float4* src = reinterpret_cast<const float4*>(X + min(m, M - 1) * ldx + k);
      const float4 lo = src[0], hi = src[1];
      const float x[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
      for (int c = 0; c < kRowCols; ++c)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[m][c] = fmaf(x[j], wf[c][j], acc[m][c]);
    }
  }
#pragma unroll
  for (int m = 0; m < MR; ++m)
#pragma unroll
    for (int c = 0; c < kRowCols; ++c) {
      const float s = warp_sum(acc[m][c]);
      if (lane == 0) part[warp][m * kRowCols + c] = s;
    }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * kRowCols * MR; i += 256) {
    const int g = i / (kRowCols * MR), e = i % (kRowCols * MR), m = e / kRowCols, n = blockIdx.x * 2 * kRowCols + g * kRowCols + e % kRowCols;
    if (m < M && n < N)
      out[m * ldo + n] = (part[4 * g][e] + part[4 * g + 1][e]) + (part[4 * g + 2][e] + part[4 * g + 3][e]);
  }
}

template <int BN>
static int launch_split(const void* W, const SplitArgs& a, long long ldw, cudaStream_t st) {
  CUtensorMap tw;
  if (const int rc = make_tmap_bf16_sw128(&tw, W, a.N, a.K, ldw, BN)) return rc;
  if (const int rc = ensure_dynamic_smem(reinterpret_cast<const void*>(gemm_split_kernel<BN>), split_smem(BN))) return rc;
  BCG_CUDA_CHECK(launch_k(gemm_split_kernel<BN>, dim3(a.tiles_m * ((a.N + BN - 1) / BN)), dim3(kSpThreads), split_smem(BN), st, tw, a));
  return BCG_OK;
}

template <int MR>
static int launch_rows(const float* X, const __nv_bfloat16* W, float* out, int M, int N, int K, long long ldx, long long ldw,
                       long long ldo, cudaStream_t st) {
  BCG_CUDA_CHECK(launch_k(gemm_rows_kernel<MR>, dim3((N + 2 * kRowCols - 1) / (2 * kRowCols)), dim3(256), 0, st, X, W, out, M, N, K, ldx,
                          ldw, ldo));
  return BCG_OK;
}

// Returns BCG_ERR_UNSUPPORTED where rows do not start on 16 bytes (the caller then takes the general kernel).
int gemm_f32(const float* X, const void* W, float* out, int M, int N, int K, long long ldx, long long ldw, long long ldo,
             cudaStream_t st) {
  if (K % 8 || ldw % 8 || ldx % 4 || ((reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(W)) & 15))
    return BCG_ERR_UNSUPPORTED;
  // four rows of 2048 -> 12288 take 29 us as rows, eight 49 us and as a tile 31 us
  if (M <= 4) {
    const auto* w = static_cast<const __nv_bfloat16*>(W);
    if (M == 1) return launch_rows<1>(X, w, out, M, N, K, ldx, ldw, ldo, st);
    if (M == 2) return launch_rows<2>(X, w, out, M, N, K, ldx, ldw, ldo, st);
    return launch_rows<4>(X, w, out, M, N, K, ldx, ldw, ldo, st);
  }
  SplitArgs a = {};
  a.x = X;
  a.w = static_cast<const __nv_bfloat16*>(W);
  a.out = out;
  a.M = M;
  a.N = N;
  a.K = K;
  a.k_blocks = (K + kSpK - 1) / kSpK;
  a.tiles_m = (M + kSpM - 1) / kSpM;
  a.ldx = ldx;
  a.ldw = ldw;
  a.ldo = ldo;
  a.vec_out = (reinterpret_cast<uintptr_t>(out) % 16 == 0 && ldo % 4 == 0) ? 1 : 0;
  // Rounds of one CTA per SM; a narrow tile takes a little more than half the time of a wide one (the conversion is the same)
  const long long wide = static_cast<long long>(a.tiles_m) * ((N + 127) / 128), narrow = static_cast<long long>(a.tiles_m) * ((N + 31) / 32);
  const int sms = num_sms();
  return (wide + sms - 1) / sms * 2 > (narrow + sms - 1) / sms ? launch_split<32>(W, a, ldw, st) : launch_split<128>(W, a, ldw, st);
}

}  // namespace bcg
