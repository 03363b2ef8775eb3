// True float32 matrix product C[M,N] = A[M,K] * W[N,K]^T on the CUDA cores (FFMA only: no
// tensor cores, no reduced-precision mode). Every output element is accumulated over k = 0..K-1
// in that order with one fused multiply-add per step, whatever M is and wherever the element
// falls in a tile, so a row's result does not depend on what else is in the batch.
// Stands where the reference's float32 run uses F.linear (miniserve/model/qwen3.py:115-131,186).
#include "common.cuh"

namespace ms {

constexpr int GBM = 64, GBN = 64, GBK = 16;

__global__ void __launch_bounds__(256)
gemm_f32_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                int lda, int ldw, int ldc, long long stride_a, long long stride_w, long long stride_c) {
  A += blockIdx.z * stride_a;  // batches of independent products (per-head matrices): one z index each
  W += blockIdx.z * stride_w;
  C += blockIdx.z * stride_c;
  __shared__ float As[GBK][GBM + 4];
  __shared__ float Ws[GBK][GBN + 4];
  pdl_prologue();
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * GBM, n0 = blockIdx.x * GBN;
  const int tx = tid & 15, ty = tid >> 4;  // 16 x 16 threads, each 4 x 4 outputs
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

  // loader mapping: 256 threads, tile 64 x 16 -> each thread 4 elements (one row, 4 consecutive k)
  const int lr = tid >> 2, lk = (tid & 3) * 4;
  for (int k0 = 0; k0 < K; k0 += GBK) {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int k = k0 + lk + e;
      const int am = m0 + lr, wn = n0 + lr;
      As[lk + e][lr] = (am < M && k < K) ? A[(size_t)am * lda + k] : 0.f;
      Ws[lk + e][lr] = (wn < N && k < K) ? W[(size_t)wn * ldw + k] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GBK; ++kk) {
      float a[4], w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
      for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int m = m0 + ty * 4 + i;
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int n = n0 + tx * 4 + j;
      if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
    }
  }
}

// The same products in larger tiles: BM x BN outputs a CTA, 8 x 8 a thread (two runs of four rows by two of four columns), k in steps of
// 16 through two shared-memory buffers, the next step's operands on their way in registers. The order of an element's sum is the same.
// Bound by FFMA issue (34 TFMA/s on the whole GPU) beside shared-memory reads: a thread's 16 operands for 64 products are what keeps
// the two even; at 4 x 4 the reads take twice the products' time.
constexpr int GK = 16;
template <int BM, int BN>
__global__ void __launch_bounds__(BM * BN / 64)
gemm_f32_tiled_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K, int lda, int ldw, int ldc,
                      long long stride_a, long long stride_w, long long stride_c, int vec) {
  constexpr int THREADS = BM * BN / 64, TX = BN / 8, LA = BM * GK / 4 / THREADS, LW = BN * GK / 4 / THREADS;  // float4 a thread brings in
  static_assert(LA * THREADS * 4 == BM * GK && LW * THREADS * 4 == BN * GK, "whole float4 a thread");
  A += blockIdx.z * stride_a;
  W += blockIdx.z * stride_w;
  C += blockIdx.z * stride_c;
  __shared__ __align__(16) float as[2][GK][BM + 4], ws[2][GK][BN + 4];
  pdl_prologue();
  const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  auto fetch = [&](const float* src, int ld, int row, int rows, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);  // (zeros behind the ends: fma(0, 0, x) is x)
    if (row < rows) {
      const float* p = src + (size_t)row * ld + k;
      if (vec && k + 4 <= K) return *reinterpret_cast<const float4*>(p);
      if (k < K) v.x = p[0];
      if (k + 1 < K) v.y = p[1];
      if (k + 2 < K) v.z = p[2];
      if (k + 3 < K) v.w = p[3];
    }
    return v;
  };
  float4 ra[LA], rw[LW];
  auto load = [&](int k0) {
#pragma unroll
    for (int i = 0; i < LA; ++i) ra[i] = fetch(A, lda, m0 + (tid + i * THREADS) / 4, M, k0 + (tid & 3) * 4);
#pragma unroll
    for (int i = 0; i < LW; ++i) rw[i] = fetch(W, ldw, n0 + (tid + i * THREADS) / 4, N, k0 + (tid & 3) * 4);
  };
  auto put = [&](int buf) {
    const int k = (tid & 3) * 4;
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int r = (tid + i * THREADS) / 4;
      as[buf][k][r] = ra[i].x; as[buf][k + 1][r] = ra[i].y; as[buf][k + 2][r] = ra[i].z; as[buf][k + 3][r] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int r = (tid + i * THREADS) / 4;
      ws[buf][k][r] = rw[i].x; ws[buf][k + 1][r] = rw[i].y; ws[buf][k + 2][r] = rw[i].z; ws[buf][k + 3][r] = rw[i].w;
    }
  };
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  load(0);
  put(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += GK, buf ^= 1) {
    const bool more = k0 + GK < K;
    if (more) load(k0 + GK);
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      float a[8], w[8];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&as[buf][kk][ty * 4]);
      *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&as[buf][kk][BM / 2 + ty * 4]);
      *reinterpret_cast<float4*>(w) = *reinterpret_cast<const float4*>(&ws[buf][kk][tx * 4]);
      *reinterpret_cast<float4*>(w + 4) = *reinterpret_cast<const float4*>(&ws[buf][kk][BN / 2 + tx * 4]);
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
    }
    if (more) put(buf ^ 1);
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + (i >> 2) * (BM / 2) + ty * 4 + (i & 3);
    if (m >= M) continue;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int n = n0 + (j >> 2) * (BN / 2) + tx * 4 + (j & 3);
      if (n < N) C[(size_t)m * ldc + n] = acc[i][j];
    }
  }
}

// Which tile: what takes the fewest outputs on the busiest SM. GBM x GBN (4 x 4 a thread, half the rate) where there are few rows.
inline int launch_gemm_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int batch, long long stride_a,
                           long long stride_w, long long stride_c, cudaStream_t stream) {
  static int sms = 0;
  if (sms == 0) {
    int dev = 0;
    MS_CHECK_CUDA(cudaGetDevice(&dev));
    MS_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  }
  const int vec = lda % 4 == 0 && ldw % 4 == 0 && stride_a % 4 == 0 && stride_w % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
  auto cost = [&](int bm, int bn, int slower) {
    const long long tiles = (long long)ceil_div(M, bm) * ceil_div(N, bn) * batch;
    return (tiles + sms - 1) / sms * bm * bn * slower;
  };
  const long long small = cost(GBM, GBN, 2), wide = cost(64, 128, 1), large = cost(128, 128, 1), narrow = cost(64, 64, 1) * 5 / 4;
#define MS_GEMM_F32(BM, BN)                                                                                                                    \
  MS_LAUNCH((gemm_f32_tiled_kernel<BM, BN>), dim3(ceil_div(N, BN), ceil_div(M, BM), batch), BM * BN / 64, 0, stream, C, A, W, M, N, K, lda, ldw, ldc, \
            stride_a, stride_w, stride_c, vec)
  if (M <= 32 || small < wide) {
    MS_LAUNCH(gemm_f32_kernel, dim3(ceil_div(N, GBN), ceil_div(M, GBM), batch), 256, 0, stream, C, A, W, M, N, K, lda, ldw, ldc, stride_a, stride_w,
              stride_c);
  } else if (large <= wide && large <= narrow) MS_GEMM_F32(128, 128);
  else if (wide <= narrow) MS_GEMM_F32(64, 128);
  else MS_GEMM_F32(64, 64);
#undef MS_GEMM_F32
  return 0;
}

}  // namespace ms

using namespace ms;

// Padding k beyond K with zeros adds fma(0, 0, acc) = acc exactly, so it does not disturb the order.
MS_EXPORT int ms_gemm_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc,
                          cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  MS_CHECK_ARG(M > 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
  MS_CHECK_ARG(lda >= K && ldw >= K && ldc >= N, "gemm_f32: leading dimensions too small");
  MS_CHECK_ARG(ceil_div(M, GBM) <= 65535, "gemm_f32: M=%d too large for one launch", M);
  return launch_gemm_f32(C, A, W, M, N, K, lda, ldw, ldc, 1, 0ll, 0ll, 0ll, stream);
}

// `batch` products of the same sizes: product b reads A + b * stride_a and W + b * stride_w and writes C + b * stride_c
// (strides in elements; rows of different products may interleave, as heads do in a [tokens, heads, d] tensor).
MS_EXPORT int ms_gemm_f32_batched(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int batch,
                                  long long stride_a, long long stride_w, long long stride_c, cudaStream_t stream) {
  if (M == 0 || N == 0 || batch == 0) return 0;
  MS_CHECK_ARG(M > 0 && N > 0 && K > 0 && batch > 0 && batch <= 65535, "gemm_f32_batched: bad sizes M=%d N=%d K=%d batch=%d", M, N, K, batch);
  MS_CHECK_ARG(lda >= K && ldw >= K && ldc >= N, "gemm_f32_batched: leading dimensions too small");
  MS_CHECK_ARG(ceil_div(M, GBM) <= 65535, "gemm_f32_batched: M=%d too large for one launch", M);
  return launch_gemm_f32(C, A, W, M, N, K, lda, ldw, ldc, batch, stride_a, stride_w, stride_c, stream);
}
