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
  pdl_prologue(A, W);
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

// The same products in tiles of BM x BN outputs a CTA, TM x TN a thread, k in steps of GK through two shared-memory buffers, the next step's
// operands on their way in registers, two neighbouring columns a multiply-add instruction (fma.rn.f32x2: each half rounds as fmaf does).
// The order of an element's sum is the same in all of them. Needs rows that start on 16 bytes.
// Bound by FFMA issue (34 TFMA/s on the whole GPU) beside shared-memory reads: a thread's 16 operands for 64 products are what keeps
// the two even; at 4 x 4 the reads take twice the products' time. Where there are fewer tiles than multiprocessors a product takes as long as
// one CTA does, so the tile's own outputs count: at 80 x 64 and k in steps of 32 (16: the next step's loads come back after the products of
// this one, 87 us) 700 rows 2048 -> 1024 columns 82 us against 111 at 64 x 128 and 281 at 4 x 4 in one buffer, 3072 -> 1024 122 / 160 / 421;
// 1024 -> 4096 146, 1024 -> 6144 191 (tiles of 128 x 128: 203). 32 x 64 and 32 x 32 for some hundred outputs a multiprocessor (100 rows
// 2048 -> 1024 39 us, 64 x 128: 111), 8 x 64 for the few rows of a decode step (8 rows 1024 -> 151936 184 us, 32 x 64: 357).
template <int BM, int BN, int TM, int TN, int GK>
struct GfTile {
  static constexpr int tx = BN / TN, ty = BM / TM, threads = tx * ty;
  static constexpr int blocks = TM * TN >= 40 ? 3 : threads >= 128 ? 5 : 8;  // a multiprocessor's
  static_assert((TM == 8 || TM == 5 || TM == 4) && (TN == 8 || TN == 4) && BM % TM == 0 && BN % TN == 0 && threads % (GK / 4) == 0);
};
template <int BM, int BN, int TM, int TN, int GK>
__global__ void __launch_bounds__((GfTile<BM, BN, TM, TN, GK>::threads), (GfTile<BM, BN, TM, TN, GK>::blocks))
gemm_f32_tiled_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K, int lda, int ldw, int ldc,
                      long long stride_a, long long stride_w, long long stride_c) {
  using I = GfTile<BM, BN, TM, TN, GK>;
  constexpr int THREADS = I::threads, PA = BM * GK / 4, PW = BN * GK / 4, LA = (PA + THREADS - 1) / THREADS, LW = (PW + THREADS - 1) / THREADS;  // pieces of 16 bytes
  __shared__ __align__(16) float as[2][GK][BM + 4], ws[2][GK][BN + 4];
  pdl_prologue();
  const int tid = threadIdx.x, tx = tid % I::tx, ty = tid / I::tx;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  A += blockIdx.z * stride_a;
  W += blockIdx.z * stride_w;
  C += blockIdx.z * stride_c;
  const int pk = tid % (GK / 4) * 4;  // (THREADS is a multiple of GK / 4: the same for all of a thread's pieces)
  auto row_of = [&](int i) { return (tid + i * THREADS) / (GK / 4); };
  const float *ap[LA], *wp[LW];  // (rows behind the end read the last one: what comes of them is not stored)
#pragma unroll
  for (int i = 0; i < LA; ++i) ap[i] = A + (size_t)min(m0 + min(row_of(i), BM - 1), M - 1) * lda + pk;
#pragma unroll
  for (int i = 0; i < LW; ++i) wp[i] = W + (size_t)min(n0 + min(row_of(i), BN - 1), N - 1) * ldw + pk;
  float4 ra[LA], rw[LW];
  auto load = [&](int k0) {
    if (k0 + GK <= K) {
#pragma unroll
      for (int i = 0; i < LA; ++i) ra[i] = behind_loadf4(ap[i] + k0);
#pragma unroll
      for (int i = 0; i < LW; ++i) rw[i] = behind_loadf4(wp[i] + k0);
    } else {  // zeros behind the last k: fma(0, 0, x) is x
      auto piece = [&](const float* p) {
        const int k = k0 + pk;
        return make_float4(k < K ? behind_load(p + k0) : 0.f, k + 1 < K ? behind_load(p + k0 + 1) : 0.f, k + 2 < K ? behind_load(p + k0 + 2) : 0.f,
                           k + 3 < K ? behind_load(p + k0 + 3) : 0.f);
      };
#pragma unroll
      for (int i = 0; i < LA; ++i) ra[i] = piece(ap[i]);
#pragma unroll
      for (int i = 0; i < LW; ++i) rw[i] = piece(wp[i]);
    }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      if (PA % THREADS != 0 && i == LA - 1 && tid + i * THREADS >= PA) break;
      float* p = &as[buf][pk][row_of(i)];
      p[0] = ra[i].x; p[BM + 4] = ra[i].y; p[2 * (BM + 4)] = ra[i].z; p[3 * (BM + 4)] = ra[i].w;
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      if (PW % THREADS != 0 && i == LW - 1 && tid + i * THREADS >= PW) break;
      float* p = &ws[buf][pk][row_of(i)];
      p[0] = rw[i].x; p[BN + 4] = rw[i].y; p[2 * (BN + 4)] = rw[i].z; p[3 * (BN + 4)] = rw[i].w;
    }
  };
  unsigned long long acc[TM][TN / 2];  // two columns each
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
  load(0);
  put(0);
  __syncthreads();
  int buf = 0;
  for (int k0 = 0; k0 < K; k0 += GK, buf ^= 1) {
    const bool more = k0 + GK < K;
    if (more) load(k0 + GK);
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      float a[TM];
      unsigned long long wj[TN / 2];
      *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(&as[buf][kk][ty * 4]);
      if constexpr (TM == 8) *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(&as[buf][kk][BM / 2 + ty * 4]);
      else if constexpr (TM == 5) a[4] = as[buf][kk][4 * I::ty + ty];
#pragma unroll
      for (int h = 0; h < TN / 4; ++h) {
        const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&ws[buf][kk][h * (4 * BN / TN) + tx * 4]);
        wj[2 * h] = w.x;
        wj[2 * h + 1] = w.y;
      }
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        unsigned long long twice;
        asm("mov.b64 %0, {%1, %1};" : "=l"(twice) : "f"(a[i]));
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][j]) : "l"(twice), "l"(wj[j]));
      }
    }
    if (more) put(buf ^ 1);
    __syncthreads();
  }
  const bool wide = ldc % 4 == 0 && stride_c % 4 == 0 && (uintptr_t)C % 16 == 0;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int m = m0 + (i < 4 ? ty * 4 + i : TM == 8 ? BM / 2 + ty * 4 + i - 4 : 4 * I::ty + ty);
    if (m >= M) continue;
#pragma unroll
    for (int half = 0; half < TN / 4; ++half) {
      const int n = n0 + half * (4 * BN / TN) + tx * 4;
      float f[4];
      asm("mov.b64 {%0, %1}, %2;" : "=f"(f[0]), "=f"(f[1]) : "l"(acc[i][2 * half]));
      asm("mov.b64 {%0, %1}, %2;" : "=f"(f[2]), "=f"(f[3]) : "l"(acc[i][2 * half + 1]));
      float* p = C + (size_t)m * ldc + n;
      if (wide && n + 4 <= N) {
        *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (n + e < N) p[e] = f[e];
      }
    }
  }
}

// The tile: what is over first. `each` is what one more tile on the busiest multiprocessor takes and `alone` what the first takes besides (its
// loads and barriers have nothing to run beside), both in tenths of a microsecond for 1024 k; measured over 1 to 2048 rows and 16 to 151936
// columns they give the time to within a tenth. gemm_f32_kernel where rows do not start on 16 bytes and where the products are over before the
// larger tiles' start is made up for: 300 rows 64 -> 1024 columns 6.6 us against 5.9.
inline int launch_gemm_f32(float* C, const float* A, const float* W, int M, int N, int K, int lda, int ldw, int ldc, int batch, long long stride_a,
                           long long stride_w, long long stride_c, cudaStream_t stream) {
  const int known = sm_count(), sms = known > 0 ? known : 148;
  const bool rows16 = lda % 4 == 0 && ldw % 4 == 0 && stride_a % 4 == 0 && stride_w % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0;
  const bool brief = K <= 64 && 2LL * ceil_div(M, GBM) * ceil_div(N, GBN) * batch <= sms;
  if (!rows16 || brief) {
    MS_LAUNCH(gemm_f32_kernel, dim3(ceil_div(N, GBN), ceil_div(M, GBM), batch), 256, 0, stream, C, A, W, M, N, K, lda, ldw, ldc, stride_a, stride_w,
              stride_c);
    return 0;
  }
  int tile = 0;
  long long least = -1;
  auto weigh = [&](int which, int bm, int bn, int each, int alone) {
    const long long tiles = (long long)ceil_div(M, bm) * ceil_div(N, bn) * batch, cost = (tiles + sms - 1) / sms * each + alone;
    if (ceil_div(M, bm) > 65535 || (least >= 0 && cost >= least)) return;
    tile = which;
    least = cost;
  };
  weigh(0, 64, 128, 450, 110);
  weigh(1, 80, 64, 350, 80);
  weigh(2, 32, 64, 200, 90);
  weigh(3, 32, 32, 115, 90);
  weigh(4, 8, 64, 95, 140);
#define MS_GEMM_F32(BM, BN, TM, TN, GK)                                                                                                      \
  MS_LAUNCH_APART((gemm_f32_tiled_kernel<BM, BN, TM, TN, GK>), dim3(ceil_div(N, BN), ceil_div(M, BM), batch),                                \
                  (GfTile<BM, BN, TM, TN, GK>::threads), 0, stream, C, A, W, M, N, K, lda, ldw, ldc, stride_a, stride_w, stride_c)
  if (tile == 0) MS_GEMM_F32(64, 128, 8, 8, 16);
  else if (tile == 1) MS_GEMM_F32(80, 64, 5, 8, 32);
  else if (tile == 2) MS_GEMM_F32(32, 64, 4, 4, 32);
  else if (tile == 3) MS_GEMM_F32(32, 32, 4, 4, 32);
  else MS_GEMM_F32(8, 64, 4, 4, 32);
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
