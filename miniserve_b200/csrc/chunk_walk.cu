// The recurrences of ``recurrence.cu`` over a prompt by chunks of 16 tokens, in 32-bit accuracy on the tensor cores.
//
//   decay rule:  S <- diag(d_t) S + k_t v_t^T;                                                   o_t = S^T q_t
//   delta rule:  S <- diag(d_t) S;  u_t = beta_t (v_t - S^T k_t);  S <- S + k_t u_t^T;           o_t = S^T q_t
//
// with d_t one decay per key channel, or (decay rule) one per head. Inside a chunk whose first token sees the state S, with G_i the
// product of the decays from the chunk's first token to i, D_ij that of the tokens behind j up to i, and u = v for the decay rule,
//
//   A_ij = beta_i (k_i . D_ij k_j) for j < i,   P_ij = q_i . D_ij k_j for j <= i
//   (I + A) U = diag(beta) (V - (G k) S):   U = U0 - W S   with   (I + A) U0 = diag(beta) V,  (I + A) W = diag(beta) (G k)
//   O = (G q) S + P U,          S_behind = G_last S + (D_(last, .) k)^T U.
//
// The first kernel works out, for all chunks at once, what does not need the state: W, q' = G q, k' = D_(last, .) k, U0, P.
// The second walks a row's chunks in order, a CTA per (16 value columns, head, row): the products of a chunk against the state
// that stays in registers. Both keep 32 bits: sums and the state are float32, and a factor of a tensor-core product is given as two
// tf32 numbers, hi = round(x) and lo = round(x - hi) (22 bits and more of x), of which the three products that matter are made.
// Against 64-bit sums the results are as far off as the token-by-token walk's (a few 1e-8 of the terms' size). A value that is not
// finite makes its column of the whole chunk NaN, in the tokens ahead of it too (a pair that is left out counts zero times it).
//
// What bounds it: the walk is a chain of tokens / 16 steps, each a few dependent tensor-core products and two barriers (one without
// the delta rule); the token-by-token walk is a chain of `tokens` steps of two lane-group sums each.
//
// The accumulator of a product is the next product's operand as it lies in the registers: a warp's slice of 8 N key channels is
// taken as N tiles of 8 of which tile i has the channels N n + i (n = 0..7), so that accumulator columns (2 t, 2 t + 1) of a lane are
// its operand's (t, t + 4), and everything a lane loads of q', W (2 N channels) or k' (N channels) is contiguous.
#include "chunk_mma.cuh"

namespace ms {

constexpr int WK_TOK = 16, WK_THREADS = 128, WK_WARPS = 4, WK_COLS = 16;
enum WalkMode : int { WALK_CHANNEL = 0, WALK_DELTA = 1, WALK_HEAD = 2 };

__device__ __forceinline__ float wk_softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

struct Tf32x2 {
  uint32_t hi, lo;
};
// hi: x rounded to 11 bits of significand, lo: what is left (12 bits and a sign, of which the last is cut off). Integer adds and masks: a
// conversion instruction takes several times their issue slots. A NaN stays one in lo whatever the addition makes of it in hi.
__device__ __forceinline__ Tf32x2 wk_split(float x) {
  Tf32x2 r;
  r.hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
  r.lo = __float_as_uint(x - __uint_as_float(r.hi)) & 0xffffe000u;
  return r;
}
__device__ __forceinline__ void wk_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
struct FragA {
  uint32_t hi[4], lo[4];
};
__device__ __forceinline__ FragA wk_frag(float x0, float x1, float x2, float x3) {
  FragA f;
  const float x[4] = {x0, x1, x2, x3};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const Tf32x2 s = wk_split(x[e]);
    f.hi[e] = s.hi;
    f.lo[e] = s.lo;
  }
  return f;
}
// A product in the accuracy of float32: main += hi hi, rest += lo hi + hi lo (an accumulator of their own: shorter chains). PART 0..2 in turn.
template <int PART>
__device__ __forceinline__ void wk_part(float (&main)[4], float (&rest)[4], const FragA& a, const Tf32x2 (&b)[2]) {
  if constexpr (PART == 0) wk_mma(rest, a.lo, b[0].hi, b[1].hi);
  else if constexpr (PART == 1) wk_mma(main, a.hi, b[0].hi, b[1].hi);
  else wk_mma(rest, a.hi, b[0].lo, b[1].lo);
}

// N consecutive floats (an address that is a multiple of their size up to 16 bytes)
template <int N>
__device__ __forceinline__ void wk_load(float (&f)[N], const float* p) {
  if constexpr (N % 4 == 0) {
#pragma unroll
    for (int e = 0; e < N; e += 4) {
      const float4 v = *reinterpret_cast<const float4*>(p + e);
      f[e] = v.x; f[e + 1] = v.y; f[e + 2] = v.z; f[e + 3] = v.w;
    }
  } else if constexpr (N == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    f[0] = v.x; f[1] = v.y;
  } else {
    f[0] = *p;
  }
}

// ---------------------------------------------------------------- the chunks of a step
// A row of n tokens has ceil(n / 16) chunks, numbered row by row. Every warp finds its own by adding up over the rows, 32 at a time: a table
// made by a launch of its own costs a small step more on the host (4 us) than these sums cost on the device.

// (row, first flat token) of a chunk, the same in every lane; row -1 behind the last chunk
__device__ __forceinline__ int2 wk_at(int chunk, const int* __restrict__ cu_q, int num_rows) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int r0 = 0; r0 < num_rows; r0 += 32) {
    const int r = r0 + lane;
    const int begin = r < num_rows ? cu_q[r] : 0, mine = r < num_rows ? (cu_q[r + 1] - begin + WK_TOK - 1) / WK_TOK : 0;
    int upto = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += x;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, chunk < base + upto);
    if (hit) {
      const int at = __ffs(hit) - 1;
      return make_int2(r0 + at, __shfl_sync(0xffffffffu, begin, at) + (chunk - base - __shfl_sync(0xffffffffu, upto - mine, at)) * WK_TOK);
    }
    base += __shfl_sync(0xffffffffu, upto, 31);
  }
  return make_int2(-1, 0);
}
// how many chunks the rows ahead of `row` have
__device__ __forceinline__ int wk_first(int row, const int* __restrict__ cu_q) {
  int sum = 0;
  for (int r = threadIdx.x & 31; r < row; r += 32) sum += (cu_q[r + 1] - cu_q[r] + WK_TOK - 1) / WK_TOK;
  return __reduce_add_sync(0xffffffffu, sum);
}

// ---------------------------------------------------------------- what a chunk needs beside the state (a decay per key channel)
// grid (chunks, H). W, q', k' [chunks, H, 16, dkp] and last [chunks, H, dkp] float32 (dkp = 32 N >= dk, zeros behind dk), u0
// [chunks, H, 16, dvp] (dvp: dv in whole sixteens, zeros behind; without the delta rule v itself), pairs = P [chunks, H, 16, 16]. z: the
// decays' logits (bias, coef, sign as in recurrence.cu); beta likewise logits.
// Bound by instruction issue: 16 x 16 pairs over dk channels with a decay each. A warp takes four tokens j at once, eight lanes
// over the channels of each, lets their keys decay from j on, and adds up over the lanes at the end (28 exchanges for four tokens).
template <typename TIn, typename TZ, bool DELTA, int N>
__global__ void __launch_bounds__(WK_THREADS)
walk_prepare_kernel(float* __restrict__ w_out, float* __restrict__ q_out, float* __restrict__ k_out, float* __restrict__ last_out,
                    float* __restrict__ u0_out, float* __restrict__ pairs, const TIn* __restrict__ q, int ld_q, const TIn* __restrict__ k,
                    int ld_k, int qk_group, const TIn* __restrict__ v, int ld_v, const TZ* __restrict__ z, int ld_z,
                    const float* __restrict__ z_bias, const float* __restrict__ decay_coef, float z_sign, const TZ* __restrict__ beta,
                    int ld_beta, const float* __restrict__ v_scale, const int* __restrict__ cu_q, int num_rows, int H, int dk, int dv, int dvp,
                    float q_scale) {
  constexpr int DKP = 32 * N;
  __shared__ __align__(16) float qs[WK_TOK][DKP], ks[WK_TOK][DKP], ds[WK_TOK][DKP];
  __shared__ __align__(16) float am[DELTA ? WK_TOK : 1][WK_TOK + 4];
  __shared__ float bs[WK_TOK], vsc[WK_TOK];
  pdl_prologue();
  const int chunk = blockIdx.x, h = blockIdx.y;
  const int2 at = wk_at(chunk, cu_q, num_rows);
  if (at.x < 0) return;
  const int t0 = at.y, n = min(WK_TOK, cu_q[at.x + 1] - t0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t qk_at = (size_t)(h / qk_group) * dk;
  const float coef = decay_coef[h];
#pragma unroll
  for (int e = 0; e < WK_TOK * DKP / WK_THREADS; ++e) {
    const int idx = e * WK_THREADS + tid, i = idx / DKP, c = idx % DKP;
    float fq = 0.f, fk = 0.f, fd = 1.f;
    if (i < n && c < dk) {
      const size_t t = (size_t)(t0 + i);
      fq = Elem<TIn>::load(q + t * ld_q + qk_at + c) * q_scale;
      fk = Elem<TIn>::load(k + t * ld_k + qk_at + c);
      fd = Elem<TZ>::load(z + t * ld_z + (size_t)h * dk + c);
      fd = expf(-coef * wk_softplus(z_sign * (fd + z_bias[(size_t)h * dk + c])));
    }
    qs[i][c] = fq;
    ks[i][c] = fk;
    ds[i][c] = fd;
  }
  if (tid < WK_TOK) {
    float b = 0.f;
    if (DELTA && tid < n) b = 1.0f / (1.0f + expf(-Elem<TZ>::load(beta + (size_t)(t0 + tid) * ld_beta + h)));
    bs[tid] = b;
    vsc[tid] = v_scale && tid < n ? v_scale[(size_t)(t0 + tid) * H + h] : 1.f;
  }
  __syncthreads();
  const size_t item = (size_t)chunk * H + h;
  {
    const int cl = lane & 7, j = warp * 4 + (lane >> 3);
    float p[4 * N] = {}, val[32];
#pragma unroll
    for (int i = 0; i < WK_TOK; ++i) {
      float a = 0.f, b = 0.f;
#pragma unroll
      for (int m = 0; m < N; ++m) {
        float fk[4], fq[4], fd[4];
        wk_load<4>(fk, &ks[i][cl * 4 + 32 * m]);
        wk_load<4>(fq, &qs[i][cl * 4 + 32 * m]);
        wk_load<4>(fd, &ds[i][cl * 4 + 32 * m]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          p[4 * m + e] = i == j ? fk[e] : p[4 * m + e] * fd[e];  // (nothing ahead of token j)
          if (DELTA) a = fmaf(fk[e], p[4 * m + e], a);
          b = fmaf(fq[e], p[4 * m + e], b);
        }
      }
      val[i] = a;
      val[16 + i] = b;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const bool up = cl & o;
#pragma unroll
      for (int i = 0; i < 4 * o; ++i) {
        const float send = up ? val[i] : val[i + 4 * o], keep = up ? val[i + 4 * o] : val[i];
        val[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const int i0 = 4 * (cl & 3);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + e;
      if (cl >= 4) pairs[(item * WK_TOK + i) * WK_TOK + j] = i >= j ? val[e] : 0.f;
      else if (DELTA) am[i][j] = i > j ? val[e] * bs[i] : 0.f;
    }
  }
  if (DELTA) __syncthreads();
  // a thread per key channel: q', W (forward substitution), k', the decay of the whole chunk; and one per value column: U0 likewise
#pragma unroll 1
  for (int c = tid; c < DKP + dvp; c += WK_THREADS) {
    float x[WK_TOK];
    if (c < DKP) {
      float passed = 1.f;
#pragma unroll
      for (int i = 0; i < WK_TOK; ++i) {
        passed *= ds[i][c];
        q_out[(item * WK_TOK + i) * DKP + c] = passed * qs[i][c];
        x[i] = passed * ks[i][c];
      }
      last_out[item * DKP + c] = passed;
      float behind = 1.f;
#pragma unroll
      for (int i = WK_TOK - 1; i >= 0; --i) {
        k_out[(item * WK_TOK + i) * DKP + c] = ks[i][c] * behind;
        behind *= ds[i][c];
      }
    } else {
      const int col = c - DKP;
#pragma unroll
      for (int i = 0; i < WK_TOK; ++i)
        x[i] = i < n && col < dv ? Elem<TIn>::load(v + (size_t)(t0 + i) * ld_v + (size_t)h * dv + col) * vsc[i] : 0.f;
    }
    if (!DELTA && c < DKP) continue;
    float* out = c < DKP ? w_out + item * WK_TOK * DKP + c : u0_out + item * WK_TOK * dvp + (c - DKP);
    const int step = c < DKP ? DKP : dvp;
#pragma unroll
    for (int i = 0; i < WK_TOK; ++i) {
      if (DELTA) {
        float y = bs[i] * x[i];
#pragma unroll
        for (int j = 0; j < i; ++j) y = fmaf(-am[i][j], x[j], y);
        x[i] = y;
      }
      out[(size_t)i * step] = x[i];
    }
  }
}

// ---------------------------------------------------------------- the walk over a row's chunks
// grid (value column tiles, H, rows). The four warps share the key channels out among themselves (8 N each): a product over the key
// channels is four partial sums that meet in shared memory, the state's own update stays inside a warp.
// Channel mode and the delta rule read what walk_prepare_kernel left (qp, wp, kp, dec, u0, pairs). Head mode reads q, k and v
// themselves, and the pairs and decays of walk_head_kernel.
// A chunk's operands come through a ring in shared memory that every lane fills and reads for itself alone (cp.async): a chunk takes
// less time than a load from L2.
template <int MODE, int N, int MT>
struct WalkItems {  // floats of one lane and chunk
  static constexpr int q = 0, w = 4 * N, k = w + (MODE == WALK_DELTA ? 4 * N : 0), last = k + 4 * N,
                       pair = last + (MODE == WALK_HEAD ? 8 : 2 * N), u = pair + 2, more = u + 2 * MT,
                       floats = (more + (MODE == WALK_HEAD ? 2 : 0) + 3) / 4 * 4;
  static constexpr int stages = MODE == WALK_HEAD ? 3 : 4;
  static constexpr int cols = MT * WK_COLS, ld = cols + 4, ldu = WK_TOK + 4;
  static constexpr int ring = stages * floats * WK_THREADS, xs = MODE == WALK_DELTA ? WK_WARPS * WK_TOK * ld : 0, os = 2 * WK_WARPS * WK_TOK * ld,
                       us = (MODE == WALK_DELTA ? 1 : 2) * cols * ldu;
  static constexpr size_t bytes = (size_t)(ring + xs + os + us) * 4;
};

// BYTES from global memory into shared memory, zeros where not `in`
template <int BYTES>
__device__ __forceinline__ void wk_cp(float* dst, const float* src, bool in) {
  const int n = in ? BYTES : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(cs_smem(dst)), "l"(src), "n"(BYTES), "r"(n) : "memory");
}
// COUNT consecutive floats of one lane: pieces of 16 bytes (or what there is) whose places in a stage are 128 lanes wide
template <int COUNT>
__device__ __forceinline__ void wk_ring_fill(float* stage, int item, const float* src, bool in, const float* any) {
  constexpr int W = COUNT % 4 == 0 ? 4 : COUNT;
#pragma unroll
  for (int e = 0; e < COUNT; e += W) wk_cp<W * 4>(stage + (item + e) * WK_THREADS + threadIdx.x * W, in ? src + e : any, in);
}
template <int COUNT>
__device__ __forceinline__ void wk_ring_read(float (&f)[COUNT], const float* stage, int item) {
  constexpr int W = COUNT % 4 == 0 ? 4 : COUNT;
#pragma unroll
  for (int e = 0; e < COUNT; e += W) {
    float x[W];
    wk_load<W>(x, stage + (item + e) * WK_THREADS + threadIdx.x * W);
#pragma unroll
    for (int i = 0; i < W; ++i) f[e + i] = x[i];
  }
}

template <int MODE, int N, int MT>
__global__ void __launch_bounds__(WK_THREADS)
walk_kernel(float* __restrict__ o, float* __restrict__ state, const float* __restrict__ qp, int ld_q, const float* __restrict__ wp,
            const float* __restrict__ kp, int ld_k, int qk_group, const float* __restrict__ dec, const float* __restrict__ v, int ld_v,
            const float* __restrict__ v_scale, const float* __restrict__ pairs, const int* __restrict__ cu_q, const int* __restrict__ q_start,
            const int* __restrict__ state_slot, int H, int dk, int dv) {
  using I = WalkItems<MODE, N, MT>;
  constexpr int DKP = 32 * N, COLS = I::cols, LD = I::ld, LDU = I::ldu, ST = I::stages;
  extern __shared__ __align__(16) float wk_smem[];
  float* ring = wk_smem;
  float* xs = ring + I::ring;  // [warp][token][LD]
  float* os = xs + I::xs;      // [2][warp][token][LD]
  float* us = os + I::os;      // [1 or 2][column][LDU]
  pdl_prologue();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int v0 = blockIdx.x * COLS, h = blockIdx.y, r = blockIdx.z;
  const int row_begin = cu_q[r], row_end = cu_q[r + 1];
  const int c0 = wk_first(r, cu_q);
  int c1 = c0 + (row_end - row_begin + WK_TOK - 1) / WK_TOK;
  asm volatile("" : "+r"(c1));  // (a number of chunks that the compiler can see to be above zero has it order the loop for fewer registers)
  if (c1 <= c0) return;
  const int slice = warp * 8 * N;      // the warp's key channels
  const int mine = slice + 2 * N * t;  // the lane's 2 N of them as a product's operand,
  const int mine_n = slice + N * g;    // and its N as an accumulator's columns
  const int tok_u = tid >> 3, col_u = (tid & 7) * 2;  // the (token, two columns) that a thread brings in and adds up
  const size_t head = (size_t)(h / qk_group) * dk;

  auto fetch = [&](int c) {  // (nothing behind the row's last chunk; the group is committed all the same)
    if (c < c1) {
      float* st = ring + (size_t)((c - c0) % ST) * (I::floats * WK_THREADS);
      const int tok0 = row_begin + (c - c0) * WK_TOK;
      const size_t item = (size_t)c * H + h;
      if constexpr (MODE == WALK_HEAD) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int tok = tok0 + j * 8 + g;
          wk_ring_fill<2 * N>(st, I::q + j * 2 * N, qp + (size_t)tok * ld_q + head + mine, tok < row_end, qp);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int tok = tok0 + 4 * t + j;
          wk_ring_fill<N>(st, I::k + j * N, kp + (size_t)tok * ld_k + head + mine_n, tok < row_end, kp);
        }
        const float* d = dec + item * (3 * WK_TOK);
        wk_ring_fill<2>(st, I::last, d + 2 * t, true, dec);
        wk_ring_fill<2>(st, I::last + 2, d + 8 + 2 * t, true, dec);
        wk_ring_fill<4>(st, I::last + 4, d + WK_TOK + 4 * t, true, dec);
        wk_ring_fill<1>(st, I::more, d + 2 * WK_TOK, true, dec);
        const int tok = tok0 + tok_u;
        const bool in = tok < row_end;
        if (v_scale) wk_ring_fill<1>(st, I::more + 1, v_scale + (size_t)tok * H + h, in, v_scale);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int col = v0 + mt * 16 + col_u + e;
            wk_ring_fill<1>(st, I::u + mt * 2 + e, v + (size_t)tok * ld_v + (size_t)h * dv + col, in && col < dv, v);
          }
      } else {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          wk_ring_fill<2 * N>(st, I::q + j * 2 * N, qp + (item * WK_TOK + j * 8 + g) * DKP + mine, true, qp);
          if constexpr (MODE == WALK_DELTA) wk_ring_fill<2 * N>(st, I::w + j * 2 * N, wp + (item * WK_TOK + j * 8 + g) * DKP + mine, true, wp);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) wk_ring_fill<N>(st, I::k + j * N, kp + (item * WK_TOK + 4 * t + j) * DKP + mine_n, true, kp);
        wk_ring_fill<2 * N>(st, I::last, dec + item * DKP + mine, true, dec);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) wk_ring_fill<2>(st, I::u + mt * 2, v + (item * WK_TOK + tok_u) * ld_v + v0 + mt * 16 + col_u, true, v);
      }
      wk_ring_fill<2>(st, I::pair, pairs + (item * WK_TOK + (warp & 1) * 8 + g) * WK_TOK + 4 * t + 2 * (warp >> 1), true, pairs);
    }
    cs_commit();
  };
  // o of the chunk that begins at tok0: the four warps' partial sums
  auto put_out = [&](int tok0, int buf) {
    const int tok = tok0 + tok_u;
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      float x[2] = {0.f, 0.f};
#pragma unroll
      for (int w = 0; w < WK_WARPS; ++w) {
        const float2 y = *reinterpret_cast<const float2*>(os + ((buf * WK_WARPS + w) * WK_TOK + tok_u) * LD + mt * 16 + col_u);
        x[0] += y.x;
        x[1] += y.y;
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int col = v0 + mt * 16 + col_u + e;
        if (tok < row_end && col < dv) o[((size_t)tok * H + h) * dv + col] = x[e];
      }
    }
  };

#pragma unroll
  for (int s = 0; s < ST - 1; ++s) fetch(c0 + s);
  float S[MT][N][4];
  float* slot = state + ((size_t)state_slot[r] * H + h) * (size_t)dv * dk;
  const bool fresh = q_start[r] == 0;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < N; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = v0 + mt * 16 + g + (e >= 2 ? 8 : 0), c = mine + N * (e & 1) + nt;
        S[mt][nt][e] = !fresh && col < dv && c < dk ? slot[(size_t)col * dk + c] : 0.f;
      }

#pragma unroll 1
  for (int c = c0; c < c1; ++c) {
    const int tok0 = row_begin + (c - c0) * WK_TOK, buf = (c - c0) & 1;
    fetch(c + ST - 1);
    cs_wait<ST - 1>();
    const float* st = ring + (size_t)((c - c0) % ST) * (I::floats * WK_THREADS);
    float fu[MT * 2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      if constexpr (MODE == WALK_HEAD) {  // (two pieces of their own)
        float x0[1], x1[1];
        wk_ring_read<1>(x0, st, I::u + 2 * mt);
        wk_ring_read<1>(x1, st, I::u + 2 * mt + 1);
        fu[2 * mt] = x0[0];
        fu[2 * mt + 1] = x1[0];
      } else {
        float x[2];
        wk_ring_read<2>(x, st, I::u + 2 * mt);
        fu[2 * mt] = x[0];
        fu[2 * mt + 1] = x[1];
      }
    }
    if constexpr (MODE == WALK_HEAD) {
      if (v_scale) {
        float x[1];
        wk_ring_read<1>(x, st, I::more + 1);
#pragma unroll
        for (int e = 0; e < MT * 2; ++e) fu[e] *= x[0];
      }
    }
    FragA a[MT][N];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt)
#pragma unroll
      for (int nt = 0; nt < N; ++nt) a[mt][nt] = wk_frag(S[mt][nt][0], S[mt][nt][2], S[mt][nt][1], S[mt][nt][3]);
    // d = the state against the two rows of 2 N channels that a lane holds of q' or W
    auto against = [&](float (&d)[MT][2][4], int item) {
      float rest[MT][2][4] = {};
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) d[mt][j][e] = 0.f;
      float f[2][2 * N];
#pragma unroll
      for (int j = 0; j < 2; ++j) wk_ring_read<2 * N>(f[j], st, item + j * 2 * N);
#pragma unroll
      for (int nt = 0; nt < N; ++nt) {
        Tf32x2 b[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) b[j][e] = wk_split(f[j][N * e + nt]);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int j = 0; j < 2; ++j) wk_part<0>(d[mt][j], rest[mt][j], a[mt][nt], b[j]);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int j = 0; j < 2; ++j) wk_part<1>(d[mt][j], rest[mt][j], a[mt][nt], b[j]);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int j = 0; j < 2; ++j) wk_part<2>(d[mt][j], rest[mt][j], a[mt][nt], b[j]);
      }
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) d[mt][j][e] += rest[mt][j][e];
    };
    float acc[MT][2][4];
    if constexpr (MODE == WALK_DELTA) {
      float x[MT][2][4];
      against(x, I::w);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) xs[(warp * WK_TOK + j * 8 + 2 * t + (e & 1)) * LD + mt * 16 + g + (e >= 2 ? 8 : 0)] = x[mt][j][e];
      __syncthreads();
      float2 y[MT][WK_WARPS];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int w = 0; w < WK_WARPS; ++w) y[mt][w] = *reinterpret_cast<const float2*>(xs + (w * WK_TOK + tok_u) * LD + mt * 16 + col_u);
      against(acc, I::q);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        us[(mt * 16 + col_u) * LDU + tok_u] = fu[2 * mt] - ((y[mt][0].x + y[mt][1].x) + (y[mt][2].x + y[mt][3].x));
        us[(mt * 16 + col_u + 1) * LDU + tok_u] = fu[2 * mt + 1] - ((y[mt][0].y + y[mt][1].y) + (y[mt][2].y + y[mt][3].y));
      }
    } else {
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int e = 0; e < 2; ++e) us[(buf * COLS + mt * 16 + col_u + e) * LDU + tok_u] = fu[2 * mt + e];
      against(acc, I::q);
    }
    __syncthreads();
    // the chunk before: its partial sums are all there (they have two buffers)
    if (c > c0) put_out(tok0 - WK_TOK, buf ^ 1);
    // ---- the state's update, and the chunk's own tokens (a quarter of those products a warp)
    float keep[2 * N], suf[4], total = 1.f;
    if constexpr (MODE == WALK_HEAD) {
      float p0[2], p1[2], x[1];
      wk_ring_read<2>(p0, st, I::last);
      wk_ring_read<2>(p1, st, I::last + 2);
      wk_ring_read<4>(suf, st, I::last + 4);
      wk_ring_read<1>(x, st, I::more);
      total = x[0];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          acc[mt][0][e] *= p0[e & 1];
          acc[mt][1][e] *= p1[e & 1];
        }
    } else {
      wk_ring_read<2 * N>(keep, st, I::last);
    }
    float fp[2];
    wk_ring_read<2>(fp, st, I::pair);
    const Tf32x2 bp[2] = {wk_split(fp[0]), wk_split(fp[1])};
    float rest[MT][N][4] = {};
    FragA au[MT][2];
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      float ua[4], ub[4];
      const float* ut = us + ((MODE == WALK_DELTA ? 0 : buf) * COLS + mt * 16 + g) * LDU + 4 * t;
      wk_load<4>(ua, ut);
      wk_load<4>(ub, ut + 8 * LDU);
#pragma unroll
      for (int s = 0; s < 2; ++s) au[mt][s] = wk_frag(ua[2 * s], ub[2 * s], ua[2 * s + 1], ub[2 * s + 1]);
#pragma unroll
      for (int nt = 0; nt < N; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[mt][nt][e] *= MODE == WALK_HEAD ? total : keep[N * (e & 1) + nt];
    }
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      float fk[2][N];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        wk_ring_read<N>(fk[e], st, I::k + (2 * s + e) * N);
        if constexpr (MODE == WALK_HEAD) {
#pragma unroll
          for (int nt = 0; nt < N; ++nt) fk[e][nt] *= suf[2 * s + e];
        }
      }
      Tf32x2 b[N][2];
#pragma unroll
      for (int nt = 0; nt < N; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) b[nt][e] = wk_split(fk[e][nt]);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < N; ++nt) wk_part<0>(S[mt][nt], rest[mt][nt], au[mt][s], b[nt]);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < N; ++nt) wk_part<1>(S[mt][nt], rest[mt][nt], au[mt][s], b[nt]);
#pragma unroll
      for (int mt = 0; mt < MT; ++mt)
#pragma unroll
        for (int nt = 0; nt < N; ++nt) wk_part<2>(S[mt][nt], rest[mt][nt], au[mt][s], b[nt]);
    }
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      float own[4] = {}, rest_own[4] = {};
      FragA f;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        f.hi[e] = warp >> 1 ? au[mt][1].hi[e] : au[mt][0].hi[e];
        f.lo[e] = warp >> 1 ? au[mt][1].lo[e] : au[mt][0].lo[e];
      }
      wk_part<0>(own, rest_own, f, bp);
      wk_part<1>(own, rest_own, f, bp);
      wk_part<2>(own, rest_own, f, bp);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        own[e] += rest_own[e];
        acc[mt][0][e] += warp & 1 ? 0.f : own[e];
        acc[mt][1][e] += warp & 1 ? own[e] : 0.f;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          os[((buf * WK_WARPS + warp) * WK_TOK + j * 8 + 2 * t + (e & 1)) * LD + mt * 16 + g + (e >= 2 ? 8 : 0)] = acc[mt][j][e];
#pragma unroll
      for (int nt = 0; nt < N; ++nt)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[mt][nt][e] += rest[mt][nt][e];
    }
  }
  __syncthreads();
  put_out(row_begin + (c1 - 1 - c0) * WK_TOK, (c1 - 1 - c0) & 1);
#pragma unroll
  for (int mt = 0; mt < MT; ++mt)
#pragma unroll
    for (int nt = 0; nt < N; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int col = v0 + mt * 16 + g + (e >= 2 ? 8 : 0), c = mine + N * (e & 1) + nt;
        if (col < dv && c < dk) slot[(size_t)col * dk + c] = S[mt][nt][e];
      }
}

// ---------------------------------------------------------------- one decay per head: the pairs of a chunk's tokens
// grid (chunks, groups of heads that share q and k). pairs[chunk, h, i, j] = q_scale (q_i . k_j) a_(j+1) .. a_i for j <= i, else 0;
// decays[chunk, h]: q_scale a_first .. a_i of 16 tokens, then a_(i+1) .. a_last of them, then a_first .. a_last. Tokens behind the row's
// end have decay 1.
template <int DK>
__global__ void __launch_bounds__(WK_THREADS)
walk_head_kernel(float* __restrict__ pairs, float* __restrict__ decays, const float* __restrict__ q, int ld_q, const float* __restrict__ k,
                 int ld_k, int qk_group, const float* __restrict__ decay, int ld_decay, const int* __restrict__ cu_q, int num_rows, int H,
                 float q_scale) {
  __shared__ __align__(16) float qs[WK_TOK][DK + 4], ks[WK_TOK][DK + 4];
  __shared__ float dot[WK_TOK][WK_TOK + 1], as[WK_TOK][33];
  pdl_prologue();
  const int chunk = blockIdx.x, grp = blockIdx.y;
  const int2 at = wk_at(chunk, cu_q, num_rows);
  if (at.x < 0) return;
  const int t0 = at.y, n = min(WK_TOK, cu_q[at.x + 1] - t0);
  const int tid = threadIdx.x;
#pragma unroll
  for (int e = 0; e < WK_TOK * DK / 4 / WK_THREADS; ++e) {
    const int idx = e * WK_THREADS + tid, i = idx / (DK / 4), c = (idx % (DK / 4)) * 4;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (i < n) {
      a = *reinterpret_cast<const float4*>(q + (size_t)(t0 + i) * ld_q + (size_t)grp * DK + c);
      b = *reinterpret_cast<const float4*>(k + (size_t)(t0 + i) * ld_k + (size_t)grp * DK + c);
    }
    *reinterpret_cast<float4*>(&qs[i][c]) = a;
    *reinterpret_cast<float4*>(&ks[i][c]) = b;
  }
  __syncthreads();
  {  // a thread's two dot products: token i with j and with j + 8
    const int i = tid >> 3, j = tid & 7;
    float s0[4] = {}, s1[4] = {};
#pragma unroll 4
    for (int c = 0; c < DK; c += 4) {
      const float4 a = *reinterpret_cast<const float4*>(&qs[i][c]), b = *reinterpret_cast<const float4*>(&ks[j][c]),
                   d = *reinterpret_cast<const float4*>(&ks[j + 8][c]);
      s0[0] = fmaf(a.x, b.x, s0[0]); s0[1] = fmaf(a.y, b.y, s0[1]); s0[2] = fmaf(a.z, b.z, s0[2]); s0[3] = fmaf(a.w, b.w, s0[3]);
      s1[0] = fmaf(a.x, d.x, s1[0]); s1[1] = fmaf(a.y, d.y, s1[1]); s1[2] = fmaf(a.z, d.z, s1[2]); s1[3] = fmaf(a.w, d.w, s1[3]);
    }
    dot[i][j] = ((s0[0] + s0[1]) + (s0[2] + s0[3])) * q_scale;
    dot[i][j + 8] = ((s1[0] + s1[1]) + (s1[2] + s1[3])) * q_scale;
  }
  for (int h0 = 0; h0 < qk_group; h0 += 32) {
    const int heads = min(32, qk_group - h0), first = grp * qk_group + h0;
    __syncthreads();
    for (int idx = tid; idx < WK_TOK * heads; idx += WK_THREADS) {
      const int i = idx / heads, e = idx - i * heads;
      as[i][e] = i < n ? decay[(size_t)(t0 + i) * ld_decay + first + e] : 1.f;
    }
    __syncthreads();
    for (int idx = tid; idx < heads * WK_TOK; idx += WK_THREADS) {  // (head, token j): the pairs that j's write is in, running over i
      const int e = idx >> 4, j = idx & 15;
      float* out = pairs + ((size_t)chunk * H + first + e) * (WK_TOK * WK_TOK) + j;
      float run = 1.f, before = 1.f;
#pragma unroll
      for (int i = 0; i < WK_TOK; ++i) {
        const float a = as[i][e];
        if (i > j) run *= a;
        if (i <= j) before *= a;
        out[i * WK_TOK] = i >= j ? dot[i][j] * run : 0.f;
      }
      float* dec = decays + ((size_t)chunk * H + first + e) * (3 * WK_TOK);
      dec[j] = before * q_scale;
      dec[WK_TOK + j] = run;
      if (j == WK_TOK - 1) dec[2 * WK_TOK] = before;
    }
  }
}

// Dynamic shared memory beyond 48 KB is asked for once per kernel. Not a dependent launch: CTAs that become resident while the kernel
// before drains gather on the SMs that are free first, and two chains on one SM walk at half the rate (16 heads of 64 x 64 with the delta
// rule over 2,048 tokens, both kernels: 140 us against 188; 32 heads of 128 x 64 with a decay per head 134 against 238).
#define MS_WALK_LAUNCH(MODE, N, MT, grid, ...)                                                                            \
  do {                                                                                                                    \
    auto walk = walk_kernel<MODE, N, MT>;                                                                                 \
    constexpr size_t bytes = WalkItems<MODE, N, MT>::bytes;                                                               \
    static const cudaError_t asked = cudaFuncSetAttribute(walk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes); \
    MS_CHECK_CUDA(asked);                                                                                                 \
    MS_LAUNCH_APART(walk, grid, WK_THREADS, bytes, stream, __VA_ARGS__);                                                  \
  } while (0)

template <typename TIn, typename TZ, bool DELTA, int N>
int launch_walk(float* o, float* state, const TIn* q, int ld_q, const TIn* k, int ld_k, int qk_group, const TIn* v, int ld_v, const TZ* z,
                int ld_z, const float* z_bias, const float* decay_coef, float z_sign, const TZ* beta, int ld_beta, const float* v_scale,
                float* scratch, const int* cu_q, const int* q_start, const int* state_slot, int num_rows, int max_chunks, int H, int dk, int dv, float q_scale, cudaStream_t stream) {
  constexpr int DKP = 32 * N;
  const size_t items = (size_t)max_chunks * H;
  const int dvp = ceil_div(dv, WK_COLS) * WK_COLS;
  float* qp = scratch;
  float* kp = qp + items * WK_TOK * DKP;
  float* last = kp + items * WK_TOK * DKP;
  float* pairs = last + items * DKP;
  float* u0 = pairs + items * WK_TOK * WK_TOK;
  float* wp = u0 + items * WK_TOK * dvp;
  auto prepare = walk_prepare_kernel<TIn, TZ, DELTA, N>;
  MS_LAUNCH(prepare, dim3(max_chunks, H), WK_THREADS, 0, stream, wp, qp, kp, last, u0, pairs, q, ld_q, k, ld_k, qk_group, v, ld_v, z, ld_z, z_bias,
            decay_coef, z_sign, beta, ld_beta, v_scale, cu_q, num_rows, H, dk, dv, dvp, q_scale);
  MS_WALK_LAUNCH(DELTA ? WALK_DELTA : WALK_CHANNEL, N, 1, dim3(dvp / WK_COLS, H, num_rows), o, state, qp, DKP, wp, kp, DKP, 1, last, u0, dvp,
                 (const float*)nullptr, pairs, cu_q, q_start, state_slot, H, dk, dv);
  return 0;
}

template <typename TIn, typename TZ, typename... Args>
int launch_walk_for(int delta, int dk, Args... args) {
#define MS_WALK(D)                                            \
  do {                                                        \
    if (dk <= 32) return launch_walk<TIn, TZ, D, 1>(args...); \
    if (dk <= 64) return launch_walk<TIn, TZ, D, 2>(args...); \
    return launch_walk<TIn, TZ, D, 4>(args...);               \
  } while (0)
  if (delta) MS_WALK(true);
  MS_WALK(false);
#undef MS_WALK
}

template <int N>
int launch_walk_head(float* o, float* state, const float* q, int ld_q, const float* k, int ld_k, int qk_group, const float* v, int ld_v,
                     const float* decay, int ld_decay, const float* v_scale, float* scratch, const int* cu_q, const int* q_start,
                     const int* state_slot, int num_rows, int max_chunks, int H, int dv, float q_scale, cudaStream_t stream) {
  constexpr int DK = 32 * N;
  static int sm_count = 0;
  if (sm_count == 0) {
    int dev = 0;
    MS_CHECK_CUDA(cudaGetDevice(&dev));
    MS_CHECK_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
  }
  float* pairs = scratch;
  float* decays = pairs + (size_t)max_chunks * H * WK_TOK * WK_TOK;
  auto prepare = walk_head_kernel<DK>;
  MS_LAUNCH(prepare, dim3(max_chunks, H / qk_group), WK_THREADS, 0, stream, pairs, decays, q, ld_q, k, ld_k, qk_group, decay, ld_decay, cu_q,
            num_rows, H, q_scale);
  // 32 value columns a CTA share what they load and split of q and k, where that leaves two CTAs an SM
  if ((long long)num_rows * H * ceil_div(dv, 2 * WK_COLS) >= 2LL * sm_count)
    MS_WALK_LAUNCH(WALK_HEAD, N, 2, dim3(ceil_div(dv, WK_COLS * 2), H, num_rows), o, state, q, ld_q, (const float*)nullptr, k, ld_k, qk_group, decays, v,
                   ld_v, v_scale, pairs, cu_q, q_start, state_slot, H, DK, dv);
  else
    MS_WALK_LAUNCH(WALK_HEAD, N, 1, dim3(ceil_div(dv, WK_COLS), H, num_rows), o, state, q, ld_q, (const float*)nullptr, k, ld_k, qk_group, decays, v,
                   ld_v, v_scale, pairs, cu_q, q_start, state_slot, H, DK, dv);
  return 0;
}

}  // namespace ms

using namespace ms;

// The most chunks that a step of so many tokens in so many rows can have.
static inline int walk_max(int tokens, int rows) { return tokens / WK_TOK + rows; }

// Floats of scratch for a step of so many tokens in so many rows. per_head: one decay per head.
MS_EXPORT long long ms_walk_scratch(int tokens, int rows, int H, int dk, int dv, int delta, int per_head) {
  const long long items = (long long)walk_max(tokens, rows) * H, dkp = dk <= 32 ? 32 : dk <= 64 ? 64 : 128;
  if (per_head) return items * (WK_TOK * WK_TOK + 3 * WK_TOK);
  return items * (WK_TOK * dkp * (delta ? 3 : 2) + dkp + WK_TOK * WK_TOK + (long long)WK_TOK * (ceil_div(dv, WK_COLS) * WK_COLS));
}

// The decay rule (delta 0) or the delta rule with a decay per key channel; operands as ms_decay_scan's, dk up to 128. o [T, H, dv] float32.
MS_EXPORT int ms_walk_scan(float* o, float* state, const void* q, int ld_q, const void* k, int ld_k, int qk_group, const void* v, int ld_v,
                           const void* z, int ld_z, const float* z_bias, const float* decay_coef, float z_sign, const void* beta, int ld_beta,
                           const float* v_scale, float* scratch, const int* cu_q, const int* q_start, const int* state_slot,
                           int num_tokens, int num_rows, int H, int dk, int dv, float q_scale, int delta, int in_dtype, int z_dtype,
                           cudaStream_t stream) {
  if (num_rows == 0 || num_tokens == 0) return 0;
  MS_CHECK_ARG(dk >= 1 && dk <= 128 && dv >= 1 && H >= 1 && H <= 65535 && num_rows <= 65535, "walk_scan: %d heads of %d x %d, %d rows", H, dk, dv, num_rows);
  MS_CHECK_ARG(qk_group > 0 && H % qk_group == 0, "walk_scan: %d heads are not a multiple of the group of %d", H, qk_group);
  MS_CHECK_ARG(!delta || beta != nullptr, "walk_scan: the delta rule needs beta");
  MS_CHECK_ARG((uintptr_t)scratch % 16 == 0, "walk_scan: scratch must start on 16 bytes");
  const int max_chunks = walk_max(num_tokens, num_rows);
#define MS_WALK(TIN, TZZ)                                                                                                                      \
  return launch_walk_for<TIN, TZZ>(delta, dk, o, state, (const TIN*)q, ld_q, (const TIN*)k, ld_k, qk_group, (const TIN*)v, ld_v, (const TZZ*)z, ld_z, \
                                   z_bias, decay_coef, z_sign, (const TZZ*)beta, ld_beta, v_scale, scratch, cu_q, q_start,      \
                                   state_slot, num_rows, max_chunks, H, dk, dv, q_scale, stream)
  if (in_dtype == MS_F32 && z_dtype == MS_F32) MS_WALK(float, float);
  if (in_dtype == MS_F32 && z_dtype == MS_BF16) MS_WALK(float, __nv_bfloat16);
  if (in_dtype == MS_BF16 && z_dtype == MS_F32) MS_WALK(__nv_bfloat16, float);
  if (in_dtype == MS_BF16 && z_dtype == MS_BF16) MS_WALK(__nv_bfloat16, __nv_bfloat16);
#undef MS_WALK
  return ms::fail("walk_scan: unsupported dtypes (%d, %d)", in_dtype, z_dtype);
}

// The decay rule with one decay per head ([T, ld_decay] float32): q, k, v float32, dk 32, 64 or 128, rows of q and k that start on 16
// bytes.
MS_EXPORT int ms_walk_scan_head(float* o, float* state, const float* q, int ld_q, const float* k, int ld_k, int qk_group, const float* v, int ld_v,
                                const float* decay, int ld_decay, const float* v_scale, float* scratch, const int* cu_q, const int* q_start,
                                const int* state_slot, int num_tokens, int num_rows, int H, int dk, int dv, float q_scale, cudaStream_t stream) {
  if (num_rows == 0 || num_tokens == 0) return 0;
  MS_CHECK_ARG((dk == 32 || dk == 64 || dk == 128) && dv >= 1 && H >= 1 && H <= 65535 && num_rows <= 65535, "walk_scan_head: %d heads of %d x %d", H, dk, dv);
  MS_CHECK_ARG(qk_group > 0 && H % qk_group == 0, "walk_scan_head: %d heads are not a multiple of the group of %d", H, qk_group);
  MS_CHECK_ARG((uintptr_t)q % 16 == 0 && (uintptr_t)k % 16 == 0 && ld_q % 4 == 0 && ld_k % 4 == 0 && (uintptr_t)scratch % 16 == 0,
               "walk_scan_head: rows of q and k must start on 16 bytes");
  const int max_chunks = walk_max(num_tokens, num_rows);
#define MS_WALK(N)                                                                                                                            \
  return launch_walk_head<N>(o, state, q, ld_q, k, ld_k, qk_group, v, ld_v, decay, ld_decay, v_scale, scratch, cu_q, q_start, \
                             state_slot, num_rows, max_chunks, H, dv, q_scale, stream)
  if (dk == 32) MS_WALK(1);
  if (dk == 64) MS_WALK(2);
  MS_WALK(4);
#undef MS_WALK
}
