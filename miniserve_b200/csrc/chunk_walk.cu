// The recurrences of ``recurrence.cu`` over a prompt by chunks of 16 tokens, in float32; the decay rule over long rows goes to ``tile_walk.cu``.
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
// (The triangular system of a chunk: the WY form of products of Householder-like factors, C. Bischof and C. Van Loan, 1987, as chunked
// linear recurrences use it.)
//
// The first kernel works out, for all chunks at once, what does not need the state: W, q' = G q, k' = D_(last, .) k, U0, P.
// The second walks a row's chunks in order, a warp per 4 value columns: the products of a chunk against the state that stays in registers.
//
// Accuracy: every sum is made of float32 multiply-adds that round to nearest, as the token-by-token walk's; products of decays, the
// last steps of the pairs' sums and the triangular system are worked out in 64 bits and rounded once. (A running product of 16 decays just
// below one is rounded down every time: in 32 bits the state of a slowly decaying head comes out three times as far off as the walk's.
// Tensor cores are further off too, factors as two tf32 numbers: 1.3 to 2.3 times the walk's errors over a few tokens, and growing with the
// row where a state lasts, 24 times at 8,192 tokens: their sums are not rounded to nearest.) Against 64-bit sums
// outputs and states are no further off than the walk's: root mean squares of the errors over 2,048 tokens 0.75 to 1.0 of the walk's
// (outputs) and 0.7 to 1.1 (states: few independent numbers), decays from 0.02 to 1; 0.27 to 0.57 with the delta rule and no decay, 1.2 where
// that rule has fewer than 16 key channels, fewer than a chunk has tokens.
// A token sees nothing of the tokens behind it, whatever they hold: a value that is not finite reaches its own token and the later
// ones. (With one decay per head the sums against the state are scaled behind the sum: a state within q's size of the largest float
// overflows.)
//
// What bounds it: the walk is a chain of tokens / 16 steps, each the products against W, an exchange among the 16 lanes of a column
// and the state's update; the token-by-token walk is a chain of `tokens` steps of two lane-group sums each.
#include <cfloat>

#include "chunk_mma.cuh"
#include "float_pairs.cuh"
#include "tile_walk.cuh"

namespace ms {

constexpr int WK_TOK = 16, WK_THREADS = 128, WK_COLS = 16;  // (WK_THREADS: of the kernels ahead of the walk; WK_COLS: what u0 is padded to)
constexpr int WK_CHAIN = 2, WK_OUT = 4, WK_FETCH = 2, WK_OWN = 8;  // warps of the walk's chain, of its outputs, of its copies; an output warp's tokens
enum WalkMode : int { WALK_CHANNEL = 0, WALK_DELTA = 1, WALK_HEAD = 2 };

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
// over the channels of each (two channels an instruction), lets their keys decay from j on, and adds up over the lanes at the end (28
// exchanges for four tokens). The sum over the lanes, products of decays and the triangular system in 64 bits (above).
// With the delta rule the triangular system is a chain of 16 steps in 64 bits, in which a CTA's warps wait for one another: six CTAs an SM (80
// registers a thread, 24 to 64 bytes of them spilled) cover it better than four. 2,048 tokens, both kernels: 16 heads of 64 x 64 139.9 -> 136.3
// us, 32 heads 225.7 -> 209.8. Without it nothing waits so long, and six measured the same as four (108.2). Operands come in fours where rows
// start on whole fours, all of a thread's loads ahead of its work: 2,048 tokens of 16 heads 32.0 us, 37.8 one by one.
template <typename TIn, typename TZ, bool DELTA, int N>
__global__ void __launch_bounds__(WK_THREADS, DELTA ? 6 : 4)
walk_prepare_kernel(float* __restrict__ w_out, float* __restrict__ q_out, float* __restrict__ k_out, float* __restrict__ last_out,
                    float* __restrict__ u0_out, float* __restrict__ pairs, const TIn* __restrict__ q, int ld_q, const TIn* __restrict__ k,
                    int ld_k, int qk_group, const TIn* __restrict__ v, int ld_v, const TZ* __restrict__ z, int ld_z,
                    const float* __restrict__ z_bias, const float* __restrict__ decay_coef, float z_sign, const TZ* __restrict__ beta,
                    int ld_beta, const float* __restrict__ v_scale, const int* __restrict__ cu_q, int num_rows, int H, int dk, int dv, int dvp,
                    float q_scale) {
  constexpr int DKP = 32 * N;
  __shared__ __align__(16) float qs[WK_TOK][DKP], ks[WK_TOK][DKP], ds[WK_TOK][DKP];
  __shared__ __align__(16) double am[DELTA ? WK_TOK : 1][WK_TOK];  // A, a column j in am[j]
  __shared__ float bs[WK_TOK], vsc[WK_TOK];
  pdl_prologue(q, k, v, z, z_bias, decay_coef, beta, v_scale, cu_q);
  const int chunk = blockIdx.x, h = blockIdx.y;
  const int2 at = wk_at(chunk, cu_q, num_rows);
  if (at.x < 0) return;
  const int t0 = at.y, n = min(WK_TOK, cu_q[at.x + 1] - t0);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t qk_at = (size_t)(h / qk_group) * dk;
  const float coef = decay_coef[h];
  auto decay = [&](float logit, int c) { return expf(-coef * softplusf(z_sign * (logit + z_bias[(size_t)h * dk + c]))); };
  if (dk % 4 == 0 && in_fours(q, ld_q) && in_fours(k, ld_k) && in_fours(z, ld_z)) {
    constexpr int EACH = WK_TOK * DKP / 4 / WK_THREADS, AT_ONCE = EACH < 2 ? EACH : 2;
#pragma unroll 1
    for (int e0 = 0; e0 < EACH; e0 += AT_ONCE) {
      float4 fq[AT_ONCE], fk[AT_ONCE], fd[AT_ONCE];
#pragma unroll
      for (int e = 0; e < AT_ONCE; ++e) {  // all of it is asked for before the first is worked on
        const int idx = (e0 + e) * WK_THREADS + tid, i = idx / (DKP / 4), c = (idx % (DKP / 4)) * 4;
        const bool in = i < n && c < dk;
        const size_t t = in ? (size_t)(t0 + i) : (size_t)t0;
        const int cc = in ? c : 0;
        fq[e] = load4(q + t * ld_q + qk_at + cc);
        fk[e] = load4(k + t * ld_k + qk_at + cc);
        fd[e] = load4(z + t * ld_z + (size_t)h * dk + cc);
      }
#pragma unroll
      for (int e = 0; e < AT_ONCE; ++e) {
        const int idx = (e0 + e) * WK_THREADS + tid, i = idx / (DKP / 4), c = (idx % (DKP / 4)) * 4;
        const bool in = i < n && c < dk;
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(&qs[i][c]) = in ? make_float4(fq[e].x * q_scale, fq[e].y * q_scale, fq[e].z * q_scale, fq[e].w * q_scale) : none;
        *reinterpret_cast<float4*>(&ks[i][c]) = in ? fk[e] : none;
        *reinterpret_cast<float4*>(&ds[i][c]) =
            in ? make_float4(decay(fd[e].x, c), decay(fd[e].y, c + 1), decay(fd[e].z, c + 2), decay(fd[e].w, c + 3)) : make_float4(1.f, 1.f, 1.f, 1.f);
      }
    }
  } else {
#pragma unroll 4
    for (int e = 0; e < WK_TOK * DKP / WK_THREADS; ++e) {
      const int idx = e * WK_THREADS + tid, i = idx / DKP, c = idx % DKP;
      float fq = 0.f, fk = 0.f, fd = 1.f;
      if (i < n && c < dk) {
        const size_t t = (size_t)(t0 + i);
        fq = Elem<TIn>::load(q + t * ld_q + qk_at + c) * q_scale;
        fk = Elem<TIn>::load(k + t * ld_k + qk_at + c);
        fd = decay(Elem<TZ>::load(z + t * ld_z + (size_t)h * dk + c), c);
      }
      qs[i][c] = fq;
      ks[i][c] = fk;
      ds[i][c] = fd;
    }
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
    f2 p[2 * N] = {};
    double val[32];
#pragma unroll
    for (int i = 0; i < WK_TOK; ++i) {
      f2 a = 0ull, b = 0ull;
#pragma unroll
      for (int m = 0; m < N; ++m) {
        const ulonglong2 fk = *reinterpret_cast<const ulonglong2*>(&ks[i][cl * 4 + 32 * m]);
        const ulonglong2 fq = *reinterpret_cast<const ulonglong2*>(&qs[i][cl * 4 + 32 * m]);
        const ulonglong2 fd = *reinterpret_cast<const ulonglong2*>(&ds[i][cl * 4 + 32 * m]);
        p[2 * m] = i == j ? fk.x : f2_mul(p[2 * m], fd.x);  // (nothing ahead of token j)
        p[2 * m + 1] = i == j ? fk.y : f2_mul(p[2 * m + 1], fd.y);
        if (DELTA) {
          f2_fma(a, fk.x, p[2 * m]);
          f2_fma(a, fk.y, p[2 * m + 1]);
        }
        f2_fma(b, fq.x, p[2 * m]);
        f2_fma(b, fq.y, p[2 * m + 1]);
      }
      val[i] = f2_sum(a);
      val[16 + i] = f2_sum(b);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const bool up = cl & o;
#pragma unroll
      for (int i = 0; i < 4 * o; ++i) {
        const double send = up ? val[i] : val[i + 4 * o], keep = up ? val[i + 4 * o] : val[i];
        val[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const int i0 = 4 * (cl & 3);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = i0 + e;
      if (cl >= 4) pairs[(item * WK_TOK + i) * WK_TOK + j] = i >= j ? (float)val[e] : 0.f;
      else if (DELTA) am[j][i] = i > j ? val[e] * (double)bs[i] : 0.0;
    }
  }
  if (DELTA) __syncthreads();
  // a thread per key channel: q', W (forward substitution), k', the decay of the whole chunk; and one per value column: U0 likewise
#pragma unroll 1
  for (int c = tid; c < DKP + dvp; c += WK_THREADS) {
    double x[WK_TOK];
    if (c < DKP) {
      double passed = 1.0;
#pragma unroll
      for (int i = 0; i < WK_TOK; ++i) {
        passed *= (double)ds[i][c];
        q_out[(item * WK_TOK + i) * DKP + c] = (float)(passed * (double)qs[i][c]);
        x[i] = passed * (double)ks[i][c];
      }
      last_out[item * DKP + c] = (float)passed;
      double behind = 1.0;
#pragma unroll
      for (int i = WK_TOK - 1; i >= 0; --i) {
        k_out[(item * WK_TOK + i) * DKP + c] = (float)((double)ks[i][c] * behind);
        behind *= (double)ds[i][c];
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
    if (DELTA) {
      asm volatile("" ::: "memory");  // (A is read again for every column: kept over the columns it takes 240 registers)
#pragma unroll
      for (int i = 0; i < WK_TOK; ++i) x[i] *= (double)bs[i];
#pragma unroll
      for (int j = 0; j + 1 < WK_TOK; ++j)
#pragma unroll
        for (int i = j + 1; i < WK_TOK; ++i) x[i] = fma(-am[j][i], x[j], x[i]);
    }
#pragma unroll
    for (int i = 0; i < WK_TOK; ++i) out[(size_t)i * step] = (float)x[i];
  }
}

// ---------------------------------------------------------------- the walk over a row's chunks
// grid (value column tiles, H, rows), 4 C columns a CTA. A column's DKP key channels lie with 16 lanes, 2 N each, in registers; a lane has
// C columns, a warp 2 C: an operand read from shared memory makes products for all of them. A product against 16 tokens' vectors is 16 sums a
// lane and column, folded over the 16 lanes all at once (lane l keeps token l's).
// The first warps carry the chain (W, u, the state behind the chunk); the others, beside them on the SM's other schedulers, make the
// outputs from the state that the chain left in shared memory, eight tokens a warp, the chunk's own tokens' part one chunk later, when u is
// there. One barrier a chunk.
// Channel mode and the delta rule read what walk_prepare_kernel left (qp, wp, kp, dec, u0, pairs). Head mode reads q, k and v
// themselves, and the pairs and decays of walk_head_kernel.
// A chunk's operands come through a ring in shared memory (cp.async), two or three chunks ahead: a chunk takes less time than a load from L2.
template <int MODE, int N, int C>
struct WalkStage {  // floats
  static constexpr int dkp = 32 * N, cols = 2 * C * WK_CHAIN, ldp = WK_TOK + 4, decays = MODE == WALK_HEAD ? 3 * WK_TOK : dkp;
  static constexpr int q = 0, k = WK_TOK * dkp, w = 2 * WK_TOK * dkp, last = w + (MODE == WALK_DELTA ? WK_TOK * dkp : 0), pair = last + decays,
                       u = pair + WK_TOK * ldp, scale = u + WK_TOK * cols, floats = scale + (MODE == WALK_HEAD ? WK_TOK : 0);
  static constexpr int stages = C == 4 ? 3 : 4, states = 2 * cols * dkp, us = 2 * cols * WK_TOK, decayed = MODE == WALK_HEAD ? cols * WK_TOK : 0;
  static constexpr size_t bytes = (size_t)(stages * floats + states + us + decayed) * 4;
};

// BYTES from global memory into shared memory, zeros where not `in`
template <int BYTES>
__device__ __forceinline__ void wk_cp(float* dst, const float* src, bool in) {
  const int n = in ? BYTES : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(cs_smem(dst)), "l"(src), "n"(BYTES), "r"(n) : "memory");
}

// a lane's 2 N channels of a row of DKP in shared memory: two for N = 1, else fours that are 64 apart
template <int N>
__device__ __forceinline__ void wk_row(f2 (&x)[N], const float* row, int l) {
  if constexpr (N == 1) {
    x[0] = *reinterpret_cast<const f2*>(row + 2 * l);
  } else {
#pragma unroll
    for (int m = 0; m < N / 2; ++m) {
      const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(row + 64 * m + 4 * l);
      x[2 * m] = y.x;
      x[2 * m + 1] = y.y;
    }
  }
}
template <int N>
__device__ __forceinline__ int wk_channel(int l, int pair, int half) {
  return N == 1 ? 2 * l + half : 64 * (pair >> 1) + 4 * l + 2 * (pair & 1) + half;
}

// The products of a lane's columns with ROWS rows, summed over the column's lanes: lane l comes back with row l's. (Eight rows: lanes l and l ^ 8
// with two parts of row l & 7's.) A lane takes row i ^ l as its i-th, so that what it keeps of an exchange is always the first half of its sums.
template <int N, int C, int ROWS>
__device__ __forceinline__ void wk_against(float (&d)[C], const f2 (&S)[C][N], const float* rows, int l) {
  float val[C][ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; ++i) {
    f2 x[N], a[C] = {};
    wk_row<N>(x, rows + (i ^ (l & (ROWS - 1))) * (32 * N), l);
#pragma unroll
    for (int p = 0; p < N; ++p)
#pragma unroll
      for (int c = 0; c < C; ++c) f2_fma(a[c], S[c][p], x[p]);
#pragma unroll
    for (int c = 0; c < C; ++c) val[c][i] = f2_sum(a[c]);
  }
#pragma unroll
  for (int o = ROWS / 2; o > 0; o >>= 1)
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int i = 0; i < o; ++i) val[c][i] += __shfl_xor_sync(0xffffffffu, val[c][i + o], o);
#pragma unroll
  for (int c = 0; c < C; ++c) d[c] = val[c][0];
}

template <int MODE, int N, int C, bool APART>
__global__ void __launch_bounds__((WK_CHAIN + WK_OUT + (APART ? WK_FETCH : 0)) * 32, C == 4 ? 2 : 1)
walk_kernel(float* __restrict__ o, float* __restrict__ state, const float* __restrict__ qp, int ld_q, const float* __restrict__ wp,
            const float* __restrict__ kp, int ld_k, int qk_group, const float* __restrict__ dec, const float* __restrict__ v, int ld_v,
            const float* __restrict__ v_scale, const float* __restrict__ pairs, const int* __restrict__ cu_q, const int* __restrict__ q_start,
            const int* __restrict__ state_slot, int H, int dk, int dv) {
  using I = WalkStage<MODE, N, C>;
  constexpr int DKP = I::dkp, COLS = I::cols, ST = I::stages, FETCHERS = (APART ? WK_FETCH : WK_OUT) * 32;
  extern __shared__ __align__(16) float wk_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, l = lane & 15;
  const int v0 = blockIdx.x * COLS, h = blockIdx.y, r = blockIdx.z;
  const int row_begin = cu_q[r], row_end = cu_q[r + 1];
  const int c0 = wk_first(r, cu_q);
  const int c1 = c0 + (row_end - row_begin + WK_TOK - 1) / WK_TOK;
  if (c1 <= c0) return;
  const bool chain = warp < WK_CHAIN;
  const int mine = (warp % WK_CHAIN) * (2 * C) + (lane >> 4) * C;  // the lane's first column of the CTA's
  float* states = wk_smem + ST * I::floats + mine * DKP;                  // [2][COLS][DKP]: the state ahead of a chunk
  float* us = wk_smem + ST * I::floats + I::states + mine * WK_TOK;       // [2][COLS][16]: u of a chunk
  float* decayed = wk_smem + ST * I::floats + I::states + I::us + mine * WK_TOK;  // (head mode) [COLS][16]: u decayed to the chunk's end

  const int ft = tid - (APART ? WK_CHAIN + WK_OUT : WK_CHAIN) * 32;  // (APART: warps that only fetch; else the output warps do)
  auto fetch = [&](int c) {  // (nothing behind the row's last chunk; the group is committed all the same)
    if (c < c1) {
      float* st = wk_smem + (size_t)((c - c0) % ST) * I::floats;
      const int tok0 = row_begin + (c - c0) * WK_TOK;
      const size_t item = (size_t)c * H + h;
      if constexpr (MODE == WALK_HEAD) {
        const size_t head = (size_t)(h / qk_group) * dk;
#pragma unroll
        for (int idx = ft; idx < WK_TOK * DKP / 4; idx += FETCHERS) {
          const int i = idx / (DKP / 4), ch = (idx % (DKP / 4)) * 4, tok = tok0 + i;
          const bool in = tok < row_end;
          wk_cp<16>(st + I::q + i * DKP + ch, in ? qp + (size_t)tok * ld_q + head + ch : qp, in);
          wk_cp<16>(st + I::k + i * DKP + ch, in ? kp + (size_t)tok * ld_k + head + ch : kp, in);
        }
        if (ft < 3 * WK_TOK / 4) wk_cp<16>(st + I::last + ft * 4, dec + item * (3 * WK_TOK) + ft * 4, true);
#pragma unroll
        for (int idx = ft; idx < WK_TOK * COLS; idx += FETCHERS) {
          const int i = idx / COLS, col = v0 + idx % COLS, tok = tok0 + i;
          const bool in = tok < row_end && col < dv;
          wk_cp<4>(st + I::u + idx, in ? v + (size_t)tok * ld_v + (size_t)h * dv + col : v, in);
        }
        if (v_scale && ft < WK_TOK) {
          const bool in = tok0 + ft < row_end;
          wk_cp<4>(st + I::scale + ft, in ? v_scale + (size_t)(tok0 + ft) * H + h : v_scale, in);
        }
      } else {
#pragma unroll
        for (int idx = ft; idx < WK_TOK * DKP / 4; idx += FETCHERS) {
          const int at = idx * 4;
          const size_t from = item * (WK_TOK * DKP) + at;
          wk_cp<16>(st + I::q + at, qp + from, true);
          wk_cp<16>(st + I::k + at, kp + from, true);
          if constexpr (MODE == WALK_DELTA) wk_cp<16>(st + I::w + at, wp + from, true);
        }
        if (ft < DKP / 4) wk_cp<16>(st + I::last + ft * 4, dec + item * DKP + ft * 4, true);
        for (int idx = ft; idx < WK_TOK * COLS / 4; idx += FETCHERS) {
          const int i = idx / (COLS / 4), col = (idx % (COLS / 4)) * 4;
          wk_cp<16>(st + I::u + i * COLS + col, v + (item * WK_TOK + i) * ld_v + v0 + col, true);
        }
      }
      if (ft < WK_TOK * WK_TOK / 4) wk_cp<16>(st + I::pair + (ft >> 2) * I::ldp + (ft & 3) * 4, pairs + item * (WK_TOK * WK_TOK) + ft * 4, true);
    }
    cs_commit();
  };

  if (APART ? warp >= WK_CHAIN + WK_OUT : !chain) {
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) fetch(c0 + s);
  }
  if (APART && warp >= WK_CHAIN + WK_OUT) {
#pragma unroll 1
    for (int c = c0; c <= c1; ++c) {
      cs_wait<ST - 2>();
      __syncthreads();  // (the one below)
      if (c < c1) fetch(c + ST - 1);
    }
    return;
  }
  f2 S[C][N];
  float* slot = state + ((size_t)state_slot[r] * H + h) * (size_t)dv * dk;
  // the chain's state into shared memory for the outputs, and from there
  auto leave = [&](int buf) {
#pragma unroll
    for (int e = 0; e < C; ++e)
#pragma unroll
      for (int p = 0; p < N; p += 2) {
        float* to = states + (buf * COLS + e) * DKP + wk_channel<N>(l, p, 0);
        if constexpr (N == 1) *reinterpret_cast<f2*>(to) = S[e][0];
        else *reinterpret_cast<ulonglong2*>(to) = make_ulonglong2(S[e][p], S[e][p + 1]);
      }
  };
  if (chain) {
    const bool fresh = q_start[r] == 0;
#pragma unroll
    for (int e = 0; e < C; ++e)
#pragma unroll
      for (int p = 0; p < N; ++p) {
        float x[2];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int col = v0 + mine + e, ch = wk_channel<N>(l, p, half);
          x[half] = !fresh && col < dv && ch < dk ? slot[(size_t)col * dk + ch] : 0.f;
        }
        S[e][p] = f2_pair(x[0], x[1]);
      }
    leave(0);
  }
  float out[C] = {};
  f2 P[WK_OWN / 2] = {};
  const int tk0 = warp >= 2 * WK_CHAIN ? WK_OWN : 0, tk = tk0 + (l & 7), j0 = l & 8;  // an output lane's token, of whose earlier ones it takes j0 .. j0 + 7

#pragma unroll 1
  for (int c = c0; c <= c1; ++c) {  // (one more trip for the last chunk's outputs)
    const int buf = (c - c0) & 1, tok0 = row_begin + (c - c0) * WK_TOK;
    if (!APART && !chain) cs_wait<ST - 2>();
    __syncthreads();  // the chunk has come, and every warp is done with the stage that the next fetch fills
    const float* st = wk_smem + (size_t)((c - c0) % ST) * I::floats;
    if (chain) {
      if (c == c1) break;
      float u[C];
#pragma unroll
      for (int e = 0; e < C; e += 2) {
        const float2 given = *reinterpret_cast<const float2*>(st + I::u + l * COLS + mine + e);
        u[e] = given.x;
        u[e + 1] = given.y;
      }
      if constexpr (MODE == WALK_DELTA) {
        float d[C];
        wk_against<N, C, WK_TOK>(d, S, st + I::w, l);
#pragma unroll
        for (int e = 0; e < C; ++e) u[e] -= d[e];
      }
      if constexpr (MODE == WALK_HEAD) {
        const float f = v_scale ? st[I::scale + l] : 1.f;
#pragma unroll
        for (int e = 0; e < C; ++e) u[e] *= f;
      }
      const float* uk = us + buf * COLS * WK_TOK;
#pragma unroll
      for (int e = 0; e < C; ++e) {
        if (tok0 + l >= row_end) u[e] = 0.f;  // (what a state that is not finite makes of a token behind the row's end)
        us[(buf * COLS + e) * WK_TOK + l] = u[e];
      }
      if constexpr (MODE == WALK_HEAD) {
        const float f = st[I::last + WK_TOK + l];
#pragma unroll
        for (int e = 0; e < C; ++e) decayed[e * WK_TOK + l] = u[e] * f;
        uk = decayed;
      }
      f2 keep[N];
      if constexpr (MODE == WALK_HEAD) {
        const float f = st[I::last + 2 * WK_TOK];
#pragma unroll
        for (int p = 0; p < N; ++p) keep[p] = f2_pair(f, f);
      } else {
        wk_row<N>(keep, st + I::last, l);
      }
      __syncwarp();
      // the first half of the tokens by itself, then the state ahead of the chunk, then the other tokens one by one: half the roundings
      // of a long-lived state, and none more of one that decays fast (whose last token, then, must come behind it)
      const bool half = row_end - tok0 <= WK_TOK / 2;
      f2 next[C][N];
#pragma unroll
      for (int e = 0; e < C; ++e)
#pragma unroll
        for (int p = 0; p < N; ++p) next[e][p] = half ? f2_mul(S[e][p], keep[p]) : 0ull;
#pragma unroll
      for (int j = 0; j < WK_TOK; j += 4) {
        if (j == WK_TOK / 2 && !half) {
#pragma unroll
          for (int e = 0; e < C; ++e)
#pragma unroll
            for (int p = 0; p < N; ++p) f2_fma(next[e][p], S[e][p], keep[p]);
        }
        float4 uj[C];
#pragma unroll
        for (int e = 0; e < C; ++e) uj[e] = *reinterpret_cast<const float4*>(uk + e * WK_TOK + j);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          f2 x[N];
          wk_row<N>(x, st + I::k + (j + i) * DKP, l);
#pragma unroll
          for (int e = 0; e < C; ++e) {
            const float f = i == 0 ? uj[e].x : i == 1 ? uj[e].y : i == 2 ? uj[e].z : uj[e].w;
            const f2 twice = f2_pair(f, f);
#pragma unroll
            for (int p = 0; p < N; ++p) f2_fma(next[e][p], twice, x[p]);
          }
        }
      }
#pragma unroll
      for (int e = 0; e < C; ++e)
#pragma unroll
        for (int p = 0; p < N; ++p) S[e][p] = next[e][p];
      leave(buf ^ 1);
      __syncwarp();  // (u is read to the end before the next chunk's takes its place)
    } else {
      if (!APART) fetch(c + ST - 1);
      if (c > c0) {  // the chunk before: P U
        const float* uc = us + (buf ^ 1) * COLS * WK_TOK;
        bool finite = true;
#pragma unroll
        for (int e = 0; e < C; ++e) finite = finite && fabsf(uc[e * WK_TOK + l]) <= FLT_MAX;
        finite = __all_sync(0xffffffffu, finite);
        if (finite) {
          f2 a[C];
#pragma unroll
          for (int e = 0; e < C; ++e) a[e] = f2_pair(out[e], 0.f);
#pragma unroll
          for (int j = 0; j < WK_OWN; j += 4)
#pragma unroll
            for (int e = 0; e < C; ++e) {
              const ulonglong2 uj = *reinterpret_cast<const ulonglong2*>(uc + e * WK_TOK + j0 + j);
              f2_fma(a[e], P[j / 2], uj.x);
              f2_fma(a[e], P[j / 2 + 1], uj.y);
            }
#pragma unroll
          for (int e = 0; e < C; ++e) out[e] = f2_sum(a[e]);
        } else {  // (zero times a later token's infinity is no zero)
#pragma unroll
          for (int j = 0; j < WK_OWN; ++j) {
            const float2 x = f2_halves(P[j / 2]);
#pragma unroll
            for (int e = 0; e < C; ++e)
              if (j0 + j <= tk) out[e] = fmaf(j & 1 ? x.y : x.x, uc[e * WK_TOK + j0 + j], out[e]);
          }
        }
        const int tok = tok0 - WK_TOK + tk;
#pragma unroll
        for (int e = 0; e < C; ++e) {
          out[e] += __shfl_xor_sync(0xffffffffu, out[e], 8);
          if ((e & 1) == (l >> 3) && tok < row_end && v0 + mine + e < dv) o[((size_t)tok * H + h) * dv + v0 + mine + e] = out[e];
        }
      }
      if (c == c1) break;
#pragma unroll
      for (int e = 0; e < C; ++e) wk_row<N>(S[e], states + (buf * COLS + e) * DKP, l);
#pragma unroll
      for (int j = 0; j < WK_OWN; j += 4) {
        const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(st + I::pair + tk * I::ldp + j0 + j);
        P[j / 2] = x.x;
        P[j / 2 + 1] = x.y;
      }
      wk_against<N, C, WK_OWN>(out, S, st + I::q + tk0 * DKP, l);
      if constexpr (MODE == WALK_HEAD) {
        const float f = st[I::last + tk];
#pragma unroll
        for (int e = 0; e < C; ++e) out[e] *= f;
      }
    }
  }
  if (!chain) return;
#pragma unroll
  for (int e = 0; e < C; ++e)
#pragma unroll
    for (int p = 0; p < N; ++p) {
      const float2 x = f2_halves(S[e][p]);
      const int col = v0 + mine + e, ch = wk_channel<N>(l, p, 0);
      if (col < dv && ch < dk) slot[(size_t)col * dk + ch] = x.x;
      if (col < dv && ch + 1 < dk) slot[(size_t)col * dk + ch + 1] = x.y;
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
  __shared__ double dot[WK_TOK][WK_TOK + 1];
  __shared__ float as[WK_TOK][33];
  pdl_prologue(decay, cu_q);
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
      a = behind_loadf4(q + (size_t)(t0 + i) * ld_q + (size_t)grp * DK + c);
      b = behind_loadf4(k + (size_t)(t0 + i) * ld_k + (size_t)grp * DK + c);
    }
    *reinterpret_cast<float4*>(&qs[i][c]) = a;
    *reinterpret_cast<float4*>(&ks[i][c]) = b;
  }
  __syncthreads();
  {  // a thread's two dot products: token i with j and with j + 8
    const int i = tid >> 3, j = tid & 7;
    f2 s0[16] = {}, s1[16] = {};  // (sums of DK / 32 products, added up in 64 bits)
#pragma unroll 1
    for (int c = 0; c < DK; c += 32)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(&qs[i][c + 4 * e]), b = *reinterpret_cast<const ulonglong2*>(&ks[j][c + 4 * e]),
                         d = *reinterpret_cast<const ulonglong2*>(&ks[j + 8][c + 4 * e]);
        f2_fma(s0[2 * e], a.x, b.x);
        f2_fma(s0[2 * e + 1], a.y, b.y);
        f2_fma(s1[2 * e], a.x, d.x);
        f2_fma(s1[2 * e + 1], a.y, d.y);
      }
    double x0 = 0.0, x1 = 0.0;
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const float2 a = f2_halves(s0[e]), b = f2_halves(s1[e]);
      x0 += (double)a.x + (double)a.y;
      x1 += (double)b.x + (double)b.y;
    }
    dot[i][j] = x0;
    dot[i][j + 8] = x1;
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
      double run = 1.0, before = 1.0;
#pragma unroll
      for (int i = 0; i < WK_TOK; ++i) {
        const double a = (double)as[i][e];
        if (i > j) run *= a;
        if (i <= j) before *= a;
        out[i * WK_TOK] = i >= j ? (float)(dot[i][j] * (run * (double)q_scale)) : 0.f;
      }
      float* dec = decays + ((size_t)chunk * H + first + e) * (3 * WK_TOK);
      dec[j] = (float)(before * (double)q_scale);
      dec[WK_TOK + j] = (float)run;
      if (j == WK_TOK - 1) dec[2 * WK_TOK] = (float)before;
    }
  }
}

// Dynamic shared memory beyond 48 KB is asked for once per kernel and device. Not a dependent launch: CTAs that become resident while the kernel
// before drains gather on the SMs that are free first, and two chains on one SM walk at half the rate.
#define MS_WALK_LAUNCH(MODE, N, C, APART, ...)                                                                                     \
  do {                                                                                                                      \
    auto walk = walk_kernel<MODE, N, C, APART>;                                                                                    \
    constexpr size_t bytes = WalkStage<MODE, N, C>::bytes;                                                                  \
    static std::atomic<unsigned long long> allowed{0};                                                                      \
    MS_CHECK_CUDA(allow_shared_memory((const void*)walk, (int)bytes, allowed));                                             \
    MS_LAUNCH_APART(walk, dim3(ceil_div(dv, WalkStage<MODE, N, C>::cols), H, num_rows), (WK_CHAIN + WK_OUT + (APART ? WK_FETCH : 0)) * 32, bytes, stream, __VA_ARGS__); \
  } while (0)
// Four columns a lane take half the reads from shared memory of two, but half the CTAs too: two until 16 columns a CTA leave two SMs of three
// one. Both kernels, 2,048 tokens, two columns against four, us: 64 CTAs of 16 columns (16 heads of 64 x 64, delta rule) 140 / 169, (8 of 64 x 128,
// decay rule) 107 / 126; 128 of them (32 of 64 x 64, delta rule) 242 / 221, (32 of 128 x 64, a decay per head) 219 / 191; 768 (three rows, 64
// of 128 x 64) 396 / 254.
// Where every CTA has a multiprocessor of its own (two columns), two more warps fetch: the output warps, which fetch elsewhere, were what a chunk waited for
// (1,640 cycles against 1,330 of the chain): 16 heads of 64 x 64, 2,048 tokens 136 -> 127, 8 of 64 x 128, 300 tokens 23.2 -> 21.5. With several CTAs a
// multiprocessor they only take issue slots (64 of 128 x 64, 64 rows of 32 tokens 319 -> 371).
#define MS_WALK_LAUNCH_FOR(MODE, N, ...)                                                                                            \
  do {                                                                                                                              \
    if (3ll * num_rows * H * ceil_div(dv, WalkStage<MODE, N, 4>::cols) >= 2ll * sms) MS_WALK_LAUNCH(MODE, N, 4, false, __VA_ARGS__); \
    else if (1ll * num_rows * H * ceil_div(dv, WalkStage<MODE, N, 2>::cols) <= sms) MS_WALK_LAUNCH(MODE, N, 2, true, __VA_ARGS__);  \
    else MS_WALK_LAUNCH(MODE, N, 2, false, __VA_ARGS__);                                                                            \
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
  const int sms = sm_count();
  MS_WALK_LAUNCH_FOR((DELTA ? WALK_DELTA : WALK_CHANNEL), N, o, state, qp, DKP, wp, kp, DKP, 1, last, u0, dvp, (const float*)nullptr, pairs, cu_q,
                     q_start, state_slot, H, dk, dv);
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
  float* pairs = scratch;
  float* decays = pairs + (size_t)max_chunks * H * WK_TOK * WK_TOK;
  auto prepare = walk_head_kernel<DK>;
  MS_LAUNCH(prepare, dim3(max_chunks, H / qk_group), WK_THREADS, 0, stream, pairs, decays, q, ld_q, k, ld_k, qk_group, decay, ld_decay, cu_q,
            num_rows, H, q_scale);
  const int sms = sm_count();
  MS_WALK_LAUNCH_FOR(WALK_HEAD, N, o, state, q, ld_q, (const float*)nullptr, k, ld_k, qk_group, decays, v, ld_v, v_scale, pairs, cu_q, q_start,
                     state_slot, H, DK, dv);
  return 0;
}

}  // namespace ms

using namespace ms;

// The most chunks that a step of so many tokens in so many rows can have.
static inline int walk_max(int tokens, int rows) { return tokens / WK_TOK + rows; }

// Floats of scratch for a step of so many tokens in so many rows. groups: of heads that share q and k, with one decay per head; 0: a decay per key channel.
MS_EXPORT long long ms_walk_scratch(int tokens, int rows, int H, int dk, int dv, int delta, int groups) {
  if (!delta && tile_walk_takes(tokens, rows, H, dk, dv, groups)) return tile_walk_scratch(tokens, rows, H, dk, dv, groups);
  const long long items = (long long)walk_max(tokens, rows) * H, dkp = dk <= 32 ? 32 : dk <= 64 ? 64 : 128;
  if (groups) return items * (WK_TOK * WK_TOK + 3 * WK_TOK);
  return items * (WK_TOK * dkp * (delta ? 3 : 2) + dkp + WK_TOK * WK_TOK + (long long)WK_TOK * (ceil_div(dv, WK_COLS) * WK_COLS));
}

// Kernels that such a step launches.
MS_EXPORT int ms_walk_kernels(int tokens, int rows, int H, int dk, int dv, int delta, int groups) {
  return !delta && tile_walk_takes(tokens, rows, H, dk, dv, groups) ? 3 : 2;
}

// The decay rule (delta 0) or the delta rule with a decay per key channel; operands as ms_decay_scan's, dk up to 128. o [T, H, dv] float32.
MS_EXPORT int ms_walk_scan(float* o, float* state, const void* q, int ld_q, const void* k, int ld_k, int qk_group, const void* v, int ld_v,
                           const void* z, int ld_z, const float* z_bias, const float* decay_coef, float z_sign, const void* beta, int ld_beta,
                           const float* v_scale, float* scratch, const int* cu_q, const int* q_start, const int* state_slot,
                           int num_tokens, int num_rows, int H, int dk, int dv, float q_scale, int delta, int in_dtype, int z_dtype,
                           int* status, cudaStream_t stream) {
  if (num_rows == 0 || num_tokens == 0) return 0;
  MS_CHECK_ARG(dk >= 1 && dk <= 128 && dv >= 1 && H >= 1 && H <= 65535 && num_rows <= 65535, "walk_scan: %d heads of %d x %d, %d rows", H, dk, dv, num_rows);
  MS_CHECK_ARG(qk_group > 0 && H % qk_group == 0, "walk_scan: %d heads are not a multiple of the group of %d", H, qk_group);
  MS_CHECK_ARG(!delta || beta != nullptr, "walk_scan: the delta rule needs beta");
  MS_CHECK_ARG((uintptr_t)scratch % 16 == 0, "walk_scan: scratch must start on 16 bytes");
  const int max_chunks = walk_max(num_tokens, num_rows);
  const bool tiles = !delta && tile_walk_takes(num_tokens, num_rows, H, dk, dv, 0);
#define MS_WALK(TIN, TZZ)                                                                                                                       \
  return tiles ? tile_walk_channel<TIN, TZZ>(o, state, (const TIN*)q, ld_q, (const TIN*)k, ld_k, qk_group, (const TIN*)v, ld_v, (const TZZ*)z,   \
                                             ld_z, z_bias, decay_coef, z_sign, v_scale, scratch, cu_q, q_start, state_slot, num_tokens,         \
                                             num_rows, H, dk, dv, q_scale, status, stream)                                                      \
               : launch_walk_for<TIN, TZZ>(delta, dk, o, state, (const TIN*)q, ld_q, (const TIN*)k, ld_k, qk_group, (const TIN*)v, ld_v,        \
                                           (const TZZ*)z, ld_z, z_bias, decay_coef, z_sign, (const TZZ*)beta, ld_beta, v_scale, scratch, cu_q,  \
                                           q_start, state_slot, num_rows, max_chunks, H, dk, dv, q_scale, stream)
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
                                const int* state_slot, int num_tokens, int num_rows, int H, int dk, int dv, float q_scale, int* status, cudaStream_t stream) {
  if (num_rows == 0 || num_tokens == 0) return 0;
  MS_CHECK_ARG((dk == 32 || dk == 64 || dk == 128) && dv >= 1 && H >= 1 && H <= 65535 && num_rows <= 65535, "walk_scan_head: %d heads of %d x %d", H, dk, dv);
  MS_CHECK_ARG(qk_group > 0 && H % qk_group == 0, "walk_scan_head: %d heads are not a multiple of the group of %d", H, qk_group);
  MS_CHECK_ARG((uintptr_t)q % 16 == 0 && (uintptr_t)k % 16 == 0 && ld_q % 4 == 0 && ld_k % 4 == 0 && (uintptr_t)scratch % 16 == 0,
               "walk_scan_head: rows of q and k must start on 16 bytes");
  if (tile_walk_takes(num_tokens, num_rows, H, dk, dv, H / qk_group))
    return tile_walk_head(o, state, q, ld_q, k, ld_k, qk_group, v, ld_v, decay, ld_decay, v_scale, scratch, cu_q, q_start, state_slot, num_tokens, num_rows, H, dk,
                          dv, q_scale, status, stream);
  const int max_chunks = walk_max(num_tokens, num_rows);
#define MS_WALK(N)                                                                                                                            \
  return launch_walk_head<N>(o, state, q, ld_q, k, ld_k, qk_group, v, ld_v, decay, ld_decay, v_scale, scratch, cu_q, q_start, \
                             state_slot, num_rows, max_chunks, H, dv, q_scale, stream)
  if (dk == 32) MS_WALK(1);
  if (dk == 64) MS_WALK(2);
  MS_WALK(4);
#undef MS_WALK
}

// ms_walk_scan_head by chunks of 64 tokens, whatever the step, in which copies do not come: those of queries from chunk `no_queries` of a row on, those of what
// chunks add to the state from `no_added` on. Each wait ends after limit_ns, the status word is raised, and the kernel ends by itself. For tests.
MS_EXPORT int ms_tile_walk_selftest(float* o, float* state, const float* q, const float* k, const float* v, const float* decay, float* scratch, const int* cu_q,
                                    const int* q_start, const int* state_slot, int num_tokens, int num_rows, int H, int dk, int dv, int* status, int no_queries,
                                    int no_added, long long limit_ns, cudaStream_t stream) {
  MS_CHECK_ARG(status != nullptr && limit_ns > 0 && limit_ns <= 1000000000LL, "tile_walk_selftest: a limit of up to a second, and a status word");
  MS_CHECK_ARG((dk == 32 || dk == 64 || dk == 128) && dv >= 1 && H >= 1 && H <= 65535 && num_rows >= 1 && num_tokens >= 1, "tile_walk_selftest: %d heads of %d x %d", H, dk, dv);
  TwWaits waits;
  waits.no_queries = no_queries, waits.no_added = no_added, waits.limit_ns = (unsigned long long)limit_ns;
  return tile_walk_head(o, state, q, H * dk, k, H * dk, 1, v, H * dv, decay, H, nullptr, scratch, cu_q, q_start, state_slot, num_tokens, num_rows, H, dk, dv, 1.f,
                        status, stream, waits);
}
MS_EXPORT long long ms_tile_walk_scratch(int tokens, int rows, int H, int dk, int dv, int groups) { return tile_walk_scratch(tokens, rows, H, dk, dv, groups); }
