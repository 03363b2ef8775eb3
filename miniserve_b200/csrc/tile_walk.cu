// The decay rule of ``recurrence.cu`` over long rows by chunks of 64 tokens, in 32-bit accuracy, on the tensor cores:
//
//   S <- diag(d_t) S + k_t v_t^T;   o_t = S^T q_t
//
// with d_t one decay per key channel or one per head. In a chunk whose first token sees the state S, with G_i the product of the decays from
// the chunk's first token to i and D_ij that of the tokens behind j up to i,
//
//   P_ij = q_i . D_ij k_j for j <= i,      O = (G q) S + P V,      S_behind = G_last S + (D_(last, .) k)^T V.
//
// Three kernels. The first makes operand tiles of queries and keys (with a decay per channel: decayed to and from the chunk's ends, and the pairs;
// with one per head: the undecayed pairs, shared by the heads that share q and k). The second takes every chunk by itself: what the chunk adds to the state, and
// the outputs that come of its own pairs. The third walks a row's chunks: S <- G_last S + (what the chunk adds), and adds (G q) S to the outputs. Where heads and
// rows leave multiprocessors idle, the third cuts rows into segments; each adds up the state from the row's first chunk on, in the same
// steps, so that a segment's outputs have the bits of the whole row's.
//
// Accuracy: a factor is the sum of three bfloat16 that hold all of its 24 bits, whatever its neighbours are (the splitting of Henry, Tang and Heinecke,
// "Leveraging the bfloat16 artificial intelligence datatype for higher-precision computations", 2019). Tensor cores cut sums off where float32 rounds them; so
// pairs of one sixteen tokens and what a chunk's last eight tokens add to the state are float32 multiply-adds, and the sums of the rest are short. Products of
// decays are worked out in 64 bits and rounded once (a running product of decays just below one is rounded down every time). A state is rounded twice in 64 tokens.
// Root mean squares of the errors over 1,400 and 2,088 tokens, against the token-by-token walk's and the chunks of 16's, decays from 0.02 to 0.99999: outputs 0.28 to 0.96
// and 0.36 to 1.00, states 0.13 to 1.02 and 0.25 to 1.00. With one channel, token or number in a hundred 1,024 to 16,384 times the others, or keys by 2^s and queries by 2^-s
// (s from -12 to 12): outputs 0.27 to 1.1 of either, with exact decays none off by more than 8e-7 of its terms' sizes. A token sees nothing of the tokens behind it, whatever they hold:
// chunks with values that are not finite, or of 2^48 and more, are worked out in plain sums, every pair by itself. (With one decay per head the
// sums against the state are scaled behind the sum: a state within q's size of the largest float overflows.)
//
// What bounds it, 64 heads of 128 x 64, three rows of 1,037, 640 and 371 tokens, 263 us by chunks of 16 and 170 here: the second kernel (91 us) issues its instructions at
// half the rate, most of them making operands and adding up results; the third (54) is a chain of 17 chunks, bound by shared memory and the state's parts; the first 24 (long scoreboard, 28 % of the issue slots; a microsecond less
// with sums of eight products everywhere, and outputs under fast decays 1.07 times as far off as by chunks of 16; two more with sums of four everywhere).
// Measured and not kept: the same products in float32 multiply-adds, 8 x 8 outputs a thread (332 us: both shared memory and the FMA pipe at 54 %); all three kernels' work
// on the chain (322); parts on a grid that a row shares, whose products add up without any cut (165, but a row's small numbers lose the bits that its largest takes: one
// value channel of 1,024 made outputs 28 times as far off).
#include <cfloat>

#include "chunk_mma.cuh"
#include "float_pairs.cuh"
#include "tile_walk.cuh"

namespace ms {

constexpr int TW_FIRST = 256, TW_WORKERS = 512, TW_THREADS = TW_WORKERS + 32, TW_COLS = 64, TW_SUB = 16;
// A chunk's pairs: the blocks of 16 x 16 below the diagonal, then those on it. With one decay per head these are not decayed yet, and in 64 bits: what they are
// multiplied with is, and the product is rounded once.
constexpr int TW_BLOCK = TW_SUB * TW_SUB, TW_DIAGONAL = 6 * TW_BLOCK;
enum TileWalkMode : int { TW_CHANNEL = 0, TW_HEAD = 1 };

// ---------------------------------------------------------------- pieces of a step's rows
// A row of n tokens has ceil(n / tokens) pieces, numbered row by row. Every warp finds its own by adding up over the rows, 32 at a time.
struct TwPiece {
  int row, begin, end, first;  // the row, its tokens, the piece's first token (flat)
  int index, count;            // which of the row's pieces
  int chunk;                   // the number of the chunk of 64 tokens that begins there
};
__device__ __forceinline__ TwPiece tw_piece(int at, int tokens, const int* __restrict__ cu_q, int num_rows) {
  const int lane = threadIdx.x & 31;
  int pieces = 0, chunks = 0;
  for (int r0 = 0; r0 < num_rows; r0 += 32) {
    const int r = r0 + lane;
    const int begin = r < num_rows ? cu_q[r] : 0, end = r < num_rows ? cu_q[r + 1] : 0;
    const int mine = (end - begin + tokens - 1) / tokens, own = (end - begin + TW_TOK - 1) / TW_TOK;
    int upto = mine, cupto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, upto, o), y = __shfl_up_sync(0xffffffffu, cupto, o);
      if (lane >= o) upto += x, cupto += y;
    }
    const unsigned hit = __ballot_sync(0xffffffffu, at < pieces + upto);
    if (hit) {
      const int l = __ffs(hit) - 1;
      TwPiece p;
      p.row = r0 + l;
      p.begin = __shfl_sync(0xffffffffu, begin, l);
      p.end = __shfl_sync(0xffffffffu, end, l);
      p.count = __shfl_sync(0xffffffffu, mine, l);
      p.index = at - pieces - (__shfl_sync(0xffffffffu, upto, l) - p.count);
      p.first = p.begin + p.index * tokens;
      p.chunk = chunks + __shfl_sync(0xffffffffu, cupto - own, l) + p.index * tokens / TW_TOK;
      return p;
    }
    pieces += __shfl_sync(0xffffffffu, upto, 31);
    chunks += __shfl_sync(0xffffffffu, cupto, 31);
  }
  TwPiece none = {-1, 0, 0, 0, 0, 0, 0};
  return none;
}

__device__ __forceinline__ int tw_below(int i, int j) { return (i * (i - 1) / 2 + j) * TW_BLOCK; }  // (floats)
__host__ __device__ constexpr int tw_pairs(bool head) { return TW_DIAGONAL + 4 * TW_BLOCK * (head ? 2 : 1); }

// A chunk's factors, for each head: the decays from the chunk's first token to each (times q's factor), where there is one per head; those of the whole chunk.
template <int MODE, int DKP>
struct TwFactors {  // floats
  static constexpr int from = 0, last = MODE == TW_HEAD ? TW_TOK : 0, floats = last + (MODE == TW_HEAD ? 4 : DKP);
};

// ---------------------------------------------------------------- numbers in three parts
// A float32 number is the sum of three bfloat16, each what is left rounded to eight bits: of all its 24 bits, whatever its neighbours are. Their
// products are exact; l l, below 2^-36 of a product, is left out. What the tensor cores lose is what falls off a sum that grows: they cut off where
// float32 sums round. So the products of the first parts, where that counts, have a short chain and an accumulator of their own.
constexpr uint32_t TW_MOST = (127u + 48u) << 23, TW_MOST_PAIRS = (127u + 72u) << 23;  // (numbers, pairs of 2^48, 2^72 and more go to the plain sums)
__device__ __forceinline__ uint32_t tw_bits(float x) { return __float_as_uint(x) & 0x7fffffffu; }
__device__ __forceinline__ uint32_t tw_pack(f2 x) {
  uint32_t r;
  const float2 h = f2_halves(x);
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(h.y), "f"(h.x));
  return r;
}
__device__ __forceinline__ f2 tw_less(f2 a, uint32_t b) {  // a - b, which is exact here
  f2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(f2_pair(__uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u))));
  return r;
}
__device__ __forceinline__ void tw_parts(uint32_t (&out)[3], f2 x) {
  out[0] = tw_pack(x);
  const f2 r = tw_less(x, out[0]);
  out[1] = tw_pack(r);
  out[2] = tw_pack(tw_less(r, out[1]));
}
__device__ __forceinline__ void tw_parts8(uint4 (&out)[3], const float* x) {
  uint32_t w[4][3];
#pragma unroll
  for (int i = 0; i < 4; ++i) tw_parts(w[i], f2_pair(x[2 * i], x[2 * i + 1]));
#pragma unroll
  for (int p = 0; p < 3; ++p) out[p] = make_uint4(w[0][p], w[1][p], w[2][p], w[3][p]);
}
// Operand tiles: 64 numbers a row, 128-byte swizzle. Where eight neighbouring numbers of a row lie (bytes).
constexpr int TW_TILE = TW_TOK * 128;
__device__ __forceinline__ int tw_at(int row, int eight) { return row * 128 + ((eight ^ (row & 7)) << 4); }

// Queries and keys of a chunk, [64][LD] in shared memory, as operand tiles in global memory: queries [part][channels / 64][64 tokens][64 channels],
// keys [part][channels][64 tokens]. Returns whether a thread's numbers are too large or none.
template <int DK, int LD>
__device__ __forceinline__ bool tw_images(uint8_t* q_to, uint8_t* k_to, const float* qs, const float* ks) {
  constexpr int CP = DK < 64 ? 64 : DK, PARTS = TW_FIRST / CP, TOKENS = TW_TOK / PARTS, PART = CP / 64 * TW_TILE;  // (CP: channels with those behind the last)
  const int tid = threadIdx.x;
  uint32_t worst = 0;
  {  // four threads a token, every fourth run of eight channels each
    const int i = tid >> 2, part = tid & 3;
#pragma unroll
    for (int e = part * 8; e < CP; e += 32) {
      float x[8];
#pragma unroll
      for (int c = 0; c < 8; c += 4) {
        const float4 y = e < DK ? *reinterpret_cast<const float4*>(qs + i * LD + e + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[c] = y.x, x[c + 1] = y.y, x[c + 2] = y.z, x[c + 3] = y.w;
        worst = max(max(max(worst, tw_bits(y.x)), tw_bits(y.y)), max(tw_bits(y.z), tw_bits(y.w)));
      }
      uint4 y[3];
      tw_parts8(y, x);
#pragma unroll
      for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(q_to + p * PART + (e >> 6) * TW_TILE + tw_at(i, (e & 63) >> 3)) = y[p];
    }
  }
  const int ch = tid % CP, t0 = tid / CP * TOKENS;
#pragma unroll
  for (int t = 0; t < TOKENS; t += 8) {
    float x[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      x[e] = ch < DK ? ks[(t0 + t + e) * LD + ch] : 0.f;
      worst = max(worst, tw_bits(x[e]));
    }
    uint4 y[3];
    tw_parts8(y, x);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(k_to + p * PART + tw_at(ch, (t0 + t) >> 3)) = y[p];
  }
  return worst >= TW_MOST;
}

// ---------------------------------------------------------------- one decay per head: operands and dot products
// grid (chunks, groups of heads that share q and k). A thread's 4 x 4 dot products (tokens wb * 16 + ty + 4 a against 32 half + tx + 8 b), sums of
// four (on the diagonal) or sixteen products, added up in 64 bits: however much smaller than others a token's numbers are, its pairs are as precise.
template <int DK>
__global__ void __launch_bounds__(TW_FIRST, 2)
tile_head_kernel(float* __restrict__ dots, uint8_t* __restrict__ q_image, uint8_t* __restrict__ k_image, int* __restrict__ plain, const float* __restrict__ q,
                 int ld_q, const float* __restrict__ k, int ld_k, const int* __restrict__ cu_q, int num_rows) {
  constexpr int LD = DK + 4;
  extern __shared__ __align__(16) float tw_smem[];
  float *qs = tw_smem, *ks = qs + TW_TOK * LD;
  pdl_prologue(cu_q);
  const int grp = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const TwPiece at = tw_piece(blockIdx.x, TW_TOK, cu_q, num_rows);
  if (at.row < 0) return;
  const int t0 = at.first, n = min(TW_TOK, at.end - t0);
#pragma unroll
  for (int e = 0; e < TW_TOK * DK / 4 / TW_FIRST; ++e) {
    const int idx = e * TW_FIRST + tid, i = idx / (DK / 4), c = (idx % (DK / 4)) * 4;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
    if (i < n) {
      a = behind_loadf4(q + (size_t)(t0 + i) * ld_q + (size_t)grp * DK + c);
      b = behind_loadf4(k + (size_t)(t0 + i) * ld_k + (size_t)grp * DK + c);
    }
    *reinterpret_cast<float4*>(qs + i * LD + c) = a;
    *reinterpret_cast<float4*>(ks + i * LD + c) = b;
  }
  __syncthreads();
  const size_t image = (size_t)at.chunk * gridDim.y + grp;
  {
    constexpr size_t bytes = (size_t)3 * (DK <= 64 ? 1 : 2) * TW_TILE;
    const bool bad = tw_images<DK, LD>(q_image + image * bytes, k_image + image * bytes, qs, ks);
    const int any = __syncthreads_or(bad);
    if (tid == 0) plain[image] = any;
  }
  const int wb = warp < 4 ? warp : 7 - warp, half = warp >> 2, ty = lane >> 3, tx = lane & 7;
  if (half != 0 && wb < 2) return;
  const int flip = (wb & 1) << 1;  // the thread's columns 8 (y ^ flip) on: those of y < 2 are the block on the diagonal, if the warp has one
  double sum[4][4] = {};
#pragma unroll 1
  for (int c0 = 0; c0 < DK; c0 += 16) {
    f2 part[4][4] = {};
#pragma unroll
    for (int c = 0; c < 16; c += 4) {
      ulonglong2 a[4], b[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        a[e] = *reinterpret_cast<const ulonglong2*>(qs + (wb * TW_SUB + ty + 4 * e) * LD + c0 + c);
        b[e] = *reinterpret_cast<const ulonglong2*>(ks + (half * 32 + tx + 8 * (e ^ flip)) * LD + c0 + c);
      }
#pragma unroll
      for (int x = 0; x < 4; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) {
          f2_fma(part[x][y], a[x].x, b[y].x);
          f2_fma(part[x][y], a[x].y, b[y].y);
          if (c == 4 && y < 2) {
            const float2 h = f2_halves(part[x][y]);
            sum[x][y] += (double)h.x + (double)h.y;
            part[x][y] = 0ull;
          }
        }
    }
#pragma unroll
    for (int x = 0; x < 4; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const float2 h = f2_halves(part[x][y]);
        sum[x][y] += y < 2 ? (double)h.x + (double)h.y : (double)(h.x + h.y);
      }
  }
  float* to = dots + image * tw_pairs(true);
  double* diagonal = reinterpret_cast<double*>(to + TW_DIAGONAL) + wb * TW_BLOCK;
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    const int j = half * 32 + tx + 8 * (y ^ flip);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int at = (ty + 4 * x) * TW_SUB + (j & 15);
      if ((j >> 4) < wb) to[tw_below(wb, j >> 4) + at] = (float)sum[x][y];
      if ((j >> 4) == wb) diagonal[at] = sum[x][y];
    }
  }
}

// ---------------------------------------------------------------- a decay per key channel: pairs, decayed queries and keys
// grid (chunks, H). q', k' [chunks, H, 64, dkp] float32 (dkp = 32 N >= dk, zeros behind dk). z: the decays' logits (bias, coef, sign as in
// recurrence.cu). The pairs of a sixteen: a warp takes four tokens j at once, eight lanes over the channels of each, lets their keys decay from
// j on, and adds up over the lanes at the end. Then a thread per sixteen and channel decays queries from the sixteen's start and keys to its
// end, which make the pairs of different sixteens, the keys decayed on over the sixteens between them. Bound by a CTA's chain (two or three a
// multiprocessor, 30 % of the issue slots): 2,048 tokens of 8 heads of 64 channels 22.7 us; 27.0 with the operands read one by one, four in flight, and
// q' and k' read back from global memory for their images.
template <typename TIn, typename TZ, int N>
__global__ void __launch_bounds__(TW_FIRST, 2)
tile_prepare_kernel(float* q_out, float* k_out, uint8_t* __restrict__ q_image, uint8_t* __restrict__ k_image, int* __restrict__ plain,
                    float* __restrict__ factors, float* __restrict__ pairs,
                    const TIn* __restrict__ q, int ld_q, const TIn* __restrict__ k, int ld_k, int qk_group, const TZ* __restrict__ z, int ld_z,
                    const float* __restrict__ z_bias, const float* __restrict__ decay_coef, float z_sign, const int* __restrict__ cu_q, int num_rows,
                    int H, int dk, float q_scale) {
  constexpr int DKP = 32 * N, LD = DKP + 4, SUBS = TW_TOK / TW_SUB;
  using F = TwFactors<TW_CHANNEL, DKP>;
  extern __shared__ __align__(16) float tw_smem[];
  float *qs = tw_smem, *ks = qs + TW_TOK * LD, *ds = ks + TW_TOK * LD;
  constexpr bool KEEP = N <= 2;  // k' stays in shared memory as well (a fourth array; at N = 4 it would leave room for one CTA)
  float* kf = KEEP ? ds + TW_TOK * LD : ks;
  __shared__ double whole[SUBS][DKP];  // a sixteen's decays
  pdl_prologue(q, k, z, z_bias, decay_coef, cu_q);
  const int h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const TwPiece at = tw_piece(blockIdx.x, TW_TOK, cu_q, num_rows);
  if (at.row < 0) return;
  const int t0 = at.first, n = min(TW_TOK, at.end - t0);
  const size_t qk_at = (size_t)(h / qk_group) * dk, item = (size_t)at.chunk * H + h;
  const float coef = decay_coef[h];
  auto decay = [&](float logit, int c) { return expf(-coef * softplusf(z_sign * (logit + z_bias[(size_t)h * dk + c]))); };
  if (dk % 4 == 0 && in_fours(q, ld_q) && in_fours(k, ld_k) && in_fours(z, ld_z)) {
    constexpr int EACH = TW_TOK * DKP / 4 / TW_FIRST, AT_ONCE = EACH < 4 ? EACH : 4;
#pragma unroll 1
    for (int e0 = 0; e0 < EACH; e0 += AT_ONCE) {
      float4 fq[AT_ONCE], fk[AT_ONCE], fd[AT_ONCE];
#pragma unroll
      for (int e = 0; e < AT_ONCE; ++e) {  // all of it is asked for before the first is worked on
        const int idx = (e0 + e) * TW_FIRST + tid, i = idx / (DKP / 4), c = (idx % (DKP / 4)) * 4;
        const bool in = i < n && c < dk;
        const size_t t = in ? (size_t)(t0 + i) : (size_t)t0;
        const int cc = in ? c : 0;
        fq[e] = load4(q + t * ld_q + qk_at + cc);
        fk[e] = load4(k + t * ld_k + qk_at + cc);
        fd[e] = load4(z + t * ld_z + (size_t)h * dk + cc);
      }
#pragma unroll
      for (int e = 0; e < AT_ONCE; ++e) {
        const int idx = (e0 + e) * TW_FIRST + tid, i = idx / (DKP / 4), c = (idx % (DKP / 4)) * 4;
        const bool in = i < n && c < dk;
        const float4 none = make_float4(0.f, 0.f, 0.f, 0.f);
        *reinterpret_cast<float4*>(qs + i * LD + c) = in ? make_float4(fq[e].x * q_scale, fq[e].y * q_scale, fq[e].z * q_scale, fq[e].w * q_scale) : none;
        *reinterpret_cast<float4*>(ks + i * LD + c) = in ? fk[e] : none;
        *reinterpret_cast<float4*>(ds + i * LD + c) =
            in ? make_float4(decay(fd[e].x, c), decay(fd[e].y, c + 1), decay(fd[e].z, c + 2), decay(fd[e].w, c + 3)) : make_float4(1.f, 1.f, 1.f, 1.f);
      }
    }
  } else {
#pragma unroll 4
    for (int e = 0; e < TW_TOK * DKP / TW_FIRST; ++e) {
      const int idx = e * TW_FIRST + tid, i = idx / DKP, c = idx % DKP;
      float fq = 0.f, fk = 0.f, fd = 1.f;
      if (i < n && c < dk) {
        const size_t t = (size_t)(t0 + i);
        fq = Elem<TIn>::load(q + t * ld_q + qk_at + c) * q_scale;
        fk = Elem<TIn>::load(k + t * ld_k + qk_at + c);
        fd = decay(Elem<TZ>::load(z + t * ld_z + (size_t)h * dk + c), c);
      }
      qs[i * LD + c] = fq;
      ks[i * LD + c] = fk;
      ds[i * LD + c] = fd;
    }
  }
  float* fac = factors + item * F::floats;
  float* out = pairs + item * tw_pairs(false);
  __syncthreads();
#pragma unroll 1
  for (int sub = warp >> 2; sub < SUBS; sub += 2) {
    const int cl = lane & 7, j = (warp & 3) * 4 + (lane >> 3), s0 = sub * TW_SUB;
    f2 p[2 * N] = {};
    double val[16];
#pragma unroll
    for (int i = 0; i < TW_SUB; ++i) {
      f2 b = 0ull;
#pragma unroll
      for (int m = 0; m < N; ++m) {
        const int c = (s0 + i) * LD + cl * 4 + 32 * m;
        const ulonglong2 fk = *reinterpret_cast<const ulonglong2*>(ks + c), fq = *reinterpret_cast<const ulonglong2*>(qs + c),
                         fd = *reinterpret_cast<const ulonglong2*>(ds + c);
        p[2 * m] = i == j ? fk.x : f2_mul(p[2 * m], fd.x);  // (nothing ahead of token j)
        p[2 * m + 1] = i == j ? fk.y : f2_mul(p[2 * m + 1], fd.y);
        f2_fma(b, fq.x, p[2 * m]);
        f2_fma(b, fq.y, p[2 * m + 1]);
      }
      val[i] = f2_sum(b);
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      const bool up = cl & o;
#pragma unroll
      for (int i = 0; i < 2 * o; ++i) {
        const double send = up ? val[i] : val[i + 2 * o], keep = up ? val[i + 2 * o] : val[i];
        val[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int i = 2 * cl + e;
      out[TW_DIAGONAL + sub * TW_BLOCK + i * TW_SUB + j] = i >= j ? (float)val[e] : 0.f;
    }
  }
  __syncthreads();
  // a thread per sixteen and channel: queries from the sixteen's start, keys to its end, in 64 bits
  constexpr int TURNS = SUBS * DKP <= TW_FIRST ? 1 : SUBS * DKP / TW_FIRST;
  const bool mine = SUBS * DKP >= TW_FIRST || tid < SUBS * DKP;
#pragma unroll 1
  for (int e = 0; e < TURNS; ++e) {
    const int idx = e * TW_FIRST + tid, sub = idx / DKP, c = idx % DKP;
    if (mine) {
      double passed = 1.0;
#pragma unroll 4
      for (int i = 0; i < TW_SUB; ++i) passed *= (double)ds[(sub * TW_SUB + i) * LD + c];
      whole[sub][c] = passed;
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int e = 0; e < TURNS; ++e) {
    const int idx = e * TW_FIRST + tid, sub = idx / DKP, c = idx % DKP;
    if (mine) {
      double before = 1.0, behind = 1.0, all = 1.0;
      for (int s = 0; s < SUBS; ++s) {
        if (s < sub) before *= whole[s][c];
        if (s > sub) behind *= whole[s][c];
        all *= whole[s][c];
      }
      if (sub == 0) fac[F::last + c] = (float)all;
      double own = 1.0;
#pragma unroll 4
      for (int i = TW_SUB - 1; i >= 0; --i) {
        const int t = sub * TW_SUB + i;
        const double x = own * (double)ks[t * LD + c];
        const float y = (float)(behind * x);
        ks[t * LD + c] = (float)x;
        if (KEEP) kf[t * LD + c] = y;
        k_out[(item * TW_TOK + t) * DKP + c] = y;
        own *= (double)ds[t * LD + c];
      }
      own = 1.0;
#pragma unroll 4
      for (int i = 0; i < TW_SUB; ++i) {
        const int t = sub * TW_SUB + i;
        own *= (double)ds[t * LD + c];
        const double x = own * (double)qs[t * LD + c];
        const float y = (float)(before * x);
        qs[t * LD + c] = (float)x;
        ds[t * LD + c] = y;  // (nobody asks for this decay any more)
        q_out[(item * TW_TOK + t) * DKP + c] = y;
      }
    }
  }
  __syncthreads();
  // sixteens `far` apart: 2 x 2 pairs a thread, 64 threads a block of 16 x 16
#pragma unroll 1
  for (int far = 1; far < SUBS; ++far) {
    if (far > 1) {  // keys over the sixteen that now lies between
      for (int idx = tid; idx < (SUBS - far) * TW_SUB * DKP; idx += TW_FIRST) {
        const int t = idx / DKP, c = idx % DKP;
        ks[t * LD + c] = (float)((double)ks[t * LD + c] * whole[t / TW_SUB + far - 1][c]);
      }
      __syncthreads();
    }
    const int jb = tid >> 6;
    if (jb < SUBS - far) {
      const int i0 = (tid & 63) >> 3, j0 = tid & 7;  // (rows i0, i0 + 8 against j0, j0 + 8)
      const float *qa = qs + ((jb + far) * TW_SUB + i0) * LD, *kb = ks + (jb * TW_SUB + j0) * LD;
      double sum[2][2] = {};
#pragma unroll 1
      for (int c0 = 0; c0 < DKP; c0 += 8) {
        f2 part[2][2] = {};
#pragma unroll
        for (int c = c0; c < c0 + 8; c += 4) {
          ulonglong2 a[2], b[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            a[e] = *reinterpret_cast<const ulonglong2*>(qa + 8 * e * LD + c);
            b[e] = *reinterpret_cast<const ulonglong2*>(kb + 8 * e * LD + c);
          }
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
              f2_fma(part[x][y], a[x].x, b[y].x);
              f2_fma(part[x][y], a[x].y, b[y].y);
            }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 2; ++y) sum[x][y] += (double)f2_sum(part[x][y]);
      }
      float* to = out + tw_below(jb + far, jb);
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) to[(i0 + 8 * x) * TW_SUB + j0 + 8 * y] = (float)sum[x][y];
    }
    __syncthreads();
  }
  if (!KEEP) {
    for (int idx = tid; idx < TW_TOK * DKP / 4; idx += TW_FIRST) {  // (what this CTA has written above)
      const int t = idx / (DKP / 4), c = (idx % (DKP / 4)) * 4;
      *reinterpret_cast<float4*>(ks + t * LD + c) = *reinterpret_cast<const float4*>(k_out + (item * TW_TOK + t) * DKP + c);
    }
    __syncthreads();
  }
  const size_t bytes = (size_t)3 * (DKP / 64) * TW_TILE;
  const bool bad = tw_images<DKP, LD>(q_image + item * bytes, k_image + item * bytes, ds, kf);
  const int any = __syncthreads_or(bad);
  if (tid == 0) plain[item] = any;
}

// ---------------------------------------------------------------- copies and products
__device__ __forceinline__ void tw_bar_init(uint64_t* bar, int count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(cs_smem(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void tw_expect(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(cs_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tw_bulk(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
               ::"r"(cs_smem(dst)), "l"(src), "r"(bytes), "r"(cs_smem(bar)) : "memory");
}
__device__ __forceinline__ void tw_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(cs_smem(bar)) : "memory");
}
__device__ __forceinline__ void tw_arrive(uint64_t* bar) {  // a warp's lanes have written or read what the barrier stands for
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncwarp();
  if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(cs_smem(bar)) : "memory");
}
__device__ __forceinline__ bool tw_wait(uint64_t* bar, int use, unsigned long long limit_ns) {  // for the use of that number
  const bool ok = mbar_wait_bounded(cs_smem(bar), use & 1, limit_ns);
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  return ok;
}
// Operand tiles in shared memory, 128-byte swizzle, groups of eight rows 1,024 bytes apart: rows are M or N, or the sums' index (COLUMNS)
__device__ __forceinline__ uint64_t tw_desc(const void* tile, uint32_t part = 16) {
  return (uint64_t)((cs_smem(tile) & 0x3FFFF) >> 4) | (uint64_t)(part >> 4) << 16 | (uint64_t)(1024 >> 4) << 32 | (uint64_t)1 << 46 | (uint64_t)2 << 61;
}
template <bool COLUMNS = false>
__device__ __forceinline__ void tw_mma(uint32_t d, uint64_t a, uint64_t b, int n, bool accumulate) {  // 64 rows
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (COLUMNS ? 1u << 16 : 0u) | ((uint32_t)(n >> 3) << 17) | (4u << 24), acc = accumulate;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
               ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc) : "memory");
}
// All products of A's parts with B's but the last two's: the largest at `d`, the rest 64 columns on
template <bool COLUMNS = false>
__device__ __forceinline__ void tw_mma_parts(uint32_t d, uint64_t a, int a_part, uint64_t b, int b_part, bool accumulate) {
  const uint64_t a1 = a + (a_part >> 4), a2 = a1 + (a_part >> 4), b1 = b + (b_part >> 4), b2 = b1 + (b_part >> 4);
  tw_mma<COLUMNS>(d, a, b, 128, accumulate);
  tw_mma<COLUMNS>(d + 64, a1, b, 64, true);
  tw_mma<COLUMNS>(d + 64, a, b2, 64, true);
  tw_mma<COLUMNS>(d + 64, a1, b1, 64, true);
  tw_mma<COLUMNS>(d + 64, a2, b, 64, true);
  tw_mma<COLUMNS>(d + 64, a1, b2, 64, true);
  tw_mma<COLUMNS>(d + 64, a2, b1, 64, true);
}
// 16 rows of 32 columns: registers 4 k + {0, 1}: row lane / 4, columns 8 k + 2 (lane % 4) + {0, 1}; 4 k + {2, 3}: eight rows on
__device__ __forceinline__ void tw_tmem_pairs(float (&r)[16], uint32_t at) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
               : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]),
                 "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
               : "r"(at));
}
// the sum of SETS pairs of accumulators, 128 columns each
template <int SETS>
__device__ __forceinline__ void tw_tmem_sums(float (&r)[16], uint32_t at) {
  float more[2 * SETS - 1][16];
  tw_tmem_pairs(r, at);
#pragma unroll
  for (int i = 1; i < 2 * SETS; ++i) tw_tmem_pairs(more[i - 1], at + 64 * (i & 1) + 128 * (i >> 1));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    if constexpr (SETS == 2) r[j] = (r[j] + more[1][j]) + (more[0][j] + more[2][j]);
    else r[j] += more[0][j];
  }
}
__device__ __forceinline__ bool tw_elect() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(pred));
  return pred != 0;
}
__device__ __forceinline__ bool tw_group_any(int id, bool flag) {  // a barrier of 256 threads with an OR over a flag
  uint32_t res;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %2, 0;\n\tbar.red.or.pred q, %1, 256, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(res) : "r"(id), "r"((uint32_t)flag) : "memory");
  return res != 0;
}
struct TwArgs {
  float *o, *state;
  const uint8_t *q_image, *k_image;
  const int* plain;  // of a chunk: queries or keys are too large, or no numbers
  const float *q, *k, *pairs, *decay, *v_scale;
  float* factors;
  const void* v;
  float q_scale;
  int ld_decay;
  float *added, *start;  // what a chunk adds to the state, [16 quads of columns][channels][4]; the state ahead of a row that is cut
  const int *cu_q, *q_start, *state_slot;
  int* status;
  int ld_q, ld_k, qk_group, ld_v, unit, num_rows, H, dk, dv, tiles, o_quads;
  TwWaits waits;
};
// outputs of a chunk that a warp read as tw_tmem_pairs has them: tokens tok and 8 on of the chunk's n, columns col, 8 on, ..
__device__ __forceinline__ void tw_add_outputs(const TwArgs& g, const float (&r)[16], float by0, float by1, int tok0, int tok, int n, int h, int col) {
  float* to = g.o + ((size_t)(tok0 + tok) * g.H + h) * g.dv + col;
#pragma unroll
  for (int j = 0; j < 16; j += 2) {
    const int row = (j >> 1) & 1, c = 8 * (j >> 2);
    const float x = r[j] * (row ? by1 : by0), y = r[j + 1] * (row ? by1 : by0);
    if (tok + 8 * row < n) {
      float* at_o = to + (row ? (size_t)8 * g.H * g.dv : 0) + c;
      if (g.o_quads) {
        if (col + c < g.dv) asm volatile("red.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(at_o), "f"(x), "f"(y) : "memory");
      } else {
        if (col + c < g.dv) atomicAdd(at_o, x);
        if (col + c + 1 < g.dv) atomicAdd(at_o + 1, y);
      }
    }
  }
}

// ---------------------------------------------------------------- a chunk by itself
// grid (chunks x column tiles, H, 2): what the chunk adds to the state (z = 0), and the outputs that come of its own pairs (z = 1). A thread has one
// column's 16 values, and 16 pairs of a token. Pairs of different sixteens are products of parts; those of one sixteen are plain sums, a column's in the
// thread that has its values: where a token's own value is all that is left, it is as precise as any. So is what the last eight tokens add to the state, which
// is most of it where decays are fast (with four, a state under decays from 0.7 to 0.99 is 1.14 times as far off as token by token).
constexpr int TW_LAST = 8;
struct TwChunk {  // bytes (last: where the pairs of one sixteen and, once they are in the values, products of decays are)
  static constexpr int b = 0, a = 3 * TW_TILE, runs = 6 * TW_TILE, near = runs + 3 * TW_TOK * 8, last = runs, fac = last + TW_LAST * (TW_COLS + 128) * 4, bars = fac + 2 * TW_TOK * 4,
                       all = bars + 64;
  static_assert(near + 4 * TW_BLOCK * 4 <= fac, "pairs and products of decays end ahead of the factors");
};
template <int MODE, int DKP, typename TV>
__global__ void __launch_bounds__(TW_FIRST, 4) tile_chunk_kernel(const TwArgs g) {
  using I = TwChunk;
  using F = TwFactors<MODE, DKP>;
  constexpr int NB = DKP / 64, IMAGE = 3 * NB * TW_TILE;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y;
  const int tile = blockIdx.x % g.tiles, v0 = tile * TW_COLS;
  const bool adds = blockIdx.z == 0;
  const TwPiece at = tw_piece(blockIdx.x / g.tiles, TW_TOK, g.cu_q, g.num_rows);
  if (at.row < 0) return;
  const int tok0 = at.first, n = min(TW_TOK, at.end - tok0);
  const size_t item = (size_t)at.chunk * g.H + h, image = MODE == TW_HEAD ? (size_t)at.chunk * (g.H / g.qk_group) + h / g.qk_group : item;
  uint64_t *k_full = reinterpret_cast<uint64_t*>(smem + I::bars), *done = k_full + 2;
  uint32_t* slot_at = reinterpret_cast<uint32_t*>(k_full + 4);
  double *as = reinterpret_cast<double*>(smem + I::runs), *upto = as + TW_TOK, *after = upto + TW_TOK;  // decays; from a sixteen's start, to its end
  float *scale = reinterpret_cast<float*>(smem + I::fac), *behind = scale + TW_TOK;
  auto copy_keys = [&](int half) {
    tw_expect(k_full + half, 3 * TW_TILE);
#pragma unroll
    for (int p = 0; p < 3; ++p) tw_bulk(smem + I::a + p * TW_TILE, g.k_image + image * IMAGE + (p * NB + half) * TW_TILE, TW_TILE, k_full + half);
  };
  if (tid == 0) {
    for (int i = 0; i < 4; ++i) tw_bar_init(k_full + i, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    if (adds) copy_keys(0);
  }
  const int quad = warp & 3, c0 = 32 * (warp >> 2), vcol = c0 + lane, vtok = 16 * quad, prow = tid >> 2, ppart = tid & 3;
  const bool has_col = v0 + vcol < g.dv;
  const float* pairs = g.pairs + (MODE == TW_HEAD ? image : item) * tw_pairs(MODE == TW_HEAD);
  float u[16];
  {
    const TV* from = static_cast<const TV*>(g.v) + (size_t)(tok0 + vtok) * g.ld_v + (size_t)h * g.dv + v0 + vcol;
    TV raw[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      raw[i] = has_col && vtok + i < n ? *from : TV(0.f);
      from += g.ld_v;
    }
    if (warp == 7) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 128;\n" ::"r"(cs_smem(slot_at)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid < TW_TOK) {
      scale[tid] = g.v_scale && tid < n ? g.v_scale[(size_t)(tok0 + tid) * g.H + h] : 1.f;
      if constexpr (MODE == TW_HEAD) {
        const double a = tid < n ? (double)g.decay[(size_t)(tok0 + tid) * g.ld_decay + h] : 1.0;
        const int i = tid & 15;
        double x = a, y = __shfl_down_sync(0xffffffffu, a, 1);
        if (i == 15) y = 1.0;
#pragma unroll
        for (int o = 1; o < 16; o <<= 1) {
          const double before = __shfl_up_sync(0xffffffffu, x, o), next = __shfl_down_sync(0xffffffffu, y, o);
          if (i >= o) x *= before;
          if (i + o < 16) y *= next;
        }
        as[tid] = a, upto[tid] = x, after[tid] = y;
        if (!adds) behind[tid] = (float)y;  // (to the end of its sixteen)
      }
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i += 4) {
      const float4 by = MODE == TW_HEAD && adds ? make_float4(1.f, 1.f, 1.f, 1.f) : *reinterpret_cast<const float4*>(scale + vtok + i);
      u[i] = Elem<TV>::load(raw + i) * by.x, u[i + 1] = Elem<TV>::load(raw + i + 1) * by.y;
      u[i + 2] = Elem<TV>::load(raw + i + 2) * by.z, u[i + 3] = Elem<TV>::load(raw + i + 3) * by.w;
    }
  }
  const uint32_t tmem = *slot_at, lanes = tmem + ((uint32_t)(32 * quad) << 16);
  const int row = 16 * quad + (lane >> 2), pcol = c0 + 2 * (lane & 3);
  bool ok = true;
  // (what does not come in time gets as long again, since the CTA must not end while it is on its way)
  auto come = [&](uint64_t* bar) { return tw_wait(bar, 0, g.waits.limit_ns) || (tw_wait(bar, 0, g.waits.limit_ns), false); };
  uint32_t worst = g.plain[image] ? 0xffffffffu : 0u;
  auto over = [&](int from, int to) {  // the decays of whole sixteens
    double x = 1.0;
    for (int b = from; b < to; ++b) x *= upto[b * TW_SUB + TW_SUB - 1];
    return x;
  };
  if (adds) {
    if constexpr (MODE == TW_HEAD) {
      if (tid < TW_TOK) {
        const int b = tid >> 4;
        behind[tid] = (float)((double)scale[tid] * (after[tid] * over(b + 1, 4)));  // (the values' factor with it: one rounding less)
        if (tile == 0) {  // (for the walk)
          float* fac = g.factors + item * F::floats;
          fac[F::from + tid] = (float)((double)g.q_scale * over(0, b) * upto[tid]);
          if (tid == 0) fac[F::last] = (float)over(0, 4);
        }
      }
      __syncthreads();
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float4 by = *reinterpret_cast<const float4*>(behind + vtok + i);
        u[i] *= by.x, u[i + 1] *= by.y, u[i + 2] *= by.z, u[i + 3] *= by.w;
      }
    }
    if (g.start && at.index == 0 && at.end - at.begin > g.unit && g.q_start[at.row] != 0) {  // the state ahead of a row that is cut: its slot is written while others read
      const float* slot = g.state + ((size_t)g.state_slot[at.row] * g.H + h) * (size_t)g.dv * g.dk;
      float* to = g.start + (((size_t)at.row * g.H + h) * g.tiles + tile) * (TW_COLS * DKP);
      for (int idx = tid; idx < TW_COLS * DKP; idx += TW_FIRST) {
        const int col = idx / DKP, ch = idx % DKP;
        to[idx] = v0 + col < g.dv && ch < g.dk ? slot[(size_t)(v0 + col) * g.dk + ch] : 0.f;
      }
    }
    float *u_last = reinterpret_cast<float*>(smem + I::last), *k_last = u_last + TW_LAST * TW_COLS;  // [8][64], [DKP][8]
    for (int idx = tid; idx < TW_LAST * DKP; idx += TW_FIRST) {
      const int t = n - TW_LAST + idx / DKP, ch = idx % DKP;
      float x = 0.f;
      if (MODE == TW_HEAD) {
        if (t >= 0 && ch < g.dk) x = g.k[(size_t)(tok0 + t) * g.ld_k + (size_t)(h / g.qk_group) * g.dk + ch];
      } else if (t >= 0) {
        x = g.k[(item * TW_TOK + t) * DKP + ch];
      }
      k_last[ch * TW_LAST + idx / DKP] = x;
    }
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      worst = max(worst, tw_bits(u[i]));
      const int t = vtok + i - (n - TW_LAST);
      if (t >= 0 && t < TW_LAST) {
        u_last[t * TW_COLS + vcol] = u[i];
        u[i] = 0.f;
      }
    }
    if (n < TW_LAST)
      for (int idx = tid; idx < (TW_LAST - n) * TW_COLS; idx += TW_FIRST) u_last[idx] = 0.f;  // (rows ahead of the chunk's first token)
    {
      uint4 y[3];
#pragma unroll
      for (int q = 0; q < 16; q += 8) {
        tw_parts8(y, u + q);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(smem + I::b + p * TW_TILE + tw_at(vcol, (vtok + q) >> 3)) = y[p];
      }
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    const bool plain = __syncthreads_or(worst >= TW_MOST);
    float* added = g.added + (item * g.tiles + tile) * (TW_COLS * DKP);
#pragma unroll 1
    for (int half = 0; half < NB; ++half) {
      if (tid == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        ok = come(k_full + half) && ok;
        const uint64_t a = tw_desc(smem + I::a), b = tw_desc(smem + I::b);
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) tw_mma_parts(tmem, a + (ks * 32 >> 4), TW_TILE, b + (ks * 32 >> 4), TW_TILE, ks > 0);
        tw_commit(done + half);
        ok = come(done + half) && ok;
        if (half + 1 < NB) copy_keys(half + 1);
        asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      }
      __syncthreads();  // (one thread waits for the products: polling by all takes a third of the instructions)
      asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
      if (!plain) {
        float r[16];
        tw_tmem_sums<1>(r, lanes + c0);
        f2 sum[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) sum[j] = f2_pair(r[2 * j], r[2 * j + 1]);
#pragma unroll
        for (int t = 0; t < TW_LAST; t += 4) {
          float k0[4], k1[4];
          *reinterpret_cast<float4*>(k0) = *reinterpret_cast<const float4*>(k_last + (64 * half + row) * TW_LAST + t);
          *reinterpret_cast<float4*>(k1) = *reinterpret_cast<const float4*>(k_last + (64 * half + row + 8) * TW_LAST + t);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float* ut = u_last + (t + e) * TW_COLS + pcol;
            const f2 by[2] = {f2_pair(k0[e], k0[e]), f2_pair(k1[e], k1[e])};
#pragma unroll
            for (int j = 0; j < 8; ++j) f2_fma(sum[j], by[j & 1], *reinterpret_cast<const f2*>(ut + 8 * (j >> 1)));
          }
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int col = pcol + 8 * (j >> 1), ch = 64 * half + row + 8 * (j & 1);
          *reinterpret_cast<f2*>(added + ((col >> 2) * DKP + ch) * 4 + (col & 3)) = sum[j];
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
      __syncthreads();
    }
    if (plain) {
      const TV* from = static_cast<const TV*>(g.v) + (size_t)tok0 * g.ld_v + (size_t)h * g.dv + v0;
      for (int idx = tid; idx < TW_COLS * DKP; idx += TW_FIRST) {
        const int ch = (idx >> 2) % DKP, col = (idx >> 2) / DKP * 4 + (idx & 3);
        float r = 0.f;
        for (int j = 0; j < n; ++j) {
          const float x = MODE == TW_HEAD ? (ch < g.dk ? g.k[(size_t)(tok0 + j) * g.ld_k + (size_t)(h / g.qk_group) * g.dk + ch] : 0.f) : g.k[(item * TW_TOK + j) * DKP + ch];
          const float y = v0 + col < g.dv ? Elem<TV>::load(from + (size_t)j * g.ld_v + col) * (MODE == TW_HEAD ? behind[j] : scale[j]) : 0.f;
          r = fmaf(x, y, r);
        }
        added[idx] = r;
      }
    }
  } else {
    float pr[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) pr[i] = 0.f;
    if (ppart < prow >> 4) {
      const float* pf = pairs + tw_below(prow >> 4, ppart) + (prow & 15) * TW_SUB;
#pragma unroll
      for (int i = 0; i < 16; i += 4) {
        const float4 x = *reinterpret_cast<const float4*>(pf + i);
        pr[i] = x.x, pr[i + 1] = x.y, pr[i + 2] = x.z, pr[i + 3] = x.w;
      }
    }
    float* near = reinterpret_cast<float*>(smem + I::near);
    if constexpr (MODE == TW_HEAD) {
      const int b = tid >> 6, iq = ((tid >> 4) & 3) * 4, j = tid & 15;
      const double* from = reinterpret_cast<const double*>(pairs + TW_DIAGONAL) + b * TW_BLOCK + j;
      double d[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) d[e] = from[(iq + e) * TW_SUB];
      double run = (double)g.q_scale;
      for (int x = j + 1; x < iq; ++x) run *= as[b * TW_SUB + x];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (iq + e > j) run *= as[b * TW_SUB + iq + e];
        near[(b * TW_SUB + iq + e) * TW_SUB + j] = iq + e >= j ? (float)(d[e] * run) : 0.f;
      }
      if (ppart < prow >> 4) {
        const float f = (float)((double)g.q_scale * upto[prow] * over(ppart + 1, prow >> 4));
#pragma unroll
        for (int i = 0; i < 16; i += 4) {
          const float4 x = *reinterpret_cast<const float4*>(behind + 16 * ppart + i);
          pr[i] = pr[i] * f * x.x, pr[i + 1] = pr[i + 1] * f * x.y, pr[i + 2] = pr[i + 2] * f * x.z, pr[i + 3] = pr[i + 3] * f * x.w;
        }
      }
    } else {
      *reinterpret_cast<float4*>(near + tid * 4) = *reinterpret_cast<const float4*>(pairs + TW_DIAGONAL + tid * 4);
    }
    {
      uint4 y[3];
#pragma unroll
      for (int q = 0; q < 16; q += 8) {
        tw_parts8(y, u + q);
#pragma unroll
        for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(smem + I::b + p * TW_TILE + tw_at(vcol, (vtok + q) >> 3)) = y[p];
      }
      if (ppart < 3) {  // (the last sixteen is in nobody's pairs)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          tw_parts8(y, pr + 8 * q);
#pragma unroll
          for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(smem + I::a + p * TW_TILE + tw_at(prow, 2 * ppart + q)) = y[p];
        }
      }
      uint32_t far = 0;
#pragma unroll
      for (int i = 0; i < 16; ++i) worst = max(worst, tw_bits(u[i])), far = max(far, tw_bits(pr[i]));
      worst = max(worst, far >= TW_MOST_PAIRS ? TW_MOST : 0u);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    const bool plain = __syncthreads_or(worst >= TW_MOST);
    if (tid == 0) {
      const uint64_t a = tw_desc(smem + I::a), b = tw_desc(smem + I::b);
#pragma unroll
      for (int ks = 0; ks < 3; ++ks) tw_mma_parts(tmem, a + (ks * 32 >> 4), TW_TILE, b + (ks * 32 >> 4), TW_TILE, ks > 0);
      tw_commit(done);
    }
    __syncwarp();
    {  // the pairs of one sixteen: outputs, to which the others are added
      const float* pf = near + quad * (TW_SUB * TW_SUB);
      f2 u2[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) u2[i] = f2_pair(u[2 * i], u[2 * i + 1]);
      float* to = g.o + ((size_t)(tok0 + vtok) * g.H + h) * g.dv + v0 + vcol;
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        f2 r = 0ull;
#pragma unroll
        for (int j = 0; j <= i; j += 4) {
          const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(pf + i * TW_SUB + j);
          f2_fma(r, x.x, u2[j / 2]);
          if (j + 2 <= i) f2_fma(r, x.y, u2[j / 2 + 1]);
        }
        if (!plain && has_col && vtok + i < n) *to = f2_sum(r);
        to += (size_t)g.H * g.dv;
      }
    }
    if (plain) {  // (zero times a later token's infinity is no zero: every pair by itself)
      const TV* from = static_cast<const TV*>(g.v) + (size_t)tok0 * g.ld_v + (size_t)h * g.dv + v0;
      for (int idx = tid; idx < n * TW_COLS; idx += TW_FIRST) {
        const int i = idx >> 6, col = idx & 63, ib = i >> 4;
        if (v0 + col >= g.dv) continue;
        float sum = 0.f;
        for (int j = 0; j <= i; ++j) {
          const int jb = j >> 4;
          float x = jb == ib ? near[(ib * TW_SUB + (i & 15)) * TW_SUB + (j & 15)] : pairs[tw_below(ib, jb) + (i & 15) * TW_SUB + (j & 15)];
          if (MODE == TW_HEAD && jb != ib) x = (float)((double)x * ((double)g.q_scale * upto[i] * over(jb + 1, ib) * after[j]));
          sum = fmaf(x, Elem<TV>::load(from + (size_t)j * g.ld_v + col) * (g.v_scale ? g.v_scale[(size_t)(tok0 + j) * g.H + h] : 1.f), sum);
        }
        g.o[((size_t)(tok0 + i) * g.H + h) * g.dv + v0 + col] = sum;
      }
    }
    if (tid == 0) {
      ok = come(done);
      asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    }
    __syncthreads();  // the products are there, and outputs to be added to
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (!plain) {
      float r[16];
      tw_tmem_sums<1>(r, lanes + c0);
      tw_add_outputs(g, r, 1.f, 1.f, tok0, row, n, h, v0 + pcol);
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
  }
  if (!ok && g.status) atomicMax(g.status, 41);
  if (warp == 7) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 128;\n" ::"r"(tmem) : "memory");
}

// ---------------------------------------------------------------- the walk over a row's chunks
// grid (segments x column tiles, H). Eight warps carry the state (a thread: a channel's 32 columns), add what the chunks add, from the row's first chunk on, and
// from the segment's first on hand it to the tensor cores as an operand; eight more scale the products with the queries and add them to the
// outputs. One warp copies the images of queries and what the chunks add, and issues the products.
// A role whose wait runs out raises the status word and waits for nothing more. The state's warps go on to their end, since they vote in every chunk; then
// they agree on whether the state may be kept. The others leave their loops; the issuing thread once what it sent for has come.
template <int MODE, int DKP>
struct TwWalk {  // bytes
  static constexpr int image = 3 * (DKP / 64) * TW_TILE, sums = DKP * TW_COLS * 4;
  static constexpr int q = 0, s = 2 * image, added = 3 * image, bars = added + 2 * sums, all = bars + 128;
  static_assert(all <= 227 * 1024, "shared memory");
  static_assert(image >= sums, "the plain sums' state lies where the state's parts are");
};
template <int MODE, int DKP>
__global__ void __launch_bounds__(TW_THREADS, 1) tile_walk_kernel(const TwArgs g) {
  using I = TwWalk<MODE, DKP>;
  using F = TwFactors<MODE, DKP>;
  constexpr int NB = DKP / 64, COLS = 32;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.x / g.tiles % g.H;
  const int tile = blockIdx.x % g.tiles, v0 = tile * TW_COLS;
  const TwPiece at = tw_piece(blockIdx.x / g.tiles / g.H, g.unit, g.cu_q, g.num_rows);
  if (at.row < 0) return;
  const int end = min(at.end, at.first + g.unit), first = at.index * g.unit / TW_TOK, steps = first + (end - at.first + TW_TOK - 1) / TW_TOK;  // chunks of the row
  const int chunk0 = at.chunk - first;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + I::bars);
  uint64_t *q_full = bars /* two */, *added_full = bars + 2 /* two */, *added_read = bars + 4 /* two */, *outputs_read = bars + 6 /* two */, *state_in = bars + 8, *done = bars + 9 /* two */, *state_read = bars + 11;
  // (done: two, since an output warp that still adds a chunk's outputs may find the products of the next two done. Those of one barrier would then be as many
  // phases ahead, which reads as not done. With two, the third's products wait for outputs_read.)
  uint32_t* slot_at = reinterpret_cast<uint32_t*>(bars + 12);
  int* plain_at = reinterpret_cast<int*>(bars + 13);             // [4]: a chunk's products with the state are plain sums
  if (tid == 0) {
    for (int i = 0; i < 12; ++i) tw_bar_init(bars + i, (i >= 4 && i <= 8) || i == 11 ? 8 : 1);
    for (int i = 0; i < 4; ++i) plain_at[i] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == TW_WORKERS / 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;\n" ::"r"(cs_smem(slot_at)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
  const uint32_t tmem = *slot_at;
  const int w = warp & 7, quad = w & 3, c0 = COLS * (w >> 2);  // of tensor memory's lanes, of the columns
  const size_t images = MODE == TW_HEAD ? g.H / g.qk_group : g.H, own = MODE == TW_HEAD ? h / g.qk_group : h;
  bool ok = true;
  auto wait = [&](uint64_t* bar, int use) { return tw_wait(bar, use, g.waits.limit_ns); };
  auto all_wait = [&](uint64_t* bar, int use) { return __all_sync(0xffffffffu, wait(bar, use)); };  // (a warp's lanes go on as one)

  if (warp == TW_WORKERS / 32) {
    // ---- copies and products
    if (tw_elect()) {
      int q_sent = 0, added_sent = 0, products = 0;
      auto copy_q = [&](int c) {
        if (c >= g.waits.no_queries) return;
        ++q_sent;
        tw_expect(q_full + ((c - first) & 1), I::image);
        tw_bulk(smem + I::q + ((c - first) & 1) * I::image, g.q_image + ((size_t)(chunk0 + c) * images + own) * I::image, I::image, q_full + ((c - first) & 1));
      };
      auto copy_added = [&](int c) {
        if (c >= g.waits.no_added) return;
        ++added_sent;
        tw_expect(added_full + (c & 1), I::sums);
        tw_bulk(smem + I::added + (c & 1) * I::sums, g.added + (((size_t)(chunk0 + c) * g.H + h) * g.tiles + tile) * (TW_COLS * DKP), I::sums, added_full + (c & 1));
      };
      copy_added(0);
      if (steps > 1) copy_added(1);
      copy_q(first);
      if (steps > first + 1) copy_q(first + 1);
      const uint64_t b = tw_desc(smem + I::s, DKP * 128);
#pragma unroll 1
      for (int c = 0; c < steps && ok; ++c) {
        const int k = c - first;
        if (k >= 0) {
          ok = wait(state_in, k) && wait(q_full + (k & 1), k >> 1) && (k < 2 || wait(outputs_read + (k & 1), (k >> 1) - 1));
          if (!ok) break;
          const uint64_t a = tw_desc(smem + I::q + (k & 1) * I::image);
#pragma unroll
          for (int blk = 0; blk < NB; ++blk)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              tw_mma_parts<true>(tmem + (k & 1) * 256 + (ks & 1) * 128, a + ((blk * TW_TILE + ks * 32) >> 4), NB * TW_TILE, b + ((blk * 4 + ks) * 2048 >> 4), DKP * 128, blk * 4 + ks > 1);
          tw_commit(done + (k & 1));
          ++products;
        }
        ok = wait(added_read + (c & 1), c >> 1);
        if (c + 2 < steps && ok) copy_added(c + 2);
        if (k >= 0) {
          ok = ok && wait(done + (k & 1), k >> 1);
          if (c + 2 < steps && ok) copy_q(c + 2);
        }
      }
      if (!ok) {
        if (g.status) atomicMax(g.status, 42);
        for (int b = 0; b < 2; ++b) {  // the last use of each of the two
          if (q_sent > b) wait(q_full + b, (q_sent - 1 - b) >> 1);
          if (added_sent > b) wait(added_full + b, (added_sent - 1 - b) >> 1);
          if (products > b) wait(done + b, (products - 1 - b) >> 1);
        }
      }
    }
    __syncwarp();
  } else if (warp < 8) {
    // ---- the state
    const bool has_ch = DKP == 128 || (quad < 2);
    const int ch = (32 * quad + lane) % DKP;
    float S[COLS];
    float* slot = g.state + ((size_t)g.state_slot[at.row] * g.H + h) * (size_t)g.dv * g.dk;
    {
      const bool fresh = g.q_start[at.row] == 0;
      const float* from = at.count > 1 ? g.start + (((size_t)at.row * g.H + h) * g.tiles + tile) * (TW_COLS * DKP) : nullptr;
#pragma unroll
      for (int j = 0; j < COLS; ++j) {
        S[j] = 0.f;
        if (!fresh) {
          if (from) S[j] = from[(size_t)(c0 + j) * DKP + ch];  // (the row's last segment writes the slot)
          else if (v0 + c0 + j < g.dv && ch < g.dk) S[j] = slot[(size_t)(v0 + c0 + j) * g.dk + ch];
        }
      }
    }
    const float* last = g.factors + ((size_t)chunk0 * g.H + h) * F::floats + F::last + (MODE == TW_HEAD ? 0 : ch);
    const int* large_at = g.plain + (size_t)chunk0 * images + own;
    float keep = last[0];
    int large = large_at[0];
    bool plain = false;
    int plain_chunks = 0;
#pragma unroll 1
    for (int c = 0; c < steps; ++c) {
      const int k = c - first;
      if (k >= 0) {
        // the state as an operand: its parts, once the products over the one before are done
        uint32_t mine = 0;
#pragma unroll
        for (int j = 0; j < COLS; ++j) mine = max(mine, tw_bits(S[j]));
        const bool was = plain;
        plain = tw_group_any(1, (has_ch && mine >= TW_MOST) || large);
        if (tid == 0) plain_at[k & 3] = plain;
        if (k > 0) ok = ok && all_wait(done + ((k - 1) & 1), (k - 1) >> 1);
        if (was) ok = ok && all_wait(state_read, plain_chunks++);  // (the plain sums have read the state)
        if (plain) {
          float* Sf = reinterpret_cast<float*>(smem + I::s);
          if (has_ch)
#pragma unroll
            for (int j = 0; j < COLS; ++j) Sf[ch * TW_COLS + c0 + j] = S[j];
        } else if (has_ch) {
          uint8_t* to = smem + I::s + ch * 128;
#pragma unroll
          for (int q = 0; q < COLS / 8; ++q) {
            uint32_t y[4][3];
#pragma unroll
            for (int j = 0; j < 4; ++j) tw_parts(y[j], f2_pair(S[8 * q + 2 * j], S[8 * q + 2 * j + 1]));
#pragma unroll
            for (int p = 0; p < 3; ++p)
              *reinterpret_cast<uint4*>(to + p * DKP * 128 + ((((c0 >> 3) + q) ^ (ch & 7)) << 4)) = make_uint4(y[0][p], y[1][p], y[2][p], y[3][p]);
          }
        }
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        tw_arrive(state_in);
      }
      const float now = keep;
      if (c + 1 < steps) {
        last += (size_t)g.H * F::floats, large_at += images;
        keep = last[0], large = large_at[0];
      }
      ok = ok && all_wait(added_full + (c & 1), c >> 1);
      const float* add = reinterpret_cast<const float*>(smem + I::added + (c & 1) * I::sums);
#pragma unroll
      for (int j = 0; j < COLS; j += 4) {
        const float4 x = *reinterpret_cast<const float4*>(add + (((c0 + j) >> 2) * DKP + ch) * 4);
        S[j] = fmaf(S[j], now, x.x), S[j + 1] = fmaf(S[j + 1], now, x.y), S[j + 2] = fmaf(S[j + 2], now, x.z), S[j + 3] = fmaf(S[j + 3], now, x.w);
      }
      tw_arrive(added_read + (c & 1));
    }
    if (!ok && lane == 0 && g.status) atomicMax(g.status, 42);
    const bool lost = tw_group_any(1, !ok);  // (a part of it did not come)
    if (!lost && has_ch && at.index == at.count - 1 && ch < g.dk) {
#pragma unroll
      for (int j = 0; j < COLS; ++j)
        if (v0 + c0 + j < g.dv) slot[(size_t)(v0 + c0 + j) * g.dk + ch] = S[j];
    }
  } else {
    // ---- the outputs
    const int row = 16 * quad + (lane >> 2), col = v0 + c0 + 2 * (lane & 3);
    const uint32_t lanes = tmem + ((uint32_t)(32 * quad) << 16);
#pragma unroll 1
    for (int c = first; c < steps; ++c) {
      const int k = c - first, tok0 = at.begin + c * TW_TOK, n = min(TW_TOK, end - tok0);
      const size_t item = (size_t)(chunk0 + c) * g.H + h;
      const float* fac = g.factors + item * F::floats;
      const float by0 = MODE == TW_HEAD ? fac[F::from + row] : 1.f, by1 = MODE == TW_HEAD ? fac[F::from + row + 8] : 1.f;
      ok = all_wait(done + (k & 1), k >> 1);
      if (!ok) break;
      if (plain_at[k & 3]) {
        tw_arrive(outputs_read + (k & 1));
        const float* Sf = reinterpret_cast<const float*>(smem + I::s);
        for (int idx = tid - TW_WORKERS / 2; idx < n * TW_COLS; idx += TW_WORKERS / 2) {
          const int i = idx >> 6, e = idx & 63;
          float r = 0.f;
          for (int x = 0; x < DKP; ++x)
            r = fmaf(MODE == TW_HEAD ? (x < g.dk ? g.q[(size_t)(tok0 + i) * g.ld_q + own * g.dk + x] : 0.f) : g.q[(item * TW_TOK + i) * DKP + x], Sf[x * TW_COLS + e], r);
          if (MODE == TW_HEAD) r *= fac[F::from + i];
          if (v0 + e < g.dv) atomicAdd(g.o + ((size_t)(tok0 + i) * g.H + h) * g.dv + v0 + e, r);
        }
        tw_arrive(state_read);
        continue;
      }
      float r[16];
      tw_tmem_sums<2>(r, lanes + (k & 1) * 256 + c0);
      tw_arrive(outputs_read + (k & 1));
      tw_add_outputs(g, r, by0, by1, tok0, row, n, h, col);
    }
    if (!ok && lane == 0 && g.status) atomicMax(g.status, 42);
  }
  __syncthreads();
  if (warp == TW_WORKERS / 32) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;\n" ::"r"(tmem) : "memory");
}

// ---------------------------------------------------------------- host
// Tokens of a segment: whole chunks, as many that heads and column tiles times segments come to no more CTAs than multiprocessors.
static int tw_unit(int tokens, int H, int tiles) {
  const int sms = sm_count(), chunks = ceil_div(tokens, TW_TOK);
  const long long ctas = (long long)H * tiles;
  const int want = ctas < sms ? (int)(sms / ctas) : 1;
  return ceil_div(chunks, want) * TW_TOK;
}
static int tw_padded(int dk) { return dk <= 64 ? 64 : 128; }

// groups: of heads that share queries and keys, with one decay per head; 0: a decay per key channel.
struct TwPlan {
  int dkp, tiles, unit, segments, chunks;
  long long images, flags, pairs, factors, keys, added, start;  // floats (images: of the queries, and as many of the keys)
  TwPlan(int tokens, int rows, int H, int dk, int dv, int groups) {
    dkp = tw_padded(dk);
    tiles = ceil_div(dv, TW_COLS);
    unit = tw_unit(tokens, H, tiles);
    segments = tokens / unit + rows;
    chunks = tokens / TW_TOK + rows;
    const long long items = (long long)chunks * H, own = (long long)chunks * (groups ? groups : H), state = (long long)tiles * TW_COLS * dkp;
    images = own * 3 * (dkp / 64) * (TW_TILE / 4);
    flags = (own + 3) / 4 * 4;
    pairs = (groups ? own : items) * tw_pairs(groups > 0);
    factors = items * (groups ? TwFactors<TW_HEAD, 64>::floats : dkp);
    keys = groups ? 0 : items * TW_TOK * dkp;
    added = items * state;
    start = tokens > unit ? (long long)rows * H * state : 0;
  }
  long long floats() const { return 2 * images + flags + pairs + factors + 2 * keys + added + start; }
};

// Three launches and a chunk of 64 tokens for the shortest row, against a chain of chunks of 16. Measured on one B200, 31 shapes of 2 to 128 heads, steps of 200 to
// 4,096 tokens in 1 to 16 rows, tiles against chunks of 16 in us. Of several rows only their number is known here, not which of them is long.
//
// A decay per channel, one row: the time of either as a sum of what is launched, what all SMs do together and the row's chain, fitted to these steps (9 % off on the
// mean, hence the 6 % that chunks of 16 are favoured by where heads are not few). 32 heads of 128 x 128: 300 tokens 69 / 53, 640 111 / 104, 800 121 / 131, 2,048 274 / 324; 8 of
// 64 x 128: 640 36 / 34, 800 37 / 39, 2,048 65 / 91; 64 of 32 x 32 (half of whose channels are padding): 2,048 243 / 174. None of 136 such steps is more than an eighth slower than
// by chunks of 16. Several rows from 640 tokens each on the mean: rows of one length lose at first (16 heads of 128 x 64, two of 650 96 / 77; 32 of 64 x 64, two of 1,024 132 / 142), one long
// row beside short ones gains (16 of 128 x 64, 4,036 tokens and three of 20, 259 / 378).
//
// One decay per head, where tiles are nearly twice as fast over long rows: few heads over one row from 420 tokens, else from 300, and 96 more for every other row, whose
// lengths may be next to nothing. 4 heads of 64 x 64: 300 tokens 21 / 18, 512 23 / 26, 2,048 34 / 82; 16 of 64 x 64: 300 24 / 18, 400 25 / 22, 512 26 / 26, 2,048 52 / 83;
// 32 of 128 x 64: 300 34 / 34, 2,048 95 / 195; 64: 300 42 / 48, 1,024 88 / 144, 2,048 162 / 285. Several rows of few heads may lose some microseconds (16 of 64 x 64, four
// of 160 tokens 27 / 22) for what one long row beside short ones gains (580 tokens and three of 20: 31 / 51).
static bool tw_one_row_pays(int tokens, int H, int dk, int dv) {
  const float p = dk <= 64 ? 1.f : 2.f, n = dk <= 32 ? 0.5f : p, chunks = tokens / 64.f + 1.f;
  const int tiles = ceil_div(dv, TW_COLS), sms = sm_count();
  const float units = (float)(tw_unit(tokens, H, tiles) / TW_TOK), segments = 2ll * H * tiles > sms ? 1.f : tokens / 64.f / units + 1.f;
  const float rounds = fmaxf(1.f, segments * H * tiles / sms);
  const float by_tiles = 21.3f + chunks * H * (0.053f * p + tiles * (0.0075f * p + 0.015f)) + tokens / 64.f * 0.42f + 1.7f * p * fminf(units, tokens / 64.f) * rounds;
  const float by_sixteens = 7.f + (tokens / 16.f + 1.f) * H * 0.0098f * n + tokens / 16.f * (0.305f + 0.074f * n + H * dv / 64.f * (0.0114f + 0.0069f * n));
  return (H * tiles < 8 ? 1.f : 1.06f) * by_tiles < by_sixteens;
}
bool tile_walk_takes(int tokens, int rows, int H, int dk, int dv, int groups) {
  const bool few = rows == 1 && (long long)H * ceil_div(dv, TW_COLS) < 24;
  const bool pays = groups ? tokens >= (few ? 420 : 300) + 96ll * (rows - 1) : rows == 1 ? tw_one_row_pays(tokens, H, dk, dv) : tokens >= 640ll * rows;
  return pays && tile_walk_scratch(tokens, rows, H, dk, dv, groups) < (1ll << 28);
}
long long tile_walk_scratch(int tokens, int rows, int H, int dk, int dv, int groups) { return TwPlan(tokens, rows, H, dk, dv, groups).floats(); }

template <int MODE, int DKP, typename TV>
static int launch_tile_walk(const TwPlan& plan, TwArgs g, float* rest, cudaStream_t stream) {
  g.added = rest;
  g.start = plan.start ? rest + plan.added : nullptr;
  g.unit = plan.unit;
  g.tiles = plan.tiles;
  g.o_quads = g.dv % 4 == 0 && (uintptr_t)g.o % 16 == 0;
  auto chunk = tile_chunk_kernel<MODE, DKP, TV>;
  auto walk = tile_walk_kernel<MODE, DKP>;
  static std::atomic<unsigned long long> allowed_chunk{0}, allowed_walk{0};
  MS_CHECK_CUDA(allow_shared_memory((const void*)chunk, TwChunk::all, allowed_chunk));
  MS_CHECK_CUDA(allow_shared_memory((const void*)walk, TwWalk<MODE, DKP>::all, allowed_walk));
  MS_LAUNCH_APART(chunk, dim3(plan.chunks * plan.tiles, g.H, 2), TW_FIRST, TwChunk::all, stream, g);
  MS_LAUNCH_APART(walk, dim3(plan.segments * plan.tiles * g.H), TW_THREADS, (TwWalk<MODE, DKP>::all), stream, g);
  return 0;
}

template <int DK>
static int launch_tile_head(const TwPlan& plan, TwArgs g, float* scratch, cudaStream_t stream) {
  uint8_t *q_image = (uint8_t*)scratch, *k_image = (uint8_t*)(scratch + plan.images);
  int* plain = (int*)(scratch + 2 * plan.images);
  float *pairs = scratch + 2 * plan.images + plan.flags, *factors = pairs + plan.pairs;
  auto prepare = tile_head_kernel<DK>;
  constexpr size_t bytes = (size_t)2 * TW_TOK * (DK + 4) * 4;
  static std::atomic<unsigned long long> allowed{0};
  MS_CHECK_CUDA(allow_shared_memory((const void*)prepare, (int)bytes, allowed));
  MS_LAUNCH(prepare, dim3(plan.chunks, g.H / g.qk_group), TW_FIRST, bytes, stream, pairs, q_image, k_image, plain, g.q, g.ld_q, g.k, g.ld_k, g.cu_q, g.num_rows);
  g.q_image = q_image, g.k_image = k_image, g.plain = plain, g.pairs = pairs, g.factors = factors;
  return launch_tile_walk<TW_HEAD, (DK < 64 ? 64 : DK), float>(plan, g, factors + plan.factors, stream);
}

int tile_walk_head(float* o, float* state, const float* q, int ld_q, const float* k, int ld_k, int qk_group, const float* v, int ld_v, const float* decay,
                   int ld_decay, const float* v_scale, float* scratch, const int* cu_q, const int* q_start, const int* state_slot, int num_tokens,
                   int num_rows, int H, int dk, int dv, float q_scale, int* status, cudaStream_t stream, const TwWaits& waits) {
  const TwPlan plan(num_tokens, num_rows, H, dk, dv, H / qk_group);
  TwArgs g = {};
  g.waits = waits;
  g.o = o, g.state = state, g.q = q, g.ld_q = ld_q, g.k = k, g.ld_k = ld_k, g.qk_group = qk_group, g.v = v, g.ld_v = ld_v, g.status = status;
  g.decay = decay, g.ld_decay = ld_decay, g.v_scale = v_scale, g.q_scale = q_scale;
  g.cu_q = cu_q, g.q_start = q_start, g.state_slot = state_slot, g.num_rows = num_rows, g.H = H, g.dk = dk, g.dv = dv;
  if (dk == 32) return launch_tile_head<32>(plan, g, scratch, stream);
  if (dk == 64) return launch_tile_head<64>(plan, g, scratch, stream);
  return launch_tile_head<128>(plan, g, scratch, stream);
}

template <typename TIn, typename TZ, int N>
static int launch_tile_channel(const TwPlan& plan, TwArgs g, float* scratch, const TIn* q, const TIn* k, const TZ* z, int ld_z, const float* z_bias,
                               const float* decay_coef, float z_sign, float q_scale, cudaStream_t stream) {
  constexpr int DKP = 32 * N;
  uint8_t *q_image = (uint8_t*)scratch, *k_image = (uint8_t*)(scratch + plan.images);
  int* plain = (int*)(scratch + 2 * plan.images);
  float *pairs = scratch + 2 * plan.images + plan.flags, *factors = pairs + plan.pairs, *qp = factors + plan.factors, *kp = qp + plan.keys;
  auto prepare = tile_prepare_kernel<TIn, TZ, N>;
  constexpr size_t bytes = (size_t)(N <= 2 ? 4 : 3) * TW_TOK * (DKP + 4) * 4;
  static std::atomic<unsigned long long> allowed{0};
  MS_CHECK_CUDA(allow_shared_memory((const void*)prepare, (int)bytes, allowed));
  MS_LAUNCH(prepare, dim3(plan.chunks, g.H), TW_FIRST, bytes, stream, qp, kp, q_image, k_image, plain, factors, pairs, q, g.ld_q, k, g.ld_k, g.qk_group, z, ld_z,
            z_bias, decay_coef, z_sign, g.cu_q, g.num_rows, g.H, g.dk, q_scale);
  g.q = qp, g.k = kp, g.q_image = q_image, g.k_image = k_image, g.plain = plain, g.pairs = pairs, g.factors = factors;
  return launch_tile_walk<TW_CHANNEL, DKP, TIn>(plan, g, kp + plan.keys, stream);
}

template <typename TIn, typename TZ>
int tile_walk_channel(float* o, float* state, const TIn* q, int ld_q, const TIn* k, int ld_k, int qk_group, const TIn* v, int ld_v, const TZ* z, int ld_z,
                      const float* z_bias, const float* decay_coef, float z_sign, const float* v_scale, float* scratch, const int* cu_q, const int* q_start,
                      const int* state_slot, int num_tokens, int num_rows, int H, int dk, int dv, float q_scale, int* status, cudaStream_t stream, const TwWaits& waits) {
  const TwPlan plan(num_tokens, num_rows, H, dk, dv, 0);
  TwArgs g = {};
  g.waits = waits;
  g.o = o, g.state = state, g.ld_q = ld_q, g.ld_k = ld_k, g.qk_group = qk_group, g.v = v, g.ld_v = ld_v, g.status = status, g.v_scale = v_scale;
  g.cu_q = cu_q, g.q_start = q_start, g.state_slot = state_slot, g.num_rows = num_rows, g.H = H, g.dk = dk, g.dv = dv;
  if (dk <= 64) return launch_tile_channel<TIn, TZ, 2>(plan, g, scratch, q, k, z, ld_z, z_bias, decay_coef, z_sign, q_scale, stream);
  return launch_tile_channel<TIn, TZ, 4>(plan, g, scratch, q, k, z, ld_z, z_bias, decay_coef, z_sign, q_scale, stream);
}

#define MS_TW_CHANNEL(TIN, TZZ)                                                                                                                     \
  template int tile_walk_channel<TIN, TZZ>(float*, float*, const TIN*, int, const TIN*, int, int, const TIN*, int, const TZZ*, int, const float*,   \
                                           const float*, float, const float*, float*, const int*, const int*, const int*, int, int, int, int, int,  \
                                           float, int*, cudaStream_t, const TwWaits&)
MS_TW_CHANNEL(float, float);
MS_TW_CHANNEL(float, __nv_bfloat16);
MS_TW_CHANNEL(__nv_bfloat16, float);
MS_TW_CHANNEL(__nv_bfloat16, __nv_bfloat16);
#undef MS_TW_CHANNEL

}  // namespace ms
