// Row-wise causal attention over the paged cache: one warp per (new token, query head).
//
// This is the attention of the true float32 path (and the fallback for head sizes the
// tensor-core kernels do not take). Its arithmetic for one (token, head) is a fixed sequence of
// float32 operations that depends only on that query, the keys and values of its own request and
// their absolute positions: keys are taken in tiles of 32 aligned to absolute position, each
// lane owns one key of the tile, scores are a sequential dot product, the tile's maximum and sum
// go through a fixed lane tree, and the running (max, sum, output) are updated tile by tile.
// So the result is the same bit for bit whether the token came in a whole prompt, in a portion,
// alone as a decode token, or beside other requests.
//
// Formula: softmax(q k^T * d^-0.5 + causal mask) v with query head h reading kv head
// h / (heads / kv_heads) (miniserve/model/attention.py:60-67, miniserve/model/qwen3.py:133-135);
// a query at absolute position p sees keys 0..p of its request, or p-window+1..p with a window; with `keep_first` the
// first keep_first keys of the request stay visible behind the window (their tiles are walked first, in order). A
// distance bias takes r1_h * ln(1 + r2_h * (p - j)) off the scaled score of key j.
#include <cfloat>
#include <type_traits>

#include "common.cuh"

namespace ms {

constexpr int ROWWISE_MAX_D = 512;  // a lane holds head_dim / 32 output channels: 8 up to a head size of 256, 16 beyond

template <typename T, int DI>
__global__ void __launch_bounds__(128)
attention_rowwise_kernel(T* __restrict__ out,            // [T, nq, d]
                         const T* __restrict__ q,        // [T, nq, d]
                         const T* __restrict__ k_pool,   // [pages, nkv, page_size, d]
                         const T* __restrict__ v_pool,
                         const int* __restrict__ positions, const int* __restrict__ row_of_token,
                         const int* __restrict__ page_indptr, const int* __restrict__ page_indices,
                         int num_tokens, int nq, int nkv, int d, float scale, int window, int sink, int page_shift,
                         int num_pages, int* __restrict__ status, const float* __restrict__ sink_values, float softcap,
                         int chunk, const float* __restrict__ dist_r1, const float* __restrict__ dist_r2, int keep_first) {
  extern __shared__ float q_smem[];  // [warps][d]
  pdl_prologue(q, k_pool, v_pool, positions, row_of_token, page_indptr, page_indices, sink_values, dist_r1, dist_r2);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long item = (long long)blockIdx.x * (blockDim.x >> 5) + warp;
  if (item >= (long long)num_tokens * nq) return;
  const int t = (int)(item / nq), h = (int)(item - (long long)t * nq);
  const int kvh = h / (nq / nkv);
  const int qpos = positions[t];
  const int row = row_of_token[t];
  const int* pages = page_indices + page_indptr[row];
  const int page_size = 1 << page_shift;
  int lo = window > 0 ? max(0, qpos - window + 1) : 0;
  if (chunk > 0) lo = max(lo, (qpos / chunk) * chunk);  // blocks of `chunk` positions counted from the sequence's start
  const float inv_cap = softcap > 0.f ? 1.0f / softcap : 0.f;

  float* qs = q_smem + warp * d;
  const T* qsrc = q + ((size_t)t * nq + h) * d;
  for (int c = lane; c < d; c += 32) qs[c] = Elem<T>::load(qsrc + c);
  __syncwarp();

  float m = -INFINITY, l = 0.f;
  float acc[DI];
#pragma unroll
  for (int i = 0; i < DI; ++i) acc[i] = 0.f;

  const float r1 = dist_r1 ? dist_r1[h] : 0.f, r2 = dist_r1 ? dist_r2[h] : 0.f;
  const int lo_tile = (lo >> 5) << 5;
  // the kept first keys' tiles (those wholly before the window's first tile), then the window's tiles
  const int kept_end = keep_first > 0 ? min((keep_first + 31) & ~31, lo_tile) : 0;
  for (int tile = kept_end > 0 ? 0 : lo_tile; tile <= qpos; tile = (tile + 32 == kept_end) ? lo_tile : tile + 32) {
    const int kj = tile + lane;
    const bool valid = kj <= qpos && (kj >= lo || kj < keep_first);
    float s = -INFINITY;
    size_t base = 0;
    if (valid) {
      const int page = pages[kj >> page_shift];
      bool usable = page >= 0;
      if (!usable) atomicExch(status, 3);
      MS_DEBUG_ONLY(if (usable && (page >= num_pages || row < 0)) {
        atomicExch(status, 5);
        usable = false;
      })
      if (usable) {
        base = (((size_t)page * nkv + kvh) * page_size + (kj & (page_size - 1))) * d;
        const T* kr = k_pool + base;
        float dot = 0.f;
        for (int c = 0; c < d; ++c) dot = fmaf(qs[c], Elem<T>::load(kr + c), dot);
        s = dot * scale;
        if (softcap > 0.f) s = softcap * tanhf(s * inv_cap);
        if (dist_r1) s -= r1 * logf(1.0f + r2 * (float)(qpos - kj));
      }
    }
    const unsigned seen = __ballot_sync(0xffffffffu, s != -INFINITY);
    const float m_tile = warp_max(s);
    const float m_new = fmaxf(m, m_tile);
    const float alpha = (m == -INFINITY) ? 0.f : expf(m - m_new);
    const float p = (s == -INFINITY) ? 0.f : expf(s - m_new);
    l = l * alpha + warp_sum(p);
#pragma unroll
    for (int i = 0; i < DI; ++i) acc[i] *= alpha;
    const int j_lo = keep_first > tile ? 0 : max(lo - tile, 0), j_hi = min(qpos - tile, 31);
    for (int j = j_lo; j <= j_hi; ++j) {
      if (!((seen >> j) & 1u)) continue;  // (a key between the kept ones and the window, or one whose page is missing)
      const float pj = __shfl_sync(0xffffffffu, p, j);
      const unsigned long long bj = __shfl_sync(0xffffffffu, (unsigned long long)base, j);
      const T* vr = v_pool + bj;
#pragma unroll
      for (int i = 0; i < DI; ++i) {
        const int c = lane + 32 * i;
        if (c < d) acc[i] = fmaf(pj, Elem<T>::load(vr + c), acc[i]);
      }
    }
    m = m_new;
  }
  if (sink) {
    // one more term in the denominator, with no value: of score 0, or of the head's own learned score
    // (which is neither scaled nor squashed). A row that sees no key at all is then all sink: output 0.
    const float s0 = sink_values ? sink_values[h] : 0.f;
    const float m_all = fmaxf(m, s0);
    const float a = (m == -INFINITY) ? 0.f : expf(m - m_all);
    l = l * a + expf(s0 - m_all);
#pragma unroll
    for (int i = 0; i < DI; ++i) acc[i] *= a;
  }
  T* o = out + ((size_t)t * nq + h) * d;
#pragma unroll
  for (int i = 0; i < DI; ++i) {
    const int c = lane + 32 * i;
    if (c < d) Elem<T>::store(o + c, acc[i] / l);
  }
}

// ---------------------------------------------------------------- the same for prompts, ROWS query rows of a request at a time
// The arithmetic of every (token, head) is the one above, operation by operation (the same bits); what differs is who does it: a CTA
// takes ROWS query rows (tokens of one request times the query heads of a kv head) and walks the key tiles once for all of them, two tiles a
// step. A warp has 8 rows from the scores to the output: a lane 4 x 4 scores (of 64 keys), then the rows of both tiles at once with a lane per key
// (the same exchanges as above; the second tile goes on from the first one's maximum), then 4 rows x 2 MD columns of the output, tile by tile.
// A tile in which a row sees nothing leaves the row as it is (alpha = 1, p = 0), so all rows may walk the tiles that any of them sees.
// Keys and values have one buffer each: the next keys come by asynchronous copies while the values are summed, the next values beside the scores.
// Bound by a warp's chain of instructions (two CTAs a multiprocessor by shared memory, 1.7 warps a scheduler, 45 % of the issue slots), shared
// memory's reads at a third (32 floats read for 64 products of a score tile, 12 for 32 of the output). 700 tokens of 16 heads of 128 on 8 kv heads
// 102 us (4 warps of 16 rows, one tile a step, in the order of the grid: 255), 2048 tokens 580. On the way: 8 rows a warp and two tiles a step
// 146; softcap and distance out of the unrolled scores and the values' loop not unrolled over the tiles (instruction fetches) 124; the order
// of the grid 102.
constexpr int AR_ROWS = 64, AR_KEYS = 32, AR_LDS = 2 * AR_KEYS + 4;

__device__ __forceinline__ void ar_cp16(void* dst, const void* src, bool in) {
  const int bytes = in ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

// Folds 16 values over the lanes of a warp, all sixteen in one go: lane l comes back with the fold of v[ar_row(l)]. The pairs are those of
// the exchange by 16, 8, 4, 2, 1 that folds one value (warp_sum), so the result is the same bit for bit.
template <typename F>
__device__ __forceinline__ float ar_fold16(float (&v)[16], F fold) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int n = 8; n > 0; n >>= 1) {
    const bool up = lane & (2 * n);
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const float send = up ? v[i] : v[i + n], keep = up ? v[i + n] : v[i];
      v[i] = fold(keep, __shfl_xor_sync(0xffffffffu, send, 2 * n));
    }
  }
  return fold(v[0], __shfl_xor_sync(0xffffffffu, v[0], 1));
}
__device__ __forceinline__ unsigned long long ar_twice(float x) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ int ar_row(int lane) { return lane >> 1; }

template <int MD, int ROWS>  // head sizes of up to 32 MD, whole fours
__global__ void __launch_bounds__(ROWS * 4, 128 / (ROWS * 2))
attention_tiled_f32_kernel(float* __restrict__ out, const float* __restrict__ q, const float* __restrict__ k_pool, const float* __restrict__ v_pool,
                           const int* __restrict__ cu_q, const int* __restrict__ q_start, const int* __restrict__ page_indptr,
                           const int* __restrict__ page_indices, int num_rows, int nq, int nkv, int d, float scale, int window, int sink,
                           int page_shift, int num_pages, int* __restrict__ status, const float* __restrict__ sink_values, float softcap, int chunk,
                           const float* __restrict__ dist_r1, const float* __restrict__ dist_r2, int keep_first, int sms) {
  constexpr int LD = 32 * MD + 4, WARPS = ROWS / 8, MC = (MD + 1) / 2, MINE = 2 * AR_KEYS / WARPS;  // MINE: keys of a step that a warp stages
  static_assert(MINE <= 32);
  extern __shared__ __align__(16) float ar_smem[];
  float* qs = ar_smem;                  // [ROWS][LD]
  float* ks = qs + ROWS * LD;           // [64][LD]
  float* vs = ks + 2 * AR_KEYS * LD;    // [64][LD] (read to column 64 MC: what lies behind a row is not stored)
  float* ss = vs + 2 * AR_KEYS * LD;    // [ROWS][AR_LDS]
  float* alphas = ss + ROWS * AR_LDS;   // [2][ROWS]
  unsigned* seen = reinterpret_cast<unsigned*>(alphas + 2 * ROWS);  // [2][ROWS]
  __shared__ int s_row, s_tile;
  __shared__ int usable[2][2 * AR_KEYS];
  pdl_prologue(q, k_pool, v_pool, cu_q, q_start, page_indptr, page_indices, sink_values, dist_r1, dist_r2);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int group = nq / nkv, per_tile = ROWS / group;
  // The late (long) tiles first, all kv heads of one tile side by side; those that share a multiprocessor with the first `sms` the other way
  // round, so that the longest has the shortest of them beside it.
  const int place_in_grid = (int)blockIdx.x >= sms && (int)blockIdx.x < 2 * sms && 2 * sms <= (int)gridDim.x ? 3 * sms - 1 - (int)blockIdx.x : (int)blockIdx.x;
  const int kvh = place_in_grid % nkv;
  if (warp == 0) {  // which request and which of its tiles
    int want = (int)gridDim.x / nkv - 1 - place_in_grid / nkv, row = -1, base = 0;
    for (int r0 = 0; r0 < num_rows && row < 0; r0 += 32) {
      const int r = r0 + lane;
      const int mine = r < num_rows ? (cu_q[r + 1] - cu_q[r] + per_tile - 1) / per_tile : 0;
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += x;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, want < base + upto);
      if (hit) {
        const int at = __ffs(hit) - 1;
        row = r0 + at;
        want -= base + __shfl_sync(0xffffffffu, upto - mine, at);
      } else {
        base += __shfl_sync(0xffffffffu, upto, 31);
      }
    }
    if (lane == 0) {
      s_row = row;
      s_tile = want;
    }
  }
  __syncthreads();
  const int row = s_row;
  if (row < 0) return;
  const int t0 = cu_q[row] + s_tile * per_tile, n_tok = min(per_tile, cu_q[row + 1] - t0);
  const int pos0 = q_start[row] + s_tile * per_tile, pos_last = pos0 + n_tok - 1;
  const int rows = n_tok * group;  // of the ROWS
  const int* pages = page_indices + page_indptr[row];
  const int page_size = 1 << page_shift;
  const float inv_cap = softcap > 0.f ? 1.0f / softcap : 0.f;
  const bool extras = softcap > 0.f || dist_r1;
  auto first_key = [&](int pos) {
    int lo = window > 0 ? max(0, pos - window + 1) : 0;
    if (chunk > 0) lo = max(lo, (pos / chunk) * chunk);
    return lo;
  };
  const int see_first = first_key(pos0), lo_tile = (see_first >> 5) << 5;  // (the first token's window begins first)
  const int kept_end = keep_first > 0 ? min((keep_first + 31) & ~31, lo_tile) : 0;
  const int vec = d / 4;
  for (int idx = tid; idx < ROWS * vec; idx += ROWS * 4) {
    const int r = idx / vec, c = (idx - r * vec) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < rows) x = *reinterpret_cast<const float4*>(q + ((size_t)(t0 + r / group) * nq + kvh * group + r % group) * d + c);
    *reinterpret_cast<float4*>(qs + r * LD + c) = x;
  }
  auto next_tile = [&](int tile) { return tile + AR_KEYS == kept_end ? lo_tile : tile + AR_KEYS; };
  // Key `lane` of the warp's own MINE (warp * MINE + lane of the step's 64): its page, asked for a step ahead, and its place in the pools;
  // negative where there is none. Keys of the first tile that lie ahead of the first token's window are not looked up: the table begins with the page ahead of
  // the window's first, and a tile may begin further back.
  const int mine = warp * MINE + lane;
  auto key_of = [&](int a, int b) { return (mine < AR_KEYS ? a : b - AR_KEYS) + mine; };
  auto page_of = [&](int a, int b) {
    const int kj = key_of(a, b);
    return lane < MINE && kj <= pos_last && (kj >= see_first || kj < keep_first) ? pages[kj >> page_shift] : -1;
  };
  auto place_of = [&](int page, int a, int b) -> long long {
    MS_DEBUG_ONLY(if (page >= num_pages) {
      atomicExch(status, 5);
      return -1;
    })
    return page < 0 ? -1 : (((long long)page * nkv + kvh) * page_size + (key_of(a, b) & (page_size - 1))) * d;
  };
  auto stage = [&](float* to, const float* pool, long long place) {
    const int c = lane * 4;
#pragma unroll
    for (int j = 0; j < MINE; ++j) {
      const long long at = __shfl_sync(0xffffffffu, place, j);
      if (c < d) ar_cp16(to + (warp * MINE + j) * LD + c, pool + (at >= 0 ? at + c : 0), at >= 0);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };

  const int r0 = warp * 8;                    // the warp's rows
  const int rg = lane >> 4, kg = lane & 15;   // a lane's four rows r0 + 4 rg + i; its keys kg + 16 jj, its columns 4 kg + 64 m
  const bool second = lane >= 16;             // of the lane's fold: row r0 + own of the step's first or second tile
  const int own = ar_row(lane) & 7;
  const int row_last = min(r0 + 8, rows) - 1;
  const int see_all = pos0 + r0 / group, see_from = first_key(pos0 + row_last / group);  // keys see_from .. see_all are seen by all the warp's rows
  float m = -INFINITY, l = 0.f;               // of row r0 + own
  unsigned long long acc[4][MC][2];           // two columns each: fma.rn.f32x2 rounds each half as fmaf does
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int mm = 0; mm < MC; ++mm)
#pragma unroll
      for (int e = 0; e < 2; ++e) acc[i][mm][e] = 0ull;

  int tile = kept_end > 0 ? 0 : lo_tile, tile2 = next_tile(tile), after = next_tile(tile2), after2 = next_tile(after), buf = 0;
  long long place = place_of(page_of(tile, tile2), tile, tile2);
  if (lane < MINE) usable[0][mine] = place >= 0;
  stage(ks, k_pool, place);
  stage(vs, v_pool, place);
  int page = page_of(after, after2);
#pragma unroll 1
  for (; tile <= pos_last; buf ^= 1) {
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // the keys
    __syncthreads();
    if (r0 < rows) {
      float s[4][4] = {};
      const float* qp = qs + (r0 + 4 * rg) * LD;
#pragma unroll 4
      for (int c = 0; c < d; c += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float4*>(qp + i * LD + c);
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(ks + (kg + 16 * j) * LD + c);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            s[i][j] = fmaf(a[i].x, b[j].x, s[i][j]);
            s[i][j] = fmaf(a[i].y, b[j].y, s[i][j]);
            s[i][j] = fmaf(a[i].z, b[j].z, s[i][j]);
            s[i][j] = fmaf(a[i].w, b[j].w, s[i][j]);
          }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) ss[(r0 + 4 * rg + i) * AR_LDS + kg + 16 * j] = s[i][j];
    }
    __syncthreads();  // the keys' buffer is free
    place = place_of(page, after, after2);
    if (lane < MINE) usable[buf ^ 1][mine] = place >= 0;
    stage(ks, k_pool, place);
    const int later = next_tile(after2), later2 = next_tile(later);
    page = page_of(later, later2);
    unsigned hidden = 0;  // bit t: a row of the warp does not see all of tile t
    if (r0 < rows) {
      float sc[16];
      bool missing = false;
#pragma unroll
      for (int t = 0; t < 2; ++t) {
        const int begin = t ? tile2 : tile, kj = begin + lane;
        const bool there = kj <= pos_last && usable[buf][t * AR_KEYS + lane];
        float* st = ss + r0 * AR_LDS + t * AR_KEYS + lane;
        if (extras) {  // (by itself: beside the plain scores its instructions would be fetched past in every step)
#pragma unroll 1
          for (int i = 0; i < 8; ++i) {
            const int r = r0 + i, h = kvh * group + r % group;
            if (r >= rows) break;
            float x = st[i * AR_LDS] * scale;
            if (softcap > 0.f) x = softcap * tanhf(x * inv_cap);
            if (dist_r1) x -= dist_r1[h] * logf(1.0f + dist_r2[h] * (float)(pos0 + r / group - kj));
            st[i * AR_LDS] = x;
          }
        }
        const float times = extras ? 1.f : scale;
        if (begin + AR_KEYS - 1 <= see_all && begin >= see_from) {
          missing = missing || !there;
#pragma unroll
          for (int i = 0; i < 8; ++i) sc[8 * t + i] = there ? st[i * AR_LDS] * times : -INFINITY;
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int r = r0 + i, qpos = pos0 + r / group;
            const bool sees = r < rows && kj <= qpos && (kj >= first_key(qpos) || kj < keep_first);
            missing = missing || (sees && !there);
            sc[8 * t + i] = sees && there ? st[i * AR_LDS] * times : -INFINITY;
          }
        }
        bool all_see = true;
#pragma unroll
        for (int i = 0; i < 8; ++i) all_see = all_see && (r0 + i >= rows || sc[8 * t + i] != -INFINITY);
        if (!__all_sync(0xffffffffu, all_see)) {
          hidden |= 1u << t;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const unsigned mask = __ballot_sync(0xffffffffu, sc[8 * t + i] != -INFINITY);
            if (lane == i) seen[t * ROWS + r0 + i] = mask;
          }
        }
      }
      if (missing) atomicExch(status, 3);
      float v[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) v[i] = sc[i];
      const float top = ar_fold16(v, [](float x, float y) { return fmaxf(x, y); }), other = __shfl_xor_sync(0xffffffffu, top, 16);
      const float m_first = fmaxf(m, second ? other : top), m_second = fmaxf(m_first, second ? top : other);
      const float before = second ? m_first : m, m_new = second ? m_second : m_first;
      const float alpha = (before == -INFINITY) ? 0.f : expf(before - m_new);
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const float mi = __shfl_sync(0xffffffffu, m_new, 2 * i);
        v[i] = (sc[i] == -INFINITY) ? 0.f : expf(sc[i] - mi);
        ss[(r0 + (i & 7)) * AR_LDS + (i >> 3) * AR_KEYS + lane] = v[i];
      }
      const float sum = ar_fold16(v, [](float x, float y) { return x + y; });
      const float l_first = __shfl_sync(0xffffffffu, l * alpha + sum, lane & 15);
      l = __shfl_sync(0xffffffffu, l_first * alpha + sum, lane | 16);
      m = m_second;
      if (!(lane & 1)) alphas[(second ? ROWS : 0) + r0 + own] = alpha;
    }
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // the values
    __syncthreads();
    if (r0 < rows) {
#pragma unroll 1
      for (int t = 0; t < 2; ++t) {
        if (t == 1 && tile2 > pos_last) break;
        unsigned mk[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int r = t * ROWS + r0 + 4 * rg + i;
          mk[i] = (hidden >> t) & 1u ? seen[r] : 0xffffffffu;
          const unsigned long long twice = ar_twice(alphas[r]);
#pragma unroll
          for (int mm = 0; mm < MC; ++mm)
#pragma unroll
            for (int e = 0; e < 2; ++e) asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(acc[i][mm][e]) : "l"(twice));
        }
        const float* pr = ss + (r0 + 4 * rg) * AR_LDS + t * AR_KEYS;
        const float* vt = vs + t * AR_KEYS * LD + 4 * kg;
        auto values = [&](auto whole) {
#pragma unroll 2
          for (int j0 = 0; j0 < AR_KEYS; j0 += 4) {
            float4 p[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) p[i] = *reinterpret_cast<const float4*>(pr + i * AR_LDS + j0);
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
              ulonglong2 v[MC];
#pragma unroll
              for (int mm = 0; mm < MC; ++mm) v[mm] = *reinterpret_cast<const ulonglong2*>(vt + (j0 + jj) * LD + 64 * mm);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const float pj = jj == 0 ? p[i].x : jj == 1 ? p[i].y : jj == 2 ? p[i].z : p[i].w;
                // (a key that a row does not see may hold anything: the row's sums must not meet it)
                if (whole.value || ((mk[i] >> (j0 + jj)) & 1u)) {
                  const unsigned long long twice = ar_twice(pj);
#pragma unroll
                  for (int mm = 0; mm < MC; ++mm) {
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][mm][0]) : "l"(twice), "l"(v[mm].x));
                    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc[i][mm][1]) : "l"(twice), "l"(v[mm].y));
                  }
                }
              }
            }
          }
        };
        if ((hidden >> t) & 1u) values(std::false_type());
        else values(std::true_type());
      }
    }
    __syncthreads();  // the values' buffer is free
    stage(vs, v_pool, place);
    tile = after;
    tile2 = after2;
    after = later;
    after2 = later2;
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  if (r0 >= rows) return;
  if (lane < 16) {  // the sink's term of the lane's row, as above
    const int r = r0 + own;
    float a = 1.f;
    if (sink) {
      const float s0 = sink_values ? sink_values[kvh * group + r % group] : 0.f;
      const float m_all = fmaxf(m, s0);
      a = (m == -INFINITY) ? 0.f : expf(m - m_all);
      l = l * a + expf(s0 - m_all);
    }
    if (!(lane & 1)) {
      alphas[r] = a;
      ss[r * AR_LDS] = l;
    }
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = r0 + 4 * rg + i;
    if (r >= rows) continue;
    const float a = alphas[r], sum = ss[r * AR_LDS];
    float* o = out + ((size_t)(t0 + r / group) * nq + kvh * group + r % group) * d;
#pragma unroll
    for (int mm = 0; mm < MC; ++mm) {
      const int c = 4 * kg + 64 * mm;
      if (c < d) {
        float4 x;
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x.x), "=f"(x.y) : "l"(acc[i][mm][0]));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(x.z), "=f"(x.w) : "l"(acc[i][mm][1]));
        if (sink) {
          x.x *= a; x.y *= a; x.z *= a; x.w *= a;
        }
        x.x /= sum; x.y /= sum; x.z /= sum; x.w /= sum;
        *reinterpret_cast<float4*>(o + c) = x;
      }
    }
  }
}

}  // namespace ms

using namespace ms;

MS_EXPORT int ms_attention_rowwise(void* out, const void* q, const void* k_pool, const void* v_pool,
                                   const int* positions, const int* row_of_token, const int* page_indptr,
                                   const int* page_indices, int num_tokens, int nq, int nkv, int head_dim, float scale,
                                   int window, int sink, int page_size, int num_pages, int* status, int dtype, cudaStream_t stream,
                                   const float* sink_values, float softcap, int chunk, const float* dist_r1, const float* dist_r2,
                                   int keep_first) {
  if (num_tokens == 0) return 0;
  MS_CHECK_ARG(keep_first >= 0 && (dist_r1 == nullptr) == (dist_r2 == nullptr), "attention: keep_first=%d, and both numbers of a distance bias",
               keep_first);
  MS_CHECK_ARG(softcap >= 0.f && chunk >= 0, "attention: softcap=%g and chunk=%d must not be negative", softcap, chunk);
  MS_CHECK_ARG(nq > 0 && nkv > 0 && nq % nkv == 0, "attention: %d query heads are not a multiple of %d kv heads", nq, nkv);
  MS_CHECK_ARG(head_dim > 0 && head_dim <= ROWWISE_MAX_D, "attention: head_dim=%d is outside 1..%d", head_dim, ROWWISE_MAX_D);
  MS_CHECK_ARG(page_size > 0 && (page_size & (page_size - 1)) == 0, "attention: page_size=%d must be a power of two", page_size);
  int page_shift = 0;
  while ((1 << page_shift) < page_size) ++page_shift;
  const int warps = 4;
  const long long items = (long long)num_tokens * nq;
  const unsigned blocks = (unsigned)((items + warps - 1) / warps);
  const size_t smem = (size_t)warps * head_dim * sizeof(float);
#define MS_ROWWISE_LAUNCH(T, DI)                                                                                        \
  MS_LAUNCH((attention_rowwise_kernel<T, DI>), blocks, warps * 32, smem, stream, (T*)out, (const T*)q, (const T*)k_pool,  \
            (const T*)v_pool, positions, row_of_token, page_indptr, page_indices, num_tokens, nq, nkv, head_dim, scale,   \
            window, sink, page_shift, num_pages, status, sink_values, softcap, chunk, dist_r1, dist_r2, keep_first)
  if (dtype == MS_F32) {
    if (head_dim <= 256) MS_ROWWISE_LAUNCH(float, 8);
    else MS_ROWWISE_LAUNCH(float, 16);
  } else {
    if (head_dim <= 256) MS_ROWWISE_LAUNCH(__nv_bfloat16, 8);
    else MS_ROWWISE_LAUNCH(__nv_bfloat16, 16);
  }
#undef MS_ROWWISE_LAUNCH
  return 0;
}

// 1 if ms_attention_tiled_f32 takes these sizes: head sizes of whole fours up to 128, groups of up to 64 query heads.
MS_EXPORT int ms_attention_tiled_f32_supports(int head_dim, int nq, int nkv) {
  return head_dim >= 4 && head_dim <= 128 && head_dim % 4 == 0 && nkv > 0 && nq % nkv == 0 && nq / nkv <= AR_ROWS && nkv <= 65535;
}

// ms_attention_rowwise for float32 and a step of whole rows: cu_q [rows + 1], q_start [rows]. The same results, bit for bit.
MS_EXPORT int ms_attention_tiled_f32(float* out, const float* q, const float* k_pool, const float* v_pool, const int* cu_q, const int* q_start,
                                     const int* page_indptr, const int* page_indices, int num_tokens, int num_rows, int nq, int nkv, int head_dim,
                                     float scale, int window, int sink, int page_size, int num_pages, int* status, cudaStream_t stream,
                                     const float* sink_values, float softcap, int chunk, const float* dist_r1, const float* dist_r2, int keep_first) {
  if (num_tokens == 0) return 0;
  MS_CHECK_ARG(ms_attention_tiled_f32_supports(head_dim, nq, nkv), "attention: %d/%d heads of %d", nq, nkv, head_dim);
  MS_CHECK_ARG(keep_first >= 0 && (dist_r1 == nullptr) == (dist_r2 == nullptr), "attention: keep_first=%d, and both numbers of a distance bias",
               keep_first);
  MS_CHECK_ARG(softcap >= 0.f && chunk >= 0, "attention: softcap=%g and chunk=%d must not be negative", softcap, chunk);
  MS_CHECK_ARG(page_size > 0 && (page_size & (page_size - 1)) == 0, "attention: page_size=%d must be a power of two", page_size);
  MS_CHECK_ARG((uintptr_t)q % 16 == 0 && (uintptr_t)k_pool % 16 == 0 && (uintptr_t)v_pool % 16 == 0 && (uintptr_t)out % 16 == 0,
               "attention: operands must start on 16 bytes");
  int page_shift = 0;
  while ((1 << page_shift) < page_size) ++page_shift;
#define MS_TILED_LAUNCH(MD, ROWS)                                                                                                               \
  do {                                                                                                                                          \
    auto kernel = attention_tiled_f32_kernel<MD, ROWS>;                                                                                         \
    constexpr size_t smem = ((ROWS + 4 * AR_KEYS) * (32 * MD + 4) + ROWS * AR_LDS + 4 * ROWS) * 4;                                              \
    static std::atomic<unsigned long long> allowed{0};                                                                                          \
    MS_CHECK_CUDA(allow_shared_memory((const void*)kernel, (int)smem, allowed));                                                                \
    const long long grid = ((long long)num_tokens / (ROWS / (nq / nkv)) + num_rows) * nkv;                                                      \
    MS_CHECK_ARG(grid <= 0x7fffffffll, "attention: %d tokens of %d kv heads are too many for one launch", num_tokens, nkv);                     \
    MS_LAUNCH_APART(kernel, (unsigned)grid, ROWS * 4, smem, stream, out, q, k_pool, v_pool, cu_q, q_start, page_indptr, page_indices, num_rows, nq, nkv,  \
                    head_dim, scale, window, sink, page_shift, num_pages, status, sink_values, softcap, chunk, dist_r1, dist_r2, keep_first,    \
                    ROWS == 32 ? sms : 1 << 29);                                                                                                \
  } while (0)
#define MS_TILED_ROWS(MD)                     \
  do {                                        \
    if (small) MS_TILED_LAUNCH(MD, 32);       \
    else MS_TILED_LAUNCH(MD, 64);             \
  } while (0)
  const int group = nq / nkv, known = sm_count(), sms = known > 0 ? known : 148;
  // 64 rows only where 32 would leave more of them without a token (one CTA a multiprocessor then, and twice the chain): 700 tokens of 16 heads
  // of 128 on 8 kv heads 146 us at 32 rows, 158 at 64, both in the plain order of the grid; 100 tokens behind 1000 170 / 228.
  const bool small = group <= 32 && 2 * (32 / group) >= 64 / group;
  if (head_dim <= 32) MS_TILED_ROWS(1);
  else if (head_dim <= 64) MS_TILED_ROWS(2);
  else MS_TILED_ROWS(4);
#undef MS_TILED_ROWS
#undef MS_TILED_LAUNCH
  return 0;
}
