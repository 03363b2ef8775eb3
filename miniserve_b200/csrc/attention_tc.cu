// Causal grouped-query attention for prompts and mixed steps on the 5th-generation tensor cores,
// for head size 128 and bfloat16: S = Q K^T and O += P V are tcgen05.mma instructions with the
// accumulators in tensor memory, operands staged by TMA straight out of the paged cache.
//
// Formula as in attention_bf16.cu (miniserve/model/attention.py:60-67,125-133): a query row at
// absolute position p sees keys 0..p of its request (or the last `window`), query head h reads kv
// head h / (heads / kv_heads), softmax in float32 with scale head_dim^-0.5.
//
// One CTA owns 256 query rows in two groups of 128 (G query heads of one kv head x 128/G
// consecutive tokens each), so that every K/V tile is fetched once for all of them. Thread r of a
// softmax group owns row r (tensor-memory lane r): per key tile it reads its row of S with
// tcgen05.ld, masks it if the tile touches the diagonal, a window's edge or the request's end,
// keeps a running maximum and sum, stores P (bfloat16) back into tensor memory, and rescales O
// only when the maximum has grown by more than 2^8 (the stale maximum is exact in the end because
// the same one scales the sum).
// Every mbarrier wait is bounded; on a timeout the kernel raises the status word and winds down.
#include <climits>

#include "common.cuh"
#include "tensor_map.cuh"

namespace ms {

constexpr int AT_D = 128, AT_ROWS = 128, AT_KEYS = 128;
constexpr int AT_FIRST = 96;  // so many of a tile's probabilities are handed over before the rest
constexpr float AT_LOG2E = 1.4426950408889634f;
constexpr int AT_BLOCK = 128 * 64 * 2;  // one [128 rows][64 bf16] swizzled block: 16 KB

__device__ __forceinline__ uint32_t at_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void at_mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(at_smem(bar)), "r"(count));
}
__device__ __forceinline__ void at_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(at_smem(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void at_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(at_smem(bar)) : "memory");
}
__device__ __forceinline__ bool at_wait(uint64_t* bar, uint32_t parity) { return mbar_wait_bounded(at_smem(bar), parity); }
__device__ __forceinline__ void at_tma_3d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
      ::"r"(at_smem(dst)), "l"(map), "r"(at_smem(bar)), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
__device__ __forceinline__ bool at_elect() {
  uint32_t pred;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(pred));
  return pred != 0;
}
// Shared-memory matrix descriptor, 128-byte swizzle: leading / stride byte offsets in bytes.
__device__ __forceinline__ uint64_t at_desc(const void* tile, uint32_t lbo, uint32_t sbo) {
  uint64_t d = (uint64_t)((at_smem(tile) & 0x3FFFF) >> 4);
  d |= (uint64_t)(lbo >> 4) << 16;
  d |= (uint64_t)(sbo >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}
__device__ __forceinline__ void at_mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void at_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(at_smem(bar)) : "memory");
}
__device__ __forceinline__ void at_tmem_ld32(uint32_t taddr, float (&r)[32]) {
  uint32_t* u = reinterpret_cast<uint32_t*>(r);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]), "=r"(u[8]),
        "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15]), "=r"(u[16]),
        "=r"(u[17]), "=r"(u[18]), "=r"(u[19]), "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]),
        "=r"(u[25]), "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
      : "r"(taddr));
}
__device__ __forceinline__ void at_tmem_st32(uint32_t taddr, const float (&r)[32]) {
  const uint32_t* u = reinterpret_cast<const uint32_t*>(r);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};\n"
      ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]),
        "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15]), "r"(u[16]), "r"(u[17]),
        "r"(u[18]), "r"(u[19]), "r"(u[20]), "r"(u[21]), "r"(u[22]), "r"(u[23]), "r"(u[24]), "r"(u[25]), "r"(u[26]),
        "r"(u[27]), "r"(u[28]), "r"(u[29]), "r"(u[30]), "r"(u[31])
      : "memory");
}
__device__ __forceinline__ float at_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
  return y;
}
// The larger of three; two multiply-adds and two sums in one instruction (the same roundings as one by one).
__device__ __forceinline__ float at_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ void at_fma2(float& x0, float& x1, float a0, float a1, float b, float c) {
  asm("{\n\t.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %4};\n\tmov.b64 c, {%5, %5};\n\t"
      "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;\n\t}\n"
      : "=f"(x0), "=f"(x1) : "f"(a0), "f"(a1), "f"(b), "f"(c));
}
__device__ __forceinline__ void at_add2(float& x0, float& x1, float a0, float a1) {
  asm("{\n\t.reg .b64 a, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 d, {%0, %1};\n\tadd.rn.f32x2 d, d, a;\n\tmov.b64 {%0, %1}, d;\n\t}\n"
      : "+f"(x0), "+f"(x1) : "f"(a0), "f"(a1));
}
#define AT_FENCE_BEFORE() asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory")
#define AT_FENCE_AFTER() asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory")

// D float32, A and B bfloat16, 128 x 128; b_mn: B is MN-major (V: [key][d] with d contiguous).
__host__ __device__ constexpr uint32_t at_idesc(bool b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? (1u << 16) : 0u) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// The kernel: 256 query rows per CTA as two groups of 128 that take turns on the tensor cores.
// Both groups (A: tokens m0 .. m0+tpc-1, B: the next tpc tokens; G heads each) attend over the
// same K/V tiles, so every tile is fetched once for twice the rows. While group A's softmax
// warps work on tile j, the tensor cores run group B's products, and the other way round. P never
// goes through shared memory: the softmax threads store it (bfloat16, two per 32-bit column) into
// the tensor-memory columns its S tile occupied, and the second product takes its A operand from
// there. Tensor memory: S/P of A [0,128), S/P of B [128,256), O of A [256,384), O of B [384,512).
// Warps 0-3: softmax A, 4-7: softmax B, 8: TMA, 9: MMA, 10-11: idle (registers are handed over by groups of four warps).
//
// Every role walks the CTA's items with counters of its own that run on from item to item, so nothing stops at an
// item's end: while a group writes its rows out of tensor memory, the tensor cores work on the other group or on the
// next item's first scores, and the next item's queries and keys are on their way. K and V have a ring of two tiles
// each with barriers of their own: K of a tile is free as soon as both groups' scores of it are done, V a softmax later.
// A copy brings a whole page of one head (4 KB at 16 tokens), both halves of its rows.
//
// What bounds it: per tile of 128 keys both groups have 4,096 cycles of tensor-core work at cuBLAS's rate (32 products of
// 128x128x16), 2,048 of ex2 in the special-function unit and about 1,100 of issue, in two chains S -> softmax -> P V that
// each wait for themselves. Measured (one B200, 16 heads of 8 kv heads, pages of 16, us for 512 / 2,048 / 4,096 / 8,192
// tokens): 20.6 / 38.1 / 96 / 333 with barriers armed anew at every item and one barrier for K and V of a tile;
// 17.4 / 34.7 / 78 / 261 as it is described above; 16.5 / 32.7 / 72 / 242 with two multiply-adds or sums an
// instruction; 15.9 / 32.2 / 67 / 229 with the first three quarters of P handed over before the last (a quarter: 233 at
// 8,192, half: 230). 8,192 tokens: 1,203 TFLOP/s. A share of the exponentials on the FMA pipes instead was slower (250 against
// 242), as were fewer or more registers for the two issuing warps than 104 (56: 620 bytes of spills there).
constexpr int AT_THREADS = 384;  // 8 softmax warps, 1 TMA warp, 1 MMA warp, 2 warps that only make up the third group of four

struct AtSmem {
  static constexpr int q = 0;                     // group A: 2 blocks, group B: 2 blocks
  static constexpr int slot = 2 * AT_BLOCK;       // a tile of K or V: [16 groups of 8 keys][2 halves of a row][8 keys][64]
  static constexpr int k = 4 * AT_BLOCK;          // 2 slots
  static constexpr int v = k + 2 * slot;          // 2 slots
  static constexpr int total = v + 2 * slot;      // 12 blocks = 192 KB
};
constexpr int AT_GROUP8 = 2048;                   // 8 keys: two swizzled blocks [8 rows][64 bf16], one per half of a row

__device__ __forceinline__ void at_mma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, bool accumulate) {
  const uint32_t acc = accumulate ? 1u : 0u;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n"
      ::"r"(tmem_d), "r"(tmem_a), "l"(db), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void at_tmem_st16(uint32_t taddr, const uint32_t (&u)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
      ::"r"(taddr), "r"(u[0]), "r"(u[1]), "r"(u[2]), "r"(u[3]), "r"(u[4]), "r"(u[5]), "r"(u[6]), "r"(u[7]), "r"(u[8]),
        "r"(u[9]), "r"(u[10]), "r"(u[11]), "r"(u[12]), "r"(u[13]), "r"(u[14]), "r"(u[15])
      : "memory");
}

// eight float32 scaled by `inv`, as eight bfloat16
__device__ __forceinline__ uint4 at_pack8(const float* v, float inv) {
  __nv_bfloat162 p0 = __floats2bfloat162_rn(v[0] * inv, v[1] * inv), p1 = __floats2bfloat162_rn(v[2] * inv, v[3] * inv);
  __nv_bfloat162 p2 = __floats2bfloat162_rn(v[4] * inv, v[5] * inv), p3 = __floats2bfloat162_rn(v[6] * inv, v[7] * inv);
  uint4 pk;
  pk.x = *reinterpret_cast<uint32_t*>(&p0);
  pk.y = *reinterpret_cast<uint32_t*>(&p1);
  pk.z = *reinterpret_cast<uint32_t*>(&p2);
  pk.w = *reinterpret_cast<uint32_t*>(&p3);
  return pk;
}
// barriers of one softmax group (128 threads, hardware barrier `id`): plain, and with an OR over a flag
__device__ __forceinline__ void at_group_sync(int id) { asm volatile("bar.sync %0, 128;\n" ::"r"(id) : "memory"); }
__device__ __forceinline__ bool at_group_any(int id, bool flag) {
  uint32_t res;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %2, 0;\n\t"
      "bar.red.or.pred q, %1, 128, p;\n\tselp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(res) : "r"(id), "r"((uint32_t)flag) : "memory");
  return res != 0;
}

// What an attention may have beyond scale, window and a sink of score 0: the score of each head's sink, a cap on
// the scores and a mask by blocks of positions (the block size travels in AtGrid, with the window). The cap works on
// the raw products, before the scale: s' = (cap / scale) tanh(s scale / cap), so that s' scale is the capped score
// and everything after it is as without a cap. tanh(y) = 1 - 2 / (1 + 2^(2 y log2 e)), absolute error about 1e-6.
struct AtExtras {
  const float* sink_values;  // [nq] or null
  float cap_raw;             // cap / scale
  float cap_c2;              // 2 log2(e) scale / cap; 0: no cap
  // a distance bias: r1_h ln(1 + r2_h (i - j)) is taken off the scaled score of query i and key j; in the raw
  // products' units that is (r1_h / (scale log2 e)) log2(1 + r2_h (i - j)). [nq] each, or null.
  const float* dist_r1;
  const float* dist_r2;
};
// the distance bias of the key `distance` positions behind the query, in the raw products' units
__device__ __forceinline__ float at_distance(float c_raw, float r2, int distance) {
  return c_raw * __log2f(fmaf(r2, (float)distance, 1.0f));
}
__device__ __forceinline__ float at_cap(float s, float cap_raw, float cap_c2) {
  return cap_raw * (1.f - __fdividef(2.f, 1.f + at_ex2(s * cap_c2)));
}

// A new running maximum for a row: the stale one is kept while the new one exceeds it by at most
// 2^8 after scaling (the same maximum scales the sum, so the result stays exact); returns the factor
// that what was accumulated so far has to be scaled by (1: nothing to do).
__device__ __forceinline__ float at_new_maximum(float m_tile, float& m_used, float scale_log2) {
  const float m_new = fmaxf(m_used, m_tile);
  if (m_used == -INFINITY) {
    m_used = m_new;
  } else if ((m_new - m_used) * scale_log2 > 8.f) {
    const float alpha = at_ex2((m_used - m_new) * scale_log2);
    m_used = m_new;
    return alpha;
  }
  return 1.f;
}
// O *= alpha for this thread's row. Called when S(j) is complete, so the product P(j-1) V(j-1) issued
// before it is complete too: O is quiet.
__device__ __forceinline__ void at_rescale(uint32_t t_o, float alpha) {
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    float ov[32];
    at_tmem_ld32(t_o + (uint32_t)(c * 32), ov);
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) ov[i] *= alpha;
    at_tmem_st32(t_o + (uint32_t)(c * 32), ov);
  }
}
// The softmax step of one row for a tile in which the row sees only the keys at offsets
// [seen_lo, seen_hi], with what EXTRAS brings. The scores are read twice, 32 columns at a time: once for the
// maximum, once for the exponentials (chunk c of P, 16 columns, lies below chunk c + 1 of S, so chunks are read
// and written in turn). A function of its own: inlined beside the all-in-registers form of interior tiles it cost
// that form its registers. (Without extras a mask is one select per score, made in registers at the call's place.)
// Returns the sum of the row's exponentials.
// `keep_off`: offsets below it are seen whatever seen_lo says (the kept first keys of a request). `dist_c`, `dist_r2`,
// `dist_0`: the distance bias's factor in raw units (0: none), its second number, and the distance of offset 0.
__device__ __noinline__ float at_softmax_masked(uint32_t t_s, uint32_t t_o, int seen_lo, int seen_hi, float scale_log2,
                                                float& m_used, float& l_sum, float cap_raw, float cap_c2, int keep_off,
                                                float dist_c, float dist_r2, int dist_0) {
  float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    float v[32];
    at_tmem_ld32(t_s + (uint32_t)(c * 32), v);
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const int off = c * 32 + i;
      float sc = cap_c2 > 0.f ? at_cap(v[i], cap_raw, cap_c2) : v[i];
      const bool seen = off <= seen_hi && (off >= seen_lo || (off < keep_off));
      if (dist_c != 0.f && seen) sc -= at_distance(dist_c, dist_r2, dist_0 - off);
      mx[i & 3] = fmaxf(mx[i & 3], seen ? sc : -INFINITY);
    }
  }
  const float alpha = at_new_maximum(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), m_used, scale_log2);
  if (__any_sync(0xffffffffu, alpha != 1.f)) {
    at_rescale(t_o, alpha);
    l_sum *= alpha;
  }
  const float m_sub = (m_used == -INFINITY ? 0.f : m_used) * scale_log2;
  float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
  for (int c = 0; c < 4; ++c) {
    float v[32];
    at_tmem_ld32(t_s + (uint32_t)(c * 32), v);
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
    uint32_t pk[16];
    if (cap_c2 > 0.f) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = at_cap(v[i], cap_raw, cap_c2);
    }
#pragma unroll
    for (int i = 0; i < 32; i += 2) {
      const int off = c * 32 + i;
      const bool seen0 = off <= seen_hi && (off >= seen_lo || (off < keep_off));
      const bool seen1 = off + 1 <= seen_hi && (off + 1 >= seen_lo || (off + 1 < keep_off));
      if (dist_c != 0.f) {
        if (seen0) v[i] -= at_distance(dist_c, dist_r2, dist_0 - off);
        if (seen1) v[i + 1] -= at_distance(dist_c, dist_r2, dist_0 - off - 1);
      }
      const float e0 = seen0 ? at_ex2(fmaf(v[i], scale_log2, -m_sub)) : 0.f;
      const float e1 = seen1 ? at_ex2(fmaf(v[i + 1], scale_log2, -m_sub)) : 0.f;
      part[(i >> 1) & 3] += e0 + e1;
      __nv_bfloat162 p2 = __floats2bfloat162_rn(e0, e1);
      pk[i >> 1] = *reinterpret_cast<uint32_t*>(&p2);
    }
    at_tmem_st16(t_s + (uint32_t)(c * 16), pk);
  }
  return (part[0] + part[1]) + (part[2] + part[3]);
}

// What one work item (a tile of 2 x 128 query rows, one group of heads, one split of the keys)
// has to do. The scheduler warp finds it from the item's number and hands it to the other roles
// through a ring of two in shared memory.
struct AtItem {
  int r, tile, tok0, q_len, m0, start, kv_len, head0, split;
  int n_tiles[2], q_first[2], q_last[2], lo_g[2], lo_max[2], shares[2];
  int tile_begin, n_all;
  // Kept first keys: the walk over key tiles runs over virtual tiles; those below `first_tile` (the window's first
  // tile) are the request's tiles 0, 1, ... that hold kept keys: virtual tile v is real tile v - walk_shift there.
  int first_tile, walk_shift;
  int has_b, alive;  // alive 0: no item, the CTA is done
  __device__ __forceinline__ int real_tile(int v) const { return v < first_tile ? v - walk_shift : v; }
};

struct AtGrid {
  int q_tiles, rows, head_groups, splits, max_tiles_per_item, window, G;
  int chunk;  // > 0: a query sees only keys from the start of its own block of this many positions on
  int keep;   // > 0: the first `keep` keys of a request stay visible behind the window (the cache keeps their pages)
};

// Tile `tile` of row r for one group of heads, its keys whole: how many key tiles that are (0: the row has no such tile).
__device__ __forceinline__ int at_tile(AtItem& it, int r, int tile, const AtGrid& gr, const int* __restrict__ cu_q, const int* __restrict__ q_start) {
  const int tpc = AT_ROWS / gr.G;  // tokens per group
  it.r = r;
  it.tile = tile;
  it.tok0 = behind_load(cu_q + r);
  it.q_len = behind_load(cu_q + r + 1) - it.tok0;
  it.m0 = tile * 2 * tpc;
  if (tile < 0 || it.m0 >= it.q_len) return 0;
  it.start = behind_load(q_start + r);
  it.kv_len = it.start + it.q_len;
  // per group: the key tiles it needs (B needs at least as many as A; B may have no rows at all)
  it.has_b = it.m0 + tpc < it.q_len;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    it.q_first[g] = it.start + it.m0 + g * tpc;
    it.q_last[g] = it.start + min(it.m0 + (g + 1) * tpc, it.q_len) - 1;
    it.lo_g[g] = gr.window > 0 ? max(0, it.q_first[g] - gr.window + 1) : 0;
    it.lo_max[g] = gr.window > 0 ? max(0, it.q_last[g] - gr.window + 1) : 0;
    if (gr.chunk > 0) {  // the first query's block starts earliest, the last query's latest
      it.lo_g[g] = max(it.lo_g[g], (it.q_first[g] / gr.chunk) * gr.chunk);
      it.lo_max[g] = max(it.lo_max[g], (it.q_last[g] / gr.chunk) * gr.chunk);
    }
  }
  it.first_tile = it.lo_g[0] / AT_KEYS;
  it.walk_shift = it.first_tile - (gr.keep > 0 ? min((gr.keep + AT_KEYS - 1) / AT_KEYS, it.first_tile) : 0);
  it.tile_begin = it.walk_shift;
  it.n_tiles[0] = (min(it.kv_len, it.q_last[0] + 1) + AT_KEYS - 1) / AT_KEYS - it.tile_begin;
  it.n_tiles[1] = it.has_b ? (min(it.kv_len, it.q_last[1] + 1) + AT_KEYS - 1) / AT_KEYS - it.tile_begin : 0;
  return max(it.n_tiles[0], it.n_tiles[1]);
}
// Key ranges longer than `max_tiles_per_item` are cut into pieces of that length (the last one
// shorter; measured faster than equal pieces, whose items all start late in the queue's order)
// that are items of their own, at most `splits` of them. A group whose keys lie in more than one piece leaves a partial result
// (unnormalised O, the maximum it is scaled by, the sum), and the last of them to finish adds
// the partial results up in the order of the pieces.
__device__ __forceinline__ int at_piece_tiles(int n_full, const AtGrid& gr) { return max(gr.max_tiles_per_item, (n_full + gr.splits - 1) / gr.splits); }
// Piece `split` of the tile: what at_tile left, cut down to it.
__device__ __forceinline__ void at_piece(AtItem& it, int head0, int split, int per_split) {
  it.head0 = head0;
  it.split = split;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    it.shares[g] = (it.n_tiles[g] + per_split - 1) / per_split;  // in how many splits the group has keys
    it.n_tiles[g] = min(max(it.n_tiles[g] - split * per_split, 0), per_split);
  }
  it.tile_begin += split * per_split;
  it.n_all = max(it.n_tiles[0], it.n_tiles[1]);
}

// The order of the items is the longest first, so that the short ones even out the end. Where rows begin at different positions, tiles are ranked by
// the position of their last key over all rows (rank 0 ends at pos_max; a row has one tile in each rank, while it has any), and all whole pieces of cut
// key ranges come before the last pieces and the tiles that are not cut; the scheduler counts items along the pairs (rank, row). With every row ranked by
// itself a portion of 900 tokens behind 4,096 had its last items of 28 tiles begin when its neighbours of 1,531 and 517 tokens were done: 89 us for
// the three, 68 now; four rows of 17 to 900 tokens behind 0 to 4,096 84 -> 63. Counting takes half a microsecond for 32 pairs, once a CTA, so
// rows that begin alike (whose order it would not change) and steps of many pairs are numbered by place: a tile's rank is its distance from the longest
// row's last one, then row, head group, split, empty ones among them. Us by place / by position: 2 rows behind 5,102 and 6,076 65 / 59, 4 behind 3,030
// to 3,860 82 / 68, 8 behind up to 3,000 46 / 42, 16 behind up to 2,000 45 / 44 and up to 4,000 86 / 87, 32 behind up to 1,500 42 / 50, 64 behind up to
// 1,000 57 / 74 and up to 3,000 107 / 156, 100 behind up to 3,000 152 / 235. The bound on the pairs lies where the two meet for 16 rows; it also leaves
// two rows that begin more than 16,384 positions apart by place, where by position they would take less (0 and 20,000 110 / 107, 1,024 and 24,000 113 / 102).
struct AtOrder {
  int pairs, pos_max;  // ranks x rows (0: by place)
};
constexpr int AT_MOST_PAIRS = 256;
__device__ __forceinline__ AtOrder at_order(const AtGrid& gr, const int* __restrict__ cu_q, const int* __restrict__ q_start, int lane) {
  if (gr.rows < 2 || gr.rows > AT_MOST_PAIRS / 2) return {0, 0};
  const int span = 2 * (AT_ROWS / gr.G);
  int last = 0, first = INT_MAX, latest = 0;
  for (int r = lane; r < gr.rows; r += 32) {
    const int len = behind_load(cu_q + r + 1) - behind_load(cu_q + r), start = behind_load(q_start + r);
    if (len > 0) {
      last = max(last, start + (len + span - 1) / span * span);
      first = min(first, start);
      latest = max(latest, start);
    }
  }
  last = __reduce_max_sync(0xffffffffu, last);
  latest = __reduce_max_sync(0xffffffffu, latest);
  first = __reduce_min_sync(0xffffffffu, first);
  if (first >= latest || (last - first) / span > AT_MOST_PAIRS / gr.rows) return {0, 0};
  return {(last - first) / span * gr.rows, last};
}

// The scheduler (all lanes of one warp): the CTA's first item is the one with its own number, the others come off a counter in global
// memory. When nothing is left, the CTA signs off on a second counter, and the last one to do so puts both back to zero for the next
// launch. Lane 0's `item` is the one claimed.
// By place, empty items (tiles past a short row's end, splits past a short key range) are stepped over: the lanes look at the 32 items from
// the claimed one on, so a run of empty items costs one round trip. By position a CTA's numbers only grow, so it counts on from where it stood.
struct AtCursor {
  int entry, items;  // entries of the order (pairs, twice) passed, and the items in them
};
__device__ __forceinline__ bool at_claim(AtItem& item, AtCursor& at, int* __restrict__ queue, const AtGrid& gr, const AtOrder& order,
                                         const int* __restrict__ cu_q, const int* __restrict__ q_start, int lane, bool first) {
  const int span = 2 * (AT_ROWS / gr.G), total = gr.q_tiles * gr.rows * gr.head_groups * gr.splits;
  for (;;) {
    int idx = (int)blockIdx.x;
    if (!first) {
      if (lane == 0) idx = (int)gridDim.x + atomicAdd(queue, 1);
      idx = __shfl_sync(0xffffffffu, idx, 0);
    }
    if (order.pairs == 0) {
      if (idx >= total) break;
      bool work = false;
      if (idx + lane < total) {
        int n = idx + lane;
        const int split = n % gr.splits;
        n /= gr.splits;
        const int head = n % gr.head_groups;
        n /= gr.head_groups;
        const int n_full = at_tile(item, n % gr.rows, gr.q_tiles - 1 - n / gr.rows, gr, cu_q, q_start), per = at_piece_tiles(n_full, gr);
        work = split * per < n_full;
        if (work) at_piece(item, head * gr.G, split, per);
      }
      const unsigned mask = __ballot_sync(0xffffffffu, work);
      if (mask & 1u) return true;
      const int run = mask ? __ffs(mask) - 1 : 32;  // this many items from idx on are empty
      if (!first && lane == 0 && run > 1) atomicMax(queue, idx + run - (int)gridDim.x);
      first = false;
      continue;
    }
    for (; at.entry < 2 * order.pairs; at.entry += 32) {
      const int entry = at.entry + lane, phase = entry >= order.pairs, pair = entry - phase * order.pairs;
      int r = 0, tile = -1, whole = 0, count = 0;
      if (entry < 2 * order.pairs) {
        const int rank = pair / gr.rows;
        r = pair - rank * gr.rows;
        const int before = order.pos_max - rank * span - behind_load(q_start + r);
        tile = before > 0 ? before / span - 1 : -1;
        const int n_full = at_tile(item, r, tile, gr, cu_q, q_start);
        if (n_full > 0) {
          const int per = at_piece_tiles(n_full, gr);
          whole = n_full / per;
          count = gr.head_groups * (phase == 0 ? whole : whole * per < n_full);
        }
      }
      int upto = count;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += x;
      }
      const int sum = __shfl_sync(0xffffffffu, upto, 31);
      if (idx < at.items + sum) {
        const int l = __ffs(__ballot_sync(0xffffffffu, idx < at.items + upto)) - 1;
        const int place = idx - at.items - __shfl_sync(0xffffffffu, upto - count, l), pieces = __shfl_sync(0xffffffffu, whole, l);
        const int in_phase = __shfl_sync(0xffffffffu, phase, l);
        const int n_full = at_tile(item, __shfl_sync(0xffffffffu, r, l), __shfl_sync(0xffffffffu, tile, l), gr, cu_q, q_start);
        const int head = in_phase ? place : place / pieces, split = in_phase ? pieces : place - head * pieces;
        at_piece(item, head * gr.G, split, at_piece_tiles(n_full, gr));
        return true;
      }
      at.items += sum;
    }
    break;
  }
  if (lane == 0 && atomicAdd(queue + 1, 1) == (int)gridDim.x - 1) {
    queue[0] = 0;
    queue[1] = 0;
  }
  return false;
}

// Persistent: one CTA per SM takes items off a queue until none is left. EXTRAS: the instantiation that takes
// sink scores, a cap and a block mask (the plain one carries none of their code).
template <bool EXTRAS>
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                        const __grid_constant__ CUtensorMap map_v, __nv_bfloat16* __restrict__ out,
                        const int* __restrict__ cu_q, const int* __restrict__ q_start, const int* __restrict__ page_indptr,
                        const int* __restrict__ page_indices, int nq, int nkv, float scale_log2, int sink, int page_shift,
                        const AtGrid gr_given, int* __restrict__ status,
                        float* __restrict__ part_o, float2* __restrict__ part_ml, int* __restrict__ queue,
                        int* __restrict__ tickets, const int* __restrict__ plan, const AtExtras ex) {
  extern __shared__ unsigned char smem_dyn[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t q_full[2], q_empty[2], k_full[2], k_empty[2], v_full[2], v_empty[2], s_full[2], p_first[2], p_full[2], o_final[2];
  __shared__ uint64_t item_full[2], item_empty[2], drained;
  __shared__ AtItem items[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int ticket_of[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  // what needs nothing of the kernels before goes before the wait for them
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      at_mbar_init(&q_full[i], 1);
      at_mbar_init(&q_empty[i], 1);
      at_mbar_init(&k_full[i], 1);
      at_mbar_init(&k_empty[i], 1);
      at_mbar_init(&v_full[i], 1);
      at_mbar_init(&v_empty[i], 1);
      at_mbar_init(&s_full[i], 1);
      at_mbar_init(&p_first[i], 128);
      at_mbar_init(&p_full[i], 128);
      at_mbar_init(&o_final[i], 1);
      at_mbar_init(&item_full[i], 1);
      at_mbar_init(&item_empty[i], 9);  // 8 softmax warps and the thread that issues products
    }
    at_mbar_init(&drained, 1);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  if (warp == 9) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(at_smem(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  AT_FENCE_BEFORE();
  __syncthreads();
  AT_FENCE_AFTER();
  const uint32_t tmem = tmem_slot;
  pdl_wait();  // (what follows reads the step's metadata by loads that stay behind it)

  // A launch that was captured into a CUDA graph takes what follows from the rows' lengths (tiles per
  // row, rows, key splits) from device memory, where the host puts it before every replay: the
  // launch itself (a CTA per SM, these arguments) is then the same for every step of its size.
  AtGrid gr = gr_given;
  if (plan != nullptr) {
    gr.q_tiles = behind_load(plan + 0);
    gr.rows = behind_load(plan + 1);
    gr.splits = behind_load(plan + 2);
    gr.max_tiles_per_item = behind_load(plan + 3);
    part_ml = reinterpret_cast<float2*>(part_o + (size_t)gr.q_tiles * gr.rows * gr.head_groups * 2 * gr.splits * (AT_ROWS * AT_D));
  }
  const int G = gr.G, window = gr.window;
  const int tpc = AT_ROWS / G;

  // The roles part for good here, and in registers too: 12 warps of 168 registers fill the register file, the softmax warps (a whole row of scores each,
  // 128 values) want more and the two warps that issue copies and products, and their two idle
  // companions, need few. Warps 8 to 11 give theirs up, warps 0 to 7 take them.
  if (warp >= 8) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 104;\n");
    if (warp == 8) {
      // ---------------------------------------------------------- TMA producer and scheduler
      // Loads go out in the order in which they are needed: queries of A, first keys, queries of B, first values,
      // then keys and values of each tile. `tiles` counts the tiles of all items; tile c lies in slot c & 1.
      const int page_size = 1 << page_shift;
      const int box_rows = min(page_size, AT_KEYS);
      int tiles = 0, queries[2] = {0, 0};
      bool ok = true;
      auto wait_free = [&](uint64_t* bar, int use) {  // before use number `use` of a slot
        if (use > 0) {
          if (lane == 0) ok = at_wait(bar, (use - 1) & 1);
          ok = __shfl_sync(0xffffffffu, ok, 0);
        }
        return ok;
      };
      const AtOrder order = at_order(gr, cu_q, q_start, lane);
      AtCursor cursor = {0, 0};
      for (int i = 0; ok; ++i) {
        AtItem mine;
        const bool alive = at_claim(mine, cursor, queue, gr, order, cu_q, q_start, lane, i == 0);
        if (!wait_free(&item_empty[i & 1], i >> 1)) break;
        AtItem& it = items[i & 1];
        if (lane == 0) {
          mine.alive = alive;
          it = mine;
          at_arrive(&item_full[i & 1]);
        }
        __syncwarp();
        if (!alive) break;
        const int* pages = page_indices + behind_load(page_indptr + it.r);
        const int kv_len = it.kv_len, head0 = it.head0, kvh = head0 / (nq / nkv), n_all = it.n_all;
        auto load_q = [&](int g) {
          if (it.n_tiles[g] == 0 || !wait_free(&q_empty[g], queries[g])) return;
          ++queries[g];
          if (lane == 0) {
            unsigned char* dst = smem + AtSmem::q + g * 2 * AT_BLOCK;
            at_expect_tx(&q_full[g], 2 * AT_BLOCK);
            at_tma_3d(dst, &map_q, &q_full[g], 0, head0, it.tok0 + it.m0 + g * tpc);
            at_tma_3d(dst + AT_BLOCK, &map_q, &q_full[g], 64, head0, it.tok0 + it.m0 + g * tpc);
          }
        };
        for (int j = 0; j < n_all && ok; ++j, ++tiles) {
          const int s = tiles & 1;
          const int key0 = it.real_tile(it.tile_begin + j) * AT_KEYS;
          const int boxes = min(AT_KEYS, ((kv_len - key0 + box_rows - 1) / box_rows) * box_rows) / box_rows;
          int group8 = 0;  // where this lane's keys begin, in groups of 8 rows of the pool
          if (lane < boxes) {
            const int key = key0 + lane * box_rows;
            // (keys that every row's window has passed are not looked up: the table begins with the page ahead of the window's first)
            const int page = key + box_rows > it.lo_g[0] || key < gr.keep ? behind_load(pages + (key >> page_shift)) : 0;
            group8 = ((max(page, 0) * nkv + kvh) * page_size + (key & (page_size - 1))) >> 3;
          }
          const uint32_t bytes = (uint32_t)boxes * box_rows * (AT_D * 2);
          if (j == 0) load_q(0);
          if (!ok || !wait_free(&k_empty[s], tiles >> 1)) break;
          if (lane == 0) at_expect_tx(&k_full[s], bytes);
          __syncwarp();
          if (lane < boxes) tma_load_4d(at_smem(smem + AtSmem::k + s * AtSmem::slot + lane * box_rows * (AT_D * 2)), &map_k, at_smem(&k_full[s]), group8);
          if (j == 0) load_q(1);
          if (!ok || !wait_free(&v_empty[s], tiles >> 1)) break;
          if (lane == 0) at_expect_tx(&v_full[s], bytes);
          __syncwarp();
          if (lane < boxes) tma_load_4d(at_smem(smem + AtSmem::v + s * AtSmem::slot + lane * box_rows * (AT_D * 2)), &map_v, at_smem(&v_full[s]), group8);
        }
        __syncwarp();
      }
      if (!ok && lane == 0) {
        atomicExch(status, 31);
        // copies in flight must not outlive the CTA: a shorter wait for each barrier's last one
#pragma unroll
        for (int s = 0; s < 2; ++s) {
          const int uses = (tiles + 1 - s) >> 1;
          if (queries[s] > 0) mbar_wait_bounded(at_smem(&q_full[s]), (queries[s] - 1) & 1, MS_WAIT_NS / 64);
          if (uses > 0) mbar_wait_bounded(at_smem(&k_full[s]), (uses - 1) & 1, MS_WAIT_NS / 64);
          if (uses > 0) mbar_wait_bounded(at_smem(&v_full[s]), (uses - 1) & 1, MS_WAIT_NS / 64);
        }
      }
    } else if (warp == 9) {
      // ---------------------------------------------------------- MMA issuer
      if (at_elect()) {
        constexpr uint32_t idesc_s = at_idesc(false), idesc_o = at_idesc(true);
        bool ok = true;
        int k_seen0 = -1, k_seen1 = -1, k_used = 0;    // per slot: the last tile waited for; bits: one group has used the tile in it
        int queries[2] = {0, 0}, steps[2] = {0, 0};    // per group: items begun, tiles whose P was taken
        int base = 0;                                  // tiles of the items before the current one
        struct Some {
          int n[2], n_all, alive;
        } cur, next;
        int fetched = 0;
        auto fetch = [&](Some& to) {
          ok = ok && at_wait(&item_full[fetched & 1], (fetched >> 1) & 1);
          if (!ok) {
            to.alive = 0;
            return;
          }
          const AtItem& it = items[fetched & 1];
          to.n[0] = it.n_tiles[0];
          to.n[1] = it.n_tiles[1];
          to.n_all = it.n_all;
          to.alive = it.alive;
          at_arrive(&item_empty[fetched & 1]);
          ++fetched;
        };
        // the scores of group g over tile j of an item whose first tile is number `first`
        auto issue_s = [&](int g, const Some& of, int first, int j) {
          const int c = first + j, s = c & 1;
          if ((s ? k_seen1 : k_seen0) < c) {
            ok = at_wait(&k_full[s], (c >> 1) & 1);
            if (!ok) return;
            if (s) k_seen1 = c;
            else k_seen0 = c;
            AT_FENCE_AFTER();
          }
          const unsigned char* kt = smem + AtSmem::k + s * AtSmem::slot;
          const unsigned char* qt = smem + AtSmem::q + g * 2 * AT_BLOCK;
  #pragma unroll
          for (int kk = 0; kk < AT_D / 16; ++kk) {
            const uint64_t da = at_desc(qt + (kk >> 2) * AT_BLOCK, 16, 1024) + (uint64_t)(2 * (kk & 3));
            const uint64_t db = at_desc(kt + (kk >> 2) * 1024, 16, AT_GROUP8) + (uint64_t)(2 * (kk & 3));
            at_mma(tmem + (uint32_t)(g * 128), da, db, idesc_s, kk != 0);
          }
          at_commit(&s_full[g]);
          if (j + 1 == of.n[g]) at_commit(&q_empty[g]);
          // the last of the groups that need the tile frees its slot
          if (((k_used >> s) & 1) || !(j < of.n[0] && j < of.n[1])) {
            k_used &= ~(1 << s);
            at_commit(&k_empty[s]);
          } else {
            k_used |= 1 << s;
          }
        };
        auto begin = [&](int g, const Some& of, int first) {
          if (!ok || of.n[g] == 0) return;
          ok = at_wait(&q_full[g], queries[g] & 1);
          if (!ok) return;
          ++queries[g];
          AT_FENCE_AFTER();
          issue_s(g, of, first, 0);
        };
        fetch(cur);
        if (cur.alive) {
          begin(0, cur, 0);
          begin(1, cur, 0);
        }
        while (ok && cur.alive) {
          bool have_next = false;
          int begun = 0;
          for (int j = 0; j < cur.n_all && ok; ++j) {
            const int c = base + j, s = c & 1;
            const unsigned char* vt = smem + AtSmem::v + s * AtSmem::slot;
            bool v_seen = false;
  #pragma unroll
            for (int g = 0; g < 2; ++g) {
              if (!ok || j >= cur.n[g]) continue;
              ok = at_wait(&p_first[g], steps[g] & 1);
              if (ok && !v_seen) ok = at_wait(&v_full[s], (c >> 1) & 1);
              if (!ok) continue;
              v_seen = true;
              AT_FENCE_AFTER();
  #pragma unroll
              for (int kk = 0; kk < AT_KEYS / 16; ++kk) {
                if (kk == AT_FIRST / 16) {
                  ok = at_wait(&p_full[g], steps[g] & 1);
                  if (!ok) break;
                  AT_FENCE_AFTER();
                }
                // A = P of this group in tensor memory: 16 keys = 8 columns of packed bf16 pairs;
                // B = V [keys][d], MN-major
                const uint64_t db = at_desc(vt + kk * 2 * AT_GROUP8, 1024, AT_GROUP8);
                at_mma_ts(tmem + (uint32_t)(256 + g * 128), tmem + (uint32_t)(g * 128 + kk * 8), db, idesc_o, (j | kk) != 0);
              }
              if (!ok) continue;
              ++steps[g];
              // the next scores overwrite this group's S/P columns: ordered after the product above
              if (j + 1 < cur.n[g]) {
                issue_s(g, cur, base, j + 1);
              } else {
                at_commit(&o_final[g]);
                // on to the next item, unless the other group has more than one tile to go (its keys come first)
                if (cur.n_all - (j + 1) <= 1) {
                  if (!have_next) fetch(next);
                  have_next = true;
                  if (next.alive) begin(g, next, base + cur.n_all);
                  begun |= 1 << g;
                }
              }
            }
            if (ok) at_commit(&v_empty[s]);
          }
          if (!have_next) fetch(next);
          base += cur.n_all;
          if (next.alive) {
  #pragma unroll
            for (int g = 0; g < 2; ++g)
              if (!(begun & (1 << g))) begin(g, next, base);
          }
          cur = next;
        }
        // arrivals that nobody else waits for must not outlive the CTA, nor products
        if (ok) {
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const int uses = (base + 1 - s) >> 1;
            if (ok && queries[s] > 0) ok = at_wait(&q_empty[s], (queries[s] - 1) & 1);
            if (ok && uses > 0) ok = at_wait(&k_empty[s], (uses - 1) & 1) && at_wait(&v_empty[s], (uses - 1) & 1);
          }
        }
        if (!ok) {
          atomicExch(status, 33);
          at_commit(&drained);
          at_wait(&drained, 0);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 200;\n");
    const int g = warp >> 2;
    const int row = threadIdx.x & 127;                // row within the group = tensor-memory lane
    const int tok = row / G, hd = row - tok * G;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t t_s = tmem + (uint32_t)(g * 128) + lane_base, t_o = tmem + (uint32_t)(256 + g * 128) + lane_base;
    int tiles = 0, steps = 0, finals = 0;  // tiles of the items before; this group's own tiles; its items
    for (int i = 0;; ++i) {
      // ---------------------------------------------------------- softmax, thread = row of its group
      bool ok = at_wait(&item_full[i & 1], (i >> 1) & 1);
      if (at_group_any(1 + g, !ok)) {
        if (row == 0) atomicExch(status, 34);
        break;
      }
      const AtItem& it = items[i & 1];
      const int r = it.r, q_tile = it.tile, tok0 = it.tok0, q_len = it.q_len, m0 = it.m0, start = it.start, kv_len = it.kv_len;
      const int head0 = it.head0, split = it.split, tile_begin = it.tile_begin, first_tile = it.first_tile, walk_shift = it.walk_shift;
      const int lo_mine = it.lo_g[g], lo_max_mine = it.lo_max[g], q_first_mine = it.q_first[g], lo_item = it.lo_g[0];
      const int n_mine = it.n_tiles[g], n_all = it.n_all, shares = it.shares[g], alive = it.alive;
      __syncwarp();
      if (lane == 0) at_arrive(&item_empty[i & 1]);  // (what follows reads the copies)
      if (!alive) break;
      const int tile_first = tiles;
      tiles += n_all;
      if (n_mine == 0) continue;
      {
        const int tok_in_req = m0 + g * tpc + tok;
        const int qpos = start + tok_in_req;
        const int block_lo = EXTRAS && gr.chunk > 0 ? (qpos / gr.chunk) * gr.chunk : 0;
        // the sink's score in units of log2 (it is neither scaled nor capped)
        const float sink_l2 = EXTRAS && ex.sink_values != nullptr ? ex.sink_values[head0 + hd] * AT_LOG2E : 0.f;
        const float dist_c = EXTRAS && ex.dist_r1 != nullptr ? ex.dist_r1[head0 + hd] / scale_log2 : 0.f;
        const float dist_r2 = EXTRAS && ex.dist_r1 != nullptr ? ex.dist_r2[head0 + hd] : 0.f;
        float m_used = -INFINITY, l_sum = 0.f;
        auto hand_over = [&](uint64_t* bar) {  // this row's stores of P so far are done
          asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
          AT_FENCE_BEFORE();
          at_arrive(bar);
        };
        for (int j = 0; j < n_mine; ++j, ++steps) {
          ok = __all_sync(0xffffffffu, ok && at_wait(&s_full[g], steps & 1));  // (a warp stops as one)
          if (!ok) break;
          AT_FENCE_AFTER();
          const int key0 = (tile_begin + j - (tile_begin + j < first_tile ? walk_shift : 0)) * AT_KEYS;
          const bool interior = key0 + AT_KEYS - 1 <= q_first_mine && key0 >= lo_max_mine;
          // Rows of V that no query may weigh: keys beyond the request's end, and keys that the window of every row of
          // this item has passed and that are not kept first keys. Their pages may have been given back and hold
          // anything (a probability of zero times a NaN is a NaN), so they are made zero.
          const int valid_keys = kv_len - key0;
          const bool passed = key0 + row < lo_item && key0 + row >= gr.keep;
          if ((valid_keys < AT_KEYS && row >= valid_keys) || passed) {
            const int c = tile_first + j;
            ok = at_wait(&v_full[c & 1], (c >> 1) & 1);  // (the copy must not land on top of the zeros)
            unsigned char* vt = smem + AtSmem::v + (c & 1) * AtSmem::slot + (row >> 3) * AT_GROUP8 + (row & 7) * 128;
  #pragma unroll
            for (int h = 0; h < 2; ++h)
  #pragma unroll
              for (int cc = 0; cc < 8; ++cc) *reinterpret_cast<uint4*>(vt + h * 1024 + cc * 16) = make_uint4(0u, 0u, 0u, 0u);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
          }
          __syncwarp();
          float part[4] = {0.f, 0.f, 0.f, 0.f};
          // a tile on the diagonal, at a window's edge or at the request's end: the keys of the tile that this row
          // sees are those at offsets [seen_lo, seen_hi]
          const int seen_hi = qpos - key0;
          const int seen_lo = max(max(lo_mine, block_lo), window > 0 ? qpos - window + 1 : 0) - key0;
          if (!EXTRAS || interior) {
            // the whole row of scores in registers, four loads in flight, one wait
            float sv[4][32];
  #pragma unroll
            for (int c = 0; c < 4; ++c) at_tmem_ld32(t_s + (uint32_t)(c * 32), sv[c]);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            if (EXTRAS && ex.cap_c2 > 0.f) {
  #pragma unroll
              for (int c = 0; c < 4; ++c)
  #pragma unroll
                for (int i = 0; i < 32; ++i) sv[c][i] = at_cap(sv[c][i], ex.cap_raw, ex.cap_c2);
            }
            if (EXTRAS && dist_c != 0.f) {
              const int d0 = qpos - key0;
  #pragma unroll
              for (int c = 0; c < 4; ++c)
  #pragma unroll
                for (int i = 0; i < 32; ++i) sv[c][i] -= at_distance(dist_c, dist_r2, d0 - (c * 32 + i));
            }
            if (!EXTRAS && !interior) {
  #pragma unroll
              for (int c = 0; c < 4; ++c)
  #pragma unroll
                for (int i = 0; i < 32; ++i) {
                  const int off = c * 32 + i;
                  sv[c][i] = off <= seen_hi && off >= seen_lo ? sv[c][i] : -INFINITY;
                }
            }
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
  #pragma unroll
            for (int c = 0; c < 4; ++c)
  #pragma unroll
              for (int i = 0; i < 32; i += 2) mx[(i >> 1) & 3] = at_max3(mx[(i >> 1) & 3], sv[c][i], sv[c][i + 1]);
            const float alpha = at_new_maximum(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), m_used, scale_log2);
            if (__any_sync(0xffffffffu, alpha != 1.f)) {
              at_rescale(t_o, alpha);
              l_sum *= alpha;
            }
            // P = 2^(s * scale - max), packed two bf16 per column into the columns S came from
            const float m_sub = (m_used == -INFINITY ? 0.f : m_used) * scale_log2;
  #pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t pk[16];
  #pragma unroll
              for (int i = 0; i < 32; i += 2) {
                // (natural pairs of registers: sums of pairs as in the masked form cost moves, 249 against 229 us at 8,192 tokens)
                float x0, x1;
                at_fma2(x0, x1, sv[c][i], sv[c][i + 1], scale_log2, -m_sub);
                const float e0 = at_ex2(x0), e1 = at_ex2(x1);
                at_add2(part[i & 2], part[(i & 2) + 1], e0, e1);
                __nv_bfloat162 p2 = __floats2bfloat162_rn(e0, e1);
                pk[i >> 1] = *reinterpret_cast<uint32_t*>(&p2);
              }
              at_tmem_st16(t_s + (uint32_t)(c * 16), pk);
              if (c == AT_FIRST / 32 - 1) hand_over(&p_first[g]);
            }
          } else {
            part[0] = at_softmax_masked(t_s, t_o, seen_lo, seen_hi, scale_log2, m_used, l_sum, ex.cap_raw, ex.cap_c2,
                                        gr.keep - key0, dist_c, dist_r2, qpos - key0);
            hand_over(&p_first[g]);
          }
          l_sum += (part[0] + part[1]) + (part[2] + part[3]);
          hand_over(&p_full[g]);
        }
        if (ok) ok = at_wait(&o_final[g], finals & 1);
        ++finals;
        // all 128 threads of the group meet here, also after a wait that gave up: all of them stop then
        if (at_group_any(1 + g, !ok)) {
          if (row == 0) atomicExch(status, 34);
          break;
        }
        AT_FENCE_AFTER();
        const bool store = tok_in_req < q_len;
        const size_t item = (size_t)(tok0 + (store ? tok_in_req : 0)) * nq + head0 + hd;  // (token, head) of this row
        __nv_bfloat16* dst = out + item * AT_D;
        if (shares <= 1) {
          {
            // a sink: one more term of score 0 in the denominator, with no value
            const float inv = 1.0f / (l_sum + (sink ? at_ex2(sink_l2 - m_used * scale_log2) : 0.f));
  #pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              float ov[32];
              at_tmem_ld32(t_o + (uint32_t)(c * 32), ov);
              asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
              if (store) {
  #pragma unroll
                for (int i = 0; i < 32; i += 8) *reinterpret_cast<uint4*>(dst + c * 32 + i) = at_pack8(ov + i, inv);
              }
            }
          }
        } else {
          // One of several splits of this group's keys. Each takes a ticket when it is done. All but the
          // last leave their partial result (unnormalised O, the maximum it is scaled by, the sum) and
          // count themselves done; the last waits until the others are (they took their tickets before
          // it and depend on nothing of it, so this is a wait for writes in flight), then adds the
          // partial results up in the order of the splits, its own from tensor memory, and writes the
          // rows. Partial results are laid out [group of rows][split][4 columns][row], so that the 128
          // threads of a group (one row each) write and read whole 512-byte lines together.
          const size_t unit = ((size_t)(q_tile * gr.rows + r) * gr.head_groups + head0 / G) * 2 + g;
          float4* po = reinterpret_cast<float4*>(part_o) + (unit * gr.splits + split) * (32 * 128) + row;
          float2* pml = part_ml + unit * gr.splits * 128 + row;
          int* ticket = tickets + unit;
          int* done = tickets + (size_t)gr.q_tiles * gr.rows * gr.head_groups * 2 + unit;
          if (row == 0) ticket_of[g] = atomicAdd(ticket, 1);
          at_group_sync(1 + g);
          const bool last = ticket_of[g] == shares - 1;
          if (!last) {
  #pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              float ov[32];
              at_tmem_ld32(t_o + (uint32_t)(c * 32), ov);
              asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
  #pragma unroll
              for (int i = 0; i < 8; ++i) po[(c * 8 + i) * 128] = make_float4(ov[4 * i], ov[4 * i + 1], ov[4 * i + 2], ov[4 * i + 3]);
            }
            pml[split * 128] = make_float2(m_used, l_sum);
            __threadfence();
            at_group_sync(1 + g);
            if (row == 0) atomicAdd(done, 1);
          } else {
            if (row == 0) {
              // bounded like every wait: a split that took its ticket and never finishes is an error, not a hang
              unsigned long long began = 0;
              bool there = false;
              for (uint32_t polls = 1; !there; ++polls) {
                there = *reinterpret_cast<volatile int*>(done) >= shares - 1;
                if (!there && (polls & 63u) == 0) {
                  unsigned long long now;
                  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(now));
                  if (began == 0) began = now;
                  else if (now - began > MS_WAIT_NS) break;
                }
              }
              if (!there) atomicExch(status, 35);
              *ticket = 0;  // both left as they were found, for the next launch
              *done = 0;
              __threadfence();
            }
            at_group_sync(1 + g);
            const float4* pall = reinterpret_cast<const float4*>(part_o) + unit * gr.splits * (32 * 128) + row;
            float m_all = m_used;
            for (int sp = 0; sp < shares; ++sp)
              if (sp != split) m_all = fmaxf(m_all, __ldcg(&pml[sp * 128]).x);
            float l_all = 0.f;
            for (int sp = 0; sp < shares; ++sp) {
              const float2 ml = sp == split ? make_float2(m_used, l_sum) : __ldcg(&pml[sp * 128]);
              l_all += ml.y == 0.f ? 0.f : at_ex2((ml.x - m_all) * scale_log2) * ml.y;
            }
            if (sink) l_all += at_ex2(sink_l2 - m_all * scale_log2);
            const float inv = 1.0f / l_all;
  #pragma unroll 1
            for (int c = 0; c < 4; ++c) {
              float own[32], acc[32];
              at_tmem_ld32(t_o + (uint32_t)(c * 32), own);
              asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
  #pragma unroll
              for (int i = 0; i < 32; ++i) acc[i] = 0.f;
              for (int sp = 0; sp < shares; ++sp) {
                if (sp == split) {
                  const float w = l_sum == 0.f ? 0.f : at_ex2((m_used - m_all) * scale_log2);
  #pragma unroll
                  for (int i = 0; i < 32; ++i) acc[i] = fmaf(w, own[i], acc[i]);
                } else {
                  const float2 ml = __ldcg(&pml[sp * 128]);
                  const float w = ml.y == 0.f ? 0.f : at_ex2((ml.x - m_all) * scale_log2);
                  const float4* src = pall + (size_t)sp * (32 * 128) + (c * 8) * 128;
  #pragma unroll
                  for (int i = 0; i < 8; ++i) {
                    const float4 v = __ldcg(src + i * 128);
                    acc[4 * i] = fmaf(w, v.x, acc[4 * i]);
                    acc[4 * i + 1] = fmaf(w, v.y, acc[4 * i + 1]);
                    acc[4 * i + 2] = fmaf(w, v.z, acc[4 * i + 2]);
                    acc[4 * i + 3] = fmaf(w, v.w, acc[4 * i + 3]);
                  }
                }
              }
              if (store) {
  #pragma unroll
                for (int i = 0; i < 32; i += 8) *reinterpret_cast<uint4*>(dst + c * 32 + i) = at_pack8(acc + i, inv);
              }
            }
          }
          at_group_sync(1 + g);  // ticket_of[g] is free for the next item
        }
      }
    }
  }
  AT_FENCE_BEFORE();
  __syncthreads();
  AT_FENCE_AFTER();
  if (warp == 9) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---------------------------------------------------------------- host side
}  // namespace ms

using namespace ms;

MS_DEFINE_LAST_ERROR(ms_attn_tc_last_error)
MS_DEFINE_PDL_SWITCH(ms_attn_tc_set_pdl)

// 1 if this kernel takes the shape: head size 128, pages of 8..128 tokens (powers of two).
MS_EXPORT int ms_attn_tc_supports(int head_dim, int page_size, int nq, int nkv) {
  return head_dim == AT_D && page_size >= 8 && page_size <= 128 && (page_size & (page_size - 1)) == 0 && nq % nkv == 0;
}

static int at_heads_per_cta(int nq, int nkv) {
  const int group = nq / nkv;
  int G = 1;
  while (G * 2 <= 8 && group % (G * 2) == 0) G *= 2;  // the largest power of two up to 8 that divides the group
  return G;
}

constexpr int AT_MIN_TILES = 8;  // the least number of key tiles that a split keeps

// How the keys of a tile of queries are shared out, from the step's geometry on the host (q_start
// and q_len of the rows the launch covers): key ranges longer than *min_tiles key tiles are cut into
// pieces of that length, at most *splits of them. One CTA fills an SM, so a step with at most one query tile per SM cannot even its load
// out through the queue (nor can one with up to two): the last tiles of a long prompt, or the few tiles of a portion far into a
// long context, walk many more keys than the rest while other SMs idle. Then key ranges longer
// than about 1.2 times the work per SM are cut (1.1 where rows begin at different positions: us with 1.0 / 1.1 / 1.2 / 1.3, 1,531 tokens beside 517 behind
// 1,024 and 900 behind 4,096 67 / 68 / 72 / 76, four rows of up to 1,100 behind up to 2,000 34 / 29.5 / 29.4 / 29.7; also where such rows
// are too far apart to be ranked by position, with 1.1 / 1.2: 600 tokens beside 500 behind 20,000 111 / 106, 700 behind 1,024 beside 300 behind 24,000
// 114 / 121, four of 200 to 400 behind up to 9,000 63 / 64, eight of 100 behind up to 4,900 47 / 47). With many more tiles than SMs the queue evens the
// load out by itself and splits only add partial results.
// Measured on B200, 16 heads in 8 groups: 256 tokens behind 30,000: 645 us whole, 109 us cut;
// 512 behind 8,192: 193 -> 72 us; one prompt of 2,048 (128 tiles, the last 16 key tiles long):
// 57 us whole, 47 us with ranges over 8 tiles cut in two, 42 us with ranges over 9.
// ms_attn_tc_scratch says how much scratch the splits need.
MS_EXPORT void ms_attn_tc_plan(const int* q_start, const int* q_len, int num_rows, int nq, int nkv, int window, int sm_count,
                               int* splits, int* min_tiles) {
  *splits = 1;
  *min_tiles = AT_MIN_TILES;
  const int G = at_heads_per_cta(nq, nkv), span = 2 * (AT_ROWS / G), head_groups = nq / G;
  long long ctas = 0, steps = 0;
  int longest = 0;
  bool alike = true;  // rows that begin alike are taken in an order of their own (at_order), which evens out less
  for (int r = 0; r < num_rows; ++r) {
    alike = alike && q_start[r] == q_start[0];
    for (int m0 = 0; m0 < q_len[r]; m0 += span) {
      const int last = q_start[r] + (m0 + span < q_len[r] ? m0 + span : q_len[r]) - 1;
      const int lo = window > 0 && q_start[r] + m0 - window + 1 > 0 ? q_start[r] + m0 - window + 1 : 0;
      const int n = (last + AT_KEYS) / AT_KEYS - lo / AT_KEYS;
      ctas += head_groups;
      steps += (long long)n * head_groups;
      longest = n > longest ? n : longest;
    }
  }
  if (ctas == 0 || ctas > 2LL * sm_count) return;
  const long long fair = (steps * (alike ? 12 : 11) + 10LL * sm_count - 1) / (10LL * sm_count);  // 1.2 (1.1) x the work per SM, rounded up
  *min_tiles = (int)(fair < 4 ? 4 : fair);
  const int want = ceil_div(longest, *min_tiles);
  *splits = want < 1 ? 1 : (want > 16 ? 16 : want);
}

// What a launch needs besides its operands: float32 for the partial results of split key ranges
// (none for one split) and int32 for the work queue and the merge tickets; the int32 must be zero
// before the first launch and are left zero by every launch.
MS_EXPORT void ms_attn_tc_scratch(int max_q_len, int num_rows, int nq, int nkv, int splits, long long* partial_floats,
                                  long long* queue_ints) {
  const int G = at_heads_per_cta(nq, nkv);
  const long long units = (long long)ceil_div(max_q_len, 2 * (AT_ROWS / G)) * num_rows * (nq / G) * 2;  // groups of 128 rows
  *partial_floats = splits > 1 ? units * splits * (AT_ROWS * AT_D + AT_ROWS * 2) : 0;
  *queue_ints = 2 + 2 * units;  // the queue's two counters, a ticket and a count of finished splits per group of rows
}

MS_EXPORT int ms_attn_tc_prefill(void* out, const void* q, const void* k_pool, const void* v_pool, const int* cu_q,
                                 const int* q_start, const int* page_indptr, const int* page_indices, int num_rows,
                                 int num_tokens, int max_q_len, int nq, int nkv, long long pool_pages, float scale,
                                 int window, int sink, int page_size, int* status, int splits, int min_tiles, float* partials,
                                 int* queue, const int* plan, cudaStream_t stream, const float* sink_values, float softcap, int chunk,
                                 const float* dist_r1, const float* dist_r2, int keep_first) {
  MS_CHECK_ARG(softcap >= 0.f && chunk >= 0, "attention_tc: softcap=%g and chunk=%d must not be negative", softcap, chunk);
  MS_CHECK_ARG(keep_first >= 0 && (keep_first == 0 || window > 0) && (dist_r1 == nullptr) == (dist_r2 == nullptr),
               "attention_tc: keep_first=%d needs a window, and a distance bias both of its numbers", keep_first);
  sink = sink || sink_values != nullptr;
  AtExtras ex;
  ex.sink_values = sink_values;
  ex.dist_r1 = dist_r1;
  ex.dist_r2 = dist_r2;
  ex.cap_raw = softcap > 0.f ? softcap / scale : 0.f;
  ex.cap_c2 = softcap > 0.f ? 2.f * AT_LOG2E * scale / softcap : 0.f;
  // plan: null, or four device ints (tiles of queries per row, rows, key splits, least key tiles per split) that
  // ms_attn_tc_write_plan fills before the launch runs; num_rows, max_q_len, splits and min_tiles are then unused
  if (num_rows == 0 && plan == nullptr) return 0;
  if (plan != nullptr) {
    num_rows = 1;
    max_q_len = num_tokens;
    splits = 2;  // (only says that there is scratch for partial results)
    min_tiles = 1;
  }
  MS_CHECK_ARG(splits >= 1 && splits <= 64 && min_tiles >= 1, "attention_tc: %d key splits of at least %d tiles", splits, min_tiles);
  // partials and queue: sized by ms_attn_tc_scratch (the work queue's two counters, then the tickets
  // of the groups whose keys are split)
  MS_CHECK_ARG(queue != nullptr, "attention_tc: the work queue is missing");
  MS_CHECK_ARG(splits == 1 || (partials != nullptr && (uintptr_t)partials % 16 == 0),
               "attention_tc: key splits need scratch for the partial results");
  MS_CHECK_ARG(ms_attn_tc_supports(AT_D, page_size, nq, nkv), "attention_tc: unsupported shape (page_size=%d)", page_size);
  MS_CHECK_ARG(((uintptr_t)q % 16 == 0) && ((uintptr_t)k_pool % 16 == 0) && ((uintptr_t)v_pool % 16 == 0), "attention_tc: operands must be 16-byte aligned");
  const int G = at_heads_per_cta(nq, nkv);
  const int tpc = AT_ROWS / G;
  TensorMapEncodeFn encode;
  if (int rc = tensor_map_encoder(&encode)) return rc;
  CUtensorMap map_q, map_k, map_v;
  {
    const cuuint64_t dims[3] = {(cuuint64_t)AT_D, (cuuint64_t)nq, (cuuint64_t)num_tokens};
    const cuuint64_t strides[2] = {(cuuint64_t)AT_D * 2, (cuuint64_t)nq * AT_D * 2};
    const cuuint32_t box[3] = {64, (cuuint32_t)G, (cuuint32_t)tpc};
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult res = encode(&map_q, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(q), dims, strides, box, elem,
                                CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    MS_CHECK_ARG(res == CUDA_SUCCESS, "attention_tc: encoding the query map failed with code %d", (int)res);
  }
  const long long pool_rows = pool_pages * nkv * page_size;
  const int box_rows = page_size < AT_KEYS ? page_size : AT_KEYS;
  if (int rc = cache_tensor_map(&map_k, k_pool, pool_rows, AT_D, box_rows)) return rc;
  if (int rc = cache_tensor_map(&map_v, v_pool, pool_rows, AT_D, box_rows)) return rc;
  int page_shift = 0;
  while ((1 << page_shift) < page_size) ++page_shift;
  constexpr size_t smem_bytes = AtSmem::total + 1024;
  static bool configured = false;
  if (!configured) {
    MS_CHECK_CUDA(cudaFuncSetAttribute(attn_prefill_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes));
    MS_CHECK_CUDA(cudaFuncSetAttribute(attn_prefill_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes));
    configured = true;
  }
  static int sm_count = 0;
  if (sm_count == 0) {
    int dev = 0;
    MS_CHECK_CUDA(cudaGetDevice(&dev));
    MS_CHECK_CUDA(cudaDeviceGetAttribute(&sm_count, cudaDevAttrMultiProcessorCount, dev));
  }
  const AtGrid gr = {ceil_div(max_q_len, 2 * tpc), num_rows, nq / G, splits, min_tiles, window, G, chunk, keep_first};
  const long long total = (long long)gr.q_tiles * gr.rows * gr.head_groups * gr.splits;
  MS_CHECK_ARG(total < (1LL << 30), "attention_tc: %lld work items are too many for one launch", total);
  // one CTA fills an SM (192 KB of shared memory, all of tensor memory) and takes items until none is left
  const unsigned grid = (unsigned)(plan == nullptr && total < sm_count ? total : sm_count);
  if (sink_values != nullptr || softcap > 0.f || chunk > 0 || dist_r1 != nullptr || keep_first > 0) {
    MS_LAUNCH(attn_prefill_tc_kernel<true>, grid, AT_THREADS, smem_bytes, stream, map_q, map_k, map_v, (__nv_bfloat16*)out, cu_q,
              q_start, page_indptr, page_indices, nq, nkv, scale * AT_LOG2E, sink, page_shift, gr, status,
              partials, reinterpret_cast<float2*>(partials + (total / gr.splits) * 2 * gr.splits * (AT_ROWS * AT_D)), queue,
              queue + 2, plan, ex);
  } else {
    MS_LAUNCH(attn_prefill_tc_kernel<false>, grid, AT_THREADS, smem_bytes, stream, map_q, map_k, map_v, (__nv_bfloat16*)out, cu_q,
              q_start, page_indptr, page_indices, nq, nkv, scale * AT_LOG2E, sink, page_shift, gr, status,
              partials, reinterpret_cast<float2*>(partials + (total / gr.splits) * 2 * gr.splits * (AT_ROWS * AT_D)), queue,
              queue + 2, plan, ex);
  }
  return 0;
}

namespace ms {
__global__ void attn_tc_plan_kernel(int* __restrict__ plan, int q_tiles, int rows, int splits, int min_tiles) {
  pdl_prologue();
  plan[0] = q_tiles;
  plan[1] = rows;
  plan[2] = splits;
  plan[3] = min_tiles;
}
}  // namespace ms

// Plans a step's attention as ms_attn_tc_plan does and puts the plan where a captured launch reads it
// (a one-thread kernel in stream order: its arguments travel with the launch, so no host buffer has to
// outlive the call). The key splits are cut down until their partial results fit partial_floats; the
// work queue must hold queue_ints.
MS_EXPORT int ms_attn_tc_write_plan(int* plan, const int* q_start, const int* q_len, int num_rows, int max_q_len, int nq, int nkv,
                                    int window, int sm_count, long long partial_floats, long long queue_ints, cudaStream_t stream) {
  MS_CHECK_ARG(plan != nullptr && num_rows > 0 && max_q_len > 0, "attention_tc: a plan needs rows");
  int splits = 1, min_tiles = AT_MIN_TILES;
  ms_attn_tc_plan(q_start, q_len, num_rows, nq, nkv, window, sm_count, &splits, &min_tiles);
  long long need_f = 0, need_i = 0;
  for (;; --splits) {
    ms_attn_tc_scratch(max_q_len, num_rows, nq, nkv, splits, &need_f, &need_i);
    if (splits == 1 || need_f <= partial_floats) break;
  }
  MS_CHECK_ARG(need_i <= queue_ints, "attention_tc: the work queue holds %lld entries, the step needs %lld", queue_ints, need_i);
  const int G = at_heads_per_cta(nq, nkv);
  MS_LAUNCH(attn_tc_plan_kernel, 1, 1, 0, stream, plan, ceil_div(max_q_len, 2 * (AT_ROWS / G)), num_rows, splits, min_tiles);
  return 0;
}
