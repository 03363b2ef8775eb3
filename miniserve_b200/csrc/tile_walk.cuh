// The decay rule over prompts by chunks of 64 tokens (``tile_walk.cu``), for the entry points of ``chunk_walk.cu``.
#pragma once
#include <climits>

#include "common.cuh"

namespace ms {

constexpr int TW_TOK = 64;

// How long the walk's waits last, and the first chunks whose queries and whose additions to the state are not copied (for tests of what happens then).
struct TwWaits {
  int no_queries = INT_MAX, no_added = INT_MAX;
  unsigned long long limit_ns = MS_WAIT_NS;
};

// Whether a step goes there. It does not know its rows' lengths, only that the longest has at least their mean. (With 1 GB of scratch and more a step
// stays on the chunks of 16: the cache pool leaves as much for it.)
bool tile_walk_takes(int tokens, int rows, int H, int dk, int dv, int groups);
long long tile_walk_scratch(int tokens, int rows, int H, int dk, int dv, int groups);  // floats; groups: of heads that share queries and keys, 0: a decay per channel

int tile_walk_head(float* o, float* state, const float* q, int ld_q, const float* k, int ld_k, int qk_group, const float* v, int ld_v, const float* decay,
                   int ld_decay, const float* v_scale, float* scratch, const int* cu_q, const int* q_start, const int* state_slot, int num_tokens,
                   int num_rows, int H, int dk, int dv, float q_scale, int* status, cudaStream_t stream, const TwWaits& waits = TwWaits());

template <typename TIn, typename TZ>
int tile_walk_channel(float* o, float* state, const TIn* q, int ld_q, const TIn* k, int ld_k, int qk_group, const TIn* v, int ld_v, const TZ* z, int ld_z,
                      const float* z_bias, const float* decay_coef, float z_sign, const float* v_scale, float* scratch, const int* cu_q, const int* q_start,
                      const int* state_slot, int num_tokens, int num_rows, int H, int dk, int dv, float q_scale, int* status, cudaStream_t stream, const TwWaits& waits = TwWaits());

}  // namespace ms
