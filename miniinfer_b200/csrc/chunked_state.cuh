// Recurrences with a decaying matrix state a head over long prompt portions, a chunk of tokens at a time (chunked_state.cu).
#pragma once

#include "common.cuh"

namespace mi {

constexpr int CHUNK_TOKENS = 64;
constexpr int CHUNK_MAX_DIM = 128;            // key channels a head
constexpr int CHUNK_STATUS_LATE = 32;

enum ChunkDecay { CHUNK_DECAY_CHANNEL = 0, CHUNK_DECAY_HEAD = 1, CHUNK_DECAY_CONSTANT = 2 };

struct ChunkedStateArgs {
  const float* qn; const float* kn;           // [tokens, qk_heads * dim], head h reads head h / (heads / qk_heads)
  const float* g;                             // decays in 0 .. 1: [tokens, heads * dim], their logarithms [tokens, heads], or [heads] (ChunkDecay)
  int decay;
  const float* beta;                          // [tokens, heads] write strengths of the delta rule, or null: S <- diag(g) S + k v^T
  float* raw;                                 // [tokens, heads * vdim]: the values in (numbers that tf32 holds, as bfloat16 ones are), the read-outs out
  float* state; long long state_stride;       // [slot][heads][dim][vdim]
  const int* q_start; const int* q_len; const int* seq_slot;
  int items, heads, qk_heads, dim, vdim;
  int min_tokens;                             // items of fewer new tokens are left alone
  int* status;                                // null, or a word that is set to CHUNK_STATUS_LATE if a bounded wait for a block's own copies ran out
};

// Whether the sizes are taken: up to CHUNK_MAX_DIM key channels, rows of whole 16 bytes.
inline bool chunked_state_takes(int dim, int vdim) { return dim > 0 && dim <= CHUNK_MAX_DIM && dim % 4 == 0 && vdim > 0 && vdim % 4 == 0; }
// Floats of scratch for a step of T tokens in `items` items (some slabs of chunks at a time share it).
long long chunked_state_scratch_floats(int T, int items, int heads, int dim, int vdim, bool delta);
int chunked_state_slabs(int T, int items, int heads, int dim, int vdim, bool delta);      // three launches each
int chunked_state_run(const ChunkedStateArgs& a, int T, float* scratch, cudaStream_t stream);

}  // namespace mi
