// One decode step of the Qwen3-shape decoder for several sequences as one persistent kernel: interface of decode_wide.cu.
#pragma once
#include "ytc_common.cuh"

namespace ytk {

constexpr int WD_MAX_B = 32;  // sequences per step

struct WdLayer {  // weights of one layer: bf16 [out, in] matrices, fp32 norm weights
  const uint16_t *qkv, *o, *gate_up, *down;
  const float *q_norm, *k_norm, *norm1, *norm2;
};

struct WdShape {
  int B, hidden, layers, heads, kv_heads, inter, vocab, max_pos;
};

struct WdStep {  // what changes from step to step, and the buffers the step works on
  int pos;       // cache slot and rotary position of the new token: keys 0 .. pos - 1 are in the cache
  float eps, scale;
  const int32_t* ids;
  const uint16_t* embed;
  const float *cos_t, *sin_t;     // [max_pos][128]
  float *k_cache, *v_cache;       // [layers][B, kv_heads, max_pos, 128]
  float *x, *qkv;                 // [B][hidden] (the result), [B][(heads + 2 kv_heads) 128]
};

// Device state of one model's wide steps (weight pointers, tensor maps, arrival words).
struct WdState {
  void* dev = nullptr;
  unsigned int epoch = 0;  // phases completed by the launches so far
  bool stale = true;       // the weight pointers have changed since the last launch
};

// Whether this model's steps can run here, on the current device.
bool wide_step_supported(const WdShape& s);
size_t wide_state_bytes(const WdShape& s);
// x of the last layer for the token `ids` of every sequence; appends one row to every cache. `state.dev` holds
// wide_state_bytes() of device memory.
int wide_step_launch(const WdShape& s, const WdStep& step, const WdLayer* layers, WdState& state, cudaStream_t st);

}  // namespace ytk
