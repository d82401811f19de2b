// Single-token decoding of the GPT-2 architecture with cached keys and values.
#pragma once
#include <cuda_runtime.h>

namespace z2h {

// Where the bf16 weights of a model lie in one packed buffer (element offsets, multiples of 64;
// -1 = absent). Offsets named o_* are inside a layer; layer l starts at layer0 + l * layer_stride.
struct DecodeLayout {
  long long wte, wpe, layer0, layer_stride, lnf_w, lnf_b;
  long long o_qkv, o_proj, o_fc, o_fc2;
  long long o_ln1_w, o_ln1_b, o_b_qkv, o_b_proj, o_ln2_w, o_ln2_b, o_b_fc, o_b_fc2;
};

// One token of up to kDecodeMaxBatch sequences, all at the same position.
struct DecodeArgs {
  DecodeLayout lay;
  const void* weights;      // bf16, packed
  void* kv;                 // bf16 [layers][2][batch][max_len][C]
  const long long* tokens;  // token of sequence b at tokens[b * token_stride]
  long long token_stride;
  float* logits;            // fp32 [batch][vocab], rounded to bf16 like the module's; null: no head
  void* scratch;            // decode_scratch_bytes(), zeroed once before the first step
  unsigned int epoch_base;  // 1 in the first step on this scratch, then decode_epochs() more in each (never less)
  int batch, C, heads, layers, vocab, pos, max_len;
  int* status;
};

constexpr int kDecodeMaxBatch = 8;

long long decode_scratch_bytes(int batch, int C, int heads);
// How far a step moves epoch_base; 0: the shape is not supported.
unsigned int decode_epochs(int batch, int C, int layers);
// 0 ok, 1 bad argument, 3 launch failed
int decode_step(const DecodeArgs& a, cudaStream_t stream);

}  // namespace z2h
