// Host entry points of the decode step as one persistent kernel (model/decode_step.cuh).  No counterpart in the reference.
#pragma once

#include <vector>

#include "../coll/comm.h"

namespace b200ipc {

struct DecodeStepShape {
  int batch, layers, hidden, hq, hkv, ffn, vocab;  // heads, FFN width and vocabulary per rank
  int max_ctx;
};
struct DecodeStepPtrs {
  // [layer][rank]
  std::vector<const void*> wqkv, wo, wgu, wdown;
  std::vector<void*> kcache, vcache;
  std::vector<const void*> head;                    // [rank]
  std::vector<const void*> gamma_attn, gamma_mlp;   // [layer]
  const void* gamma_final;
  void* h;                                          // [batch, hidden] embeddings of the tokens; overwritten
  std::vector<void*> hidden_out;                    // [rank] [batch, hidden]
  int64_t* ids;                                     // [batch]
  void* workspace;
};

// Whether the kernel takes a step: every rank in this process, 1 to 64 sequences, head dimension 128, 1 / 2 / 4 / 8 query heads
// per KV head, a hidden size that the row-parallel GEMMs of the chain of kernels take, at least one position in the cache.
bool decode_step_takes(const Comm& comm, const DecodeStepShape& s, int pos);
// Whether it is also ahead of the chain of kernels, as far as that depends on the step.
bool decode_step_pays(const Comm& comm, const DecodeStepShape& s, int pos);
size_t decode_step_workspace_bytes(const Comm& comm, const DecodeStepShape& s);
// Of the flags kMuteSends is known: one CTA stays away from the meeting points, so the waits there run out.
void decode_step(Comm& comm, DType t, const DecodeStepShape& s, const DecodeStepPtrs& p, int pos, float eps, float theta, cudaStream_t stream,
                 uint32_t flags = 0);

}  // namespace b200ipc
