// The action chunk as a chain of kernels replayed from CUDA graphs (pi05_steps.cu): what the engine hands over at bind.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "pi05_common.cuh"

namespace pi05 {

struct StepSetup {
  int device, sms, batch, prefix;
  const void* const* in;                     // the 25 inputs
  float* actions;
  unsigned int* status;
  int* state;                                // {Euler step, finished blocks of the step tail, Euler steps of this chunk}
  float *temb, *hid, *cond, *mod, *x, *part; // part: partial sums of split projections and attentions
  size_t part_floats;                        // what `part` holds (steps_part_floats)
  uint32_t *rope, *rope4;                    // [token][128]; the same words as gemm::rope_at orders them
  __nv_bfloat16 *h, *an, *q, *k, *v, *attn, *act;
  const void *pool_k, *pool_v;               // prefix cache; strides in elements
  long long token_stride, layer_stride, page_stride;
  int num_pages;
  const int* page_table;
  int pages_per_obs, page_tokens;
  long long wait_limit;
  int withhold;                              // debug: the QKV projection of this layer waits for data that never comes; -1: none
};

// The prologue for all Euler steps, and one step of all layers.
struct StepGraphs {
  cudaGraphExec_t prologue = nullptr, step = nullptr;
  long long wait_limit = 0;                  // what the graphs were captured with
  int kernels_prologue = 0, kernels_step = 0;
};

// How a binding is cut: query tokens per CTA of the attention and CTAs that share the keys of a tile, K splits of the O and down
// projections, FP32 words of partial sums.
struct StepPlan {
  int tok_tile, splits, o_splits, down_splits;
  int chunks;                                // of 128 keys, the most that a CTA of the attention takes
  bool join, with_o;                         // the suffix in the last chunk of the prefix; attention and O projection in one kernel (all keys at once)
  size_t part_floats;
};
StepPlan steps_plan(int sms, int batch, int prefix, int page_tokens);
// The cuts of a binding, and the kernels of its launch (`g`: of the captured chain), as a JSON object.
std::string steps_describe(int sms, int batch, int prefix, int page_tokens, const StepGraphs& g);
// FP32 words of partial sums that up to `max_batch` observations with up to `max_prefix` prefix tokens need.
size_t steps_part_floats(int sms, int max_batch, int max_prefix);
// Captures and instantiates the graphs; frees what `g` held.
int steps_build(const StepSetup& s, StepGraphs* g, std::string* error);
// Enqueues one chunk: the graphs where they fit, else kernel by kernel.  Allocates nothing and does not wait.  `capturing`: the stream
// is being captured.
int steps_launch(const StepGraphs& g, const StepSetup& s, int n_steps, int n_layers, bool capturing, cudaStream_t stream, std::string* error);
void steps_free(StepGraphs* g);

}  // namespace pi05
