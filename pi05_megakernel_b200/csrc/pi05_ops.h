// Host side of the tcgen05 projections and attention (pi05_ops.cu): tensor maps, how a projection is cut, launches.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <atomic>
#include <utility>

#include "pi05_attention.cuh"
#include "pi05_attention_o.cuh"
#include "pi05_gemm.cuh"

namespace pi05 {

// Launch with programmatic stream serialisation (the kernel may become resident and set up while the one before it in the
// stream runs; `early` false: without it) and, with `cluster` > 1, as clusters of that many CTAs.
template <typename... Params, typename... Args>
cudaError_t launch_kernel(void (*kernel)(Params...), dim3 grid, int block, size_t smem, cudaStream_t stream, int cluster, bool early, Args&&... args) {
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = grid; cfg.blockDim = dim3(block); cfg.dynamicSmemBytes = smem; cfg.stream = stream;
  cudaLaunchAttribute at[2];
  int n = 0;
  if (early) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n].val.programmaticStreamSerializationAllowed = 1;
    ++n;
  }
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = cluster; at[n].val.clusterDim.y = 1; at[n].val.clusterDim.z = 1;
    ++n;
  }
  cfg.attrs = at; cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), int grid, int block, size_t smem, cudaStream_t stream, int cluster, Args&&... args) {
  return launch_kernel(kernel, grid, block, smem, stream, cluster, true, std::forward<Args>(args)...);
}

// An operand [rows, K] BF16 row-major as {64 k, rows, K / 64}, box {64, box_rows, blocks}, 128-byte swizzle: one copy brings
// `blocks` 64-k blocks of box_rows rows.  Rows beyond `rows` read as zeros.
bool map_k(CUtensorMap* m, const void* base, uint64_t k, uint64_t rows, uint32_t box_rows, uint32_t blocks);
// Keys or values as the attention's tiled copies read them: {64 dims, tokens, 4 blocks, layers, pages} with strides in elements,
// box {64, box_tokens, box_blocks, 1, 1}; tokens beyond `tokens` read as zeros.
bool map_kv(CUtensorMap* m, const void* base, uint64_t tokens, uint64_t layers, uint64_t pages, uint64_t token_stride,
            uint64_t layer_stride, uint64_t page_stride, uint32_t box_tokens, uint32_t box_blocks);

// How one projection of `tokens` x n features over k is cut.
struct GemmPlan {
  int epi;            // gemm::EPI_*
  bool pair, sk;
  int bn, ks, splits, m_tiles, rows, arows, units, grid, stages, bufs, off_out, smem, kblocks;
  int w_rows, w_kb;   // rows and 64-k blocks of one weight copy (the box of the weights' maps)
};
// pairs: 1 / 0 leaves only cuts on CTA pairs / on single CTAs, -1 all.
GemmPlan plan_gemm(int sms, int tokens, int n, int k, int epi, int pairs = -1);
// The stream-K cut of a projection with partial sums: 128 x 256 tiles, one equal range of 64-k blocks per CTA.
GemmPlan plan_gemm_sk(int sms, int tokens, int n, int k);
// Fills in what the plan decides and the destination maps, and launches.  `width` and the pointers have to be set.  `early`: may
// start while the kernel before it in the stream runs.
cudaError_t launch_gemm(const GemmPlan& g, gemm::Args& p, cudaStream_t stream, bool early = true);
cudaError_t launch_attention(attn::Args& p, int observations, cudaStream_t stream);
// Shared-memory opt-in of the kernel behind a plan, before its first launch on a device.  (Only what is used: the first touch loads a
// kernel's code, and all of them together take 20 ms.)
cudaError_t opt_in_gemm(const GemmPlan& g, int device);
cudaError_t opt_in_attention(int tok_tile, bool join, int device);
// Attention and O projection in one kernel (prefixes of up to attno::MAX_PREFIX tokens).
cudaError_t launch_attention_o(const attno::Args& p, int observations, int smem, cudaStream_t stream);
cudaError_t opt_in_attention_o(int device);
// Runs `body` (launch settings that may be made twice) once per device, from whichever threads: `done` has a bit per device.
template <typename F>
cudaError_t once_per_device(std::atomic<uint64_t>* done, int device, F body) {
  const uint64_t bit = device < 64 ? 1ull << device : 0;
  if (done->load() & bit) return cudaSuccess;
  const cudaError_t e = body();
  if (e == cudaSuccess) done->fetch_or(bit);
  return e;
}
// One split of L1 and shared memory for all kernels of a chain: an SM that has to change it drains first, which would keep a
// kernel's CTAs from becoming resident beside the ones of the kernel before.
cudaError_t chain_opt_in(const void* kernel, int smem);

}  // namespace pi05
