// Host side of the tcgen05 projections and attention: tensor maps, how a projection is cut, launches.
#include "pi05_ops.h"

#include <algorithm>

namespace pi05 {
namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encoder() {
  static EncodeTiledFn fn = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
        qres != cudaDriverEntryPointSuccess)
      ptr = nullptr;
    return reinterpret_cast<EncodeTiledFn>(ptr);
  }();
  return fn;
}

// Bytes of the staging buffer of a tile's results (gemm::Staging).
int staging_bytes(int epi, int bn) {
  using namespace gemm;
  if (epi == EPI_PART) return bn == 32 ? 0 : bn == 64 ? Staging<EPI_PART, 64>::BYTES : bn == 128 ? Staging<EPI_PART, 128>::BYTES : Staging<EPI_PART, 256>::BYTES;
  if (epi == EPI_GEGLU) return bn == 64 || bn == 112 ? 0 : bn == 128 ? Staging<EPI_GEGLU, 128>::BYTES : bn == 224 ? Staging<EPI_GEGLU, 224>::BYTES : Staging<EPI_GEGLU, 256>::BYTES;
  return bn == 32 ? 0 : bn == 64 ? Staging<EPI_QKV, 64>::BYTES : bn == 128 ? Staging<EPI_QKV, 128>::BYTES : Staging<EPI_QKV, 256>::BYTES;
}

typedef void (*GemmKernel)(const gemm::Args);
struct Cut { int epi, bn, ks; bool pair, sk; GemmKernel kernel; };

// Every cut that is built: each is the choice for some number of tokens, 1 to 4096 of a prefill or 1 to 16 observations.
#define CUT(E, BN, PAIR, KS, SK) {gemm::E, BN, KS, PAIR, SK, gemm::gemm_kernel<gemm::E, BN, PAIR, KS, SK>}
const Cut kCuts[] = {
    CUT(EPI_QKV, 32, false, 4, false), CUT(EPI_QKV, 32, false, 2, false), CUT(EPI_QKV, 64, false, 2, false), CUT(EPI_QKV, 128, false, 2, false),
    CUT(EPI_QKV, 128, true, 2, false), CUT(EPI_QKV, 256, true, 1, false),
    CUT(EPI_GEGLU, 64, false, 2, false), CUT(EPI_GEGLU, 128, false, 2, false), CUT(EPI_GEGLU, 128, true, 2, false), CUT(EPI_GEGLU, 112, false, 2, false),
    CUT(EPI_GEGLU, 224, true, 1, false), CUT(EPI_GEGLU, 256, true, 1, false),
    CUT(EPI_PART, 32, false, 2, false), CUT(EPI_PART, 64, false, 2, false), CUT(EPI_PART, 128, false, 2, false), CUT(EPI_PART, 64, true, 2, false),
    CUT(EPI_PART, 128, true, 2, false), CUT(EPI_PART, 256, true, 1, false), CUT(EPI_PART, 256, false, 1, true),
};
#undef CUT

// Loads, ring, staging and shared memory of a cut whose tile, grid and accumulators are decided.
void lay_out(GemmPlan* g, int stages_wanted) {
  const bool two = !g->pair && (g->epi == gemm::EPI_QKV || g->epi == gemm::EPI_GEGLU);
  g->w_rows = g->pair || two ? g->bn / 2 : g->bn;
  g->w_kb = two ? 1 : g->ks;
  const int w_bytes = (g->pair ? g->bn / 2 : g->bn) * 128, stage = g->ks * (g->arows * 128 + w_bytes);
  // results are staged in the ring when the CTA has one tile (its operands are consumed by then), else behind it
  const bool behind = g->bufs > 1;
  const int out = g->sk ? 2 * 16384 : staging_bytes(g->epi, g->bn);
  const int budget = 218 * 1024 - (behind ? out : 0);
  g->stages = std::min({gemm::MAX_STAGES, budget / stage, stages_wanted});
  const int ring = g->stages * stage;
  g->off_out = behind ? ring : 0;
  // the MMA reads 128 rows from the last activation block on
  g->smem = std::max({ring, (g->stages - 1) * stage + (g->ks - 1) * g->arows * 128 + 128 * 128, g->off_out + out}) + 1024;
}

}  // namespace

bool map_k(CUtensorMap* m, const void* base, uint64_t k, uint64_t rows, uint32_t box_rows, uint32_t blocks) {
  EncodeTiledFn enc = encoder();
  if (!enc) return false;
  cuuint64_t dims[3] = {64, rows, k / 64};
  cuuint64_t strides[2] = {k * 2, 128};
  cuuint32_t box[3] = {64, box_rows, blocks};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool map_kv(CUtensorMap* m, const void* base, uint64_t tokens, uint64_t layers, uint64_t pages, uint64_t token_stride,
            uint64_t layer_stride, uint64_t page_stride, uint32_t box_tokens, uint32_t box_blocks) {
  EncodeTiledFn enc = encoder();
  if (!enc) return false;
  cuuint64_t dims[5] = {64, tokens, 4, layers, pages};
  cuuint64_t strides[4] = {token_stride * 2, 64 * 2, layer_stride * 2, page_stride * 2};
  cuuint32_t box[5] = {64, box_tokens, box_blocks, 1, 1};
  cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The cheapest of the cuts that are built, by a model of the launch's time in SM cycles: rounds x 64-k blocks x the slower of the
// tensor core (N / 2 cycles per K16 instruction) and shared memory (128 B per cycle: the rows of both operands that an
// instruction reads, 64 or 128 of the activations, and the copies that bring them), not less than the weights' way from HBM
// (3.3 KB per cycle), plus what every launch pays, an epilogue that grows with the tile, the start of a cluster for pairs
// of CTAs (measured: a launch on pairs takes 0.4-0.8 us longer than the same on single CTAs) and the way of partial sums through
// L2 and the row kernel.  Its constants are fitted to cuts that were timed by themselves, 50 to 800 tokens: it knows nothing of the
// kernel behind, which starts up to 2 us later behind a launch on more than half of the SMs.
// K of the projections whose sums meet in the residual kernel is split in powers of two, down to four 64-k blocks.
GemmPlan plan_gemm(int sms, int tokens, int n, int k, int epi, int pairs) {
  GemmPlan best = {};
  double best_cost = 1e30;
  for (const Cut& c : kCuts)
    for (int splits = 1; c.epi == epi && !c.sk && splits <= (epi == gemm::EPI_PART ? 8 : 1); splits *= 2) {
      GemmPlan g = {};
      g.epi = epi; g.pair = c.pair; g.bn = c.bn; g.ks = c.ks; g.splits = splits;
      g.kblocks = k / gemm::BK / splits;
      g.m_tiles = (tokens + 127) / 128;
      if ((g.pair && g.m_tiles < 2) || (pairs >= 0 && (int)g.pair != pairs)) continue;
      if (g.pair) g.m_tiles = (g.m_tiles + 1) / 2 * 2;
      // K is split where the tiles of a whole K leave SMs idle, and not to even out rounds: prefill of 2700 tokens 10.9 ms, with K of the
      // down projection over two CTAs 11.3
      const int n_tiles = (n + g.bn - 1) / g.bn;              // (224 features divide no width: what is left of the last tile is computed and clipped)
      if (g.kblocks < 4 || (splits > 1 && g.m_tiles * n_tiles >= sms)) continue;
      // Stages of four 64-k blocks where a whole K fits the ring that way: 50 tokens 4.66 against 4.69 ms a chunk; the gate / up, O and
      // down projections got slower on them (+1 to 3%), and every one on stages of a single block (+1 to 2%)
      if (c.ks == 4 && tokens > 64) continue;
      g.rows = (tokens + g.m_tiles - 1) / g.m_tiles;
      g.arows = (g.rows + 7) / 8 * 8;
      // 112 and 224 features (56 and 112 of gate and of up) are for widths that they cut into whole rounds: 4096 in two rounds of 74 pairs beside 1.73 of
      // 256 (both widths in turn in one process: sixteen observations of 128 tokens 10.32 -> 10.20 ms, of 600 11.51 -> 11.42; prefill of 256 tokens 1.52 -> 1.48), 16384 in two rounds of 148 CTAs beside 3.5 of 64 (prefill of 128 tokens
      // 1.32 -> 1.26).  In a single round either way they only pay where the MMAs take long: 5 observations (tiles of 125 tokens) 6.32 -> 6.21, 9 (113) 8.06 -> 7.96,
      // but 7 (88) 7.11 -> 7.28: the narrower tile occupies 148 SMs, not 128, and the next kernel's CTAs start late
      if ((g.bn == 224 || g.bn == 112) && g.m_tiles * n_tiles <= sms && (tokens + g.m_tiles - 1) / g.m_tiles <= 96) continue;
      const int w_bytes = (g.pair ? g.bn / 2 : g.bn) * 128, ctas = g.m_tiles * n_tiles * splits, rounds = (ctas + sms - 1) / sms;
      // cycles of a 64-k block: the tensor core's, or what its operands take through shared memory
      const double smem = (4 * ((!g.pair && g.rows <= 64 ? 2048 : 4096) + g.bn * (g.pair ? 16 : 32)) + g.arows * 128 + w_bytes) / 128.0;
      double cost = std::max(rounds * g.kblocks * (std::max({2.0 * g.bn, 100.0, smem}) + 70.0 / g.ks), (double)n * k * 2 / 3300) + 2000 +
                    g.bn * (epi == gemm::EPI_GEGLU ? 24 : 8) + (g.pair ? 2400 : 0);
      if (splits > 1) cost += std::max(500.0 * splits, splits * (double)tokens * n * 4 / 1800);
      if (cost >= best_cost) continue;
      g.units = g.pair ? ctas / 2 : ctas;
      g.grid = std::min(ctas, g.pair ? sms / 2 * 2 : sms);
      g.bufs = g.grid < ctas ? 2 : 1;
      lay_out(&g, g.bufs > 1 ? gemm::MAX_STAGES : g.kblocks / g.ks);
      // (a ring of two 64-k blocks, beside the staging of 256 features, leaves the tensor core idle half of the time: prefill of 680
      // tokens 3.32 ms on such a cut, 2.77 on the next best; 1280 tokens 5.55 and 4.90)
      if (g.stages * g.ks < 3) continue;
      best = g;
      best_cost = cost;
    }
  return best;
}

GemmPlan plan_gemm_sk(int sms, int tokens, int n, int k) {
  GemmPlan g = {};
  g.epi = gemm::EPI_PART; g.sk = true; g.bn = 256; g.ks = 1; g.splits = 1; g.bufs = 2;
  g.kblocks = k / gemm::BK;
  g.m_tiles = (tokens + 127) / 128;
  g.rows = g.m_tiles > 1 ? 128 : tokens;
  g.arows = (g.rows + 7) / 8 * 8;
  g.units = g.m_tiles * (n / g.bn);
  const long long work = (long long)g.units * g.kblocks;
  g.grid = work < sms ? (int)work : sms;
  lay_out(&g, gemm::MAX_STAGES);
  return g;
}

cudaError_t launch_gemm(const GemmPlan& g, gemm::Args& p, cudaStream_t stream, bool early) {
  const Cut* cut = nullptr;
  for (const Cut& c : kCuts)
    if (c.epi == g.epi && c.bn == g.bn && c.pair == g.pair && c.ks == g.ks && c.sk == g.sk) cut = &c;
  if (!cut) return cudaErrorInvalidValue;
  p.rows = g.rows; p.arows = g.arows;
  p.m_groups = g.pair ? g.m_tiles / 2 : g.m_tiles; p.splits = g.splits; p.kblocks = g.kblocks;
  p.stages = g.stages; p.bufs = g.bufs; p.off_out = g.off_out;
  p.units = g.units - p.unit0;
  const int ctas = g.pair ? 2 * p.units : p.units, grid = g.sk || g.grid < ctas ? g.grid : ctas;
  return launch_kernel(cut->kernel, grid, gemm::THREADS_G, g.smem, stream, g.pair ? 2 : 1, early, p);
}

namespace {
typedef void (*AttentionKernel)(const attn::Args);
struct Tile { int rows; bool join; AttentionKernel kernel; };
#define TILE(ROWS) {ROWS, false, attn::attention_kernel<ROWS, false>}, {ROWS, true, attn::attention_kernel<ROWS, true>}
const Tile kTiles[] = {TILE(16), TILE(32), TILE(48), TILE(64), TILE(112)};
#undef TILE
}  // namespace

cudaError_t launch_attention(attn::Args& p, int observations, cudaStream_t stream) {
  const int rows = p.tok_tile * NQH;
  for (const Tile& t : kTiles)
    if (t.rows == rows && t.join == (p.m_rows > 0))
      return launch_chained(t.kernel, observations * p.tiles * p.splits, attn::THREADS, attn::smem_for(rows), stream, p.splits, p);
  return cudaErrorInvalidValue;
}

cudaError_t chain_opt_in(const void* kernel, int smem) {
  cudaError_t e = cudaSuccess;
  if (smem) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  return e;
}

cudaError_t opt_in_gemm(const GemmPlan& g, int device) {
  static std::atomic<uint64_t> done[sizeof kCuts / sizeof kCuts[0]];
  for (const Cut& c : kCuts)
    if (c.epi == g.epi && c.bn == g.bn && c.pair == g.pair && c.ks == g.ks && c.sk == g.sk)
      return once_per_device(&done[&c - kCuts], device, [&] { return chain_opt_in((const void*)c.kernel, 222 * 1024); });
  return cudaErrorInvalidValue;
}

cudaError_t opt_in_attention(int tok_tile, bool join, int device) {
  static std::atomic<uint64_t> done[sizeof kTiles / sizeof kTiles[0]];
  for (const Tile& t : kTiles)
    if (t.rows == tok_tile * NQH && t.join == join)
      return once_per_device(&done[&t - kTiles], device, [&] { return chain_opt_in((const void*)t.kernel, attn::smem_for(t.rows)); });
  return cudaErrorInvalidValue;
}

cudaError_t launch_attention_o(const attno::Args& p, int observations, int smem, cudaStream_t stream) {
  return launch_chained(attno::attention_o_kernel<attno::NTHREADS>, observations * NQH * attno::GROUPS, attno::NTHREADS, smem, stream, 1, p);
}

cudaError_t opt_in_attention_o(int device) {
  static std::atomic<uint64_t> done;
  return once_per_device(&done, device, [] { return chain_opt_in((const void*)attno::attention_o_kernel<attno::NTHREADS>, attno::MAX_SMEM); });
}

}  // namespace pi05
