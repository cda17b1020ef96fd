// Gemma-2B prefix-LM prefill on B200 (sm_100a): the step before the action chunk, which turns the embedded prefix
// (image tokens + prompt) into the per-layer key / value cache the chunk engine attends over.
//
// Semantics follow the reference's eager definition (reference/pi05.py:167-195): per layer RMSNorm, q / k / v projections,
// RoPE at the positions of the valid tokens, bidirectional attention among valid tokens, O projection + residual, and
// the GeGLU MLP + residual; every matmul output, product and sum is rounded to BF16 where the reference's BF16 tensors
// round.  The outputs are the post-RoPE keys and the values, [layers, tokens, 1, 256] BF16, the layout pi05_bind takes as
// inputs 22 and 23, so the chunk engine chains after this without a copy.  Of the last layer only the keys and values are
// computed: nothing behind them reaches an output.
//
// A layer is seven launches - QKV projection (+ RoPE), attention, O projection, residual + RMSNorm, gate / up projection
// (+ GeGLU), down projection, residual + RMSNorm - of the tcgen05 kernels in pi05_gemm.cuh and pi05_attention.cuh and of the
// row kernel below, chained with programmatic dependent launches.  The down projection (K = 16384) is a stream-K launch while
// its tiles do not fill half of the SMs.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <new>
#include <string>

#include "../../include/pi05_b200.h"
#include "pi05_ops.h"
using namespace pi05;

namespace pf {

using gemm::hi16;
using gemm::lo16;
using gemm::pack2;
using gemm::rb;

constexpr int H = 2048;            // Gemma-2B width
constexpr int FFN = 16384;         // MLP width
constexpr int LAYERS = 18;
constexpr int SK_TILES = 32;       // most tiles of a stream-K down projection (four tiles of tokens x 8 of features)

// Positions = cumsum(valid) - 1 (reference/pi05.py:173) and the BF16 cos / sin of every (token, rotary index)
// (reference/pi05.py:218-229: FP32 inverse frequencies and phases), 32 tokens per block; block 0 clears the status words.
__global__ void __launch_bounds__(256) tables_kernel(const uint8_t* __restrict__ valid, int tokens, uint32_t* __restrict__ rope,
                                                     unsigned int* status) {
  __shared__ int s_cnt, s_pos[32];
  __shared__ float s_inv[128];
  const int tid = threadIdx.x, lane = tid & 31, t0 = blockIdx.x * 32;
  if (tid == 0) s_cnt = 0;
  if (tid < 128) s_inv[tid] = 1.0f / (float)pow(10000.0, (double)((float)(2 * tid) / 256.0f));
  if (blockIdx.x == 0 && tid < 2) status[tid] = 0u;
  __syncthreads();
  int n = 0;
  for (int i = tid; i < t0; i += 256) n += valid[i] ? 1 : 0;
  for (int sh = 16; sh; sh >>= 1) n += __shfl_xor_sync(0xffffffffu, n, sh);
  if (lane == 0 && n) atomicAdd(&s_cnt, n);
  __syncthreads();
  if (tid < 32) {
    const unsigned bits = __ballot_sync(0xffffffffu, t0 + tid < tokens && valid[t0 + tid] != 0);
    s_pos[tid] = s_cnt + __popc(bits & (0xffffffffu >> (31 - tid))) - 1;
  }
  __syncthreads();
  for (int i = tid; i < 32 * 128; i += 256) {
    const int t = t0 + (i >> 7);
    if (t >= tokens) break;
    const float phase = (float)s_pos[i >> 7] * s_inv[i & 127];
    rope[gemm::rope_at(tokens, t, i & 127)] = pack2((float)cos((double)phase), (float)sin((double)phase));
  }
}

struct NormArgs {
  const __nv_bfloat16* src;        // the residual stream before this kernel
  __nv_bfloat16 *x, *out;          // the residual stream after it, and its norm
  const __nv_bfloat16* w;
  const float* part;
  int m_tiles;
  // stream-K: of every tile the first contributing CTA and their number, and the owner slots' offset
  short first[SK_TILES], count[SK_TILES];
  int owner0;
};

// x = bf16(src + bf16(sum of the parts)); out = Gemma RMSNorm of x (the reference's rms(x, weight, gemma=True),
// reference/pi05.py:178, 192): FP32 normalisation, scale by (1 + weight), one rounding to BF16.  One token per block, four
// columns per thread.  S: slices of partial sums ([S][tokens][2048]); 0: no projection before (the embeddings); -1 and -2: the slots
// of a stream-K launch ([slot][128][256]), -2 with registers for 20 of them, which only a launch of a block per SM at most can afford (256 tokens 1.44 ms, on -2 1.45).
template <int S>
__global__ void __launch_bounds__(512) norm_kernel(const __grid_constant__ NormArgs p) {
  __shared__ float red[16];
  const int c0 = threadIdx.x * 4;
  ptx::grid_dep_launch();
  const size_t at = (size_t)blockIdx.x * H + c0;
  const uint2 wv = __ldg(reinterpret_cast<const uint2*>(p.w + c0));
  ptx::grid_dep_wait();
  const uint2 xv = __ldcg(reinterpret_cast<const uint2*>(p.src + at));
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
  if (S > 0) {
    const size_t slice = (size_t)gridDim.x * H;
    float4 v[S > 0 ? S : 1];
#pragma unroll
    for (int s = 0; s < S; ++s) v[s] = __ldcg(reinterpret_cast<const float4*>(p.part + s * slice + at));
#pragma unroll
    for (int s = 0; s < S; ++s) { a.x += v[s].x; a.y += v[s].y; a.z += v[s].z; a.w += v[s].w; }
  } else if (S < 0) {
    const int tile = (c0 >> 8) * p.m_tiles + (int)(blockIdx.x >> 7);
    const float* q = p.part + (size_t)(blockIdx.x & 127) * 256 + (c0 & 255);
    a = __ldcg(reinterpret_cast<const float4*>(q + (size_t)(p.owner0 + tile) * 32768));
    const int first = p.first[tile], count = p.count[tile];
    const float4* q4 = reinterpret_cast<const float4*>(q + (size_t)first * 32768);
    int s = 0;
    if constexpr (S == -2) {
      // up to 20 slots, all on their way before the first is added: in eights, 19 of them took three trips to L2 (61 tokens: 3.6 us of a kernel of 5; prefill of
      // 128 tokens 1.20 -> 1.18 ms).  What is read beyond the last contributor's is another slot
      float4 v[20];
#pragma unroll
      for (int k = 0; k < 20; k += 4)
        if (k < count) ptx::ld_l2_f4x4(reinterpret_cast<float4(&)[4]>(v[k]), q4 + (size_t)k * 8192, 8192);
#pragma unroll
      for (int k = 0; k < 20; ++k)
        if (k < count) { a.x += v[k].x; a.y += v[k].y; a.z += v[k].z; a.w += v[k].w; }
      s = 20;
    }
#pragma unroll 8
    for (; s < count; ++s) {
      const float4 w = __ldcg(q4 + (size_t)s * 8192);
      a.x += w.x; a.y += w.y; a.z += w.z; a.w += w.w;
    }
  }
  float v[4] = {lo16(xv.x), hi16(xv.x), lo16(xv.y), hi16(xv.y)};
  if (S != 0) {
    v[0] = rb(v[0] + rb(a.x)); v[1] = rb(v[1] + rb(a.y)); v[2] = rb(v[2] + rb(a.z)); v[3] = rb(v[3] + rb(a.w));
  }
  *reinterpret_cast<uint2*>(p.x + at) = make_uint2(pack2(v[0], v[1]), pack2(v[2], v[3]));
  float ss = (v[0] * v[0] + v[1] * v[1]) + (v[2] * v[2] + v[3] * v[3]);
  for (int d = 16; d; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = ss;
  __syncthreads();
  ss = red[threadIdx.x & 15];
  for (int d = 8; d; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
  const float rs = rsqrtf(ss * (1.0f / H) + EPS);
  const float w[4] = {lo16(wv.x), hi16(wv.x), lo16(wv.y), hi16(wv.y)};
#pragma unroll
  for (int e = 0; e < 4; ++e) v[e] = __fmul_rn(__fmul_rn(v[e], rs), __fadd_rn(1.0f, w[e]));
  *reinterpret_cast<uint2*>(p.out + at) = make_uint2(pack2(v[0], v[1]), pack2(v[2], v[3]));
}

typedef void (*NormKernel)(const NormArgs);
NormKernel norm_kernel_for(int splits) {
  return splits == 1 ? norm_kernel<1> : splits == 2 ? norm_kernel<2> : splits == 4 ? norm_kernel<4> : norm_kernel<8>;
}

}  // namespace pf

// =========================================================================================== host side
struct pi05_prefill {
  int device = 0, sms = 0, max_tokens = 0;
  const void* weights[PI05_PREFILL_NUM_WEIGHTS] = {};
  uint8_t* ws = nullptr;
  size_t ws_bytes = 0;
  bool bound = false;
  long long wait_limit = 4000000000ll;
  std::string last_error;
  // workspace offsets
  size_t off_status, off_x, off_n, off_q, off_mixed, off_act, off_rope, off_part;
  size_t part_floats = 0;          // FP32 words of partial sums at off_part
};

namespace {

struct Guard {
  int prev = -1;
  bool ok;
  explicit Guard(int dev) { if (cudaGetDevice(&prev) != cudaSuccess) prev = -1; ok = cudaSetDevice(dev) == cudaSuccess; }
  ~Guard() { if (prev >= 0) cudaSetDevice(prev); }
};

size_t up(size_t v) { return (v + 255) / 256 * 256; }

// How a prefill of `tokens` tokens is launched on a GPU of `sms` SMs: the decisions pi05_prefill_run takes and
// pi05_prefill_plan reports.
struct PrefillPlan {
  int m_tiles;        // 128-token tiles
  bool pairs;         // gate/up and O projections (and the down projection unless it is stream-K) on CTA pairs (256-token tiles)
  bool sk_down;       // down projection as a stream-K launch of 128 x 256 tiles
  GemmPlan qkv, o, gu, down;
  int tok_tile;       // query tokens per attention CTA
};

PrefillPlan plan_prefill(int sms, int tokens) {
  PrefillPlan pl;
  pl.m_tiles = (tokens + 127) / 128;
  // The down projection (K = 16384) as a stream-K launch while its 128-feature tiles would leave more than half of the SMs
  // without work for the longest GEMM of the layer, else cut like the others.
  pl.sk_down = pl.m_tiles * (pf::H / 128) * 2 <= sms;
  // CTA pairs work on 256 tokens at a time: with a single tile of tokens the second CTA of every pair would idle.
  pl.pairs = pl.m_tiles >= 2;
  pl.qkv = plan_gemm(sms, tokens, QKVW, pf::H, gemm::EPI_QKV);
  pl.o = plan_gemm(sms, tokens, pf::H, QD, gemm::EPI_PART, pl.pairs);
  pl.gu = plan_gemm(sms, tokens, 2 * pf::FFN, pf::H, gemm::EPI_GEGLU, pl.pairs);
  pl.down = pl.sk_down ? plan_gemm_sk(sms, tokens, pf::H, pf::FFN) : plan_gemm(sms, tokens, pf::H, pf::FFN, gemm::EPI_PART, 1);
  // The widest tile of query tokens that does not cost a second wave of CTAs: 512 tokens 2.23 ms on tiles of 4, 2.37 on 2 and 2.26
  // on 8; 968 tokens 3.40 on 8 and 3.75 on 4.
  pl.tok_tile = 14;
  for (int t : {8, 6, 4, 2})
    if ((tokens + t - 1) / t <= sms) pl.tok_tile = t;
  return pl;
}

// FP32 words of partial sums of a prefill.
size_t part_floats(const PrefillPlan& pl, int tokens) {
  const size_t o = (size_t)pl.o.splits * tokens * pf::H;
  const size_t d = pl.sk_down ? (size_t)(pl.down.grid + pl.down.units) * 128 * 256 : (size_t)pl.down.splits * tokens * pf::H;
  return std::max(o, d);
}

// The most that a prefill of up to `max_tokens` needs, asked of every count: the cuts do not only follow the number of 128-token
// tiles (148 SMs: K of the down projection over eight CTAs from 641 to 682 tokens, over two from 683 on).  0.24 ms for 968.
size_t most_part_floats(int sms, int max_tokens) {
  size_t most = 0;
  for (int t = 1; t <= max_tokens; ++t) most = std::max(most, part_floats(plan_prefill(sms, t), t));
  return most;
}

cudaError_t prefill_opt_in(int device) {
  static std::atomic<uint64_t> done;
  return once_per_device(&done, device, [] {
    cudaError_t e = cudaSuccess;
    const void* all[] = {(const void*)pf::tables_kernel, (const void*)pf::norm_kernel<-2>, (const void*)pf::norm_kernel<-1>, (const void*)pf::norm_kernel<0>,
                         (const void*)pf::norm_kernel<1>, (const void*)pf::norm_kernel<2>, (const void*)pf::norm_kernel<4>,
                         (const void*)pf::norm_kernel<8>};
    for (const void* k : all)
      if (e == cudaSuccess) e = chain_opt_in(k, 0);
    return e;
  });
}

}  // namespace

extern "C" {

int pi05_prefill_create(int device, int max_tokens, pi05_prefill_t* out) {
  if (!out) return PI05_ERR_ARGUMENT;
  *out = nullptr;
  if (device < 0 || device >= 64 || max_tokens < 1 || max_tokens > 4096) return PI05_ERR_ARGUMENT;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) { cudaGetLastError(); return PI05_ERR_NO_DEVICE; }
  if (device >= ndev) return PI05_ERR_ARGUMENT;
  cudaDeviceProp prop;
  if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) { cudaGetLastError(); return PI05_ERR_NO_DEVICE; }
  if (prop.major != 10) return PI05_ERR_NO_DEVICE;
  pi05_prefill* h = new (std::nothrow) pi05_prefill();
  if (!h) return PI05_ERR_ARGUMENT;
  h->device = device;
  h->sms = prop.multiProcessorCount;
  h->max_tokens = max_tokens;
  const size_t P = (size_t)max_tokens;
  size_t off = 0;
  auto add = [&](size_t bytes) { const size_t at = off; off = up(off + bytes); return at; };
  h->off_status = add(256);
  h->off_x = add(P * pf::H * 2);
  h->off_n = add(P * pf::H * 2);
  h->off_q = add(P * QD * 2);
  h->off_mixed = add(P * QD * 2);
  h->off_act = add(P * (size_t)pf::FFN * 2);
  h->off_rope = add(P * 128 * 4);
  h->part_floats = most_part_floats(h->sms, max_tokens);
  h->off_part = add(h->part_floats * 4);
  h->ws_bytes = off;
  *out = h;
  return PI05_OK;
}

int pi05_prefill_workspace_bytes(pi05_prefill_t h, size_t* bytes) {
  if (!h || !bytes) return PI05_ERR_ARGUMENT;
  *bytes = h->ws_bytes;
  return PI05_OK;
}

const char* pi05_prefill_last_error(pi05_prefill_t h) { return h ? h->last_error.c_str() : "bad handle"; }

int pi05_prefill_bind(pi05_prefill_t h, const void* const weights[PI05_PREFILL_NUM_WEIGHTS], void* workspace,
                      size_t workspace_bytes) {
  if (!h || !weights || !workspace) return PI05_ERR_ARGUMENT;
  if (workspace_bytes < h->ws_bytes || (reinterpret_cast<uintptr_t>(workspace) & 255)) {
    h->last_error = "workspace too small or not 256-byte aligned";
    return PI05_ERR_ARGUMENT;
  }
  for (int i = 0; i < PI05_PREFILL_NUM_WEIGHTS; ++i) {
    if (!weights[i] || (reinterpret_cast<uintptr_t>(weights[i]) & 15)) {
      h->last_error = "weight " + std::to_string(i) + " is null or not 16-byte aligned";
      return PI05_ERR_ARGUMENT;
    }
    h->weights[i] = weights[i];
  }
  h->ws = static_cast<uint8_t*>(workspace);
  h->bound = true;
  return PI05_OK;
}

int pi05_prefill_run(pi05_prefill_t h, const void* embeddings, const void* valid, int tokens, void* keys, void* values,
                     int n_layers, void* stream_) {
  if (!h || !embeddings || !valid || !keys || !values) return PI05_ERR_ARGUMENT;
  if (!h->bound) return PI05_ERR_NOT_BOUND;
  if (tokens < 1 || tokens > h->max_tokens || n_layers < 1 || n_layers > pf::LAYERS) return PI05_ERR_ARGUMENT;
  if ((reinterpret_cast<uintptr_t>(embeddings) & 15) || (reinterpret_cast<uintptr_t>(keys) & 15) ||
      (reinterpret_cast<uintptr_t>(values) & 15)) {
    h->last_error = "embeddings, keys and values must be 16-byte aligned";
    return PI05_ERR_ARGUMENT;
  }
  Guard guard(h->device);
  if (!guard.ok) return PI05_ERR_CUDA;
  cudaStream_t stream = (cudaStream_t)stream_;
  cudaError_t e = prefill_opt_in(h->device);
  if (e != cudaSuccess) { h->last_error = cudaGetErrorString(e); return PI05_ERR_CUDA; }
  const int P = tokens;
  auto ptr = [&](size_t off) { return h->ws + off; };
  __nv_bfloat16* x = reinterpret_cast<__nv_bfloat16*>(ptr(h->off_x));
  __nv_bfloat16* nrm = reinterpret_cast<__nv_bfloat16*>(ptr(h->off_n));
  __nv_bfloat16* q = reinterpret_cast<__nv_bfloat16*>(ptr(h->off_q));
  __nv_bfloat16* mixed = reinterpret_cast<__nv_bfloat16*>(ptr(h->off_mixed));
  __nv_bfloat16* act = reinterpret_cast<__nv_bfloat16*>(ptr(h->off_act));
  uint32_t* rope = reinterpret_cast<uint32_t*>(ptr(h->off_rope));
  unsigned int* status = reinterpret_cast<unsigned int*>(ptr(h->off_status));
  float* part = reinterpret_cast<float*>(ptr(h->off_part));
  const __nv_bfloat16* const* w = reinterpret_cast<const __nv_bfloat16* const*>(h->weights);
  enum { LN1 = 0, LN2, LQ, LK, LV, LO, LG, LU, LD };
  __nv_bfloat16* K = static_cast<__nv_bfloat16*>(keys);
  __nv_bfloat16* V = static_cast<__nv_bfloat16*>(values);
  const PrefillPlan pl = plan_prefill(h->sms, P);
  if (part_floats(pl, P) > h->part_floats) { h->last_error = "the workspace does not hold the partial sums of this prompt"; return PI05_ERR_UNSUPPORTED; }
  for (const GemmPlan* g : {&pl.qkv, &pl.o, &pl.gu, &pl.down})
    if (e == cudaSuccess) e = opt_in_gemm(*g, h->device);
  if (e == cudaSuccess) e = opt_in_attention(pl.tok_tile, false, h->device);
  if (e != cudaSuccess) { h->last_error = cudaGetErrorString(e); return PI05_ERR_CUDA; }

  // tensor maps: activations (rows = tokens, zero beyond), weights (all layers stacked), keys / values for the attention
  CUtensorMap a_qkv, a_o, a_gu, a_dn, wq, wk, wv, wo, wg, wu, wd;
  attn::Args ap;
  memset(&ap, 0, sizeof ap);
  const uint64_t L = pf::LAYERS;
  auto act_map = [&](CUtensorMap* m, const void* base, int k, const GemmPlan& g) { return map_k(m, base, k, P, g.arows, g.ks); };
  auto weight_map = [&](CUtensorMap* m, int which, int k, int rows, const GemmPlan& g) { return map_k(m, w[which], k, L * rows, g.w_rows, g.w_kb); };
  const bool ok = act_map(&a_qkv, nrm, pf::H, pl.qkv) && act_map(&a_o, mixed, QD, pl.o) && act_map(&a_gu, nrm, pf::H, pl.gu) &&
                  act_map(&a_dn, act, pf::FFN, pl.down) && weight_map(&wq, LQ, pf::H, QD, pl.qkv) && weight_map(&wk, LK, pf::H, HD, pl.qkv) &&
                  weight_map(&wv, LV, pf::H, HD, pl.qkv) && weight_map(&wo, LO, QD, pf::H, pl.o) && weight_map(&wg, LG, pf::H, pf::FFN, pl.gu) &&
                  weight_map(&wu, LU, pf::H, pf::FFN, pl.gu) && weight_map(&wd, LD, pf::FFN, pf::H, pl.down) &&
                  map_kv(&ap.pk, K, P, L, 1, HD, (uint64_t)P * HD, L * P * HD, attn::KCH, 2) &&
                  map_kv(&ap.pv, V, P, L, 1, HD, (uint64_t)P * HD, L * P * HD, 64, 4) &&
                  map_k(&ap.q, q, HD, (uint64_t)P * NQH, pl.tok_tile * NQH, HD / 64);
  if (!ok) { h->last_error = "cuTensorMapEncodeTiled failed"; return PI05_ERR_CUDA; }
  ap.pk_tail = ap.pk; ap.pv_tail = ap.pv; ap.sk = ap.pk; ap.sv = ap.pv;
  ap.valid = static_cast<const uint8_t*>(valid); ap.out = mixed;
  ap.pages_per_obs = 1; ap.page_tokens = P; ap.k_rows = attn::KCH; ap.prefix = P; ap.obs_tokens = P;
  ap.tok_tile = pl.tok_tile; ap.tiles = (P + pl.tok_tile - 1) / pl.tok_tile; ap.splits = 1;
  ap.status = status; ap.limit = h->wait_limit;

  auto project = [&](const GemmPlan& g, const CUtensorMap& a, const CUtensorMap& b0, const CUtensorMap* b1, const CUtensorMap* b2,
                     int width, int layer, int unit0 = 0) {
    if (e != cudaSuccess) return;
    gemm::Args p;
    memset(&p, 0, sizeof p);
    p.a = a; p.b0 = b0;
    if (b1) p.b1 = *b1;
    if (b2) p.b2 = *b2;
    p.tokens = P; p.layer = layer; p.width = width; p.unit0 = unit0; p.status = status; p.limit = h->wait_limit;
    p.q = q; p.k = K + (size_t)layer * P * HD; p.v = V + (size_t)layer * P * HD; p.rope = rope; p.act = act; p.part = part;
    e = launch_gemm(g, p, stream);
  };
  pf::NormArgs n;
  memset(&n, 0, sizeof n);
  n.x = x; n.out = nrm; n.part = part; n.m_tiles = pl.m_tiles;
  if (pl.sk_down) {
    n.owner0 = pl.down.grid;
    for (int c = 0; c < pl.down.grid; ++c) {      // every CTA whose range begins inside a tile contributes to that tile
      const long long at = gemm::Segments::begin(pl.down.units, pl.down.kblocks, c, pl.down.grid);
      const int tile = (int)(at / pl.down.kblocks);
      if (at % pl.down.kblocks && n.count[tile]++ == 0) n.first[tile] = (short)c;
    }
  }
  auto norm = [&](pf::NormKernel kernel, const __nv_bfloat16* src, const __nv_bfloat16* weight) {
    n.src = src; n.w = weight;
    if (e == cudaSuccess) e = launch_chained(kernel, P, 512, 0, stream, 1, n);
  };

  pf::tables_kernel<<<(P + 31) / 32, 256, 0, stream>>>(static_cast<const uint8_t*>(valid), P, rope, status);
  e = cudaGetLastError();
  norm(pf::norm_kernel<0>, static_cast<const __nv_bfloat16*>(embeddings), w[LN1]);
  for (int l = 0; l < n_layers && e == cudaSuccess; ++l) {
    if (l + 1 == n_layers) {                      // keys and values only: the tiles behind the eight query heads
      project(pl.qkv, a_qkv, wq, &wk, &wv, 0, l, pl.qkv.units / (NQH + 2) * NQH);
      break;
    }
    project(pl.qkv, a_qkv, wq, &wk, &wv, 0, l);
    ap.layer = l;
    if (e == cudaSuccess) e = launch_attention(ap, 1, stream);
    project(pl.o, a_o, wo, nullptr, nullptr, pf::H, l);
    norm(pf::norm_kernel_for(pl.o.splits), x, w[LN2] + (size_t)l * pf::H);
    project(pl.gu, a_gu, wg, &wu, nullptr, pf::FFN, l);
    project(pl.down, a_dn, wd, nullptr, nullptr, pf::H, l);
    norm(pl.sk_down ? (P <= h->sms ? pf::norm_kernel<-2> : pf::norm_kernel<-1>) : pf::norm_kernel_for(pl.down.splits), x, w[LN1] + (size_t)(l + 1) * pf::H);
  }
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) { h->last_error = std::string("kernel launch: ") + cudaGetErrorString(e); return PI05_ERR_CUDA; }
  return PI05_OK;
}

int pi05_prefill_plan(int sms, int tokens, int cta, int info[PI05_PREFILL_PLAN_INFO], int* segments, int capacity, int* count) {
  if (sms < 2 || sms > 1024 || tokens < 1 || tokens > 4096 || !info || !count || capacity < 0 || (capacity && !segments))
    return PI05_ERR_ARGUMENT;
  const PrefillPlan pl = plan_prefill(sms, tokens);
  const GemmPlan& d = pl.down;
  info[0] = pl.m_tiles; info[1] = pl.pairs; info[2] = pl.sk_down;
  info[3] = pl.sk_down ? d.units : 0; info[4] = pl.sk_down ? d.kblocks : 0; info[5] = pl.sk_down ? d.grid : 0;
  *count = 0;
  if (!pl.sk_down) return PI05_OK;
  if (cta < 0 || cta >= d.grid) return PI05_ERR_ARGUMENT;
  const long long end = gemm::Segments::begin(d.units, d.kblocks, cta + 1, d.grid);
  for (long long at = gemm::Segments::begin(d.units, d.kblocks, cta, d.grid); at < end; ++*count) {
    const int tile = (int)(at / d.kblocks), kb0 = (int)(at % d.kblocks);
    const int kb1 = (int)std::min<long long>(d.kblocks, kb0 + (end - at));
    if (*count < capacity) { segments[3 * *count] = tile; segments[3 * *count + 1] = kb0; segments[3 * *count + 2] = kb1; }
    at += kb1 - kb0;
  }
  return PI05_OK;
}

int pi05_prefill_partials(int sms, int max_tokens, int tokens, size_t* held, size_t* needed) {
  if (sms < 2 || sms > 1024 || max_tokens < 1 || max_tokens > 4096 || tokens < 1 || tokens > max_tokens || !held || !needed)
    return PI05_ERR_ARGUMENT;
  *held = most_part_floats(sms, max_tokens);
  *needed = part_floats(plan_prefill(sms, tokens), tokens);
  return PI05_OK;
}

int pi05_prefill_status(pi05_prefill_t h, void* stream, int* code, int* where) {
  if (!h || !code || !where) return PI05_ERR_ARGUMENT;
  if (!h->ws) return PI05_ERR_NOT_BOUND;
  Guard guard(h->device);
  if (!guard.ok) return PI05_ERR_CUDA;
  unsigned int st[2] = {0, 0};
  cudaError_t e = cudaMemcpyAsync(st, h->ws + h->off_status, sizeof st, cudaMemcpyDeviceToHost, (cudaStream_t)stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) { h->last_error = cudaGetErrorString(e); return PI05_ERR_CUDA; }
  *code = (int)st[0];
  *where = (int)(st[1] >> 16);               // the block
  return st[0] ? PI05_ERR_DEVICE_TIMEOUT : PI05_OK;
}

int pi05_prefill_destroy(pi05_prefill_t h) {
  if (!h) return PI05_ERR_ARGUMENT;
  delete h;
  return PI05_OK;
}

}  // extern "C"
