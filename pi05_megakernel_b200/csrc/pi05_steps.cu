// The action chunk as a chain of kernels, one set per layer pass, replayed from CUDA graphs.
//
// A layer pass is seven kernels - QKV projection (+ RoPE), attention, O projection, gated residual + adaRMS, gate / up
// projection (+ GeGLU), down projection, gated residual + adaRMS; of short prefixes attention and O projection are one - and an Euler step is 18 of them, the last residual being
// the step tail.  The step's kernels are captured once per binding; the Euler step index and the number of steps live in
// device memory, so the same graph is launched once per step.  What the graphs do not fit - fewer layers, a stream that is being
// captured, another wait limit than at bind - is launched kernel by kernel: a launch never builds a graph.  Every kernel but the
// first of a step is launched with programmatic stream serialisation: its CTAs become
// resident, set up and request their weights (or cached keys) while the kernel before it runs, and wait for it only
// before they touch what it wrote.  Measured on B200, a hop along such a chain (last store to first load) costs 1.25 us
// against 1.75-2.3 us for a device-scope counter of a persistent kernel, and every stage may use all SMs.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <string>

#include "../../include/pi05_b200.h"
#include "pi05_ops.h"
#include "pi05_steps.h"

namespace pi05 {
namespace {

static_assert(WAIT_W_EMPTY == PI05_WAIT_WEIGHT_SLOT && WAIT_W_FULL == PI05_WAIT_WEIGHT_DATA && WAIT_A_EMPTY == PI05_WAIT_ACT_SLOT &&
              WAIT_T_EMPTY == PI05_WAIT_TMEM_SLOT && WAIT_T_FULL == PI05_WAIT_TMEM_DATA && WAIT_DRAIN == PI05_WAIT_DRAIN &&
              attn::WAIT_KV_EMPTY == PI05_WAIT_KV_SLOT && attn::WAIT_KV_FULL == PI05_WAIT_KV_DATA && attn::WAIT_Q_FULL == PI05_WAIT_QUERIES &&
              attn::WAIT_S_EMPTY == PI05_WAIT_SCORE_SLOT && attn::WAIT_S_FULL == PI05_WAIT_SCORES && attn::WAIT_P_FULL == PI05_WAIT_PROBS &&
              attn::WAIT_P_EMPTY == PI05_WAIT_PROBS_SLOT && attn::WAIT_O_FULL == PI05_WAIT_OUTPUT, "status codes of the interface");

using gemm::hi16;
using gemm::lo16;
using gemm::pack2;
using gemm::rb;

// ------------------------------------------------------------------------------------------- prologue
struct TableArgs {
  float t_steps[NS];
  float* temb;
  uint32_t *rope, *rope4;                    // [token][128] (no kernel of the chain reads it: the region that callers know as "rope"), and as the QKV epilogue reads it
  const uint8_t* mask;
  int* state;
  int prefix, n_steps;
};

// Time embedding (FP64, reference/pi05.py:232-237), RoPE tables of the suffix positions (reference/pi05.py:218-229, they
// start at the observation's number of valid prefix tokens) and the step state.  blockIdx.y = observation.
__global__ void __launch_bounds__(256) tables_kernel(const TableArgs p) {
  const int b = blockIdx.y, tid = threadIdx.x, gtid = blockIdx.x * 256 + tid, gn = gridDim.x * 256;
  __shared__ int s_cnt;
  if (tid == 0) s_cnt = 0;
  __syncthreads();
  int n = 0;
  for (int i = tid; i < p.prefix; i += 256) n += p.mask[(size_t)b * p.prefix + i] ? 1 : 0;
  for (int sh = 16; sh; sh >>= 1) n += __shfl_xor_sync(0xffffffffu, n, sh);
  if ((tid & 31) == 0 && n) atomicAdd(&s_cnt, n);
  __syncthreads();
  const int nvalid = s_cnt;
  for (int i = gtid; i < T * (HD / 2); i += gn) {
    const int t = i / (HD / 2), j = i % (HD / 2);
    const float e = (float)(2 * j) / (float)HD;
    const float inv = 1.0f / (float)pow(10000.0, (double)e);
    const float phase = (float)(nvalid + t) * inv;
    const uint32_t cs = pack2((float)cos((double)phase), (float)sin((double)phase));
    p.rope[(size_t)b * T * (HD / 2) + i] = cs;
    p.rope4[gemm::rope_at(gridDim.y * T, b * T + t, j)] = cs;
  }
  if (b == 0) {
    for (int i = gtid; i < NS * W; i += gn) {
      const int s = i / W, j = i % W, f = j % (W / 2);
      const double step = 1.0 / (W / 2 - 1);
      const double frac = f < (W / 4) ? step * f : 1.0 - step * (W / 2 - 1 - f);
      const double period = 4e-3 * pow(4.0 / 4e-3, frac);
      const double phase = (double)p.t_steps[s] * (1.0 / period * 2 * 3.141592653589793);
      p.temb[i] = (float)(j < W / 2 ? sin(phase) : cos(phase));
    }
    if (gtid < 3) p.state[gtid] = gtid == 2 ? p.n_steps : 0;
  }
}

struct MatArgs {
  const float* in;                           // [10][1024]
  const float *w[3], *b[3];                  // modulation: attention norms, feed-forward norms, final norm
  float* out;
};

// One layer of the time MLP for the ten time steps at once: out[s][row] = silu(W[row][:] . in[s][:] + bias[row]).  A warp
// per row; the whole row is requested before the kernel before this one has finished.
__global__ void __launch_bounds__(256) time_mlp_kernel(const MatArgs p) {
  const int lane = threadIdx.x & 31, row = blockIdx.x * 8 + (threadIdx.x >> 5);
  ptx::grid_dep_launch();
  float4 w[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) w[j] = ptx::ldg_stream_f4(p.w[0] + (size_t)row * W + j * 128 + lane * 4);
  const float bias = __ldg(p.b[0] + row);
  ptx::grid_dep_wait();
  float mine = 0.f;
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    float a = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float4 v = __ldcg(reinterpret_cast<const float4*>(p.in + s * W) + j * 32 + lane);
      a = fmaf(w[j].x, v.x, a); a = fmaf(w[j].y, v.y, a); a = fmaf(w[j].z, v.z, a); a = fmaf(w[j].w, v.w, a);
    }
    for (int sh = 16; sh; sh >>= 1) a += __shfl_xor_sync(0xffffffffu, a, sh);
    if (lane == s) mine = a;
  }
  if (lane < NS) {
    const float y = mine + bias;
    p.out[(size_t)lane * W + row] = y / (1.0f + expf(-y));
  }
}

// The 37 modulation layers for the ten time steps at once: out[s][row] = W[row][:] . in[s][:] + bias[row]; the 474 MB of FP32
// weights are streamed from HBM exactly once.  A warp takes four rows; lane l covers k = 4 l .. 4 l + 3 of every 128, the
// ten vectors lie in shared memory, products are accumulated in packed FP32 pairs.  What bounds it is how much is on its way from HBM: a lane copies the
// 16 bytes of each row that it will use itself into a ring of four stages of 128 columns, 96 KB in flight per SM.  (With the next 128 columns in registers,
// 32 KB in flight, a chunk took 26 to 38 us longer: 4.223 and 4.196 ms at prefix 128.)
constexpr int MOD_THREADS = 512, MOD_STAGES = 4, MOD_R = 4;
constexpr int MOD_SMEM = NS * W * 4 + MOD_THREADS / 32 * MOD_STAGES * MOD_R * 512;
__global__ void __launch_bounds__(MOD_THREADS, 1) modulation_kernel(const MatArgs p) {
  constexpr int R = MOD_R;
  extern __shared__ __align__(16) float s_dyn[];
  float4* c = reinterpret_cast<float4*>(s_dyn);             // [10][256]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float4* ring = c + NS * W / 4 + warp * (MOD_STAGES * R * 32) + lane;
  ptx::grid_dep_launch();
  const int nrows = NNORM * MODW, step = gridDim.x * (MOD_THREADS / 32) * R;
  auto weights = [&](int row0, const float*& bias) -> const float* {
    const int n = row0 / MODW, j = row0 - n * MODW, which = n == NNORM - 1 ? 2 : (n & 1);
    const size_t r = which == 2 ? (size_t)j : (size_t)(n >> 1) * MODW + j;
    bias = p.b[which] + r;
    return p.w[which] + r * W + lane * 4;
  };
  int row0 = (blockIdx.x * (MOD_THREADS / 32) + warp) * R;
  const float *wrow = nullptr, *bias = nullptr;
  if (row0 < nrows) wrow = weights(row0, bias);
  auto request = [&](const float* w, int j) {
    if (w)
#pragma unroll
      for (int r = 0; r < R; ++r) ptx::copy_async_16(ring + ((j & (MOD_STAGES - 1)) * R + r) * 32, w + (size_t)r * W + j * 128);
    ptx::copy_async_commit();
  };
#pragma unroll
  for (int j = 0; j < MOD_STAGES - 1; ++j) request(wrow, j);
  ptx::grid_dep_wait();
  for (int i = tid; i < NS * W / 4; i += MOD_THREADS) c[i] = __ldcg(reinterpret_cast<const float4*>(p.in) + i);
  __syncthreads();
  for (; row0 < nrows; row0 += step) {
    float2 acc[R][NS];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int s = 0; s < NS; ++s) acc[r][s] = make_float2(0.f, 0.f);
    const float *bcur = bias, *wnext = nullptr;
    if (row0 + step < nrows) wnext = weights(row0 + step, bias);
#pragma unroll
    for (int j = 0; j < W / 128; ++j) {
      if (j + MOD_STAGES - 1 < W / 128) request(wrow, j + MOD_STAGES - 1);
      else request(wnext, j + MOD_STAGES - 1 - W / 128);
      ptx::copy_async_wait<MOD_STAGES - 1>();
      float4 w[R];
#pragma unroll
      for (int r = 0; r < R; ++r) w[r] = ring[((j & (MOD_STAGES - 1)) * R + r) * 32];
#pragma unroll
      for (int s = 0; s < NS; ++s) {
        const float4 v = c[s * (W / 4) + j * 32 + lane];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          acc[r][s] = ptx::fma2(make_float2(w[r].x, w[r].y), make_float2(v.x, v.y), acc[r][s]);
          acc[r][s] = ptx::fma2(make_float2(w[r].z, w[r].w), make_float2(v.z, v.w), acc[r][s]);
        }
      }
    }
    wrow = wnext;
    // 40 sums over the 32 lanes: fold the lanes' halves together while halving the number of values each lane keeps
    float v[40];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
      for (int s = 0; s < NS; ++s) v[r * NS + s] = acc[r][s].x + acc[r][s].y;
#pragma unroll
    for (int i = 0; i < 20; ++i) {
      const float keep = lane & 16 ? v[i + 20] : v[i], send = lane & 16 ? v[i] : v[i + 20];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
#pragma unroll
    for (int i = 0; i < 10; ++i) {
      const float keep = lane & 8 ? v[i + 10] : v[i], send = lane & 8 ? v[i] : v[i + 10];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      const float keep = lane & 4 ? v[i + 5] : v[i], send = lane & 4 ? v[i] : v[i + 5];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
      v[i] += __shfl_xor_sync(0xffffffffu, v[i], 2);
      v[i] += __shfl_xor_sync(0xffffffffu, v[i], 1);
    }
    if ((lane & 3) == 0) {
      const int base = (lane & 16 ? 20 : 0) + (lane & 8 ? 10 : 0) + (lane & 4 ? 5 : 0);
#pragma unroll
      for (int i = 0; i < 5; ++i) {
        const int r = (base + i) / NS, s = (base + i) % NS;
        p.out[(size_t)s * NNORM * MODW + row0 + r] = v[i] + __ldg(bcur + r);
      }
    }
  }
}

// ------------------------------------------------------------------------------------------- row kernels
struct NormArgs {
  const float* part;                         // [splits][tokens][1024] partial sums of the projection before
  __nv_bfloat16 *h, *out;
  const float* mod;
  const int* state;
  int gate_norm, next_norm;
};

// h += bf16(bf16(sum of the parts) * bf16(gate)); out = adaRMS(h) with the next norm's scale and shift
// (reference/pi05.py:240-279).  One token per block, four columns per thread (every load of a warp covers whole lines).
template <int S>
__global__ void __launch_bounds__(256) residual_norm_kernel(const NormArgs p) {
  __shared__ float red[2][8];
  const int c0 = threadIdx.x * 4;
  ptx::grid_dep_launch();
  // the modulation was finished before the step began (its first kernel does not start early), and the step counter only moves at
  // the end of a step
  const float* mod_s = p.mod + (size_t)__ldcg(p.state) * NNORM * MODW;
  const float4 g = __ldcg(reinterpret_cast<const float4*>(mod_s + (size_t)p.gate_norm * MODW + 2 * W + c0));
  const float4 sc = __ldcg(reinterpret_cast<const float4*>(mod_s + (size_t)p.next_norm * MODW + c0));
  const float4 sh = __ldcg(reinterpret_cast<const float4*>(mod_s + (size_t)p.next_norm * MODW + W + c0));
  const float gate[4] = {g.x, g.y, g.z, g.w}, scale[4] = {sc.x, sc.y, sc.z, sc.w}, shift[4] = {sh.x, sh.y, sh.z, sh.w};
  const size_t at = (size_t)blockIdx.x * W + c0, slice = (size_t)gridDim.x * W / 4;
  const float4* a4 = reinterpret_cast<const float4*>(p.part + at);
  // The first pass is a dry one: it brings the code (fetched once per launch otherwise, at several cycles an instruction) and the
  // address translations into the caches while the kernel before this one runs.  50 tokens: 0.9 us from the end of that kernel
  // to the last store, 1.2 without
#pragma unroll 1
  for (int pass = 0; pass < 2; ++pass) {
    if (pass) ptx::grid_dep_wait();
    float4 a[S];
    if constexpr (S == 8) {
      ptx::ld_l2_f4x4(reinterpret_cast<float4(&)[4]>(a[0]), a4, slice);
      ptx::ld_l2_f4x4(reinterpret_cast<float4(&)[4]>(a[4]), a4 + 4 * slice, slice);
    } else {
#pragma unroll
      for (int s = 0; s < S; ++s) a[s] = __ldcg(a4 + s * slice);
    }
    const uint2 hv = __ldcg(reinterpret_cast<const uint2*>(p.h + at));
#pragma unroll
    for (int s = 1; s < S; ++s) { a[0].x += a[s].x; a[0].y += a[s].y; a[0].z += a[s].z; a[0].w += a[s].w; }
    const float av[4] = {a[0].x, a[0].y, a[0].z, a[0].w}, hw[4] = {lo16(hv.x), hi16(hv.x), lo16(hv.y), hi16(hv.y)};
    float v[4], ss = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[e] = rb(hw[e] + rb(rb(av[e]) * rb(gate[e])));
      ss += v[e] * v[e];
    }
    if (pass) *reinterpret_cast<uint2*>(p.h + at) = make_uint2(pack2(v[0], v[1]), pack2(v[2], v[3]));
    for (int d = 16; d; d >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, d);
    if ((threadIdx.x & 31) == 0) red[pass][threadIdx.x >> 5] = ss;
    __syncthreads();
    ss = ((red[pass][0] + red[pass][1]) + (red[pass][2] + red[pass][3])) + ((red[pass][4] + red[pass][5]) + (red[pass][6] + red[pass][7]));
    const float rs = 1.0f / sqrtf(ss * (1.0f / W) + EPS);
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = __fadd_rn(__fmul_rn(__fmul_rn(v[e], rs), __fadd_rn(1.0f, scale[e])), shift[e]);
    if (pass) *reinterpret_cast<uint2*>(p.out + at) = make_uint2(pack2(o[0], o[1]), pack2(o[2], o[3]));
  }
}

struct TailArgs {
  const float* part;
  __nv_bfloat16 *h, *out;
  const float* mod;
  int* state;
  const float *noise, *ain_w, *ain_b, *aout_w, *aout_b;
  float *x, *actions;
  const unsigned int* status;
  float dt;
  int gate_norm, tokens, splits;
};

constexpr int TAIL_THREADS = 256;
constexpr int TAIL_SMEM = W * ADIM * 4 + W * 4;

// The end of an Euler step (INIT: the beginning of the first): residual of the last layer, final adaRMS, action_out, Euler
// update, and - unless it was the last step - action_in and the first layer's norm for the next step (reference/pi05.py:282-309).
// A block works through tokens blockIdx.x, + gridDim.x, ...; action_in's weights wait in shared memory and action_out's in
// registers, both requested before the kernel before this one has finished.
template <bool INIT>
__global__ void __launch_bounds__(TAIL_THREADS, 1) tail_kernel(const TailArgs p) {
  extern __shared__ __align__(16) float s_dyn[];
  float4* s_in = reinterpret_cast<float4*>(s_dyn);          // [1024 rows][8 pieces], piece c of row r at c ^ (r & 7)
  float* s_row = s_dyn + W * ADIM;                          // [1024]
  __shared__ float red[8], s_x[ADIM];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c0 = tid * 4;
  ptx::grid_dep_launch();
  const int4 state = INIT ? make_int4(-1, 0, 0, 0) : __ldcg(reinterpret_cast<const int4*>(p.state));
  const int step = state.x;
  const bool last = !INIT && step + 1 == state.z;
  float4 wo[4][8];                                          // action_out rows 4 warp .. 4 warp + 3, columns 4 lane + 128 j
  if (!INIT) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int j = 0; j < 8; ++j) wo[r][j] = __ldg(reinterpret_cast<const float4*>(p.aout_w + (size_t)(warp * 4 + r) * W) + lane + 32 * j);
  }
  if (!last)
    for (int i = tid; i < W * 8; i += TAIL_THREADS) s_in[(i & ~7) | ((i & 7) ^ ((i >> 3) & 7))] = __ldg(reinterpret_cast<const float4*>(p.ain_w) + i);
  auto block_sum = [&](float v) {
    for (int sh = 16; sh; sh >>= 1) v += __shfl_xor_sync(0xffffffffu, v, sh);
    __syncthreads();
    if (lane == 0) red[warp] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += red[i];
    return s;
  };
  ptx::grid_dep_wait();
  for (int t = blockIdx.x; t < p.tokens; t += gridDim.x) {
    if (!INIT) {
      const size_t at = (size_t)t * W + c0;
      const float* mod_s = p.mod + (size_t)step * NNORM * MODW;
      const float4 g = __ldcg(reinterpret_cast<const float4*>(mod_s + (size_t)p.gate_norm * MODW + 2 * W + c0));
      const float4 sc = __ldcg(reinterpret_cast<const float4*>(mod_s + (size_t)(NNORM - 1) * MODW + c0));
      const float4 sh = __ldcg(reinterpret_cast<const float4*>(mod_s + (size_t)(NNORM - 1) * MODW + W + c0));
      const uint2 hv = __ldcg(reinterpret_cast<const uint2*>(p.h + at));
      float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
      for (int s = 0; s < p.splits; ++s) {
        const float4 b = __ldcg(reinterpret_cast<const float4*>(p.part + ((size_t)s * p.tokens) * W + at));
        a.x += b.x; a.y += b.y; a.z += b.z; a.w += b.w;
      }
      float v[4];
      v[0] = rb(lo16(hv.x) + rb(rb(a.x) * rb(g.x)));
      v[1] = rb(hi16(hv.x) + rb(rb(a.y) * rb(g.y)));
      v[2] = rb(lo16(hv.y) + rb(rb(a.z) * rb(g.z)));
      v[3] = rb(hi16(hv.y) + rb(rb(a.w) * rb(g.w)));
      const float rs = 1.0f / sqrtf(block_sum((v[0] * v[0] + v[1] * v[1]) + (v[2] * v[2] + v[3] * v[3])) * (1.0f / W) + EPS);
      const float sca[4] = {sc.x, sc.y, sc.z, sc.w}, sha[4] = {sh.x, sh.y, sh.z, sh.w};
#pragma unroll
      for (int e = 0; e < 4; ++e)
        s_row[c0 + e] = rb(__fadd_rn(__fmul_rn(__fmul_rn(v[e], rs), __fadd_rn(1.0f, sca[e])), sha[e]));
      __syncthreads();
      float dot[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 n = reinterpret_cast<const float4*>(s_row)[lane + 32 * j];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          dot[r] = fmaf(wo[r][j].x, n.x, dot[r]); dot[r] = fmaf(wo[r][j].y, n.y, dot[r]);
          dot[r] = fmaf(wo[r][j].z, n.z, dot[r]); dot[r] = fmaf(wo[r][j].w, n.w, dot[r]);
        }
      }
#pragma unroll
      for (int r = 0; r < 4; ++r)
        for (int sh2 = 16; sh2; sh2 >>= 1) dot[r] += __shfl_xor_sync(0xffffffffu, dot[r], sh2);
      if (lane < 4) {
        const int a4 = warp * 4 + lane;
        const float d = lane == 0 ? dot[0] : lane == 1 ? dot[1] : lane == 2 ? dot[2] : dot[3];
        const float xn = __fadd_rn(p.x[(size_t)t * ADIM + a4], __fmul_rn(p.dt, d + __ldg(p.aout_b + a4)));
        p.x[(size_t)t * ADIM + a4] = xn;
        s_x[a4] = xn;
        // a chunk in which a bounded wait gave up must not be mistaken for a result
        if (last) p.actions[(size_t)t * ADIM + a4] = ptx::ld_relaxed(p.status) != 0u ? __int_as_float(0x7fc00000) : xn;
      }
    } else if (tid < ADIM) {
      const float xv = __ldg(p.noise + (size_t)t * ADIM + tid);
      p.x[(size_t)t * ADIM + tid] = xv;
      s_x[tid] = xv;
    }
    __syncthreads();
    if (last) continue;
    // h = bf16(Win x + b) and the next norm, columns tid, tid + 256, ..
    const float* mod_n = p.mod + (size_t)(step + 1) * NNORM * MODW;
    float y[4], ss = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int col = tid + TAIL_THREADS * e;
      float a = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float4 w4 = s_in[col * 8 + (k ^ (col & 7))];
        a = fmaf(w4.x, s_x[4 * k], a); a = fmaf(w4.y, s_x[4 * k + 1], a);
        a = fmaf(w4.z, s_x[4 * k + 2], a); a = fmaf(w4.w, s_x[4 * k + 3], a);
      }
      y[e] = rb(a + __ldg(p.ain_b + col));
      ss += y[e] * y[e];
      p.h[(size_t)t * W + col] = __float2bfloat16_rn(y[e]);
    }
    const float rs = 1.0f / sqrtf(block_sum(ss) * (1.0f / W) + EPS);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int col = tid + TAIL_THREADS * e;
      p.out[(size_t)t * W + col] = __float2bfloat16_rn(
          __fadd_rn(__fmul_rn(__fmul_rn(y[e], rs), __fadd_rn(1.0f, __ldcg(mod_n + col))), __ldcg(mod_n + W + col)));
    }
  }
  if (!INIT) {
    // the last block to finish moves the step counter: every block has read it by then
    __syncthreads();
    if (tid == 0) {
      __threadfence();
      if (atomicAdd(p.state + 1, 1) == (int)gridDim.x - 1) {
        p.state[1] = 0;
        p.state[0] = step + 1;
      }
    }
  }
}

// =========================================================================================== host side
// How the attention of `batch` observations is cut: `tok_tile` query tokens per CTA, the keys of a tile over `splits` CTAs of a
// cluster, the suffix in the last chunk of the prefix (`join`) or in one of its own.
struct AttnPlan { int tok_tile, tiles, splits; bool join; };

// Whether attention and O projection run as one kernel: where all keys fit into shared memory and a CTA per head and 128 output features is at most one
// round.  Prefix 128: 4.66 -> 4.36 ms, 40: 4.61 -> 4.22, two observations at 100: 5.01 -> 4.97; three would be two rounds.
bool with_o(int sms, int batch, int prefix) {
  return prefix <= attno::MAX_PREFIX && batch * NQH * attno::GROUPS <= sms;
}

// Whether the suffix joins the last chunk of the prefix: cached keys there, padded to 8, and the 50 of the suffix are at most 128, and the cached ones
// are one copy (a page holds them).  968 tokens: eight chunks instead of nine.
bool joins(int prefix, int page_tokens) {
  const int rows = (prefix - (prefix - 1) / attn::KCH * attn::KCH + 7) / 8 * 8;
  return rows <= 72 && (rows <= 64 || prefix <= page_tokens || page_tokens % attn::KCH == 0);
}

// The cuts of `batch` observations and the part of their cost (in us, below) that does not depend on the keys: per chunk, `fixed`; `share`: of the
// fetches of cached keys that contend.
struct AttnCuts {
  struct Cut { int tok_tile, tiles, splits, shift, rounds; double chunk, fixed, share; } cut[20];
  int n;
};
AttnCuts attention_cuts(int sms, int batch) {
  AttnCuts a;
  a.n = 0;
  for (int t : {2, 4, 6, 8, 14})
    for (int shift = 0; shift < 4; ++shift) {
      const int splits = 1 << shift, tiles = (T + t - 1) / t, ctas = batch * tiles * splits;
      // (a cluster is resident as a whole, and those of four and eight CTAs leave some SMs without: four observations of 968 tokens on 144 CTAs in
      // clusters of four 8.4 ms, on 112 7.0)
      if (splits > 1 && ctas > (splits == 8 ? sms * 3 / 4 : splits == 4 ? sms * 7 / 8 : sms)) continue;
      AttnCuts::Cut& c = a.cut[a.n++];
      c.tok_tile = t; c.tiles = tiles; c.splits = splits; c.shift = shift; c.rounds = (ctas + sms - 1) / sms;
      c.chunk = 1.28 + 0.03 * t;
      c.fixed = (t <= 4 ? 0.28 * (t - 2) : 0.42 * t - 1.1) + (splits > 1 ? 1.5 + 0.2 * t + (batch > 1 ? 0.9 : 0.0) : 0.0);
      c.share = 0.5 + 0.5 * std::min(ctas, sms) / sms;
    }
  return a;
}

// `prefix_chunks` chunks of 128 cached tokens; `may_join`: the suffix fits into the last of them; `pages`: 0 where an observation's keys lie in one page, else 64 or
// 128, the tokens that one copy brings of several pages.  The times behind the cost, in us, were fitted to every cut
// timed by itself at 1 to 16 observations and 128 to 968 tokens, and then to whole chunks: a chunk of 128 keys, what a tile costs besides, a merge (dearer
// with several observations, whose next kernels' CTAs wait for the clusters to leave), the copies of a joined chunk.  One chunk per CTA on a cluster of four:
// 300 tokens 4.84 -> 4.64 ms (apart, 2 tokens x 4 CTAs, against joined on one), 384 4.86 -> 4.62; joined: 968 tokens 5.05 -> 4.85, two observations 5.99 -> 5.87.
// Over several pages (fitted to all cuts at 1 to 16 observations, 129 to 1024 tokens) a chunk of cached keys costs 0.15 us more, on pages of 64 0.45, the half of it
// where few CTAs fetch them, and joining the suffix saves the less the more chunks a CTA takes, behind which its own chunk would hide. Without these terms three
// observations of 552 tokens on pages of 64 took 7.29 ms on joined tiles of 2 tokens, against 6.72 on 6 tokens x 4 CTAs, sixteen of 959 on pages of 128 12.76 against
// 12.63 apart.
AttnPlan plan_attention(const AttnCuts& cuts, int prefix_chunks, bool may_join, int pages) {
  AttnPlan best = {};
  double best_cost = 1e30;
  const double page_cost = pages == 0 ? 0.0 : pages == attn::KCH ? 0.15 : 0.45;
  for (int join = may_join ? 1 : 0; join >= 0; --join)
    for (int i = 0; i < cuts.n; ++i) {
      const AttnCuts::Cut& c = cuts.cut[i];
      const int chunks = prefix_chunks + (join ? 0 : 1), per_cta = (chunks + c.splits - 1) >> c.shift;
      if (c.splits > chunks) continue;
      const double joined = !join ? 0.0 : pages ? 0.18 * per_cta + (pages == attn::KCH ? 0.3 : 0.0) : 0.8;
      const double paged = page_cost * c.share * (per_cta - (join || c.splits > 1 ? 0 : 1));
      const double cost = (per_cta * c.chunk + paged + joined) * c.rounds + c.fixed;
      if (cost >= best_cost) continue;
      best_cost = cost;
      best.tok_tile = c.tok_tile; best.tiles = c.tiles; best.splits = c.splits; best.join = join != 0;
    }
  return best;
}
AttnPlan plan_attention_for(int sms, int batch, int prefix, int page_tokens) {
  return plan_attention(attention_cuts(sms, batch), (prefix + attn::KCH - 1) / attn::KCH, joins(prefix, page_tokens), prefix <= page_tokens ? 0 : page_tokens % attn::KCH ? 64 : attn::KCH);
}

typedef void (*NormKernel)(const NormArgs);
NormKernel norm_kernel_for(int splits) {
  return splits == 1 ? residual_norm_kernel<1> : splits == 2 ? residual_norm_kernel<2> : splits == 4 ? residual_norm_kernel<4> : residual_norm_kernel<8>;
}

// Launch settings of the chain's own kernels, once per device.
cudaError_t opt_in(int device) {
  static std::atomic<uint64_t> done;
  return once_per_device(&done, device, [] {
    const struct { const void* kernel; int smem; } all[] = {
        {(const void*)tail_kernel<false>, TAIL_SMEM}, {(const void*)tail_kernel<true>, TAIL_SMEM},
        {(const void*)residual_norm_kernel<1>, 0}, {(const void*)residual_norm_kernel<2>, 0},
        {(const void*)residual_norm_kernel<4>, 0}, {(const void*)residual_norm_kernel<8>, 0},
        {(const void*)modulation_kernel, MOD_SMEM}, {(const void*)time_mlp_kernel, 0}, {(const void*)tables_kernel, 0}};
    cudaError_t e = cudaSuccess;
    for (const auto& k : all)
      if (e == cudaSuccess) e = chain_opt_in(k.kernel, k.smem);
    return e;
  });
}

// The kernels of a chunk, launched into `stream`, which may be one that is being captured.
struct Chain {
  const StepSetup& s;
  int n_steps, n_layers, kernels = 0, fused_smem = 0;
  cudaStream_t stream;
  cudaError_t e;
  std::string what;
  GemmPlan pq, po, pg, pd;
  CUtensorMap a_qkv, a_short, a_o, a_gu, a_dn, wq, wk, wv, wo, wg, wu, wd;
  attn::Args ap;
  attno::Args fp;
  bool join, fused;                                // attention and O projection as one kernel

  Chain(const StepSetup& setup, int steps, int layers, cudaStream_t into) : s(setup), n_steps(steps), n_layers(layers), stream(into) {
    const int tokens = T * s.batch;
    pq = plan_gemm(s.sms, tokens, QKVW, W, gemm::EPI_QKV);
    po = plan_gemm(s.sms, tokens, W, QD, gemm::EPI_PART);
    pg = plan_gemm(s.sms, tokens, 2 * FF, W, gemm::EPI_GEGLU);
    pd = plan_gemm(s.sms, tokens, W, FF, gemm::EPI_PART);
    const AttnPlan pa = plan_attention_for(s.sms, s.batch, s.prefix, s.page_tokens);
    join = pa.join;
    memset(&ap, 0, sizeof ap);
    ap.tok_tile = pa.tok_tile; ap.tiles = pa.tiles; ap.splits = pa.splits;
    e = opt_in(s.device);
    for (const GemmPlan* g : {&pq, &po, &pg, &pd})
      if (e == cudaSuccess && !(g == &po && with_o(s.sms, s.batch, s.prefix))) e = opt_in_gemm(*g, s.device);
    fused = with_o(s.sms, s.batch, s.prefix);
    if (fused) po.splits = NQH;
    if (e == cudaSuccess) e = fused ? opt_in_attention_o(s.device) : opt_in_attention(ap.tok_tile, join, s.device);
    if (e == cudaSuccess) encode();
  }

  template <typename... P, typename... A>
  void put(void (*kernel)(P...), int grid, int block, size_t smem, int cluster, A&&... args) {
    if (e != cudaSuccess) return;
    e = launch_chained(kernel, grid, block, smem, stream, cluster, std::forward<A>(args)...);
    ++kernels;
  }

  TailArgs tail_args() const {
    TailArgs t;
    memset(&t, 0, sizeof t);
    t.part = s.part; t.h = s.h; t.out = s.an; t.mod = s.mod; t.state = s.state;
    t.noise = (const float*)s.in[21];
    t.ain_w = (const float*)s.in[0]; t.ain_b = (const float*)s.in[1];
    t.aout_w = (const float*)s.in[6]; t.aout_b = (const float*)s.in[7];
    t.x = s.x; t.actions = s.actions; t.status = s.status; t.dt = (float)(-1.0 / NS);
    t.gate_norm = 2 * (n_layers - 1) + 1; t.tokens = T * s.batch; t.splits = pd.splits;
    return t;
  }

  void prologue() {
    if (e != cudaSuccess) return;
    TableArgs t;
    const double dt = -1.0 / NS;
    for (int i = 0; i < NS; ++i) t.t_steps[i] = (float)(1.0 + i * dt);
    t.temb = s.temb; t.rope = s.rope; t.rope4 = s.rope4; t.mask = (const uint8_t*)s.in[24]; t.state = s.state; t.prefix = s.prefix; t.n_steps = n_steps;
    e = launch_kernel(tables_kernel, dim3(std::max(8, s.sms / s.batch), s.batch), 256, 0, stream, 1, false, t);
    ++kernels;
    MatArgs m;
    memset(&m, 0, sizeof m);
    m.in = s.temb; m.w[0] = (const float*)s.in[2]; m.b[0] = (const float*)s.in[3]; m.out = s.hid;
    put(time_mlp_kernel, W / 8, 256, 0, 1, m);
    m.in = s.hid; m.w[0] = (const float*)s.in[4]; m.b[0] = (const float*)s.in[5]; m.out = s.cond;
    put(time_mlp_kernel, W / 8, 256, 0, 1, m);
    m.in = s.cond; m.out = s.mod;
    m.w[0] = (const float*)s.in[15]; m.b[0] = (const float*)s.in[16];
    m.w[1] = (const float*)s.in[17]; m.b[1] = (const float*)s.in[18];
    m.w[2] = (const float*)s.in[19]; m.b[2] = (const float*)s.in[20];
    put(modulation_kernel, s.sms, MOD_THREADS, MOD_SMEM, 1, m);
    put(tail_kernel<true>, std::min(T * s.batch, s.sms), TAIL_THREADS, TAIL_SMEM, 1, tail_args());
  }

  void project(const GemmPlan& g, const CUtensorMap& a, const CUtensorMap* b0, const CUtensorMap* b1, const CUtensorMap* b2,
               int width, int layer, bool early = true) {
    if (e != cudaSuccess) return;
    gemm::Args p;
    memset(&p, 0, sizeof p);
    p.a = a; p.b0 = *b0;
    if (b1) p.b1 = *b1;
    if (b2) p.b2 = *b2;
    p.tokens = T * s.batch; p.layer = layer; p.width = width; p.status = s.status; p.limit = s.wait_limit;
    p.q = s.q; p.k = s.k; p.v = s.v; p.rope = s.rope4; p.act = s.act; p.part = s.part;
    e = launch_gemm(g, p, stream, early);
    ++kernels;
  }

  void encode() {
    const uint64_t L = NL, M = T * s.batch;
    ap.merge = s.part;
    // full pages, and the last page of an observation cut at its last valid token; 128 keys are one copy where pages allow it
    const int tail = s.prefix - (s.prefix - 1) / s.page_tokens * s.page_tokens;
    ap.k_rows = s.pages_per_obs == 1 || s.page_tokens % attn::KCH == 0 ? attn::KCH : 64;
    auto keys = [&](CUtensorMap* m, int rows) {
      return map_kv(m, s.pool_k, rows, L, s.num_pages, s.token_stride, s.layer_stride, s.page_stride, ap.k_rows, ap.k_rows / 64);
    };
    auto values = [&](CUtensorMap* m, int rows) {
      return map_kv(m, s.pool_v, rows, L, s.num_pages, s.token_stride, s.layer_stride, s.page_stride, 64, 4);
    };
    auto weights = [&](CUtensorMap* m, int which, int k, int rows, const GemmPlan& g) { return map_k(m, s.in[which], k, L * rows, g.w_rows, g.w_kb); };
    if (join) {
      ap.m_rows = (s.prefix - (s.prefix - 1) / attn::KCH * attn::KCH + 7) / 8 * 8;
      ap.m_suf = 56 + (ap.m_rows % 16 == 0 ? 8 : 0);
    }
    auto joined = [&](CUtensorMap* m, const void* pool) { return !ap.m_rows || map_kv(m, pool, tail, L, s.num_pages, s.token_stride, s.layer_stride, s.page_stride, ap.m_rows, 1); };
    auto joined_suffix = [&](CUtensorMap* m, const void* kv) { return !ap.m_rows || map_kv(m, kv, T, 1, s.batch, HD, (uint64_t)T * HD, (uint64_t)T * HD, ap.m_suf, 1); };
    if (!(joined(&ap.jk, s.pool_k) && joined(&ap.jv, s.pool_v) && joined_suffix(&ap.jsk, s.k) && joined_suffix(&ap.jsv, s.v) &&
          map_k(&a_qkv, s.an, W, M, pq.arows, pq.ks) && map_k(&a_short, s.an, W, M, pq.arows - 8, pq.ks) &&
          map_k(&a_o, s.attn, QD, M, po.arows, po.ks) && map_k(&a_gu, s.an, W, M, pg.arows, pg.ks) &&
          map_k(&a_dn, s.act, FF, M, pd.arows, pd.ks) && weights(&wq, 8, W, QD, pq) && weights(&wk, 9, W, HD, pq) && weights(&wv, 10, W, HD, pq) &&
          weights(&wo, 11, QD, W, po) && weights(&wg, 12, W, FF, pg) && weights(&wu, 13, W, FF, pg) && weights(&wd, 14, FF, W, pd) &&
          map_k(&ap.q, s.q, HD, M * NQH, ap.tok_tile * NQH, HD / 64) &&
          keys(&ap.pk, s.page_tokens) &&
          keys(&ap.pk_tail, tail) && values(&ap.pv, s.page_tokens) && values(&ap.pv_tail, tail) &&
          map_kv(&ap.sk, s.k, T, 1, s.batch, HD, (uint64_t)T * HD, (uint64_t)T * HD, attn::KCH, 2) &&
          map_kv(&ap.sv, s.v, T, 1, s.batch, HD, (uint64_t)T * HD, (uint64_t)T * HD, 64, 4))) {
      e = cudaErrorUnknown;
      what = "cuTensorMapEncodeTiled failed";
      return;
    }
    ap.page_table = s.page_table; ap.pages_per_obs = s.pages_per_obs; ap.page_tokens = s.page_tokens;
    ap.valid = (const uint8_t*)s.in[24]; ap.out = s.attn; ap.prefix = s.prefix; ap.suffix = T; ap.obs_tokens = T;
    ap.early = 1; ap.status = s.status; ap.limit = s.wait_limit;
    if (fused) encode_fused(tail);
  }

  // Attention with the O projection: the prefix in its first page, or (pages of 64 tokens) in two.
  void encode_fused(int tail) {
    const uint64_t M = T * s.batch;
    const attno::Layout l = attno::layout(s.prefix);
    memset(&fp, 0, sizeof fp);
    const bool two = s.prefix > s.page_tokens;
    fp.rows0 = two ? s.page_tokens : l.rows - attno::SUF;
    fp.rows1 = l.rows - attno::SUF - fp.rows0;
    auto cache = [&](CUtensorMap* m, const void* pool, int tokens, int box) {
      return map_kv(m, pool, tokens, NL, s.num_pages, s.token_stride, s.layer_stride, s.page_stride, box, 1);
    };
    auto suffix = [&](CUtensorMap* m, const void* kv) { return map_kv(m, kv, T, 1, s.batch, HD, (uint64_t)T * HD, (uint64_t)T * HD, attno::SUF, 1); };
    if (!(map_k(&fp.q, s.q, QD, M, attno::QROWS, HD / 64) && cache(&fp.pk0, s.pool_k, two ? s.page_tokens : tail, fp.rows0) && cache(&fp.pv0, s.pool_v, two ? s.page_tokens : tail, fp.rows0) &&
          (!two || (cache(&fp.pk1, s.pool_k, tail, fp.rows1) && cache(&fp.pv1, s.pool_v, tail, fp.rows1))) && suffix(&fp.sk, s.k) && suffix(&fp.sv, s.v) &&
          map_k(&fp.wo, s.in[11], QD, (uint64_t)NL * W, attno::FEAT, HD / 64))) {
      e = cudaErrorUnknown;
      what = "cuTensorMapEncodeTiled failed";
      return;
    }
    fp.wo_base = (const __nv_bfloat16*)s.in[11];
    fp.page_table = s.page_table; fp.valid = (const uint8_t*)s.in[24]; fp.part = s.part;
    fp.pages_per_obs = s.pages_per_obs; fp.prefix = s.prefix; fp.tokens = T * s.batch;
    fp.off_v = l.off_v; fp.off_q = l.off_q; fp.off_wo = l.off_wo; fp.wo_early = l.wo_early; fused_smem = l.smem;
    fp.status = s.status; fp.limit = s.wait_limit;
  }

  void step() {
    const int tokens = T * s.batch;
    NormArgs n;
    n.part = s.part; n.h = s.h; n.out = s.an; n.mod = s.mod; n.state = s.state;
    for (int l = 0; l < n_layers && e == cudaSuccess; ++l) {
      // (withheld: copies of fewer bytes than their barrier is told to expect)
      project(pq, l == s.withhold ? a_short : a_qkv, &wq, &wk, &wv, 0, l, l > 0);      // (what a step leaves behind is complete before the next one's first kernel starts)
      if (fused) {
        fp.layer = l;
        if (e == cudaSuccess) { e = launch_attention_o(fp, s.batch, fused_smem, stream); ++kernels; }
      } else {
        ap.layer = l;
        if (e == cudaSuccess) { e = launch_attention(ap, s.batch, stream); ++kernels; }
        project(po, a_o, &wo, nullptr, nullptr, W, l);
      }
      n.gate_norm = 2 * l; n.next_norm = 2 * l + 1;
      put(norm_kernel_for(po.splits), tokens, 256, 0, 1, n);
      project(pg, a_gu, &wg, &wu, nullptr, FF, l);
      project(pd, a_dn, &wd, nullptr, nullptr, W, l);
      if (l + 1 < n_layers) {
        n.gate_norm = 2 * l + 1; n.next_norm = 2 * l + 2;
        put(norm_kernel_for(pd.splits), tokens, 256, 0, 1, n);
      }
    }
    put(tail_kernel<false>, std::min(tokens, s.sms), TAIL_THREADS, TAIL_SMEM, 1, tail_args());
  }

  // Captures what `body` launches into an executable graph.
  template <typename F>
  cudaGraphExec_t graph(F body) {
    if (e != cudaSuccess) return nullptr;
    cudaGraph_t g = nullptr;
    cudaGraphExec_t x = nullptr;
    kernels = 0;
    e = cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return nullptr;
    body();
    const cudaError_t end = cudaStreamEndCapture(stream, &g);
    if (e == cudaSuccess) e = end;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&x, g, 0);
    if (e == cudaSuccess) e = cudaGraphUpload(x, stream);
    if (g) cudaGraphDestroy(g);
    if (e != cudaSuccess && x) { cudaGraphExecDestroy(x); x = nullptr; }
    return x;
  }
};

}  // namespace

namespace {
size_t attention_floats(int batch, const AttnPlan& a) { return a.splits > 1 ? (size_t)batch * a.tiles * a.splits * attn::part_floats(a.tok_tile * NQH) : 0; }
}  // namespace

StepPlan steps_plan(int sms, int batch, int prefix, int page_tokens) {
  const AttnPlan a = plan_attention_for(sms, batch, prefix, page_tokens);
  const bool o = with_o(sms, batch, prefix);
  StepPlan p;
  p.tok_tile = o ? T : a.tok_tile; p.splits = o ? 1 : a.splits;
  p.with_o = o; p.join = !o && a.join;
  p.chunks = o ? 1 : ((prefix + attn::KCH - 1) / attn::KCH + (a.join ? 0 : 1) + a.splits - 1) / a.splits;
  p.o_splits = o ? NQH : plan_gemm(sms, T * batch, W, QD, gemm::EPI_PART).splits;
  p.down_splits = plan_gemm(sms, T * batch, W, FF, gemm::EPI_PART).splits;
  p.part_floats = std::max((size_t)std::max(p.o_splits, p.down_splits) * T * batch * W, o ? 0 : attention_floats(batch, a));
  return p;
}

std::string steps_describe(int sms, int batch, int prefix, int page_tokens, const StepGraphs& g) {
  const int tokens = T * batch;
  const AttnPlan a = plan_attention_for(sms, batch, prefix, page_tokens);
  const bool o = with_o(sms, batch, prefix);
  const struct { const char* name; GemmPlan plan; } all[] = {{"qkv", plan_gemm(sms, tokens, QKVW, W, gemm::EPI_QKV)},
                                                              {"o", plan_gemm(sms, tokens, W, QD, gemm::EPI_PART)},
                                                              {"gate_up", plan_gemm(sms, tokens, 2 * FF, W, gemm::EPI_GEGLU)},
                                                              {"down", plan_gemm(sms, tokens, W, FF, gemm::EPI_PART)}};
  char buf[256];
  snprintf(buf, sizeof buf, "{\"prologue_launches\": %d, \"launches_per_layer\": %d, \"attention\": {\"query_tokens\": %d, \"ctas_per_tile\": %d, \"ctas\": %d}",
           g.kernels_prologue, g.kernels_step / NL, o ? T : a.tok_tile, o ? 1 : a.splits, o ? batch * NQH * attno::GROUPS : batch * a.tiles * a.splits);
  std::string out = buf;
  for (const auto& x : all) {
    if (o && x.plan.epi == gemm::EPI_PART && x.plan.kblocks * x.plan.splits == QD / gemm::BK) {      // part of the attention
      snprintf(buf, sizeof buf, ", \"o\": {\"within\": \"attention\", \"features_per_cta\": %d, \"k_splits\": %d}", attno::FEAT, NQH);
      out += buf;
      continue;
    }
    snprintf(buf, sizeof buf, ", \"%s\": {\"tile_tokens\": %d, \"tile_features\": %d, \"cta_pairs\": %s, \"k_splits\": %d, \"ctas\": %d, \"stages\": %d}", x.name,
             x.plan.rows, x.plan.bn, x.plan.pair ? "true" : "false", x.plan.splits, x.plan.grid, x.plan.stages);
    out += buf;
  }
  return out + "}";
}

// Every number of chunks of every batch is asked: the longest prefix does not need the most (148 SMs, four observations: tiles of 8
// tokens over four CTAs at 968 tokens, of 4 over two at 1100).
size_t steps_part_floats(int sms, int max_batch, int max_prefix) {
  size_t most = 0;
  for (int b = 1; b <= max_batch; ++b) {
    const int splits = std::max(plan_gemm(sms, T * b, W, QD, gemm::EPI_PART).splits, plan_gemm(sms, T * b, W, FF, gemm::EPI_PART).splits);
    most = std::max(most, (size_t)std::max(splits, with_o(sms, b, 1) ? NQH : 0) * T * b * W);
    const AttnCuts cuts = attention_cuts(sms, b);
    for (int chunks = 1; chunks <= (max_prefix + attn::KCH - 1) / attn::KCH; ++chunks)
      for (int pages : {0, 64, attn::KCH})
        for (bool join : {false, true}) most = std::max(most, attention_floats(b, plan_attention(cuts, chunks, join, pages)));
  }
  return most;
}

namespace {
int failed(const Chain& c, const char* doing, std::string* error) {
  *error = doing + (": " + (c.what.empty() ? std::string(cudaGetErrorString(c.e)) : c.what));
  cudaGetLastError();
  return PI05_ERR_CUDA;
}
}  // namespace

int steps_build(const StepSetup& s, StepGraphs* g, std::string* error) {
  steps_free(g);
  if (steps_plan(s.sms, s.batch, s.prefix, s.page_tokens).part_floats > s.part_floats) {
    *error = "the workspace does not hold the partial sums of this binding";
    return PI05_ERR_UNSUPPORTED;
  }
  Chain c(s, NS, NL, nullptr);
  if (c.e == cudaSuccess) c.e = cudaStreamCreateWithFlags(&c.stream, cudaStreamNonBlocking);
  g->prologue = c.graph([&] { c.prologue(); });
  g->kernels_prologue = c.kernels;
  g->step = c.graph([&] { c.step(); });
  g->kernels_step = c.kernels;
  if (c.stream) {
    const cudaError_t done = cudaStreamSynchronize(c.stream);
    if (c.e == cudaSuccess) c.e = done;
    cudaStreamDestroy(c.stream);
  }
  if (c.e != cudaSuccess) {
    steps_free(g);
    return failed(c, "capture of the chunk's kernels", error);
  }
  g->wait_limit = s.wait_limit;
  return PI05_OK;
}

int steps_launch(const StepGraphs& g, const StepSetup& s, int n_steps, int n_layers, bool capturing, cudaStream_t stream, std::string* error) {
  // a graph cannot be launched into a stream that is being captured
  const bool graphs = g.step && !capturing && n_layers == NL && s.wait_limit == g.wait_limit && s.withhold < 0;
  if (graphs && n_steps == NS) {
    cudaError_t e = cudaGraphLaunch(g.prologue, stream);
    for (int i = 0; i < n_steps && e == cudaSuccess; ++i) e = cudaGraphLaunch(g.step, stream);
    if (e == cudaSuccess) return PI05_OK;
    *error = std::string("graph launch: ") + cudaGetErrorString(e);
    return PI05_ERR_CUDA;
  }
  Chain c(s, n_steps, n_layers, stream);
  c.prologue();
  for (int i = 0; i < n_steps && c.e == cudaSuccess; ++i) {
    if (graphs) c.e = cudaGraphLaunch(g.step, stream);
    else c.step();
  }
  return c.e == cudaSuccess ? PI05_OK : failed(c, "launch of the chunk's kernels", error);
}

void steps_free(StepGraphs* g) {
  if (g->prologue) cudaGraphExecDestroy(g->prologue);
  if (g->step) cudaGraphExecDestroy(g->step);
  *g = StepGraphs();
}

}  // namespace pi05
