// The projections of the action chunk and of the prefix prefill as tcgen05 GEMMs: out[tokens, N] = A[tokens, K] . W[N, K]^T with
// a fused epilogue.
//
// One CTA (or CTA pair, cta_group::2) works on output tiles of `rows` <= 128 tokens per CTA x BN features x a K range.  The
// kernels of a chunk (and of a short prefill) form one dependent chain of ~2-5 us each, so what matters is the time from the
// end of one to the first MMA of the next:
//   * weights do not depend on the chain, so a CTA fills its whole weight ring before it waits for the kernel before it
//     (programmatic dependent launch);
//   * a stage holds both operands of KS 64-k blocks behind one barrier, and its MMAs and the commit that frees it are one asm
//     block.  Weights and activations have a producer warp each, and a copy brings all KS blocks of an operand;
//   * what a stage takes is the way of its operands through shared memory (128 B per cycle: 4 KB of activations and 1-2 KB of
//     weights read per MMA, and the copies that write them): an MMA reads 128 rows of activations however few are valid.  A
//     tile of up to 64 rows is an MMA of 64: at 50 tokens a stage of 128 k x 64 features takes 0.27 us instead of 0.38, a layer
//     pass 28.3 us instead of 30.2;
//   * the tile's tokens are balanced (rows = ceil(tokens / tiles)) and only those rows are copied; the MMA still reads 64
//     or 128 rows, the ones beyond the tile are whatever shared memory holds and end in accumulator lanes nobody reads;
//   * K is split over several CTAs where whole-K tiles would leave SMs without work.  Every split stores its FP32 partial
//     sums to a slice of its own and a row kernel adds the slices (atomics made the end of the kernel ~1 us later; folding the
//     row kernel's normalisation into the projections around it and adding the splits within a cluster made a layer pass
//     slower, since the row kernel is what the weights of the next projection arrive under);
//   * results of all but the smallest tiles leave through shared memory, from where all epilogue threads store whole lines (a thread per row
//     stores 16 bytes to 32 different lines, which the LSU takes one at a time: 2 us at 128 features per thread; a bulk copy per row: 1.5 us;
//     tiled copies by one thread: 1.3 us for 115 rows of 128 FP32 sums, 30 B per cycle, against 0.5);
//   * SK ("stream-K"): tiles x 64-k blocks, taken as one sequence, are cut into one contiguous, equal range per CTA, so that a
//     long K with few tiles keeps every SM busy for the same time.  A range that begins inside a tile (a contributor's) leaves
//     its partial sums in the slot of its CTA, one that begins with a tile (the owner's) in the slot of the tile; the residual
//     kernel adds them.  Nobody waits for anybody;
//   * with more tiles than CTAs the launch is persistent with two accumulators, so that a tile's epilogue runs under the
//     next tile's MMAs.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "pi05_common.cuh"
#include "ptx_sm100.cuh"

namespace gemm {
using namespace pi05;

// Warp 0 weight producer, warp 1 MMA issuer, the next eight epilogue (two per TMEM lane quadrant; four of them are no faster), the last one activation
// producer.
constexpr int EPI_THREADS = 256, THREADS_G = 96 + EPI_THREADS, WARP_A = THREADS_G / 32 - 1;
constexpr int BK = 64;             // k per stage (one 128-byte swizzle row)
constexpr int MAX_STAGES = 16;

enum { EPI_QKV = 0, EPI_GEGLU = 1, EPI_PART = 2 };
struct Args {
  CUtensorMap a;                   // activations as {64 k, rows, K / 64}, box {64, arows, KS}
  CUtensorMap b0, b1, b2;          // weights likewise, box {64, rows of a load, 64-k blocks of a load}.  QKV: wq, wk, wv; GEGLU: gate, up
  int tokens, rows, arows, m_groups, splits, kblocks, units, layer, stages, bufs, off_out;   // kblocks: 64-k blocks per unit
  int width;                       // GEGLU: MLP width; PART: features of the output (rows of a layer's weights)
  int unit0;                       // first unit of the launch (QKV of a last layer: keys and values only)
  unsigned int* status;
  long long limit;
  __nv_bfloat16 *q, *k, *v;        // EPI_QKV: [tokens, 2048], [tokens, 256], [tokens, 256]
  const uint32_t* rope;            // [128 / 4][tokens][4]: cos BF16 | sin BF16 << 16 (rope_at)
  __nv_bfloat16* act;              // EPI_GEGLU: [tokens, width]
  float* part;                     // EPI_PART: [splits][tokens, width]; SK: [slots][128][BN]
};

// Word of the rotary table: four dims of a token together, tokens next to each other, so that the 32 tokens of an epilogue warp read whole lines.
// With a token's 128 words in a row, a warp's load touched 32 lines, which the load unit takes one at a time: 2 us of a QKV epilogue of 128 features.
__host__ __device__ __forceinline__ size_t rope_at(int tokens, int token, int dim) { return ((size_t)(dim >> 2) * tokens + token) * 4 + (dim & 3); }

__device__ __forceinline__ float rb(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float lo16(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi16(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// 0.5 x (1 + tanh z) = x / (1 + exp(-2 z)) with z = 0.79788 (x + 0.044715 x^3): one exponential and one reciprocal, no
// cancellation for negative x.  The constants carry the factor -2 log2 e.
__device__ __forceinline__ float gelu_tanh(float x) {
  const float e = ptx::ex2_approx(x * fmaf(x * x, -0.10294324f, -2.3022082f));
  return x * ptx::rcp_approx(1.0f + e);
}

// Staging of a tile's results: boxes of 128 rows x BOX bytes (swizzled, so that neither its writers nor its readers meet in a bank), COUNT of them; 0: the
// tile is small and its rows are stored directly.  PART: 32 FP32 columns a box; GEGLU and QKV: 64 BF16 (QKV of 64
// features: 32, each half of the tile a box; GEGLU of 224: 16, which 112 results are a multiple of; GEGLU of 112 is stored directly, 56 results a row, like the 64 of
// which it is a wider form: staged it was not tried).
template <int EPI, int BN>
struct Staging {
  static constexpr int COUNT = EPI == EPI_PART ? (BN >= 64 ? BN / 32 : 0) : EPI == EPI_GEGLU ? (BN == 224 ? 7 : BN == 112 ? 0 : BN / 128) : (BN == 256 ? 4 : BN >= 64 ? 2 : 0);
  static constexpr int BOX = EPI == EPI_QKV && BN == 64 ? 64 : EPI == EPI_GEGLU && BN == 224 ? 32 : 128;
  static constexpr int BYTES = COUNT * 128 * BOX;
  // 16-byte piece `c` (counted over the whole row of BN results) of row `row`
  static __device__ __forceinline__ uint32_t at(int row, int c) {
    constexpr int PER = BOX / 16;
    const uint32_t sw = BOX == 128 ? (row & 7) : BOX == 64 ? ((row >> 1) & 3) : ((row >> 2) & 1);
    return (uint32_t)(c / PER) * (128 * BOX) + row * BOX + (((c % PER) ^ sw) << 4);
  }
};

// This thread's token row of the accumulator (TMEM lanes of its warp, BN columns from t0); `part` of PARTS is the share of the columns
// (of each half of the tile for QKV and GEGLU) that its warp handles.  `out` is the staging buffer; PART fills `boxes` boxes of
// it from column 32 box0 on.
// Eight columns at a time in loops that stay loops: an instruction that runs once costs several cycles to fetch.
template <int EPI, int BN>
__device__ __forceinline__ void epilogue_row(const Args& p, uint32_t t0, int nt, int split, int row, int token, bool live, bool mine, int part, uint32_t out,
                                             int box0, int boxes) {
  using St = Staging<EPI, BN>;
  constexpr bool STAGED = St::COUNT > 0;
  constexpr int PARTS = EPI_THREADS / 128;
  constexpr bool EVEN = BN / 2 / PARTS % 8 == 0;            // else the warps take eight columns in turn
  constexpr int FIRST = EVEN ? BN / 2 / PARTS : 8;
  const int tok = live ? token : 0;
  if constexpr (EPI == EPI_PART) {
    const int cols = (STAGED ? boxes * 32 : BN) / PARTS, c0 = (STAGED ? box0 * 32 : 0) + part * cols;
    uint4* g = reinterpret_cast<uint4*>(p.part + ((size_t)split * p.tokens + tok) * p.width + nt * BN + c0);
#pragma unroll 1
    for (int c = 0; c < cols; c += 16) {
      uint32_t r[16];
      ptx::tmem_ld_32x16(t0 + c0 + c, r);
      ptx::tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (STAGED) { if (mine) ptx::st_shared_v4(out + St::at(row, (part * cols + c) / 4 + j), r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]); }
        else if (live) g[c / 4 + j] = make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
    }
  } else {
    // QKV and GEGLU need columns c and c + BN / 2 of the tile together (rotary partner, gate with up)
    constexpr int PER = HD / BN;                            // QKV: tiles per head
    const int head = nt / PER, dim0 = (nt % PER) * (BN / 2);
    const uint4* cs4 = reinterpret_cast<const uint4*>(p.rope) + (size_t)(dim0 / 4) * p.tokens + tok;
    __nv_bfloat16* g = EPI == EPI_GEGLU ? p.act + (size_t)tok * p.width + nt * (BN / 2)
                       : (head < NQH ? p.q + (size_t)tok * QD + head * HD : (head == NQH ? p.k : p.v) + (size_t)tok * HD) + dim0;
#pragma unroll 1
    for (int c = part * FIRST; c < (EVEN ? (part + 1) * FIRST : BN / 2); c += EVEN ? 8 : 8 * PARTS) {
      uint32_t r1[8], r2[8], o1[4], o2[4];
      ptx::tmem_ld_32x8(t0 + c, r1);
      ptx::tmem_ld_32x8(t0 + BN / 2 + c, r2);
      uint4 wa, wb;
      if (EPI == EPI_QKV) { wa = __ldg(cs4 + (c / 4) * p.tokens); wb = __ldg(cs4 + (c / 4 + 1) * p.tokens); }
      ptx::tmem_wait_ld();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t x = pack2(__uint_as_float(r1[2 * j]), __uint_as_float(r1[2 * j + 1]));
        const uint32_t y = pack2(__uint_as_float(r2[2 * j]), __uint_as_float(r2[2 * j + 1]));
        if (EPI == EPI_GEGLU) {
          const uint32_t z = pack2(gelu_tanh(lo16(x)), gelu_tanh(hi16(x)));
          // (a product of two BF16 is exact in FP32: one rounding either way)
          const __nv_bfloat162 a = __hmul2_rn(*reinterpret_cast<const __nv_bfloat162*>(&z), *reinterpret_cast<const __nv_bfloat162*>(&y));
          o1[j] = *reinterpret_cast<const uint32_t*>(&a);
        } else {
          // RoPE (reference/pi05.py:218-229 on BF16 tensors): x cos + rotate_half(x) sin, every product and the sum rounded
          // to BF16; dim d pairs with dim d + 128.  A table word holds cos | sin << 16 of one dim.
          const uint32_t w0 = j == 0 ? wa.x : j == 1 ? wa.z : j == 2 ? wb.x : wb.z, w1 = j == 0 ? wa.y : j == 1 ? wa.w : j == 2 ? wb.y : wb.w;
          const uint32_t cw = __byte_perm(w0, w1, 0x5410), sw = __byte_perm(w0, w1, 0x7632);
          const __nv_bfloat162 co = *reinterpret_cast<const __nv_bfloat162*>(&cw), si = *reinterpret_cast<const __nv_bfloat162*>(&sw);
          const __nv_bfloat162 xv = *reinterpret_cast<const __nv_bfloat162*>(&x), yv = *reinterpret_cast<const __nv_bfloat162*>(&y);
          const __nv_bfloat162 a = __hadd2_rn(__hmul2_rn(xv, co), __hmul2_rn(__hneg2(yv), si));
          const __nv_bfloat162 b = __hadd2_rn(__hmul2_rn(yv, co), __hmul2_rn(xv, si));
          o1[j] = head <= NQH ? *reinterpret_cast<const uint32_t*>(&a) : x;
          o2[j] = head <= NQH ? *reinterpret_cast<const uint32_t*>(&b) : y;
        }
      }
      if (STAGED) { if (mine) ptx::st_shared_v4(out + St::at(row, c / 8), o1[0], o1[1], o1[2], o1[3]); }
      else if (live && (BN != 112 || nt * (BN / 2) + c < p.width)) *reinterpret_cast<uint4*>(g + c) = make_uint4(o1[0], o1[1], o1[2], o1[3]);
      if (EPI == EPI_QKV) {
        if (STAGED) { if (mine) ptx::st_shared_v4(out + St::at(row, (BN / 2 + c) / 8), o2[0], o2[1], o2[2], o2[3]); }
        else if (live) *reinterpret_cast<uint4*>(g + 128 + c) = make_uint4(o2[0], o2[1], o2[2], o2[3]);
      }
    }
  }
}

// The staged tile (PART: boxes box0 .. box0 + boxes - 1 of it) to its place in memory: 16 bytes per thread, whole lines per warp.
// (Tiled copies, a thread issuing one per box, moved 30 B per cycle: 1.3 us for 115 rows of 128 FP32 sums.)
template <int EPI, int BN, bool SK>
__device__ __forceinline__ void copy_out(const Args& p, uint32_t stage, int nt, int split, int token0, int box0, int tid) {
  using St = Staging<EPI, BN>;
  constexpr int PER = EPI == EPI_PART ? (SK ? 16 : BN / 4) : EPI == EPI_GEGLU ? BN / 16 : BN / 8;      // 16-byte pieces of a row
  const int left = p.tokens - token0, rows = left < p.rows ? left : p.rows;
  uint4* g;
  int pitch, jump = 0;                                      // of a row; QKV: from the first half of the pieces to the second
  if constexpr (EPI == EPI_PART) {
    pitch = (SK ? BN : p.width) / 4;
    g = reinterpret_cast<uint4*>(p.part) + (SK ? (size_t)split * 128 * pitch : ((size_t)split * p.tokens + token0) * pitch + nt * (BN / 4)) + box0 * 8;
  } else if constexpr (EPI == EPI_GEGLU) {
    pitch = p.width / 8;
    g = reinterpret_cast<uint4*>(p.act) + (size_t)token0 * pitch + nt * (BN / 16);
  } else {
    constexpr int HEAD = HD / BN;
    const int head = nt / HEAD;
    pitch = (head < NQH ? QD : HD) / 8;
    g = reinterpret_cast<uint4*>(head < NQH ? p.q + head * HD : head == NQH ? p.k : p.v) + (size_t)token0 * pitch + (nt % HEAD) * (BN / 16);
    jump = 128 / 8 - PER / 2;
  }
  constexpr int UNROLL = BN >= 128 ? 4 : 2;
#pragma unroll UNROLL
  for (int i = tid; i < rows * PER; i += EPI_THREADS) {
    const int row = i / PER, c = i % PER;
    if (EPI == EPI_GEGLU && BN == 224 && nt * 14 + c >= pitch) continue;      // (the last tile of a width that 112 does not divide)
    g[(size_t)row * pitch + c + (EPI == EPI_QKV && c >= PER / 2 ? jump : 0)] = ptx::ld_shared_v4(stage + St::at(row, c));
  }
}

// The contiguous ranges of (tile, 64-k block) units of a stream-K launch, in which a tile's blocks are neighbours.
struct Segments {
  __host__ __device__ static long long begin(int tiles, int kblocks, int cta, int ctas) { return (long long)tiles * kblocks * cta / ctas; }
};

// KS: 64-k blocks per stage.
template <int EPI, int BN, bool PAIR, int KS, bool SK>
__global__ void __launch_bounds__(THREADS_G) gemm_kernel(const __grid_constant__ Args p) {
  static_assert(!SK || (EPI == EPI_PART && BN == 256 && !PAIR && KS == 1), "stream-K: partial sums of 128 x 256 tiles");
  constexpr int WR = PAIR ? BN / 2 : BN;                  // weight rows this CTA loads per 64-k block
  constexpr bool TWO = !PAIR && (EPI == EPI_QKV || EPI == EPI_GEGLU);      // .. from two places, block by block
  constexpr int W_BYTES = WR * 128, HALF = (BN / 2) * 128, OUT = Staging<EPI, BN>::BYTES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  __shared__ uint64_t bars[2 * MAX_STAGES + 4];
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t rank = PAIR ? ptx::cluster_ctarank() : 0u;                // pair: the even CTA issues
  const int per_unit = PAIR ? 2 : 1;
  const int ustep = (int)gridDim.x / per_unit, unit0 = p.unit0 + (int)blockIdx.x / per_unit;
  // a stage: KS activation blocks, then KS weight blocks
  const uint32_t a_stride = (uint32_t)p.arows * 128, w_off = KS * a_stride, st_stride = w_off + KS * W_BYTES, ring = ptx::smem_u32(smem);
  const uint32_t full = ptx::smem_u32(bars), empty = full + 8 * MAX_STAGES, t_full = empty + 8 * MAX_STAGES, t_empty = t_full + 16;
  const bool leader = ptx::elect_one();
  const int stages = p.stages;
  const int tcols = p.bufs * (BN < 32 ? 32 : BN > 128 ? 256 : BN > 64 ? 128 : BN);      // a power of two

  if (warp == 0) {
    // a stage is full when both producers' arrivals (weights, activations) and every byte of both have come; a lane per stage, since
    // a CTA that starts when the kernel before it leaves pays for every cycle up to here
    if (lane < stages) { ptx::mbar_init(full + 8 * lane, 2); ptx::mbar_init(empty + 8 * lane, 1); }
    if (lane < 2) { ptx::mbar_init(t_full + 8 * lane, 1); ptx::mbar_init(t_empty + 8 * lane, OUT == 0 ? EPI_THREADS : (PAIR ? 2 : 1) * EPI_THREADS / 32); }
    ptx::fence_mbar_init();
    ptx::fence_proxy_async_shared();
  }
  __syncwarp();
  if (PAIR) ptx::cluster_sync();           // every CTA's barriers exist before another's copies count on them

  // The CTA's work, unit after unit: tile (mt, nt), slice of the partial sums, first stage and number of stages of its K range.
  // Regular: groups of tokens fastest (neighbours share weights), then K split, then features.
  struct Work { int mt, nt, split, st0, nst; };
  auto first = [&]() -> long long { return SK ? Segments::begin(p.units, p.kblocks, blockIdx.x, gridDim.x) : unit0; };
  const long long last = SK ? Segments::begin(p.units, p.kblocks, blockIdx.x + 1, gridDim.x) : p.unit0 + p.units;
  auto take = [&](long long& at, Work& w) -> bool {
    if (at >= last) return false;
    if (SK) {
      const int tile = (int)(at / p.kblocks);
      w.st0 = (int)(at - (long long)tile * p.kblocks);
      w.nst = (int)(last - at < p.kblocks - w.st0 ? last - at : p.kblocks - w.st0);
      w.nt = tile / p.m_groups;
      w.mt = tile - w.nt * p.m_groups;
      w.split = w.st0 ? (int)blockIdx.x : (int)gridDim.x + tile;      // slot of the partial sums
      at += w.nst;
    } else {
      const int unit = (int)at;
      const int rest = unit / p.m_groups, mg = unit - rest * p.m_groups;
      w.nt = rest / p.splits;
      w.split = rest - w.nt * p.splits;
      w.mt = PAIR ? 2 * mg + (int)rank : mg;
      w.nst = p.kblocks / KS;
      w.st0 = w.split * w.nst;
      at += ustep;
    }
    return true;
  };
  if (warp == 0) {
    // ---- weight producer: does not wait for the kernel before this one, nor does anybody wait for it but the MMAs
    ptx::bar_arrive(6, THREADS_G);
    const uint32_t bytes = (PAIR ? 2 : 1) * KS * W_BYTES;
    uint32_t slot = 0, par = 1;
    bool ok = true;
    long long at = first();
    Work w;
    while (ok && take(at, w)) {
      const CUtensorMap *m0 = &p.b0, *m1 = &p.b0;
      int r0, r1;
      if (EPI == EPI_QKV) {                // tile = BN / 2 dims of a head and their rotary partners
        constexpr int PER = HD / BN;
        const int head = w.nt / PER, d0 = (w.nt % PER) * (BN / 2);
        m0 = m1 = head < NQH ? &p.b0 : head == NQH ? &p.b1 : &p.b2;
        r0 = head < NQH ? p.layer * QD + head * HD + d0 : p.layer * HD + d0;
        r1 = r0 + 128;
      } else if (EPI == EPI_GEGLU) {
        m1 = &p.b1;
        r0 = r1 = p.layer * p.width + w.nt * (BN / 2);
      } else {
        r0 = p.layer * p.width + w.nt * BN;
        r1 = r0 + BN / 2;
      }
      if (PAIR && rank) { m0 = m1; r0 = r1; }
      for (int i = 0; i < w.nst; ++i) {
        const int kb = (w.st0 + i) * KS;
        if (!(ok = ptx::wait_bar(p.status, p.limit, empty + 8 * slot, par, WAIT_W_EMPTY))) break;
        if (leader) {
          const uint32_t dst = ring + slot * st_stride + w_off;
          if (rank == 0) ptx::mbar_expect_tx(full + 8 * slot, bytes);
          if (PAIR) {
            ptx::tma_load_3d_pair(dst, m0, ptx::map_to_rank(full + 8 * slot, 0), 0, r0, kb);
          } else if (TWO) {
#pragma unroll
            for (int h = 0; h < KS; ++h) {
              ptx::tma_load_3d(dst + h * W_BYTES, m0, full + 8 * slot, 0, r0, kb + h);
              ptx::tma_load_3d(dst + h * W_BYTES + HALF, m1, full + 8 * slot, 0, r1, kb + h);
            }
          } else {
            ptx::tma_load_3d(dst, m0, full + 8 * slot, 0, r0, kb);
          }
        }
        if (++slot == (uint32_t)stages) { slot = 0; par ^= 1; }
      }
    }
  } else {
    if (warp == 1) {
      if (PAIR) { ptx::tmem_alloc_pair(ptx::smem_u32(&s_tmem), tcols); ptx::tmem_relinquish_pair(); }
      else { ptx::tmem_alloc(ptx::smem_u32(&s_tmem), tcols); ptx::tmem_relinquish(); }
      ptx::grid_dep_launch();              // after the allocation: a later kernel cannot take the columns first
    } else if (warp == WARP_A && leader) {
      ptx::prefetch_tensormap(&p.a);
    }
    ptx::tc_fence_before();
    ptx::named_bar_sync(6, THREADS_G);     // the barriers are initialised, the tensor memory is allocated
    ptx::tc_fence_after();
  }
  const uint32_t tmem = s_tmem;

  if (warp == WARP_A) {
    // ---- activation producer.  It waits for the kernel before this one right before its first copy, when everything that copy takes is computed
    bool waited = false;
    const uint32_t bytes = (PAIR ? 2 : 1) * KS * a_stride;
    uint32_t slot = 0, par = 1;
    bool ok = true;
    long long at = first();
    Work w;
    while (ok && take(at, w))
      for (int i = 0; i < w.nst; ++i) {
        if (!(ok = ptx::wait_bar(p.status, p.limit, empty + 8 * slot, par, WAIT_A_EMPTY))) break;
        if (leader) {
          const uint32_t dst = ring + slot * st_stride;
          if (rank == 0) ptx::mbar_expect_tx(full + 8 * slot, bytes);
          if (!waited) ptx::grid_dep_wait();
          if (PAIR) ptx::tma_load_3d_pair(dst, &p.a, ptx::map_to_rank(full + 8 * slot, 0), 0, w.mt * p.rows, (w.st0 + i) * KS);
          else ptx::tma_load_3d(dst, &p.a, full + 8 * slot, 0, w.mt * p.rows, (w.st0 + i) * KS);
        }
        waited = true;
        if (++slot == (uint32_t)stages) { slot = 0; par ^= 1; }
      }
  } else if (warp == 1) {
    // ---- MMA issuer (of a pair: the even CTA only)
    if (rank == 0) {
      const uint32_t idesc = ptx::umma_idesc_bf16(PAIR ? 256 : p.rows <= 64 ? 64 : 128, BN);
      const uint32_t adesc0 = (uint32_t)ptx::umma_smem_desc(ring), bdesc0 = (uint32_t)ptx::umma_smem_desc(ring + w_off);
      uint32_t slot = 0, par = 0, it = 0, off = 0;
      bool ok = true;
      long long at = first();
      Work w;
      for (; ok && take(at, w); ++it) {
        const uint32_t buf = it & 1;
        if (!(ok = ptx::wait_bar(p.status, p.limit, t_empty + 8 * buf, ((it >> 1) & 1) ^ 1, WAIT_T_EMPTY))) break;
        ptx::tc_fence_after();
        const uint32_t d = tmem + buf * BN;
        uint32_t acc = 0;
#pragma unroll 1
        for (int i = 0; i < w.nst; ++i) {
          if (!(ok = ptx::wait_bar(p.status, p.limit, full + 8 * slot, par, WAIT_W_FULL))) break;
          const uint32_t cur = off, bar = empty + 8 * slot;
          off += st_stride >> 4;
          if (++slot == (uint32_t)stages) { slot = 0; par ^= 1; off = 0; }
          ptx::umma_bf16_stage<PAIR, KS>(d, adesc0 + cur, bdesc0 + cur, idesc, acc, bar, a_stride >> 4, W_BYTES >> 4, leader ? 1u : 0u);
          acc = 1;
        }
        if (ok && leader) {
          if (PAIR) ptx::umma_commit_pair(t_full + 8 * buf, 3);
          else ptx::umma_commit(t_full + 8 * buf);
        }
      }
    }
  } else if (warp >= 2) {
    // ---- epilogue: warp w reads TMEM lanes 32 (w % 4) ..; thread = token row of the tile, a share of its columns.  A wait that
    // gives up does not end the loop: the other epilogue warps count on this one at their barriers
    // (a tile of up to 64 rows is an MMA of 64, whose rows lie in the first 16 lanes of every warp)
    const bool m64 = !PAIR && p.rows <= 64;
    const int quad = warp & 3, qrow = m64 ? quad * 16 : quad * 32, row = qrow + lane, part = (warp - 2) >> 2;
    const uint32_t release = PAIR ? ptx::map_to_rank(t_empty, 0) : 0u;
    uint32_t it = 0;
    bool ok = true;
    long long at = first();
    Work w;
    const uint32_t stage = ptx::smem_u32(smem) + p.off_out;
    constexpr int BOXES = SK ? 2 : Staging<EPI, BN>::COUNT;          // boxes staged at a time
    for (; take(at, w); ++it) {
      const uint32_t buf = it & 1;
      const int token = w.mt * p.rows + row;
      if (EPI == EPI_QKV && BN >= 64) {    // the rotary words of this tile into L1 while the MMAs run: from L2 they cost a round trip per eight columns
        ptx::grid_dep_wait();
        constexpr int PARTS = EPI_THREADS / 128;
        const uint4* cs4 = reinterpret_cast<const uint4*>(p.rope) + (size_t)(w.nt % (HD / BN) * (BN / 8) + part * (BN / 8 / PARTS)) * p.tokens;
        if (row < p.rows && token < p.tokens)
#pragma unroll 4
          for (int c = 0; c < BN / 8 / PARTS; ++c) ptx::touch(cs4 + (size_t)c * p.tokens + token);
        __syncwarp();
      }
      ok &= ptx::wait_bar(p.status, p.limit, t_full + 8 * buf, (it >> 1) & 1, WAIT_T_FULL);
      ptx::tc_fence_after();
      const uint32_t t0 = tmem + buf * BN + ((uint32_t)(quad * 32) << 16);
#pragma unroll 1
      for (int box0 = 0; box0 < (SK ? Staging<EPI, BN>::COUNT : 1); box0 += SK ? BOXES : 1) {
        if (OUT > 0 && (it > 0 || box0 > 0)) ptx::named_bar_sync(1, EPI_THREADS);     // what was staged before has left the buffer
        if (qrow < p.rows)
          epilogue_row<EPI, BN>(p, t0, w.nt, w.split, row, token, ok && row < p.rows && token < p.tokens && (!m64 || lane < 16), !m64 || lane < 16, part, stage, box0, BOXES);
        if (!SK || box0 + BOXES >= Staging<EPI, BN>::COUNT) {   // the accumulator has been read
          ptx::tc_fence_before();
          if constexpr (OUT == 0) {
            ptx::mbar_arrive(t_empty + 8 * buf);
          } else {                         // by warps, since the stores are still to come: 256 arrivals on a barrier go one after the other
            __syncwarp();
            if (lane == 0) {
              if (PAIR) ptx::mbar_arrive_cluster(release + 8 * buf);
              else ptx::mbar_arrive(t_empty + 8 * buf);
            }
          }
        }
        if constexpr (OUT > 0) {
          ptx::named_bar_sync(1, EPI_THREADS);
          if (ok) copy_out<EPI, BN, SK>(p, stage, w.nt, w.split, w.mt * p.rows, box0, tid - 64);
        }
      }
    }
  }
  __syncthreads();
  if (PAIR) ptx::cluster_sync();           // neither CTA leaves (or frees tensor memory) while the other may still use what is in it
  if (warp == 1) {
    ptx::tc_fence_after();
    if (PAIR) ptx::tmem_dealloc_pair(tmem, tcols);
    else ptx::tmem_dealloc(tmem, tcols);
  }
}

}  // namespace gemm
