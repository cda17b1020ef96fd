// Attention on the tcgen05 tensor cores, used by the action chunk (50 suffix tokens over a prefix cache) and by the prefix
// prefill (every token over every token): several query tokens x 8 heads share the one KV head, so a tile of up to 128 query
// rows is one MMA operand.
//
//   * One CTA = one tile of `tok_tile` query tokens against a contiguous share of the keys, in chunks of 64.  A cluster of
//     `splits` CTAs shares the keys of a tile and merges through distributed shared memory (below).
//   * Warp 0 streams Q, the key chunks and the value chunks with TMA (the 256 dims of a token as four 64-dim segments of
//     128-byte swizzled rows); warp 1 issues S = Q K^T of chunk i + 1 before O += P V of chunk i; warps 2..9 are the
//     softmax threads, two per query row, each with half of the chunk's keys and half of the output's dims.  V is the
//     K-dimension operand as it lies in memory (rows = keys): the MMA takes it as an MN-major B operand, so nothing is
//     ever transposed.
//   * The keys are passed over once.  The exponent's reference is the maximum of the first chunk; the accumulator is only
//     rescaled when a later chunk exceeds it by more than RESCALE (nats), so that almost no chunk pays for it.  Numerator
//     and denominator always use the same reference, hence the result does not depend on when it moves.
//   * Scores are rounded to BF16 before the scale 1 / 16, and probabilities before P V, as the reference's BF16 matmuls
//     round (reference/pi05.py:184-188, 254-265).
//   * The key and value chunks of the cached prefix do not depend on the kernel before this one: with `early` the first
//     ones are requested before the grid dependency is waited for.
//   * Shared memory is cut by the tile's rows (only those of Q and P are stored; the MMAs read 128 rows, the ones beyond are
//     whatever follows and end in accumulator lanes nobody reads): small tiles leave room for three key / value stages, all
//     that a CTA of a short or well split prefix ever needs, so that nothing of it waits for a stage to be freed.
//   * Merge of a cluster: each CTA stores its accumulator and (max, sum) per row to global memory, column by column so that a
//     warp's 32 rows are one line; after a cluster barrier every rank adds its 256 / splits columns of all `splits` parts,
//     each scaled by exp(m - M) / L.  (The same exchange through distributed shared memory ran at 8-14 B/clk per SM in
//     either direction and took 6-7 us.)
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "ptx_sm100.cuh"

namespace attn {

constexpr int HD = 256, NQH = 8, KCH = 64, THREADS = 320;
constexpr int K_BYTES = KCH * HD * 2;                         // four 64-dim segments of [64 keys x 128 B]
constexpr int MAX_STG = 3;                                    // key / value stages
constexpr int MERGE_COLS = HD + 2;                            // FP32 columns of a part: the accumulator, maximum, sum
constexpr int SMEM_LIMIT = 226 * 1024;                        // dynamic shared memory without the alignment slack
constexpr int TM_O = 0, TM_S = 256, TM_COLS = 512;            // TMEM columns: O [128 x 256], two S buffers [128 x 64]
constexpr int MASK_WORDS = 130;                               // validity bits of up to 4096 prefix tokens + the suffix
constexpr float RESCALE = 5.0f;
// Shared memory of a tile of `rows` query rows: Q as four 64-dim blocks [rows x 128 B], two P buffers [rows x 64 keys], then
// the key and the value stages.
__host__ __device__ constexpr int stages_for(int rows) {
  return (SMEM_LIMIT - 4 * rows * 128 - 2 * rows * 128) / (2 * K_BYTES) < MAX_STG ? (SMEM_LIMIT - 6 * rows * 128) / (2 * K_BYTES) : MAX_STG;
}
__host__ __device__ constexpr int smem_for(int rows) { return 6 * rows * 128 + 2 * stages_for(rows) * K_BYTES + 1024; }
static_assert(stages_for(128) == 2 && smem_for(128) + 2048 <= 227 * 1024 && stages_for(40) == 3, "attention shared memory");
struct Args {
  CUtensorMap q;                           // [tokens x 8 rows, 256 dims], box {64, 8 x tok_tile}
  CUtensorMap pk, pk_tail, pv, pv_tail;    // prefix keys / values {64 dims, page tokens, 4, layers, pages}, box {64, 64, 4, 1, 1}
  CUtensorMap o;                           // the output as [observations][rows per observation][256], box {64, rows, 1}
  CUtensorMap sk, sv;                      // suffix keys / values {64, tokens, 4, observations}, box {64, 64, 4, 1}
  const int* page_table;                   // [observation][pages_per_obs], or null: page = observation
  const uint8_t* valid;                    // [observation][prefix]
  __nv_bfloat16* out;                      // [tokens, 2048]
  float* merge;                            // splits > 1: [tile][split][MERGE_COLS][rows]
  int pages_per_obs, page_tokens, prefix, suffix;      // suffix: keys behind the prefix (0: none)
  int obs_tokens, tok_tile, tiles, splits, layer, early, stages;
  unsigned int* status;
  long long limit;
};

__device__ __forceinline__ float rb(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float lo16(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi16(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

template <int = 0>   // a template, so that only the file that launches it holds its code
__global__ void __launch_bounds__(THREADS, 1) attention_kernel(const __grid_constant__ Args p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // barriers: q, k_full[3], k_empty[3], v_full[3], v_empty[3], s_full[2], s_empty[2], p_full[2], p_empty[2], o_full
  __shared__ uint64_t bars[22];
  __shared__ uint32_t s_tmem;
  __shared__ uint32_t s_mask[MASK_WORDS];
  // one value per row exchanged between threads: maxima [chunk parity][half][row] (BF16) during the loop, then sums
  // [half][row]
  __shared__ __align__(8) uint8_t s_row[128 * 8];
  __nv_bfloat16 (*s_max)[2][128] = reinterpret_cast<__nv_bfloat16 (*)[2][128]>(s_row);
  float (*s_sum)[128] = reinterpret_cast<float (*)[128]>(s_row);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = blockIdx.x % p.splits, unit = blockIdx.x / p.splits;
  const int ob = unit / p.tiles, tile = unit % p.tiles;
  const int npc = (p.prefix + KCH - 1) / KCH, total = npc + (p.suffix > 0 ? 1 : 0);
  const int cbeg = total * split / p.splits, n = total * (split + 1) / p.splits - cbeg;    // n >= 1: splits <= total
  const int rows = p.tok_tile * NQH;
  const uint32_t b0 = ptx::smem_u32(bars);
  const uint32_t q_full = b0, k_full = b0 + 8, k_empty = b0 + 32, v_full = b0 + 56, v_empty = b0 + 80;
  const uint32_t s_full = b0 + 104, s_empty = b0 + 120, p_full = b0 + 136, p_empty = b0 + 152, o_full = b0 + 168;
  const uint32_t q_base = ptx::smem_u32(smem), blk = rows * 128;            // one 64-dim block of Q, one P buffer
  const int stg = p.stages, off_k = 6 * rows * 128;
  const uint32_t p_base = q_base + 4 * blk, k_base = q_base + off_k, v_base = k_base + stg * K_BYTES;
  const bool leader = ptx::elect_one();

  if (tid == 0) {
    ptx::mbar_init(q_full, 1);
    for (int i = 0; i < stg; ++i) {
      ptx::mbar_init(k_full + 8 * i, 1); ptx::mbar_init(k_empty + 8 * i, 1);
      ptx::mbar_init(v_full + 8 * i, 1); ptx::mbar_init(v_empty + 8 * i, 1);
    }
    for (int i = 0; i < 2; ++i) {
      ptx::mbar_init(s_full + 8 * i, 1); ptx::mbar_init(s_empty + 8 * i, 256);
      ptx::mbar_init(p_full + 8 * i, 256); ptx::mbar_init(p_empty + 8 * i, 1);
    }
    ptx::mbar_init(o_full, 1);
    ptx::fence_mbar_init();
    ptx::fence_proxy_async_shared();
  }
  __syncwarp();
  // one chunk of keys (isv = 0) or values (isv = 1) into its stage
  auto load_chunk = [&](int i, int slot, int isv) {
    const int c = cbeg + i;
    const uint32_t bar = (isv ? v_full : k_full) + 8 * slot, dst = (isv ? v_base : k_base) + slot * K_BYTES;
    ptx::mbar_expect_tx(bar, K_BYTES);
    if (c < npc) {
      // logical page of the chunk -> page of the pool; the last page goes through the map that ends at the last valid row
      const int lp = p.pages_per_obs == 1 ? 0 : c * KCH / p.page_tokens, row = c * KCH - lp * p.page_tokens;
      const int page = p.page_table ? __ldg(p.page_table + ob * p.pages_per_obs + lp) : ob;
      const bool tail = lp == (p.prefix - 1) / p.page_tokens;
      ptx::tma_load_5d(dst, tail ? (isv ? &p.pv_tail : &p.pk_tail) : (isv ? &p.pv : &p.pk), bar, 0, row, 0, p.layer, page);
    } else {
      ptx::tma_load_4d(dst, isv ? &p.sv : &p.sk, bar, 0, 0, 0, ob);
    }
  };
  int early = 0;                           // chunks requested before the dependency is waited for
  if (warp == 0) {
    if (p.early) {
      for (; early < stg && early < n && cbeg + early < npc; ++early)
        if (leader) { load_chunk(early, early, 0); load_chunk(early, early, 1); }
    }
    if (leader) { ptx::prefetch_tensormap(&p.q); ptx::prefetch_tensormap(&p.sk); ptx::prefetch_tensormap(&p.sv); }
  } else if (warp == 1) {
    ptx::tmem_alloc(ptx::smem_u32(&s_tmem), TM_COLS);
    ptx::tmem_relinquish();
    ptx::grid_dep_launch();                // after the allocation: a later kernel cannot take the columns first
  } else {
    // validity bits of this CTA's keys (an input, not an output of the kernel before)
    for (int w = warp - 2; w < 2 * n; w += 8) {
      const int t = (cbeg * 2 + w) * 32 + lane, s = t - npc * KCH;
      const bool ok = s < 0 ? t < p.prefix && p.valid[(size_t)ob * p.prefix + t] != 0 : s < p.suffix;
      const unsigned bits = __ballot_sync(0xffffffffu, ok);
      if (lane == 0) s_mask[w] = bits;
    }
  }
  ptx::tc_fence_before();
  __syncthreads();
  ptx::tc_fence_after();
  const uint32_t tmem = s_tmem;
  ptx::grid_dep_wait();

  // softmax threads: TMEM lanes 32 (warp % 4) .., key half (warps 2..5: keys 0..31 of a chunk, warps 6..9: keys 32..63)
  const int quad = warp & 3, row = quad * 32 + lane, half = warp >= 6 ? 1 : 0;
  const uint32_t trow = tmem + ((uint32_t)(quad * 32) << 16);
  const bool busy = warp >= 2 && quad * 32 < rows;        // a warp whose rows are all beyond the tile only keeps the barriers going
  bool ok = true;
  float m = -1e30f, l = 0.f;
  constexpr float LOG2E = 1.4426950408889634f;

  if (warp == 0) {
    // ---- producer
    if (leader) {
      ptx::mbar_expect_tx(q_full, 4 * blk);
      for (int kb = 0; kb < 4; ++kb)
        ptx::tma_load_2d(q_base + kb * blk, &p.q, q_full, kb * 64, (ob * p.obs_tokens + tile * p.tok_tile) * NQH);
    }
    for (int i = early, slot = early % stg, par = (early / stg & 1) ^ 1; i < n; ++i) {
      if (!ptx::wait_bar(p.status, p.limit, k_empty + 8 * slot, par, 1)) break;
      if (leader) load_chunk(i, slot, 0);
      if (!ptx::wait_bar(p.status, p.limit, v_empty + 8 * slot, par, 2)) break;
      if (leader) load_chunk(i, slot, 1);
      if (++slot == stg) { slot = 0; par ^= 1; }
    }
  } else if (warp == 1) {
    // ---- MMA issuer
    const uint32_t idesc_s = ptx::umma_idesc_bf16(128, KCH), idesc_o = ptx::umma_idesc_bf16(128, HD) | ptx::UMMA_B_MN_MAJOR;
    const uint64_t qdesc = ptx::umma_smem_desc(q_base), kdesc = ptx::umma_smem_desc(k_base);
    const uint64_t pdesc = ptx::umma_smem_desc(p_base);
    const uint64_t vdesc = ptx::umma_smem_desc_mn(v_base, KCH * 128);
    bool go = ptx::wait_bar(p.status, p.limit, q_full, 0, 3);
    int ks = 0, kpar = 0, vs = 0, vpar = 0;
    auto issue_s = [&](int i) -> bool {
      const int slot = i & 1;
      if (!ptx::wait_bar(p.status, p.limit, k_full + 8 * ks, kpar, 4)) return false;
      if (!ptx::wait_bar(p.status, p.limit, s_empty + 8 * slot, ((i >> 1) & 1) ^ 1, 5)) return false;
      ptx::tc_fence_after();
      if (leader) {
#pragma unroll
        for (int kb = 0; kb < 4; ++kb)
          ptx::umma_bf16_k64(tmem + TM_S + slot * KCH, qdesc + (uint64_t)((kb * blk) >> 4),
                             kdesc + (uint64_t)((ks * K_BYTES + kb * (KCH * 128)) >> 4), idesc_s, kb ? 1u : 0u, 2, 2);
        ptx::umma_commit(s_full + 8 * slot);
        ptx::umma_commit(k_empty + 8 * ks);
      }
      if (++ks == stg) { ks = 0; kpar ^= 1; }
      return true;
    };
    auto issue_pv = [&](int i) -> bool {
      const int slot = i & 1;
      if (!ptx::wait_bar(p.status, p.limit, v_full + 8 * vs, vpar, 6)) return false;
      if (!ptx::wait_bar(p.status, p.limit, p_full + 8 * slot, (i >> 1) & 1, 7)) return false;
      ptx::tc_fence_after();
      if (leader) {
        // 16 keys per MMA: 32 bytes further in P's swizzled rows, 16 rows of 128 B further in V
        ptx::umma_bf16_k64(tmem + TM_O, pdesc + (uint64_t)((slot * blk) >> 4), vdesc + (uint64_t)((vs * K_BYTES) >> 4),
                           idesc_o, i ? 1u : 0u, 2, 16 * 128 / 16);
        ptx::umma_commit(p_empty + 8 * slot);
        ptx::umma_commit(v_empty + 8 * vs);
      }
      if (++vs == stg) { vs = 0; vpar ^= 1; }
      return true;
    };
    for (int i = 0; go && i < n; ++i) {
      go = issue_s(i);
      if (go && i >= 1) go = issue_pv(i - 1);
    }
    if (go) go = issue_pv(n - 1);
    if (go && leader) ptx::umma_commit(o_full);
  } else {
    // ---- softmax threads.  A wait that gives up does not end the loop: the other warp of the quadrant counts on this one at
    // their named barrier, and every further wait returns at once
    constexpr float SCALE_LOG2E = 0.0625f * LOG2E;
    const uint32_t prow = p_base + row * 128, psw = row & 7;
    for (int i = 0; i < n; ++i) {
      const int slot = i & 1;
      ok &= ptx::wait_bar(p.status, p.limit, s_full + 8 * slot, (i >> 1) & 1, 8);
      ptx::tc_fence_after();
      if (!busy) {
        ptx::tc_fence_before();
        ptx::mbar_arrive(s_empty + 8 * slot);
        ptx::mbar_arrive(p_full + 8 * slot);
        continue;
      }
      // Both passes over the row's 32 scores go eight columns at a time in loops that stay loops (the scores are read from
      // TMEM twice): an instruction that runs once costs several cycles to fetch.
      const uint32_t mask = s_mask[2 * i + half], scol = trow + TM_S + slot * KCH + half * 32;
      // maximum of the raw scores: rounding to BF16 and the scale are monotonic, so they are applied to it once
      float mine = -INFINITY;
#pragma unroll 1
      for (int j0 = 0; j0 < 32; j0 += 8) {
        uint32_t r[8];
        ptx::tmem_ld_32x8(scol + j0, r);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (mask >> (j0 + j) & 1) mine = fmaxf(mine, __uint_as_float(r[j]));
      }
      s_max[slot][half][row] = __float2bfloat16_rn(mine);
      ptx::named_bar_sync(1 + quad, 64);                  // the row's other half is in the other warp of this quadrant
      const float cm = fmaxf(rb(mine), __bfloat162float(s_max[slot][half ^ 1][row])) * 0.0625f;
      if (i == 0) {
        m = fmaxf(cm, -1e30f);
      } else if (__any_sync(0xffffffffu, cm > m + RESCALE)) {
        // rare (and the same decision in both warps of the quadrant): move the reference of the rows that need it and
        // rescale this half of what they have accumulated
        const float mn = cm > m + RESCALE ? cm : m, f = ptx::ex2_approx((m - mn) * LOG2E);
        m = mn;
        l *= f;
        ok &= ptx::wait_bar(p.status, p.limit, p_empty + 8 * ((i - 1) & 1), ((i - 1) >> 1) & 1, 9);
        ptx::tc_fence_after();
#pragma unroll 1
        for (int c0 = half * (HD / 2); c0 < (half + 1) * (HD / 2); c0 += 32) {
          uint32_t o[32];
          ptx::tmem_ld_32x32(trow + TM_O + c0, o);
          ptx::tmem_wait_ld();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * f);
          ptx::tmem_st_32x32(trow + TM_O + c0, o);
        }
        ptx::tmem_wait_st();
        ptx::tc_fence_before();
      }
      // the P buffer is free once the P V of chunk i - 2 has read it
      ok &= ptx::wait_bar(p.status, p.limit, p_empty + 8 * slot, ((i >> 1) & 1) ^ 1, 10);
      // p = exp(bf16(s) / 16 - m) as one FMA and one ex2 per score; masked ones are replaced afterwards
      const float mneg = -m * LOG2E;
      const uint32_t dst = prow + slot * blk;
#pragma unroll 1
      for (int j0 = 0; j0 < 32; j0 += 8) {
        uint32_t r[8], pk[4];
        ptx::tmem_ld_32x8(scol + j0, r);
        ptx::tmem_wait_ld();
        const uint32_t mk = mask >> j0;
        float ls[2] = {0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          const uint32_t s0 = pack2(__uint_as_float(r[j]), __uint_as_float(r[j + 1]));
          float a = ptx::ex2_approx(fmaf(lo16(s0), SCALE_LOG2E, mneg)), b = ptx::ex2_approx(fmaf(hi16(s0), SCALE_LOG2E, mneg));
          a = mk & (1u << j) ? a : 0.f;
          b = mk & (2u << j) ? b : 0.f;
          ls[0] += a;
          ls[1] += b;
          pk[j >> 1] = pack2(a, b);
        }
        l += ls[0] + ls[1];
        // 16-byte piece c of the row sits at piece c ^ (row & 7) of its 128-byte line
        if (row < rows) ptx::st_shared_v4(dst + (((uint32_t)(half * 4 + (j0 >> 3)) ^ psw) << 4), pk[0], pk[1], pk[2], pk[3]);
        __syncwarp();
      }
      ptx::tc_fence_before();
      ptx::mbar_arrive(s_empty + 8 * slot);
      __syncwarp();
      ptx::fence_proxy_async_shared();
      ptx::tc_fence_before();
      ptx::mbar_arrive(p_full + 8 * slot);
    }
    ok &= ptx::wait_bar(p.status, p.limit, o_full, 0, 11);
    ptx::tc_fence_after();
  }
  __syncthreads();
  if (warp >= 2) s_sum[half][row] = l;
  __syncthreads();
  if (warp >= 2) l += s_sum[half ^ 1][row];               // both halves of the row's sum
  __syncthreads();

  // ---- O / l -> BF16: row = token_local * 8 + head, so the tile's rows are one contiguous block of [tokens, 2048].  They leave
  // through shared memory by tiled copies (which clip what lies beyond the observation's tokens)
  const int left = p.obs_tokens - tile * p.tok_tile, out_rows = (left < p.tok_tile ? left : p.tok_tile) * NQH;
  uint4* base = reinterpret_cast<uint4*>(p.out + (size_t)(ob * p.obs_tokens + tile * p.tok_tile) * NQH * HD);
  const int c_half = half * (HD / 2);
  if (p.splits == 1) {
    const uint32_t stage = q_base;                        // four swizzled 64-dim blocks, over Q (every MMA has completed)
    if (busy) {
      const float il = 1.0f / l;
#pragma unroll 1
      for (int c0 = 0; c0 < HD / 2; c0 += 16) {
        uint32_t r[16];
        ptx::tmem_ld_32x16(trow + TM_O + c_half + c0, r);
        ptx::tmem_wait_ld();
        const int ch = (c_half + c0) >> 3;                // 16-byte piece of the row
        const uint32_t line = stage + (ch >> 3) * blk + row * 128;
        if (row < rows)
#pragma unroll
          for (int j = 0; j < 2; ++j)
            ptx::st_shared_v4(line + ((((uint32_t)ch + j) & 7) ^ (row & 7)) * 16,
                              pack2(__uint_as_float(r[8 * j]) * il, __uint_as_float(r[8 * j + 1]) * il),
                              pack2(__uint_as_float(r[8 * j + 2]) * il, __uint_as_float(r[8 * j + 3]) * il),
                              pack2(__uint_as_float(r[8 * j + 4]) * il, __uint_as_float(r[8 * j + 5]) * il),
                              pack2(__uint_as_float(r[8 * j + 6]) * il, __uint_as_float(r[8 * j + 7]) * il));
        __syncwarp();
      }
      ptx::tc_fence_before();
      ptx::fence_proxy_async_shared();
    }
    __syncthreads();
    if (tid == 64 && ok) {
#pragma unroll 1
      for (int kb = 0; kb < 4; ++kb) ptx::tma_store_3d(&p.o, stage + kb * blk, kb * 64, tile * rows, ob);
      ptx::bulk_commit();
      ptx::bulk_wait_read();
    }
  } else {
    const size_t pstride = (size_t)MERGE_COLS * rows;
    float* parts = p.merge + (size_t)unit * p.splits * pstride;
    if (busy) {
      float* mine = parts + split * pstride + row;
#pragma unroll 1
      for (int c0 = c_half; c0 < c_half + HD / 2; c0 += 32) {
        uint32_t r[32];
        ptx::tmem_ld_32x32(trow + TM_O + c0, r);
        ptx::tmem_wait_ld();
        if (row < rows)
#pragma unroll
          for (int j = 0; j < 32; ++j) __stcg(mine + (c0 + j) * rows, __uint_as_float(r[j]));
        __syncwarp();
      }
      if (row < rows) __stcg(mine + (HD + half) * rows, half ? l : m);
      __syncwarp();
      ptx::tc_fence_before();
    }
    ptx::cluster_sync();                                  // the parts of every CTA of the tile are in memory
    // this rank's 256 / splits columns (splits is 2, 4 or 8): a thread takes eight columns of a row, a warp 32 rows
    const int nc = (HD / 8) / p.splits, blocks = (out_rows + 31) >> 5;
#pragma unroll 1
    for (int i = warp; i < blocks * nc; i += THREADS / 32) {
      const int rr = (i / nc) * 32 + lane, c = split * nc + i % nc;
      if (rr >= out_rows) continue;
      const float* q = parts + rr;
      float M = -1e30f, L = 0.f, a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int s = 0; s < p.splits; s += 2) {             // two parts at a time: 20 loads in flight
        float v[2][8], pm[2], pl[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float* qs = q + (s + h) * pstride;
          pm[h] = __ldcg(qs + HD * rows);
          pl[h] = __ldcg(qs + (HD + 1) * rows);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[h][j] = __ldcg(qs + (c * 8 + j) * rows);
        }
        const float mn = fmaxf(M, fmaxf(pm[0], pm[1])), g = ptx::ex2_approx((M - mn) * LOG2E);
        const float f0 = ptx::ex2_approx((pm[0] - mn) * LOG2E), f1 = ptx::ex2_approx((pm[1] - mn) * LOG2E);
        M = mn;
        L = L * g + (pl[0] * f0 + pl[1] * f1);
#pragma unroll
        for (int j = 0; j < 8; ++j) a[j] = a[j] * g + (v[0][j] * f0 + v[1][j] * f1);
      }
      const float il = 1.0f / L;
      base[rr * (HD / 8) + c] = make_uint4(pack2(a[0] * il, a[1] * il), pack2(a[2] * il, a[3] * il), pack2(a[4] * il, a[5] * il),
                                           pack2(a[6] * il, a[7] * il));
    }
  }
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, TM_COLS);
  }
}

}  // namespace attn
