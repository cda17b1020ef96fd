// Attention on the tcgen05 tensor cores, used by the action chunk (50 suffix tokens over a prefix cache) and by the prefix
// prefill (every token over every token): the 8 heads of several query tokens share the one KV head, so a tile of N = 8 x tokens
// query rows is one MMA operand.
//
//   * Everything is computed transposed: S^T = K Q^T (128 keys x N), O^T = V^T P (2 x 128 dims x N).  What bounds a CTA is
//     shared memory (128 B per cycle: operands read by the MMAs and copies written), and an MMA reads 128 rows of its A operand
//     whatever is valid.  With the keys, and the dims of V, as A those rows are always full, and the few query rows are
//     B, which may be as narrow as it is: 128 keys cost 1.2 us with 16 query rows and 1.7 us with 112, against 2.3 us for
//     up to 128 rows the other way round.
//   * One CTA = one tile of query tokens against a contiguous share of the keys, in chunks of 128.  The suffix joins the last chunk of the
//     prefix where it fits (up to 72 cached keys there), else it is a chunk of its own; a chunk of up to 64 valid keys skips the other half of V.  `splits` CTAs of a cluster share the keys of a tile
//     and merge through global memory (below).
//   * Warp 0 streams the keys and values with TMA into a ring of 32 KB units, in the order in which the MMAs consume them:
//     K (dims 0-127, dims 128-255) of chunk i + 1, V (keys 0-63, keys 64-127) of chunk i, ..; warp 1 fetches Q and issues S^T of chunk i + 1
//     before O^T of chunk i; warps 2..9 are the softmax threads: thread = one key and half of the query rows.  V and P are
//     taken as they lie, as MN-major operands: nothing is ever transposed in memory.
//   * The keys are passed over once, and after the first chunk without looking for their maximum: the exponent's reference of a
//     row is its maximum over the first chunk, and only when a probability of a later chunk comes out above 2^RESCALE is the
//     reference moved, the accumulator rescaled and the chunk done again.  Numerator and denominator always use the same
//     reference, hence the result does not depend on when it moves.
//   * Scores are rounded to BF16 before the scale 1 / 16, and probabilities before P V, as the reference's BF16 matmuls
//     round (reference/pi05.py:184-188, 254-265).
//   * The cached prefix does not depend on the kernel before this one: with `early` as much of it as the ring holds is requested
//     before the grid dependency is waited for.
//   * Merge of a cluster: each CTA stores its accumulator [row][256] and (reference, sum) per row to global memory; after a
//     cluster barrier every rank adds N / splits rows of all parts, each scaled by exp(m - M) / L.  (The same exchange through
//     distributed shared memory, by ld / st.shared::cluster or by bulk copies, ran at 6-14 B/clk per SM.)
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include "ptx_sm100.cuh"

namespace attn {

constexpr int HD = 256, NQH = 8, KCH = 128, THREADS = 320, SOFTMAX = 256;
constexpr int UNIT = 32 * 1024;                               // ring unit: 128 keys x 128 dims of K or 64 keys x 256 dims of V
constexpr int SEG = KCH * 128;                                // one 64-dim block of a K unit
constexpr int MASK_WORDS = 136;                               // validity bits of up to 4096 prefix tokens + the suffix
constexpr float RESCALE = 7.5f, RESCALE_LOG = 5.0f;           // of exponents to the base 2 / e: 5 log2 e < 7.5, a moved reference satisfies the bound
// Shared memory of a tile of N query rows: Q as four 64-dim blocks [N x 128 B], P as [128 keys x 64 query rows] segments, the ring.
__host__ __device__ constexpr int p_bytes(int n) { return (n > 64 ? 2 : 1) * KCH * 128; }
__host__ __device__ constexpr int units_for(int n) {
  return (226 * 1024 - 512 * n - p_bytes(n)) / UNIT < 6 ? (226 * 1024 - 512 * n - p_bytes(n)) / UNIT : 6;
}
__host__ __device__ constexpr int smem_for(int n) { return 512 * n + p_bytes(n) + units_for(n) * UNIT + 1024; }
static_assert(units_for(16) == 6 && units_for(64) == 5 && units_for(112) == 4 && smem_for(32) + 2048 <= 227 * 1024 && smem_for(112) + 5120 <= 227 * 1024, "attention shared memory");
// FP32 words that a CTA of a split tile leaves behind.
__host__ __device__ constexpr int part_floats(int n) { return n * (HD + 2); }

struct Args {
  CUtensorMap q;                           // [tokens x 8 rows, 256 dims] as {64, rows, 4}, box {64, N, 4}
  CUtensorMap pk, pk_tail, pv, pv_tail;    // prefix keys / values {64 dims, page tokens, 4, layers, pages}; K: box {64, k_rows, k_rows / 64,
                                           // 1, 1}, V: box {64, 64, 4, 1, 1}; *_tail: the same, cut at the last valid token of a last page
  CUtensorMap sk, sv;                      // suffix keys / values {64, tokens, 4, 1, observations}, box {64, 128, 2, 1, 1} and {64, 64, 4, 1, 1}
  CUtensorMap jk, jv, jsk, jsv;            // a last chunk that the suffix joins, a 64-dim segment a copy: m_rows cached keys, then m_suf rows of the suffix
  const int* page_table;                   // [observation][pages_per_obs], or null: page = observation
  const uint8_t* valid;                    // [observation][prefix]
  __nv_bfloat16* out;                      // [tokens, 2048]
  float* merge;                            // splits > 1: [tile][split][part_floats]
  int pages_per_obs, page_tokens, prefix, suffix;      // suffix: keys behind the prefix (0: none; up to 64)
  int k_rows;                              // 128: 128 keys of a chunk are one copy; 64: pages of 64 tokens
  int m_rows, m_suf;                       // 0, or the cached keys of the joined chunk padded to 8 and what the suffix is padded to (16 rows together)
  int obs_tokens, tok_tile, tiles, splits, layer, early;
  unsigned int* status;
  long long limit;
};

// Wait kinds of the status word, behind those of the projections (pi05::WAIT_*).
enum { WAIT_KV_EMPTY = 9, WAIT_KV_FULL, WAIT_Q_FULL, WAIT_S_EMPTY, WAIT_S_FULL, WAIT_P_FULL, WAIT_P_EMPTY, WAIT_O_FULL };

__device__ __forceinline__ float rb(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float lo16(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi16(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }
// Maximum over the warp.
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

template <int N, bool JOIN>     // query rows of a tile; the suffix joins the last chunk of the prefix
__global__ void __launch_bounds__(THREADS, 1) attention_kernel(const __grid_constant__ Args p) {
  constexpr int R = N / 2;                                    // query rows per softmax thread
  constexpr int UNITS = units_for(N), QBLK = N * 128;
  constexpr int TM_S = 0, TM_O = 2 * N, TM_COLS = N <= 16 ? 64 : N <= 32 ? 128 : N <= 64 ? 256 : 512;    // two S^T buffers, two halves of O^T
  constexpr float LOG2E = 1.4426950408889634f, SCALE_LOG2E = 0.0625f * LOG2E;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // barriers: q, full[6], empty[6], s_full[2], s_empty[2], p_full, p_empty, o_full
  __shared__ uint64_t bars[20];
  __shared__ uint32_t s_tmem;
  __shared__ uint32_t s_mask[MASK_WORDS];
  __shared__ float s_red[4][N];            // what the four warps of a half exchange: maxima, at the end sums
  // a warp's own, of its half's rows: factor of a move, summand of the exponents, at the end factor of the result.  Every warp works out what it needs:
  // one barrier less than by a thread per row
  __shared__ __align__(16) float s_row[4][N];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int split = blockIdx.x % p.splits, unit = blockIdx.x / p.splits;
  const int ob = unit / p.tiles, tile = unit % p.tiles;
  const int npc = (p.prefix + KCH - 1) / KCH, late = JOIN ? npc - 1 : npc, total = npc + (!JOIN && p.suffix > 0 ? 1 : 0);    // late: the chunk with suffix keys
  const int cbeg = total * split / p.splits, n = total * (split + 1) / p.splits - cbeg;    // n >= 1: splits <= total
  const uint32_t b0 = ptx::smem_u32(bars);
  const uint32_t q_full = b0, full = b0 + 8, empty = b0 + 56, s_full = b0 + 104, s_empty = b0 + 120, p_full = b0 + 136, p_empty = b0 + 144,
                 o_full = b0 + 152;
  const uint32_t q_base = ptx::smem_u32(smem), p_base = q_base + 4 * QBLK, ring = p_base + p_bytes(N);
  const bool leader = ptx::elect_one();

  // Units of V of this CTA's chunk i (of a joined chunk: halves of the dims, laid out like K; else halves of the keys).  The ring's order is
  // K0 | K1 V0 | K2 V1 | .. | V(n-1); a suffix at the end goes behind the values of the chunk before it, which do not depend on the kernel
  // before this one.
  auto nv = [&](int i) { const int c = cbeg + i; return c < late ? (p.prefix - c * KCH > 64 ? 2 : 1) : JOIN ? 2 : 1; };
  const bool swapped = n >= 2 && cbeg + n > late;

  if (warp == 0) {
    // all 20 (the last of them unused), a lane each: s_empty[2] and p_full are the softmax threads'
    if (lane < 20) ptx::mbar_init(b0 + 8 * lane, (lane >= 15 && lane <= 17) ? SOFTMAX : 1);
    ptx::fence_mbar_init();
    ptx::fence_proxy_async_shared();
  }
  __syncwarp();

  // softmax threads: key 32 (warp % 4) + lane of a chunk, query rows [half R, half R + R)
  const int quad = warp & 3, half = warp >= 6 ? 1 : 0;
  bool ok = true;

  if (warp == 0) {
    // ---- producer
    ptx::bar_arrive(2, THREADS);           // nobody waits for the requests below
    bool waited = false;
    int j = 0, slot = 0;                   // unit in the ring's order
    uint32_t par = 1;
    const bool paged = p.pages_per_obs > 1;
    const int last = paged ? (p.prefix - 1) / p.page_tokens : 0, page0 = paged || !p.page_table ? ob : __ldg(p.page_table + ob);
    auto page_of = [&](int key, int& row, bool& tail) {      // key: first of 64 or 128 keys of a page; beyond the prefix: rows that read as zeros
      row = key;
      tail = true;
      if (!paged) return page0;
      int lp = key / p.page_tokens;
      row = key - lp * p.page_tokens;
      if (lp > last) { lp = last; row = p.page_tokens; }
      tail = lp == last;
      return __ldg(p.page_table + ob * p.pages_per_obs + lp);
    };
    // half of the joined chunk's keys or values (dims 128 u ..): 1: the cached rows, 2: the suffix
    auto joined = [&](int isv, int u, int sl, int what) {
      const uint32_t bar = full + 8 * sl, dst = ring + sl * UNIT;
      if (what & 1) {
        int row;
        bool tail;
        const int page = page_of(late * KCH, row, tail);
        if (leader) {
          ptx::mbar_expect_tx(bar, 2 * (p.m_rows + p.m_suf) * 128);
#pragma unroll 1
          for (int s = 0; s < 2; ++s) ptx::tma_load_5d(dst + s * SEG, isv ? &p.jv : &p.jk, bar, 0, row, 2 * u + s, p.layer, page);
        }
        __syncwarp();
      }
      if (what & 2) {
        if (!waited) { ptx::grid_dep_wait(); waited = true; }
        if (leader)
#pragma unroll 1
          for (int s = 0; s < 2; ++s) ptx::tma_load_5d(dst + s * SEG + p.m_rows * 128, isv ? &p.jsv : &p.jsk, bar, 0, 0, 2 * u + s, 0, ob);
        __syncwarp();
      }
    };
    auto emit = [&](int i, int isv, int u) {
      const int c = cbeg + i;
      if (JOIN && c == late) {
        if (ok && j >= UNITS) ok = ptx::wait_bar(p.status, p.limit, empty + 8 * slot, par, WAIT_KV_EMPTY);
        if (ok) joined(isv, u, slot, 3);
        ++j;
        if (++slot == UNITS) { slot = 0; par ^= 1; }
        return;
      }
      if (!waited && (!p.early || c >= npc)) {
        ptx::grid_dep_wait();
        waited = true;
      }
      if (ok && j >= UNITS) ok = ptx::wait_bar(p.status, p.limit, empty + 8 * slot, par, WAIT_KV_EMPTY);
      if (ok && leader) {
        const uint32_t bar = full + 8 * slot, dst = ring + slot * UNIT;
        ptx::mbar_expect_tx(bar, UNIT);
        int row;
        bool tail;
        if (c >= npc) {
          ptx::tma_load_5d(dst, isv ? &p.sv : &p.sk, bar, 0, 0, isv ? 0 : 2 * u, 0, ob);
        } else if (isv) {
          const int page = page_of(c * KCH + 64 * u, row, tail);
          ptx::tma_load_5d(dst, tail ? &p.pv_tail : &p.pv, bar, 0, row, 0, p.layer, page);
        } else if (p.k_rows == KCH) {
          const int page = page_of(c * KCH, row, tail);
          ptx::tma_load_5d(dst, tail ? &p.pk_tail : &p.pk, bar, 0, row, 2 * u, p.layer, page);
        } else {
#pragma unroll 1
          for (int h = 0; h < 2; ++h) {
            const int page = page_of(c * KCH + 64 * h, row, tail);
            ptx::tma_load_5d(dst + h * 64 * 128, tail ? &p.pk_tail : &p.pk, bar, 0, row, 2 * u, p.layer, page);
            ptx::tma_load_5d(dst + SEG + h * 64 * 128, tail ? &p.pk_tail : &p.pk, bar, 0, row, 2 * u + 1, p.layer, page);
          }
        }
      }
      __syncwarp();
      ++j;
      if (++slot == UNITS) { slot = 0; par ^= 1; }
    };
    // groups of units: K0, then (K_i, V_(i-1)) or, a suffix, (V_(i-1), K_i), then V_(n-1)
    if (JOIN && n == 1 && cbeg == late) {                 // the joined chunk alone: all of its cached rows before the wait
#pragma unroll 1
      for (int g = 0; g < 8; ++g) joined(g >> 1 & 1, g & 1, g & 3, g < 4 ? 1 : 2);
    } else
#pragma unroll 1
    for (int g = 0; g < 2 * n; ++g) {
      const int i = (g + 1) >> 1;                             // groups 2 i - 1 and 2 i are chunk i's keys and the values before it
      const bool isv = i == n || (g > 0 && ((g & 1) == 0) != (swapped && i == n - 1));
      const int ch = isv ? i - 1 : i;
      const int units = isv ? nv(ch) : 2;
      for (int u = 0; u < units; ++u) emit(ch, isv ? 1 : 0, u);
    }
  } else {
    if (warp == 1) {
      ptx::tmem_alloc(ptx::smem_u32(&s_tmem), TM_COLS);
      ptx::tmem_relinquish();
      ptx::grid_dep_launch();              // after the allocation: a later kernel cannot take the columns first
      if (leader) { ptx::prefetch_tensormap(&p.q); ptx::prefetch_tensormap(&p.sk); ptx::prefetch_tensormap(&p.sv); }
      __syncwarp();
    } else {
      // validity bits of this CTA's keys (an input, not an output of the kernel before)
      for (int w = warp - 2; w < 4 * n; w += 8) {
        const int t = (cbeg * 4 + w) * 32 + lane, s = t - late * KCH - (JOIN ? p.m_rows : 0);
        const bool good = t < p.prefix ? p.valid[(size_t)ob * p.prefix + t] != 0 : s >= 0 && s < p.suffix;
        const unsigned bits = __ballot_sync(0xffffffffu, good);
        if (lane == 0) s_mask[w] = bits;
      }
    }
    ptx::tc_fence_before();
    ptx::named_bar_sync(2, THREADS);
    ptx::tc_fence_after();
  }
  const uint32_t tmem = s_tmem;            // (not for warp 0)

  if (warp == 1) {
    // ---- MMA issuer
    const uint32_t idesc_s = ptx::umma_idesc_bf16(KCH, N), idesc_o = ptx::umma_idesc_bf16(128, N) | ptx::UMMA_A_MN_MAJOR | ptx::UMMA_B_MN_MAJOR;
    // lower words of the descriptors (the upper one is the same for all)
    const uint32_t qdesc = (uint32_t)ptx::umma_smem_desc(q_base), kdesc = (uint32_t)ptx::umma_smem_desc(ring);
    const uint32_t pdesc = (uint32_t)ptx::umma_smem_desc_mn(p_base, SEG), vdesc = (uint32_t)ptx::umma_smem_desc_mn(ring, 64 * 128);
    const uint32_t on = leader ? 1u : 0u;
    if (leader) {
      ptx::mbar_expect_tx(q_full, 4 * QBLK);
      ptx::grid_dep_wait();                // Q is this warp's, which is the one that waits for it: warp 0 may still be at the cache
      ptx::tma_load_3d(q_base, &p.q, q_full, 0, (ob * p.obs_tokens + tile * p.tok_tile) * NQH, 0);
    }
    __syncwarp();
    bool go = ptx::wait_bar(p.status, p.limit, q_full, 0, WAIT_Q_FULL);
    // The units in the ring's order, which is the order of use but for a suffix at the end.  What bounds this loop, next to shared memory,
    // is the warp's own instructions between two MMAs.
    int slot = 0;
    uint32_t par = 0;
    auto next = [&](int& sl, uint32_t& pr) { if (++sl == UNITS) { sl = 0; pr ^= 1; } };
    auto issue_s = [&](int i, int& sl, uint32_t& pr) -> bool {
      const int buf = i & 1;
      if (i > 1) {
        if (!ptx::wait_bar(p.status, p.limit, s_empty + 8 * buf, ((i >> 1) & 1) ^ 1, WAIT_S_EMPTY)) return false;
        ptx::tc_fence_after();
      }
#pragma unroll 1
      for (int u = 0; u < 2; ++u) {
        if (!ptx::wait_bar(p.status, p.limit, full + 8 * sl, pr, WAIT_KV_FULL)) return false;
        const uint32_t kd = kdesc + sl * (UNIT >> 4), qd = qdesc + u * (2 * QBLK >> 4);
        ptx::umma_bf16_k64<2, 2>(tmem + TM_S + buf * N, kd, qd, idesc_s, (uint32_t)u, on);
        ptx::umma_bf16_k64<2, 2>(tmem + TM_S + buf * N, kd + (SEG >> 4), qd + (QBLK >> 4), idesc_s, 1u, on);
        if (leader) {
          ptx::umma_commit(empty + 8 * sl);
          if (u == 1) ptx::umma_commit(s_full + 8 * buf);
        }
        __syncwarp();
        next(sl, pr);
      }
      return true;
    };
    auto issue_pv = [&](int i) -> bool {
      const int units = nv(i);
      if (!ptx::wait_bar(p.status, p.limit, p_full, i & 1, WAIT_P_FULL)) return false;
      ptx::tc_fence_after();
      if (JOIN && cbeg + i == late) {
        const int steps = (p.m_rows + p.m_suf) / 16;
#pragma unroll 1
        for (int u = 0; u < 2; ++u) {
          if (!ptx::wait_bar(p.status, p.limit, full + 8 * slot, par, WAIT_KV_FULL)) return false;
          const uint32_t vd = vdesc + ((SEG - 64 * 128) << 12) + slot * (UNIT >> 4), od = tmem + TM_O + u * N;      // (segments 128 keys apart)
          int s = 0;
#pragma unroll 1
          for (; s + 4 <= steps; s += 4) ptx::umma_bf16_k64<128, 128>(od, vd + s * 128, pdesc + s * 128, idesc_o, i || s ? 1u : 0u, on);
#pragma unroll 1
          for (; s < steps; ++s) ptx::umma_bf16_k16(od, vd + s * 128, pdesc + s * 128, idesc_o, i || s ? 1u : 0u, on);
          if (leader) {
            ptx::umma_commit(empty + 8 * slot);
            if (u == 1) ptx::umma_commit(p_empty);
          }
          __syncwarp();
          next(slot, par);
        }
        return true;
      }
#pragma unroll 1
      for (int u = 0; u < units; ++u) {
        if (!ptx::wait_bar(p.status, p.limit, full + 8 * slot, par, WAIT_KV_FULL)) return false;
        // 16 keys per MMA: 16 rows of 128 B further in V and in P
        const uint32_t vd = vdesc + slot * (UNIT >> 4), pd = pdesc + u * (64 * 128 >> 4), acc = i || u ? 1u : 0u;
        ptx::umma_bf16_k64<128, 128>(tmem + TM_O, vd, pd, idesc_o, acc, on);
        ptx::umma_bf16_k64<128, 128>(tmem + TM_O + N, vd + ((2 * 64 * 128) >> 4), pd, idesc_o, acc, on);
        if (leader) {
          ptx::umma_commit(empty + 8 * slot);
          if (u == units - 1) ptx::umma_commit(p_empty);
        }
        __syncwarp();
        next(slot, par);
      }
      return true;
    };
#pragma unroll 1
    for (int i = 0; go && i <= n; ++i) {   // S of chunk i, then P V of the one before
      int sl = slot;
      uint32_t pr = par;
      const bool suffix = swapped && i == n - 1;            // its keys stand behind the values of the chunk before it
      if (suffix)
        for (int u = nv(i - 1); u > 0; --u) next(sl, pr);
      if (i < n) go = issue_s(i, sl, pr);
      if (!suffix) { slot = sl; par = pr; }
      if (go && i >= 1) go = issue_pv(i - 1);
      if (suffix) { slot = sl; par = pr; }
    }
    if (go && leader) ptx::umma_commit(o_full);
    __syncwarp();
  } else if (warp >= 2) {
    // ---- softmax threads.  A wait that gives up does not end the loop: the other warps count on this one at their named
    // barriers, and every further wait returns at once
    const int r0 = half * R;
    const uint32_t trow = tmem + ((uint32_t)(quad * 32) << 16) + r0;
    float l[R];
#pragma unroll
    for (int r = 0; r < R; ++r) l[r] = 0.f;
    constexpr int ROWS = (R + 31) / 32;                       // rows of the half per lane, with their references
    float m[ROWS];
#pragma unroll 1
    for (int i = 0; i < n; ++i) {
      const int buf = i & 1;
      ok &= ptx::wait_bar(p.status, p.limit, s_full + 8 * buf, (i >> 1) & 1, WAIT_S_FULL);
      ptx::tc_fence_after();
      const bool key = s_mask[4 * i + quad] >> lane & 1;      // this thread's key counts
      const uint32_t scol = trow + TM_S + buf * N;
      // the key's line of P: piece c (8 query rows) at c ^ (key & 7), 64 query rows per segment
      const uint32_t line = p_base + (quad * 32 + lane) * 128, psw = lane & 7;
#pragma unroll 1
      for (int tries = i > 0 ? 1 : 0;; ++tries) {             // 0: no reference yet
        if (tries > 0) {
          // p = exp(bf16(s) / 16 - m) as one FMA and one ex2 per score; the vote looks at the exponents
          float t[R], top = -INFINITY;
          {
            uint32_t x[R];
#pragma unroll
            for (int c = 0; c < R; c += 8) ptx::tmem_ld_32x8(scol + c, *reinterpret_cast<uint32_t(*)[8]>(&x[c]));
            ptx::tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < R; c += 4) {
              const float4 mn = *reinterpret_cast<const float4*>(&s_row[quad][r0 + c]);
              const uint32_t x0 = pack2(__uint_as_float(x[c]), __uint_as_float(x[c + 1])), x1 = pack2(__uint_as_float(x[c + 2]), __uint_as_float(x[c + 3]));
              t[c] = fmaf(lo16(x0), SCALE_LOG2E, mn.x); t[c + 1] = fmaf(hi16(x0), SCALE_LOG2E, mn.y);
              t[c + 2] = fmaf(lo16(x1), SCALE_LOG2E, mn.z); t[c + 3] = fmaf(hi16(x1), SCALE_LOG2E, mn.w);
              top = fmaxf(fmaxf(top, fmaxf(t[c], t[c + 1])), fmaxf(t[c + 2], t[c + 3]));
            }
          }
          if (i == 0 || !ptx::named_bar_or(1, SOFTMAX, key && top > RESCALE) || tries > 2) {
            uint32_t pk[R / 2];
#pragma unroll
            for (int r = 0; r < R; r += 2) {
              const float e0 = key ? ptx::ex2_approx(t[r]) : 0.f, e1 = key ? ptx::ex2_approx(t[r + 1]) : 0.f;
              l[r] += e0;
              l[r + 1] += e1;
              pk[r / 2] = pack2(e0, e1);
            }
            // the P buffer is free once the P V of the chunk before has read it
            if (i > 0) ok &= ptx::wait_bar(p.status, p.limit, p_empty, (i - 1) & 1, WAIT_P_EMPTY);
#pragma unroll
            for (int c = 0; c < R; c += 8) {
              const uint32_t piece = (uint32_t)(r0 + c) >> 3;
              ptx::st_shared_v4(line + (piece >> 3) * SEG + (((piece & 7) ^ psw) << 4), pk[c / 2], pk[c / 2 + 1], pk[c / 2 + 2], pk[c / 2 + 3]);
            }
            break;
          }
        }
        // rare, but for the first chunk: find the maximum (of the raw scores: rounding to BF16 and the scale are monotonic)
#pragma unroll 1
        for (int c = 0; c < R; c += 8) {
          uint32_t s[8];
          ptx::tmem_ld_32x8(scol + c, s);
          ptx::tmem_wait_ld();
          float mx = 0.f;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float v = warp_max(key ? __uint_as_float(s[k]) : -INFINITY);
            if (lane == k) mx = v;
          }
          if (lane < 8) s_red[quad][r0 + c + lane] = mx;
          __syncwarp();
        }
        ptx::named_bar_sync(1, SOFTMAX);
#pragma unroll
        for (int j = 0; j < ROWS; ++j) {
          const int k = r0 + lane + 32 * j;
          if (k < r0 + R) {
            const float cm = rb(fmaxf(fmaxf(s_red[0][k], s_red[1][k]), fmaxf(s_red[2][k], s_red[3][k]))) * 0.0625f;
            float f = 1.f;
            if (i == 0) m[j] = fmaxf(cm, -1e30f);
            else if (cm > m[j] + RESCALE_LOG) { f = ptx::ex2_approx((m[j] - cm) * LOG2E); m[j] = cm; }
            s_row[quad][k] = i == 0 ? -m[j] * LOG2E : f;
          }
        }
        __syncwarp();
        if (i > 0) {
          // rescale what has been accumulated
#pragma unroll
          for (int r = 0; r < R; ++r) l[r] *= s_row[quad][r0 + r];
          ok &= ptx::wait_bar(p.status, p.limit, p_empty, (i - 1) & 1, WAIT_P_EMPTY);
          ptx::tc_fence_after();
#pragma unroll 1
          for (int c = 0; c < 2 * R; c += 8) {
            const int row = c < R ? c : c - R;
            const uint32_t at = trow + TM_O + (c < R ? 0 : N) + row;
            uint32_t o[8];
            ptx::tmem_ld_32x8(at, o);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int k = 0; k < 8; ++k) o[k] = __float_as_uint(__uint_as_float(o[k]) * s_row[quad][r0 + row + k]);
            ptx::tmem_st_32x8(at, o);
          }
          ptx::tmem_wait_st();
          __syncwarp();
#pragma unroll
          for (int j = 0; j < ROWS; ++j)
            if (lane + 32 * j < R) s_row[quad][r0 + lane + 32 * j] = -m[j] * LOG2E;
          __syncwarp();
        }
      }
      __syncwarp();
      ptx::tc_fence_before();
      ptx::mbar_arrive(s_empty + 8 * buf);
      ptx::fence_proxy_async_shared();
      ptx::mbar_arrive(p_full);
    }
    // the rows' sums over all keys, while the last P V runs
    if (n == 1) ptx::named_bar_sync(1, SOFTMAX);              // (with more chunks their votes lie between the maxima's readers and this)
#pragma unroll
    for (int c = 0; c < R; c += 8) {
      float mine = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float v = l[c + k];
#pragma unroll
        for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        if (lane == k) mine = v;
      }
      if (lane < 8) s_red[quad][r0 + c + lane] = mine;
    }
    __syncwarp();
    ptx::named_bar_sync(1, SOFTMAX);
    float* part = p.merge + (size_t)(unit * p.splits + split) * part_floats(N);
#pragma unroll
    for (int j = 0; j < ROWS; ++j) {
      const int k = r0 + lane + 32 * j;
      if (k < r0 + R) {
        const float sum = (s_red[0][k] + s_red[1][k]) + (s_red[2][k] + s_red[3][k]);
        if (p.splits == 1) s_row[quad][k] = sum > 0.f ? 1.0f / sum : 0.f;     // (no valid key: zeros)
        else if (quad == 0) __stcg(reinterpret_cast<float2*>(part + N * HD) + k, make_float2(m[j], sum));
      }
    }
    __syncwarp();
    ok &= ptx::wait_bar(p.status, p.limit, o_full, 0, WAIT_O_FULL);
    ptx::tc_fence_after();

    // ---- O^T / l -> BF16 [row][256] (row = token_local * 8 + head: the tile's rows are one contiguous block of [tokens, 2048])
    if (p.splits == 1) {
      // straight to memory, 64 bytes of a row per warp and store: through shared memory and tiled copies, with their fence, barrier
      // and wait, a layer pass took 0.3 us longer at 16 query rows per tile and 0.8 us at 48
      const int left = p.obs_tokens - tile * p.tok_tile, out_rows = (left < p.tok_tile ? left : p.tok_tile) * NQH;
      __nv_bfloat16* base = p.out + (size_t)(ob * p.obs_tokens + tile * p.tok_tile) * NQH * HD + quad * 32 + lane;
#pragma unroll 1
      for (int c = 0; c < 2 * R; c += 8) {
        const int d = c < R ? 0 : 1, row = r0 + (d ? c - R : c);
        uint32_t o[8];
        ptx::tmem_ld_32x8(trow + TM_O + d * N + (row - r0), o);
        ptx::tmem_wait_ld();
        if (row < out_rows && ok)
#pragma unroll
          for (int k = 0; k < 8; ++k) base[(row + k) * HD + d * 128] = __float2bfloat16_rn(__uint_as_float(o[k]) * s_row[quad][row + k]);
        __syncwarp();
      }
      ptx::tc_fence_before();
    } else {
#pragma unroll 1
      for (int c = 0; c < 2 * R; c += 8) {
        const int d = c < R ? 0 : 1, row = r0 + (d ? c - R : c);
        uint32_t o[8];
        ptx::tmem_ld_32x8(trow + TM_O + d * N + (row - r0), o);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 8; ++k) __stcg(part + (row + k) * HD + d * 128 + quad * 32 + lane, __uint_as_float(o[k]));
      }
      ptx::tc_fence_before();
    }
  }
  __syncthreads();
  if (p.splits > 1) {
    ptx::cluster_sync();                                      // the parts of every CTA of the tile are in memory
    const int left = p.obs_tokens - tile * p.tok_tile, out_rows = (left < p.tok_tile ? left : p.tok_tile) * NQH;
    uint4* base = reinterpret_cast<uint4*>(p.out + (size_t)(ob * p.obs_tokens + tile * p.tok_tile) * NQH * HD);
    // a warp takes a row of this rank's, a lane eight dims
    for (int row = split * (N / p.splits) + warp; row < (split + 1) * (N / p.splits) && row < out_rows; row += THREADS / 32) {
      const float* q = p.merge + (size_t)unit * p.splits * part_floats(N);
      float M = -1e30f, L = 0.f, a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      float4 x[8], y[8];                                      // every part is on its way before the first is used
      float2 ml[8];
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const float* qs = q + (s < p.splits ? s : 0) * part_floats(N);
        ml[s] = __ldcg(reinterpret_cast<const float2*>(qs + N * HD) + row);
        x[s] = __ldcg(reinterpret_cast<const float4*>(qs + row * HD + lane * 8));
        y[s] = __ldcg(reinterpret_cast<const float4*>(qs + row * HD + lane * 8) + 1);
        if (s >= p.splits) ml[s] = make_float2(-1e30f, 0.f);
        M = fmaxf(M, ml[s].x);
      }
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const float f = s < p.splits ? ptx::ex2_approx((ml[s].x - M) * LOG2E) : 0.f;
        L += ml[s].y * f;
        a[0] += x[s].x * f; a[1] += x[s].y * f; a[2] += x[s].z * f; a[3] += x[s].w * f;
        a[4] += y[s].x * f; a[5] += y[s].y * f; a[6] += y[s].z * f; a[7] += y[s].w * f;
      }
      const float il = L > 0.f ? 1.0f / L : 0.f;
      base[row * (HD / 8) + lane] = make_uint4(pack2(a[0] * il, a[1] * il), pack2(a[2] * il, a[3] * il), pack2(a[4] * il, a[5] * il),
                                               pack2(a[6] * il, a[7] * il));
    }
  }
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, TM_COLS);
  }
}

}  // namespace attn
