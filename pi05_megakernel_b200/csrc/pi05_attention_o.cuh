// Attention and O projection of the action chunk in one kernel, for prefixes whose keys and values fit into shared memory beside everything
// else (up to 128 tokens) and few observations.
//
// A CTA takes one query head of an observation and 128 output features: it computes the attention of all 50 tokens of the head - the eight CTAs
// of a head compute the same - and multiplies it by its 128 x 256 block of Wo.  Its 50 x 128 partial sums go to the slice of the head, and the
// residual kernel adds the eight heads as it adds K splits.  What that buys is a stage less in the chain: at 50 tokens and 128 cached keys
// attention and O projection took 5.15 + 3.9 us of a layer pass of 26.6, most of it waiting (a hop, the first operands, two
// softmax rounds one after the other, drain and output of two kernels).
//
//   * All keys lie in shared memory, [prefix, padded to 8 rows | suffix] as rows of 64-dim segments, and are taken in one pass: S^T = K Q^T
//     as one or two MMAs of 128 key rows, softmax over all of them at once by 16 warps (thread = one key and half of the query rows),
//     O^T = V^T P, and D = Wo O^T with the normalised, BF16-rounded O^T as B operand.  The same roundings as in pi05_attention.cuh.
//   * Shared memory: K | V | Q.  P and (where it has no place of its own) the block of Wo take K's place once the scores are done, O^T
//     takes Q's.  Cached keys and values are requested before the kernel before this one has finished, Wo too or at least brought into L2.
//   * Reductions over a warp's 32 keys fold values and lanes together (32 rows: 16 shuffles of packed pairs for the maximum, 31 for the sum).
#pragma once
#include "pi05_attention.cuh"
#include "pi05_common.cuh"

namespace attno {
using attn::HD;
using attn::lo16;
using attn::hi16;
using attn::pack2;

constexpr int NTHREADS = 576, SOFTMAX = 512, N = 64, R = 32, TOK = pi05::T, SUF = 56, QROWS = 56, FEAT = 128, GROUPS = pi05::W / FEAT;
constexpr int MAX_PREFIX = 128, WO_BYTES = FEAT * HD * 2, OT_BYTES = HD * 128;
constexpr int MAX_SMEM = 221 * 1024;       // of `layout`, and 5 KB of static shared memory
static_assert(MAX_SMEM + 5632 <= 227 * 1024, "shared memory");

struct Args {
  CUtensorMap q;                           // {64 dims, tokens, 32}, box {64, 56, 4}
  CUtensorMap pk0, pk1, pv0, pv1;          // cached keys / values {64 dims, page tokens, 4, layers, pages}, boxes of rows0 and rows1 tokens; cut at the last valid token
  CUtensorMap sk, sv;                      // suffix keys / values {64, 50, 4, 1, observations}, box {64, 56, 1, 1, 1}
  CUtensorMap wo;                          // {64 k, layers x 1024 features, 32}, box {64, 128, 4}
  const __nv_bfloat16* wo_base;
  const int* page_table;
  const uint8_t* valid;                    // [observation][prefix]
  float* part;                             // [8 heads][tokens][1024]
  int pages_per_obs, prefix, layer, tokens;        // tokens: 50 x observations
  int rows0, rows1;                        // rows of the prefix in the first page and in the second (0: none); their sum is the prefix, padded to 8
  int off_v, off_q, off_wo, wo_early;
  unsigned int* status;
  long long limit;
};

// What the kernel needs for a prefix: rows of keys, places in shared memory.
struct Layout { int rows, off_v, off_q, off_wo, wo_early, smem; };
inline Layout layout(int prefix) {
  Layout l;
  l.rows = (prefix + 7) / 8 * 8 + SUF;
  const int kv = l.rows * 512, p = (l.rows + 15) / 16 * 16 * 128;
  l.wo_early = 2 * kv + OT_BYTES + WO_BYTES <= MAX_SMEM - 1024;
  l.off_v = l.wo_early || kv > p + WO_BYTES ? kv : p + WO_BYTES;
  l.off_q = l.off_v + kv;
  l.off_wo = l.wo_early ? l.off_q + OT_BYTES : p;
  l.smem = l.off_q + OT_BYTES + (l.wo_early ? WO_BYTES : 0) + 1024;
  return l;
}

__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) {
  const __nv_bfloat162 m = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&m);
}

// (A template so that every file that includes this one may, and only the one that launches the kernel compiles it.)
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) attention_o_kernel(const __grid_constant__ Args p) {
  constexpr int TM_S = 0, TM_O = 128, TM_D = 0, TM_COLS = 256;       // two S^T, two halves of O^T; D takes the place of S^T
  constexpr float LOG2E = 1.4426950408889634f, SCALE_LOG2E = 0.0625f * LOG2E;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  // k (prefix), ks (suffix), v, q, w, s[2], p, o[2], ot[2], d
  __shared__ uint64_t bars[13];
  __shared__ uint32_t s_tmem;
  __shared__ uint32_t s_max[8][N / 2];     // a warp row's maxima, BF16 pairs
  __shared__ float s_sum[8][N];
  __shared__ __align__(16) float s_mneg[N], s_f[N];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int group = blockIdx.x % GROUPS, head = blockIdx.x / GROUPS % pi05::NQH, ob = blockIdx.x / (GROUPS * pi05::NQH);
  const int r8 = p.rows0 + p.rows1, rows = r8 + SUF, seg = rows * 128, steps = (rows + 15) / 16;
  const bool two = rows > 128;
  const uint32_t b0 = ptx::smem_u32(bars);
  const uint32_t k_full = b0, ks_full = b0 + 8, v_full = b0 + 16, q_full = b0 + 24, w_full = b0 + 32, s_full = b0 + 40, p_full = b0 + 56, o_full = b0 + 64,
                 ot_full = b0 + 80, d_full = b0 + 96;
  const uint32_t k_base = ptx::smem_u32(smem), v_base = k_base + p.off_v, q_base = k_base + p.off_q, wo_base = k_base + p.off_wo;
  const bool leader = ptx::elect_one();
  bool ok = true;

  if (warp == 0) {
    if (lane < 13) ptx::mbar_init(b0 + 8 * lane, lane == 7 ? SOFTMAX : lane == 10 || lane == 11 ? SOFTMAX / 2 : 1);
    ptx::fence_mbar_init();
    ptx::fence_proxy_async_shared();
    __syncwarp();
    // ---- producer
    ptx::bar_arrive(2, THREADS);           // nobody waits for the requests below
    if (leader) {
      const int page0 = p.pages_per_obs > 1 ? __ldg(p.page_table + ob * p.pages_per_obs) : p.page_table ? __ldg(p.page_table + ob) : ob;
      const int page1 = p.rows1 ? __ldg(p.page_table + ob * p.pages_per_obs + 1) : 0;
      auto prefix = [&](const CUtensorMap* m0, const CUtensorMap* m1, uint32_t dst, uint32_t bar) {
#pragma unroll 1
        for (int s = 0; s < 4; ++s) {
          ptx::tma_load_5d(dst + s * seg, m0, bar, 0, 0, s, p.layer, page0);
          if (p.rows1) ptx::tma_load_5d(dst + s * seg + p.rows0 * 128, m1, bar, 0, 0, s, p.layer, page1);
        }
      };
      ptx::mbar_expect_tx(k_full, 4 * r8 * 128);
      prefix(&p.pk0, &p.pk1, k_base, k_full);
      ptx::mbar_expect_tx(v_full, 4 * rows * 128);
      prefix(&p.pv0, &p.pv1, v_base, v_full);
      if (p.wo_early) {
        ptx::mbar_expect_tx(w_full, WO_BYTES);
        ptx::tma_load_3d(wo_base, &p.wo, w_full, 0, p.layer * pi05::W + group * FEAT, head * 4);
      }
    }
    __syncwarp();
    if (leader) {
      ptx::mbar_expect_tx(ks_full, 4 * SUF * 128);
      ptx::grid_dep_wait();                // right before the first copy, when everything that it takes is computed
#pragma unroll 1
      for (int s = 0; s < 4; ++s) ptx::tma_load_5d(k_base + s * seg + r8 * 128, &p.sk, ks_full, 0, 0, s, 0, ob);
#pragma unroll 1
      for (int s = 0; s < 4; ++s) ptx::tma_load_5d(v_base + s * seg + r8 * 128, &p.sv, v_full, 0, 0, s, 0, ob);
    }
    __syncwarp();
    if (!p.wo_early) {                     // behind P in the place of the keys, once the scores are done
      ok = ptx::wait_bar(p.status, p.limit, s_full, 0, attn::WAIT_S_FULL);
      if (two) ok = ok && ptx::wait_bar(p.status, p.limit, s_full + 8, 0, attn::WAIT_S_FULL);
      if (ok && leader) {
        ptx::mbar_expect_tx(w_full, WO_BYTES);
        ptx::tma_load_3d(wo_base, &p.wo, w_full, 0, p.layer * pi05::W + group * FEAT, head * 4);
      }
      __syncwarp();
    }
  } else {
    if (warp == 1) {
      ptx::tmem_alloc(ptx::smem_u32(&s_tmem), TM_COLS);
      ptx::tmem_relinquish();
      ptx::grid_dep_launch();              // after the allocation: a later kernel cannot take the columns first
      if (leader) { ptx::prefetch_tensormap(&p.q); ptx::prefetch_tensormap(&p.sk); ptx::prefetch_tensormap(&p.sv); ptx::prefetch_tensormap(&p.wo); }
      __syncwarp();
    } else if (!p.wo_early) {
      // this CTA's block of Wo into L2: 128 rows of four lines, a line each
      const int et = tid - 64;
      const char* line = reinterpret_cast<const char*>(p.wo_base + ((size_t)p.layer * pi05::W + group * FEAT + (et >> 2)) * pi05::QD + head * HD) + (et & 3) * 128;
      asm volatile("prefetch.global.L2 [%0];" ::"l"(line));
    }
    ptx::tc_fence_before();
    ptx::named_bar_sync(2, THREADS);
    ptx::tc_fence_after();
  }
  const uint32_t tmem = s_tmem;            // (not for warp 0)

  if (warp == 1) {
    // ---- MMA issuer
    const uint32_t idesc_s = ptx::umma_idesc_bf16(128, N), idesc_o = idesc_s | ptx::UMMA_A_MN_MAJOR | ptx::UMMA_B_MN_MAJOR, idesc_d = idesc_s | ptx::UMMA_B_MN_MAJOR;
    const uint32_t qdesc = (uint32_t)ptx::umma_smem_desc(q_base), kdesc = (uint32_t)ptx::umma_smem_desc(k_base), wdesc = (uint32_t)ptx::umma_smem_desc(wo_base);
    const uint32_t vdesc = (uint32_t)ptx::umma_smem_desc_mn(v_base, seg), pdesc = (uint32_t)ptx::umma_smem_desc_mn(k_base, 16384),
                   odesc = (uint32_t)ptx::umma_smem_desc_mn(q_base, 16384);
    const uint32_t on = leader ? 1u : 0u;
    if (leader) {
      ptx::mbar_expect_tx(q_full, 4 * QROWS * 128);
      ptx::grid_dep_wait();
      ptx::tma_load_3d(q_base, &p.q, q_full, 0, ob * TOK, head * 4);
    }
    __syncwarp();
    bool go = ptx::wait_bar(p.status, p.limit, k_full, 0, attn::WAIT_KV_FULL);
    if (go && r8 < 128) go = ptx::wait_bar(p.status, p.limit, ks_full, 0, attn::WAIT_KV_FULL);
    go = go && ptx::wait_bar(p.status, p.limit, q_full, 0, attn::WAIT_Q_FULL);
#pragma unroll 1
    for (int c = 0; go && c < (two ? 2 : 1); ++c) {
      if (c && r8 >= 128) go = ptx::wait_bar(p.status, p.limit, ks_full, 0, attn::WAIT_KV_FULL);
      if (!go) break;
#pragma unroll
      for (int s = 0; s < 4; ++s)
        ptx::umma_bf16_k64<2, 2>(tmem + TM_S + c * N, kdesc + ((s * seg + c * 16384) >> 4), qdesc + (s * QROWS * 128 >> 4), idesc_s, s ? 1u : 0u, on);
      if (leader) ptx::umma_commit(s_full + 8 * c);
      __syncwarp();
    }
    go = go && ptx::wait_bar(p.status, p.limit, v_full, 0, attn::WAIT_KV_FULL);
    go = go && ptx::wait_bar(p.status, p.limit, p_full, 0, attn::WAIT_P_FULL);
    if (go) {
      ptx::tc_fence_after();
      // (where the rows are an odd number of eights, the last 16 keys reach into the next segment's values, behind the last one into Q, and into O^T while its
      // first half is being written there: finite values times the zeros that P has in those rows)
#pragma unroll 1
      for (int d = 0; d < 2; ++d) {
        const uint32_t vd = vdesc + (d * 2 * seg >> 4), od = tmem + TM_O + d * N;
        int s = 0;
#pragma unroll 1
        for (; s + 4 <= steps; s += 4) ptx::umma_bf16_k64<128, 128>(od, vd + s * 128, pdesc + s * 128, idesc_o, s ? 1u : 0u, on);
#pragma unroll 1
        for (; s < steps; ++s) ptx::umma_bf16_k16(od, vd + s * 128, pdesc + s * 128, idesc_o, s ? 1u : 0u, on);
        if (leader) ptx::umma_commit(o_full + 8 * d);
        __syncwarp();
      }
    }
    go = go && ptx::wait_bar(p.status, p.limit, w_full, 0, pi05::WAIT_W_FULL);
#pragma unroll 1
    for (int d = 0; go && d < 2; ++d) {
      go = ptx::wait_bar(p.status, p.limit, ot_full + 8 * d, 0, attn::WAIT_P_FULL);
      if (!go) break;
      ptx::tc_fence_after();
#pragma unroll
      for (int b = 0; b < 2; ++b)          // 64 dims: a block of Wo, 64 rows of O^T
        ptx::umma_bf16_k64<2, 128>(tmem + TM_D, wdesc + ((2 * d + b) * FEAT * 128 >> 4), odesc + ((2 * d + b) * 64 * 128 >> 4), idesc_d, d || b ? 1u : 0u, on);
      if (d == 1 && leader) ptx::umma_commit(d_full);
      __syncwarp();
    }
  } else if (warp >= 2) {
    // ---- softmax threads: key 128 chunk + 32 quad + lane, query rows 32 half ..; a wait that gives up does not end the role: the other warps
    // count on this one at their named barriers
    const int et = tid - 64, part = (warp - 2) >> 2, chunk = part >> 1, half = part & 1, quad = warp & 3, r0 = half * R;
    const int kk = chunk * 128 + quad * 32 + lane;
    const bool active = chunk * 128 + quad * 32 < rows;       // the warp has rows of P
    const bool key = kk < p.prefix ? p.valid[(size_t)ob * p.prefix + kk] != 0 : kk >= r8 && kk < r8 + TOK;
    const uint32_t trow = tmem + ((uint32_t)(quad * 32) << 16);
    uint32_t x[R / 2];
    if (active) {
      ok &= ptx::wait_bar(p.status, p.limit, s_full + 8 * chunk, 0, attn::WAIT_S_FULL);
      ptx::tc_fence_after();
      uint32_t s[R];
#pragma unroll
      for (int c = 0; c < R; c += 16) ptx::tmem_ld_32x16(trow + TM_S + chunk * N + r0 + c, *reinterpret_cast<uint32_t(*)[16]>(&s[c]));
      ptx::tmem_wait_ld();
      uint32_t m[R / 2];
#pragma unroll
      for (int i = 0; i < R / 2; ++i) {
        x[i] = pack2(__uint_as_float(s[2 * i]), __uint_as_float(s[2 * i + 1]));
        m[i] = key ? x[i] : 0xff80ff80u;
      }
#pragma unroll
      for (int w = 8; w; w >>= 1)          // lanes 2 w apart share their values, each keeps half of them
#pragma unroll
        for (int i = 0; i < w; ++i) {
          const uint32_t keep = lane & (2 * w) ? m[i + w] : m[i], send = lane & (2 * w) ? m[i] : m[i + w];
          m[i] = max2(keep, __shfl_xor_sync(0xffffffffu, send, 2 * w));
        }
      m[0] = max2(m[0], __shfl_xor_sync(0xffffffffu, m[0], 1));
      if (!(lane & 1)) s_max[chunk * 4 + quad][half * (R / 2) + (lane >> 1)] = m[0];
      ptx::tc_fence_before();
    }
    ptx::named_bar_sync(1, SOFTMAX);
    const int nq = (rows + 31) / 32;       // warp rows of keys
    if (et < N) {
      float m = -INFINITY;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < nq) { const uint32_t v = s_max[q][et >> 1]; m = fmaxf(m, et & 1 ? hi16(v) : lo16(v)); }
      s_mneg[et] = -fmaxf(m * 0.0625f, -1e30f) * LOG2E;       // (no valid key: every probability is 0)
    }
    ptx::named_bar_sync(1, SOFTMAX);
    if (active) {
      // p = exp(bf16(s) / 16 - m); query rows beyond the 50 tokens get zeros
      float e[R];
#pragma unroll
      for (int c = 0; c < R; c += 4) {
        const float4 mn = *reinterpret_cast<const float4*>(&s_mneg[r0 + c]);
        const float mv[4] = {mn.x, mn.y, mn.z, mn.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int r = c + k;
          e[r] = 0.f;
          if (key && (r < TOK - R || half == 0)) e[r] = ptx::ex2_approx(fmaf(r & 1 ? hi16(x[r / 2]) : lo16(x[r / 2]), SCALE_LOG2E, mv[k]));
        }
      }
      const uint32_t line = k_base + kk * 128;
      if (kk < steps * 16)
#pragma unroll
        for (int c = 0; c < R; c += 8)
          ptx::st_shared_v4(line + ((((uint32_t)(r0 + c) >> 3) ^ (lane & 7)) << 4), pack2(e[c], e[c + 1]), pack2(e[c + 2], e[c + 3]), pack2(e[c + 4], e[c + 5]),
                            pack2(e[c + 6], e[c + 7]));
      ptx::fence_proxy_async_shared();
      ptx::mbar_arrive(p_full);
#pragma unroll
      for (int w = 16; w; w >>= 1)
#pragma unroll
        for (int i = 0; i < w; ++i) {
          const float keep = lane & w ? e[i + w] : e[i], send = lane & w ? e[i] : e[i + w];
          e[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
      s_sum[chunk * 4 + quad][r0 + lane] = e[0];
    } else {
      ptx::mbar_arrive(p_full);
    }
    ptx::named_bar_sync(1, SOFTMAX);
    if (et < N) {
      float sum = 0.f;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < nq) sum += s_sum[q][et];
      s_f[et] = sum > 0.f ? 1.0f / sum : 0.f;                 // (no valid key: zeros)
    }
    ptx::named_bar_sync(1, SOFTMAX);
    // ---- O^T / l -> BF16, as the B operand of the projection: half d of the dims, 32 tokens
    {
      const int d = part >> 1, t0 = (part & 1) * 32;
      ok &= ptx::wait_bar(p.status, p.limit, o_full + 8 * d, 0, attn::WAIT_O_FULL);
      ptx::tc_fence_after();
      uint32_t o[32];
#pragma unroll
      for (int c = 0; c < 32; c += 16) ptx::tmem_ld_32x16(trow + TM_O + d * N + t0 + c, *reinterpret_cast<uint32_t(*)[16]>(&o[c]));
      ptx::tmem_wait_ld();
      const uint32_t line = q_base + (d * 128 + quad * 32 + lane) * 128;
#pragma unroll
      for (int c = 0; c < 32; c += 8) {
        const float4 f0 = *reinterpret_cast<const float4*>(&s_f[t0 + c]), f1 = *reinterpret_cast<const float4*>(&s_f[t0 + c + 4]);
        ptx::st_shared_v4(line + ((((uint32_t)(t0 + c) >> 3) ^ (lane & 7)) << 4),
                          pack2(__uint_as_float(o[c]) * f0.x, __uint_as_float(o[c + 1]) * f0.y), pack2(__uint_as_float(o[c + 2]) * f0.z, __uint_as_float(o[c + 3]) * f0.w),
                          pack2(__uint_as_float(o[c + 4]) * f1.x, __uint_as_float(o[c + 5]) * f1.y), pack2(__uint_as_float(o[c + 6]) * f1.z, __uint_as_float(o[c + 7]) * f1.w));
      }
      ptx::tc_fence_before();
      ptx::fence_proxy_async_shared();
      ptx::mbar_arrive(ot_full + 8 * d);
    }
    // ---- the 50 x 128 partial sums: feature = lane of the accumulator, 16 tokens per warp
    ok &= ptx::wait_bar(p.status, p.limit, d_full, 0, pi05::WAIT_T_FULL);
    ptx::tc_fence_after();
    uint32_t a[16];
    ptx::tmem_ld_32x16(trow + TM_D + part * 16, a);
    ptx::tmem_wait_ld();
    float* out = p.part + ((size_t)head * p.tokens + ob * TOK + part * 16) * pi05::W + group * FEAT + quad * 32 + lane;
    if (ok)
#pragma unroll
      for (int t = 0; t < 16; ++t)
        if (part * 16 + t < TOK) __stcg(out + (size_t)t * pi05::W, __uint_as_float(a[t]));
    ptx::tc_fence_before();
  }
  __syncthreads();
  if (warp == 1) {
    ptx::tc_fence_after();
    ptx::tmem_dealloc(tmem, TM_COLS);
  }
}

}  // namespace attno
