// Thin inline-PTX wrappers for sm_100a: mbarrier, TMA (cp.async.bulk.tensor), tcgen05 MMA / TMEM,
// proxy fences, device-scope release/acquire, warp MMA (mma.sync) and ldmatrix for the attention stage.
// No load here uses cluster multicast in any form.
#pragma once
#include <cuda_bf16.h>
#include <stdint.h>

namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// ----------------------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
// One probe of the barrier's phase with the given parity; true when that phase has completed.
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n.reg .pred P;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 P, [%1], %2;\n"
      "selp.u32 %0, 1, 0, P;\n}"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// ----------------------------------------------------------------------------- fences
// Generic-proxy writes -> visible to later async-proxy (TMA) reads of global memory.
__device__ __forceinline__ void fence_proxy_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ----------------------------------------------------------------------------- device-scope flags
__device__ __forceinline__ void red_release_add(unsigned int* addr, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* addr) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(addr) : "memory");
  return v;
}
__device__ __forceinline__ unsigned int ld_relaxed(const unsigned int* addr) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(addr) : "memory");
  return v;
}
// System scope: counters that another GPU updates or reads over NVLink.
__device__ __forceinline__ void red_release_sys_add(unsigned int* addr, unsigned int v) {
  asm volatile("red.release.sys.global.add.u32 [%0], %1;" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_sys(const unsigned int* addr) {
  unsigned int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void red_add_f32(float* addr, float v) {
  asm volatile("red.relaxed.gpu.global.add.f32 [%0], %1;" ::"l"(addr), "f"(v) : "memory");
}

// ----------------------------------------------------------------------------- TMA
// 2-D tiled load global -> this CTA's shared memory, completion on an mbarrier of this CTA.
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(c0), "r"(c1) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// 4-D tiled load (innermost coordinate first).
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1, int c2, int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3) : "memory");
}
// 5-D tiled load (innermost coordinate first).
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1, int c2, int c3,
                                            int c4) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4) : "memory");
}
__device__ __forceinline__ void tma_load_2d_hint(uint32_t dst, const void* tmap, uint32_t bar, int c0, int c1,
                                                 uint64_t policy) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint"
      " [%0], [%1, {%3, %4}], [%2], %5;"
      ::"r"(dst), "l"(tmap), "r"(bar), "r"(c0), "r"(c1), "l"(policy) : "memory");
}
__device__ __forceinline__ uint64_t policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void prefetch_tensormap(const void* tmap) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(tmap) : "memory");
}

// 2^x, approximate (one special-function instruction; denormal results flush to zero).
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 16 bytes of a read-only table into L1.
__device__ __forceinline__ void touch(const uint4* p) {
  uint32_t a, b, c, d;
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "l"(p));
}
// Two FP32 fused multiply-adds in one instruction.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long ra, rb, rc, rd;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rc) : "f"(c.x), "f"(c.y));
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(rd) : "l"(ra), "l"(rb), "l"(rc));
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}

// ----------------------------------------------------------------------------- programmatic dependent launch
// A kernel launched with programmatic stream serialisation may start while the kernel before it in the stream is still
// running; grid_dep_wait blocks until that kernel has completed and its writes are visible, grid_dep_launch lets the
// kernel after this one start early in the same way.  Both do nothing in a kernel launched the ordinary way.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// ----------------------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait_ld() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// Shared-memory matrix descriptor, K-major operand, 128-byte swizzle: rows of 128 B, 8-row groups 1024 B apart.
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3fffu)   // start address >> 4
         | (1ull << 16)                         // leading byte offset (unused with 128-B swizzle, K-major)
         | (64ull << 32)                        // stride byte offset 1024 B >> 4
         | (1ull << 46)                         // descriptor version of this architecture
         | (2ull << 61);                        // SWIZZLE_128B
}
// Instruction descriptor: BF16 x BF16 -> FP32, both operands K-major, dense.
__device__ __forceinline__ uint32_t umma_idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// The same for an operand that is MN-major (its rows run along K): 64 M / N elements per 128-byte swizzled row, eight K
// rows per 1024-byte group, the next 64 M / N elements `segment` bytes further; the instruction descriptor of a B operand
// in this layout carries UMMA_B_MN_MAJOR.
__device__ __forceinline__ uint64_t umma_smem_desc_mn(uint32_t saddr, uint32_t segment) {
  return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)(segment >> 4) << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
constexpr uint32_t UMMA_A_MN_MAJOR = 1u << 15, UMMA_B_MN_MAJOR = 1u << 16;
// One pipeline stage of the GEMM CTAs in one piece: eight K = 16 MMAs over a 128-k stage (four 32-byte steps in each
// of the two 64-k operand atoms, which lie a_atom / b_atom descriptor units apart) and the commit that frees the stage.
template <uint32_t A_ATOM, uint32_t B_ATOM>
__device__ __forceinline__ void umma_bf16_stage8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                                 uint32_t accumulate, uint32_t commit_bar) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 a1, a2, a3, a4, a5, a6, a7, b1, b2, b3, b4, b5, b6, b7;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "add.u64 a1, %1, 2;\n add.u64 a2, %1, 4;\n add.u64 a3, %1, 6;\n add.u64 a4, %1, %6;\n"
      "add.u64 a5, a4, 2;\n add.u64 a6, a4, 4;\n add.u64 a7, a4, 6;\n"
      "add.u64 b1, %2, 2;\n add.u64 b2, %2, 4;\n add.u64 b3, %2, 6;\n add.u64 b4, %2, %7;\n"
      "add.u64 b5, b4, 2;\n add.u64 b6, b4, 4;\n add.u64 b7, b4, 6;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a1, b1, %3, 1;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a2, b2, %3, 1;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a3, b3, %3, 1;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a4, b4, %3, 1;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a5, b5, %3, 1;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a6, b6, %3, 1;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a7, b7, %3, 1;\n"
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%5];\n}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(commit_bar),
        "n"((unsigned long long)A_ATOM), "n"((unsigned long long)B_ATOM) : "memory");
}
// One pipeline stage of KS 64-k blocks in one piece: 4 KS MMAs of K = 16 (32-byte steps inside the 128-byte swizzle rows of
// a block, blocks `ablock` / `bblock` descriptor units apart) and the commit that frees the stage, on one CTA or on a pair
// (whose commit arrives in both CTAs).  `alo`, `blo`: lower words of the descriptors; the upper word is the same for all.
constexpr uint32_t UMMA_DESC_HI = 64u | (1u << 14) | (2u << 29);
template <bool PAIR, int KS>
__device__ __forceinline__ void umma_bf16_stage(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t idesc, uint32_t accumulate,
                                                uint32_t commit_bar, uint32_t ablock, uint32_t bblock, uint32_t on) {
#define PI05_UMMA1(G, AO, BO, P0)                                              \
  "add.u32 al, a0, " AO ";\n add.u32 bl, b0, " BO ";\n"                        \
  "mov.b64 da, {al, %8};\n mov.b64 db, {bl, %8};\n"                            \
  "@q tcgen05.mma.cta_group::" G ".kind::f16 [%0], da, db, %3, " P0 ";\n"
#define PI05_UMMA4(G, P0) PI05_UMMA1(G, "0", "0", P0) PI05_UMMA1(G, "2", "2", "t") PI05_UMMA1(G, "4", "4", "t") PI05_UMMA1(G, "6", "6", "t")
#define PI05_UMMA_HEAD "{\n.reg .pred p, q, t;\n.reg .b32 a0, b0, al, bl;\n.reg .b64 da, db;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %9, 0;\n" \
                       "setp.eq.b32 t, 0, 0;\nmov.b32 a0, %1;\nmov.b32 b0, %2;\n"
#define PI05_UMMA_NEXT "add.u32 a0, a0, %6;\n add.u32 b0, b0, %7;\n"
#define PI05_UMMA_COMMIT1 "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%5];\n}"
#define PI05_UMMA_COMMIT2 ".reg .b16 m;\nmov.b16 m, 3;\n@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%5], m;\n}"
#define PI05_UMMA_ARGS ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "r"(commit_bar), "r"(ablock), "r"(bblock), "n"(UMMA_DESC_HI), "r"(on) : "memory"
  if constexpr (KS == 4) {
    static_assert(!PAIR, "four blocks a stage: single CTAs");
    asm volatile(PI05_UMMA_HEAD PI05_UMMA4("1", "p") PI05_UMMA_NEXT PI05_UMMA4("1", "t") PI05_UMMA_NEXT PI05_UMMA4("1", "t") PI05_UMMA_NEXT
                 PI05_UMMA4("1", "t") PI05_UMMA_COMMIT1 PI05_UMMA_ARGS);
  } else if constexpr (PAIR && KS == 1)
    asm volatile(PI05_UMMA_HEAD PI05_UMMA4("2", "p") PI05_UMMA_COMMIT2 PI05_UMMA_ARGS);
  else if constexpr (PAIR)
    asm volatile(PI05_UMMA_HEAD PI05_UMMA4("2", "p") PI05_UMMA_NEXT PI05_UMMA4("2", "t") PI05_UMMA_COMMIT2 PI05_UMMA_ARGS);
  else if constexpr (KS == 1)
    asm volatile(PI05_UMMA_HEAD PI05_UMMA4("1", "p") PI05_UMMA_COMMIT1 PI05_UMMA_ARGS);
  else
    asm volatile(PI05_UMMA_HEAD PI05_UMMA4("1", "p") PI05_UMMA_NEXT PI05_UMMA4("1", "t") PI05_UMMA_COMMIT1 PI05_UMMA_ARGS);
#undef PI05_UMMA4
#undef PI05_UMMA1
#undef PI05_UMMA_HEAD
#undef PI05_UMMA_NEXT
#undef PI05_UMMA_COMMIT1
#undef PI05_UMMA_COMMIT2
#undef PI05_UMMA_ARGS
}
// Four K = 16 MMAs on one CTA, ASTEP / BSTEP descriptor units (16 bytes) apart, by the lane for which `on` is set; the rest as above.
template <int ASTEP, int BSTEP>
__device__ __forceinline__ void umma_bf16_k64(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t idesc, uint32_t accumulate, uint32_t on) {
#define PI05_UMMA1(P0) "mov.b64 da, {al, %5};\n mov.b64 db, {bl, %5};\n@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, " P0 ";\n"
#define PI05_UMMA_STEP "add.u32 al, al, %7;\n add.u32 bl, bl, %8;\n"
  asm volatile("{\n.reg .pred p, q, t;\n.reg .b32 al, bl;\n.reg .b64 da, db;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %6, 0;\nsetp.eq.b32 t, 0, 0;\n"
               "mov.b32 al, %1;\nmov.b32 bl, %2;\n" PI05_UMMA1("p") PI05_UMMA_STEP PI05_UMMA1("t") PI05_UMMA_STEP PI05_UMMA1("t") PI05_UMMA_STEP
               PI05_UMMA1("t") "}"
               ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "n"(UMMA_DESC_HI), "r"(on), "n"(ASTEP), "n"(BSTEP) : "memory");
#undef PI05_UMMA1
#undef PI05_UMMA_STEP
}
// One of them.
__device__ __forceinline__ void umma_bf16_k16(uint32_t d_tmem, uint32_t alo, uint32_t blo, uint32_t idesc, uint32_t accumulate, uint32_t on) {
  asm volatile("{\n.reg .pred p, q;\n.reg .b64 da, db;\nsetp.ne.b32 p, %4, 0;\nsetp.ne.b32 q, %6, 0;\nmov.b64 da, {%1, %5};\n mov.b64 db, {%2, %5};\n"
               "@q tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}"
               ::"r"(d_tmem), "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "n"(UMMA_DESC_HI), "r"(on) : "memory");
}
// One lane of a converged warp (always the same one), for instructions that a single thread must issue while the
// loop around them stays warp-uniform.
__device__ __forceinline__ bool elect_one() {
  uint32_t leader;
  asm volatile("{\n.reg .pred P;\n.reg .b32 r;\nelect.sync r|P, 0xffffffff;\nselp.u32 %0, 1, 0, P;\n}" : "=r"(leader));
  return leader != 0;
}
// Arrive once on an mbarrier of this CTA when every tcgen05 op issued so far by this thread has completed.
__device__ __forceinline__ void umma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns: thread i of the warp gets lane (base_lane + i), columns col..col+31.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}

// The store that mirrors tmem_ld_32x8, and the wait that orders it before later tcgen05 loads of the same thread.
__device__ __forceinline__ void tmem_st_32x8(uint32_t taddr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr) : "memory");
}

// ----------------------------------------------------------------------------- CTA pairs (cta_group::2)
// Two CTAs of a cluster (ranks 2 i and 2 i + 1) share one MMA: M = 256 rows, each CTA holding its 128 rows of A, its half
// of B's rows and its 128 lanes of the accumulator at the same shared-memory / TMEM offsets; one thread of the even CTA
// issues.  Allocation, release and deallocation of TMEM are executed by the same warp of both CTAs.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The shared::cluster address of `saddr` (an address in this CTA's shared memory) in the CTA of rank `rank`.
__device__ __forceinline__ uint32_t map_to_rank(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_slot), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Tiled load into this CTA's shared memory whose bytes count on an mbarrier of the pair's even CTA (`cluster_bar`).
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const void* tmap, uint32_t cluster_bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(tmap), "r"(cluster_bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// Arrive on the barrier at this offset in both CTAs of the pair (`mask`: their ranks in the cluster) when every tcgen05 op issued
// so far has completed.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, unsigned short mask) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(bar), "h"(mask) : "memory");
}


// Bounded wait on an mbarrier of this CTA, by a whole converged warp: a wait that runs out records (kind, block) in the
// status words once.  The vote keeps the result warp-uniform and the warp converged, which
// the .aligned tcgen05 instructions behind a wait rely on.  The waiting itself is one function per kernel: the code of a
// kernel that runs for a few microseconds is fetched once, and what it does not repeat it pays for.
//   The time counts from the end of the kernel before this one, which every wait of a CTA is behind, and is cut to SETTLED (1 ms) where
// another wait has run out.  `limit` is not below SETTLED, and a CTA's longest healthy wait is some 10 us, so a wait only gives up where
// nothing in the CTA has moved for that long: no other warp of it has copies or MMAs in flight or is about to issue any while it
// frees its tensor memory and leaves.  (A mark or a vote at the end of every role would see to that as well, but costs 2 to 4% of a chunk.)
constexpr long long SETTLED = 2000000;
static __device__ __noinline__ bool wait_bar_slow(unsigned int* status, long long limit, uint32_t bar, uint32_t parity, int kind) {
  grid_dep_wait();
  const long long t0 = clock64();
  for (unsigned i = 0;; ++i) {
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    if ((i & 63u) == 63u) {
      bool stop = ld_relaxed(status) != 0u && clock64() - t0 > SETTLED;
      if (!stop && clock64() - t0 > limit) {
        if (atomicCAS(status, 0u, (unsigned)kind) == 0u) status[1] = blockIdx.x << 16;
        stop = true;
      }
      if (__any_sync(0xffffffffu, stop)) break;
    }
  }
  // what the CTA may still have in flight finishes within microseconds
  const long long t1 = clock64();
  while (clock64() - t1 < 200000) __nanosleep(1000);
  return false;
}
__device__ __forceinline__ bool wait_bar(unsigned int* status, long long limit, uint32_t bar, uint32_t parity, int kind) {
  if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
  return wait_bar_slow(status, limit, bar, parity, kind);
}

// ----------------------------------------------------------------------------- warp MMA + ldmatrix (attention)
__device__ __forceinline__ void ldmatrix_x4(uint32_t saddr, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(saddr) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t saddr, uint32_t& a, uint32_t& b, uint32_t& c, uint32_t& d) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(a), "=r"(b), "=r"(c), "=r"(d) : "r"(saddr) : "memory");
}
// D(16x8, f32) += A(16x16, bf16, row) * B(16x8, bf16, col)
__device__ __forceinline__ void mma_16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                          uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16-byte store to a shared-memory address given in the shared state space (lets the compiler keep global loads
// of later iterations ahead of it: the two spaces cannot alias).
__device__ __forceinline__ void st_shared_v4(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d));
}

__device__ __forceinline__ uint4 ld_shared_v4(uint32_t saddr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(saddr) : "memory");
  return v;
}
// 16 bytes from each of four places through L2, all on their way before the first is used.
__device__ __forceinline__ void ld_l2_f4x4(float4 (&v)[4], const float4* p, size_t step) {
  asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%16];\n ld.global.cg.v4.f32 {%4, %5, %6, %7}, [%17];\n"
               "ld.global.cg.v4.f32 {%8, %9, %10, %11}, [%18];\n ld.global.cg.v4.f32 {%12, %13, %14, %15}, [%19];"
               : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[0].z), "=f"(v[0].w), "=f"(v[1].x), "=f"(v[1].y), "=f"(v[1].z), "=f"(v[1].w),
                 "=f"(v[2].x), "=f"(v[2].y), "=f"(v[2].z), "=f"(v[2].w), "=f"(v[3].x), "=f"(v[3].y), "=f"(v[3].z), "=f"(v[3].w)
               : "l"(p), "l"(p + step), "l"(p + 2 * step), "l"(p + 3 * step) : "memory");
}

__device__ __forceinline__ void named_bar_sync(int id, int nthreads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int nthreads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(nthreads) : "memory");
}
// The same barrier with the disjunction of a predicate over its threads.
__device__ __forceinline__ bool named_bar_or(int id, int nthreads, bool pred) {
  int r;
  asm volatile("{\n.reg .pred p, q;\nsetp.ne.u32 p, %3, 0;\nbarrier.cta.red.or.pred q, %1, %2, p;\nselp.u32 %0, 1, 0, q;\n}"
               : "=r"(r) : "r"(id), "r"(nthreads), "r"(pred ? 1 : 0) : "memory");
  return r != 0;
}
// 16 bytes from global to shared memory past L1, as part of the thread's current group; the wait returns when all but the last N groups are there.
__device__ __forceinline__ void copy_async_16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// Streaming 16-byte load that does not allocate in L1.
__device__ __forceinline__ float4 ldg_stream_f4(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}

}  // namespace ptx
