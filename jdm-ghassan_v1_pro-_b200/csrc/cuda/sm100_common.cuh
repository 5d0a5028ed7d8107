// Thin inline-PTX layer for Blackwell (sm_100a): mbarrier, TMA (cp.async.bulk.tensor),
// tcgen05 (alloc / mma / commit / ld / fences) and shared-memory matrix descriptors.
// Every wait in this file is bounded, by polls (mbar_wait: the caller gets `false` and is expected to
// record an error code and drain) or by cycles (wait_or_report, wait_or_leave: they record it themselves).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>

namespace gb {

// status codes written to the device-side error word (named for the user in ops/_lib.py: STATUS_NAMES)
enum : int {
  ST_OK = 0,
  ST_TIMEOUT_FULL = 101,      // consumer never saw the TMA bytes land
  ST_TIMEOUT_EMPTY = 102,     // producer never got a free smem stage
  ST_TIMEOUT_TMEM_FULL = 103, // epilogue never saw the accumulator commit
  ST_TIMEOUT_TMEM_EMPTY = 104,// MMA warp never got an accumulator buffer back
  ST_TIMEOUT_PEER = 201,      // a flag owned by another rank never changed
  ST_BAD_ARGUMENT = 301,
  ST_EP_OVERFLOW = 302,       // expert parallelism: more rows routed to this rank's experts than its buffers hold
  ST_TIMEOUT_AUX = 105,       // an epilogue warp never saw the bytes of its own TMA load
};

}  // namespace gb

// Result of the launch just issued, for the C launchers: 0, or -(1000 + cudaError_t) so that the caller can name it.
static inline int gb_launch_rc() {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(1000 + static_cast<int>(e));
}

// Programmatic dependent launch for chains of short kernels (the decode step): the next kernel's blocks are set up
// while this one drains.  A kernel launched through GB_PDL_LAUNCH must call gb::pdl_wait() before it writes global memory and
// before it reads anything that the launch ahead of it may write; until then nothing that launch wrote is guaranteed
// visible.  What only earlier launches write may be read before: a launch starts once every block of the one ahead is past its own
// wait.  GB200_NO_PDL=1 turns the attribute off.
#include <cstdlib>
#include "smem_limit.h"
static inline cudaLaunchConfig_t gb_pdl_config(dim3 grid, dim3 block, size_t smem, cudaStream_t st, cudaLaunchAttribute* attr) {
  static const int enabled = []() { const char* e = std::getenv("GB200_NO_PDL"); return (e && e[0] == '1') ? 0 : 1; }();
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  attr->id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr->val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = enabled ? 1 : 0;
  return cfg;
}
#define GB_PDL_LAUNCH(kernel, grid, block, st, ...)                                   \
  do {                                                                                \
    cudaLaunchAttribute gb_attr_;                                                     \
    cudaLaunchConfig_t gb_cfg_ = gb_pdl_config(grid, block, 0, st, &gb_attr_);        \
    (void)cudaLaunchKernelEx(&gb_cfg_, kernel, __VA_ARGS__);                          \
  } while (0)
// The same with dynamic shared memory, opting in to more than 48 KB of it.  (Where that is refused, so is the launch, which says why.)
#define GB_PDL_LAUNCH_SMEM(kernel, grid, block, smem, st, ...)                                                       \
  do {                                                                                                               \
    cudaLaunchAttribute gb_attr_;                                                                                    \
    cudaLaunchConfig_t gb_cfg_ = gb_pdl_config(grid, block, smem, st, &gb_attr_);                                    \
    (void)gb_allow_smem(reinterpret_cast<const void*>(kernel), smem);                                                \
    (void)cudaLaunchKernelEx(&gb_cfg_, kernel, __VA_ARGS__);                                                         \
  } while (0)

namespace gb {

// Wait until the kernels before this one have finished and their writes are visible, then let the kernel after it begin its own set-up.  The first
// statement of every kernel that GB_PDL_LAUNCH starts, but for those that first ask for constants (weights in gemm_skinny_sm100.cu, layers_gemv.cu,
// layers_latent.cu, the norms of decode.cu and layers_common.cu, the offsets in piece_add_kernel) or, where the caller says that the launch ahead leaves them
// alone (`early`, `b_static`), for state and cache rows of earlier steps (token attention, the Mamba step): the headers say which arguments the
// launch ahead must not write.  A kernel with tensor memory allocates it first: were the next kernel let in before, its blocks could take the columns
// and then wait for this kernel, which waits for them.
__device__ __forceinline__ void pdl_wait() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// ----------------------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void fence_barrier_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Polls a few times inside one instruction sequence, so that callers' loops keep one straight path.
__device__ __forceinline__ bool mbar_try_wait_some(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred P1, P2;\n\t.reg .u32 n;\n\t"
      "mov.u32 n, 64;\n\t"
      "L_POLL_%=:\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\t"
      "@P1 bra L_DONE_%=;\n\t"
      "sub.u32 n, n, 1;\n\t"
      "setp.ne.u32 P2, n, 0;\n\t"
      "@P2 bra L_POLL_%=;\n\t"
      "L_DONE_%=:\n\t"
      "selp.b32 %0, 1, 0, P1;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// One lane of a converged warp.
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t on;
  asm volatile("{\n\t.reg .pred P;\n\telect.sync _|P, 0xffffffff;\n\tselp.b32 %0, 1, 0, P;\n\t}" : "=r"(on));
  return on;
}
#ifndef GB_SPIN_LIMIT
#define GB_SPIN_LIMIT (1u << 24)
#endif
// Bounded wait: true when the phase completed, false when the poll budget ran out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  for (uint32_t i = 0; i < GB_SPIN_LIMIT; ++i) {
    if (mbar_try_wait(bar, parity)) return true;
  }
  return false;
}

// Bounded wait shared by all roles of a CTA: gives up once another role has given up (looked at before anything else), or after
// ~2 s, and reports that in the status word, which says that the results are void.
static constexpr long long WAIT_CYCLES = 4000000000LL;      // ~2 s
__device__ __forceinline__ bool wait_poll(uint64_t* bar, uint32_t parity, int* status, int code, volatile int* abort_flag, long long limit) {
  const long long t0 = clock64();
  while (!*abort_flag) {
#pragma unroll 1
    for (int i = 0; i < 256; ++i)
      if (mbar_try_wait(bar, parity)) return true;
    if (clock64() - t0 > limit) {
      atomicCAS(status, 0, code);
      *abort_flag = 1;
    }
  }
  return false;
}
static __device__ __noinline__ void wait_or_report_slow(uint64_t* bar, uint32_t parity, int* status, int code, volatile int* abort_flag,
                                                        long long limit) {
  (void)wait_poll(bar, parity, status, code, abort_flag, limit);
}
static __device__ __noinline__ void wait_or_leave_slow(uint64_t* bar, uint32_t parity, int* status, int code, volatile int* abort_flag,
                                                       long long limit) {
  if (!wait_poll(bar, parity, status, code, abort_flag, limit)) asm volatile("exit;");
}
// For MMA issuers and epilogues: after a failure the loops go on, on whatever the buffers hold, and no later wait of the CTA takes longer
// than its first polls.  A loop that left on a wait's result would no longer be provably uniform over the warp, and the operands
// of the MMAs would lose their uniform registers.  What still runs stays in the CTA's own buffers and barriers.
__device__ __forceinline__ void wait_or_report(uint64_t* bar, uint32_t parity, int* status, int code, volatile int* abort_flag,
                                               long long limit = WAIT_CYCLES) {
  if (!mbar_try_wait_some(bar, parity)) wait_or_report_slow(bar, parity, status, code, abort_flag, limit);
}
// For the warps that load: after a failure the thread ends, so that nothing more is expected of a barrier or loaded into a stage that may
// be in use; the barriers of the block and the cluster wait for the threads that are left.  Not for a warp that holds anything
// (tensor memory).  Clearing `on` instead, which makes it an ordinary predicate, cost the two-CTA GEMM 2 to 6 %.
__device__ __forceinline__ void wait_or_leave(uint64_t* bar, uint32_t parity, int* status, int code, volatile int* abort_flag,
                                              long long limit = WAIT_CYCLES) {
  if (!mbar_try_wait_some(bar, parity)) wait_or_leave_slow(bar, parity, status, code, abort_flag, limit);
}

// ----------------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_load_2d(const CUtensorMap* map, uint64_t* bar, void* dst, int c0, int c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(const CUtensorMap* map, uint64_t* bar, void* dst, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
      : "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

// ----------------------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
               : "memory");
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
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 32 lanes x 32 columns of 32-bit cells: thread t of the warp receives lane (base_lane + t),
// columns [col, col+32).  `taddr` = (lane << 16) | column.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// store 32 lanes x 16 columns (thread t -> lane base+t)
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      :
      : "r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// ----------------------------------------------------------------------------- CTA pairs (cta_group::2)
// Two CTAs of a cluster of two drive one 256-row MMA: each holds 128 rows of A, half of B and 128 accumulator lanes.
// CTA 0 of the pair issues the MMAs; every barrier that both CTAs signal lives in CTA 0 and is addressed through
// mapa.  None of the loads below is a multicast: each CTA fetches its own operand halves.
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_nctaid_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
// shared::cluster address of `addr` (a shared::cta address of this CTA) as seen in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t mapa_shared(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// arrive on a barrier given by its shared::cluster address (possibly in the other CTA of the pair)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// ----------------------------------------------------------------------------- issue from a warp that runs converged
// Every lane passes the same operands and the lane with `on` != 0 issues; `on` comes from elect_one().  The operands then stay
// in uniform registers, which is where these instructions want them.  Measured in the two-CTA GEMM, cycles per 64-deep k-block
// (four MMAs and a commit; the MMAs themselves take 512 at 256 columns and 256 at 128): 747 issued from an `if (lane == 0)`
// branch, whatever the tile's width; 548 with the whole warp in the loop and `on = lane == 0`; 512 and 444 with elect_one().
// The forms of one CTA are plain; *_pair_on are cta_group::2 (loads count their bytes on a barrier that may be the other CTA's;
// the commit arrives at this shared-memory offset in every CTA of the mask, a signal, no data is copied).
// D[tmem] (+)= A[smem desc] * B[smem desc]; fp16/bf16 operands, fp32 accumulate.
__device__ __forceinline__ void umma_f16_on(uint32_t on, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                            uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}
// The same with the A operand in tensor memory.
__device__ __forceinline__ void umma_f16_ts_on(uint32_t on, uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc,
                                               uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}
// All previously issued MMAs of the issuing lane arrive on `bar` when they have completed.
__device__ __forceinline__ void umma_commit_on(uint32_t on, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}"
      :
      : "r"(smem_u32(bar)), "r"(on)
      : "memory");
}
__device__ __forceinline__ void umma_f16_pair_on(uint32_t on, uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                                 uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      :
      : "r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate), "r"(on)
      : "memory");
}
__device__ __forceinline__ void umma_commit_pair_on(uint32_t on, uint64_t* bar, uint16_t cta_mask) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %2, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
      :
      : "r"(smem_u32(bar)), "h"(cta_mask), "r"(on)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx_on(uint32_t on, uint64_t* bar, uint32_t bytes) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %2, 0;\n\t"
      "@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(smem_u32(bar)),
      "r"(bytes), "r"(on)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_on(uint32_t on, const CUtensorMap* map, uint64_t* bar, void* dst, int c0, int c1) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(on)
      : "memory");
}
__device__ __forceinline__ void tma_load_2d_pair_on(uint32_t on, const CUtensorMap* map, uint32_t bar_cluster_addr, void* dst,
                                                    int c0, int c1) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(on)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d_pair_on(uint32_t on, const CUtensorMap* map, uint32_t bar_cluster_addr, void* dst,
                                                    int c0, int c1, int c2) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %6, 0;\n\t"
      "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
      :
      : "r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(c0), "r"(c1), "r"(c2), "r"(on)
      : "memory");
}

// ----------------------------------------------------------------------------- TMA stores (shared -> global)
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* src, int c0, int c1, int c2) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
// global[tile] += shared[tile], element type from the tensor map (fp32 here)
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, const void* src, int c0, int c1, int c2) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// at most N of this thread's bulk groups may still be reading their shared-memory source
template <int N> __device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N> __device__ __forceinline__ void bulk_wait() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}

// ------------------------------------------------------------------ descriptors
// Shared-memory matrix descriptor (tcgen05 / "UMMA"), 128-byte swizzle:
//   bits [0,14)  start address >> 4        bits [16,30) leading byte offset >> 4
//   bits [32,46) stride byte offset >> 4   bits [46,48) version = 1
//   bits [61,64) layout type (2 = SWIZZLE_128B)
__device__ __forceinline__ uint64_t make_smem_desc_sw128(uint32_t smem_addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= uint64_t((smem_addr >> 4) & 0x3FFF);
  d |= uint64_t((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= uint64_t((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(2) << 61;
  return d;
}
// Instruction descriptor for kind::f16 with fp32 accumulation.
//   fmt: 0 = fp16 operands, 1 = bf16.  *_mn_major: 0 = K-major operand, 1 = MN-major.
__host__ __device__ inline uint32_t make_idesc_f16(int fmt, int a_mn_major, int b_mn_major, int M, int N) {
  uint32_t d = 0;
  d |= 1u << 4;                       // D format = F32
  d |= uint32_t(fmt) << 7;            // A format
  d |= uint32_t(fmt) << 10;           // B format
  d |= uint32_t(a_mn_major) << 15;
  d |= uint32_t(b_mn_major) << 16;
  d |= uint32_t(N >> 3) << 17;
  d |= uint32_t(M >> 4) << 24;
  return d;
}

// ------------------------------------------------------------------ small helpers
template <typename T> struct Cvt;
template <> struct Cvt<__half> {
  static __device__ __forceinline__ float to_f(__half v) { return __half2float(v); }
  static __device__ __forceinline__ __half from_f(float v) { return __float2half_rn(v); }
  static __device__ __forceinline__ uint32_t pack2(float a, float b) {
    __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ float2 unpack2(uint32_t u) {
    return __half22float2(*reinterpret_cast<__half2*>(&u));
  }
};
template <> struct Cvt<__nv_bfloat16> {
  static __device__ __forceinline__ float to_f(__nv_bfloat16 v) { return __bfloat162float(v); }
  static __device__ __forceinline__ __nv_bfloat16 from_f(float v) { return __float2bfloat16_rn(v); }
  static __device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
  }
  static __device__ __forceinline__ float2 unpack2(uint32_t u) {
    return __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&u));
  }
};
template <> struct Cvt<float> {
  static __device__ __forceinline__ float to_f(float v) { return v; }
  static __device__ __forceinline__ float from_f(float v) { return v; }
};

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace gb

// ------------------------------------------------------------------ host-side TMA map encoding
// cuTensorMapEncodeTiled is fetched through the runtime so the library does not link libcuda.
typedef CUresult (*gb_encode_tiled_fn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                       const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                                       CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                                       CUtensorMapFloatOOBfill);
gb_encode_tiled_fn gb_get_encode_tiled();
// 2-D row-major 16-bit matrix [rows, cols] with leading dimension `ld` (elements); box = [box_rows, box_cols],
// 128-byte swizzle when box_cols*2 == 128.  Returns 0 on success.
int gb_make_tmap_2d_16b(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                        uint32_t box_rows, uint32_t box_cols, int is_bf16);
// 3-D view [groups][rows][cols] of an output (or epilogue input) matrix for TMA stores / loads of 128-byte-wide boxes:
// dtype 0 fp16, 1 bf16, 2 fp32; row pitch `ld` and group pitch `group_stride` in elements; box = [1, box_rows,
// 128 / element size] with the 128-byte swizzle.  Returns 0 on success.
// MN-major 16-bit operand stored [k_rows, mn] (mn a multiple of 64) viewed as [mn / 64][k_rows][64]: one box
// [chunks, box_k, 64] lands as `chunks` consecutive 64-wide, 128-byte-swizzled column blocks.  Returns 0 on success.
int gb_make_tmap_mn_chunks(CUtensorMap* out, const void* base, uint64_t k_rows, uint64_t mn, uint64_t ld, uint32_t box_k,
                           uint32_t chunks, int is_bf16);
int gb_make_tmap_3d_box128(CUtensorMap* out, const void* base, int dtype, uint64_t cols, uint64_t rows, uint64_t groups,
                           uint64_t ld, uint64_t group_stride, uint32_t box_rows);
