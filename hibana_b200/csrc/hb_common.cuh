// Common device helpers for the sm_100a kernel library: PTX wrappers for mbarrier, TMA, tcgen05 / TMEM,
// bounded waits that fail soft, and small numeric helpers.
//
// Every wait in this library is bounded. A wait that runs out records a code in the launch's status word,
// raises a CTA-wide abort flag in shared memory, and the kernel drains its own copies, frees its TMEM and
// returns; nothing traps and nothing spins forever.
#pragma once
#include <cstdint>
#include <cstring>
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace hb {

constexpr int kNumSms = 148;      // two dies of 74 (hardware/b200.py NUM_SMS)

// Status codes written to the status word (first writer wins; 0 = OK).
enum Status : int {
  kOk = 0,
  kTimeoutFull = 1,     // consumer gave up waiting for a TMA stage
  kTimeoutEmpty = 2,    // producer gave up waiting for a free stage
  kTimeoutAccum = 3,    // epilogue gave up waiting for the accumulator
  kTimeoutPeer = 4,     // a wait on another rank's flag ran out
  kTimeoutCounter = 5,  // a wait on an arrival counter ran out
  kBadShape = 6,
  kTimeoutDrain = 7,
  kTimeoutLowLatency = 8,   // the low-latency all-reduce never saw a peer's word
  kTimeoutGate = 9,         // a flag-gated GEMM tile never saw its source rank's rows
  kOverflow = 10,           // an expert-parallel receive buffer was too small for the rows routed to it
};

#ifndef HB_SPIN_LIMIT
#define HB_SPIN_LIMIT (1u << 22)
#endif
// Wall limit of a single wait in nanoseconds (globaltimer); the iteration limit is the backstop.
#ifndef HB_WAIT_NS
#define HB_WAIT_NS 2000000000ull
#endif

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Iteration cap of a peer wait whose wall limit is `limit_ns`: one poll of peer-visible memory takes far longer than
// 16 ns, so the nanosecond limit is what ends a failed wait and this cap only backs it up (a `limit_ns` of several
// seconds is honoured in full).
__device__ __forceinline__ unsigned long long spin_cap(unsigned long long limit_ns) { return (limit_ns >> 4) + 65536ull; }
__device__ __forceinline__ void set_status(int* status, int code) {
  if (status != nullptr) atomicCAS(status, 0, code);
}

// ---------------------------------------------------------------- checked indices (the -DHB_BOUNDS build flavour)
// Kernels that index a pool with a number they were handed (a KV slot from the block table, a recurrent-state slot,
// a token id) pass it through `index_ok`. In the normal build that is `true` and compiles away. In the bounds
// flavour the limits come from a device-side table the host fills (`hb_bounds_set`); an index outside its limit
// is recorded once (kernel, index, limit) and the caller skips the access, so a bad index shows up as a report
// the host reads with `hb_bounds_read`, never as a fault.
enum BoundsWhich : int { kBoundKvSlots = 0, kBoundStateSlots = 1, kBoundVocab = 2, kBoundRows = 3, kBoundKinds = 4 };
enum BoundsKernel : int {
  kKerRopeKvWrite = 1, kKerKvCopy = 2, kKerConvState = 3, kKerMambaScan = 4, kKerGdnScan = 5, kKerAttnDecode = 6,
  kKerAttnGeneral = 7, kKerEmbedding = 8,
};
#ifdef HB_BOUNDS
struct BoundsState {
  long long limit[kBoundKinds];
  long long index, bound;
  int hits, kernel;
};
extern __device__ BoundsState g_bounds;
__device__ __forceinline__ bool index_ok(long long idx, int which, int kernel) {
  const long long lim = g_bounds.limit[which];
  if (lim <= 0 || (idx >= 0 && idx < lim)) return true;   // limit never set: unchecked
  if (atomicAdd(&g_bounds.hits, 1) == 0) {
    g_bounds.kernel = kernel;
    g_bounds.index = idx;
    g_bounds.bound = lim;
  }
  return false;
}
#else
__device__ __forceinline__ constexpr bool index_ok(long long, int, int) { return true; }
#endif

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void fence_proxy_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// One arrival + expected transaction bytes.
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// Adds expected transaction bytes WITHOUT arriving (for barriers whose arrival count is made of thread arrivals).
__device__ __forceinline__ void mbar_add_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Non-blocking probe (try_wait may suspend the thread for a while; a role that polls two barriers uses this one).
__device__ __forceinline__ bool mbar_test_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// Bounded wait. Returns false when it gave up (either this wait ran out or another role raised `abort`).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int* status,
                                          int code) {
  // Fast path: no clock read (a wait that is about to succeed must cost nothing but the polls themselves).
#pragma unroll 1
  for (int it = 0; it < 512; ++it)
    if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = globaltimer_ns();
  for (uint32_t it = 0; it < HB_SPIN_LIMIT; ++it) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((it & 255u) == 255u) {
      if (*abort) return false;
      if (globaltimer_ns() - t0 > HB_WAIT_NS) break;
    }
  }
  *abort = 1;
  set_status(status, code);
  return false;
}

// Read-only 32-bit load that asks L2 to keep the line (evict_last): for small tables every kernel of a step reads
// again (block tables, context lengths) while gigabytes of weights and KV stream through L2 in between.
__device__ __forceinline__ int ldg_keep(const int* p) {
  int v;
  asm volatile(
      "{\n\t.reg .b64 pol;\n\t"
      "createpolicy.fractional.L2::evict_last.b64 pol, 1.0;\n\t"
      "ld.global.nc.L2::cache_hint.b32 %0, [%1], pol;\n\t}"
      : "=r"(v)
      : "l"(p));
  return v;
}

// ---------------------------------------------------------------- TMA (bulk tensor copies, never multicast)
// ---- thread-block clusters (distributed shared memory) and programmatic dependent launch
__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {   // every thread of every CTA of the cluster
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// The same meeting without ordering of memory: for CTAs that only must not leave while a peer still reads their shared memory
// (whose values the peer has used by then: in every warp an instruction that needs them, such as a store of them, has been issued;
// a load whose value nothing needs may still be under way). The release above first waits for the thread's global stores to be
// acknowledged, which nobody in the cluster reads: 1.3 us at the end of a split-K projection.
__device__ __forceinline__ void cluster_sync_exit() {
  asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_smem_addr, uint32_t cta) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_smem_addr), "r"(cta));
  return r;
}
__device__ __forceinline__ float ld_dsmem_f32(uint32_t cluster_addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(cluster_addr) : "memory");
  return v;
}
__device__ __forceinline__ float4 ld_dsmem_v4(uint32_t cluster_addr) {   // 16-byte aligned
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(cluster_addr)
               : "memory");
  return v;
}
// The grid this one depends on (programmatic stream serialisation) has completed and its writes are visible.
// A no-op when the kernel was launched without the attribute.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The same for a kernel with const __restrict__ parameters that earlier kernels of the step wrote: the compiler may move a load through
// such a pointer ahead of the wait (a promise about the whole kernel overrides the asm's clobber), so they are named here and come out
// as values that do not exist before it. Loads through them are plain ones then, not read-only ones.
template <typename P>
__device__ __forceinline__ void behind_wait(P& p) {          // (stays a global address: no generic loads)
  size_t a = __cvta_generic_to_global(p);
  asm volatile("" : "+l"(a)::"memory");
  p = static_cast<P>(__cvta_global_to_generic(a));
}
template <typename P, typename... Q>
__device__ __forceinline__ void grid_dep_wait(P& p, Q&... q) {
  grid_dep_wait();
  behind_wait(p);
  (behind_wait(q), ...);
}
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Load of what an earlier kernel of the step wrote where a const __restrict__ view or __ldg would be wanted for speed (loads that need
// not keep their order with this kernel's stores): stays behind the wait, and is a plain load, not a read-only one.
template <typename T>
__device__ __forceinline__ T ld_step(const T* p) {
  static_assert(sizeof(T) == 2 || sizeof(T) == 4 || sizeof(T) == 8 || sizeof(T) == 16, "2, 4, 8 or 16 bytes");
  T r;
  if constexpr (sizeof(T) == 2) {
    unsigned short v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
    memcpy(&r, &v, 2);
  } else if constexpr (sizeof(T) == 4) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    memcpy(&r, &v, 4);
  } else if constexpr (sizeof(T) == 8) {
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    memcpy(&r, &v, 8);
  } else {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    memcpy(&r, &v, 16);
  }
  return r;
}

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// The same with shared-memory addresses (kept in uniform registers by warp-uniform callers).
__device__ __forceinline__ void tma_load_2d(uint32_t smem_dst, const CUtensorMap* m, uint32_t bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(bar), "r"(x), "r"(y)
      : "memory");
}
__device__ __forceinline__ void bulk_load(uint32_t smem_dst, const void* gsrc, uint32_t bytes, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_dst),
      "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y,
                                            int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], "
      "[%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// Untiled bulk copy global -> shared; both addresses 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(gsrc)), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// Launch as a programmatic dependent of the kernel before it in the stream (when the library-wide switch is on,
// see hb_gemm_set_pdl): the grid may be scheduled while its predecessor drains, which hides launch latency. The rules:
//   * a CTA calls grid_dep_wait() before it reads anything that ANY kernel of the step wrote, and before it writes anything. CTAs that do
//     neither (grouped GEMM tiles without rows) may leave without it, but one CTA of every grid waits: a grid none of whose CTAs
//     does could end before its predecessor, and its dependents' waits with it.
//     Kernels may call grid_dep_launch() ahead of their own wait (norms, RoPE + KV write, attention, merges, scans, GEMMs do), so
//     when a dependent starts, kernels further back than its predecessor may still run;
//   * before the wait only what was complete long ago may be read: norm weights, static scales, a model's weights (projections fetch
//     theirs early only where the caller promises that, see hb_gemm_plain), and, where the caller promises it for a decode
//     step, its tables, older keys and recurrent states (hb_attn_decode_early, hb_state_early: attention, convolution, scans). The
//     promise holds because the step's embedding gather triggers only after its own wait: nothing behind the gather starts before
//     everything in front of it has ended. A kernel of the step that writes such data runs ahead of the gather;
//   * one exception: the one-CTA grouped GEMM (gemm.cu) reads the routing plan before its wait, to leave early. That is safe
//     because the kernel in front of it (the activation quantiser, the row gather) triggers only after its own wait, which
//     the plan kernel's end precedes, or is another grouped GEMM behind such a kernel. One that is put in between must do
//     the same.
// At level 1 only GEMMs are launched as dependents, so an early trigger matters where a GEMM follows. Level 2 is the default:
// the launch latency (0.4 us in a graph) and prologue of most kernels of a step pass behind their predecessors. Kernels that are
// launched with <<<>>> (qsa.cu, hyper.cu, ggml.cu, ssm_window.cu, ep.cu, comm.cu, attn_decode_tc.cu, the fp8 quantisers, the speculative
// ones of sample.cu) start when all in front of them have ended and let their successor start when they end.
extern "C" int hb_gemm_get_pdl(void);
extern "C" int hb_take_plain(void);     // see hb_gemm_plain
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, int cluster, size_t smem, cudaStream_t st,
                                      Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  cfg.attrs = at;
  if (hb_gemm_get_pdl() >= 2 && !hb_take_plain()) {     // level 1: GEMMs only; level 2: these kernels as well
    at[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
  }
  if (cluster > 1) {
    at[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
    at[cfg.numAttrs].val.clusterDim.x = cluster;
    at[cfg.numAttrs].val.clusterDim.y = at[cfg.numAttrs].val.clusterDim.z = 1;
    ++cfg.numAttrs;
  }
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dep(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
  return launch_dep_cluster(kern, grid, block, 1, smem, st, static_cast<Args&&>(args)...);
}

// ---------------------------------------------------------------- tcgen05 / TMEM
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_dst, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {  // whole warp
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// Arrives on the mbarrier once all tcgen05 operations issued so far by this thread have completed.
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// True in one lane of a converged warp. tcgen05 and TMA instructions take their operands from uniform registers: inside
// `if (elect_one())` of warp-uniform code the compiler knows that one lane runs and keeps descriptors and addresses there;
// under `if (lane == 0)` it moves every operand over for every instruction (see gemm.cu for what that cost).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}
// D[tmem] (+)= A[smem desc] * B[smem desc]; kind::f16 covers fp16/bf16 inputs with fp32 accumulation.
__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// The same with A from TMEM: row i in lane i, two consecutive K elements per 32-bit column (8 columns per instruction).
__device__ __forceinline__ void mma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
      "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Block-scaled FP4 (e2m1 values, ue4m3 scale per 16 elements), K = 64 per instruction.
__device__ __forceinline__ void mma_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
__device__ __forceinline__ void mma_nvf4(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate, uint32_t sfa_tmem, uint32_t sfb_tmem) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(
          d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
// Shared -> TMEM copy of one 32 x 128-bit block replicated to the four 32-lane quarters (scale factors).
__device__ __forceinline__ void tmem_cp_32x128b_x4(uint32_t taddr, uint64_t sdesc) {
  asm volatile("tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// 32 lanes x 32 consecutive fp32 columns: thread t of the warp gets columns [c, c+32) of TMEM lane base+t.
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
__device__ __forceinline__ void tmem_st_32x32(uint32_t taddr, const uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]),
      "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]),
      "r"(r[29]), "r"(r[30]), "r"(r[31]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_32x16(uint32_t taddr, const uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15};" ::"r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
      "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}

// Shared-memory matrix descriptor of a K-major operand tile stored with 128-byte swizzle: rows of 128 bytes,
// groups of 8 rows 1024 bytes apart. The tile base must be 1024-byte aligned; advancing along K inside the
// 128-byte row adds (bytes >> 4) to the low word.
__device__ __forceinline__ uint64_t make_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);  // start address
  d |= static_cast<uint64_t>(1) << 16;                  // leading byte offset (unused with swizzle)
  d |= static_cast<uint64_t>(1024 >> 4) << 32;          // stride byte offset between 8-row groups
  d |= static_cast<uint64_t>(1) << 46;                  // descriptor version (Blackwell)
  d |= static_cast<uint64_t>(2) << 61;                  // SWIZZLE_128B
  return d;
}
// MN-major operand tile with 128-byte swizzle: 64 contiguous 2-byte elements along M/N per 128-byte row,
// 8 K-rows per 1024-byte atom; atoms along M/N are `lbo_bytes` apart and atoms along K `sbo_bytes` apart.
__device__ __forceinline__ uint64_t make_desc_sw128_mn(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
  d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// Unswizzled K-major descriptor for the 32-row x 16-byte scale-factor blocks (8-row groups 128 bytes apart).
__device__ __forceinline__ uint64_t make_desc_sf(uint32_t saddr) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((saddr & 0x3FFFFu) >> 4);
  d |= static_cast<uint64_t>(128 >> 4) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  return d;
}
// Instruction descriptor, kind::f16, bf16 x bf16 -> fp32, both operands K-major unless flagged.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int m, int n, int a_mn_major = 0, int b_mn_major = 0) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a_mn_major) << 15) |
         (static_cast<uint32_t>(b_mn_major) << 16) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}
// Instruction descriptor, kind::f8f6f4 with e4m3 x e4m3 -> fp32 (operand format code 0 = E4M3), K = 32.
__host__ __device__ constexpr uint32_t make_idesc_e4m3(int m, int n) {
  return (1u << 4) | (0u << 7) | (0u << 10) | (static_cast<uint32_t>(n >> 3) << 17) |
         (static_cast<uint32_t>(m >> 4) << 24);
}
// Instruction descriptor, kind::mxf4nvf4: e2m1 x e2m1, ue4m3 scales, K = 64.
__host__ __device__ constexpr uint32_t make_idesc_nvf4(int m, int n) {
  return (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (0u << 23) |
         (static_cast<uint32_t>(m >> 4) << 24);
}

// ---------------------------------------------------------------- numeric helpers
__device__ __forceinline__ float bf16_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&t);
}
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
// e2m1 code (4 bits, sign in bit 3) of a float already divided by its block scale; round to nearest even
// on the e2m1 grid {0, .5, 1, 1.5, 2, 3, 4, 6}.
__device__ __forceinline__ uint32_t float_to_e2m1(float x) {
  const float a = fabsf(x);
  uint32_t c;
  if (a <= 0.25f) c = 0;
  else if (a < 0.75f) c = 1;
  else if (a <= 1.25f) c = 2;
  else if (a < 1.75f) c = 3;
  else if (a <= 2.5f) c = 4;
  else if (a < 3.5f) c = 5;
  else if (a <= 5.0f) c = 6;
  else c = 7;
  return c | (x < 0.f ? 8u : 0u);
}
// Two floats -> one byte of e2m1 codes (low nibble = `lo`), round to nearest even, saturating: the hardware
// conversion, same grid and tie rule as float_to_e2m1.
__device__ __forceinline__ uint32_t e2m1x2(float lo, float hi) {
  uint32_t r;
  asm("{\n\t.reg .b8 t;\n\tcvt.rn.satfinite.e2m1x2.f32 t, %1, %2;\n\tcvt.u32.u8 %0, t;\n\t}"
      : "=r"(r)
      : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ float e2m1_to_float(uint32_t c) {
  const float t[8] = {0.f, .5f, 1.f, 1.5f, 2.f, 3.f, 4.f, 6.f};
  const float v = t[c & 7];
  return (c & 8) ? -v : v;
}
// float -> e4m3 byte (saturating, round to nearest even) and back.
__device__ __forceinline__ uint32_t float_to_e4m3(float x) {
  uint32_t r;
  asm("{\n\t.reg .b16 t;\n\tcvt.rn.satfinite.e4m3x2.f32 t, %1, %2;\n\tcvt.u32.u16 %0, t;\n\t}"
      : "=r"(r)
      : "f"(0.f), "f"(x));
  return r & 0xFFu;
}
__device__ __forceinline__ float e4m3_to_float(uint32_t b) {
  uint32_t h2;
  const uint16_t in = static_cast<uint16_t>(b & 0xFFu);
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h2) : "h"(in));
  return __half2float(__ushort_as_half(static_cast<unsigned short>(h2 & 0xFFFFu)));
}

}  // namespace hb
