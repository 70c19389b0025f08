// Prefill-sized NVFP4 GEMM for sm_100a on SM pairs: D[m, n] = A[m, K] * B[n, K]^T, tokens on the A side.
//
// Two CTAs of a cluster share one 256 x 256 output tile (tcgen05 cta_group::2, M = 256): each stages its own 128 rows
// of A and HALF of B, and the leader's MMA reads both shared memories. A 128 x 256 tile on one SM has to read
// 12 KB and land 13.5 KB of shared memory per 128-cycle FP4 instruction, more than the 128 bytes per cycle an SM has;
// the pair reads 8 KB and lands 9.5 KB per SM and instruction, which is what lets the tensor cores run at FP4 rate.
//
// The kernel is persistent: a cluster walks the work units u = cluster, cluster + clusters, ... . Two accumulators
// alternate, so that the epilogue of a unit runs under the MMAs of the next one. 2 x 256 columns leave no TMEM for the
// scale factors (16 + 32 columns): the second accumulator starts at column 208 and shares 48 columns with the
// first. The epilogue therefore reads the shared columns first (64 of them, into registers) and releases them at
// once; the tensor cores wait for that part only.
//
// Bound by what L2 delivers to the SMs (12.5 TB/s measured with the MMAs taken out: 39 KB per CTA and K tile), then by the
// last wave. Against one CTA per 128 x 256 tile, K 5120 unless noted: 2048 x 34816 with SiLU-mul + requantisation 362 ->
// 170 us (4.3 PFLOP/s), 2048 x 7168 93 -> 48, 2048 x 5120 (K 17408) 176 -> 87, 4096 x 34816 690 -> 305 (4.8 PFLOP/s),
// 300 x 5120 (K 17408) 60 -> 34. The sums run in the same order: results are the same bit for bit.
//
// The last wave of full tiles is cut into narrower units (128 or 64 columns) when that shortens it: 2048 x 5120 makes
// 160 tiles for 74 clusters, 12 of which would otherwise keep the whole chip for a third full wave.
#include <algorithm>

#include "gemm.cuh"

#include "hb_common.cuh"
#include "rownorm.cuh"

extern "C" int hb_gemm_get_pdl(void);

namespace hb {
namespace {

constexpr int PAIR_M = 256;                   // rows of a unit (128 per CTA)
constexpr int PAIR_N = 256;                   // columns of a full unit
constexpr int THREADS = 192;                  // producer warp, MMA warp, four epilogue warps
constexpr int STAGES = 5;
constexpr int A_BYTES = 128 * 128;            // 128 rows x 256 packed e2m1
constexpr int B_BYTES = 128 * 128;            // this CTA's half of the 256 columns
constexpr int SFA_BYTES = 2048;               // one 128-row block x 4 K atoms
constexpr int SFB_BYTES = 4096;               // two 128-column blocks x 4 K atoms (each CTA holds all columns' scales)
constexpr int STAGE_BYTES = A_BYTES + B_BYTES + SFA_BYTES + SFB_BYTES;
constexpr int ROW_PITCH = 144;                // staged output row: 128 bytes + 16 (conflict-free 16-byte accesses)
constexpr int Q_PITCH = 80;                   // staged requantised row: 64 packed bytes, 8 scale bytes, padding
constexpr int STAGING_BYTES = 4 * 32 * ROW_PITCH;
constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + STAGING_BYTES + 256;
constexpr int ACC1_COL = 208;                 // first column of the second accumulator
constexpr int SFA_COL = 464;                  // 4 K atoms x 4 columns
constexpr int SFB_COL = 480;                  // 4 K atoms x 8 columns
static_assert(ACC1_COL + PAIR_N == SFA_COL && SFB_COL + 32 == 512, "TMEM map");

struct PairParams {
  int m, n, k_tiles;
  int m_tiles, full_units, sub_width, units;   // units past full_units are sub_width columns wide
  __nv_bfloat16* out;
  long long ldo;
  const __nv_bfloat16* residual;
  float alpha;
  const float* alpha_ptr;
  int early_launch;
  uint8_t* q_out;
  uint8_t* q_sf;
  const float* q_gscale;
  int q_ka;
  long long q_ld;
  int* status;
};

struct Unit {
  int m0, n0, width;
  bool live;     // a narrow unit of a ragged last tile can lie past the last column
};
__device__ __forceinline__ Unit unit_at(const PairParams& p, int u) {
  Unit x;
  int t = u, sub = 0;
  x.width = PAIR_N;
  if (u >= p.full_units) {
    const int per = PAIR_N / p.sub_width;
    t = p.full_units + (u - p.full_units) / per;
    sub = (u - p.full_units) % per;
    x.width = p.sub_width;
  }
  // rows fastest: the row tiles that read the same weights run side by side, so the weights leave HBM once
  x.m0 = (t % p.m_tiles) * PAIR_M;
  x.n0 = (t / p.m_tiles) * PAIR_N + sub * x.width;
  x.live = x.n0 < p.n;
  return x;
}

// ---- the cta_group::2 forms of the wrappers in hb_common.cuh
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_dst, uint32_t ncols) {   // one whole warp of each CTA
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_dst)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// Tile load into this CTA's shared memory whose bytes are counted on the leader's barrier (a cluster address).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t smem_dst, const CUtensorMap* m, uint32_t leader_bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], "
      "[%2];" ::"r"(smem_dst),
      "l"(reinterpret_cast<uint64_t>(m)), "r"(leader_bar), "r"(x), "r"(y)
      : "memory");
}
// Arrives on the barrier at this offset of both CTAs once the pair's tcgen05 operations issued so far are done.
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"(static_cast<uint16_t>(3))
      : "memory");
}
__device__ __forceinline__ void tmem_cp_32x128b_x4_pair(uint32_t taddr, uint64_t sdesc) {   // both CTAs, own operands
  asm volatile("tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;" ::"r"(taddr), "l"(sdesc) : "memory");
}
__device__ __forceinline__ void mma_nvf4_pair(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                              uint32_t accumulate, uint32_t sfa_tmem, uint32_t sfb_tmem) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::mxf4nvf4.block_scale.block16 [%0], %1, %2, %3, [%5], [%6], p;\n\t}" ::"r"(
          d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(sfa_tmem), "r"(sfb_tmem)
      : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}

__device__ __forceinline__ float silu_fast(float x) { return __fdividef(x, 1.f + __expf(-x)); }

// One epilogue warp's 32 rows of a unit. `acc` is the accumulator's address for the warp's lanes, `release` the leader's
// acc_free barrier. Steps of 64 columns; the first step covers the columns the two accumulators share.
template <int EPI>
__device__ __forceinline__ void epilogue_unit(const PairParams& p, const Unit& x, int buf, uint32_t acc, int row0,
                                              uint8_t* staging, float alpha, float q_inv_gs, uint32_t release, int lane) {
  const int steps = x.width / 64;
  uint8_t* my_row = staging + lane * (EPI == kEpiSiluMulQuant ? Q_PITCH : ROW_PITCH);
#pragma unroll 1
  for (int j = 0; j < steps; ++j) {
    const int s = buf == 0 ? steps - 1 - j : j;
    uint32_t r[2][32];
    tmem_ld_32x32(acc + s * 64, r[0]);
    tmem_ld_32x32(acc + s * 64 + 32, r[1]);
    tmem_ld_wait();
    if (j == 0) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(release);
    }
    if constexpr (EPI == kEpiSiluMulQuant) {
      // 32 accumulator columns are 16 gate / up pairs: one 16-feature NVFP4 group of the thread's token. Same
      // arithmetic in the same order as the stand-alone quantiser.
      uint2 packed[2];
      uint32_t sf[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float y[16];
#pragma unroll
        for (int t = 0; t < 16; ++t)
          y[t] = __bfloat162float(__float2bfloat16(silu_fast(__uint_as_float(r[h][2 * t]) * alpha) *
                                                   (__uint_as_float(r[h][2 * t + 1]) * alpha)));
        sf[h] = quant16(y, q_inv_gs, &packed[h]);
      }
      *reinterpret_cast<uint4*>(my_row + s * 16) = make_uint4(packed[0].x, packed[0].y, packed[1].x, packed[1].y);
      *reinterpret_cast<uint16_t*>(my_row + 64 + s * 2) = static_cast<uint16_t>(sf[0] | (sf[1] << 8));
    } else if constexpr (EPI == kEpiSiluMul) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t w[8];
#pragma unroll
        for (int t = 0; t < 8; ++t)
          w[t] = pack_bf16(
              silu_fast(__uint_as_float(r[h][4 * t]) * alpha) * (__uint_as_float(r[h][4 * t + 1]) * alpha),
              silu_fast(__uint_as_float(r[h][4 * t + 2]) * alpha) * (__uint_as_float(r[h][4 * t + 3]) * alpha));
        *reinterpret_cast<uint4*>(my_row + h * 32) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(my_row + h * 32 + 16) = make_uint4(w[4], w[5], w[6], w[7]);
      }
    } else {
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i)
            w[i] = pack_bf16(__uint_as_float(r[h][8 * t + 2 * i]) * alpha, __uint_as_float(r[h][8 * t + 2 * i + 1]) * alpha);
          *reinterpret_cast<uint4*>(my_row + h * 64 + t * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
    if constexpr (EPI != kEpiSiluMulQuant) {
      // whole 16-byte chunks, consecutive lanes along a row: 128 (64 with SiLU-mul) contiguous bytes per row
      constexpr int CHUNKS = EPI == kEpiSiluMul ? 4 : 8;
      const int col0 = EPI == kEpiSiluMul ? (x.n0 >> 1) + s * 32 : x.n0 + s * 64;
      const int col_end = EPI == kEpiSiluMul ? p.n >> 1 : p.n;
      const int ch = lane % CHUNKS;
      const int gcol = col0 + ch * 8;
      __syncwarp();
#pragma unroll
      for (int r0 = 0; r0 < 32; r0 += 32 / CHUNKS) {
        const int lr = r0 + lane / CHUNKS;
        const int grow = row0 + lr;
        if (grow < p.m && gcol + 8 <= col_end) {
          uint4 v = *reinterpret_cast<const uint4*>(staging + lr * ROW_PITCH + ch * 16);
          const long long o = static_cast<long long>(grow) * p.ldo + gcol;
          if constexpr (EPI == kEpiResidual) {
            const uint4 rr = *reinterpret_cast<const uint4*>(p.residual + o);
            v.x = pack_bf16(bf16_lo(v.x) + bf16_lo(rr.x), bf16_hi(v.x) + bf16_hi(rr.x));
            v.y = pack_bf16(bf16_lo(v.y) + bf16_lo(rr.y), bf16_hi(v.y) + bf16_hi(rr.y));
            v.z = pack_bf16(bf16_lo(v.z) + bf16_lo(rr.z), bf16_hi(v.z) + bf16_hi(rr.z));
            v.w = pack_bf16(bf16_lo(v.w) + bf16_lo(rr.w), bf16_hi(v.w) + bf16_hi(rr.w));
          }
          *reinterpret_cast<uint4*>(p.out + o) = v;
        }
      }
      __syncwarp();
    }
  }
  if constexpr (EPI == kEpiSiluMulQuant) {
    __syncwarp();
    // packed bytes: width / 4 per row, 16-byte chunks of two groups (the feature count is a multiple of 64)
    const int rows_per = 32 / steps;
    const int ch = lane % steps;
    for (int r0 = 0; r0 < 32; r0 += rows_per) {
      const int lr = r0 + lane / steps;
      const int grow = row0 + lr;
      if (grow < p.m && x.n0 + ch * 64 + 64 <= p.n)
        *reinterpret_cast<uint4*>(p.q_out + static_cast<size_t>(grow) * p.q_ld + (x.n0 >> 2) + ch * 16) =
            *reinterpret_cast<const uint4*>(staging + lr * Q_PITCH + ch * 16);
    }
    if (row0 + lane < p.m) {
      for (int g2 = 0; g2 < steps; ++g2)
        if (x.n0 + g2 * 64 + 64 <= p.n)
          *reinterpret_cast<uint16_t*>(p.q_sf + row_sf_off(row0 + lane, (x.n0 >> 5) + 2 * g2, p.q_ka)) =
              *reinterpret_cast<const uint16_t*>(my_row + 64 + 2 * g2);
    }
    __syncwarp();
  }
}

template <int EPI>
__global__ void __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                 const __grid_constant__ CUtensorMap tb_sub, const __grid_constant__ CUtensorMap tsfa,
                 const __grid_constant__ CUtensorMap tsfb, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + STAGES * STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + STAGING_BYTES);   // the leader's count both CTAs' bytes
  uint64_t* empty = full + STAGES;
  uint64_t* accum = empty + STAGES;     // [2] accumulator complete (both CTAs)
  uint64_t* acc_free = accum + 2;       // leader: the shared columns of the last unit have been read (8 warps)
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_free + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0);   // warp-uniform for the compiler too
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const int cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&accum[0], 1);
    mbar_init(&accum[1], 1);
    mbar_init(acc_free, 8);
    *abort = 0;
    fence_mbar_init();
    prefetch_tmap(&ta);
    prefetch_tmap(&tb);
    prefetch_tmap(&tsfa);
    prefetch_tmap(&tsfb);
  }
  if (warp == 1) tmem_alloc_pair(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // both CTAs' barriers are initialised before either side signals the other's
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  if (p.early_launch) grid_dep_launch();

  const uint32_t smem_base = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
  if (warp == 0) {
    // The whole warp walks the loop (waits included) and one elected lane issues: see elect_one.
    const uint32_t full0 = __shfl_sync(0xffffffffu, map_to_cta(smem_u32(full), 0), 0);   // the leader's barriers
    int i = 0;             // stage counter over all units
    auto side_a = [&](const Unit& x, int kt, int s) {
      const uint32_t st = smem_base + s * STAGE_BYTES;
      tma_load_2d_pair(st, &ta, full0 + s * 8, kt * 128, x.m0 + static_cast<int>(rank) * 128);
      tma_load_2d_pair(st + A_BYTES + B_BYTES, &tsfa, full0 + s * 8, kt * 256, (x.m0 >> 7) + static_cast<int>(rank));
    };
    auto side_b = [&](const Unit& x, int kt, int s) {
      const uint32_t st = smem_base + s * STAGE_BYTES;
      tma_load_2d_pair(st + A_BYTES, x.width == PAIR_N ? &tb : &tb_sub, full0 + s * 8, kt * 128,
                       x.n0 + static_cast<int>(rank) * (x.width >> 1));
      tma_load_2d_pair(st + A_BYTES + B_BYTES + SFA_BYTES, &tsfb, full0 + s * 8, kt * 256, x.n0 >> 7);
    };
    auto tx_bytes = [](const Unit& x) {
      return 2u * (A_BYTES + SFA_BYTES + SFB_BYTES + static_cast<uint32_t>(x.width) * 64u);
    };
    // The first ring of stages: weights first (they depend on nothing), then the wait for the kernel that produces
    // the activations, then the activations.
    int pre = 0;
    {
      const Unit x = unit_at(p, cluster);
      if (cluster < p.units && x.live) pre = min(STAGES, p.k_tiles);
      if (elect_one())
        for (int kt = 0; kt < pre; ++kt) {
          if (rank == 0) mbar_expect_tx(&full[kt], tx_bytes(x));
          side_b(x, kt, kt);
        }
      __syncwarp();
      grid_dep_wait();
      if (elect_one())
        for (int kt = 0; kt < pre; ++kt) side_a(x, kt, kt);
      __syncwarp();
    }
    bool ok = true;
    for (int u = cluster; u < p.units && ok; u += clusters) {
      const Unit x = unit_at(p, u);
      if (!x.live) continue;
      for (int kt = 0; kt < p.k_tiles; ++kt, ++i) {
        if (i < pre) continue;
        const int s = i % STAGES;
        if (i >= STAGES)
          ok = __all_sync(0xffffffffu, mbar_wait(&empty[s], ((i / STAGES) & 1) ^ 1, abort, p.status, kTimeoutEmpty));
        if (!ok) break;
        if (elect_one()) {
          if (rank == 0) mbar_expect_tx(&full[s], tx_bytes(x));
          side_b(x, kt, s);
          side_a(x, kt, s);
        }
        __syncwarp();
      }
    }
    if (!ok && rank == 0 && lane == 0) {
      // Bounded wait for the copies still in flight so that none lands after the CTAs have gone.
      volatile int ignore = 0;
      for (int j = max(i - STAGES, 0); j < i; ++j)
        mbar_wait(&full[j % STAGES], (j / STAGES) & 1, &ignore, nullptr, kTimeoutDrain);
    }
  } else if (warp == 1) {
    // The whole warp walks the loop (waits included) and one elected lane issues: see elect_one.
    if (rank == 0) {
      const uint32_t sfa_t = tmem_base + SFA_COL, sfb_t = tmem_base + SFB_COL;
      int i = 0, it = 0;
      bool ok = true;
      for (int u = cluster; u < p.units && ok; u += clusters) {
        const Unit x = unit_at(p, u);
        if (!x.live) continue;
        const uint32_t idesc = make_idesc_nvf4(PAIR_M, PAIR_N) -
                               (static_cast<uint32_t>((PAIR_N - x.width) >> 3) << 17);
        const uint32_t acc = tmem_base + ((it & 1) ? ACC1_COL : 0);
        const uint32_t sfb_u = sfb_t + ((x.n0 & 64) ? 2 : 0);    // a 64-column unit in the upper half of a block
        if (it > 0) ok = __all_sync(0xffffffffu, mbar_wait(acc_free, (it - 1) & 1, abort, p.status, kTimeoutAccum));
        if (!ok) break;
        tc_fence_after();
        for (int kt = 0; kt < p.k_tiles; ++kt, ++i) {
          const int s = i % STAGES;
          ok = __all_sync(0xffffffffu, mbar_wait(&full[s], (i / STAGES) & 1, abort, p.status, kTimeoutFull));
          if (!ok) break;
          tc_fence_after();
          const uint32_t st = smem_base + s * STAGE_BYTES;
          const uint64_t adesc = make_desc_sw128(st);
          const uint64_t bdesc = make_desc_sw128(st + A_BYTES);
          const uint32_t sf = st + A_BYTES + B_BYTES;
          if (elect_one()) {
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
              tmem_cp_32x128b_x4_pair(sfa_t + kb * 4, make_desc_sf(sf + kb * 512));
              tmem_cp_32x128b_x4_pair(sfb_t + kb * 8, make_desc_sf(sf + SFA_BYTES + kb * 512));
              tmem_cp_32x128b_x4_pair(sfb_t + kb * 8 + 4, make_desc_sf(sf + SFA_BYTES + 2048 + kb * 512));
            }
#pragma unroll
            for (int kb = 0; kb < 4; ++kb)
              mma_nvf4_pair(acc, adesc + kb * 2, bdesc + kb * 2, idesc, (kt > 0 || kb > 0) ? 1u : 0u, sfa_t + kb * 4,
                            sfb_u + kb * 8);
            tc_commit_pair(&empty[s]);
            if (kt == p.k_tiles - 1) tc_commit_pair(&accum[it & 1]);
          }
          __syncwarp();
        }
        ++it;
      }
    }
  } else {
    grid_dep_wait();
    const int q = warp & 3;      // TMEM lane quarter this warp may read
    const uint32_t tlane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    const uint32_t release = map_to_cta(smem_u32(acc_free), 0);
    uint8_t* mine = staging + q * 32 * ROW_PITCH;
    float alpha = p.alpha;
    if (p.alpha_ptr != nullptr) alpha *= *p.alpha_ptr;
    const float q_inv_gs = EPI == kEpiSiluMulQuant ? 1.f / *p.q_gscale : 0.f;
    int it = 0;
    for (int u = cluster; u < p.units; u += clusters) {
      const Unit x = unit_at(p, u);
      if (!x.live) continue;
      const int buf = it & 1;
      if (!mbar_wait(&accum[buf], (it >> 1) & 1, abort, p.status, kTimeoutAccum)) break;
      tc_fence_after();
      epilogue_unit<EPI>(p, x, buf, tlane + (buf ? ACC1_COL : 0), x.m0 + static_cast<int>(rank) * 128 + q * 32, mine,
                         alpha, q_inv_gs, release, lane);
      ++it;
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();      // nobody leaves while the pair's MMAs, commits or arrivals may still touch its memory
  if (warp == 1) tmem_dealloc_pair(tmem_base, 512);
}

template <int EPI>
cudaError_t launch(const CUtensorMap& ta, const CUtensorMap& tb, const CUtensorMap& tb_sub, const CUtensorMap& tsfa,
                   const CUtensorMap& tsfb, const PairParams& p, int clusters, cudaStream_t stream) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * clusters);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = SMEM_BYTES;
  cfg.stream = stream;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = hb_gemm_get_pdl() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, gemm_pair_kernel<EPI>, ta, tb, tb_sub, tsfa, tsfb, p);
}

// Clusters of two that the device holds at once (0 = the kernels could not be set up).
template <int EPI>
int resident_clusters() {
  if (cudaFuncSetAttribute(gemm_pair_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) != cudaSuccess)
    return 0;
  cudaLaunchConfig_t q = {};
  q.gridDim = dim3(2);
  q.blockDim = dim3(THREADS);
  q.dynamicSmemBytes = SMEM_BYTES;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
  q.attrs = at;
  q.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<EPI>, &q) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace

bool gemm_pair_ok(const GemmArgs& a) {
  if (a.kind != kGemmNvfp4 || a.swap || a.peer != nullptr || a.grp_cnt != nullptr || a.tok_scale != nullptr ||
      a.splits > 1 || a.bn != 256)
    return false;
  if (a.epilogue == kEpiSiluMulQuant) return true;      // gemm_launch has checked its layout
  if (a.epilogue != kEpiStore && a.epilogue != kEpiResidual && a.epilogue != kEpiSiluMul) return false;
  // 16-byte output chunks
  const int cols = a.epilogue == kEpiSiluMul ? 16 : 8;
  return a.rb % cols == 0 && a.ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(a.residual) & 15) == 0;
}

cudaError_t gemm_pair_launch(const GemmArgs& a, cudaStream_t stream) {
  static const int resident = [] {
    int n = resident_clusters<kEpiStore>();
    n = std::min(n, resident_clusters<kEpiResidual>());
    n = std::min(n, resident_clusters<kEpiSiluMul>());
    return std::min(n, resident_clusters<kEpiSiluMulQuant>());
  }();
  if (resident < 1) return cudaErrorInvalidConfiguration;
  PairParams p;
  p.m = a.ra; p.n = a.rb; p.k_tiles = (a.k + 255) / 256;
  p.m_tiles = (a.ra + PAIR_M - 1) / PAIR_M;
  const int n_tiles = (a.rb + PAIR_N - 1) / PAIR_N;
  const int tiles = p.m_tiles * n_tiles;
  // Width of the units that the last, partial wave of full tiles is cut into: the one with the shortest estimate. A K tile
  // of a wave costs the larger of the MMAs (0.28 us at 256 columns) and of the bytes the wave's clusters fetch through L2,
  // which delivers 12.5 TB/s to all SMs together (measured; a full wave of 256-column units is bound by it): 22 KB plus
  // 64 bytes per column and CTA. Narrow units spread a few tiles over idle SMs but fetch the A rows again.
  const int rem = tiles % resident;
  p.sub_width = PAIR_N;
  double best = 1e30;
  for (int w = PAIR_N; w >= 64 && rem != 0; w /= 2) {
    double t = 0;
    for (int left = rem * (PAIR_N / w); left > 0; left -= resident) {
      const int live = std::min(left, resident);
      t += std::max(0.28 * w / PAIR_N, 2.0 * live * (22528 + 64 * w) / 12.5e6) + 0.01;
    }
    if (t < best * 0.97) {
      best = t;
      p.sub_width = w;
    }
  }
  p.full_units = p.sub_width == PAIR_N ? tiles : tiles - rem;
  p.units = p.full_units + (tiles - p.full_units) * (PAIR_N / p.sub_width);
  p.out = static_cast<__nv_bfloat16*>(a.out); p.ldo = a.ldo;
  p.residual = static_cast<const __nv_bfloat16*>(a.residual);
  p.alpha = a.alpha; p.alpha_ptr = a.alpha_ptr;
  p.early_launch = hb_gemm_get_pdl() >= 2;
  p.q_out = static_cast<uint8_t*>(a.q_out); p.q_sf = static_cast<uint8_t*>(a.q_sf); p.q_gscale = a.q_gscale;
  p.q_ka = a.q_ka; p.q_ld = a.q_ld;
  p.status = a.status;

  const uint64_t cols = static_cast<uint64_t>(a.k / 2);
  const uint32_t sub_rows = static_cast<uint32_t>(p.sub_width / 2);
  const TmapKey ka{a.a, static_cast<uint64_t>(a.ra), cols, static_cast<uint64_t>(a.lda / 2), 128, 128, 1};
  const TmapKey kb{a.b, static_cast<uint64_t>(a.rb), cols, static_cast<uint64_t>(a.ldb / 2), 128, 128, 1};
  const TmapKey kb_sub{a.b, static_cast<uint64_t>(a.rb), cols, static_cast<uint64_t>(a.ldb / 2), sub_rows, 128, 1};
  // scale factors as rows of 128-row blocks: 64 8-byte words per K atom
  const uint64_t pa = static_cast<uint64_t>(a.sf_k_atoms_a) * 512, pb = static_cast<uint64_t>(a.sf_k_atoms_b) * 512;
  const TmapKey ksa{a.sfa, static_cast<uint64_t>((a.ra + 127) / 128), pa / 8, pa, 1, 256, 2};
  const TmapKey ksb{a.sfb, static_cast<uint64_t>((a.rb + 127) / 128), pb / 8, pb, 2, 256, 2};
  CUtensorMap ta, tb, tb_sub, tsfa, tsfb;
  if (!get_tmap_2d(ka, &ta) || !get_tmap_2d(kb, &tb) || !get_tmap_2d(kb_sub, &tb_sub) || !get_tmap_2d(ksa, &tsfa) ||
      !get_tmap_2d(ksb, &tsfb))
    return cudaErrorInvalidValue;
  const int clusters = std::min(resident, p.units);
  switch (a.epilogue) {
    case kEpiStore: return launch<kEpiStore>(ta, tb, tb_sub, tsfa, tsfb, p, clusters, stream);
    case kEpiResidual: return launch<kEpiResidual>(ta, tb, tb_sub, tsfa, tsfb, p, clusters, stream);
    case kEpiSiluMul: return launch<kEpiSiluMul>(ta, tb, tb_sub, tsfa, tsfb, p, clusters, stream);
    case kEpiSiluMulQuant: return launch<kEpiSiluMulQuant>(ta, tb, tb_sub, tsfa, tsfb, p, clusters, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace hb
