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
//
// Grouped (mixture-of-experts) mode: a unit is (chunk of up to 256 rows of an expert's segment, 256 of its weight rows), from
// the work list that the routing plan left on the device. An expert of a 4096-token chunk has about 176 rows, and its
// GEMM is 4 to 11 K tiles long: as one CTA per 128 x 128 tile, set-up and epilogue took most of the time (fc1 and
// fc2 of 512 experts, 1024 x 2688, 904 / 4096 tokens of 22 experts each: 544 us on average; as units 349 / 359 and 217 / 238). fc1
// requantises its activation for fc2 in the epilogue, straight from registers: staged in shared memory, which the MMAs keep busy, it
// took 40 us longer, and with four warps per lane quarter instead of two 90 more. Rows of A that lie past the segment are not
// fetched and their warps skip the epilogue: 305 / 321 and 205 / 226 us. What is left is the epilogue of fc1 (237 us without) and 1.1 us
// between the units of a cluster, which share accumulator columns; the weights' bytes take 121.
#include <algorithm>

#include "gemm.cuh"

#include "hb_common.cuh"
#include "rownorm.cuh"

extern "C" int hb_gemm_get_pdl(void);

namespace hb {
namespace {

constexpr int PAIR_M = 256;                   // rows of a unit (128 per CTA)
constexpr int PAIR_N = 256;                   // columns of a full unit
constexpr int EPI_WARPS = 8;                  // two per TMEM lane quarter, half of a unit's columns each
constexpr int THREADS = 64 + EPI_WARPS * 32;  // producer warp, MMA warp, epilogue warps
constexpr int STAGES = 5;
constexpr int A_BYTES = 128 * 128;            // 128 rows x 256 packed e2m1
constexpr int B_BYTES = 128 * 128;            // this CTA's half of the 256 columns
constexpr int SFA_BYTES = 2048;               // one 128-row block x 4 K atoms
constexpr int SFB_BYTES = 4096;               // two 128-column blocks x 4 K atoms (each CTA holds all columns' scales)
constexpr int STAGE_BYTES = A_BYTES + B_BYTES + SFA_BYTES + SFB_BYTES;
constexpr int ROW_PITCH = 80;                 // staged output row: 64 bytes (conflict-free 16-byte accesses)
constexpr int STAGING_BYTES = EPI_WARPS * 32 * ROW_PITCH;
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
  // grouped mode
  const int* grp_start;     // [E] first row of the expert's segment (a multiple of 128)
  const int* grp_cnt;       // [E] its rows
  const int* grp_tiles;     // work list: expert * 4096 + chunk of 256 rows
  const int* grp_ntiles;
  int grp_rows_b;           // weight rows per expert (n columns)
  int n_tiles;              // units per list entry; the last one is sub_width wide if that covers its columns
};

struct Unit {
  int m0, n0, width;      // first row, first column, columns
  int b0;                 // first row of the weight matrix
  int m_end;              // rows from here on are not stored
  float alpha;
  bool live;              // a narrow unit of a ragged last tile can lie past the last column
};

// The units of one cluster in order. In grouped mode a unit's place takes two dependent loads: the entry after the next and
// the segment of the next one are under way while the current unit is worked on.
template <bool GRP>
struct UnitWalk {
  const PairParams& p;
  int u, stride, units;
  int code_far = 0;                                   // list entry of unit u + 2 stride
  int code_next = 0, start_next = 0, cnt_next = 0;    // entry, segment and scale of unit u + stride
  float alpha_next = 0.f;
  int code = 0, start = 0, cnt = 0;
  float alpha = 0.f;

  __device__ __forceinline__ UnitWalk(const PairParams& params, int cluster, int clusters) : p(params), u(cluster), stride(clusters) {
    if constexpr (GRP) {
      units = *p.grp_ntiles * p.n_tiles;
      code_far = entry(u);
      fetch();
      code_far = entry(u + stride);
      step();
      code_far = entry(u + 2 * stride);
    } else {
      units = p.units;
    }
  }
  __device__ __forceinline__ int entry(int unit) const { return unit < units ? p.grp_tiles[unit / p.n_tiles] : 0; }
  __device__ __forceinline__ void fetch() {
    code_next = code_far;
    start_next = p.grp_start[code_next >> 12];
    cnt_next = p.grp_cnt[code_next >> 12];
    alpha_next = p.alpha_ptr != nullptr ? p.alpha_ptr[code_next >> 12] : 1.f;
  }
  __device__ __forceinline__ void step() {
    code = code_next; start = start_next; cnt = cnt_next; alpha = alpha_next;
    fetch();
  }
  __device__ __forceinline__ bool more() const { return u < units; }
  __device__ __forceinline__ void next() {
    u += stride;
    if constexpr (GRP) {
      step();
      code_far = entry(u + 2 * stride);
    }
  }
  __device__ __forceinline__ int width() const {
    if constexpr (GRP) return u % p.n_tiles == p.n_tiles - 1 ? p.sub_width : PAIR_N;
    return u >= p.full_units ? p.sub_width : PAIR_N;
  }
  __device__ __forceinline__ Unit unit() const {
    Unit x;
    x.width = width();
    if constexpr (GRP) {
      x.m0 = start + (code & 4095) * PAIR_M;
      x.n0 = (u % p.n_tiles) * PAIR_N;
      x.b0 = (code >> 12) * p.grp_rows_b + x.n0;
      x.m_end = start + cnt;
      x.alpha = p.alpha * alpha;
      x.live = true;
    } else {
      int t = u, sub = 0;
      if (u >= p.full_units) {
        const int per = PAIR_N / p.sub_width;
        t = p.full_units + (u - p.full_units) / per;
        sub = (u - p.full_units) % per;
      }
      // rows fastest: the row tiles that read the same weights run side by side, so the weights leave HBM once
      x.m0 = (t % p.m_tiles) * PAIR_M;
      x.n0 = (t / p.m_tiles) * PAIR_N + sub * x.width;
      x.b0 = x.n0;
      x.m_end = p.m;
      x.alpha = 0.f;      // one scale for all units: read once by the epilogue
      x.live = x.n0 < p.n;
    }
    return x;
  }
};

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

// One epilogue warp's part of a unit: 32 rows x half of its columns, in steps of 32 columns (one tcgen05.ld), two steps in
// registers at a time. `acc` is the accumulator's address for the warp's lanes, `release` the leader's acc_free barrier.
// The columns that the two accumulators share come first: the last ones of the first, the first ones of the second.
template <int EPI, bool GRP>
__device__ __forceinline__ void epilogue_unit(const PairParams& p, const Unit& x, int buf, int half, uint32_t acc, int row0,
                                              uint8_t* staging, float alpha, float q_inv_gs, uint32_t release, int lane) {
  if (GRP && row0 >= x.m_end) {                     // none of these rows is stored (the segment's padding)
    __syncwarp();
    if (lane == 0) mbar_arrive_cluster(release);
    return;
  }
  const int steps = x.width / 64, groups = (steps + 1) / 2;
  const int col0 = half * (x.width / 2);            // first column of this half, within the unit
  uint8_t* my_row = staging + lane * ROW_PITCH;
  const int row = row0 + lane;
#pragma unroll 1
  for (int j = 0; j < groups; ++j) {
    const int s0 = 2 * (buf == 0 ? groups - 1 - j : j);
    uint32_t r[2][32];
    tmem_ld_32x32(acc + col0 + s0 * 32, r[0]);
    if (s0 + 1 < steps) tmem_ld_32x32(acc + col0 + s0 * 32 + 32, r[1]);
    tmem_ld_wait();
    if (j == 0) {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(release);
    }
    if constexpr (EPI == kEpiSiluMulQuant || EPI == kEpiRelu2Quant) {
      // The thread's token: two steps are 32 or 64 features, 16 or 32 packed bytes and two or four scale bytes, which go straight
      // from registers to whole or half sectors. Same arithmetic in the same order as the stand-alone quantiser. Whole steps are
      // in range or none: ungrouped SiLU-mul calls have a multiple of 64 gate and up columns, grouped calls of 64 features.
      constexpr int GROUPS = EPI == kEpiSiluMulQuant ? 1 : 2;     // 16-feature groups of a step
      constexpr int SHIFT = EPI == kEpiSiluMulQuant ? 5 : 4;      // columns per group, log2
      uint2 pk[2 * GROUPS];
      uint32_t sfw = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        if (s0 + h >= steps) break;
#pragma unroll
        for (int g = 0; g < GROUPS; ++g) {
          float y[16];
#pragma unroll
          for (int t = 0; t < 16; ++t) {
            if constexpr (EPI == kEpiSiluMulQuant) {
              y[t] = __bfloat162float(__float2bfloat16(silu_fast(__uint_as_float(r[h][2 * t]) * alpha) *
                                                       (__uint_as_float(r[h][2 * t + 1]) * alpha)));
            } else {      // squared ReLU, rounded as a bf16 store would
              const float v = __uint_as_float(r[h][g * 16 + t]) * alpha;
              y[t] = __bfloat162float(__float2bfloat16(v > 0.f ? v * v : 0.f));
            }
          }
          sfw |= quant16(y, q_inv_gs, &pk[h * GROUPS + g]) << (8 * (h * GROUPS + g));
        }
      }
      const int c = x.n0 + col0 + s0 * 32;          // first column
      const int ng = c >= p.n ? 0 : s0 + 1 < steps && c + 64 <= p.n ? 2 * GROUPS : GROUPS;      // groups in range
      if (row < x.m_end && ng > 0) {
        uint8_t* dst = p.q_out + static_cast<size_t>(row) * p.q_ld + (c >> SHIFT) * 8;
        uint8_t* sf = p.q_sf + row_sf_off(row, c >> SHIFT, p.q_ka);      // the groups of a K atom are neighbouring bytes
        if (ng == 2 * GROUPS) {
          *reinterpret_cast<uint4*>(dst) = make_uint4(pk[0].x, pk[0].y, pk[1].x, pk[1].y);
          if constexpr (GROUPS == 2) {
            *reinterpret_cast<uint4*>(dst + 16) = make_uint4(pk[2].x, pk[2].y, pk[3].x, pk[3].y);
            *reinterpret_cast<uint32_t*>(sf) = sfw;
          } else {
            *reinterpret_cast<uint16_t*>(sf) = static_cast<uint16_t>(sfw);
          }
        } else {
          *reinterpret_cast<uint2*>(dst) = pk[0];
          sf[0] = static_cast<uint8_t>(sfw);
          if constexpr (GROUPS == 2) {
            *reinterpret_cast<uint2*>(dst + 8) = pk[1];
            sf[1] = static_cast<uint8_t>(sfw >> 8);
          }
        }
      }
    } else
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int s = s0 + h;
      if (s >= steps) break;
      const int c = x.n0 + col0 + s * 32;           // first column of the step
      {
        // bf16 rows through shared memory: whole 16-byte chunks, consecutive lanes along a row
        constexpr int CHUNKS = EPI == kEpiSiluMul ? 2 : 4;
#pragma unroll
        for (int t = 0; t < CHUNKS; ++t) {
          uint32_t w[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if constexpr (EPI == kEpiSiluMul) {
              const int e = 16 * t + 4 * i;
              w[i] = pack_bf16(silu_fast(__uint_as_float(r[h][e]) * alpha) * (__uint_as_float(r[h][e + 1]) * alpha),
                               silu_fast(__uint_as_float(r[h][e + 2]) * alpha) * (__uint_as_float(r[h][e + 3]) * alpha));
            } else {
              w[i] = pack_bf16(__uint_as_float(r[h][8 * t + 2 * i]) * alpha, __uint_as_float(r[h][8 * t + 2 * i + 1]) * alpha);
            }
          }
          *reinterpret_cast<uint4*>(my_row + t * 16) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        const int col_end = EPI == kEpiSiluMul ? p.n >> 1 : p.n;
        const int ch = lane % CHUNKS;
        const int gcol = (EPI == kEpiSiluMul ? c >> 1 : c) + ch * 8;
        __syncwarp();
#pragma unroll
        for (int r0 = 0; r0 < 32; r0 += 32 / CHUNKS) {
          const int lr = r0 + lane / CHUNKS;
          const int grow = row0 + lr;
          if (grow < x.m_end && gcol + 8 <= col_end) {
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
  }
  if constexpr (EPI == kEpiSiluMulQuant || EPI == kEpiRelu2Quant) {
    constexpr int SHIFT = EPI == kEpiSiluMulQuant ? 5 : 4;
    if (row < x.m_end && half == 1 && x.n0 + x.width >= p.n)      // groups that pad the last K tile of the next GEMM read as zero
      for (int w = p.n >> SHIFT; w < p.q_ka * 4; ++w) p.q_sf[row_sf_off(row, w, p.q_ka)] = 0;
  }
}

template <int EPI, bool GRP>
__global__ void __launch_bounds__(THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap ta64,
                 const __grid_constant__ CUtensorMap ta32, const __grid_constant__ CUtensorMap tb,
                 const __grid_constant__ CUtensorMap tb_sub, const __grid_constant__ CUtensorMap tsfa,
                 const __grid_constant__ CUtensorMap tsfb, const PairParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = smem + STAGES * STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(staging + STAGING_BYTES);   // the leader's count both CTAs' bytes
  uint64_t* empty = full + STAGES;
  uint64_t* accum = empty + STAGES;     // [2] accumulator complete (both CTAs)
  uint64_t* acc_free = accum + 2;       // leader: the shared columns of the last unit have been read (both CTAs' warps)
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
    mbar_init(acc_free, 2 * EPI_WARPS);
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
    // Grouped: rows of A that a CTA fetches, in whole boxes. What lies beyond the segment's rows is not worth its way from L2: the
    // MMA then reads whatever the stage held, into rows that nobody stores.
    auto box_rows = [](const Unit& x, int r) {
      if constexpr (!GRP) return 128;
      const int n = x.m_end - x.m0 - r * 128;
      return n > 64 ? 128 : n > 32 ? 64 : n > 0 ? 32 : 0;
    };
    auto side_a = [&](const Unit& x, int kt, int s) {
      const uint32_t st = smem_base + s * STAGE_BYTES;
      const int box = box_rows(x, static_cast<int>(rank));
      if (GRP && box == 0) return;
      tma_load_2d_pair(st, !GRP || box == 128 ? &ta : box == 64 ? &ta64 : &ta32, full0 + s * 8, kt * 128,
                       x.m0 + static_cast<int>(rank) * 128);
      tma_load_2d_pair(st + A_BYTES + B_BYTES, &tsfa, full0 + s * 8, kt * 256, (x.m0 >> 7) + static_cast<int>(rank));
    };
    auto side_b = [&](const Unit& x, int kt, int s) {
      const uint32_t st = smem_base + s * STAGE_BYTES;
      tma_load_2d_pair(st + A_BYTES, x.width == PAIR_N ? &tb : &tb_sub, full0 + s * 8, kt * 128,
                       x.b0 + static_cast<int>(rank) * (x.width >> 1));
      tma_load_2d_pair(st + A_BYTES + B_BYTES + SFA_BYTES, &tsfb, full0 + s * 8, kt * 256, x.b0 >> 7);
    };
    auto tx_bytes = [&](const Unit& x) {
      uint32_t bytes = 2u * (SFB_BYTES + static_cast<uint32_t>(x.width) * 64u);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const int box = box_rows(x, r);
        bytes += static_cast<uint32_t>(box) * 128u + (box > 0 ? SFA_BYTES : 0);
      }
      return bytes;
    };
    // The first ring of stages: weights first (they depend on nothing), then the wait for the kernel that produces
    // the activations, then the activations.
    // (In grouped mode the unit itself comes from the plan's kernels, so all of it waits.)
    int pre = 0;
    if constexpr (!GRP) {
      const UnitWalk<false> w(p, cluster, clusters);
      const Unit x = w.unit();
      if (w.more() && x.live) pre = min(STAGES, p.k_tiles);
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
    } else {
      grid_dep_wait();
    }
    bool ok = true;
    for (UnitWalk<GRP> w(p, cluster, clusters); w.more() && ok; w.next()) {
      Unit x = w.unit();
      if (!x.live) continue;
      if constexpr (GRP) {
        x.m0 = __shfl_sync(0xffffffffu, x.m0, 0);
        x.b0 = __shfl_sync(0xffffffffu, x.b0, 0);
        x.m_end = __shfl_sync(0xffffffffu, x.m_end, 0);
      }
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
      // (of a grouped unit this warp needs no more than its width, which is not in the work list)
      int units = p.units;
      if constexpr (GRP) {
        grid_dep_wait();
        units = __shfl_sync(0xffffffffu, *p.grp_ntiles, 0) * p.n_tiles;
      }
      for (int u = cluster; u < units && ok; u += clusters) {
        int width = PAIR_N, n0 = 0;
        if constexpr (GRP) {
          if (u % p.n_tiles == p.n_tiles - 1) width = p.sub_width;
        } else {
          UnitWalk<false> w(p, u, clusters);
          const Unit x = w.unit();
          if (!x.live) continue;
          width = x.width;
          n0 = x.n0;
        }
        const uint32_t idesc = make_idesc_nvf4(PAIR_M, PAIR_N) - (static_cast<uint32_t>((PAIR_N - width) >> 3) << 17);
        const uint32_t acc = tmem_base + ((it & 1) ? ACC1_COL : 0);
        const uint32_t sfb_u = sfb_t + ((n0 & 64) ? 2 : 0);      // a 64-column unit in the upper half of a block
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
    const int half = (warp - 2) >> 2;
    uint8_t* mine = staging + (warp - 2) * 32 * ROW_PITCH;
    float alpha = p.alpha;
    if (!GRP && p.alpha_ptr != nullptr) alpha *= *p.alpha_ptr;
    const float q_inv_gs = EPI == kEpiSiluMulQuant || EPI == kEpiRelu2Quant ? 1.f / *p.q_gscale : 0.f;
    int it = 0;
    for (UnitWalk<GRP> w(p, cluster, clusters); w.more(); w.next()) {
      const Unit x = w.unit();
      if (!x.live) continue;
      if constexpr (GRP) alpha = x.alpha;
      const int buf = it & 1;
      // one verdict per warp: lanes that give up on a wait must not leave the others alone in a warp-wide TMEM load
      if (!__all_sync(0xffffffffu, mbar_wait(&accum[buf], (it >> 1) & 1, abort, p.status, kTimeoutAccum))) break;
      tc_fence_after();
      epilogue_unit<EPI, GRP>(p, x, buf, half, tlane + (buf ? ACC1_COL : 0), x.m0 + static_cast<int>(rank) * 128 + q * 32, mine,
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

template <int EPI, bool GRP>
cudaError_t launch(const CUtensorMap& ta, const CUtensorMap& ta64, const CUtensorMap& ta32, const CUtensorMap& tb,
                   const CUtensorMap& tb_sub, const CUtensorMap& tsfa, const CUtensorMap& tsfb, const PairParams& p, int clusters,
                   cudaStream_t stream) {
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
  cfg.numAttrs = hb_gemm_get_pdl() && !hb_take_plain() ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, gemm_pair_kernel<EPI, GRP>, ta, ta64, ta32, tb, tb_sub, tsfa, tsfb, p);
}

// Clusters of two that the device holds at once (0 = the kernels could not be set up).
template <int EPI, bool GRP>
int resident_clusters() {
  if (cudaFuncSetAttribute(gemm_pair_kernel<EPI, GRP>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES) !=
      cudaSuccess)
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
  if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel<EPI, GRP>, &q) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  return n;
}

}  // namespace

bool gemm_pair_ok(const GemmArgs& a) {
  if (a.kind != kGemmNvfp4 || a.peer != nullptr || a.ep != nullptr || a.tok_scale != nullptr || a.bn != 256) return false;
  const bool grouped = a.grp_cnt != nullptr;
  if (grouped) {
    if (!a.swap || a.grp_tiles == nullptr || a.grp_rows_a % 128 != 0) return false;
  } else if (a.swap || a.splits > 1) {
    return false;
  }
  if (a.epilogue == kEpiSiluMulQuant) return true;      // gemm_launch has checked its layout
  if (a.epilogue == kEpiRelu2Quant) return grouped;
  if (a.epilogue != kEpiStore && (grouped || (a.epilogue != kEpiResidual && a.epilogue != kEpiSiluMul))) return false;
  // 16-byte output chunks
  const int cols = a.epilogue == kEpiSiluMul ? 16 : 8;
  return (grouped ? a.grp_rows_a : a.rb) % cols == 0 && a.ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 &&
         (reinterpret_cast<uintptr_t>(a.residual) & 15) == 0;
}

cudaError_t gemm_pair_launch(const GemmArgs& a, cudaStream_t stream) {
  static const int resident = [] {
    int n = resident_clusters<kEpiStore, false>();
    n = std::min(n, resident_clusters<kEpiResidual, false>());
    n = std::min(n, resident_clusters<kEpiSiluMul, false>());
    n = std::min(n, resident_clusters<kEpiSiluMulQuant, false>());
    n = std::min(n, resident_clusters<kEpiStore, true>());
    n = std::min(n, resident_clusters<kEpiRelu2Quant, true>());
    return std::min(n, resident_clusters<kEpiSiluMulQuant, true>());
  }();
  if (resident < 1) return cudaErrorInvalidConfiguration;
  const bool grouped = a.grp_cnt != nullptr;
  // tokens are the A side here; a grouped call names its weights first
  const void *act = grouped ? a.b : a.a, *act_sf = grouped ? a.sfb : a.sfa;
  const void *wgt = grouped ? a.a : a.b, *wgt_sf = grouped ? a.sfa : a.sfb;
  const int rows = grouped ? a.rb : a.ra, wgt_rows = grouped ? a.ra : a.rb;
  const int act_ka = grouped ? a.sf_k_atoms_b : a.sf_k_atoms_a, wgt_ka = grouped ? a.sf_k_atoms_a : a.sf_k_atoms_b;
  const int64_t act_ld = grouped ? a.ldb : a.lda, wgt_ld = grouped ? a.lda : a.ldb;
  PairParams p;
  p.m = rows; p.n = grouped ? a.grp_rows_a : a.rb; p.k_tiles = (a.k + 255) / 256;
  p.m_tiles = (rows + PAIR_M - 1) / PAIR_M;
  p.n_tiles = (p.n + PAIR_N - 1) / PAIR_N;
  int clusters;
  if (grouped) {
    const int last = p.n - (p.n_tiles - 1) * PAIR_N;      // a multiple of 128
    p.sub_width = last <= 128 ? 128 : PAIR_N;
    p.full_units = p.units = 0;                           // the list's length is on the device
    clusters = resident;
  } else {
    const int tiles = p.m_tiles * p.n_tiles;
    // Width of the units that the last, partial wave of full tiles is cut into: the one with the shortest estimate. A K
    // tile of a wave costs the larger of the MMAs (0.28 us at 256 columns) and of the bytes the wave's clusters fetch
    // through L2, which delivers 12.5 TB/s to all SMs together (measured; a full wave of 256-column units is bound by
    // it): 22 KB plus 64 bytes per column and CTA. Narrow units spread a few tiles over idle SMs but fetch the A rows
    // again.
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
    clusters = std::min(resident, p.units);
  }
  p.out = static_cast<__nv_bfloat16*>(a.out); p.ldo = a.ldo;
  p.residual = static_cast<const __nv_bfloat16*>(a.residual);
  p.alpha = a.alpha; p.alpha_ptr = a.alpha_ptr;
  p.early_launch = hb_gemm_get_pdl() >= 2;
  p.q_out = static_cast<uint8_t*>(a.q_out); p.q_sf = static_cast<uint8_t*>(a.q_sf); p.q_gscale = a.q_gscale;
  p.q_ka = a.q_ka; p.q_ld = a.q_ld;
  p.status = a.status;
  p.grp_start = a.grp_start; p.grp_cnt = a.grp_cnt; p.grp_tiles = a.grp_tiles; p.grp_ntiles = a.grp_ntiles;
  p.grp_rows_b = a.grp_rows_a;

  const uint64_t cols = static_cast<uint64_t>(a.k / 2);
  const uint32_t sub_rows = static_cast<uint32_t>(p.sub_width / 2);
  const uint64_t pitch_a = static_cast<uint64_t>(act_ld / 2), pitch_b = static_cast<uint64_t>(wgt_ld / 2);
  const TmapKey ka{act, static_cast<uint64_t>(rows), cols, pitch_a, 128, 128, 1};
  const TmapKey kb{wgt, static_cast<uint64_t>(wgt_rows), cols, pitch_b, 128, 128, 1};
  const TmapKey kb_sub{wgt, static_cast<uint64_t>(wgt_rows), cols, pitch_b, sub_rows, 128, 1};
  // scale factors as rows of 128-row blocks: 64 8-byte words per K atom
  const uint64_t pa = static_cast<uint64_t>(act_ka) * 512, pb = static_cast<uint64_t>(wgt_ka) * 512;
  const TmapKey ksa{act_sf, static_cast<uint64_t>((rows + 127) / 128), pa / 8, pa, 1, 256, 2};
  const TmapKey ksb{wgt_sf, static_cast<uint64_t>((wgt_rows + 127) / 128), pb / 8, pb, 2, 256, 2};
  CUtensorMap ta, ta64, ta32, tb, tb_sub, tsfa, tsfb;
  TmapKey k64 = ka, k32 = ka;
  if (grouped) {
    k64.box_rows = 64;
    k32.box_rows = 32;
  }
  if (!get_tmap_2d(ka, &ta) || !get_tmap_2d(k64, &ta64) || !get_tmap_2d(k32, &ta32) || !get_tmap_2d(kb, &tb) ||
      !get_tmap_2d(kb_sub, &tb_sub) || !get_tmap_2d(ksa, &tsfa) || !get_tmap_2d(ksb, &tsfb))
    return cudaErrorInvalidValue;
#define HB_PAIR(EPI, GRP) launch<EPI, GRP>(ta, ta64, ta32, tb, tb_sub, tsfa, tsfb, p, clusters, stream)
  switch (a.epilogue) {
    case kEpiStore: return grouped ? HB_PAIR(kEpiStore, true) : HB_PAIR(kEpiStore, false);
    case kEpiResidual: return HB_PAIR(kEpiResidual, false);
    case kEpiSiluMul: return HB_PAIR(kEpiSiluMul, false);
    case kEpiSiluMulQuant: return grouped ? HB_PAIR(kEpiSiluMulQuant, true) : HB_PAIR(kEpiSiluMulQuant, false);
    case kEpiRelu2Quant: return HB_PAIR(kEpiRelu2Quant, true);
    default: return cudaErrorInvalidValue;
  }
#undef HB_PAIR
}

}  // namespace hb
