// Paged GQA prefill attention on the 5th-generation tensor cores (tcgen05.mma, accumulators in TMEM). Head dim 256 runs the
// kernel described here; head dims up to 128 run its two-stream form, attn_prefill_pp_kernel below, and bf16 pools with enough
// query rows the form with two Q tiles per CTA, attn_prefill_q2_kernel.
//
// One CTA owns one (sequence, kv head, block of query tokens). The block's query rows are packed as
// (token, group member) pairs, 128 rows = floor(128 / g) tokens x g query heads of the kv head, so a K / V tile
// gathered once from the token-granular pool serves the whole GQA group. Per 128-key tile:
//
//   producers (3 warps)   gather K and V rows by slot id with 16-byte cp.async into 128-byte-swizzled tiles
//                         (the layout TMA would produce; rows of a paged pool are not a TMA box). K and V have
//                         separate 2-stage rings: a K stage is free as soon as its S MMA has run, so K runs one
//                         tile ahead of V;
//   issuer (1 lane)       S = Q K^T (kind::f16, both operands K-major) into one of two TMEM score buffers, two
//                         tiles ahead of the softmax; once the softmax warps have published P, O += P V (V as
//                         MN-major B operand) accumulates in TMEM;
//   softmax (4 warps)     thread r owns query row r = TMEM lane r: one tcgen05.ld of the whole score row, row max,
//                         exp2, bf16 P tile into swizzled shared memory. The running maximum that O and the row
//                         sum refer to is only raised (and O rescaled in TMEM) when the new maximum exceeds it by
//                         more than 2^8, so the rescale is rare and the tensor pipe overlaps the softmax.
//
// e4m3 pools (F8) run the same pipeline in fp16, to which every e4m3 code expands exactly: eight producer warps load
// 16 codes per lane, expand them in registers and store the swizzled tiles (two loads in flight per lane: K of the next
// tile, V of this one). Q rows become fp16 under a power-of-two row scale (exact down to 2^-31 of the row's
// largest element), and P is the sum of two fp16 tiles, hi + lo: O += hi V + lo V. So that small weights do not fall on the
// fp16 subnormal grid, O and the row sum refer to a value below the running maximum (pf_reference): weights down to 2^-14
// of the largest keep 22 bits, smaller ones are exact to 2^-36 of it. Against the fp32 CUDA-core kernel of attn.cu: 1237 +
// 263 tokens, 24 / 4 heads of 256: 2170 -> 87 us. What bounds it is the chain scores -> softmax -> P -> O of each tile, not
// the MMAs.
//
// Few rows on a long context leave most SMs idle, so the context can be cut into splits (merged by hb_attn_merge): 4 rows
// on 30000 keys, 24 / 4 heads of 256: 1050 us as one range, 63 us in 37.
//
// Causal masking follows the ragged-batch rule of the engine: row token j of a sequence with R new rows and
// context ctx sees keys [0, ctx - R + j]. All waits are bounded; a timeout raises the status word and every role
// leaves.
//
// Replaces the reference's FlashInfer ragged-prefill wrapper + prefix kernel + LSE merge
// (hibana/kernels/ops.py:131-161, hibana/model/attention.py:73-96, hibana/kernels/csrc/verify_attn.cu prefix_kernel).
#include "kv_tma.cuh"
#include "hb_api.h"
#include "hb_common.cuh"

namespace hb {
namespace {

template <bool F8>
struct PfRoles {                  // warps 0-3 softmax, then the producers, then the MMA issuer
  static constexpr int PROD_WARPS = F8 ? 8 : 3;
  static constexpr int ISSUER = 4 + PROD_WARPS;
  static constexpr int PRODUCERS = PROD_WARPS * 32;
  static constexpr int THREADS = (ISSUER + 1) * 32;
};
constexpr int PF_ROWS = 128;      // packed query rows per CTA
constexpr int PF_STAGES = 2;

struct PfParams {
  const __nv_bfloat16* q;
  const __nv_bfloat16* k_pool;
  const __nv_bfloat16* v_pool;
  long long pool_stride;      // elements between slots
  long long head_stride;      // elements between kv heads
  int tma_xh, tma_yh;         // tensor-map coordinates per kv head (kv_tma.cuh)
  const int* kv_indices;
  long long ld_idx;
  const int* seq_rows;
  const int* ctx_len;
  const int* q_indptr;
  __nv_bfloat16* out;
  float* part_o;              // splits > 1: [T, Hq, splits, D] partial outputs and their log2 sums [T, Hq, splits]
  float* part_lse;
  int hq, hkv, splits;
  int use_tma;                // pools are TMA-addressable: contiguous slot runs travel as bulk tensor copies
  float scale_log2;
  float kv_scale;             // dequantisation scale of an e4m3 pool
  int causal;
  int* status;
  unsigned long long* prof;   // optional cycle counters (null = off)
};

template <int D, bool F8>
struct PfCfg {
  static constexpr int KT = D > 128 ? 64 : 128;               // keys per tile (head dim 256: 64, to fit shared memory)
  static constexpr int HALVES = D / 64;                      // 64-element (128-byte) column blocks of a row
  static constexpr int Q_BYTES = PF_ROWS * D * 2;
  static constexpr int KV_TILE = KT * D * 2;              // one stage of K or of V
  static constexpr int P_BYTES = PF_ROWS * KT * 2;
  static constexpr int BAR_OFF = Q_BYTES + 2 * PF_STAGES * KV_TILE + P_BYTES * (F8 ? 2 : 1);
  static constexpr int SMEM = BAR_OFF + 256 + (F8 ? PF_ROWS * 4 : 0) + 1024;   // F8: one scale per packed query row
  static constexpr int TMEM_COLS = 512;                      // S0 [0, KT) S1 [KT, 2 KT) O [2 KT, 2 KT + D)
  static constexpr float RESCALE_GAP = F8 ? 4.f : 8.f;       // log2 units; F8: weights stay below 2^(11 + 4), in fp16 range
};

__device__ __forceinline__ void cp16(uint32_t saddr, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr), "l"(g) : "memory");
}
__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// What a row's weights refer to (log2 units) when `mx` is its largest raw score. F8: 2^11 below the maximum. Without that, the
// weights below 2^-14 of the maximum would be fp16 subnormals and those below 2^-25 vanish, although the row sum counts
// them: with one dominant key of small V over 30011 keys at 2^-24 the output was 2.5e-2 off, now 4e-6 (the output is bf16). As
// part of the reference it costs nothing per weight; as a factor on every weight it cost 3 %. Maxima of 2^20 and more stay
// as they are: there a difference is rounded to steps that could take a weight out of the fp16 range.
template <bool F8>
__device__ __forceinline__ float pf_reference(float mx, float scale_log2) {
  const float m = __fmul_rn(mx, scale_log2);
  return F8 && fabsf(m) < 1048576.f ? m - 11.f : m;
}
// Cycle accounting of one representative thread per role (softmax thread 0, producer 0, the issuer), summed over
// CTAs into p.prof: where each role's time goes. Costs one predictable branch per site when off.
#define PF_T0() const long long _t0 = p.prof ? clock64() : 0
#define PF_ACC(slot, cond) do { if (p.prof && (cond)) atomicAdd(p.prof + (slot), (unsigned long long)(clock64() - _t0)); } while (0)

// Bounded wait with a warp-uniform verdict, for warps that go on to warp-wide tcgen05.ld / st.
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile int* abort, int* status, int code) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort, status, code));
}
__device__ __forceinline__ void st_zero16(uint32_t saddr) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(saddr), "r"(0) : "memory");
}

// Byte offset of 16-byte chunk `part` of row `r` in a tile of `rows` rows whose 128-byte column blocks are stored
// one after another, each with the 128-byte swizzle (chunk index xor row % 8).
__device__ __forceinline__ uint32_t sw_off(int r, int part, int rows) {
  return static_cast<uint32_t>((part >> 3) * rows * 128 + r * 128 + (((part & 7) ^ (r & 7)) << 4));
}

// 16 e4m3 codes -> 16 fp16 in two 16-byte chunks, at 16-byte columns 2 `part` and 2 `part` + 1 of row r of a tile.
__device__ __forceinline__ void store_f16_row16(uint32_t tile, int r, int part, int rows, const uint4& a) {
  const uint32_t w[4] = {a.x, a.y, a.z, a.w};
  uint32_t h[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    asm("{\n\t.reg .b16 lo, hi;\n\tmov.b32 {lo, hi}, %2;\n\tcvt.rn.f16x2.e4m3x2 %0, lo;\n\tcvt.rn.f16x2.e4m3x2 %1, hi;\n\t}"
        : "=r"(h[2 * i]), "=r"(h[2 * i + 1])
        : "r"(w[i]));
  }
#pragma unroll
  for (int c = 0; c < 2; ++c)
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(tile + sw_off(r, 2 * part + c, rows)), "r"(h[4 * c]),
                 "r"(h[4 * c + 1]), "r"(h[4 * c + 2]), "r"(h[4 * c + 3])
                 : "memory");
}

// What one CTA works on: a block of query tokens of a sequence, one kv head, one range of its keys.
struct PfBlock {
  int g, b, kvh, split, row0, R, tok0, nrows, ctx, kbeg, kmax, ntiles;
  __device__ __forceinline__ PfBlock(const PfParams& p, int KT) {
    g = p.hq / p.hkv;
    const int tok_per_blk = PF_ROWS / g;
    b = blockIdx.z;
    kvh = blockIdx.y;
    split = static_cast<int>(blockIdx.x) % p.splits;
    const int qb = (gridDim.x - 1 - blockIdx.x) / p.splits;   // heaviest (latest) query blocks first
    row0 = p.q_indptr ? p.q_indptr[b] : b;
    R = p.q_indptr ? p.q_indptr[b + 1] - row0 : 1;
    tok0 = qb * tok_per_blk;
    const int ntok = min(tok_per_blk, R - tok0);
    nrows = ntok * g;                                         // none: past the sequence's rows
    ctx = p.ctx_len[b];
    // keys [0, vis) are visible to at least one row of the block, of which this CTA takes [kbeg, kmax): splits are whole
    // tiles, so that only the last one ends inside a tile
    const int vis = p.causal ? min(ctx, ctx - R + tok0 + ntok) : ctx;
    const int per = ((ctx + p.splits - 1) / p.splits + KT - 1) / KT * KT;
    kbeg = split * per;
    kmax = min(vis, kbeg + per);
    ntiles = kmax > kbeg ? (kmax - kbeg + KT - 1) / KT : 0;
  }
};

// F8: the block's Q rows as fp16 under a power-of-two row scale, by `threads` threads (a multiple of 32).
template <int D>
__device__ __forceinline__ void pf_fill_q16(const PfParams& p, const PfBlock& x, uint8_t* q_s, float* row_scale, int tid,
                                            int threads) {
  constexpr int CPR = D / 8;
  const int g = x.g, nrows = x.nrows, row0 = x.row0, tok0 = x.tok0, kvh = x.kvh;
  // CPR = 16 or 32 consecutive lanes hold a row
  for (int c = tid; c < PF_ROWS * CPR; c += threads) {      // both are multiples of 32: warp-uniform
    const int r = c / CPR, part = c % CPR;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (r < nrows)
      v = *reinterpret_cast<const uint4*>(
          p.q + (static_cast<long long>(row0 + tok0 + r / g) * p.hq + kvh * g + r % g) * D + part * 8);
    uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t mx = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) mx = max(mx, max(w[e] & 0x7FFFu, (w[e] >> 16) & 0x7FFFu));
#pragma unroll
    for (int sh = 1; sh < CPR; sh <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, sh));
    const int e2 = static_cast<int>(mx >> 7) - 127;
    const int up = mx == 0 || e2 > 127 ? 0 : min(14 - e2, 126);      // largest element to [2^14, 2^15)
    const float f = __uint_as_float(static_cast<uint32_t>(127 + up) << 23);
    if (part == 0) row_scale[r] = __uint_as_float(static_cast<uint32_t>(127 - up) << 23);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const __half2 h = __floats2half2_rn(bf16_lo(w[e]) * f, bf16_hi(w[e]) * f);
      w[e] = *reinterpret_cast<const uint32_t*>(&h);
    }
    *reinterpret_cast<uint4*>(q_s + sw_off(r, part, PF_ROWS)) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// The producer warps: K and V tiles of the block's keys into their rings of NS stages (and, for bf16 pools, the Q rows). Tile t
// is announced on full barrier t % NF.
template <int D, bool F8, int PF_PRODUCERS, int NS, int NF>
__device__ __forceinline__ void pf_produce(const PfParams& p, const PfBlock& x, const CUtensorMap& tmk, const CUtensorMap& tmv,
                                           uint8_t* q_s, uint8_t* k_s, uint8_t* v_s, uint64_t* kfull, uint64_t* vfull,
                                           uint64_t* kempty, uint64_t* vempty, volatile int* abort, int ptid, int lane) {
  using C = PfCfg<D, F8>;
  constexpr int KT = C::KT;
  constexpr int CPR = D / 8;   // 16-byte chunks per row
  const int g = x.g, b = x.b, kvh = x.kvh, row0 = x.row0, tok0 = x.tok0, nrows = x.nrows, kbeg = x.kbeg, kmax = x.kmax,
            ntiles = x.ntiles;
  const int* idx_row = p.kv_indices + static_cast<long long>(p.seq_rows ? p.seq_rows[b] : b) * p.ld_idx;
  if constexpr (F8) {
    constexpr int CH = D / 16;                              // 16-code chunks per row
    constexpr int PER = KT * CH / PF_PRODUCERS;             // chunks of a tile per thread
    constexpr int RSTEP = PF_PRODUCERS / CH;
    static_assert(KT * CH % PF_PRODUCERS == 0 && PF_PRODUCERS % CH == 0, "whole chunks per thread");
    const int part = ptid % CH, r0 = ptid / CH;
    int sl_now[PER], sl_next[PER];
    uint4 kreg[PER], vreg[PER];
    auto slots = [&](int t, int (&sl)[PER]) {               // -1 beyond the visible keys
#pragma unroll
      for (int i = 0; i < PER; ++i) {
        const int key = kbeg + t * KT + r0 + i * RSTEP;
        sl[i] = t < ntiles && key < kmax ? ld_step(idx_row + key) : -1;
      }
    };
    auto load = [&](const void* pool, const int (&sl)[PER], uint4 (&reg)[PER]) {
#pragma unroll
      for (int i = 0; i < PER; ++i)
        reg[i] = sl[i] < 0 ? make_uint4(0, 0, 0, 0)
                           : ld_step(reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(pool) +
                                                                  static_cast<long long>(sl[i]) * p.pool_stride +
                                                                  kvh * p.head_stride + part * 16));
    };
    auto store = [&](uint8_t* tile, const uint4 (&reg)[PER], uint64_t* bar) {
#pragma unroll
      for (int i = 0; i < PER; ++i) store_f16_row16(smem_u32(tile), r0 + i * RSTEP, part, KT, reg[i]);
      fence_proxy_async_smem();
      mbar_arrive(bar);
    };
    slots(0, sl_now);
    slots(1, sl_next);
    load(p.k_pool, sl_now, kreg);
    for (int t = 0; t < ntiles; ++t) {
      const int s = t % NS;
      const uint32_t ph = ((t / NS) - 1) & 1;
      load(p.v_pool, sl_now, vreg);
      if (t >= NS && !mbar_wait(&kempty[s], ph, abort, p.status, kTimeoutEmpty)) break;
      store(k_s + s * C::KV_TILE, kreg, &kfull[t % NF]);
      load(p.k_pool, sl_next, kreg);
#pragma unroll
      for (int i = 0; i < PER; ++i) sl_now[i] = sl_next[i];
      slots(t + 2, sl_next);
      if (t >= NS && !mbar_wait(&vempty[s], ph, abort, p.status, kTimeoutEmpty)) break;
      store(v_s + s * C::KV_TILE, vreg, &vfull[t % NF]);
    }
  } else {
  // Q rows (zero padded); they travel in the first cp.async group, i.e. with K tile 0.
  for (int c = ptid; c < PF_ROWS * CPR; c += PF_PRODUCERS) {
    const int r = c / CPR, part = c % CPR;
    const uint32_t dst = smem_u32(q_s) + sw_off(r, part, PF_ROWS);
    if (r < nrows) {
      const int tok = tok0 + r / g, gg = r % g;
      cp16(dst, p.q + (static_cast<long long>(row0 + tok) * p.hq + kvh * g + gg) * D + part * 8);
    } else {
      st_zero16(dst);
    }
  }
  // A tile is moved as four 32-key sub-blocks, one producer warp each (warp j % 3). Lane l fetches the slot id
  // of key l of the sub-block. Slots of a sequence are handed out in ascending runs, so most sub-blocks sit in
  // 32 consecutive pool rows: then one lane issues a bulk tensor copy per 128-byte column block (box = 32 rows
  // x 64 elements, 128-byte swizzle, row pitch = one pool slot) that completes on the tile's barrier by
  // transaction bytes. Otherwise (fragmented pool, tail of the context) the warp gathers the rows with 16-byte
  // cp.async: the LSU path keeps only ~16 KB in flight per SM, an order of magnitude less than the TMA unit.
  const int pw = ptid >> 5;
  constexpr int SB = (KT / 32 + 2) / 3;   // sub-blocks per warp and tile
  // Slot ids of this warp's sub-blocks of tile t (one per lane); -1 beyond the visible keys.
  auto fetch_slots = [&](int t, int (&sl)[SB]) {
#pragma unroll
    for (int i = 0; i < SB; ++i) {
      const int j = pw + 3 * i;
      const int key = kbeg + t * KT + j * 32 + lane;
      sl[i] = (j < KT / 32 && t < ntiles && key < kmax) ? ld_step(idx_row + key) : -1;
    }
  };
  auto copy_tile = [&](int t, const int (&sl)[SB], const __nv_bfloat16* pool, const CUtensorMap* tm, uint8_t* ring,
                       uint64_t* bar) {
    uint8_t* tile = ring + (t % NS) * C::KV_TILE;
#pragma unroll
    for (int i = 0; i < SB; ++i) {
      const int j = pw + 3 * i;
      if (j >= KT / 32) break;
      const int slot = sl[i];
      const int slot0 = __shfl_sync(0xffffffffu, slot, 0);
      const bool run = p.use_tma && __all_sync(0xffffffffu, slot >= 0 && slot == slot0 + lane);
      if (run) {
        if (elect_one()) {
          mbar_add_tx(bar, 32 * D * 2);   // bytes only: the lane's arrival comes with the other producers'
#pragma unroll
          for (int h = 0; h < C::HALVES; ++h)
            tma_load_2d(tile + h * (KT * 128) + j * (32 * 128), tm, bar, kvh * p.tma_xh + h * 64,
                        kvh * p.tma_yh + slot0);
        }
      } else {
        // lane -> (row = i * (32 / CPR) + lane / CPR, 16-byte column = lane % CPR)
        constexpr int RPI = 32 / CPR;
        const int part = lane % CPR;
        const uint32_t dst0 = smem_u32(tile) + (part >> 3) * (KT * 128);
#pragma unroll
        for (int ii = 0; ii < 32 / RPI; ++ii) {
          const int rr = ii * RPI + lane / CPR;
          const int s1 = __shfl_sync(0xffffffffu, slot, rr);
          const int r = j * 32 + rr;
          const uint32_t dst = dst0 + r * 128 + (((part & 7) ^ (r & 7)) << 4);
          if (s1 >= 0)
            cp16(dst, pool + static_cast<long long>(s1) * p.pool_stride + kvh * p.head_stride + part * 8);
          else st_zero16(dst);
        }
      }
    }
  };
  // cp.async groups in order: K0, [K1, V0], [K2, V1], ...  After iteration t commits V(t), "at most two groups
  // pending" means K(t) and V(t - 1) have landed: fence them for the tensor-core proxy and signal.
  bool live = ntiles > 0;
  int sl_v[SB], sl_k[SB], sl_pre[SB];   // slots of tile t (V copy), t + 1 (K copy), t + 2 (in flight)
  fetch_slots(0, sl_v);
  fetch_slots(1, sl_k);
  if (live) copy_tile(0, sl_v, p.k_pool, &tmk, k_s, &kfull[0]);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int t = 0; live && t < ntiles; ++t) {
    fetch_slots(t + 2, sl_pre);   // latency hides behind the stage waits below
    if (t + 1 < ntiles) {
      {
        PF_T0();
        if (t + 1 >= NS && !mbar_wait(&kempty[(t + 1) % NS], (((t + 1) / NS) - 1) & 1, abort,
                                             p.status, kTimeoutEmpty)) {
          live = false;
          break;
        }
        PF_ACC(6, ptid == 0);
      }
      {
        PF_T0();
        copy_tile(t + 1, sl_k, p.k_pool, &tmk, k_s, &kfull[(t + 1) % NF]);
        PF_ACC(8, ptid == 0);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    {
      PF_T0();
      if (t >= NS &&
          !mbar_wait(&vempty[t % NS], ((t / NS) - 1) & 1, abort, p.status, kTimeoutEmpty)) {
        live = false;
        break;
      }
      PF_ACC(7, ptid == 0);
    }
    {
      PF_T0();
      copy_tile(t, sl_v, p.v_pool, &tmv, v_s, &vfull[t % NF]);
      PF_ACC(8, ptid == 0);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    PF_T0();
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    PF_ACC(9, ptid == 0);
    fence_proxy_async_smem();
    mbar_arrive(&kfull[t % NF]);
    if (t >= 1) mbar_arrive(&vfull[(t - 1) % NF]);
#pragma unroll
    for (int i = 0; i < SB; ++i) {
      sl_v[i] = sl_k[i];
      sl_k[i] = sl_pre[i];
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");   // nothing may land after the CTA has gone
  fence_proxy_async_smem();
  if (live) mbar_arrive(&vfull[(ntiles - 1) % NF]);
  }
}

template <int D, bool F8>
__global__ void __launch_bounds__(PfRoles<F8>::THREADS, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap tmk, const __grid_constant__ CUtensorMap tmv, const PfParams p) {
  grid_dep_launch();
  grid_dep_wait();
  using C = PfCfg<D, F8>;
  constexpr int KT = C::KT;
  constexpr int PF_PRODUCERS = PfRoles<F8>::PRODUCERS, ISSUER = PfRoles<F8>::ISSUER;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;
  uint8_t* k_s = smem + C::Q_BYTES;
  uint8_t* v_s = k_s + PF_STAGES * C::KV_TILE;
  uint8_t* p_s = v_s + PF_STAGES * C::KV_TILE;
  uint64_t* kfull = reinterpret_cast<uint64_t*>(smem + C::BAR_OFF);
  uint64_t* vfull = kfull + PF_STAGES;
  uint64_t* kempty = vfull + PF_STAGES;
  uint64_t* vempty = kempty + PF_STAGES;
  uint64_t* s_ready = vempty + PF_STAGES;   // [2], one per score buffer
  uint64_t* p_ready = s_ready + 2;
  uint64_t* pv_ready = p_ready + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_ready + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float* row_scale = reinterpret_cast<float*>(smem + C::BAR_OFF + 256);   // F8

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // warp-uniform for the compiler too
  const PfBlock x(p, KT);
  if (x.nrows <= 0) return;   // uniform: before any barrier or TMEM allocation
  const int g = x.g, kvh = x.kvh, row0 = x.row0, R = x.R, tok0 = x.tok0, nrows = x.nrows, ctx = x.ctx, split = x.split,
            kbeg = x.kbeg, ntiles = x.ntiles;

  if (tid == 0) {
    for (int s = 0; s < PF_STAGES; ++s) {
      mbar_init(&kfull[s], PF_PRODUCERS);
      mbar_init(&vfull[s], PF_PRODUCERS);
      mbar_init(&kempty[s], 1);
      mbar_init(&vempty[s], 1);
    }
    mbar_init(&s_ready[0], 1);
    mbar_init(&s_ready[1], 1);
    mbar_init(p_ready, PF_ROWS);
    mbar_init(pv_ready, 1);
    *abort = 0;
    fence_mbar_init();
    if (p.use_tma) {
      prefetch_tmap(&tmk);
      prefetch_tmap(&tmv);
    }
  }
  if (warp == ISSUER) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  if constexpr (F8) {
    pf_fill_q16<D>(p, x, q_s, row_scale, tid, PfRoles<F8>::THREADS);
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);
  const uint32_t o_tmem = tmem_base + 2 * KT;

  if (warp >= 4 && warp < ISSUER) {
    // ------------------------------------------------------------------ producers
    pf_produce<D, F8, PF_PRODUCERS, PF_STAGES, PF_STAGES>(p, x, tmk, tmv, q_s, k_s, v_s, kfull, vfull, kempty, vempty, abort,
                                                          tid - 128, lane);
  } else if (warp == ISSUER) {
    // ------------------------------------------------------------------ MMA issuer
    {   // the whole warp walks the loop, one elected lane issues (hb_common.cuh, elect_one)
      // operand format codes of kind::f16: 0 = fp16, 1 = bf16 (bits 7 and 10)
      constexpr uint32_t kBf16 = (1u << 7) | (1u << 10);
      constexpr uint32_t idesc_qk = make_idesc_bf16(PF_ROWS, KT) & ~(F8 ? kBf16 : 0u);
      constexpr uint32_t idesc_pv = make_idesc_bf16(PF_ROWS, D, 0, 1) & ~(F8 ? kBf16 : 0u);
      const uint32_t q_a = __shfl_sync(0xffffffffu, smem_u32(q_s), 0);
      const uint32_t k_0 = q_a + C::Q_BYTES, v_0 = k_0 + PF_STAGES * C::KV_TILE, p_a = v_0 + PF_STAGES * C::KV_TILE;
      // S(t) = Q K(t)^T into score buffer t % 2; releases the K stage and publishes the scores when done.
      auto issue_qk = [&](int t) -> bool {
        const int s = t % PF_STAGES;
        {
          PF_T0();
          if (!warp_wait(&kfull[s], (t / PF_STAGES) & 1, abort, p.status, kTimeoutFull)) return false;
          PF_ACC(5, lane == 0);
        }
        tc_fence_after();
        const uint32_t k_a = k_0 + s * C::KV_TILE;
        const uint32_t s_t = tmem_base + (t & 1) * KT;
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < D / 16; ++ks) {
            const uint32_t in_row = (ks & 3) * 32;   // 16 elements = 32 bytes inside the 128-byte swizzled row
            mma_f16(s_t, make_desc_sw128(q_a + (ks >> 2) * (PF_ROWS * 128) + in_row),
                    make_desc_sw128(k_a + (ks >> 2) * (KT * 128) + in_row), idesc_qk, ks > 0 ? 1u : 0u);
          }
          tc_commit(&kempty[s]);
          tc_commit(&s_ready[t & 1]);
        }
        __syncwarp();
        return true;
      };
      bool ok = ntiles > 0 && issue_qk(0);
      if (ok && ntiles > 1) ok = issue_qk(1);
      for (int t = 0; ok && t < ntiles; ++t) {
        const int s = t % PF_STAGES;
        {
          PF_T0();
          if (!warp_wait(p_ready, t & 1, abort, p.status, kTimeoutAccum)) break;
          PF_ACC(3, lane == 0);
        }
        {
          PF_T0();
          if (!warp_wait(&vfull[s], (t / PF_STAGES) & 1, abort, p.status, kTimeoutFull)) break;
          PF_ACC(4, lane == 0);
        }
        tc_fence_after();
        const uint32_t v_a = v_0 + s * C::KV_TILE;
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < KT / 16; ++kk) {
            const uint64_t adesc = make_desc_sw128(p_a + (kk >> 2) * (PF_ROWS * 128) + (kk & 3) * 32);
            // 16 keys = two 8-row groups 1024 bytes apart; the D / 64 column blocks are KT * 128 bytes apart
            const uint64_t bdesc = make_desc_sw128_mn(v_a + kk * 2048, KT * 128, 1024);
            mma_f16(o_tmem, adesc, bdesc, idesc_pv, (t > 0 || kk > 0) ? 1u : 0u);
            if constexpr (F8)      // the low parts of the weights
              mma_f16(o_tmem, make_desc_sw128(p_a + C::P_BYTES + (kk >> 2) * (PF_ROWS * 128) + (kk & 3) * 32), bdesc,
                      idesc_pv, 1u);
          }
          tc_commit(&vempty[s]);
          tc_commit(pv_ready);
        }
        __syncwarp();
        // score buffer t % 2 was read completely before p_ready(t): refill it two tiles ahead
        if (t + 2 < ntiles) ok = issue_qk(t + 2);
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + output (warps 0-3)
    const int r = tid;                                   // packed query row = TMEM lane
    const uint32_t tlane = static_cast<uint32_t>(warp * 32) << 16;
    const bool row_ok = r < nrows;
    const int tok = tok0 + r / g;
    // last visible key position (inclusive)
    const int lim = row_ok ? (p.causal ? ctx - R + tok : ctx - 1) : -1;
    const float scale_log2 = F8 ? p.scale_log2 * p.kv_scale * row_scale[r] : p.scale_log2;
    float m_ref = -INFINITY, l = 0.f;   // O and l are relative to 2^m_ref
    const uint32_t p_row = smem_u32(p_s) + r * 128;
    bool ok = true;
    const long long t_begin = p.prof ? clock64() : 0;
    for (int t = 0; t < ntiles; ++t) {
      {
        PF_T0();
        if (!warp_wait(&s_ready[t & 1], (t >> 1) & 1, abort, p.status, kTimeoutAccum)) {
          ok = false;
          break;
        }
        PF_ACC(0, tid == 0);
      }
      tc_fence_after();
      const int k0 = kbeg + t * KT;
      const uint32_t s_t = tmem_base + (t & 1) * KT + tlane;
      // The two passes over the score row are rolled loops over 32-column chunks: fully unrolled, the softmax body
      // alone is several thousand instructions, and streaming that through the instruction cache every tile cost
      // more than the arithmetic. `rel` = last visible column of this tile for this row (>= 127: no masking).
      const int rel = lim - k0;
      const long long t_math = p.prof ? clock64() : 0;
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
      for (int c0 = 0; c0 < KT; c0 += 32) {
        uint32_t v[32];
        tmem_ld_32x32(s_t + c0, v);
        tmem_ld_wait();
        const int rc = rel - c0;
#pragma unroll
        for (int j = 0; j < 32; ++j)
          mx4[j & 3] = fmaxf(mx4[j & 3], j <= rc ? __uint_as_float(v[j]) : -INFINITY);
      }
      const float m_tile = pf_reference<F8>(fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])), scale_log2);
      // P(t) overwrites the buffer O += P(t - 1) V(t - 1) reads, and a rescale touches O: both need that MMA done.
      {
        PF_T0();
        if (t > 0 && !warp_wait(pv_ready, (t - 1) & 1, abort, p.status, kTimeoutAccum)) {
          ok = false;
          break;
        }
        PF_ACC(1, tid == 0);
      }
      if (t == 0) {
        m_ref = m_tile;
      } else if (__any_sync(0xffffffffu, m_tile > m_ref + C::RESCALE_GAP)) {
        // Raise the reference (all lanes of the warp: tcgen05.ld / st are warp-wide) and rescale O and l.
        const float m_new = fmaxf(m_ref, m_tile);
        const float alpha = m_new == -INFINITY ? 1.f : ex2(m_ref - m_new);
        m_ref = m_new;
        l *= alpha;
        tc_fence_after();
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t o[32];
          tmem_ld_32x32(o_tmem + tlane + c0, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          tmem_st_32x32(o_tmem + tlane + c0, o);
        }
        tmem_st_wait();
      }
      const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
      float sum4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 1
      for (int c0 = 0; c0 < KT; c0 += 32) {
        uint32_t v[32];
        tmem_ld_32x32(s_t + c0, v);
        tmem_ld_wait();
        const int rc = rel - c0;
        uint32_t w[16];
        uint32_t wl[F8 ? 16 : 1];
#pragma unroll
        for (int j = 0; j < 32; j += 2) {
          // F8: product and difference rounded one after the other, as the maximum was, so that the largest score gives
          // the same power of two whatever its size (a fused product of scores near 2^40 would overflow the exponential)
          const float x0 = F8 ? __fadd_rn(__fmul_rn(__uint_as_float(v[j]), scale_log2), neg_m)
                              : fmaf(__uint_as_float(v[j]), scale_log2, neg_m);
          const float x1 = F8 ? __fadd_rn(__fmul_rn(__uint_as_float(v[j + 1]), scale_log2), neg_m)
                              : fmaf(__uint_as_float(v[j + 1]), scale_log2, neg_m);
          const float p0 = j <= rc ? ex2(x0) : 0.f;
          const float p1 = j + 1 <= rc ? ex2(x1) : 0.f;
          sum4[(j >> 1) & 3] += p0 + p1;
          if constexpr (F8) {
            const __half2 hi = __floats2half2_rn(p0, p1);
            const __half2 lo = __floats2half2_rn(p0 - __low2float(hi), p1 - __high2float(hi));
            w[j >> 1] = *reinterpret_cast<const uint32_t*>(&hi);
            wl[j >> 1] = *reinterpret_cast<const uint32_t*>(&lo);
          } else {
            w[j >> 1] = pack_bf16(p0, p1);
          }
        }
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) {
          const int part = (c0 >> 3) + ch;   // 16-byte chunk (8 keys) of the row
          const uint32_t dst = p_row + (part >> 3) * (PF_ROWS * 128) + (((part & 7) ^ (r & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(w[4 * ch]), "r"(w[4 * ch + 1]),
                       "r"(w[4 * ch + 2]), "r"(w[4 * ch + 3])
                       : "memory");
          if constexpr (F8)
            asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + C::P_BYTES), "r"(wl[4 * ch]),
                         "r"(wl[4 * ch + 1]), "r"(wl[4 * ch + 2]), "r"(wl[4 * ch + 3])
                         : "memory");
        }
      }
      l += (sum4[0] + sum4[1]) + (sum4[2] + sum4[3]);
      if (p.prof && tid == 0) atomicAdd(p.prof + 13, (unsigned long long)(clock64() - t_math));
      {
        PF_T0();
        tc_fence_before();
        fence_proxy_async_smem();
        mbar_arrive(p_ready);
        PF_ACC(14, tid == 0);
      }
    }
    if (p.prof && tid == 0) {
      atomicAdd(p.prof + 10, (unsigned long long)(clock64() - t_begin));
      atomicAdd(p.prof + 11, (unsigned long long)ntiles);
    }
    if (ok && ntiles > 0) ok = warp_wait(pv_ready, (ntiles - 1) & 1, abort, p.status, kTimeoutAccum);
    if (ok) {
      tc_fence_after();
      float inv = l > 0.f ? 1.f / l : 0.f;
      if constexpr (F8) inv *= p.kv_scale;
      const long long rh = static_cast<long long>(row0 + tok) * p.hq + kvh * g + r % g;
      __nv_bfloat16* dst = p.out + rh * D;
      if (p.splits > 1 && row_ok) p.part_lse[rh * p.splits + split] = l > 0.f ? m_ref + log2f(l) : -INFINITY;
#pragma unroll
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t o[32];
        if (ntiles > 0) {
          tmem_ld_32x32(o_tmem + tlane + c0, o);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = 0;
        }
        if (row_ok && p.splits > 1) {
          float* part = p.part_o + (rh * p.splits + split) * D + c0;
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            *reinterpret_cast<float4*>(part + j) =
                make_float4(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv,
                            __uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv);
        } else if (row_ok) {
#pragma unroll
          for (int j = 0; j < 32; j += 8)
            *reinterpret_cast<uint4*>(dst + c0 + j) =
                make_uint4(pack_bf16(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv),
                           pack_bf16(__uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv),
                           pack_bf16(__uint_as_float(o[j + 4]) * inv, __uint_as_float(o[j + 5]) * inv),
                           pack_bf16(__uint_as_float(o[j + 6]) * inv, __uint_as_float(o[j + 7]) * inv));
        }
      }
      tc_fence_before();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == ISSUER) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

// Head dims up to 128: two softmax warpgroups. One warpgroup's softmax is the longest link of the chain scores -> softmax ->
// P -> O, and with one warp per scheduler its latencies show (3500 of 4480 cycles per 128-key tile). Here the even and the
// odd tiles are two independent streams, each with its own softmax warpgroup, issuer lane, score buffer, accumulator and
// running maximum, on the same Q and the same K / V rings; the streams meet once, at the end. P replaces
// the scores it came from in TMEM and enters O += P V as the A operand from there (F8: 16 columns of hi, 16 of lo per
// 32 keys), so it never passes through shared memory.
// One layer, 40 / 8 heads of 128, bf16: 2048 tokens 138 -> 113 us, 4096 in five prompts 239 -> 204, 2048 new tokens over 30000
// keys 2780 -> 1700; e4m3, 4096 tokens, 32 / 2 heads: 390 -> 282 (8050 on the CUDA cores). Per tile of a stream 6400 cycles are left, 2400 of them
// softmax; the rest is the chain of barriers around the two MMAs and K tiles that arrive late (copies of 32 rows; with
// warps of their own for K and V they came no earlier, and the layer took 125 us).
constexpr int PP_STAGES = 3;      // K and V rings, shared by both streams
// Full barriers of a ring. A wait on a phase parity cannot tell phase n from phase n + 2, so whoever waits on a barrier has to
// wait for every one of its phases. With one barrier per stage a stream would see only every second phase: tile t could
// pass its wait while the other stream's tile t - 3, whose bulk copies may land later than those of tile t - 2, is still on
// its way into that stage. Two barriers per stage make each of them one stream's own (t % 6 is even or odd as t is). The
// empty barriers need no such care: their only waiters, the producers, wait for all phases.
constexpr int PP_FULL = 2 * PP_STAGES;
struct PpPlace {
  int stage, full, parity;        // ring stage, full barrier, and the parity of that barrier's phase
};
__host__ __device__ constexpr PpPlace pp_place(int t) { return {t % PP_STAGES, t % PP_FULL, (t / PP_FULL) & 1}; }
template <bool F8>
struct PpRoles {                  // warps 0-3 and 4-7 softmax, then the producers, then one issuer per stream
  static constexpr int PROD_WARPS = F8 ? 8 : 3;
  static constexpr int ISSUER = 8 + PROD_WARPS;
  static constexpr int PRODUCERS = PROD_WARPS * 32;
  static constexpr int THREADS = (ISSUER + 2) * 32;
};
template <int D, bool F8>
struct PpCfg {
  static constexpr int KT = 128;
  static constexpr int BAR_OFF = PfCfg<D, F8>::Q_BYTES + 2 * PP_STAGES * PfCfg<D, F8>::KV_TILE;
  static constexpr int SCALE_OFF = BAR_OFF + 256;                  // F8: one scale per packed query row
  static_assert((2 * PP_FULL + 2 * PP_STAGES + 6) * 8 + 8 <= 256, "barriers, TMEM address and abort flag");
  static constexpr int SMEM = SCALE_OFF + (F8 ? PF_ROWS * 4 : 0) + 1024;
  static_assert(PfCfg<D, F8>::KT == KT && 2 * KT + 2 * D <= 512, "a score buffer and an accumulator per stream");
};

// Two fp32 operations per instruction (same rounding as the scalar forms).
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// The weights of one row's `keys` scores at s_t (32 columns at a time): replaces the scores by P and returns their sum. `rel` is the
// last visible column; WHOLE rows see all of them.
template <bool F8, bool WHOLE>
__device__ __forceinline__ float pp_weights(uint32_t s_t, int keys, int rel, float scale_log2, float neg_m) {
  const uint64_t scale2 = pack2(scale_log2, scale_log2), neg2 = pack2(neg_m, neg_m);
  uint64_t sum2[2] = {0ull, 0ull};
#pragma unroll 1
  for (int c0 = 0; c0 < keys; c0 += 32) {
    uint32_t v[32];
    tmem_ld_32x32(s_t + c0, v);
    tmem_ld_wait();
    const int rc = rel - c0;
    uint32_t w[16];
    uint32_t wl[F8 ? 16 : 1];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      // F8: product and difference rounded one after the other, as the maximum was, so that the largest score gives
      // the same power of two whatever its size (a fused product of scores near 2^40 would overflow the exponential; the paired
      // mul and add came out fused)
      float p0, p1;
      if constexpr (F8) {
        p0 = __fadd_rn(__fmul_rn(__uint_as_float(v[j]), scale_log2), neg_m);
        p1 = __fadd_rn(__fmul_rn(__uint_as_float(v[j + 1]), scale_log2), neg_m);
      } else {
        unpack2(fma2(pack2(__uint_as_float(v[j]), __uint_as_float(v[j + 1])), scale2, neg2), p0, p1);
      }
      p0 = WHOLE || j <= rc ? ex2(p0) : 0.f;
      p1 = WHOLE || j + 1 <= rc ? ex2(p1) : 0.f;
      sum2[(j >> 1) & 1] = add2(sum2[(j >> 1) & 1], pack2(p0, p1));
      if constexpr (F8) {
        const __half2 hi = __floats2half2_rn(p0, p1);
        const __half2 lo = __floats2half2_rn(p0 - __low2float(hi), p1 - __high2float(hi));
        w[j >> 1] = *reinterpret_cast<const uint32_t*>(&hi);
        wl[j >> 1] = *reinterpret_cast<const uint32_t*>(&lo);
      } else {
        w[j >> 1] = pack_bf16(p0, p1);
      }
    }
    tmem_st_32x16(s_t + c0, w);                        // over the scores just read
    if constexpr (F8) tmem_st_32x16(s_t + c0 + 16, wl);
  }
  float a, b;
  unpack2(add2(sum2[0], sum2[1]), a, b);
  return a + b;
}

template <int D, bool F8>
__global__ void __launch_bounds__(PpRoles<F8>::THREADS, 1)
attn_prefill_pp_kernel(const __grid_constant__ CUtensorMap tmk, const __grid_constant__ CUtensorMap tmv, const PfParams p) {
  grid_dep_launch();
  grid_dep_wait();
  using C = PfCfg<D, F8>;
  constexpr int KT = C::KT;
  constexpr int ISSUER = PpRoles<F8>::ISSUER;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* q_s = smem;
  uint8_t* k_s = smem + C::Q_BYTES;
  uint8_t* v_s = k_s + PP_STAGES * C::KV_TILE;
  uint64_t* kfull = reinterpret_cast<uint64_t*>(smem + PpCfg<D, F8>::BAR_OFF);
  uint64_t* vfull = kfull + PP_FULL;
  uint64_t* kempty = vfull + PP_FULL;
  uint64_t* vempty = kempty + PP_STAGES;
  uint64_t* s_ready = vempty + PP_STAGES;      // from here on one per stream
  uint64_t* p_ready = s_ready + 2;
  uint64_t* pv_done = p_ready + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  float2* ml = reinterpret_cast<float2*>(q_s);     // at the end, over Q: running maximum and sum of both streams' rows
  float* row_scale = reinterpret_cast<float*>(smem + PpCfg<D, F8>::SCALE_OFF);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // warp-uniform for the compiler too
  const PfBlock x(p, KT);
  if (x.nrows <= 0) return;   // uniform: before any barrier or TMEM allocation
  const int ntiles = x.ntiles;

  if (tid == 0) {
    for (int s = 0; s < PP_FULL; ++s) {
      mbar_init(&kfull[s], PpRoles<F8>::PRODUCERS);
      mbar_init(&vfull[s], PpRoles<F8>::PRODUCERS);
    }
    for (int s = 0; s < PP_STAGES; ++s) {
      mbar_init(&kempty[s], 1);
      mbar_init(&vempty[s], 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(&s_ready[s], 1);
      mbar_init(&p_ready[s], PF_ROWS);
      mbar_init(&pv_done[s], 1);
    }
    *abort = 0;
    fence_mbar_init();
    if (p.use_tma) {
      prefetch_tmap(&tmk);
      prefetch_tmap(&tmv);
    }
  }
  if (warp == ISSUER) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if constexpr (F8) {
    pf_fill_q16<D>(p, x, q_s, row_scale, tid, PpRoles<F8>::THREADS);
    fence_proxy_async_smem();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp >= 8 && warp < ISSUER) {
    pf_produce<D, F8, PpRoles<F8>::PRODUCERS, PP_STAGES, PP_FULL>(p, x, tmk, tmv, q_s, k_s, v_s, kfull, vfull, kempty, vempty,
                                                                  abort, tid - 256, lane);
  } else if (warp >= ISSUER) {
    // ------------------------------------------------------------------ MMA issuer of one stream
    constexpr uint32_t kBf16 = (1u << 7) | (1u << 10);      // operand format codes of kind::f16: 0 = fp16, 1 = bf16
    constexpr uint32_t idesc_qk = make_idesc_bf16(PF_ROWS, KT) & ~(F8 ? kBf16 : 0u);
    constexpr uint32_t idesc_pv = make_idesc_bf16(PF_ROWS, D, 0, 1) & ~(F8 ? kBf16 : 0u);
    const int st = warp - ISSUER;
    const uint32_t q_a = __shfl_sync(0xffffffffu, smem_u32(q_s), 0);
    const uint32_t s_t = tmem_base + st * KT, o_t = tmem_base + 2 * KT + st * D;
    for (int t = st, i = 0; t < ntiles; t += 2, ++i) {
      const PpPlace at = pp_place(t);
      const int s = at.stage;
      const uint32_t k_a = q_a + C::Q_BYTES + s * C::KV_TILE, v_a = k_a + PP_STAGES * C::KV_TILE;
      // the score buffer holds P(t - 2) until that tile's O += P V is done
      if (i > 0 && !warp_wait(&pv_done[st], (i - 1) & 1, abort, p.status, kTimeoutAccum)) break;
      {
        PF_T0();
        if (!warp_wait(&kfull[at.full], at.parity, abort, p.status, kTimeoutFull)) break;
        PF_ACC(5, lane == 0 && st == 0);
      }
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t in_row = (ks & 3) * 32;   // 16 elements = 32 bytes inside the 128-byte swizzled row
          mma_f16(s_t, make_desc_sw128(q_a + (ks >> 2) * (PF_ROWS * 128) + in_row),
                  make_desc_sw128(k_a + (ks >> 2) * (KT * 128) + in_row), idesc_qk, ks > 0 ? 1u : 0u);
        }
        tc_commit(&kempty[s]);
        tc_commit(&s_ready[st]);
      }
      __syncwarp();
      {
        PF_T0();
        if (!warp_wait(&p_ready[st], i & 1, abort, p.status, kTimeoutAccum)) break;
        PF_ACC(3, lane == 0 && st == 0);
      }
      {
        PF_T0();
        if (!warp_wait(&vfull[at.full], at.parity, abort, p.status, kTimeoutFull)) break;
        PF_ACC(4, lane == 0 && st == 0);
      }
      tc_fence_after();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < KT / 16; ++kk) {
          // 16 keys = two 8-row groups 1024 bytes apart; the D / 64 column blocks are KT * 128 bytes apart
          const uint64_t bdesc = make_desc_sw128_mn(v_a + kk * 2048, KT * 128, 1024);
          const uint32_t a_t = s_t + (kk >> 1) * 32 + (kk & 1) * 8;      // 8 columns of packed pairs
          mma_f16_ts(o_t, a_t, bdesc, idesc_pv, (i > 0 || kk > 0) ? 1u : 0u);
          if constexpr (F8) mma_f16_ts(o_t, a_t + 16, bdesc, idesc_pv, 1u);   // the low parts of the weights
        }
        tc_commit(&vempty[s]);
        tc_commit(&pv_done[st]);
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------------ softmax of one stream, half of the output columns
    const int st = warp >> 2;
    const int r = tid & (PF_ROWS - 1);                   // packed query row = TMEM lane
    const uint32_t tlane = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_t = tmem_base + st * KT + tlane, o_t = tmem_base + 2 * KT + st * D + tlane;
    const bool row_ok = r < x.nrows;
    const int tok = x.tok0 + r / x.g;
    // last visible key position (inclusive)
    const int lim = row_ok ? (p.causal ? x.ctx - x.R + tok : x.ctx - 1) : -1;
    const float scale_log2 = F8 ? p.scale_log2 * p.kv_scale * row_scale[r] : p.scale_log2;
    float m_ref = -INFINITY, l = 0.f;   // O and l of this stream are relative to 2^m_ref
    bool ok = true;
    const long long t_begin = p.prof ? clock64() : 0;
    for (int t = st, i = 0; t < ntiles; t += 2, ++i) {
      {
        PF_T0();
        ok = warp_wait(&s_ready[st], i & 1, abort, p.status, kTimeoutAccum);
        PF_ACC(0, tid == 0);
      }
      if (!ok) break;
      tc_fence_after();
      // `rel` = last visible column of this tile for this row; a warp whose rows see the whole tile skips the masking.
      const int rel = lim - (x.kbeg + t * KT);
      const bool whole = __all_sync(0xffffffffu, rel >= KT - 1);
      const long long t_math = p.prof ? clock64() : 0;
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll 1
      for (int c0 = 0; c0 < KT; c0 += 32) {
        uint32_t v[32];
        tmem_ld_32x32(s_t + c0, v);
        tmem_ld_wait();
        if (whole) {
#pragma unroll
          for (int j = 0; j < 32; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], __uint_as_float(v[j]));
        } else {
          const int rc = rel - c0;
#pragma unroll
          for (int j = 0; j < 32; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], j <= rc ? __uint_as_float(v[j]) : -INFINITY);
        }
      }
      const float m_tile = pf_reference<F8>(fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])), scale_log2);
      if (i == 0) {
        m_ref = m_tile;
      } else if (__any_sync(0xffffffffu, m_tile > m_ref + C::RESCALE_GAP)) {
        // Raise the reference (all lanes of the warp: tcgen05.ld / st are warp-wide) and rescale O and l. The scores
        // were issued after this stream's last O += P V had completed.
        const float m_new = fmaxf(m_ref, m_tile);
        const float alpha = m_new == -INFINITY ? 1.f : ex2(m_ref - m_new);
        m_ref = m_new;
        l *= alpha;
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 32) {
          uint32_t o[32];
          tmem_ld_32x32(o_t + c0, o);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          tmem_st_32x32(o_t + c0, o);
        }
      }
      const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
      const float sum = whole ? pp_weights<F8, true>(s_t, KT, rel, scale_log2, neg_m)
                              : pp_weights<F8, false>(s_t, KT, rel, scale_log2, neg_m);
      l += sum;
      tmem_st_wait();
      if (p.prof && tid == 0) atomicAdd(p.prof + 13, (unsigned long long)(clock64() - t_math));
      tc_fence_before();
      mbar_arrive(&p_ready[st]);
    }
    if (p.prof && tid == 0) {
      atomicAdd(p.prof + 10, (unsigned long long)(clock64() - t_begin));
      atomicAdd(p.prof + 11, (unsigned long long)((ntiles + 1) / 2));
    }
    // This stream's last O += P V (the other's barrier has phases this thread did not follow), then both streams': from
    // here on no MMA is left, Q included. A stream without tiles (one-tile blocks) has no O.
    const int n0 = (ntiles + 1) / 2, n1 = ntiles / 2, mine = st == 0 ? n0 : n1;
    if (ok && mine > 0) ok = warp_wait(&pv_done[st], (mine - 1) & 1, abort, p.status, kTimeoutAccum);
    __syncwarp();
    asm volatile("bar.sync 1, 256;" ::: "memory");
    ml[st * PF_ROWS + r] = make_float2(m_ref, l);
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (ok) {
      tc_fence_after();
      // (without tiles nobody has waited for the copy of Q, which then lands where `ml` is)
      const float2 none = make_float2(-INFINITY, 0.f);
      const float2 a = ntiles > 0 ? ml[r] : none, b = ntiles > 0 ? ml[PF_ROWS + r] : none;
      const float m = fmaxf(a.x, b.x);
      float wa = a.x == -INFINITY ? 0.f : ex2(a.x - m), wb = b.x == -INFINITY ? 0.f : ex2(b.x - m);
      const float total = a.y * wa + b.y * wb;
      float inv = total > 0.f ? 1.f / total : 0.f;
      if constexpr (F8) inv *= p.kv_scale;
      wa *= inv;
      wb *= inv;
      const long long rh = static_cast<long long>(x.row0 + tok) * p.hq + x.kvh * x.g + r % x.g;
      __nv_bfloat16* dst = p.out + rh * D;
      if (p.splits > 1 && row_ok && st == 0)
        p.part_lse[rh * p.splits + x.split] = total > 0.f ? m + log2f(total) : -INFINITY;
      const uint32_t o0 = tmem_base + 2 * KT + tlane, o1 = o0 + D;
#pragma unroll
      for (int c0 = st * (D / 2); c0 < (st + 1) * (D / 2); c0 += 32) {
        uint32_t u[32];
        float o[32];
        if (n0 > 0) {
          tmem_ld_32x32(o0 + c0, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = __uint_as_float(u[j]) * wa;
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = 0.f;
        }
        if (n1 > 0) {
          tmem_ld_32x32(o1 + c0, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = fmaf(__uint_as_float(u[j]), wb, o[j]);
        }
        if (row_ok && p.splits > 1) {
          float* part = p.part_o + (rh * p.splits + x.split) * D + c0;
#pragma unroll
          for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4*>(part + j) = make_float4(o[j], o[j + 1], o[j + 2], o[j + 3]);
        } else if (row_ok) {
#pragma unroll
          for (int j = 0; j < 32; j += 8)
            *reinterpret_cast<uint4*>(dst + c0 + j) = make_uint4(pack_bf16(o[j], o[j + 1]), pack_bf16(o[j + 2], o[j + 3]),
                                                                 pack_bf16(o[j + 4], o[j + 5]), pack_bf16(o[j + 6], o[j + 7]));
        }
      }
      tc_fence_before();
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == ISSUER) tmem_dealloc(tmem_base, 512);
}

// bf16 pools, head dims up to 128: two Q tiles per CTA. The kernel above reads every K / V tile for one tile of 128 packed rows
// (64 KB from L2 per 128 x 128 scores, near what L2 delivers if the softmax kept up), and the chain scores -> softmax -> P -> O of
// a stream left the tensor cores idle for four fifths of the time. Here the two streams are two Q tiles on the same K / V tiles:
// half the traffic, and no merge of accumulators at the end. Tiles are 64 keys, so that a stream has two score buffers in TMEM and the
// scores of the next tile are there before the softmax of this one ends: the softmax warps never wait for an MMA in the steady
// state. Q is loaded by the softmax warps while the producers fetch the first tiles, and the heaviest blocks of all heads and
// sequences start first. Bounds per 64 keys and pair of Q tiles: MMAs 1280 cycles (Q K^T reads 6 KB of shared memory per
// instruction), exponentials 1024; 1830 to 1930 are spent, 1330 of them in a softmax whose exponentials share their unit with the
// other stream's. One layer, 40 / 8 heads of 128: 2048 tokens 111 -> 62 us, from scattered slots 200 -> 75, five prompts of 4096
// 202 -> 104, 4096 tokens 313 -> 175, 2048 new ones over 8192 keys 465 -> 303; 32 / 32 heads of 64, 2048 tokens 75 -> 41; 29 tokens
// 13.1 -> 8.8.
// The reference of a row's weights: a weight that is the reference itself is 1 and has no rounding error, and it is the largest weights
// whose rounding to bf16 shows. So the reference follows the maximum exactly for the first 256 keys (what the two streams of the kernel
// above see first), afterwards in steps of 2^4. With the maximum of the first 64 keys and steps of 2^8 the error against 64 bits
// was up to 11 % above that kernel's, now it is the same or less. 40 / 8 heads of 128, queries times 1 / 1.5 / 3, 1e-3: 512 tokens,
// above 1.977 / 1.913 / 1.826, before 2.013 / 2.015 / 2.024, now 1.974 / 1.913 / 1.796; 2048 tokens 2.047 / 2.017 / 2.029,
// 2.084 / 2.107 / 2.145, 2.046 / 2.010 / 1.911 (rounding the result alone: 1.66). It costs 2048 tokens 61.8 -> 62.5 us, 512
// 17.4 -> 18.4, five prompts of 4096 102 -> 104.
constexpr int Q2_SETTLE = 4;      // tiles
constexpr float Q2_GAP = 4.f;     // log2
constexpr int Q2_KT = 64;
constexpr int Q2_STAGES = 4;      // tiles of the K and of the V ring
constexpr int Q2_THREADS = 512;   // warps 0-3 and 4-7 softmax, 8 and 9 fetch K, 10 and 11 V, 12 and 13 issue S = Q K^T, 14 and 15 O += P V
template <int D>
struct Q2Cfg {
  static constexpr int Q_TILE = PF_ROWS * D * 2;
  static constexpr int KV_TILE = Q2_KT * D * 2;
  static constexpr int BAR_OFF = 2 * Q_TILE + 2 * Q2_STAGES * KV_TILE;
  static constexpr int SMEM = BAR_OFF + 256 + 1024;
  static_assert((4 * Q2_STAGES + 13) * 8 + 8 <= 256, "barriers, TMEM address and abort flag");
  static_assert(SMEM <= 227 * 1024 && 4 * Q2_KT + 2 * D <= 512, "shared memory, TMEM");
};

// A CTA's two Q tiles: `tpb` tokens each from tok0 on, of which tile st has rows(st) packed rows and tiles(st) key tiles.
struct Q2Block {
  int g, b, kvh, tpb, row0, R, tok0, ctx, kmax, ntiles;
  int rows0, rows1, tiles0, tiles1;
  __device__ __forceinline__ int rows(int st) const { return st ? rows1 : rows0; }
  __device__ __forceinline__ int tiles(int st) const { return st ? tiles1 : tiles0; }
  __device__ __forceinline__ Q2Block(const PfParams& p) {
    g = p.hq / p.hkv;
    tpb = PF_ROWS / g;
    kvh = blockIdx.x;
    b = blockIdx.y;
    row0 = p.q_indptr ? p.q_indptr[b] : b;
    R = p.q_indptr ? p.q_indptr[b + 1] - row0 : 1;
    ctx = p.ctx_len[b];
    tok0 = static_cast<int>(gridDim.z - 1 - blockIdx.z) * 2 * tpb;       // heaviest (latest) blocks first
    const int n0 = max(0, min(tpb, R - tok0)), n1 = max(0, min(tpb, R - tok0 - tpb));
    const int vis0 = visible(p, tok0, n0), vis1 = visible(p, tok0 + tpb, n1);
    rows0 = n0 * g;
    rows1 = n1 * g;
    tiles0 = (vis0 + Q2_KT - 1) / Q2_KT;
    tiles1 = (vis1 + Q2_KT - 1) / Q2_KT;
    kmax = max(vis0, vis1);
    ntiles = max(tiles0, tiles1);
  }
  // keys that `n` tokens from `tok` on see
  __device__ __forceinline__ int visible(const PfParams& p, int tok, int n) const {
    return n > 0 ? max(0, p.causal ? min(ctx, ctx - R + tok + n) : ctx) : 0;
  }
};

// P of one row from its scores, written over them in TMEM; returns their sum. `rel` is the last visible column; WHOLE rows
// see all of them.
template <bool WHOLE>
__device__ __forceinline__ float q2_weights(const uint32_t (&v)[2][32], uint32_t s_t, int rel, float scale_log2, float neg_m) {
  const uint64_t scale2 = pack2(scale_log2, scale_log2), neg2 = pack2(neg_m, neg_m);
  uint64_t sum2[2] = {0ull, 0ull};
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    uint32_t w[16];
#pragma unroll
    for (int j = 0; j < 32; j += 2) {
      float p0, p1;
      unpack2(fma2(pack2(__uint_as_float(v[c][j]), __uint_as_float(v[c][j + 1])), scale2, neg2), p0, p1);
      p0 = WHOLE || c * 32 + j <= rel ? ex2(p0) : 0.f;
      p1 = WHOLE || c * 32 + j + 1 <= rel ? ex2(p1) : 0.f;
      sum2[(j >> 1) & 1] = add2(sum2[(j >> 1) & 1], pack2(p0, p1));
      w[j >> 1] = pack_bf16(p0, p1);
    }
    tmem_st_32x16(s_t + c * 32, w);
  }
  float a, b;
  unpack2(add2(sum2[0], sum2[1]), a, b);
  return a + b;
}

template <int D>
__global__ void __launch_bounds__(Q2_THREADS, 1)
attn_prefill_q2_kernel(const __grid_constant__ CUtensorMap tmk, const __grid_constant__ CUtensorMap tmv, const PfParams p) {
  grid_dep_launch();
  grid_dep_wait();
  using C = Q2Cfg<D>;
  constexpr int KT = Q2_KT, CPR = D / 8;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* ring = smem + 2 * C::Q_TILE;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::BAR_OFF);
  uint64_t* empty = full + 2 * Q2_STAGES;      // [K, V][stage], as `full`
  uint64_t* q_ready = empty + 2 * Q2_STAGES;
  uint64_t* s_ready = q_ready + 1;             // [stream][score buffer]
  // Softmax and issuers run up to a tile apart. A wait on a phase parity cannot tell phase n from n + 2, so the even and the odd
  // tiles of a stream have barriers of their own: the next phase of one (tile t + 2) cannot complete before tile t is through.
  uint64_t* p_ready = s_ready + 4;
  uint64_t* pv_done = p_ready + 4;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 4);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);   // warp-uniform for the compiler too
  const Q2Block x(p);
  if (x.rows0 <= 0) return;   // uniform: before any barrier or TMEM allocation

  if (tid == 256) {
    for (int i = 0; i < 2 * Q2_STAGES; ++i) {
      mbar_init(&full[i], 2);                  // one arrival per producer warp of a tile
      mbar_init(&empty[i], 2);                 // one per stream
    }
    mbar_init(q_ready, 256);
    for (int i = 0; i < 4; ++i) {
      mbar_init(&s_ready[i], 1);
      mbar_init(&p_ready[i], PF_ROWS);
      mbar_init(&pv_done[i], 1);
    }
    *abort = 0;
    fence_mbar_init();
    if (p.use_tma) {
      prefetch_tmap(&tmk);
      prefetch_tmap(&tmv);
    }
  }
  if (warp == 12) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  if (warp < 8) {      // Q rows, zero padded: row rr of tile st is (token tok0 + st * tpb + rr / g, head kvh * g + rr % g)
    const uint32_t inv_g = (65536u + x.g - 1) / x.g;      // rr * inv_g >> 16 == rr / g for rr < 128
#pragma unroll 4
    for (int i = 0; i < 2 * PF_ROWS * CPR / 256; ++i) {
      const int c = tid + i * 256, r = c / CPR, part = c % CPR, st = r >> 7, rr = r & 127;
      const uint32_t dst = smem_u32(smem + st * C::Q_TILE) + sw_off(rr, part, PF_ROWS);
      if (rr < x.rows(st)) {
        const int t = static_cast<int>(rr * inv_g >> 16);
        cp16(dst, p.q + (static_cast<long long>(x.row0 + x.tok0 + st * x.tpb + t) * p.hq + x.kvh * x.g + rr - t * x.g) * D +
                      part * 8);
      } else {
        st_zero16(dst);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

  if (warp >= 8 && warp < 12) {
    // ------------------------------------------------------------------ producers: K or V, half a tile (32 keys) per warp
    const bool is_v = warp >= 10;
    const int j = warp & 1;
    const __nv_bfloat16* pool = is_v ? p.v_pool : p.k_pool;
    const CUtensorMap* tm = is_v ? &tmv : &tmk;
    const int* idx_row = p.kv_indices + static_cast<long long>(p.seq_rows ? p.seq_rows[x.b] : x.b) * p.ld_idx;
    auto fetch_slot = [&](int t) {             // -1 beyond the visible keys
      const int key = t * KT + j * 32 + lane;
      return t < x.ntiles && key < x.kmax ? ld_step(idx_row + key) : -1;
    };
    auto place = [&](int t) { return (is_v ? Q2_STAGES : 0) + t % Q2_STAGES; };
    int slot = fetch_slot(0), next = fetch_slot(1);
    uint32_t late = 0;                         // bit i: the rows of tile t - i were gathered and have not been announced
    int done = 0;
    auto announce = [&](int t) {
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&full[place(t)]);
    };
    for (int t = 0; t < x.ntiles; ++t) {
      const int at = place(t);
      if (t >= Q2_STAGES && !warp_wait(&empty[at], (t / Q2_STAGES - 1) & 1, abort, p.status, kTimeoutEmpty)) break;
      uint8_t* tile = ring + at * C::KV_TILE;
      const int slot0 = __shfl_sync(0xffffffffu, slot, 0);
      const bool run = p.use_tma && __all_sync(0xffffffffu, slot >= 0 && slot == slot0 + lane);
      late <<= 1;
      if (run) {      // 32 consecutive pool rows: bulk tensor copies
        if (elect_one()) {
          mbar_expect_tx(&full[at], 32 * D * 2);
#pragma unroll
          for (int h = 0; h < D / 64; ++h)
            tma_load_2d(tile + h * (KT * 128) + j * (32 * 128), tm, &full[at], x.kvh * p.tma_xh + h * 64,
                        x.kvh * p.tma_yh + slot0);
        }
        __syncwarp();
      } else {        // fragmented pool, tail of the context: 16-byte copies, announced with the next tile
        constexpr int RPI = 32 / CPR;
        const int part = lane % CPR;
#pragma unroll 4
        for (int ii = 0; ii < 32 / RPI; ++ii) {
          const int rr = ii * RPI + lane / CPR;
          const int s1 = __shfl_sync(0xffffffffu, slot, rr);
          const uint32_t dst = smem_u32(tile) + sw_off(j * 32 + rr, part, KT);
          if (s1 >= 0)
            cp16(dst, pool + static_cast<long long>(s1) * p.pool_stride + x.kvh * p.head_stride + part * 8);
          else
            st_zero16(dst);
        }
        late |= 1;
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      if (late & 2) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        announce(t - 1);
      }
      slot = next;
      next = fetch_slot(t + 2);
      ++done;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");   // nothing may land after the CTA has gone
    if (done > 0 && (late & 1)) announce(done - 1);
    if (*abort) {      // nor may the bulk copies (bounded: a tile whose other half was never issued does not complete)
      volatile int ignore = 0;
      for (int t = max(done - Q2_STAGES, 0); t < done; ++t)
        mbar_wait(&full[place(t)], (t / Q2_STAGES) & 1, &ignore, nullptr, kTimeoutDrain);
    }
  } else if (warp >= 12) {
    // ------------------------------------------------------------------ MMA issuers: a stream's Q K^T or its P V
    // (One warp for both issued 1.6 times as slowly: an issue blocks while the pipe is busy, and a wait, passed or not, costs 100
    // cycles.) The other stream may see more tiles: those are only passed on.
    const int st = warp & 1, n = x.ntiles, mine = x.tiles(st);
    const uint32_t smem_a = __shfl_sync(0xffffffffu, smem_u32(smem), 0);
    const uint32_t ring_a = smem_a + 2 * C::Q_TILE, s_0 = tmem_base + st * 2 * KT, o_t = tmem_base + 4 * KT + st * D;
    if (warp < 14) {
      constexpr uint32_t idesc_qk = make_idesc_bf16(PF_ROWS, KT);
      const uint32_t q_a = smem_a + st * C::Q_TILE;
      bool ok = warp_wait(q_ready, 0, abort, p.status, kTimeoutFull);
      for (int t = 0; ok && t < n; ++t) {
        const int at = t % Q2_STAGES, sb = st * 2 + (t & 1);
        {
          PF_T0();
          ok = warp_wait(&full[at], (t / Q2_STAGES) & 1, abort, p.status, kTimeoutFull);
          PF_ACC(5, lane == 0 && st == 0);
        }
        // score buffer t % 2 holds P(t - 2) until that tile's O += P V is done
        if (ok && t >= 2 && t < mine) ok = warp_wait(&pv_done[sb], ((t >> 1) - 1) & 1, abort, p.status, kTimeoutAccum);
        if (!ok) break;
        if (t < mine) {
          tc_fence_after();
          const uint32_t k_a = ring_a + at * C::KV_TILE, s_t = s_0 + (t & 1) * KT;
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < D / 16; ++ks) {
              const uint32_t in_row = (ks & 3) * 32;   // 16 elements = 32 bytes inside the 128-byte swizzled row
              mma_f16(s_t, make_desc_sw128(q_a + (ks >> 2) * (PF_ROWS * 128) + in_row),
                      make_desc_sw128(k_a + (ks >> 2) * (KT * 128) + in_row), idesc_qk, ks > 0 ? 1u : 0u);
            }
            tc_commit(&empty[at]);
            tc_commit(&s_ready[sb]);
          }
        } else if (lane == 0) {
          mbar_arrive(&empty[at]);
        }
        __syncwarp();
      }
    } else {
      constexpr uint32_t idesc_pv = make_idesc_bf16(PF_ROWS, D, 0, 1);
      for (int t = 0; t < n; ++t) {
        const int at = Q2_STAGES + t % Q2_STAGES, sb = st * 2 + (t & 1);
        bool ok;
        {
          PF_T0();
          ok = warp_wait(&full[at], (t / Q2_STAGES) & 1, abort, p.status, kTimeoutFull);
          PF_ACC(4, lane == 0 && st == 0);
        }
        if (ok && t < mine) {
          PF_T0();
          ok = warp_wait(&p_ready[sb], (t >> 1) & 1, abort, p.status, kTimeoutAccum);
          PF_ACC(3, lane == 0 && st == 0);
        }
        if (!ok) break;
        if (t < mine) {
          tc_fence_after();
          const uint32_t v_a = ring_a + at * C::KV_TILE, s_t = s_0 + (t & 1) * KT;
          if (elect_one()) {
#pragma unroll
            for (int kk = 0; kk < KT / 16; ++kk)
              // 16 keys = two 8-row groups 1024 bytes apart; P: 8 columns of packed pairs per 16 keys
              mma_f16_ts(o_t, s_t + (kk >> 1) * 32 + (kk & 1) * 8, make_desc_sw128_mn(v_a + kk * 2048, KT * 128, 1024),
                         idesc_pv, (t > 0 || kk > 0) ? 1u : 0u);
            tc_commit(&empty[at]);
            tc_commit(&pv_done[sb]);
          }
        } else if (lane == 0) {
          mbar_arrive(&empty[at]);
        }
        __syncwarp();
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax and output of one stream
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    fence_proxy_async_smem();
    mbar_arrive(q_ready);
    const int st = warp >> 2;
    const int r = tid & (PF_ROWS - 1);                   // packed query row = TMEM lane
    const uint32_t tlane = static_cast<uint32_t>((warp & 3) * 32) << 16;
    const uint32_t s_0 = tmem_base + st * 2 * KT + tlane, o_t = tmem_base + 4 * KT + st * D + tlane;
    const bool row_ok = r < x.rows(st);
    const int tok = x.tok0 + st * x.tpb + r / x.g;
    const int mine = x.tiles(st);
    // last visible key position (inclusive); rows that are not there (zeros of Q) see everything: masking would keep their warp, and
    // with it the tile, on the slower path (128 x 64 scores of 125 rows: 2400 cycles, 1920 with 128 rows)
    const int lim = !row_ok ? 0x40000000 : p.causal ? x.ctx - x.R + tok : x.ctx - 1;
    float m_ref = -INFINITY, l = 0.f;   // O and l are relative to 2^m_ref
    bool ok = true;
    const long long t_begin = p.prof ? clock64() : 0;
    for (int t = 0; t < mine; ++t) {
      {
        PF_T0();
        ok = warp_wait(&s_ready[st * 2 + (t & 1)], (t >> 1) & 1, abort, p.status, kTimeoutAccum);
        PF_ACC(0, tid == 0);
      }
      if (!ok) break;
      tc_fence_after();
      const long long t_math = p.prof ? clock64() : 0;
      const uint32_t s_t = s_0 + (t & 1) * KT;
      uint32_t v[2][32];
      tmem_ld_32x32(s_t, v[0]);
      tmem_ld_32x32(s_t + 32, v[1]);
      // `rel` = last visible column of this tile for this row; a warp whose rows see the whole tile skips the masking.
      const int rel = lim - t * KT;
      const bool whole = __all_sync(0xffffffffu, rel >= KT - 1);
      tmem_ld_wait();
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      if (whole) {
#pragma unroll
        for (int j = 0; j < KT; ++j) mx4[j & 3] = fmaxf(mx4[j & 3], __uint_as_float(v[j >> 5][j & 31]));
      } else {
#pragma unroll
        for (int j = 0; j < KT; ++j)
          mx4[j & 3] = fmaxf(mx4[j & 3], j <= rel ? __uint_as_float(v[j >> 5][j & 31]) : -INFINITY);
      }
      const float m_tile = pf_reference<false>(fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])), p.scale_log2);
      if (t == 0) {
        m_ref = m_tile;
      } else if (__any_sync(0xffffffffu, m_tile > m_ref + (t < Q2_SETTLE ? 0.f : Q2_GAP))) {
        // Raise the reference (all lanes of the warp: tcgen05.ld / st are warp-wide) and rescale O and l, once O += P V of
        // the tile before has completed. The scores make room for 64 columns of O at a time and are read again.
        ok = warp_wait(&pv_done[st * 2 + ((t - 1) & 1)], ((t - 1) >> 1) & 1, abort, p.status, kTimeoutAccum);
        if (!ok) break;
        tc_fence_after();
        const float m_new = fmaxf(m_ref, m_tile);
        const float alpha = m_new == -INFINITY ? 1.f : ex2(m_ref - m_new);
        m_ref = m_new;
        l *= alpha;
#pragma unroll 1
        for (int c0 = 0; c0 < D; c0 += 64) {
          tmem_ld_32x32(o_t + c0, v[0]);
          tmem_ld_32x32(o_t + c0 + 32, v[1]);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 64; ++j) v[j >> 5][j & 31] = __float_as_uint(__uint_as_float(v[j >> 5][j & 31]) * alpha);
          tmem_st_32x32(o_t + c0, v[0]);
          tmem_st_32x32(o_t + c0 + 32, v[1]);
        }
        tmem_ld_32x32(s_t, v[0]);
        tmem_ld_32x32(s_t + 32, v[1]);
        tmem_ld_wait();
      }
      const float neg_m = m_ref == -INFINITY ? 0.f : -m_ref;
      l += whole ? q2_weights<true>(v, s_t, rel, p.scale_log2, neg_m) : q2_weights<false>(v, s_t, rel, p.scale_log2, neg_m);
      tmem_st_wait();
      if (p.prof && tid == 0) atomicAdd(p.prof + 13, (unsigned long long)(clock64() - t_math));
      tc_fence_before();
      mbar_arrive(&p_ready[st * 2 + (t & 1)]);
    }
    if (p.prof && tid == 0) {
      atomicAdd(p.prof + 10, (unsigned long long)(clock64() - t_begin));
      atomicAdd(p.prof + 11, (unsigned long long)mine);
    }
    if (ok && mine > 0) ok = warp_wait(&pv_done[st * 2 + ((mine - 1) & 1)], ((mine - 1) >> 1) & 1, abort, p.status, kTimeoutAccum);
    if (ok) {
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* dst = p.out + (static_cast<long long>(x.row0 + tok) * p.hq + x.kvh * x.g + r % x.g) * D;
#pragma unroll
      for (int c0 = 0; c0 < D; c0 += 32) {
        uint32_t o[32];
        if (mine > 0) {
          tmem_ld_32x32(o_t + c0, o);
          tmem_ld_wait();
        } else {                                         // no visible key
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = 0;
        }
        if (row_ok) {
#pragma unroll
          for (int j = 0; j < 32; j += 8)
            *reinterpret_cast<uint4*>(dst + c0 + j) =
                make_uint4(pack_bf16(__uint_as_float(o[j]) * inv, __uint_as_float(o[j + 1]) * inv),
                           pack_bf16(__uint_as_float(o[j + 2]) * inv, __uint_as_float(o[j + 3]) * inv),
                           pack_bf16(__uint_as_float(o[j + 4]) * inv, __uint_as_float(o[j + 5]) * inv),
                           pack_bf16(__uint_as_float(o[j + 6]) * inv, __uint_as_float(o[j + 7]) * inv));
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 12) tmem_dealloc(tmem_base, 512);
}

template <int D>
int launch_prefill_q2(const PfParams& p, const CUtensorMap* tk, const CUtensorMap* tv, int max_rows, int batch,
                      cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(attn_prefill_q2_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, Q2Cfg<D>::SMEM) !=
        cudaSuccess)
      return 3;
    attr = true;
  }
  const int tokens = 2 * (PF_ROWS / (p.hq / p.hkv));
  launch_dep(attn_prefill_q2_kernel<D>, dim3(p.hkv, batch, (max_rows + tokens - 1) / tokens), dim3(Q2_THREADS),
             Q2Cfg<D>::SMEM, st, *tk, *tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

template <int D, bool F8>
int launch_prefill_pp(const PfParams& p, const CUtensorMap* tk, const CUtensorMap* tv, int qblocks, int batch,
                      cudaStream_t st) {
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(attn_prefill_pp_kernel<D, F8>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             PpCfg<D, F8>::SMEM) != cudaSuccess)
      return 3;
    attr = true;
  }
  launch_dep(attn_prefill_pp_kernel<D, F8>, dim3(qblocks * p.splits, p.hkv, batch), dim3(PpRoles<F8>::THREADS), PpCfg<D, F8>::SMEM, st,
             *tk, *tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

template <int D, bool F8>
int launch_prefill(const PfParams& p, const CUtensorMap* tk, const CUtensorMap* tv, int qblocks, int batch,
                   cudaStream_t st) {
  using C = PfCfg<D, F8>;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(attn_prefill_kernel<D, F8>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) !=
        cudaSuccess)
      return 3;
    attr = true;
  }
  launch_dep(attn_prefill_kernel<D, F8>, dim3(qblocks * p.splits, p.hkv, batch), dim3(PfRoles<F8>::THREADS), C::SMEM, st, *tk, *tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace
}  // namespace hb

using namespace hb;

static unsigned long long* g_pf_prof = nullptr;

extern "C" {

// Cycle counters of the prefill kernel's roles: `buf` = 16 zeroed uint64 on the device (null switches it off).
// [0] softmax waits for scores, [1] softmax waits for the previous O update, [3] issuer waits for P,
// [4] issuer waits for V, [5] issuer waits for K, [6] / [7] producer waits for a free K / V stage,
// [8] producer issues copies, [9] producer waits for landed copies, [10] softmax loop total, [11] tiles,
// [12] softmax score load, [13] softmax math incl. the wait for the previous O update, [14] publish P.
void hb_attn_prefill_profile(void* buf) { g_pf_prof = static_cast<unsigned long long*>(buf); }

// Ring stage, full barrier and barrier parity of tile `t` in the two-stream kernel: place[0..2].
void hb_attn_prefill_place(int t, int* place) {
  const PpPlace at = pp_place(t);
  place[0] = at.stage;
  place[1] = at.full;
  place[2] = at.parity;
}

// bf16 KV with head dim 64, 128 or 256, or e4m3 KV (`kv_fp8`: x = code * kv_scale) with head dim 128 or 256, slot and head
// strides multiples of 16 and 16-byte aligned pools; group size hq / hkv <= 128. `max_rows` bounds the new rows of any
// sequence. With splits > 1 the context is cut into that many ranges of whole tiles, a CTA each, whose normalised
// partial rows and log2 sums go to part_o / part_lse for hb_attn_merge. splits = 1: one range, and bf16 pools with head dim 64 or
// 128 run two Q tiles per CTA where a sequence may have two; 0: one range, one Q tile per CTA.
int hb_attn_prefill(const void* q, const void* k_pool, const void* v_pool, long long pool_stride,
                    long long head_stride,
                    const void* kv_indices, long long ld_idx, const void* seq_rows, const void* ctx_len,
                    const void* q_indptr, void* out, void* part_o, void* part_lse, int splits, int batch, int max_rows,
                    int hq, int hkv, int d, float scale,
                    int kv_fp8, float kv_scale, int causal, long long pool_slots, void* status, void* stream) {
  if (batch <= 0 || max_rows <= 0) return 0;
  if (hq % hkv != 0 || hq / hkv > PF_ROWS) return 1;
  if (kv_fp8 && (pool_stride % 16 != 0 || head_stride % 16 != 0 ||
                 ((reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool)) & 15) != 0))
    return 1;
  PfParams p;
  p.q = static_cast<const __nv_bfloat16*>(q);
  p.k_pool = static_cast<const __nv_bfloat16*>(k_pool);
  p.v_pool = static_cast<const __nv_bfloat16*>(v_pool);
  p.pool_stride = pool_stride;
  p.head_stride = head_stride;
  p.kv_indices = static_cast<const int*>(kv_indices);
  p.ld_idx = ld_idx;
  p.seq_rows = static_cast<const int*>(seq_rows);
  p.ctx_len = static_cast<const int*>(ctx_len);
  p.q_indptr = static_cast<const int*>(q_indptr);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.part_o = static_cast<float*>(part_o);
  p.part_lse = static_cast<float*>(part_lse);
  p.splits = splits < 1 ? 1 : splits;
  if (p.splits > 1 && (part_o == nullptr || part_lse == nullptr)) return 1;
  p.hq = hq; p.hkv = hkv;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.kv_scale = kv_scale;
  p.causal = causal;
  p.status = static_cast<int*>(status);
  p.prof = g_pf_prof;
  const int tok_per_blk = PF_ROWS / (hq / hkv);
  const int qblocks = (max_rows + tok_per_blk - 1) / tok_per_blk;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  static const CUtensorMap dummy = {};
  const CUtensorMap *tk = &dummy, *tv = &dummy;
  if (kv_fp8) {      // producers load through registers: no tensor maps
    p.use_tma = p.tma_xh = p.tma_yh = 0;
    if (d == 128) return launch_prefill_pp<128, true>(p, tk, tv, qblocks, batch, st);
    if (d == 256) return launch_prefill<256, true>(p, tk, tv, qblocks, batch, st);
    return 1;
  }
  const KvTma t = make_kv_tma(k_pool, v_pool, pool_stride, head_stride, pool_slots, hkv, d, 32);
  p.use_tma = t.ok;
  p.tma_xh = t.xh;
  p.tma_yh = t.yh;
  if (t.ok) {
    tk = &t.k;
    tv = &t.v;
  }
  // two Q tiles per CTA: the caller knows whether there are enough of them (ops/attention.py, two_q_tiles)
  const bool q2 = splits == 1 && qblocks > 1 && batch <= 65535 && qblocks <= 2 * 65535;
  if (d == 64)
    return q2 ? launch_prefill_q2<64>(p, tk, tv, max_rows, batch, st) : launch_prefill_pp<64, false>(p, tk, tv, qblocks, batch, st);
  if (d == 128)
    return q2 ? launch_prefill_q2<128>(p, tk, tv, max_rows, batch, st) : launch_prefill_pp<128, false>(p, tk, tv, qblocks, batch, st);
  if (d == 256) return launch_prefill<256, false>(p, tk, tv, qblocks, batch, st);
  return 1;
}

}  // extern "C"
