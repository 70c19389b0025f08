// Flash-decoding for paged GQA attention with up to 16 query rows per (sequence, kv head): decode (one token x
// GQA group <= 16) and short speculative verify blocks. Bandwidth-bound by design:
//
//   * K / V tiles of KT keys live in shared memory as 128-byte-swizzled column blocks ([KT rows x 128 bytes] per
//     64 head-dim elements), the layout a bulk tensor copy produces. The pool hands a sequence its slots in
//     ascending runs, so most tiles are KT consecutive pool rows and travel as one TMA box per column block
//     (row pitch = one pool slot): the TMA unit keeps far more bytes in flight than the LSU path, which tops out
//     near 16 KB outstanding per SM (~3.5 TB/s over the chip). Tiles that are not one run (fragmented pool, the
//     tail of the context) are gathered row by row with 16-byte cp.async into the same layout;
//   * each of the 4 warps of a CTA owns a private 3-stage ring of KT-key tiles and walks its own share of the keys,
//     so the main loop has no block-wide barrier and no flag wait: a warp waits only on its own cp.async groups;
//   * S = Q K^T and O += P V run on the tensor cores (m16n8k16 bf16, fp32 accumulate) with the query rows padded to
//     one 16-row tile; the online softmax lives in registers; the 4 warps' partial (m, l, O) merge through shared
//     memory at the end, and KV splits merge through the LSE kernel of attn.cu.
//
// e4m3 pools (F8): the tiles hold the codes, which expand to fp16 in registers on their way into the MMAs (exactly; two
// codes per conversion). The softmax weights enter O += P V times 2^15 as two fp16 terms, hi + lo: weights down to 2^-18 of
// the largest keep 22 bits, smaller ones are exact to 2^-40 of it (split_f16). Measured per layer against the CUDA-core kernel of attn.cu:
// 2 x 30011 keys, 40 / 8 heads of 128: 116 -> 36 us (3.4 TB/s); 16 x 8192, 32 / 2 heads: 180 -> 53 us; 4 x 5003, 24 / 4
// heads of 256: 102 -> 20 us.
//
// The KV range of a split is derived on the device from ctx_len, so one captured launch serves any context.
// Replaces the FlashInfer decode wrapper the reference plans per step (hibana/engine/graphs.py:55,
// hibana/engine/executor.py:161-169) and the multi-row verify kernel (hibana/kernels/csrc/verify_attn.cu:469).
#include "kv_tma.cuh"
#include "hb_api.h"
#include "hb_common.cuh"
#include "rownorm.cuh"

namespace hb {
namespace {

constexpr int DEC_STAGES = 3;

struct DecParams {
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
  float* part_o;
  float* part_lse;
  int hq, hkv, splits;
  float scale_log2;
  float kv_scale;             // dequantisation scale of an e4m3 pool (1 for bf16)
  int causal;
  int use_tma;
  int early;                  // tables, and keys before this forward's rows, are complete: see hb_attn_decode_early
  // Fused RoPE + KV write (see hb_attn_decode_rope): rows [Hq * D | Hkv * D | Hkv * D] of the projection, null = off
  const __nv_bfloat16* qkv;
  long long ld_qkv;
  const int* positions;
  const int* slots;
  const float* inv_freq;
  float kv_inv_scale;
  int* status;
  unsigned long long* prof;   // optional cycle counters of warp 0 (null = off)
  // Fused split merge: one int per (sequence, kv head), zero between launches. The CTA that finds splits - 1
  // earlier arrivals merges the partials of its (sequence, kv head) itself, so no merge kernel follows.
  int* split_counter;
  // Optional NVFP4 output of the merged (or unsplit) rows, the activation operand of the o projection:
  // q_out [rows, hq * D / 2] packed e2m1, q_sf swizzled ue4m3 scales, *q_gscale the static per-tensor scale.
  uint8_t* q_out;
  uint8_t* q_sf;
  const float* q_gscale;
  int q_ka;
};

__device__ __forceinline__ void ldsm_x4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void mma_f16_sync(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two e4m3 bytes -> two fp16 (exact; byte 0 in the low half).
__device__ __forceinline__ uint32_t e4m3x2_f16(uint32_t two) {
  uint32_t r;
  asm("{\n\t.reg .b16 t;\n\tcvt.u16.u32 t, %1;\n\tcvt.rn.f16x2.e4m3x2 %0, t;\n\t}" : "=r"(r) : "r"(two));
  return r;
}
// Softmax weights of two keys (at most 1) times 2^15 as fp16 pairs hi + lo. Without the factor, weights below 2^-14 would
// fall on the fp16 subnormal grid and those below 2^-25 vanish, although the row sum counts them: with one dominant key of
// small V over 30011 keys at 2^-24 the output was 2.5e-2 off, with it 2.5e-7 (fp32 weights: 1e-9; the output is bf16).
constexpr float kWeightScale = 32768.f, kWeightUnscale = 1.f / 32768.f;
__device__ __forceinline__ void split_f16(float a, float b, uint32_t* hi, uint32_t* lo) {
  a *= kWeightScale;
  b *= kWeightScale;
  const __half2 h = __floats2half2_rn(a, b);
  const __half2 l = __floats2half2_rn(a - __low2float(h), b - __high2float(h));
  *hi = *reinterpret_cast<const uint32_t*>(&h);
  *lo = *reinterpret_cast<const uint32_t*>(&l);
}

// Transposes an 8x8 matrix of 16-bit elements held one 32-bit pair per lane (the mma fragment layout).
__device__ __forceinline__ uint32_t movmatrix_trans(uint32_t a) {
  uint32_t d;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
  return d;
}

__device__ __forceinline__ void cp16(uint32_t saddr, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(saddr), "l"(g) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_wait2() { asm volatile("cp.async.wait_group 2;" ::: "memory"); }

template <int D, bool F8>
struct DecCfg {
  // Two CTAs share an SM: one streams while the other runs its prologue or merge. An e4m3 tile is half the bytes of a
  // bf16 one and twice the arithmetic per byte: twice the warps, the same bytes in flight.
  static constexpr int WARPS = F8 ? 4 : 2;
  static constexpr int THREADS = WARPS * 32;
  static constexpr int ESZ = F8 ? 1 : 2;
  static constexpr int KT = D >= 256 ? 16 : 32;        // keys per warp tile
  static constexpr int BLOCK_ELEMS = 128 / ESZ;         // elements of a 128-byte column block
  static constexpr int HALVES = D / BLOCK_ELEMS;        // column blocks per row
  static constexpr int BLOCK_BYTES = KT * 128;          // one column block of a tile
  static constexpr int TILE_BYTES = KT * D * ESZ;       // one of K or V
  static constexpr int STAGE_BYTES = 2 * TILE_BYTES;
  static constexpr int WARP_BYTES = DEC_STAGES * STAGE_BYTES;
  static constexpr int QROWB = D * 2 + 16;              // padded Q row: conflict-free ldmatrix
  static constexpr int Q_BYTES = 16 * QROWB;
  static constexpr int BAR_OFF = WARPS * WARP_BYTES + Q_BYTES;
  static constexpr int ROPE_OFF = BAR_OFF + 256;        // +0 barriers and abort flags, +128 row scales, +192 merge flag
  static constexpr int NEW_OFF = ROPE_OFF + D / 2 * 8;  // fused RoPE: the row's (cos, sin), then its new K and V rows
  static constexpr int SMEM = NEW_OFF + 2 * D * ESZ + 1024;
  static_assert(16 * D * 4 + 16 * 8 <= WARP_BYTES, "merge scratch must fit a warp's ring");
  static_assert(BLOCK_BYTES % 1024 == 0, "column blocks must keep the swizzle atom alignment");
};

// Byte offset of 16-byte chunk c of row `row` in a swizzled tile of KT rows.
template <int KT>
__device__ __forceinline__ uint32_t dsw(int row, int c) {
  return static_cast<uint32_t>((c >> 3) * (KT * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4));
}

// Chunk c (8 elements) of a row of head dim D at `src`, rotated by the angles cs[D / 2]: the arithmetic of rope_kv_write_kernel.
template <int D>
__device__ __forceinline__ void rope_chunk(const __nv_bfloat16* src, int c, const float2* cs, float (&o)[8]) {
  const bool low = c < D / 16;
  const int pc = low ? c + D / 16 : c - D / 16;
  const uint4 a = *reinterpret_cast<const uint4*>(src + c * 8), b = *reinterpret_cast<const uint4*>(src + pc * 8);
  float v[8], pv[8];
  unpack8(a, v);
  unpack8(b, pv);
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float2 t = cs[(low ? c : pc) * 8 + e];
    // (spelled out with the roundings that rope_kv_write_kernel has: left to the compiler they differ between kernels)
    o[e] = low ? __fmaf_rn(v[e], t.x, -__fmul_rn(pv[e], t.y)) : __fmaf_rn(pv[e], t.y, __fmul_rn(v[e], t.x));
  }
}

template <int D, bool T8, bool F8>
__global__ void __launch_bounds__(DecCfg<D, F8>::THREADS, 2)
attn_decode_kernel(const __grid_constant__ CUtensorMap tmk, const __grid_constant__ CUtensorMap tmv, const DecParams p) {
  using C = DecCfg<D, F8>;
  constexpr int DEC_WARPS = C::WARPS;
  grid_dep_launch();   // what follows (merge, output projection) waits for this grid before it reads anything
  // May run as a programmatic dependent of the RoPE + KV-write kernel. With `early` the tables and the tiles of keys that are
  // older than this forward are fetched before the wait: three round trips to L2 (lengths, slots, tiles) pass behind the
  // projection and the RoPE.
  if (!p.early) grid_dep_wait();
  constexpr int KT = C::KT, ROWB = C::QROWB;
  constexpr int NB = KT / 8;     // score n-blocks per tile
  constexpr int KS = D / 16;     // k-steps of Q K^T
  constexpr int ONB = D / 8;     // output n-blocks
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g4 = lane >> 2, t4 = lane & 3;
  uint8_t* ring = smem + warp * C::WARP_BYTES;
  uint8_t* qs = smem + DEC_WARPS * C::WARP_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::BAR_OFF) + warp * DEC_STAGES;   // this warp's barriers
  volatile int* abort = reinterpret_cast<volatile int*>(smem + C::BAR_OFF + DEC_WARPS * DEC_STAGES * 8) + warp;
  if (lane == 0) {
    for (int s = 0; s < DEC_STAGES; ++s) mbar_init(&full[s], 1);
    *abort = 0;
    fence_mbar_init();
  }

  const int b = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z;
  const int g = p.hq / p.hkv;
  const int row0 = p.q_indptr ? ldg_keep(p.q_indptr + b) : b;
  const int R = p.q_indptr ? ldg_keep(p.q_indptr + b + 1) - row0 : 1;
  const int nq = R * g;   // <= 16 guaranteed by the host
  const int ctx = ldg_keep(p.ctx_len + b);
  const int per = (((ctx + p.splits - 1) / p.splits + KT - 1) / KT) * KT;
  const int k0 = split * per;
  const int k1 = min(ctx, k0 + per);
  const int ntiles = k1 > k0 ? (k1 - k0 + KT - 1) / KT : 0;

  const int* idx_row = p.kv_indices + static_cast<long long>(p.seq_rows ? ldg_keep(p.seq_rows + b) : b) * p.ld_idx;

  // Issues the copies of this warp's `it`-th tile into its ring stage: one bulk tensor copy per column block of
  // K and of V when the tile's slots are KT consecutive pool rows, else a row-by-row cp.async gather. `tma_mode`
  // remembers per stage which way the tile in flight travels, `tma_phase` the parity of the stage's barrier.
  uint32_t tma_mode = 0, tma_phase = 0;
  // Slot id of key `lane` of this warp's tile `it` (-1 beyond the split). Fetched one tile ahead of its use so
  // that the index load's latency is not on the issue path.
  auto fetch_slot = [&](int it) -> int {
    const int base = k0 + (warp + it * DEC_WARPS) * KT;
    int slot = (warp + it * DEC_WARPS < ntiles && lane < KT && base + lane < k1) ? ldg_keep(idx_row + base + lane) : -1;
    if (slot >= 0 && !index_ok(slot, kBoundKvSlots, kKerAttnDecode)) slot = 0;   // reported; the dummy slot is read
    return slot;
  };
  auto issue = [&](int it, int my_slot) {
    const int tile = warp + it * DEC_WARPS;
    if (tile < ntiles) {
      const int st = it % DEC_STAGES;
      const int base = k0 + tile * KT;
      uint8_t* kt = ring + st * C::STAGE_BYTES;
      const uint32_t kdst = smem_u32(kt);
      const uint32_t vdst = kdst + C::TILE_BYTES;
      constexpr int CPR = D * C::ESZ / 16;  // 16-byte chunks per row
      constexpr int RPI = 32 / CPR > 0 ? 32 / CPR : 1;   // rows per warp instruction
      const int slot0 = __shfl_sync(0xffffffffu, my_slot, 0);
      const bool run = p.use_tma && __all_sync(0xffffffffu, lane >= KT || (my_slot >= 0 && my_slot == slot0 + lane));
      if (run) {
        tma_mode |= 1u << st;
        // lane 0 posts the byte count, then 2 * HALVES lanes issue one box each (K / V x column block)
        if (lane == 0) mbar_expect_tx(&full[st], 2 * C::TILE_BYTES);
        __syncwarp();
        if (lane < 2 * C::HALVES) {
          const int h = lane >> 1, is_v = lane & 1;
          tma_load_2d(kt + is_v * C::TILE_BYTES + h * C::BLOCK_BYTES, is_v ? &tmv : &tmk, &full[st],
                      kvh * p.tma_xh + h * C::BLOCK_ELEMS, kvh * p.tma_yh + slot0);
        }
      } else {
        tma_mode &= ~(1u << st);
        if constexpr (CPR <= 32) {
          const int part = lane % CPR, sub = lane / CPR;
#pragma unroll
          for (int r = 0; r < KT; r += RPI) {
            const int key = r + sub;
            const int slot = __shfl_sync(0xffffffffu, my_slot, key);
            const uint32_t so = dsw<KT>(key, part);
            if (slot >= 0) {
              const long long off = (static_cast<long long>(slot) * p.pool_stride +
                                     static_cast<long long>(kvh) * p.head_stride) * C::ESZ + part * 16;
              cp16(kdst + so, reinterpret_cast<const uint8_t*>(p.k_pool) + off);
              cp16(vdst + so, reinterpret_cast<const uint8_t*>(p.v_pool) + off);
            } else {
              asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(kdst + so), "r"(0) : "memory");
              asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};" ::"r"(vdst + so), "r"(0) : "memory");
            }
          }
        }
      }
    }
    cp_commit();
  };

  __syncwarp();      // this warp's barriers are initialised
  int issued = 0;
  const bool rope = p.qkv != nullptr;
  float2* cs = reinterpret_cast<float2*>(smem + C::ROPE_OFF);
  uint8_t* fresh = smem + C::NEW_OFF;                       // the new token's K row, then its V row, as the pool holds them
  const bool owns_new = rope && ntiles > 0 && k1 == ctx;    // this range ends with the new token
  if (p.early) {
    // Tiles that end before this forward's rows (a tile past the range issues nothing). With fused RoPE the one new row is put
    // into its tile by this CTA, so that no tile has to wait.
    while (issued < 2 && (rope || min(k1, k0 + (warp + issued * DEC_WARPS + 1) * KT) <= ctx - R)) {
      issue(issued, fetch_slot(issued));
      ++issued;
    }
    if (rope) {
      const float pos = static_cast<float>(ldg_keep(p.positions + b));
      for (int j = tid; j < D / 2; j += DEC_WARPS * 32) {
        float sn, co;
        sincosf(pos * p.inv_freq[j], &sn, &co);
        cs[j] = make_float2(co, sn);
      }
      __syncthreads();
    }
    grid_dep_wait();
  }
  if (owns_new) {      // K and V of the new token: into the pool and, for this CTA's own tile, into shared memory
    const __nv_bfloat16* krow = p.qkv + b * p.ld_qkv + (p.hq + kvh) * D;
    int slot = ldg_keep(p.slots + b);
    if (slot >= 0 && !index_ok(slot, kBoundKvSlots, kKerRopeKvWrite)) slot = -1;   // reported; nothing is written
    for (int i = tid; i < 2 * (D / 8); i += DEC_WARPS * 32) {
      const bool is_v = i >= D / 8;
      const int c = is_v ? i - D / 8 : i;
      float f[8];
      if (is_v) unpack8(*reinterpret_cast<const uint4*>(krow + p.hkv * D + c * 8), f);
      else rope_chunk<D>(krow, c, cs, f);
      uint8_t* pool = const_cast<uint8_t*>(reinterpret_cast<const uint8_t*>(is_v ? p.v_pool : p.k_pool)) +
                      (static_cast<long long>(slot) * p.pool_stride + static_cast<long long>(kvh) * p.head_stride) * C::ESZ;
      if constexpr (F8) {
        uint32_t w[2] = {0, 0};
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e >> 2] |= float_to_e4m3(f[e] * p.kv_inv_scale) << (8 * (e & 3));
        *reinterpret_cast<uint2*>(fresh + (is_v ? D : 0) + c * 8) = make_uint2(w[0], w[1]);
        if (slot >= 0) *reinterpret_cast<uint2*>(pool + c * 8) = make_uint2(w[0], w[1]);
      } else {
        const uint4 v = pack8(f);
        *reinterpret_cast<uint4*>(fresh + (is_v ? 2 * D : 0) + c * 16) = v;
        if (slot >= 0) *reinterpret_cast<uint4*>(pool + c * 16) = v;
      }
    }
  }

  // Q rows (zero padded to 16) into shared memory. For an e4m3 pool Q becomes fp16, the type K and V expand to
  // exactly: every row is scaled by a power of two that takes its largest element to [2^14, 2^15), so all that is more
  // than 2^-31 of the largest keeps its eight significant bits; the inverse factor joins the softmax scale.
  float* row_scale = reinterpret_cast<float*>(smem + C::BAR_OFF + 128);
  for (int i = tid; i < 16 * (D / 8); i += DEC_WARPS * 32) {
    const int qi = i / (D / 8), c = i % (D / 8);
    uint4 v = make_uint4(0, 0, 0, 0);
    if (qi < nq) {
      const int rr = qi / g, gg = qi % g;
      if (rope) {
        float f[8];
        rope_chunk<D>(p.qkv + b * p.ld_qkv + (kvh * g + gg) * D, c, cs, f);
        v = pack8(f);
      } else {
        v = *reinterpret_cast<const uint4*>(p.q + (static_cast<long long>(row0 + rr) * p.hq + kvh * g + gg) * D + c * 8);
      }
    }
    if constexpr (F8) {
      uint32_t w[4] = {v.x, v.y, v.z, v.w};
      // bit pattern of the largest magnitude (a whole row sits in D / 8 = 16 or 32 consecutive lanes)
      uint32_t mx = 0;
#pragma unroll
      for (int e = 0; e < 4; ++e) mx = max(mx, max(w[e] & 0x7FFFu, (w[e] >> 16) & 0x7FFFu));
#pragma unroll
      for (int sh = 1; sh < D / 8; sh <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, sh));
      const int e2 = static_cast<int>(mx >> 7) - 127;          // exponent of the largest element
      const int up = mx == 0 || e2 > 127 ? 0 : min(14 - e2, 126);
      const float f = __uint_as_float(static_cast<uint32_t>(127 + max(up, -126)) << 23);
      if (c == 0) row_scale[qi] = __uint_as_float(static_cast<uint32_t>(127 - max(up, -126)) << 23);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const __half2 h = __floats2half2_rn(bf16_lo(w[e]) * f, bf16_hi(w[e]) * f);
        w[e] = *reinterpret_cast<const uint32_t*>(&h);
      }
      v = make_uint4(w[0], w[1], w[2], w[3]);
    }
    *reinterpret_cast<uint4*>(qs + qi * ROWB + c * 16) = v;
  }
  __syncthreads();

  // Up to 8 query rows (T8): the tile math runs transposed, S^T = K Q^T and O^T = V^T P^T, so the keys (resp. the
  // head dim) take the 16-row side of m16n8k16 and the query rows its 8 columns: half the MMAs of the 16-row
  // form. Q is then the B operand (n = query row, k = head dim).
  uint32_t qf[T8 ? 1 : KS][4];
  uint32_t qb[T8 ? KS : 1][2];
  if constexpr (F8) {
    // The contraction index of Q K^T is permuted inside each block of 16 head dims so that a thread's four K bytes
    // are one 32-bit word: positions 2 t4, 2 t4 + 1 | 2 t4 + 8, 2 t4 + 9 stand for dims 4 t4 .. 4 t4 + 3.
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) {
      const uint2 a = *reinterpret_cast<const uint2*>(qs + g4 * ROWB + (ks * 16 + 4 * t4) * 2);
      if constexpr (T8) {
        qb[ks][0] = a.x;
        qb[ks][1] = a.y;
      } else {
        const uint2 b2 = *reinterpret_cast<const uint2*>(qs + (g4 + 8) * ROWB + (ks * 16 + 4 * t4) * 2);
        qf[ks][0] = a.x;
        qf[ks][1] = b2.x;
        qf[ks][2] = a.y;
        qf[ks][3] = b2.y;
      }
    }
  } else if constexpr (!T8) {
    const uint32_t base = smem_u32(qs) + ((lane & 7) + ((lane >> 3) & 1) * 8) * ROWB + (lane >> 4) * 16;
#pragma unroll
    for (int ks = 0; ks < KS; ++ks) ldsm_x4(qf[ks], base + ks * 32);
  } else {
    const uint32_t base = smem_u32(qs) + (lane & 7) * ROWB + (lane >> 3) * 16;
#pragma unroll
    for (int ks = 0; ks < KS; ks += 2) {
      uint32_t r[4];
      ldsm_x4(r, base + ks * 32);
      qb[ks][0] = r[0];
      qb[ks][1] = r[1];
      qb[ks + 1][0] = r[2];
      qb[ks + 1][1] = r[3];
    }
  }

  // 16-row form: o[n-block][4], rows g4 / g4 + 8. Transposed form: o[16-wide head-dim block][4] = (d g4 | g4 + 8)
  // x (query rows 2 t4, 2 t4 + 1); "lo" / "hi" then name those two query rows.
  constexpr int OB = T8 ? D / 16 : ONB;
  float o[OB][4];
#pragma unroll
  for (int i = 0; i < OB; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
  float m_lo = -INFINITY, m_hi = -INFINITY, l_lo = 0.f, l_hi = 0.f;
  // Causal limits of this thread's two rows (keys [0, limit) visible).
  const int row_lo = T8 ? 2 * t4 : g4, row_hi = T8 ? 2 * t4 + 1 : g4 + 8;
  const int lim_lo = p.causal ? ctx - R + (row_lo / g) + 1 : ctx;
  const int lim_hi = p.causal ? ctx - R + (row_hi / g) + 1 : ctx;
  const float scale_lo = F8 ? p.scale_log2 * p.kv_scale * row_scale[row_lo] : p.scale_log2;
  const float scale_hi = F8 ? p.scale_log2 * p.kv_scale * row_scale[row_hi] : p.scale_log2;

  const bool prof = p.prof != nullptr && tid == 0;
  const long long t_start = prof ? clock64() : 0;
  long long c_issue = 0, c_wait = 0, c_math = 0;
  for (; issued < 2; ++issued) issue(issued, fetch_slot(issued));
  int slot_next = fetch_slot(2);
  for (int it = 0; warp + it * DEC_WARPS < ntiles; ++it) {
    // Stage (it + 2) % 3 was read in iteration it - 1: every lane is past it, order it before the async writes.
    __syncwarp();
    long long t0 = prof ? clock64() : 0;
    issue(it + 2, slot_next);
    slot_next = fetch_slot(it + 3);
    long long t1 = prof ? clock64() : 0;
    cp_wait2();
    const int st = it % DEC_STAGES;
    if (tma_mode & (1u << st)) {
      const bool got = mbar_wait(&full[st], (tma_phase >> st) & 1u, abort, p.status, kTimeoutFull);
      tma_phase ^= 1u << st;
      if (!__all_sync(0xffffffffu, got)) break;
    }
    __syncwarp();
    const long long t2 = prof ? clock64() : 0;
    c_issue += t1 - t0;
    c_wait += t2 - t1;
    c_math -= t2;
    const uint32_t kbase = smem_u32(ring + st * C::STAGE_BYTES);
    const uint32_t vbase = kbase + C::TILE_BYTES;
    const int tile = warp + it * DEC_WARPS;
    const int kpos0 = k0 + tile * KT;
    if (owns_new && tile == ntiles - 1) {      // the new token's row over what the copy found in its slot
      constexpr int CPR = D * C::ESZ / 16;
      uint8_t* dst = ring + st * C::STAGE_BYTES;
      for (int i = lane; i < 2 * CPR; i += 32) {
        const int c = i % CPR, is_v = i / CPR;
        *reinterpret_cast<uint4*>(dst + is_v * C::TILE_BYTES + dsw<KT>(ctx - 1 - kpos0, c)) =
            *reinterpret_cast<const uint4*>(fresh + i * 16);
      }
      __syncwarp();
    }

    if constexpr (!T8) {
    float s[NB][4];
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
        if constexpr (F8) {
#pragma unroll
          for (int ks = 0; ks < KS; ks += 4) {
            uint32_t kb[4];
            ldsm_x4(kb, kbase + dsw<KT>(j * 8 + (lane & 7), ks + (lane >> 3)));
#pragma unroll
            for (int i = 0; i < 4; ++i)
              mma_f16_sync(s[j], qf[ks + i], e4m3x2_f16(kb[i]), e4m3x2_f16(kb[i] >> 16));
          }
        } else
#pragma unroll
        for (int ks = 0; ks < KS; ks += 2) {
          uint32_t kb[4];
          ldsm_x4(kb, kbase + dsw<KT>(j * 8 + (lane & 7), ks * 2 + (lane >> 3)));
          mma_bf16(s[j], qf[ks], kb[0], kb[1]);
          mma_bf16(s[j], qf[ks + 1], kb[2], kb[3]);
        }
      }
      float mx_lo = -INFINITY, mx_hi = -INFINITY;
#pragma unroll
      for (int j = 0; j < NB; ++j) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int kp = kpos0 + j * 8 + 2 * t4 + e;
          const bool in = kp < k1;
          s[j][e] = (in && kp < lim_lo) ? s[j][e] * scale_lo : -INFINITY;
          s[j][2 + e] = (in && kp < lim_hi) ? s[j][2 + e] * scale_hi : -INFINITY;
          mx_lo = fmaxf(mx_lo, s[j][e]);
          mx_hi = fmaxf(mx_hi, s[j][2 + e]);
        }
      }
      mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 1));
      mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, 2));
      mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 1));
      mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, 2));
      const float mn_lo = fmaxf(m_lo, mx_lo), mn_hi = fmaxf(m_hi, mx_hi);
      const float a_lo = mn_lo == -INFINITY ? 1.f : exp2f(m_lo - mn_lo);
      const float a_hi = mn_hi == -INFINITY ? 1.f : exp2f(m_hi - mn_hi);
      m_lo = mn_lo;
      m_hi = mn_hi;
      l_lo *= a_lo;
      l_hi *= a_hi;
      uint32_t pf[NB / 2][4];
      uint32_t pl[F8 ? NB / 2 : 1][4];   // low halves of the fp16 weights
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const float p0 = mn_lo == -INFINITY ? 0.f : exp2f(s[j][0] - mn_lo);
        const float p1 = mn_lo == -INFINITY ? 0.f : exp2f(s[j][1] - mn_lo);
        const float p2 = mn_hi == -INFINITY ? 0.f : exp2f(s[j][2] - mn_hi);
        const float p3 = mn_hi == -INFINITY ? 0.f : exp2f(s[j][3] - mn_hi);
        l_lo += p0 + p1;
        l_hi += p2 + p3;
        if constexpr (F8) {
          split_f16(p0, p1, &pf[j >> 1][(j & 1) * 2], &pl[j >> 1][(j & 1) * 2]);
          split_f16(p2, p3, &pf[j >> 1][(j & 1) * 2 + 1], &pl[j >> 1][(j & 1) * 2 + 1]);
        } else {
          pf[j >> 1][(j & 1) * 2] = pack_bf16(p0, p1);
          pf[j >> 1][(j & 1) * 2 + 1] = pack_bf16(p2, p3);
        }
      }
#pragma unroll
      for (int nb = 0; nb < ONB; ++nb) {
        o[nb][0] *= a_lo;
        o[nb][1] *= a_lo;
        o[nb][2] *= a_hi;
        o[nb][3] *= a_hi;
      }
#pragma unroll
      for (int kk = 0; kk < KT / 16; ++kk) {
        if constexpr (F8) {
          // A transposing load hands a thread the bytes of dims 2 g4, 2 g4 + 1 of two keys: accumulator blocks
          // 2 c and 2 c + 1 are the even and the odd dims of 16-dim block c.
#pragma unroll
          for (int c = 0; c < D / 16; c += 2) {
            uint32_t vw[4];
            ldsm_x4_t(vw, vbase + dsw<KT>(kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, c + (lane >> 4)));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint32_t w0 = __byte_perm(vw[2 * i], 0, 0x3120), w1 = __byte_perm(vw[2 * i + 1], 0, 0x3120);
              const uint32_t e0 = e4m3x2_f16(w0), e1 = e4m3x2_f16(w1);
              const uint32_t o0 = e4m3x2_f16(w0 >> 16), o1 = e4m3x2_f16(w1 >> 16);
              mma_f16_sync(o[2 * (c + i)], pf[kk], e0, e1);
              mma_f16_sync(o[2 * (c + i) + 1], pf[kk], o0, o1);
              mma_f16_sync(o[2 * (c + i)], pl[kk], e0, e1);
              mma_f16_sync(o[2 * (c + i) + 1], pl[kk], o0, o1);
            }
          }
        } else
#pragma unroll
        for (int nb = 0; nb < ONB; nb += 2) {
          uint32_t vb[4];
          ldsm_x4_t(vb, vbase + dsw<KT>(kk * 16 + ((lane >> 3) & 1) * 8 + (lane & 7), nb + (lane >> 4)));
          mma_bf16(o[nb], pf[kk], vb[0], vb[1]);
          mma_bf16(o[nb + 1], pf[kk], vb[2], vb[3]);
        }
      }
    } else {
      constexpr int MT = KT / 16;   // 16-key blocks of the tile
      float st[MT][4];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        st[mt][0] = st[mt][1] = st[mt][2] = st[mt][3] = 0.f;
        if constexpr (F8) {
#pragma unroll
          for (int ks = 0; ks < KS; ks += 2) {
            uint32_t kw[4];
            ldsm_x4(kw, kbase + dsw<KT>(mt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, ks + (lane >> 4)));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint32_t ka[4] = {e4m3x2_f16(kw[2 * i]), e4m3x2_f16(kw[2 * i + 1]), e4m3x2_f16(kw[2 * i] >> 16),
                                      e4m3x2_f16(kw[2 * i + 1] >> 16)};
              mma_f16_sync(st[mt], ka, qb[ks + i][0], qb[ks + i][1]);
            }
          }
        } else
#pragma unroll
        for (int ks = 0; ks < KS; ++ks) {
          uint32_t ka[4];
          ldsm_x4(ka, kbase + dsw<KT>(mt * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, ks * 2 + (lane >> 4)));
          mma_bf16(st[mt], ka, qb[ks][0], qb[ks][1]);
        }
      }
      // st[mt] = {key g4: rows lo, hi | key g4 + 8: rows lo, hi} of key block mt
      float mx_lo = -INFINITY, mx_hi = -INFINITY;
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int kp = kpos0 + mt * 16 + g4 + 8 * e;
          const bool in = kp < k1;
          st[mt][2 * e] = (in && kp < lim_lo) ? st[mt][2 * e] * scale_lo : -INFINITY;
          st[mt][2 * e + 1] = (in && kp < lim_hi) ? st[mt][2 * e + 1] * scale_hi : -INFINITY;
          mx_lo = fmaxf(mx_lo, st[mt][2 * e]);
          mx_hi = fmaxf(mx_hi, st[mt][2 * e + 1]);
        }
      }
#pragma unroll
      for (int sh = 4; sh < 32; sh <<= 1) {   // keys live across the g4 lane groups
        mx_lo = fmaxf(mx_lo, __shfl_xor_sync(0xffffffffu, mx_lo, sh));
        mx_hi = fmaxf(mx_hi, __shfl_xor_sync(0xffffffffu, mx_hi, sh));
      }
      const float mn_lo = fmaxf(m_lo, mx_lo), mn_hi = fmaxf(m_hi, mx_hi);
      const float a_lo = mn_lo == -INFINITY ? 1.f : exp2f(m_lo - mn_lo);
      const float a_hi = mn_hi == -INFINITY ? 1.f : exp2f(m_hi - mn_hi);
      m_lo = mn_lo;
      m_hi = mn_hi;
      l_lo *= a_lo;
      l_hi *= a_hi;
      uint32_t pb[MT][2];   // P^T as B operand: (k = key, n = query row)
      uint32_t pl[F8 ? MT : 1][2];
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float p0 = mn_lo == -INFINITY ? 0.f : exp2f(st[mt][2 * e] - mn_lo);
          const float p1 = mn_hi == -INFINITY ? 0.f : exp2f(st[mt][2 * e + 1] - mn_hi);
          l_lo += p0;
          l_hi += p1;
          if constexpr (F8) {
            uint32_t hi, lo;
            split_f16(p0, p1, &hi, &lo);
            pb[mt][e] = movmatrix_trans(hi);
            pl[mt][e] = movmatrix_trans(lo);
          } else {
            pb[mt][e] = movmatrix_trans(pack_bf16(p0, p1));
          }
        }
      }
#pragma unroll
      for (int ob = 0; ob < OB; ++ob) {
        o[ob][0] *= a_lo;
        o[ob][1] *= a_hi;
        o[ob][2] *= a_lo;
        o[ob][3] *= a_hi;
      }
#pragma unroll
      for (int kk = 0; kk < MT; ++kk) {
        if constexpr (F8) {
          // rows g4 and g4 + 8 of accumulator block ob are dims 2 g4 and 2 g4 + 1 of 16-dim block ob
#pragma unroll
          for (int ob = 0; ob < OB; ob += 2) {
            uint32_t vw[4];
            ldsm_x4_t(vw, vbase + dsw<KT>(kk * 16 + (lane & 7) + ((lane >> 3) & 1) * 8, ob + (lane >> 4)));
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const uint32_t w0 = __byte_perm(vw[2 * i], 0, 0x3120), w1 = __byte_perm(vw[2 * i + 1], 0, 0x3120);
              const uint32_t va[4] = {e4m3x2_f16(w0), e4m3x2_f16(w0 >> 16), e4m3x2_f16(w1), e4m3x2_f16(w1 >> 16)};
              mma_f16_sync(o[ob + i], va, pb[kk][0], pb[kk][1]);
              mma_f16_sync(o[ob + i], va, pl[kk][0], pl[kk][1]);
            }
          }
        } else
#pragma unroll
        for (int ob = 0; ob < OB; ++ob) {
          uint32_t va[4];   // V^T block (16 head-dim x 16 keys) through transposing loads
          ldsm_x4_t(va, vbase + dsw<KT>(kk * 16 + ((lane >> 4) & 1) * 8 + (lane & 7), ob * 2 + ((lane >> 3) & 1)));
          mma_bf16(o[ob], va, pb[kk][0], pb[kk][1]);
        }
      }
    }
    if (prof) c_math += clock64();
  }
  const long long t_loop_end = prof ? clock64() : 0;
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  // ---- merge the 4 warps through each warp's own (now idle) ring
  float* mo = reinterpret_cast<float*>(ring);          // [16][D]
  float* ml = mo + 16 * D;                             // [16][2] (m, l)
  if constexpr (!T8) {
    // Row sums live split over the 4 threads of a row group.
    l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 1);
    l_lo += __shfl_xor_sync(0xffffffffu, l_lo, 2);
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 1);
    l_hi += __shfl_xor_sync(0xffffffffu, l_hi, 2);
    if constexpr (F8) {
#pragma unroll
      for (int c = 0; c < D / 16; ++c) {
        *reinterpret_cast<float4*>(mo + g4 * D + c * 16 + 4 * t4) =
            make_float4(o[2 * c][0], o[2 * c + 1][0], o[2 * c][1], o[2 * c + 1][1]);
        *reinterpret_cast<float4*>(mo + (g4 + 8) * D + c * 16 + 4 * t4) =
            make_float4(o[2 * c][2], o[2 * c + 1][2], o[2 * c][3], o[2 * c + 1][3]);
      }
    } else
#pragma unroll
    for (int nb = 0; nb < OB; ++nb) {
      *reinterpret_cast<float2*>(mo + g4 * D + nb * 8 + 2 * t4) = make_float2(o[nb][0], o[nb][1]);
      *reinterpret_cast<float2*>(mo + (g4 + 8) * D + nb * 8 + 2 * t4) = make_float2(o[nb][2], o[nb][3]);
    }
    if (t4 == 0) {
      ml[g4 * 2] = m_lo;
      ml[g4 * 2 + 1] = l_lo;
      ml[(g4 + 8) * 2] = m_hi;
      ml[(g4 + 8) * 2 + 1] = l_hi;
    }
  } else {
    // Row sums live split over the 8 lane groups that hold different keys.
#pragma unroll
    for (int sh = 4; sh < 32; sh <<= 1) {
      l_lo += __shfl_xor_sync(0xffffffffu, l_lo, sh);
      l_hi += __shfl_xor_sync(0xffffffffu, l_hi, sh);
    }
    if constexpr (F8) {
#pragma unroll
      for (int ob = 0; ob < OB; ++ob) {
        *reinterpret_cast<float2*>(mo + row_lo * D + ob * 16 + 2 * g4) = make_float2(o[ob][0], o[ob][2]);
        *reinterpret_cast<float2*>(mo + row_hi * D + ob * 16 + 2 * g4) = make_float2(o[ob][1], o[ob][3]);
      }
    } else
#pragma unroll
    for (int ob = 0; ob < OB; ++ob) {
      mo[row_lo * D + ob * 16 + g4] = o[ob][0];
      mo[row_hi * D + ob * 16 + g4] = o[ob][1];
      mo[row_lo * D + ob * 16 + g4 + 8] = o[ob][2];
      mo[row_hi * D + ob * 16 + g4 + 8] = o[ob][3];
    }
    if (g4 == 0) {
      ml[row_lo * 2] = m_lo;
      ml[row_lo * 2 + 1] = l_lo;
      ml[row_hi * 2] = m_hi;
      ml[row_hi * 2 + 1] = l_hi;
    }
  }
  __syncthreads();
  const bool fused_merge = p.splits > 1 && p.split_counter != nullptr;
  const bool direct = p.splits == 1;
  // NVFP4 output goes through `fin` (the Q tile's shared memory: Q lives in registers by now) so that one thread
  // owns a whole 16-element group; values are rounded to bf16 first, as the separate quantiser would see them.
  __nv_bfloat16* fin = reinterpret_cast<__nv_bfloat16*>(qs);
  {
    for (int i = tid; i < nq * D; i += DEC_WARPS * 32) {
      const int qi = i / D, d = i % D;
      float mt = -INFINITY;
#pragma unroll
      for (int w = 0; w < DEC_WARPS; ++w)
        mt = fmaxf(mt, reinterpret_cast<const float*>(smem + w * C::WARP_BYTES)[16 * D + qi * 2]);
      float acc = 0.f, lt = 0.f;
      if (mt > -INFINITY) {
#pragma unroll
        for (int w = 0; w < DEC_WARPS; ++w) {
          const float* wo = reinterpret_cast<const float*>(smem + w * C::WARP_BYTES);
          const float mw = wo[16 * D + qi * 2];
          const float sc = mw == -INFINITY ? 0.f : exp2f(mw - mt);
          acc += sc * wo[qi * D + d];
          lt += sc * wo[16 * D + qi * 2 + 1];
        }
      }
      float val = lt > 0.f ? acc / lt : 0.f;
      if constexpr (F8) val *= p.kv_scale * kWeightUnscale;
      const int rr = qi / g, gg = qi % g;
      const long long rh = static_cast<long long>(row0 + rr) * p.hq + kvh * g + gg;
      if (direct) {
        if (p.q_out == nullptr) p.out[rh * D + d] = __float2bfloat16(val);
        else fin[i] = __float2bfloat16(val);
      } else {
        p.part_o[(rh * p.splits + split) * D + d] = val;
        if (d == 0) p.part_lse[rh * p.splits + split] = lt > 0.f ? mt + log2f(lt) : -INFINITY;
      }
    }
  }
  bool finish = direct && p.q_out != nullptr;
  if (fused_merge) {
    // Last arriver of this (sequence, kv head) merges: every CTA publishes its partial (fence, then one counted
    // arrival); the one that counts splits - 1 before it re-arms the counter and reads all partials back from L2.
    int* last_flag = reinterpret_cast<int*>(smem + C::BAR_OFF + 192);
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      int* cnt = p.split_counter + b * p.hkv + kvh;
      const int old = atomicAdd(cnt, 1);
      const int last = old == p.splits - 1;
      if (last) *cnt = 0;
      *last_flag = last;
    }
    __syncthreads();
    if (*last_flag) {
      __threadfence();
      // The merge is latency-bound (a few hundred values per CTA, every one a chain of L2 reads), so the reads are
      // batched: all log-sum-exps of this (sequence, kv head) land in shared memory in one round trip, then every
      // thread keeps four outputs in flight per pass over the splits.
      float* lse_s = reinterpret_cast<float*>(smem);          // [nq][splits], the rings are idle
      const int S = p.splits;
      for (int i = tid; i < nq * S; i += DEC_WARPS * 32) {
        const int qi = i / S, s2 = i - qi * S;
        const long long rh = static_cast<long long>(row0 + qi / g) * p.hq + kvh * g + qi % g;
        lse_s[i] = __ldcg(p.part_lse + rh * S + s2);
      }
      __syncthreads();
      constexpr int V = 4;
      for (int base = 0; base < nq * D; base += V * DEC_WARPS * 32) {
        float o[V], mx[V], wsum[V];
        long long rhv[V];
        int qv[V], dv[V];
        bool live[V];
#pragma unroll
        for (int v = 0; v < V; ++v) {
          const int i = base + v * DEC_WARPS * 32 + tid;
          live[v] = i < nq * D;
          qv[v] = live[v] ? i / D : 0;
          dv[v] = live[v] ? i % D : 0;
          rhv[v] = static_cast<long long>(row0 + qv[v] / g) * p.hq + kvh * g + qv[v] % g;
          float m = -INFINITY;
          for (int s2 = 0; s2 < S; ++s2) m = fmaxf(m, lse_s[qv[v] * S + s2]);
          mx[v] = m;
          o[v] = 0.f;
          wsum[v] = 0.f;
        }
#pragma unroll 2
        for (int s2 = 0; s2 < S; ++s2) {
          float x[V];
#pragma unroll
          for (int v = 0; v < V; ++v) x[v] = live[v] ? __ldcg(p.part_o + (rhv[v] * S + s2) * D + dv[v]) : 0.f;
#pragma unroll
          for (int v = 0; v < V; ++v) {
            const float w = mx[v] > -INFINITY ? exp2f(lse_s[qv[v] * S + s2] - mx[v]) : 0.f;
            if (w > 0.f) o[v] += w * x[v];
            wsum[v] += w;
          }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
          if (!live[v]) continue;
          const float r = wsum[v] > 0.f ? o[v] / wsum[v] : 0.f;
          const int i = base + v * DEC_WARPS * 32 + tid;
          if (p.q_out == nullptr) p.out[rhv[v] * D + dv[v]] = __float2bfloat16(r);
          else fin[i] = __float2bfloat16(r);
        }
      }
      finish = p.q_out != nullptr;
    }
  }
  if (finish) {
    __syncthreads();
    const float inv_gs = 1.f / *p.q_gscale;
    constexpr int GPR = D / 16;   // groups per (row, head)
    for (int it = tid; it < nq * GPR; it += DEC_WARPS * 32) {
      const int qi = it / GPR, gi = it % GPR;
      float x[16];
      load16(fin + qi * D + gi * 16, x);
      uint2 packed;
      const uint32_t sfb = quant16(x, inv_gs, &packed);
      const int rr = qi / g, gg = qi % g;
      const int row = row0 + rr, head = kvh * g + gg;
      *reinterpret_cast<uint2*>(p.q_out + (static_cast<size_t>(row) * p.hq + head) * (D / 2) + gi * 8) = packed;
      p.q_sf[row_sf_off(row, head * GPR + gi, p.q_ka)] = static_cast<uint8_t>(sfb);
    }
  }
  if (prof) {
    const long long t_end = clock64();
    atomicAdd(p.prof + 0, static_cast<unsigned long long>(c_issue));
    atomicAdd(p.prof + 1, static_cast<unsigned long long>(c_wait));
    atomicAdd(p.prof + 2, static_cast<unsigned long long>(c_math));
    atomicAdd(p.prof + 3, static_cast<unsigned long long>(t_loop_end - t_start));
    atomicAdd(p.prof + 4, static_cast<unsigned long long>(t_end - t_loop_end));
    atomicAdd(p.prof + 5, static_cast<unsigned long long>((ntiles + DEC_WARPS - 1 - warp) / DEC_WARPS));
    atomicAdd(p.prof + 6, 1ull);
  }
}

template <int D, bool T8, bool F8>
int launch_decode(const DecParams& p0, const void* k_pool, const void* v_pool, long long pool_slots, int batch,
                  cudaStream_t st) {
  DecParams p = p0;
  using C = DecCfg<D, F8>;
  static bool attr = false;
  if (!attr) {
    if (cudaFuncSetAttribute(attn_decode_kernel<D, T8, F8>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM) !=
        cudaSuccess)
      return 3;
    attr = true;
  }
  static const CUtensorMap dummy = {};
  const CUtensorMap *tk = &dummy, *tv = &dummy;
  const KvTma t = make_kv_tma(k_pool, v_pool, p.pool_stride, p.head_stride, pool_slots, p.hkv, D, C::KT, C::ESZ);
  p.use_tma = t.ok;
  p.tma_xh = t.xh;
  p.tma_yh = t.yh;
  if (t.ok) {
    tk = &t.k;
    tv = &t.v;
  }
  launch_dep(attn_decode_kernel<D, T8, F8>, dim3(batch, p.hkv, p.splits), dim3(C::THREADS), C::SMEM, st, *tk, *tv, p);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // namespace
}  // namespace hb

using namespace hb;

static unsigned long long* g_dec_prof = nullptr;
struct DecFuse {
  int* counter = nullptr;
  void* q_out = nullptr;
  void* q_sf = nullptr;
  const void* q_gscale = nullptr;
  int q_ka = 0;
};
static thread_local DecFuse g_dec_fuse;
static thread_local int g_dec_early = 0;
struct DecRope {
  const void *qkv = nullptr, *positions = nullptr, *slots = nullptr, *inv_freq = nullptr;
  long long ld = 0;
  float kv_inv_scale = 1.f;
};
static thread_local DecRope g_dec_rope;

extern "C" {

// Cycle counters of warp 0 of every CTA, summed: `buf` = 8 zeroed uint64 on the device (null switches it off).
// [0] issuing copies, [1] waiting for a tile, [2] tile math, [3] main loop, [4] merge + store, [5] tiles of warp 0,
// [6] CTAs.
void hb_attn_decode_profile(void* buf) { g_dec_prof = static_cast<unsigned long long*>(buf); }

// Arms the fused tail for the NEXT hb_attn_decode call of this thread (consumed by that call): `split_counter`
// (one zeroed int per sequence x kv head, re-armed by the kernel) makes the last-arriving split CTA merge the
// partials, so no hb_attn_merge follows; q_out / q_sf / q_gscale (may be null) make the kernel write the rows as
// NVFP4 instead of bf16 (`out` is then not written).
void hb_attn_decode_fuse(void* split_counter, void* q_out, void* q_sf, const void* q_gscale, int q_ka) {
  g_dec_fuse.counter = static_cast<int*>(split_counter);
  g_dec_fuse.q_out = q_out; g_dec_fuse.q_sf = q_sf; g_dec_fuse.q_gscale = q_gscale; g_dec_fuse.q_ka = q_ka;
}

// Promises, for the NEXT hb_attn_decode call of this thread, that its tables (block table, context lengths, row offsets) and the keys
// and values in front of every sequence's last rows were complete before the forward began, and that a kernel which triggers
// its successor only after its own wait (the embedding gather) ran since: the kernel may then read them ahead of its wait.
void hb_attn_decode_early(void) { g_dec_early = 1; }

// RoPE and KV write inside the NEXT hb_attn_decode call of this thread (with hb_attn_decode_early, one row per sequence): row b of
// `qkv` [Hq * D | Hkv * D | Hkv * D] is rotated over all of D at positions[b], its K and V go to slots[b] (whose place in the
// block table is the sequence's last) and take part in the attention from shared memory; `q` is not read. 16-byte aligned rows
// of qkv and of the pools; `kv_inv_scale` as hb_rope_kv_write has it. The separate kernel was 4.4 us of every layer's chain.
void hb_attn_decode_rope(const void* qkv, long long ld_qkv, const void* positions, const void* slots, const void* inv_freq,
                         float kv_inv_scale) {
  g_dec_rope.kv_inv_scale = kv_inv_scale;
  g_dec_rope.qkv = qkv; g_dec_rope.ld = ld_qkv; g_dec_rope.positions = positions; g_dec_rope.slots = slots;
  g_dec_rope.inv_freq = inv_freq;
}

// bf16 KV, or e4m3 (`kv_fp8`: x = code * kv_scale; head dim 128 or 256, slot and head strides multiples of 16, 16-byte
// aligned pools); rows_per_seq * (hq / hkv) must be <= 16. Partials go through hb_attn_merge when splits > 1 unless
// hb_attn_decode_fuse armed the in-kernel merge.
int hb_attn_decode(const void* q, const void* k_pool, const void* v_pool, long long pool_stride,
                   long long head_stride,
                   const void* kv_indices, long long ld_idx, const void* seq_rows, const void* ctx_len,
                   const void* q_indptr, void* out, void* part_o, void* part_lse, int batch, int max_rows, int hq,
                   int hkv, int d, int splits, float scale, int kv_fp8, float kv_scale, int causal, long long pool_slots,
                   void* status, void* stream) {
  const int early = g_dec_early;
  g_dec_early = 0;
  const DecRope rope = g_dec_rope;
  g_dec_rope = DecRope{};
  if (batch <= 0) return 0;
  if (kv_fp8 && (pool_stride % 16 != 0 || head_stride % 16 != 0 ||
                 ((reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool)) & 15) != 0))
    return 1;
  if (hq % hkv != 0 || max_rows * (hq / hkv) > 16) return 1;
  DecParams p;
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
  p.hq = hq; p.hkv = hkv; p.splits = splits < 1 ? 1 : splits;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.kv_scale = kv_fp8 ? kv_scale : 1.f;
  p.causal = causal;
  p.status = static_cast<int*>(status);
  p.prof = g_dec_prof;
  p.split_counter = g_dec_fuse.counter;
  p.q_out = static_cast<uint8_t*>(g_dec_fuse.q_out);
  p.q_sf = static_cast<uint8_t*>(g_dec_fuse.q_sf);
  p.q_gscale = static_cast<const float*>(g_dec_fuse.q_gscale);
  p.q_ka = g_dec_fuse.q_ka;
  g_dec_fuse = DecFuse{};
  p.early = early;
  p.qkv = static_cast<const __nv_bfloat16*>(rope.qkv);
  p.ld_qkv = rope.ld;
  p.positions = static_cast<const int*>(rope.positions);
  p.slots = static_cast<const int*>(rope.slots);
  p.inv_freq = static_cast<const float*>(rope.inv_freq);
  p.kv_inv_scale = rope.kv_inv_scale;
  if (p.qkv != nullptr) {
    const int align = kv_fp8 ? 16 : 8;      // pool strides are in elements
    if (!early || q_indptr != nullptr || max_rows != 1 || p.slots == nullptr || p.positions == nullptr || p.inv_freq == nullptr ||
        rope.ld % 8 != 0 || (reinterpret_cast<uintptr_t>(rope.qkv) & 15) != 0 || pool_stride % align != 0 ||
        head_stride % align != 0 || ((reinterpret_cast<uintptr_t>(k_pool) | reinterpret_cast<uintptr_t>(v_pool)) & 15) != 0)
      return 1;
  }
  if (p.q_out != nullptr && p.splits > 1 && p.split_counter == nullptr) return 1;
  if (p.splits > 1 && (part_o == nullptr || part_lse == nullptr)) return 1;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool t8 = max_rows * (hq / hkv) <= 8;
  if (kv_fp8) {
    if (d == 128) return t8 ? launch_decode<128, true, true>(p, k_pool, v_pool, pool_slots, batch, st)
                            : launch_decode<128, false, true>(p, k_pool, v_pool, pool_slots, batch, st);
    if (d == 256) return t8 ? launch_decode<256, true, true>(p, k_pool, v_pool, pool_slots, batch, st)
                            : launch_decode<256, false, true>(p, k_pool, v_pool, pool_slots, batch, st);
    return 1;
  }
  if (d == 64) return t8 ? launch_decode<64, true, false>(p, k_pool, v_pool, pool_slots, batch, st)
                         : launch_decode<64, false, false>(p, k_pool, v_pool, pool_slots, batch, st);
  if (d == 128) return t8 ? launch_decode<128, true, false>(p, k_pool, v_pool, pool_slots, batch, st)
                          : launch_decode<128, false, false>(p, k_pool, v_pool, pool_slots, batch, st);
  if (d == 256) return t8 ? launch_decode<256, true, false>(p, k_pool, v_pool, pool_slots, batch, st)
                          : launch_decode<256, false, false>(p, k_pool, v_pool, pool_slots, batch, st);
  return 1;
}

}  // extern "C"
