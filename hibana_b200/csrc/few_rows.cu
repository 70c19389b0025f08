// bf16 projection of up to 16 rows: out[t, f] = sum_k x[t, k] * w[f, k], fp32 accumulation, bf16 or fp32 out.
//
// For the small bf16 matrices of a decode step (routers, latent projections, gate projections: 1 to 32 MB) a tcgen05 tile is
// mostly set-up: tensor maps, barriers, TMEM, split-K clusters. Here a CTA owns 16 features; its warps take K in turns of 32 elements,
// weights straight from memory into mma.sync fragments (the contraction index is permuted inside a step so that a lane's
// share is one 16-byte load per row; the same for x), DEPTH steps in flight, the first of them before the wait for the kernel
// that produces x. Partial sums meet in shared memory, warp by warp. Bound by the latency of a few dependent loads and the launch,
// not by bytes; so as much of K as possible is in flight at once.
//
// In a chain of launches, tcgen05 / this, us: 512 x 4096 5.8 / 3.1 (1 row), 1024 x 4096 6.0 / 3.3, 2048 x 2048 5.3 / 2.9, 4096 x 1024
// 5.5 / 3.4, 4096 x 4096 9.5 / 7.8; 16 rows 6.0 / 5.3, 6.2 / 5.5, 5.7 / 3.5, 5.6 / 3.5, 9.8 / 11. Relative error against 64 bits (fp32
// accumulation in both): 512 x 4096 4.9e-7 / 1.4e-7 at 1 row, 4.8e-7 / 2.4e-7 at 16; 4096 x 1024 1.7e-7 / 0.9e-7; 256 x 1000, whose K the
// tcgen05 form cuts finer than these warps do, 1.3e-7 / 1.3e-7 (2.3e-7 with one accumulator).
#include "hb_api.h"
#include "hb_common.cuh"

namespace hb {
namespace {

constexpr int FEATS = 16;

__device__ __forceinline__ void mma_bf16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
      "{%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NB = blocks of 8 rows of x. SPLIT CTAs (a cluster) share a block of features, each with its turns of K; the first adds their sums up.
template <int NB, int WARPS, int DEPTH, int SPLIT = 1>
__global__ void __launch_bounds__(WARPS * 32)
few_rows_kernel(const __nv_bfloat16* x, long long ldx, const __nv_bfloat16* __restrict__ w, long long ldw, int m, int n, int k,
                void* out, long long ldo, int f32) {
  __shared__ float red[WARPS][8 * NB][FEATS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g4 = lane >> 2, t4 = lane & 3;
  __shared__ float parts[SPLIT][SPLIT > 1 ? 8 * NB * FEATS : 1];     // of the first CTA: the sums of each
  const int part = SPLIT > 1 ? blockIdx.x % SPLIT : 0, turn = part * WARPS + warp;
  const int f0 = blockIdx.x / SPLIT * FEATS;
  const int kl = (turn * 4 + t4) * 8;                       // this lane's first element of its warp's first step
  constexpr int STRIDE = SPLIT * WARPS * 32;                // elements between two steps of a warp
  const int steps = k > turn * 32 ? (k - turn * 32 + STRIDE - 1) / STRIDE : 0;
  const uint4 zero = make_uint4(0, 0, 0, 0);
  auto weights = [&](int i, int half) -> uint4 {
    const int f = f0 + g4 + 8 * half, kk = kl + i * STRIDE;
    return f < n && kk < k ? __ldg(reinterpret_cast<const uint4*>(w + f * ldw + kk)) : zero;
  };
  auto rows = [&](int i, int blk) -> uint4 {
    const int t = blk * 8 + g4, kk = kl + i * STRIDE;
    return t < m && kk < k ? ld_step(reinterpret_cast<const uint4*>(x + t * ldx + kk)) : zero;
  };
  uint4 a[DEPTH][2], b[DEPTH][NB];
  grid_dep_launch();
  if (SPLIT > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");     // (its shared memory may be written)
#pragma unroll
  for (int i = 0; i < DEPTH; ++i) {
    a[i][0] = weights(i, 0);
    a[i][1] = weights(i, 1);
  }
  grid_dep_wait();
#pragma unroll
  for (int i = 0; i < DEPTH; ++i)
#pragma unroll
    for (int q = 0; q < NB; ++q) b[i][q] = rows(i, q);
  float acc[2][NB][4];       // of the even and the odd instructions: the longer a chain, the more its fp32 additions lose
#pragma unroll
  for (int q = 0; q < 2 * NB; ++q) acc[q & 1][q >> 1][0] = acc[q & 1][q >> 1][1] = acc[q & 1][q >> 1][2] = acc[q & 1][q >> 1][3] = 0.f;
  for (int i0 = 0; i0 < steps; i0 += DEPTH) {
#pragma unroll
    for (int i = 0; i < DEPTH; ++i) {
      // (steps past the end multiply zeros)
#pragma unroll
      for (int q = 0; q < NB; ++q) {
        mma_bf16(acc[0][q], a[i][0].x, a[i][1].x, a[i][0].y, a[i][1].y, b[i][q].x, b[i][q].y);
        mma_bf16(acc[1][q], a[i][0].z, a[i][1].z, a[i][0].w, a[i][1].w, b[i][q].z, b[i][q].w);
      }
      if (i0 + DEPTH < steps) {
        a[i][0] = weights(i0 + DEPTH + i, 0);
        a[i][1] = weights(i0 + DEPTH + i, 1);
#pragma unroll
        for (int q = 0; q < NB; ++q) b[i][q] = rows(i0 + DEPTH + i, q);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < NB; ++q)
#pragma unroll
    for (int e = 0; e < 4; ++e) red[warp][q * 8 + 2 * t4 + (e & 1)][g4 + 8 * (e >> 1)] = acc[0][q][e] + acc[1][q][e];
  __syncthreads();
  auto sum = [&](int i) {
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < WARPS; ++j) s += red[j][i / FEATS][i % FEATS];
    return s;
  };
  auto store = [&](int i, float s) {
    const int t = i / FEATS, f = f0 + i % FEATS;
    if (f >= n) return;
    if (f32) static_cast<float*>(out)[t * ldo + f] = s;
    else static_cast<__nv_bfloat16*>(out)[t * ldo + f] = __float2bfloat16(s);
  };
  if constexpr (SPLIT == 1) {
    for (int i = threadIdx.x; i < m * FEATS; i += WARPS * 32) store(i, sum(i));
  } else {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    for (int i = threadIdx.x; i < m * FEATS; i += WARPS * 32) {
      const float s = sum(i);
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(map_to_cta(smem_u32(&parts[part][i]), 0)), "f"(s) : "memory");
    }
    cluster_sync_all();
    if (part == 0)
      for (int i = threadIdx.x; i < m * FEATS; i += WARPS * 32) {
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < SPLIT; ++j) s += parts[j][i];
        store(i, s);
      }
  }
}

}  // namespace
}  // namespace hb

using namespace hb;

extern "C" {

// x [m <= 16, k], w [n, k] bf16 with row pitches ldx, ldw; k and the pitches multiples of 8, both 16-byte aligned. `f32`: out is fp32.
int hb_few_rows_bf16(const void* x, long long ldx, const void* w, long long ldw, int m, int n, int k, void* out, long long ldo,
                     int f32, void* stream) {
  if (m < 1 || m > 16 || n < 1 || k < 1 || k % 8 != 0 || ldx % 8 != 0 || ldw % 8 != 0 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w)) & 15) != 0)
    return 1;
  // One wave of CTAs: sixteen warps take 4096 elements of K at once. More CTAs (or 9 to 16 rows, whose fragments of x take registers):
  // eight warps, several CTAs to an SM. A matrix of a megabyte runs beside a larger projection on a parallel branch: four warps
  // (12K to 16K registers) find room next to its CTAs of 192 threads, sixteen would wait until that projection has left the SM, which put
  // 11 us a layer on the critical path of the delta rule's gates.
  // From 2048 elements of K on eight CTAs share a block of features, all of K in flight at once: beside the projection, which
  // keeps the memory busy, each round of loads takes 3 us, and the gates of 4 rows (96 x 5120) left 5 us after the convolution.
  const int ctas = (n + FEATS - 1) / FEATS;
  const bool small = static_cast<long long>(n) * k <= (1 << 19);
  const int split = small && k >= 2048 ? 8 : 1;
  auto kern = split > 1 ? (m <= 8 ? few_rows_kernel<1, 4, 8, 8> : few_rows_kernel<2, 4, 4, 8>)
              : small ? (m <= 8 ? few_rows_kernel<1, 4, 8> : few_rows_kernel<2, 4, 4>)
              : m <= 8 ? (ctas <= 148 && k > 1024 ? few_rows_kernel<1, 16, 8> : few_rows_kernel<1, 8, 8>)
                       : (k > 1024 ? few_rows_kernel<2, 8, 8> : few_rows_kernel<2, 8, 4>);
  const int warps = small ? 4 : m <= 8 && ctas <= 148 && k > 1024 ? 16 : 8;
  launch_dep_cluster(kern, dim3(ctas * split), dim3(warps * 32), split, 0, static_cast<cudaStream_t>(stream),
                     static_cast<const __nv_bfloat16*>(x), ldx, static_cast<const __nv_bfloat16*>(w), ldw, m, n, k, out, ldo, f32);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

}  // extern "C"
