// K ranges in a cluster: S = 2 or 4 CTAs of a cluster have each multiplied the same 128 x 128 tile over its own range of K
// blocks; every CTA then adds up the S partial sums of its W = 128 / S columns in the order of the ranges. The partial sums
// travel through distributed shared memory into a buffer of the owner, [S ranges][128 rows][W columns] fp32 (64 KB, in the
// operand stages) with its 16-byte chunks swizzled by row, so that neither the lanes' row-wise stores nor the loads of the
// owner meet in a bank.
//
// Order of calls, by all threads of all CTAs of the cluster:
//   MMAs finished -> cluster_sync_all() -> ranges_push -> cluster_sync_all() -> ranges_sum
// The first barrier says that no operand stage of the cluster is read any more, the second that all partial sums have landed
// (and no CTA leaves while a neighbour writes to it).
#pragma once
#include "ptx.cuh"

namespace tnnb {

// Epilogue warp (TMEM lane quarter q, column half `half` of the 128): 32 rows x 64 columns to their owners.
__device__ __forceinline__ void ranges_push(uint32_t buf, uint32_t tmem, int rank, int W, int q, int half, int lane) {
  const int row = q * 32 + lane, swz = row & 7;
  const uint32_t mine = buf + (uint32_t)(rank * 128 + row) * (W * 4);
#pragma unroll 1
  for (int c = 0; c < 2; ++c) {
    const int c0 = half * 64 + c * 32;
    uint32_t r[32];
    tmem_ld_32x32_wait(tmem + (static_cast<uint32_t>(q * 32) << 16) + c0, r);  // warp-collective
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const int col = c0 + g * 4, owner = col / W, chunk = (col - owner * W) >> 2;
      const uint32_t dst = mapa_shared(mine + ((chunk ^ swz) << 4), owner);
      asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst), "r"(r[4 * g]), "r"(r[4 * g + 1]), "r"(r[4 * g + 2]),
                   "r"(r[4 * g + 3])
                   : "memory");
    }
  }
}

// Row q * 32 + lane, columns half * 32 .. + 31 of the owner's W: the sum over all ranges.
__device__ __forceinline__ void ranges_sum(const uint8_t* buf, int ranges, int W, int q, int half, int lane, uint32_t (&r)[32]) {
  const int row = q * 32 + lane, swz = row & 7;
  float acc[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) acc[k] = 0.f;
#pragma unroll 1
  for (int s = 0; s < ranges; ++s) {
    const uint8_t* src = buf + (s * 128 + row) * (W * 4);
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      const float4 v = *reinterpret_cast<const float4*>(src + (((half * 8 + g) ^ swz) << 4));
      acc[4 * g] += v.x, acc[4 * g + 1] += v.y, acc[4 * g + 2] += v.z, acc[4 * g + 3] += v.w;
    }
  }
#pragma unroll
  for (int k = 0; k < 32; ++k) r[k] = __float_as_uint(acc[k]);
}

}  // namespace tnnb
