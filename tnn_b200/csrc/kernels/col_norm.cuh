// Per-column normalisation with running statistics inside a product's epilogue: v * scale + shift, with
// scale = gamma / sqrt(var + eps) and shift = beta - mean * scale. One lane works out one column, and the 32 lanes of a warp hand
// theirs round: every lane of an epilogue warp has all 32 columns of its own row.
#pragma once
#include "ptx.cuh"

namespace tnnb {

struct ColNorm {
  const __nv_bfloat16 *gamma, *beta;  // or null: 1 and 0
  const float *mean, *var;
  float eps;
};

struct ColNormRaw {
  float gamma, beta, mean, var;
};

// The values of column `col` (those of an identity past N): loaded apart from their use, which may then come much later.
__device__ __forceinline__ ColNormRaw col_norm_load(const ColNorm& n, int col, int N) {
  ColNormRaw r = {1.f, 0.f, 0.f, 1.f};
  if (col < N) {
    if (n.gamma) r.gamma = __bfloat162float(n.gamma[col]);
    if (n.beta) r.beta = __bfloat162float(n.beta[col]);
    r.mean = n.mean[col];
    r.var = n.var[col];
  }
  return r;
}
__device__ __forceinline__ void col_norm_of(const ColNorm& n, const ColNormRaw& r, float& scale, float& shift) {
  scale = r.gamma * rsqrtf(r.var + n.eps);
  shift = r.beta - r.mean * scale;
}
__device__ __forceinline__ void col_norm(const ColNorm& n, int col, float& scale, float& shift) {
  col_norm_of(n, col_norm_load(n, col, col + 1), scale, shift);
}

// 32 columns of a row as pairs: lane k holds the scale and shift of column k.
__device__ __forceinline__ void col_norm_apply(uint64_t (&v)[16], float scale, float shift) {
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    const uint64_t sc = pack_f2(__shfl_sync(0xffffffffu, scale, 2 * k), __shfl_sync(0xffffffffu, scale, 2 * k + 1));
    const uint64_t sh = pack_f2(__shfl_sync(0xffffffffu, shift, 2 * k), __shfl_sync(0xffffffffu, shift, 2 * k + 1));
    v[k] = fma_f2(v[k], sc, sh);
  }
}

}  // namespace tnnb
