// NHWC convolution support kernels and pooling.
//
// Convolutions run on the tcgen05 GEMM (gemm_tcgen05.cu): 1x1 / stride-1 layers are
// a GEMM over the activation tensor as it is; every other geometry goes through
// the patch matrices built here:
//   im2col   cols[(n,oh,ow), (kh,kw,c)] = x[n, oh*s+kh-p, ow*s+kw-p, c]  (0 outside)
//   col2im   dx[n,h,w,c] = sum over the taps (kh,kw) that read pixel (h,w) of
//            dcols[(n,oh,ow),(kh,kw,c)]   - a gather, so no atomics
// Weights [O,KH,KW,C] are already the [O, K] operand of that GEMM.
// Semantics follow the reference CPU engine (src/nn/engines/cpu_engine.cpp:617-734,
// pools :66-210; average pooling divides by the in-image count as in
// src/nn/engines/cuda_engine.cu:141-194). The reference calls cuDNN conv graphs
// (cudnn_engine.cu:328-578) and scatter kernels with atomics for the pool backward.
#include "ptx.cuh"

TNNB_BOUNDS_TU(conv_pool)

namespace tnnb {

typedef __nv_bfloat16 bf16;

struct ConvGeo {
  int N, H, W, C, KH, KW, SH, SW, PH, PW, OH, OW;
  int Kld;  // row pitch of the patch matrix in elements (>= KH*KW*C, multiple of 8)
};

// VEC = 8: C % 8 == 0, one 16-byte move per thread. VEC = 1 (any C, e.g. the 3-channel stem): each thread still
// writes one 16-byte group of eight consecutive columns of the row (Kld % 8 == 0), gathering its eight elements
// with scalar loads - the write side, which is the larger one, stays coalesced.
template <int VEC>
__global__ void im2col_kernel(const bf16* __restrict__ x, bf16* __restrict__ cols, ConvGeo g) {
  if (VEC == 8) {
    const int cv = g.C / 8;
    const long long per_row = (long long)g.KH * g.KW * cv;
    const long long total = (long long)g.N * g.OH * g.OW * per_row;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
      const int c = (int)(i % cv);
      long long r = i / cv;
      const int kw = (int)(r % g.KW); r /= g.KW;
      const int kh = (int)(r % g.KH); r /= g.KH;
      const long long pix = r;  // (n, oh, ow)
      const int ow = (int)(pix % g.OW);
      const int oh = (int)((pix / g.OW) % g.OH);
      const int n = (int)(pix / ((long long)g.OW * g.OH));
      const int ih = oh * g.SH + kh - g.PH, iw = ow * g.SW + kw - g.PW;
      const long long doff = pix * g.Kld + ((long long)(kh * g.KW + kw) * g.C) + c * 8;
      if (!TNNB_CHECK(doff + 7, (long long)g.N * g.OH * g.OW * g.Kld)) continue;
      bf16* dst = cols + doff;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (ih >= 0 && ih < g.H && iw >= 0 && iw < g.W) {
        const long long soff = (((long long)n * g.H + ih) * g.W + iw) * g.C + c * 8;
        if (TNNB_CHECK(soff + 7, (long long)g.N * g.H * g.W * g.C)) v = *reinterpret_cast<const uint4*>(x + soff);
      }
      *reinterpret_cast<uint4*>(dst) = v;
    }
  } else {
    const int K = g.KH * g.KW * g.C;
    const int groups = g.Kld / 8;  // 16-byte groups per row, padding columns included (written as zeros)
    const long long total = (long long)g.N * g.OH * g.OW * groups;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
      const int gi = (int)(i % groups);
      const long long pix = i / groups;
      const int ow = (int)(pix % g.OW);
      const int oh = (int)((pix / g.OW) % g.OH);
      const int n = (int)(pix / ((long long)g.OW * g.OH));
      const bf16* img = x + (long long)n * g.H * g.W * g.C;
      __align__(16) bf16 v[8];
      // In NHWC the (kw, c) run of one filter row is contiguous in the image, so a column index k = kh * KW*C + kp
      // maps to img[(ih * W + iw0) * C + kp]; the horizontal bounds become a range of kp. One division per thread
      // instead of six per element - with three channels this kernel is bound by integer arithmetic, not by memory.
      const int kwc = g.KW * g.C;
      const int ih0 = oh * g.SH - g.PH, iw0 = ow * g.SW - g.PW;
      const int lo = (iw0 < 0 ? -iw0 : 0) * g.C;
      const int hi = (g.W - iw0 < g.KW ? g.W - iw0 : g.KW) * g.C;
      int kh = (gi * 8) / kwc;
      int kp = gi * 8 - kh * kwc;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        bf16 e = __float2bfloat16(0.f);
        const int ih = ih0 + kh;
        if (gi * 8 + j < K && ih >= 0 && ih < g.H && kp >= lo && kp < hi) {
          const long long off = ((long long)ih * g.W + iw0) * g.C + kp;
          if (TNNB_CHECK(off, (long long)g.H * g.W * g.C)) e = img[off];
        }
        v[j] = e;
        if (++kp == kwc) {
          kp = 0;
          ++kh;
        }
      }
      *reinterpret_cast<uint4*>(cols + pix * g.Kld + gi * 8) = *reinterpret_cast<const uint4*>(v);
    }
  }
}

// im2col through shared memory: a block builds the patch rows of `R` output rows of one image. It brings the input rows
// those need - (R - 1) * SH + KH of them, zero-padded on all sides - into shared memory once, and every thread then writes
// one fixed column group (eight columns, 16 bytes) of successive pixels, so that the place of its eight elements in the
// window is worked out once per block instead of once per group, and consecutive threads write consecutive addresses.
// The gather kernel above is bound by the integer arithmetic of that place: 224 x 224 x 3, 7 x 7 stride 2, 256 images
// took 856 us for 1.05 GB, this one takes 218; 64 x 64 x 32, 3 x 3, 256 images: 291 and 110 us. Shapes: im2col_rows().
// VEC = 8: C % 8 == 0, a group is one 16-byte element of the window. VEC = 1: any C, eight two-byte loads.
// A shared-memory row holds image columns [-PW, W + right) with image column 0 on a 16-byte boundary.
struct Im2colRows {
  int R, lp, rowlen, rows_in;  // output rows per block; elements left of image column 0; row pitch; input rows per block
  int row_blocks;              // ceil(OH / R)
  int vec_rows;                // image rows are whole 16-byte vectors
};
template <int VEC>
__global__ void __launch_bounds__(256)
im2col_rows_kernel(const bf16* __restrict__ x, bf16* __restrict__ cols, ConvGeo g, Im2colRows q) {
  extern __shared__ __align__(16) uint8_t im_smem[];
  bf16* win = reinterpret_cast<bf16*>(im_smem);
  const int n = blockIdx.x / q.row_blocks, oh0 = (blockIdx.x - n * q.row_blocks) * q.R;
  const int ih0 = oh0 * g.SH - g.PH;
  const int wc = g.W * g.C;
  const bf16* img = x + (long long)n * g.H * wc;
  const bf16 zero = __float2bfloat16(0.f);
  if (q.vec_rows) {
    const int per_row = q.rowlen / 8, v0 = q.lp / 8, v1 = v0 + wc / 8;
    for (int i = threadIdx.x; i < q.rows_in * per_row; i += 256) {
      const int r = i / per_row, v = i - r * per_row, ih = ih0 + r;
      uint4 val = make_uint4(0, 0, 0, 0);
      if (ih >= 0 && ih < g.H && v >= v0 && v < v1) {
        const long long off = (long long)ih * wc + (v - v0) * 8;
        if (TNNB_CHECK(off + 7, (long long)g.H * wc)) val = *reinterpret_cast<const uint4*>(img + off);
      }
      *reinterpret_cast<uint4*>(win + i * 8) = val;
    }
  } else {
    for (int i = threadIdx.x; i < q.rows_in * q.rowlen; i += 256) {
      const int r = i / q.rowlen, e = i - r * q.rowlen - q.lp, ih = ih0 + r;
      bf16 val = zero;
      if (ih >= 0 && ih < g.H && e >= 0 && e < wc) {
        const long long off = (long long)ih * wc + e;
        if (TNNB_CHECK(off, (long long)g.H * wc)) val = img[off];
      }
      win[i] = val;
    }
  }
  __syncthreads();
  const int groups = g.Kld / 8;
  const int per_trip = 256 / groups;  // pixels per trip of the block (groups <= 256)
  const int gi = threadIdx.x % groups, p0 = threadIdx.x / groups;
  if (p0 >= per_trip) return;
  const int kwc = g.KW * g.C, K = g.KH * kwc;
  const int shift = q.lp - g.PW * g.C;  // window column 0 of output column 0
  constexpr int NOFF = VEC == 8 ? 1 : 8;
  int off[NOFF];
#pragma unroll
  for (int j = 0; j < NOFF; ++j) {
    const int k = gi * 8 + j, kh = k / kwc;
    off[j] = k < K ? kh * q.rowlen + (k - kh * kwc) + shift : -1;
  }
  if (VEC == 8 && off[0] < 0) return;  // columns beyond the patch stay as they are
  const int pixels = min(q.R, g.OH - oh0) * g.OW;
  bf16* dst = cols + (((long long)n * g.OH + oh0) * g.OW) * g.Kld + gi * 8;
  int r = p0 / g.OW, ow = p0 - r * g.OW;
  for (int p = p0; p < pixels; p += per_trip) {
    const bf16* w = win + r * g.SH * q.rowlen + ow * g.SW * g.C;
    uint4 v;
    if (VEC == 8) {
      v = *reinterpret_cast<const uint4*>(w + off[0]);
    } else {
      uint32_t h[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint16_t a = off[NOFF == 1 ? 0 : 2 * j] >= 0 ? *reinterpret_cast<const uint16_t*>(w + off[NOFF == 1 ? 0 : 2 * j]) : 0;
        const uint16_t b = off[NOFF == 1 ? 0 : 2 * j + 1] >= 0 ? *reinterpret_cast<const uint16_t*>(w + off[NOFF == 1 ? 0 : 2 * j + 1]) : 0;
        h[j] = (uint32_t)a | ((uint32_t)b << 16);
      }
      v = make_uint4(h[0], h[1], h[2], h[3]);
    }
    const long long doff = (long long)p * g.Kld;
    if (TNNB_CHECK((((long long)n * g.OH + oh0) * g.OW + p) * g.Kld + gi * 8 + 7, (long long)g.N * g.OH * g.OW * g.Kld))
      *reinterpret_cast<uint4*>(dst + doff) = v;
    ow += per_trip;
    while (ow >= g.OW) {
      ow -= g.OW;
      ++r;
    }
  }
}

// Launch shape of im2col_rows_kernel, or false where it does not apply (a row window larger than 48 KB, more than 256
// column groups). Output rows per block, as far as 24 KB of input rows allow: enough that a block writes 4096 groups (16 a
// thread), or eight rows where the grid keeps eight blocks per SM, so that input rows serve several output rows (224 x 224 x
// 3, 7 x 7 stride 2, 256 images: 218 us, without that 246). Small calls take fewer rows again until there are two blocks per
// SM: 32 x 32 x 3, 3 x 3, one image 2.3 us instead of 5.2, 224 x 224 x 3, 7 x 7, one image 4.1 and 5.8. (At 28 x 28 x 1, 5 x 5, 256
// images that costs: 8.5 instead of 5.6.)
static bool im2col_rows(const ConvGeo& g, const void* x, int vec, Im2colRows& q) {
  const int wc = g.W * g.C, groups = g.Kld / 8;
  if (groups > 256 || groups < 1) return false;
  const long long need = ((long long)(g.OW - 1) * g.SW + g.KW - g.PW) * g.C;  // elements right of image column 0 a window touches
  q.lp = (g.PW * g.C + 7) / 8 * 8;
  const long long right = need > wc ? need : wc;
  const long long rowlen = (q.lp + right + 7) / 8 * 8;
  if (rowlen * g.KH * 2 > 48 * 1024) return false;
  q.rowlen = (int)rowlen;
  q.vec_rows = (wc % 8 == 0) && !((uintptr_t)x & 15);
  if (vec == 8 && !q.vec_rows) return false;
  int R = 1;
  while (R < g.OH && (long long)R * g.OW * groups < 4096 && (((R) * g.SH + g.KH) * rowlen * 2 <= 24 * 1024)) ++R;
  while (R < 8 && R < g.OH && ((R * g.SH + g.KH) * rowlen * 2 <= 24 * 1024) && (long long)g.N * ((g.OH + R) / (R + 1)) >= 148 * 8) ++R;
  while (R > 1 && (long long)g.N * ((g.OH + R - 1) / R) < 148 * 2) --R;
  q.R = R;
  q.rows_in = (R - 1) * g.SH + g.KH;
  q.row_blocks = (g.OH + R - 1) / R;
  return (long long)g.N * q.row_blocks < (1ll << 31);
}

template <int VEC>
__global__ void col2im_kernel(const bf16* __restrict__ dcols, bf16* __restrict__ dx, ConvGeo g) {
  const int cv = g.C / VEC;
  const long long total = (long long)g.N * g.H * g.W * cv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const int c = (int)(i % cv);
    long long r = i / cv;
    const int w = (int)(r % g.W); r /= g.W;
    const int h = (int)(r % g.H);
    const int n = (int)(r / g.H);
    float acc[VEC];
#pragma unroll
    for (int k = 0; k < VEC; ++k) acc[k] = 0.f;
    // the output pixels whose window covers (h, w), as index ranges (two divisions per axis, see pool_bwd_kernel)
    const int th = h + g.PH, tw = w + g.PW;
    const int oh_hi = min(th / g.SH, g.OH - 1), ow_hi = min(tw / g.SW, g.OW - 1);
    const int oh_lo = th - g.KH + 1 > 0 ? (th - g.KH + g.SH) / g.SH : 0;
    const int ow_lo = tw - g.KW + 1 > 0 ? (tw - g.KW + g.SW) / g.SW : 0;
    for (int oh = oh_lo; oh <= oh_hi; ++oh) {
      const int kh = th - oh * g.SH;
      for (int ow = ow_lo; ow <= ow_hi; ++ow) {
        const int kw = tw - ow * g.SW;
        const long long soff = (((long long)n * g.OH + oh) * g.OW + ow) * g.Kld + (long long)(kh * g.KW + kw) * g.C + c * VEC;
        if (!TNNB_CHECK(soff + VEC - 1, (long long)g.N * g.OH * g.OW * g.Kld)) continue;
        const bf16* src = dcols + soff;
        if (VEC == 8) {
          uint4 raw = *reinterpret_cast<const uint4*>(src);
          const bf16* t8 = reinterpret_cast<const bf16*>(&raw);
#pragma unroll
          for (int k = 0; k < 8; ++k) acc[k] += __bfloat162float(t8[k]);
        } else {
          acc[0] += __bfloat162float(*src);
        }
      }
    }
    bf16* dst = dx + i * VEC;
    if (VEC == 8) {
      __align__(16) bf16 o[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) o[k] = __float2bfloat16(acc[k]);
      *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<uint4*>(o);
    } else {
      *dst = __float2bfloat16(acc[0]);
    }
  }
}

// Which row a thread works on and which of its elements: `blocks_per_row` blocks share a row, or (0) rows of fewer than
// 128 elements are laid end to end over the threads.
struct PoolSlot {
  int row, first, step;
};
__device__ __forceinline__ PoolSlot pool_slot(int blocks_per_row, int per_row) {
  PoolSlot s;
  if (blocks_per_row) {
    s.row = blockIdx.x / blocks_per_row;
    s.first = (blockIdx.x - s.row * blocks_per_row) * 256 + threadIdx.x;
    s.step = blocks_per_row * 256;
  } else {
    const unsigned t = blockIdx.x * 256u + threadIdx.x;
    s.row = (int)(t / (unsigned)per_row);
    s.first = (int)(t - (unsigned)s.row * per_row);
    s.step = per_row;
  }
  return s;
}

// MAX: window clipped to the image, uint8 window-relative argmax saved (the first of equal maxima; 255 when nothing in the
// window exceeds -infinity, and then the output is 0); otherwise the average over the in-image elements. For the usual
// 2 x 2 and 3 x 3 windows (KS) all loads of a window are issued before the first comparison, and the maximum is taken on
// packed bf16 pairs: one compare-to-mask and two selects per tap and pair carry value and position together. The same
// comparisons on eight fp32 values per tap, with the average's sums beside them, were bound by instruction issue:
// 256 x 112 x 112 x 64, 3 x 3 stride 2 (565 MB), 268 us, now 154; 256 x 32 x 32 x 128, 2 x 2, 29 and 15 us.
template <int KS, bool MAX>
__global__ void __launch_bounds__(256)
pool_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, unsigned char* __restrict__ idx, ConvGeo g, int blocks_per_row) {
  const int cv = g.C / 8;
  const PoolSlot ps = pool_slot(blocks_per_row, g.OW * cv);
  const int row = ps.row;  // n * OH + oh
  if (row >= g.N * g.OH) return;
  const int n = row / g.OH, oh = row - n * g.OH;
  const int KH = KS ? KS : g.KH, KW = KS ? KS : g.KW;
  const int ih0 = oh * g.SH - g.PH;
  const bf16* img = x + (long long)n * g.H * g.W * g.C;
  const long long out0 = (long long)row * g.OW * cv;
  for (int i = ps.first; i < g.OW * cv; i += ps.step) {
    const int ow = i / cv, c = i - ow * cv;
    const int iw0 = ow * g.SW - g.PW;
    uint32_t best[4], pos[4];  // two channels per word
    float sum[8];
#pragma unroll
    for (int k = 0; k < 4; ++k) best[k] = 0xff80ff80u, pos[k] = 0x00ff00ffu;
#pragma unroll
    for (int k = 0; k < 8; ++k) sum[k] = 0.f;
    int cnt = 0;
    auto take = [&](const uint4& raw, uint32_t t) {
      const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
      if (MAX) {
        const uint32_t tt = t | (t << 16);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t m = __hgt2_mask(*reinterpret_cast<const __nv_bfloat162*>(&w[k]), *reinterpret_cast<const __nv_bfloat162*>(&best[k]));
          best[k] = (w[k] & m) | (best[k] & ~m);
          pos[k] = (tt & m) | (pos[k] & ~m);
        }
      } else {
        ++cnt;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          sum[2 * k] += __uint_as_float(w[k] << 16);
          sum[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
        }
      }
    };
    if (KS) {
      constexpr int T = KS ? KS * KS : 1, K1 = KS ? KS : 1;
      uint4 raw[T];
      bool ok[T];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int ih = ih0 + t / K1, iw = iw0 + t % K1;
        ok[t] = ih >= 0 && ih < g.H && iw >= 0 && iw < g.W;
        raw[t] = make_uint4(0, 0, 0, 0);
        if (ok[t]) raw[t] = *reinterpret_cast<const uint4*>(img + ((long long)ih * g.W + iw) * g.C + c * 8);
      }
#pragma unroll
      for (int t = 0; t < T; ++t)
        if (ok[t]) take(raw[t], (uint32_t)t);
    } else {
      for (int kh = 0; kh < KH; ++kh) {
        const int ih = ih0 + kh;
        if (ih < 0 || ih >= g.H) continue;
        for (int kw = 0; kw < KW; ++kw) {
          const int iw = iw0 + kw;
          if (iw < 0 || iw >= g.W) continue;
          take(*reinterpret_cast<const uint4*>(img + ((long long)ih * g.W + iw) * g.C + c * 8), (uint32_t)(kh * KW + kw));
        }
      }
    }
    const long long oi = (out0 + i) * 8;
    uint32_t o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (MAX) {  // an untouched half (position 255) is 0
        o[k] = best[k] & (((pos[k] & 0xffffu) == 255u ? 0u : 0xffffu) | ((pos[k] >> 16) == 255u ? 0u : 0xffff0000u));
      } else {
        __nv_bfloat162 h = __floats2bfloat162_rn(cnt ? sum[2 * k] / cnt : 0.f, cnt ? sum[2 * k + 1] / cnt : 0.f);
        o[k] = *reinterpret_cast<uint32_t*>(&h);
      }
    }
    *reinterpret_cast<uint4*>(y + oi) = make_uint4(o[0], o[1], o[2], o[3]);
    if (MAX && idx)
      *reinterpret_cast<uint2*>(idx + oi) = make_uint2(__byte_perm(pos[0], pos[1], 0x6420), __byte_perm(pos[2], pos[3], 0x6420));
  }
}

// Average over large windows (the pool in front of a classifier: 7 x 7 and one output pixel per image): one thread per output
// pixel and eight channels, sixteen loads of its window in flight where the loop above has one. The elements are added in
// the order of that loop, so that the result does not depend on the kernel: a rounding that flips here moves the gradient of
// a deep network by 0.006 of its 2-norm. Us with one load in flight and now: 7 x 7 x 2048 channels, 7 images 13.1 and 6.5, 256
// images (51 MB) 14.0 and 8.3; 8 x 8 x 512, 1024 images 17.7 and 8.7; 4 x 4 x 512, 8192 images (134 MB) 29.2 and 25.6; 4 x 4
// windows of 56 x 56 x 64, 64 images 45.8 and 33.0. Twice as many loads in flight: 10.4 us for the first. (Eight lanes sharing a
// window: 3.1 us for the first, but 13.1 for the second, and another order.)
__global__ void __launch_bounds__(64)
pool_avg_window_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, ConvGeo g, long long total) {
  const int cv = g.C / 8;
  const long long i = (long long)blockIdx.x * 64 + threadIdx.x;
  if (i >= total) return;
  const long long pix = i / cv;  // (n * OH + oh) * OW + ow
  const int c = (int)(i - pix * cv);
  const long long row = pix / g.OW;
  const int ow = (int)(pix - row * g.OW);
  const int n = (int)(row / g.OH), oh = (int)(row - (long long)n * g.OH);
  const int h0 = max(oh * g.SH - g.PH, 0), h1 = min(oh * g.SH - g.PH + g.KH, g.H);
  const int w0 = max(ow * g.SW - g.PW, 0), w1 = min(ow * g.SW - g.PW + g.KW, g.W);
  const int ww = max(w1 - w0, 0), cnt = max(h1 - h0, 0) * ww;
  float sum[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const bf16* src = x + (((long long)n * g.H + h0) * g.W + w0) * g.C + c * 8;
  int left = ww;  // elements of the window's row that are still to come
  for (int t = 0; t < cnt; t += 16) {
    uint4 raw[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      raw[u] = make_uint4(0, 0, 0, 0);
      if (t + u < cnt) raw[u] = *reinterpret_cast<const uint4*>(src);
      src += g.C;
      if (--left == 0) {
        left = ww;
        src += (long long)(g.W - ww) * g.C;
      }
    }
#pragma unroll
    for (int u = 0; u < 16; ++u) {  // behind the end zeros
      const uint32_t w[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        sum[2 * k] += __uint_as_float(w[k] << 16);
        sum[2 * k + 1] += __uint_as_float(w[k] & 0xffff0000u);
      }
    }
  }
  uint32_t o[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    __nv_bfloat162 h = __floats2bfloat162_rn(cnt ? sum[2 * k] / cnt : 0.f, cnt ? sum[2 * k + 1] / cnt : 0.f);
    o[k] = *reinterpret_cast<uint32_t*>(&h);
  }
  *reinterpret_cast<uint4*>(y + i * 8) = make_uint4(o[0], o[1], o[2], o[3]);
}

// Gather form of the pool backward: every input pixel sums the outputs whose window covers it (max: only where the saved
// argmax points back at it; average: dy / in-image count). Output rows whose window covers input row h:
// oh * SH - PH <= h < oh * SH - PH + KH. NW is the number of windows that can cover a pixel along an axis when that is one
// or two (KH <= NW * SH and KW <= NW * SW): all their loads are then in flight together, and for the maximum the saved
// positions of eight channels are compared in two byte-wise instructions whose masks select the gradient's bf16 pairs. NW = 0
// takes any window in a loop. Of the zoo's pools the 3 x 3 maximum at stride 3 comes here with NW = 1 and the averages over
// whole images (4 x 4 to 8 x 8 at stride 1) with NW = 0; maxima at stride 2 go to the patch kernel below. One window at a
// time and channel by channel, 256 x 112 x 112 x 64, 3 x 3 stride 2, took 496 us, this form 420 (the patch kernel 165).
template <int NW, bool MAX>
__global__ void __launch_bounds__(256)
pool_bwd_kernel(const bf16* __restrict__ dy, const unsigned char* __restrict__ idx, bf16* __restrict__ dx, ConvGeo g, int blocks_per_row) {
  const int cv = g.C / 8;
  const PoolSlot ps = pool_slot(blocks_per_row, g.W * cv);
  const int row = ps.row;  // n * H + h
  if (row >= g.N * g.H) return;
  const int n = row / g.H, h = row - n * g.H;
  const int th = h + g.PH;
  const int oh_hi = min(th / g.SH, g.OH - 1);
  const int oh_lo = th - g.KH + 1 > 0 ? (th - g.KH + g.SH) / g.SH : 0;
  const long long img0 = (long long)n * g.OH * g.OW;
  for (int i = ps.first; i < g.W * cv; i += ps.step) {
    const int w = i / cv, c = i - w * cv;
    float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    const int tw = w + g.PW;
    const int ow_hi = min(tw / g.SW, g.OW - 1);
    const int ow_lo = tw - g.KW + 1 > 0 ? (tw - g.KW + g.SW) / g.SW : 0;
    auto add = [&](const uint4& raw, const uint2& ir, int oh, int ow) {
      const uint32_t gw[4] = {raw.x, raw.y, raw.z, raw.w};
      if (MAX) {
        const uint32_t me = (uint32_t)((th - oh * g.SH) * g.KW + (tw - ow * g.SW)) * 0x01010101u;
#ifdef TNNB_BOUNDS_CHECK
        const unsigned char* b8 = reinterpret_cast<const unsigned char*>(&ir);
        for (int k = 0; k < 8; ++k)
          if (b8[k] != 255) (void)TNNB_CHECK(b8[k], g.KH * g.KW);  // a saved position outside the window (255 = empty window)
#endif
        const uint32_t e0 = __vcmpeq4(ir.x, me), e1 = __vcmpeq4(ir.y, me);
        const uint32_t m[4] = {__byte_perm(e0, 0, 0x1100), __byte_perm(e0, 0, 0x3322), __byte_perm(e1, 0, 0x1100), __byte_perm(e1, 0, 0x3322)};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t v = gw[k] & m[k];
          acc[2 * k] += __uint_as_float(v << 16);
          acc[2 * k + 1] += __uint_as_float(v & 0xffff0000u);
        }
      } else {
        const int h0 = max(oh * g.SH - g.PH, 0), h1 = min(oh * g.SH - g.PH + g.KH, g.H);
        const int w0 = max(ow * g.SW - g.PW, 0), w1 = min(ow * g.SW - g.PW + g.KW, g.W);
        const float inv = 1.f / (float)max((h1 - h0) * (w1 - w0), 1);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          acc[2 * k] += __uint_as_float(gw[k] << 16) * inv;
          acc[2 * k + 1] += __uint_as_float(gw[k] & 0xffff0000u) * inv;
        }
      }
    };
    if (NW) {
      constexpr int T = NW ? NW * NW : 1, N1 = NW ? NW : 1;
      uint4 raw[T];
      uint2 ir[T];
      bool ok[T];
#pragma unroll
      for (int t = 0; t < T; ++t) {
        const int oh = oh_lo + t / N1, ow = ow_lo + t % N1;
        const long long o = ((img0 + (long long)oh * g.OW + ow) * cv + c) * 8;
        ok[t] = oh <= oh_hi && ow <= ow_hi && TNNB_CHECK(o + 7, (long long)g.N * g.OH * g.OW * g.C);
        raw[t] = make_uint4(0, 0, 0, 0);
        ir[t] = make_uint2(0, 0);
        if (ok[t]) {
          raw[t] = *reinterpret_cast<const uint4*>(dy + o);
          if (MAX) ir[t] = *reinterpret_cast<const uint2*>(idx + o);
        }
      }
#pragma unroll
      for (int t = 0; t < T; ++t)
        if (ok[t]) add(raw[t], ir[t], oh_lo + t / N1, ow_lo + t % N1);
    } else {
      for (int oh = oh_lo; oh <= oh_hi; ++oh)
        for (int ow = ow_lo; ow <= ow_hi; ++ow) {
          const long long o = ((img0 + (long long)oh * g.OW + ow) * cv + c) * 8;
          if (!TNNB_CHECK(o + 7, (long long)g.N * g.OH * g.OW * g.C)) continue;
          add(*reinterpret_cast<const uint4*>(dy + o), MAX ? *reinterpret_cast<const uint2*>(idx + o) : make_uint2(0, 0), oh, ow);
        }
    }
    uint32_t o4[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      __nv_bfloat162 hh = __floats2bfloat162_rn(acc[2 * k], acc[2 * k + 1]);
      o4[k] = *reinterpret_cast<uint32_t*>(&hh);
    }
    *reinterpret_cast<uint4*>(dx + ((long long)row * g.W * cv + i) * 8) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
  }
}

// Max-pool backward at stride 2 with windows of up to NW * 2 elements along an axis. A thread owns the 2 x 2 input pixels
// whose (h + PH) / 2 and (w + PW) / 2 are the same pair (mh, mw): exactly the windows mh - NW + 1 .. mh and mw - NW + 1 ..
// mw can cover them, so NW * NW gradients and positions are loaded once for four pixels instead of up to NW * NW times per
// pixel, and a thread has four stores in flight. One pixel per thread left the memory system waiting for 114 thousand
// short blocks: 256 x 112 x 112 x 64, 3 x 3: 420 us, now 165 (565 MB); 256 x 32 x 32 x 128, 2 x 2: 45 and 17 us.
template <int NW>
__global__ void __launch_bounds__(256)
pool_bwd_patch_kernel(const bf16* __restrict__ dy, const unsigned char* __restrict__ idx, bf16* __restrict__ dx, ConvGeo g,
                      int blocks_per_row, int mh0, int mw0, int prows, int pcols) {
  const int cv = g.C / 8;
  const PoolSlot ps = pool_slot(blocks_per_row, pcols * cv);
  const int row = ps.row;  // n * prows + patch row
  if (row >= g.N * prows) return;
  const int n = row / prows, mh = mh0 + row - n * prows;
  const long long img0 = (long long)n * g.OH * g.OW;
  for (int i = ps.first; i < pcols * cv; i += ps.step) {
    const int pc = i / cv, c = i - pc * cv, mw = mw0 + pc;
    uint4 raw[NW * NW];
    uint2 ir[NW * NW];
    bool ok[NW * NW];
#pragma unroll
    for (int t = 0; t < NW * NW; ++t) {
      const int oh = mh - NW + 1 + t / NW, ow = mw - NW + 1 + t % NW;
      const long long o = ((img0 + (long long)oh * g.OW + ow) * cv + c) * 8;
      ok[t] = oh >= 0 && oh < g.OH && ow >= 0 && ow < g.OW && TNNB_CHECK(o + 7, (long long)g.N * g.OH * g.OW * g.C);
      raw[t] = make_uint4(0, 0, 0, 0);
      ir[t] = make_uint2(0xffffffffu, 0xffffffffu);
      if (ok[t]) {
        raw[t] = *reinterpret_cast<const uint4*>(dy + o);
        ir[t] = *reinterpret_cast<const uint2*>(idx + o);
#ifdef TNNB_BOUNDS_CHECK
        const unsigned char* b8 = reinterpret_cast<const unsigned char*>(&ir[t]);
        for (int k = 0; k < 8; ++k)
          if (b8[k] != 255) (void)TNNB_CHECK(b8[k], g.KH * g.KW);
#endif
      }
    }
#pragma unroll
    for (int px = 0; px < 4; ++px) {
      const int th = 2 * mh + (px >> 1), tw = 2 * mw + (px & 1);
      const int h = th - g.PH, w = tw - g.PW;
      if (h < 0 || h >= g.H || w < 0 || w >= g.W) continue;
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
      for (int t = 0; t < NW * NW; ++t) {
        const int kh = (px >> 1) + 2 * (NW - 1 - t / NW), kw = (px & 1) + 2 * (NW - 1 - t % NW);
        if (kh >= g.KH || kw >= g.KW) continue;  // the window ends before this pixel (same for every thread)
        const uint32_t me = (uint32_t)(kh * g.KW + kw) * 0x01010101u;
        const uint32_t e0 = __vcmpeq4(ir[t].x, me), e1 = __vcmpeq4(ir[t].y, me);
        const uint32_t gw[4] = {raw[t].x, raw[t].y, raw[t].z, raw[t].w};
        const uint32_t m[4] = {__byte_perm(e0, 0, 0x1100), __byte_perm(e0, 0, 0x3322), __byte_perm(e1, 0, 0x1100), __byte_perm(e1, 0, 0x3322)};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t v = gw[k] & m[k];
          acc[2 * k] += __uint_as_float(v << 16);
          acc[2 * k + 1] += __uint_as_float(v & 0xffff0000u);
        }
      }
      uint32_t o4[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        __nv_bfloat162 hh = __floats2bfloat162_rn(acc[2 * k], acc[2 * k + 1]);
        o4[k] = *reinterpret_cast<uint32_t*>(&hh);
      }
      *reinterpret_cast<uint4*>(dx + ((((long long)n * g.H + h) * g.W + w) * cv + c) * 8) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
    }
  }
}

// Grid of the pooling kernels over `rows` rows of `per_row` elements (see PoolSlot); 0 when a grid cannot hold it.
static int pool_grid(long long rows, int per_row, int& blocks_per_row) {
  blocks_per_row = 0;
  if (rows >= (1ll << 31)) return 0;
  if (per_row < 128) {
    const long long total = rows * per_row;
    if (total < (1ll << 31)) return (int)((total + 255) / 256);
  }
  blocks_per_row = (per_row + 255) / 256;
  if (rows * blocks_per_row >= (1ll << 31)) blocks_per_row = 1;
  return (int)(rows * blocks_per_row);
}

// Filter of a data gradient: out[c, u, v, o] = w[o, rh + sh * (nh - 1 - u), rw + sw * (nw - 1 - v), c], i.e. the filter
// rotated by 180 degrees with its channel axes swapped (stride 1: rh = 0, sh = 1, nh = KH), or the taps that reach one
// parity class of input pixels. Per tap a transpose of 64 x 64 channel tiles through shared memory, 16 bytes per access on
// both sides, where a flip and a strided copy were two launches that read or wrote two bytes at a time (128 to 512
// channels, 3 x 3: 9.9 us together, now 2.7).
__global__ void __launch_bounds__(256)
conv_weight_t_kernel(const bf16* __restrict__ w, bf16* __restrict__ out, int O, int KH, int KW, int C, int rh, int sh, int nh,
                     int rw, int sw, int nw) {
  __shared__ uint16_t tile[64][66];
  const int c0 = blockIdx.x * 64, o0 = blockIdx.y * 64;
  const int u = blockIdx.z / nw, v = blockIdx.z - u * nw;
  const int kh = rh + sh * (nh - 1 - u), kw = rw + sw * (nw - 1 - v);
  const long long in_pitch = (long long)KH * KW * C, out_pitch = (long long)nh * nw * O;
  const bf16* src = w + (long long)(kh * KW + kw) * C + c0;
#pragma unroll
  for (int i = threadIdx.x; i < 512; i += 256) {
    const int o = i >> 3, c8 = (i & 7) * 8;
    const uint4 val = *reinterpret_cast<const uint4*>(src + (o0 + o) * in_pitch + c8);
    uint32_t* d = reinterpret_cast<uint32_t*>(&tile[o][c8]);
    d[0] = val.x; d[1] = val.y; d[2] = val.z; d[3] = val.w;
  }
  __syncthreads();
  bf16* dst = out + (long long)(u * nw + v) * O + o0;
#pragma unroll
  for (int i = threadIdx.x; i < 512; i += 256) {
    const int c = i >> 3, o8 = (i & 7) * 8;
    uint32_t p[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) p[j] = (uint32_t)tile[o8 + 2 * j][c] | ((uint32_t)tile[o8 + 2 * j + 1][c] << 16);
    *reinterpret_cast<uint4*>(dst + (c0 + c) * out_pitch + o8) = make_uint4(p[0], p[1], p[2], p[3]);
  }
}

static inline int grid1d(long long n, int block) {
  long long g = (n + block - 1) / block;
  const long long cap = 148ll * 32;
  return (int)(g < 1 ? 1 : (g > cap ? cap : g));
}

}  // namespace tnnb

using namespace tnnb;

static ConvGeo make_geo(int N, int H, int W, int C, int KH, int KW, int SH, int SW, int PH, int PW, int Kld) {
  ConvGeo g{N, H, W, C, KH, KW, SH, SW, PH, PW, (H + 2 * PH - KH) / SH + 1, (W + 2 * PW - KW) / SW + 1, Kld};
  return g;
}

#define RC_LAST()                                       \
  do {                                                  \
    cudaError_t e__ = cudaGetLastError();               \
    return e__ == cudaSuccess ? 0 : -(int)e__ - 1000;   \
  } while (0)

extern "C" {

// cols: [N*OH*OW, Kld] bf16; columns >= KH*KW*C (padding of the pitch) are left untouched.
int tnnb_im2col(const void* x, void* cols, int N, int H, int W, int C, int KH, int KW, int SH, int SW, int PH, int PW,
                int Kld, void* stream) {
  ConvGeo g = make_geo(N, H, W, C, KH, KW, SH, SW, PH, PW, Kld);
  if (g.OH <= 0 || g.OW <= 0 || Kld < KH * KW * C) return -2;
  if (Kld % 8 || ((uintptr_t)cols & 15)) return -3;
  if (N <= 0 || Kld == 0) RC_LAST();  // nothing to write
  const bool vec = (C % 8 == 0) && !((uintptr_t)x & 15);
  const long long total = (long long)N * g.OH * g.OW * (vec ? (long long)KH * KW * (C / 8) : Kld / 8);
  Im2colRows q;
  if (im2col_rows(g, x, vec ? 8 : 1, q)) {
    const int grid = g.N * q.row_blocks;
    const size_t smem = (size_t)q.rows_in * q.rowlen * 2;
    if (vec) im2col_rows_kernel<8><<<grid, 256, smem, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)cols, g, q);
    else im2col_rows_kernel<1><<<grid, 256, smem, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)cols, g, q);
    RC_LAST();
  }
  if (vec) im2col_kernel<8><<<grid1d(total, 256), 256, 0, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)cols, g);
  else im2col_kernel<1><<<grid1d(total, 256), 256, 0, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)cols, g);
  RC_LAST();
}

int tnnb_col2im(const void* dcols, void* dx, int N, int H, int W, int C, int KH, int KW, int SH, int SW, int PH, int PW,
                int Kld, void* stream) {
  ConvGeo g = make_geo(N, H, W, C, KH, KW, SH, SW, PH, PW, Kld);
  if (g.OH <= 0 || g.OW <= 0) return -2;
  const bool vec = (C % 8 == 0) && (Kld % 8 == 0) && !(((uintptr_t)dx | (uintptr_t)dcols) & 15);
  const long long total = (long long)N * H * W * (vec ? C / 8 : C);
  if (vec) col2im_kernel<8><<<grid1d(total, 256), 256, 0, (cudaStream_t)stream>>>((const bf16*)dcols, (bf16*)dx, g);
  else col2im_kernel<1><<<grid1d(total, 256), 256, 0, (cudaStream_t)stream>>>((const bf16*)dcols, (bf16*)dx, g);
  RC_LAST();
}

// w [O, KH, KW, C] -> out [C, nh, nw, O] (see conv_weight_t_kernel). O and C multiples of 64, 16-byte aligned tensors.
int tnnb_conv_weight_t(const void* w, void* out, int O, int KH, int KW, int C, int rh, int sh, int nh, int rw, int sw, int nw,
                       void* stream) {
  if (O <= 0 || C <= 0 || O % 64 || C % 64 || (((uintptr_t)w | (uintptr_t)out) & 15)) return -3;
  if (nh <= 0 || nw <= 0 || rh < 0 || rw < 0 || sh <= 0 || sw <= 0 || rh + sh * (nh - 1) >= KH || rw + sw * (nw - 1) >= KW) return -2;
  if (O / 64 > 65535 || nh * nw > 65535) return -3;
  conv_weight_t_kernel<<<dim3(C / 64, O / 64, nh * nw), 256, 0, (cudaStream_t)stream>>>((const bf16*)w, (bf16*)out, O, KH, KW, C, rh, sh, nh,
                                                                                       rw, sw, nw);
  RC_LAST();
}

// Images per launch of a pooling kernel, which numbers its rows with 31 bits; a larger batch is taken in parts.
static int pool_part(int N, int rows) { return (int)min((long long)N, max(1ll, ((1ll << 31) - 1) / rows)); }

static int pool_fwd_part(const void* x, void* y, void* idx, int N, int H, int W, int C, int KH, int KW, int SH, int SW, int PH,
                         int PW, int mode, void* stream) {
  const ConvGeo g = make_geo(N, H, W, C, KH, KW, SH, SW, PH, PW, 0);
  // Windows of 16 elements and more: faster at every size but 7 x 7 x 2048, 1024 images (39.0 us in the loop, 43.8); below, one
  // trip holds nothing but the window and the unrolled forms for 2 x 2 and 3 x 3 do the same.
  const long long outputs = (long long)N * g.OH * g.OW * (C / 8);
  if (mode == 1 && KH * KW >= 16 && outputs < (1ll << 36)) {
    pool_avg_window_kernel<<<(int)((outputs + 63) / 64), 64, 0, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)y, g, outputs);
    RC_LAST();
  }
  const long long rows = (long long)N * g.OH;
  int bpr;
  const int grid = pool_grid(rows, g.OW * (C / 8), bpr);
  if (!grid) return -3;
#define TNNB_POOL(KS)                                                                                                                \
  do {                                                                                                                              \
    if (mode == 0) pool_fwd_kernel<KS, true><<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)y, (unsigned char*)idx, g, bpr); \
    else pool_fwd_kernel<KS, false><<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)y, (unsigned char*)idx, g, bpr);  \
  } while (0)
  if (KH == 2 && KW == 2) TNNB_POOL(2);
  else if (KH == 3 && KW == 3) TNNB_POOL(3);
  else TNNB_POOL(0);
#undef TNNB_POOL
  RC_LAST();
}

// C % 8 == 0 and pool windows of at most 254 elements. idx (uint8, same shape as y) may be null.
int tnnb_pool_fwd(const void* x, void* y, void* idx, int N, int H, int W, int C, int KH, int KW, int SH, int SW, int PH,
                  int PW, int mode, void* stream) {
  if (C % 8 || KH * KW > 254) return -3;
  const ConvGeo g = make_geo(N, H, W, C, KH, KW, SH, SW, PH, PW, 0);
  if (g.OH <= 0 || g.OW <= 0 || N <= 0 || C == 0) RC_LAST();
  const int part = pool_part(N, g.OH);
  for (int n = 0; n < N; n += min(part, N - n)) {
    const long long in = (long long)n * H * W * C, out = (long long)n * g.OH * g.OW * C;
    const int rc = pool_fwd_part((const bf16*)x + in, (bf16*)y + out, idx ? (unsigned char*)idx + out : nullptr, min(part, N - n), H, W, C,
                                 KH, KW, SH, SW, PH, PW, mode, stream);
    if (rc) return rc;
  }
  return 0;
}

static int pool_bwd_part(const void* dy, const void* idx, void* dx, int N, int H, int W, int C, int KH, int KW, int SH, int SW,
                         int PH, int PW, int mode, void* stream) {
  const ConvGeo g = make_geo(N, H, W, C, KH, KW, SH, SW, PH, PW, 0);
  int bpr;
  if (mode == 0 && SH == 2 && SW == 2 && KH <= 4 && KW <= 4 && PH >= 0 && PW >= 0) {  // a patch's windows: one or two per axis
    const int mh0 = PH / 2, mw0 = PW / 2;
    const int prows = (H - 1 + PH) / 2 - mh0 + 1, pcols = (W - 1 + PW) / 2 - mw0 + 1;
    const int grid = pool_grid((long long)N * prows, pcols * (C / 8), bpr);
    if (!grid) return -3;
    if (KH <= 2 && KW <= 2)
      pool_bwd_patch_kernel<1><<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)dy, (const unsigned char*)idx, (bf16*)dx, g, bpr, mh0, mw0, prows, pcols);
    else
      pool_bwd_patch_kernel<2><<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)dy, (const unsigned char*)idx, (bf16*)dx, g, bpr, mh0, mw0, prows, pcols);
    RC_LAST();
  }
  const long long rows = (long long)N * H;
  const int grid = pool_grid(rows, W * (C / 8), bpr);
  if (!grid) return -3;
  const int nw = (KH <= SH && KW <= SW) ? 1 : (KH <= 2 * SH && KW <= 2 * SW) ? 2 : 0;
#define TNNB_POOL(NW)                                                                                                                \
  do {                                                                                                                              \
    if (mode == 0) pool_bwd_kernel<NW, true><<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)dy, (const unsigned char*)idx, (bf16*)dx, g, bpr); \
    else pool_bwd_kernel<NW, false><<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)dy, (const unsigned char*)idx, (bf16*)dx, g, bpr); \
  } while (0)
  if (nw == 1) TNNB_POOL(1);
  else if (nw == 2) TNNB_POOL(2);
  else TNNB_POOL(0);
#undef TNNB_POOL
  RC_LAST();
}

int tnnb_pool_bwd(const void* dy, const void* idx, void* dx, int N, int H, int W, int C, int KH, int KW, int SH, int SW,
                  int PH, int PW, int mode, void* stream) {
  if (C % 8) return -3;
  const ConvGeo g = make_geo(N, H, W, C, KH, KW, SH, SW, PH, PW, 0);
  if (H <= 0 || W <= 0 || N <= 0 || C == 0) RC_LAST();
  const int part = pool_part(N, H);
  for (int n = 0; n < N; n += min(part, N - n)) {
    const long long in = (long long)n * H * W * C, out = (long long)n * g.OH * g.OW * C;
    const int rc = pool_bwd_part((const bf16*)dy + out, idx ? (const unsigned char*)idx + out : nullptr, (bf16*)dx + in, min(part, N - n), H,
                                 W, C, KH, KW, SH, SW, PH, PW, mode, stream);
    if (rc) return rc;
  }
  return 0;
}

}  // extern "C"
