// bf16 GEMM for sm_100a: TMA -> 128B-swizzled shared memory -> tcgen05.mma
// with the fp32 accumulator in TMEM -> tcgen05.ld epilogue.
//
//   D[M,N] (+)= op(A)[M,K] * op(B)[N,K]^T   (+ bias, GELU, dGELU, ReLU, residual)
//
// Either operand may be "K-major" (stored [rows, K], K contiguous) or
// "MN-major" (stored [K, rows], rows contiguous), which is what lets one
// kernel serve the three products of a dense layer without a transpose pass:
//   forward  Y  = X  * W^T      A K-major,  B K-major
//   dgrad    dX = dY * W        A K-major,  B MN-major
//   wgrad    dW += dY^T * X     A MN-major, B MN-major, fp32 atomic split-K
// The reference obtains these from cublasGemmEx / cuDNN matmul graphs
// (src/math/cuda/gemm.cu:72-112, src/nn/engines/cudnn_engine.cu:113-326).
//
// Structure: persistent CTAs (one per SM), 10 warps.
//   warp 0      TMA producer (one lane), STAGES-deep ring of (A,B) k-blocks
//   warp 1      TMEM owner + MMA issuer (one lane), two accumulators so the
//               epilogue of tile i overlaps the main loop of tile i+1
//   warps 2-9   epilogue: TMEM -> registers -> fused math -> per-warp staging tile in shared
//               memory -> global memory in whole 128-byte lines
//               (two warps per 32-lane TMEM quarter, each owning half of the columns)
// Two kernels share this structure: a single-CTA one (128 x 256, 128 x 128 or 128 x 64 tiles) and a CTA-pair
// one (`cta_group::2`, 256 x 256 tiles over two SMs), which is the default for large problems.
// Every barrier wait is bounded; on expiry the kernel records a status code,
// raises a CTA-wide abort flag and unwinds (TMEM is always released).
#include "gemm_tcgen05.h"

#include <cstdlib>
#include <mutex>

#include "col_norm.cuh"
#include "k_ranges.cuh"
#include "launch.cuh"
#include "ptx.cuh"
#include "tp_flags.cuh"

namespace tnnb {

// Tensor-parallel extension of the CTA-pair kernel (tnnb_gemm_tp; protocol in tp_flags.cuh).
//   mode 1  all-gather -> GEMM: rows of A that another rank owns are pushed into the local A buffer by
//           that rank; the TMA producer polls the row block's counter before it loads a tile of such rows.
//           Tiles of the locally owned rows run first. The push itself is done by two extra warps of this very
//           kernel (push_n > 0): while the tensor cores work on the local tiles they copy this rank's rows
//           into every peer's buffer with plain 16-byte stores, piece by piece in row order, and bump the
//           peer's row-block counter after each piece - the transfer hides behind the local half of the GEMM
//           on both sides and blocks nobody but the two warps that issue it.
//   mode 2  GEMM -> reduce-scatter: the epilogue stores the bf16 partial sums of rows another rank owns
//           straight into that rank's inbox (peer stores) and the rows this rank owns into the local
//           output (with the bias); remote tiles run first and their counters are bumped as soon as the
//           CTA has finished its last remote tile. The kernel itself never waits for a peer.
struct TpExt {
  int mode, tp, rank;
  int rows_per_rank;   // rows of M owned by each rank (multiple of 128)
  int pair_blocks_per_rank;  // rows_per_rank / 256, or 0 when that is not whole (tile order then stays plain)
  const uint32_t* pass;      // device word: number of passes including the current one
  int* status;
  // mode 1
  const uint32_t* a_ready;   // [M/128] cumulative rows landed per 128-row block of A (local memory)
  int push_n;                // number of peers this rank's rows of A are sent to by this kernel (0: none)
  int push_first_block;      // first 128-row block (inside this rank's rows) the kernel sends; earlier ones were sent by the producer
  const __nv_bfloat16* push_src;        // this rank's A buffer (all M rows; only its own rows are read)
  long long push_ld;                    // row pitch of A in elements (the same on every rank)
  __nv_bfloat16* push_dst[TP_MAX - 1];  // peer i's A buffer
  uint32_t* push_ready[TP_MAX - 1];     // peer i's counters [M/128]
  // mode 2
  void* out[TP_MAX];         // out[o]: [rows_per_rank, ldo] block that receives the rows owned by rank o
  long long ldo;
  uint32_t* arrived[TP_MAX]; // arrived[o]: rank o's counters, one per 128-row block of its rows
};

struct GemmParams {
  int M, N, K;
  int num_m_blocks, num_n_blocks, num_k_blocks;
  int split_k, kb_per_split;
  void* D;
  long long ldd;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* aux_in;
  __nv_bfloat16* aux_out;
  long long ld_aux;
  const __nv_bfloat16* resid;
  long long ld_res;
  ColNorm norm;  // EPI_NORM
  int flags;
  int* status;
  int lines;      // epilogue_lines; else epilogue_rows
  int stages;     // operand stages in use
  int epi_tiles;  // staging tiles per epilogue warp: 1, or one per 64 columns of an aux tensor
  // batched form (single-CTA kernel): `batch` independent products. Item i of an operand is head (i + off) % heads of
  // sequence (i + off) / heads, two strides apart, so that heads are read out of and written into packed [B, S, ., H, D]
  // tensors as they lie.
  int batch;
  int a_heads, a_off, b_heads, b_off, d_heads, d_off;
  long long d_stride_h, d_stride_b;  // of the output, in elements of D
};

// Shared memory of a CTA, from a 1024-byte boundary on: operand stages, staging tiles of the epilogue warps (1024-byte aligned
// as well: tile loads are swizzled by address), barriers.
static constexpr int EPI_WARPS = 8;   // two per 32-lane quarter of tensor memory, each with half of the columns
static constexpr int EPI_TILE = 4096;  // [32 rows][128 bytes]
static constexpr int BAR_BYTES = 512;
static constexpr int BAR_AUX = 256;    // byte of the barrier block where those of the epilogue warps' tile loads begin

template <int BN>
struct GemmCfg {
  static constexpr int BM = 128;
  static constexpr int BK = 64;
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int STAGES = (BN == 256) ? 4 : (BN == 128) ? 6 : 8;  // one less with two staging tiles per epilogue warp
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + BAR_BYTES + EPI_WARPS * EPI_TILE;
};

// Where a tile's result goes: the call's output, or (tensor-parallel reduce-scatter) the block of the rank
// that owns the tile's rows, with the bias applied only by the owner.
struct EpiOut {
  void* D;
  long long ldd;
  int flags;
};

// 16-byte accesses to a row from `at` on: every row of the tensor has to start on such a boundary, so the base as well as the pitch.
__device__ __forceinline__ bool row_vectors(const void* at, long long ld, int per16) {
  return ld % per16 == 0 && (reinterpret_cast<uintptr_t>(at) & 15) == 0;
}

// Fused element-wise part of the epilogue for 32 accumulator columns of one row (row < M, col0 < N). EPI_NORM and what follows it
// exist in epilogue_lines only (its entry point refuses outputs that are not for it).
__device__ __forceinline__ void epilogue_math(const GemmParams& p, const EpiOut& eo, float (&v)[32], int row, int col0) {
  const int flags = eo.flags;
  const bool full = (col0 + 32 <= p.N);

  if (flags & EPI_BIAS) {
    if (full && ((reinterpret_cast<uintptr_t>(p.bias + col0) & 15) == 0)) {
#pragma unroll
      for (int j = 0; j < 32; j += 8) {  // the same address in every lane: a broadcast
        const uint4 raw = *reinterpret_cast<const uint4*>(p.bias + col0 + j);
        const __nv_bfloat16* t = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[j + k] += __bfloat162float(t[k]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (full || col0 + j < p.N) v[j] += __bfloat162float(p.bias[col0 + j]);
    }
  }
  if (flags & EPI_GELU) {
    if (p.aux_out) {
      __nv_bfloat16* z = p.aux_out + (long long)row * p.ld_aux + col0;
      if (full && row_vectors(z, p.ld_aux, 8)) {
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
          __align__(16) __nv_bfloat16 t[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) t[k] = __float2bfloat16(v[j + k]);
          *reinterpret_cast<uint4*>(z + j) = *reinterpret_cast<uint4*>(t);
        }
      } else {
        for (int j = 0; j < 32; ++j)
          if (col0 + j < p.N) z[j] = __float2bfloat16(v[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = gelu_tanh(v[j]);
  }
  if (flags & EPI_DGELU) {
    const __nv_bfloat16* z = p.aux_in + (long long)row * p.ld_aux + col0;
    if (full && row_vectors(z, p.ld_aux, 8)) {
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        uint4 raw = *reinterpret_cast<const uint4*>(z + j);
        const __nv_bfloat16* t = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[j + k] *= gelu_tanh_grad(__bfloat162float(t[k]));
      }
    } else {
      for (int j = 0; j < 32; ++j)
        if (col0 + j < p.N) v[j] *= gelu_tanh_grad(__bfloat162float(z[j]));
    }
  }
  if (flags & EPI_RELU) {
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
  }
  if (flags & EPI_RESID) {
    const __nv_bfloat16* rs = p.resid + (long long)row * p.ld_res + col0;
    if (full && row_vectors(rs, p.ld_res, 8)) {
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        uint4 raw = *reinterpret_cast<const uint4*>(rs + j);
        const __nv_bfloat16* t = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
        for (int k = 0; k < 8; ++k) v[j + k] += __bfloat162float(t[k]);
      }
    } else {
      for (int j = 0; j < 32; ++j)
        if (col0 + j < p.N) v[j] += __bfloat162float(rs[j]);
    }
  }
}

// Row-per-lane store of 32 columns (each lane writes its own row): used for ragged edges and for the
// output forms the coalescing path below does not cover.
__device__ __forceinline__ void epilogue_store_rowwise(const GemmParams& p, const EpiOut& eo, const float (&v)[32], int row, int col0) {
  const int flags = eo.flags;
  const bool full = (col0 + 32 <= p.N);
  if (flags & EPI_ATOMIC) {
    float* d = reinterpret_cast<float*>(eo.D) + (long long)row * eo.ldd + col0;
    if (full && row_vectors(d, eo.ldd, 4)) {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(d + j), "f"(v[j]),
                     "f"(v[j + 1]), "f"(v[j + 2]), "f"(v[j + 3])
                     : "memory");
      }
    } else {
      for (int j = 0; j < 32; ++j)
        if (col0 + j < p.N) atomicAdd(d + j, v[j]);
    }
  } else if (flags & EPI_OUT_F32) {
    float* d = reinterpret_cast<float*>(eo.D) + (long long)row * eo.ldd + col0;
    if (full && row_vectors(d, eo.ldd, 4)) {
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        float4 o = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
        if (flags & EPI_ACCUM) {
          float4 old = *reinterpret_cast<float4*>(d + j);
          o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
        }
        *reinterpret_cast<float4*>(d + j) = o;
      }
    } else {
      for (int j = 0; j < 32; ++j)
        if (col0 + j < p.N) d[j] = (flags & EPI_ACCUM) ? d[j] + v[j] : v[j];
    }
  } else {
    __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(eo.D) + (long long)row * eo.ldd + col0;
    if (full && row_vectors(d, eo.ldd, 8)) {
#pragma unroll
      for (int j = 0; j < 32; j += 8) {
        __align__(16) __nv_bfloat16 t[8];
        if (flags & EPI_ACCUM) {
          uint4 raw = *reinterpret_cast<const uint4*>(d + j);
          const __nv_bfloat16* o = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
          for (int k = 0; k < 8; ++k) t[k] = __float2bfloat16(v[j + k] + __bfloat162float(o[k]));
        } else {
#pragma unroll
          for (int k = 0; k < 8; ++k) t[k] = __float2bfloat16(v[j + k]);
        }
        *reinterpret_cast<uint4*>(d + j) = *reinterpret_cast<uint4*>(t);
      }
    } else {
      for (int j = 0; j < 32; ++j)
        if (col0 + j < p.N)
          d[j] = __float2bfloat16((flags & EPI_ACCUM) ? v[j] + __bfloat162float(d[j]) : v[j]);
    }
  }
}


// ---- coalescing epilogue ------------------------------------------------------------------------
// tcgen05.ld hands every lane one ROW of the accumulator, so a direct store touches 32 different
// 128-byte lines per instruction. Each epilogue warp therefore owns a 4 KB staging tile in shared
// memory ([32 rows][128 B], 16-byte chunks XOR-swizzled by row): lanes write their row into it, and the
// warp reads it back with 8 lanes per row so that every global store / reduction instruction covers
// four complete 128-byte lines.
__device__ __forceinline__ uint32_t stage_off(int row, int chunk) { return row * 128 + ((chunk ^ (row & 7)) << 4); }

// bf16 output, 64 columns [col0, col0+64) of rows [row_base, row_base+32): lane = row has written its
// 64 values (as packed bf16) to the staging tile. Requires D on a 16-byte boundary, ldd % 8 == 0 and col0 + 64 <= N.
__device__ __forceinline__ void stage_flush_bf16(const GemmParams& p, const EpiOut& eo, const uint8_t* stage, int lane, int row_base,
                                                 int col0) {
  __syncwarp();
  __nv_bfloat16* D = reinterpret_cast<__nv_bfloat16*>(eo.D);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int r = i * 4 + (lane >> 3), c = lane & 7;
    const uint4 v = *reinterpret_cast<const uint4*>(stage + stage_off(r, c));
    if (row_base + r < p.M) *reinterpret_cast<uint4*>(D + (long long)(row_base + r) * eo.ldd + col0 + c * 8) = v;
  }
  __syncwarp();
}

// One warp's share of a tile: `nchunks` groups of 32 accumulator columns starting at TMEM address t_addr /
// global column col_base, rows row_base + lane, bf16 output. Chooses the coalescing path where its conditions hold. Only for
// products whose tiles go to several ranks (they refuse fp32 outputs and EPI_ACCUM).
__device__ __forceinline__ void epilogue_warp(const GemmParams& p, const EpiOut& eo, uint32_t t_addr, int nchunks, int row_base,
                                              int col_base, int lane, uint8_t* stage) {
  const int row = row_base + lane;
  const bool staged_ok = row_vectors(eo.D, eo.ldd, 8);
#pragma unroll 1
  for (int c = 0; c < nchunks; c += 2) {
    const int col0 = col_base + c * 32;
    if (col0 >= p.N) {  // whole pair of chunks is outside the matrix (tcgen05.ld is not needed)
      continue;
    }
    const bool pair_staged = staged_ok && (col0 + 64 <= p.N) && (c + 1 < nchunks);
    // both chunks of the pair are requested from tensor memory before the single wait: the epilogue is bound by the
    // latency of its dependent chain (two warps per scheduler), not by issue slots
    uint32_t rr[2][32];
    tmem_ld_32x32(t_addr + c * 32, rr[0]);  // warp-collective: never under a per-lane condition
    if (c + 1 < nchunks) tmem_ld_32x32(t_addr + (c + 1) * 32, rr[1]);
    tmem_ld_wait();
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (c + h >= nchunks) break;
      const int cc = col0 + h * 32;
      if (cc >= p.N) continue;
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(rr[h][j]);
      if (row < p.M) epilogue_math(p, eo, v, row, cc);
      if (!pair_staged) {
        if (row < p.M) epilogue_store_rowwise(p, eo, v, row, cc);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            __nv_bfloat162 h2 = __floats2bfloat162_rn(v[8 * k + 2 * j], v[8 * k + 2 * j + 1]);
            w[j] = *reinterpret_cast<uint32_t*>(&h2);
          }
          *reinterpret_cast<uint4*>(stage + stage_off(lane, h * 4 + k)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        if (h == 1) stage_flush_bf16(p, eo, stage, lane, row_base, col0);
      }
    }
  }
}

// ---- epilogue in lines ------------------------------------------------------------------------------
// For outputs with 16-byte aligned base and pitch. A warp takes 32 columns of its 32 rows
// at a time: accumulators -> registers -> fused math on pairs of fp32 values -> its staging tile -> whole 128-byte lines. A
// bf16 tensor that is read beside the output (EPI_DGELU, EPI_RESID) is fetched by TMA into the very staging tile the result
// replaces, as soon as the tile before has been written out: the load runs under the main loop. The accumulator is handed back
// once it lies in registers.
//
// What bounds products with few K blocks is this path, and in it the latency of each step rather than issue slots: what a
// step needs is on its way before the step begins. Us per launch with scalar math on two groups at a time, aux values and
// pre-activations accessed row by row by the lanes, and so:
//                             plain          bias + GELU + pre-act.   * GELU'        + residual
//   8192 x 3072 x 768     34.4 and 33.5          59.1 and 43.5      69.6 and 43.5   48.5 and 41.2
//   8192 x 768 x 3072     31.9 and 30.5          39.7 and 34.5      42.2 and 37.3   35.5 and 35.5
//   32125 x 1024 x 256    27.7 and 22.3          55.5 and 40.5      74.8 and 43.0   49.4 and 35.0
//   802816 x 256 x 64      116 and 94             297 and 205        398 and 207     243 and 160
//   8192 x 3072 x 3072     110 and 110            141 and 138        140 and 137     123 and 125  (power cap: +- 5 %)
// Outputs that are added to, row by row with scalar math, row by row, and so: fp32 8192 x 768 x 768 42.1, 32.5 and 19.7, 802816 x 64 x 256
// 430, 211 and 135; bf16 (D as its own residual) 24.6, 23.6 and 17.1, 162, 282 and 100.
// Taken back: results stored by the copy unit (cp.async.bulk.tensor; with one staging tile per warp each store waits for the
// one before to be read, and it writes whole 16-byte units past a ragged row's end): 802816 x 256 x 64 146 us. Sixteen epilogue
// warps of 96 registers: 32125 x 1024 x 256 with GELU 40 us, but 8192 x 3072 x 768 plain 35.5 and 0.6 us more per launch.

// The kernels exist for several kinds of epilogue, each with the code of a few flags only. With the code of all of them in one
// kernel every launch waits for instructions, also those of the branches it jumps over (us, one kernel and by kind):
// 69 x 768 x 768 8.1 and 7.3, 1218 x 256 x 256 6.1 and 5.1, 802816 x 64 x 64 74.9 and 38.8; on CTA pairs 50176 x 1024 x 256 32.6
// and 31.0, with a bias 45.3 and 37.1, with bias, GELU and pre-activation 66.0 and 60.4, + residual 53.6 and 51.0.
enum EpiKind : int {
  KIND_PLAIN,  // bias, ReLU, fp32 outputs
  KIND_GELU,   // bias, GELU, pre-activation
  KIND_DGELU,  // * GELU'
  KIND_TAIL,   // bias, norm, ReLU, residual
  KIND_ANY,    // every combination, outputs that are added to, and those that are not written in lines (epilogue_rows)
};
__host__ __device__ constexpr int kind_flags(int kind) {
  return kind == KIND_PLAIN  ? EPI_BIAS | EPI_RELU | EPI_ATOMIC | EPI_OUT_F32
         : kind == KIND_GELU  ? EPI_BIAS | EPI_GELU
         : kind == KIND_DGELU ? EPI_DGELU
         : kind == KIND_TAIL  ? EPI_BIAS | EPI_NORM | EPI_RELU | EPI_RELU_LAST | EPI_RESID
                              : ~0;
}
template <int KIND>
__device__ __forceinline__ int epi_flags(const GemmParams& p) {
  return p.flags & kind_flags(KIND);  // the bits a kind does not have are constants to the compiler
}

struct EpiWarp {
  uint8_t* tile;  // this warp's staging tiles
  uint64_t* bar;  // its tile loads
  uint32_t phase;
};

template <int KIND>
__device__ __forceinline__ bool epi_reads_aux(const GemmParams& p) {
  return (epi_flags<KIND>(p) & (EPI_DGELU | EPI_RESID)) != 0;
}

// Fetch the aux values of 32 rows x WCOLS columns, 64 per staging tile (one lane; the warp has finished with the tiles).
template <int WCOLS>
__device__ __forceinline__ void epi_fetch(const EpiWarp& w, const CUtensorMap& tmX, int row, int col) {
  fence_proxy_async_smem();
  mbar_expect_tx(w.bar, (WCOLS + 63) / 64 * EPI_TILE);
#pragma unroll
  for (int i = 0; i < (WCOLS + 63) / 64; ++i) tma_load_2d(w.tile + i * EPI_TILE, &tmX, w.bar, col + i * 64, row);
}

// Bias of 32 columns, packed; zeros past N.
__device__ __forceinline__ void epi_load_bias(const GemmParams& p, int col0, uint32_t (&b)[16]) {
  const __nv_bfloat16* src = p.bias + col0;
  if (col0 + 32 <= p.N && (reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint4 v = reinterpret_cast<const uint4*>(src)[k];  // the same address in every lane: a broadcast
      b[4 * k] = v.x, b[4 * k + 1] = v.y, b[4 * k + 2] = v.z, b[4 * k + 3] = v.w;
    }
  } else {
    const unsigned short* s16 = reinterpret_cast<const unsigned short*>(src);
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      const uint32_t lo = col0 + 2 * k < p.N ? s16[2 * k] : 0, hi = col0 + 2 * k + 1 < p.N ? s16[2 * k + 1] : 0;
      b[k] = lo | (hi << 16);
    }
  }
}

// 32 columns of a row into the staging tile, as bf16 chunks chunk0 .. chunk0 + 3 or as eight fp32 chunks. `row` = this lane's row
// of the tile, `x16` = (lane & 7) * 16, the swizzle.
__device__ __forceinline__ void epi_put_bf16(uint8_t* row, uint32_t x16, int chunk0, const uint64_t (&v)[16]) {
#pragma unroll
  for (int k = 0; k < 4; ++k)
    *reinterpret_cast<uint4*>(row + (((chunk0 + k) * 16) ^ x16)) =
        make_uint4(f2_to_bf16x2(v[4 * k]), f2_to_bf16x2(v[4 * k + 1]), f2_to_bf16x2(v[4 * k + 2]), f2_to_bf16x2(v[4 * k + 3]));
}
__device__ __forceinline__ void epi_put_f32(uint8_t* row, uint32_t x16, const uint64_t (&v)[16]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) *reinterpret_cast<ulonglong2*>(row + ((k * 16) ^ x16)) = make_ulonglong2(v[2 * k], v[2 * k + 1]);
}

// A staging tile into memory, eight lanes per row of 128 bytes; this lane's vectors go to column `col` (columns below `end`
// exist) of rows row_base + lane / 8, + 4, ... of `base`. Between two warp barriers.
enum EpiWrite : int { WRITE_STORE, WRITE_RED, WRITE_ADD };  // store, red.add, add to what this lane reads first (the last two fp32)
template <typename T>
__device__ __forceinline__ void epi_flush(void* base, long long ld, int M, int row_base, int col, int end, int how, const uint8_t* tile,
                                          int lane) {
  constexpr int PER16 = 16 / sizeof(T);
  const int c = lane & 7, sub = lane >> 3;
  const int rows = M - row_base - sub;  // this lane's rows are 0, 4, 8, ... while below
  T* dst = static_cast<T*>(base) + (long long)(row_base + sub) * ld + col;
  const uint8_t* even = tile + sub * 128 + ((c ^ sub) << 4);  // this lane's vectors in rows sub, sub + 8, ...
  const uint8_t* odd = tile + sub * 128 + ((c ^ (sub + 4)) << 4) + 512;  // ... and in rows sub + 4, sub + 12, ...
  if (col + PER16 <= end) {
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = *reinterpret_cast<const uint4*>(((i & 1) ? odd : even) + (i >> 1) * 1024);
    if (sizeof(T) == 4 && how == WRITE_ADD) {
      float4 o[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i * 4 < rows) o[i] = *reinterpret_cast<const float4*>(dst + i * 4 * ld);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i * 4 < rows)
          *reinterpret_cast<float4*>(dst + i * 4 * ld) = make_float4(__uint_as_float(v[i].x) + o[i].x, __uint_as_float(v[i].y) + o[i].y,
                                                                     __uint_as_float(v[i].z) + o[i].z, __uint_as_float(v[i].w) + o[i].w);
      return;
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i * 4 < rows) {
        if (sizeof(T) == 4 && how == WRITE_RED)
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(__uint_as_float(v[i].x)),
                       "f"(__uint_as_float(v[i].y)), "f"(__uint_as_float(v[i].z)), "f"(__uint_as_float(v[i].w))
                       : "memory");
        else
          *reinterpret_cast<uint4*>(dst) = v[i];
      }
      dst += 4 * ld;
    }
  } else if (col < end) {  // the last vector of a row whose length is not a whole number of vectors
#pragma unroll 1
    for (int i = 0; i < 8 && i * 4 < rows; ++i) {
      const T* v = reinterpret_cast<const T*>(((i & 1) ? odd : even) + (i >> 1) * 1024);
#pragma unroll 1
      for (int j = 0; j < end - col; ++j) {
        if constexpr (sizeof(T) == 4) {
          if (how == WRITE_RED) {
            atomicAdd(dst + j, v[j]);
            continue;
          }
          if (how == WRITE_ADD) {
            dst[j] += v[j];
            continue;
          }
        }
        dst[j] = v[j];
      }
      dst += 4 * ld;
    }
  }
}

// 32 accumulator columns of one row through the fused math into the staging tile: `half` says which half of its 128-byte row
// (bf16). The rounded pre-activation of EPI_GELU takes the other half (half = 1).
template <int KIND>
__device__ __forceinline__ void epi_chunk(const GemmParams& p, uint8_t* tile, const uint32_t (&r)[32], const uint32_t (&bias)[16],
                                          float scale, float shift, bool writes_z, int half, int lane) {
  const int flags = epi_flags<KIND>(p);
  uint8_t* row = tile + lane * 128;
  const uint32_t x16 = (lane & 7) << 4;
  uint64_t v[16];
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = pack_f2(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1]));
  if (flags & EPI_BIAS) {
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = add_f2(v[k], bf16x2_to_f2(bias[k]));
  }
  if (flags & EPI_NORM) col_norm_apply(v, scale, shift);
  if (flags & EPI_GELU) {
    if (writes_z) epi_put_bf16(row, x16, 0, v);
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = gelu_tanh_f2(v[k]);
  }
  if (flags & EPI_DGELU) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint4 a = *reinterpret_cast<const uint4*>(row + (((half * 4 + k) * 16) ^ x16));
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) v[4 * k + i] = mul_f2(v[4 * k + i], gelu_tanh_grad_f2(bf16x2_to_f2(aw[i])));
    }
  }
  if (flags & EPI_RELU) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      float lo, hi;
      unpack_f2(v[k], lo, hi);
      v[k] = pack_f2(fmaxf(lo, 0.f), fmaxf(hi, 0.f));
    }
  }
  if (flags & EPI_RESID) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint4 a = *reinterpret_cast<const uint4*>(row + (((half * 4 + k) * 16) ^ x16));
      const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) v[4 * k + i] = add_f2(v[4 * k + i], bf16x2_to_f2(aw[i]));
    }
  }
  if (flags & EPI_RELU_LAST) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      float lo, hi;
      unpack_f2(v[k], lo, hi);
      v[k] = pack_f2(fmaxf(lo, 0.f), fmaxf(hi, 0.f));
    }
  }
  if (flags & (EPI_ATOMIC | EPI_OUT_F32)) epi_put_f32(row, x16, v);
  else epi_put_bf16(row, x16, half * 4, v);
}

// 32 accumulator columns from col0 on (rows row_base + lane) through the math and, where the staging tile is complete, into
// memory: `odd` says that they are the second half of the tile's 64 columns, `last` that no more columns follow.
template <int KIND>
__device__ __forceinline__ void epi_finish(const GemmParams& p, const EpiOut& eo, uint8_t* tile, const uint32_t (&r)[32],
                                           const uint32_t (&bias)[16], float scale, float shift, int row_base, int col0, int odd,
                                           bool last, int end, int lane) {
  const bool f32 = (epi_flags<KIND>(p) & (EPI_ATOMIC | EPI_OUT_F32)) != 0;
  const bool writes_z = (epi_flags<KIND>(p) & EPI_GELU) && p.aux_out;
  const int half = writes_z ? 1 : odd;
  epi_chunk<KIND>(p, tile, r, bias, scale, shift, writes_z, half, lane);
  if (!(f32 || half == 1 || last)) return;
  __syncwarp();
  const int l8 = lane & 7;
  if (f32) {
    const int how = (epi_flags<KIND>(p) & EPI_ATOMIC) ? WRITE_RED : (epi_flags<KIND>(p) & EPI_ACCUM) ? WRITE_ADD : WRITE_STORE;
    epi_flush<float>(eo.D, eo.ldd, p.M, row_base, col0 + l8 * 4, end, how, tile, lane);
  } else if (writes_z) {  // 64 bytes of each row to either tensor
    epi_flush<__nv_bfloat16>(l8 < 4 ? p.aux_out : eo.D, l8 < 4 ? p.ld_aux : eo.ldd, p.M, row_base, col0 + (l8 & 3) * 8, end,
                             WRITE_STORE, tile, lane);
  } else {
    epi_flush<__nv_bfloat16>(eo.D, eo.ldd, p.M, row_base, col0 - half * 32 + l8 * 8, end, WRITE_STORE, tile, lane);
  }
  __syncwarp();
}

// One warp's share of a tile: WCOLS columns in groups of 32 at TMEM addresses t, t + 32, ..., from the `jump`-th group on at
// t2, t2 + 32, ...; rows row_base + lane, global columns from col_base on. next_row / next_col: where this warp's next tile
// lies (next_col < 0: there is none). wait_full() waits for the accumulator, release() hands it back. false: a wait ran out.
template <int WCOLS, int KIND, typename Wait, typename Release>
__device__ __forceinline__ bool epilogue_lines(const GemmParams& p, const EpiOut& eo, const CUtensorMap& tmX, EpiWarp& w, uint32_t t,
                                               uint32_t t2, int jump, int row_base, int col_base, int next_row, int next_col, int lane,
                                               volatile uint32_t* abort_flag, Wait wait_full, Release release) {
  constexpr int n = WCOLS / 32;
  const bool reads = epi_reads_aux<KIND>(p);
  const int end = min(p.N, col_base + WCOLS);
  // 64 columns per load from tensor memory in the short kernels, 32 in the others, whose code for each group is long
  constexpr int STEP = (KIND == KIND_PLAIN && n % 2 == 0) ? 2 : 1;
  uint32_t bias[16], bias_next[16], r[STEP][32];
  ColNormRaw raw_next{};
  if (epi_flags<KIND>(p) & EPI_BIAS) epi_load_bias(p, col_base, bias_next);
  if (epi_flags<KIND>(p) & EPI_NORM) raw_next = col_norm_load(p.norm, col_base + lane, p.N);
  if (!wait_full()) return false;
  tc_fence_after();
  if (reads) {
    if (!__all_sync(0xffffffffu, wait_or_abort(w.bar, w.phase, abort_flag))) return false;
    w.phase ^= 1;
  }
#pragma unroll 1
  for (int c0 = 0; c0 < n; c0 += STEP) {
    const uint32_t at = c0 < jump ? t + c0 * 32 : t2 + (c0 - jump) * 32;  // `jump` is a multiple of STEP
    if constexpr (STEP == 2) tmem_ld_32x64_wait(at, r[0], r[1]);  // warp-collective: never under a per-lane condition
    else tmem_ld_32x32_wait(at, r[0]);
    if (c0 + STEP == n) {
      tc_fence_before();
      __syncwarp();
      release();
    }
#pragma unroll
    for (int i = 0; i < STEP; ++i) {
      const int c = c0 + i, col0 = col_base + c * 32;
      uint8_t* tile = w.tile + (reads ? (c >> 1) * EPI_TILE : 0);
      if (epi_flags<KIND>(p) & EPI_BIAS) {  // loaded one group ahead: a bias from L2 costs as much as the rest of a group
#pragma unroll
        for (int k = 0; k < 16; ++k) bias[k] = bias_next[k];
        if (c + 1 < n) epi_load_bias(p, col0 + 32, bias_next);
      }
      float scale = 1.f, shift = 0.f;
      if (epi_flags<KIND>(p) & EPI_NORM) {
        col_norm_of(p.norm, raw_next, scale, shift);
        if (c + 1 < n) raw_next = col_norm_load(p.norm, col0 + 32 + lane, p.N);
      }
      epi_finish<KIND>(p, eo, tile, r[i], bias, scale, shift, row_base, col0, c & 1, c + 1 == n, end, lane);
    }
  }
  if (reads && lane == 0 && next_col >= 0) epi_fetch<WCOLS>(w, tmX, next_row, next_col);
  return true;
}

// The same share of a tile for outputs without aligned vectors and for two tensors beside the output:
// every lane loads and stores its own row, in vectors where those are aligned.
template <int WCOLS, typename Wait, typename Release>
__device__ __forceinline__ bool epilogue_rows(const GemmParams& p, const EpiOut& eo, uint32_t t, uint32_t t2, int jump, int row,
                                              int col_base, Wait wait_full, Release release) {
  if (!wait_full()) return false;
  tc_fence_after();
#pragma unroll 1
  for (int c = 0; c < WCOLS / 32; ++c) {
    const int col0 = col_base + c * 32;
    uint32_t r[32];
    tmem_ld_32x32_wait(c < jump ? t + c * 32 : t2 + (c - jump) * 32, r);
    float v[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
    if (row < p.M && col0 < p.N) {
      epilogue_math(p, eo, v, row, col0);
      epilogue_store_rowwise(p, eo, v, row, col0);
    }
  }
  tc_fence_before();
  __syncwarp();
  release();
  return true;
}

// After an abort: a tile load that nobody waited for lands before the CTA's shared memory goes away.
__device__ __forceinline__ void epi_drain(const EpiWarp& w, int lane) {
  if (lane != 0) return;
  const uint64_t t0 = globaltimer_ns();
  while (!mbar_try_wait(w.bar, w.phase))
    if (globaltimer_ns() - t0 > 200000000ull) break;
}

// BATCHED: the tensor maps have two more dimensions (head and sequence) and the work list runs over items x tiles; used for
// the per-head products of attention with head sizes the flash kernels do not cover.
template <int BN, int A_MN, int B_MN, int KIND, bool BATCHED = false>
__global__ void __launch_bounds__(64 + 32 * EPI_WARPS, 1)
gemm_bf16_tcgen05_kernel(const __grid_constant__ CUtensorMap tmA,
                         const __grid_constant__ CUtensorMap tmB, const GemmParams p, const __grid_constant__ CUtensorMap tmX) {
  using Cfg = GemmCfg<BN>;
  const int stages = p.stages;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  uint8_t* epi_tiles = smem + stages * Cfg::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(epi_tiles + EPI_WARPS * p.epi_tiles * EPI_TILE);
  uint64_t* aux_bars = full + BAR_AUX / 8;  // one per epilogue warp
  uint64_t* empty = full + Cfg::STAGES;
  uint64_t* tfull = empty + Cfg::STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int tiles = p.num_m_blocks * p.num_n_blocks;
  const int per_batch = tiles * p.split_k;
  const int total_work = per_batch * (BATCHED ? p.batch : 1);

  // The K blocks [kb0, kb1) of a work item, and the copy of one of them into an operand stage.
  auto k_range = [&](int work, int& kb0, int& kb1) {
    const int ks = (BATCHED ? work % per_batch : work) / tiles;
    kb0 = ks * p.kb_per_split;
    kb1 = min(kb0 + p.kb_per_split, p.num_k_blocks);
  };
  // (Where an item lies is worked out once: with the divisions in `load` the one thread that issues the copies was what a
  // long K waited for, 69 x 768 x 3072 in one range 17.4 and 19.9 us.)
  struct Place {
    int row, col, ah, ab, bh, bb;
  };
  auto place_of = [&](int work) {
    const int bi = BATCHED ? work / per_batch : 0;
    const int ai = BATCHED ? bi + p.a_off : 0, ab = BATCHED ? ai / p.a_heads : 0, ah = ai - ab * (BATCHED ? p.a_heads : 0);
    const int bj = BATCHED ? bi + p.b_off : 0, bb = BATCHED ? bj / p.b_heads : 0, bh = bj - bb * (BATCHED ? p.b_heads : 0);
    const int t = (work - bi * per_batch) % tiles;
    const int nb = t / p.num_m_blocks;
    return Place{(t - nb * p.num_m_blocks) * 128, nb * BN, ah, ab, bh, bb};
  };
  auto load = [&](const Place& at, int kb, int stage) {
    mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
    uint8_t* a_dst = smem + stage * Cfg::STAGE_BYTES;
    uint8_t* b_dst = a_dst + Cfg::A_BYTES;
    if (A_MN == 0) {
      if (BATCHED) tma_load_4d(a_dst, &tmA, &full[stage], kb * 64, at.row, at.ah, at.ab);
      else tma_load_2d(a_dst, &tmA, &full[stage], kb * 64, at.row);
    } else {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (BATCHED) tma_load_4d(a_dst + i * 8192, &tmA, &full[stage], at.row + i * 64, kb * 64, at.ah, at.ab);
        else tma_load_2d(a_dst + i * 8192, &tmA, &full[stage], at.row + i * 64, kb * 64);
      }
    }
    if (B_MN == 0) {
      if (BATCHED) tma_load_4d(b_dst, &tmB, &full[stage], kb * 64, at.col, at.bh, at.bb);
      else tma_load_2d(b_dst, &tmB, &full[stage], kb * 64, at.col);
    } else {
#pragma unroll
      for (int i = 0; i < BN / 64; ++i) {
        if (BATCHED) tma_load_4d(b_dst + i * 8192, &tmB, &full[stage], at.col + i * 64, kb * 64, at.bh, at.bb);
        else tma_load_2d(b_dst + i * 8192, &tmB, &full[stage], at.col + i * 64, kb * 64);
      }
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], EPI_WARPS);
    }
    for (int i = 0; i < EPI_WARPS; ++i) mbar_init(&aux_bars[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
    // The first stages are filled while the other warps get tensor memory and meet at the barrier: about 1000 of the 7500
    // clocks of a small product.
    grid_dep_wait();
    int kb0, kb1;
    k_range(blockIdx.x, kb0, kb1);
    const Place at = place_of(blockIdx.x);
    for (int i = 0; i < stages && kb0 + i < kb1; ++i) load(at, kb0 + i, i);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 2 * BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_launch();
  grid_dep_wait();

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      int last_stage = -1;
      uint32_t last_phase = 0;
      bool ok = true;
      for (int work = blockIdx.x; ok && work < total_work; work += gridDim.x) {
        int kb0, kb1;
        k_range(work, kb0, kb1);
        const Place at = place_of(work);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (work != (int)blockIdx.x || kb - kb0 >= stages) {  // else it is on its way already
            if (!wait_or_abort(&empty[stage], phase ^ 1, abort_flag)) {
              raise_abort(p.status, abort_flag, ST_TIMEOUT_PRODUCER);
              ok = false;
              break;
            }
            load(at, kb, stage);
          }
          last_stage = stage;
          last_phase = phase;
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
      if (!ok && last_stage >= 0) drain_stages(full, stages, last_stage, last_phase);  // before the CTA retires
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(128, BN, A_MN, B_MN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int work = blockIdx.x; ok && work < total_work; work += gridDim.x) {
        int kb0, kb1;
        k_range(work, kb0, kb1);
        if (!wait_or_abort(&tempty[acc], acc_phase ^ 1, abort_flag)) {
          raise_abort(p.status, abort_flag, ST_TIMEOUT_MMA);
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&full[stage], phase, abort_flag)) {
            raise_abort(p.status, abort_flag, ST_TIMEOUT_MMA);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint32_t b_addr = a_addr + Cfg::A_BYTES;
          // one descriptor per operand and k-block; its address field counts 16-byte units, so a k-step is an add
          const uint64_t ad0 = A_MN ? make_smem_desc(a_addr, 8192, 1024) : make_smem_desc(a_addr, 16, 1024);
          const uint64_t bd0 = B_MN ? make_smem_desc(b_addr, 8192, 1024) : make_smem_desc(b_addr, 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            tc_mma_ss(d_tmem, ad0 + k * (A_MN ? 128 : 2), bd0 + k * (B_MN ? 128 : 2), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
          tc_commit(&empty[stage]);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        tc_commit(&tfull[acc]);
        acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else {
    const int q = warp & 3;            // TMEM lane quarter this warp may read
    constexpr int WCOLS = BN / (EPI_WARPS / 4);  // columns per warp
    const int wcol = ((warp - 2) >> 2) * WCOLS;
    int acc = 0;
    uint32_t acc_phase = 0;
    EpiWarp ew = {epi_tiles + (warp - 2) * p.epi_tiles * EPI_TILE, aux_bars + (warp - 2), 0};
    // rows and columns of this warp in a work item
    auto place = [&](int work, int& row, int& col) {
      const int t = (BATCHED ? work % per_batch : work) % tiles;
      const int nb = t / p.num_m_blocks;
      row = (t - nb * p.num_m_blocks) * 128 + q * 32;
      col = nb * BN + wcol;
    };
    const bool lines = KIND != KIND_ANY || p.lines;
    const bool reads = lines && epi_reads_aux<KIND>(p);
    if (reads && lane == 0 && (int)blockIdx.x < total_work) {
      int row, col;
      place(blockIdx.x, row, col);
      epi_fetch<WCOLS>(ew, tmX, row, col);
    }
    bool ok = true;
    for (int work = blockIdx.x; work < total_work; work += gridDim.x) {
      int row_base, col_base, next_row = 0, next_col = -1;
      place(work, row_base, col_base);
      if (work + (int)gridDim.x < total_work) place(work + gridDim.x, next_row, next_col);
      const uint32_t t_addr = tmem_base + acc * BN + (static_cast<uint32_t>(q * 32) << 16) + wcol;
      long long d_off = 0;
      if (BATCHED) {
        const int di = work / per_batch + p.d_off, db = di / p.d_heads, dh = di - db * p.d_heads;
        d_off = (db * p.d_stride_b + dh * p.d_stride_h) * ((p.flags & (EPI_ATOMIC | EPI_OUT_F32)) ? 4 : 2);
      }
      const EpiOut eo = {static_cast<uint8_t*>(p.D) + d_off, p.ldd, p.flags};
      const auto release = [&] {
        if (lane == 0) mbar_arrive(&tempty[acc]);
      };
      const auto wait_full = [&] { return __all_sync(0xffffffffu, wait_or_abort(&tfull[acc], acc_phase, abort_flag)); };
      ok = lines ? epilogue_lines<WCOLS, KIND>(p, eo, tmX, ew, t_addr, t_addr, WCOLS / 32, row_base, col_base, next_row, next_col, lane,
                                           abort_flag, wait_full, release)
                   : epilogue_rows<WCOLS>(p, eo, t_addr, t_addr, WCOLS / 32, row_base + lane, col_base, wait_full, release);
      if (!ok) break;
      acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (!ok) {
      if (lane == 0) raise_abort(p.status, abort_flag, ST_TIMEOUT_EPILOGUE);
      if (reads) epi_drain(ew, lane);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// ------------------------------------------------------- K ranges in a cluster
// Products of a few 128 x 128 tiles: a cluster of S = 2 or 4 CTAs works on ONE tile, each on its own range of K blocks, and
// then every CTA adds up the S partial sums of its 128 / S columns, in the order of the ranges, and takes them through the
// fused math (k_ranges.cuh). What bounds such a product is the walk of one CTA over all of K (a K block of two 128 x 64 tiles
// takes 0.27 us: the 64 bytes per clock that one SM gets from L2), while most SMs idle. No atomics, no buffer in memory, the
// same result every time; error against fp64 no larger than with one range (shorter chains in the tensor core, which
// truncates: 69 x 768 x 3072 3.2e-6, 1.5e-6 with 2, 7.3e-7 with 4). Times: pick_ranges.
template <int B_MN, int KIND>
__global__ void __launch_bounds__(64 + 32 * EPI_WARPS, 1)
gemm_bf16_tcgen05_ranges_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GemmParams p,
                                const __grid_constant__ CUtensorMap tmX) {
  using Cfg = GemmCfg<128>;
  constexpr int STAGES = Cfg::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* epi_tiles = smem + STAGES * Cfg::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(epi_tiles + EPI_WARPS * EPI_TILE);
  uint64_t* aux_bars = full + BAR_AUX / 8;
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ranges = p.split_k, rank = (int)cluster_ctarank();  // the cluster is one row of `ranges` CTAs
  const int tile = (int)blockIdx.x / ranges;
  const int nb = tile / p.num_m_blocks, mb = tile - nb * p.num_m_blocks;
  const int kb0 = rank * p.kb_per_split, kb1 = min(kb0 + p.kb_per_split, p.num_k_blocks);  // never empty (host)
  const int W = 128 / ranges;
  auto load = [&](int i) {  // K block kb0 + i
    const int kb = kb0 + i, stage = i % STAGES;
    mbar_expect_tx(&full[stage], Cfg::STAGE_BYTES);
    uint8_t* a_dst = smem + stage * Cfg::STAGE_BYTES;
    uint8_t* b_dst = a_dst + Cfg::A_BYTES;
    tma_load_2d(a_dst, &tmA, &full[stage], kb * 64, mb * 128);
    if (B_MN == 0) {
      tma_load_2d(b_dst, &tmB, &full[stage], kb * 64, nb * 128);
    } else {
      tma_load_2d(b_dst, &tmB, &full[stage], nb * 128, kb * 64);
      tma_load_2d(b_dst + 8192, &tmB, &full[stage], nb * 128 + 64, kb * 64);
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    for (int i = 0; i < EPI_WARPS; ++i) mbar_init(&aux_bars[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
    grid_dep_wait();
    for (int i = 0; i < STAGES && kb0 + i < kb1; ++i) load(i);  // while the other warps set themselves up
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, 128);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  grid_dep_launch();
  grid_dep_wait();

  // epilogue warps: rows of this warp, and the columns it adds up (none for the second four warps with W <= 32)
  const int q = warp & 3, half = (warp - 2) >> 2;
  const int row_base = mb * 128 + q * 32;
  const int col_base = nb * 128 + rank * W + half * 32, end = min(p.N, col_base + 32);
  const bool adds = warp >= 2 && half * 32 < W;
  const bool reads = epi_reads_aux<KIND>(p);
  EpiWarp ew = {epi_tiles + (warp - 2) * EPI_TILE, aux_bars + (warp - 2), 0};
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      int last = min(STAGES, kb1 - kb0) - 1;
      for (int i = STAGES; i < kb1 - kb0; ++i) {
        if (!wait_or_abort(&empty[i % STAGES], ((i / STAGES) & 1) ^ 1, abort_flag)) {
          raise_abort(p.status, abort_flag, ST_TIMEOUT_PRODUCER);
          break;
        }
        load(i);
        last = i;
      }
      drain_stages(full, STAGES, last % STAGES, (last / STAGES) & 1);  // the cluster's partial sums are written over the stages
    }
    __syncwarp();
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(128, 128, 0, B_MN);
      for (int kb = kb0; ok && kb < kb1; ++kb) {
        const int i = kb - kb0, stage = i % STAGES;
        ok = wait_or_abort(&full[stage], (i / STAGES) & 1, abort_flag);
        if (!ok) {
          raise_abort(p.status, abort_flag, ST_TIMEOUT_MMA);
          break;
        }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + stage * Cfg::STAGE_BYTES);
        const uint32_t b_addr = a_addr + Cfg::A_BYTES;
        const uint64_t ad0 = make_smem_desc(a_addr, 16, 1024);
        const uint64_t bd0 = B_MN ? make_smem_desc(b_addr, 8192, 1024) : make_smem_desc(b_addr, 16, 1024);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          tc_mma_ss(tmem_base, ad0 + k * 2, bd0 + k * (B_MN ? 128 : 2), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
        tc_commit(&empty[stage]);
      }
      if (ok) tc_commit(tfull);
    }
    __syncwarp();
  } else {
    if (reads && adds && lane == 0) epi_fetch<64>(ew, tmX, row_base, col_base);
    ok = __all_sync(0xffffffffu, wait_or_abort(tfull, 0, abort_flag));
    if (!ok && lane == 0) raise_abort(p.status, abort_flag, ST_TIMEOUT_EPILOGUE);
  }
  // Every CTA passes both barriers, also after a wait that ran out (the result is then wrong and the status says so).
  cluster_sync_all();  // all MMAs of the cluster have finished: the operand stages are free
  if (warp >= 2 && ok) {
    tc_fence_after();
    ranges_push(smem_u32(smem), tmem_base, rank, W, q, half, lane);
    tc_fence_before();
  }
  __syncwarp();
  cluster_sync_all();  // the partial sums of this CTA's columns are here; no CTA leaves before its neighbours have written
  if (adds && ok) {
    uint32_t r[32], bias[16];
    ranges_sum(smem, ranges, W, q, half, lane, r);
    if (epi_flags<KIND>(p) & EPI_BIAS) epi_load_bias(p, col_base, bias);
    if (reads) ok = __all_sync(0xffffffffu, wait_or_abort(ew.bar, 0, abort_flag));
    float scale = 1.f, shift = 0.f;
    if (epi_flags<KIND>(p) & EPI_NORM) col_norm_of(p.norm, col_norm_load(p.norm, col_base + lane, p.N), scale, shift);
    if (ok) epi_finish<KIND>(p, EpiOut{p.D, p.ldd, p.flags}, ew.tile, r, bias, scale, shift, row_base, col_base, 0, true, end, lane);
    else if (lane == 0) raise_abort(p.status, abort_flag, ST_TIMEOUT_EPILOGUE);
  }
  if (!ok && reads && adds) epi_drain(ew, lane);

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 128);
  }
}

// ------------------------------------------------------------- CTA-pair kernel
// The same product on 256 x 256 tiles computed by a CTA PAIR (cluster of two, `cta_group::2`): each CTA
// stages its own 128 rows of A and HALF of the B tile (128 of the 256 N rows) per k-block, the even CTA's
// MMA thread issues one 256 x 256 x 16 instruction that reads both CTAs' shared memory and writes 128
// accumulator rows into each CTA's TMEM. Per SM this halves the B traffic through shared memory, which is
// what limits the single-CTA kernel (12 KB per instruction read by the tensor core plus the same written
// by TMA), and leaves room for six stages.
//   full[s]   lives in the even CTA; both CTAs' TMA loads count their bytes on it (no multicast of data)
//   empty[s]  one per CTA, signalled by a multicast tcgen05.commit
//   tfull[a]  one per CTA (multicast commit); tempty[a] in the even CTA, 8 local + 8 remote warp arrivals
template <int BN, int COMM = 0>
struct Gemm2Cfg {
  static constexpr int A_BYTES = 128 * 64 * 2;
  static constexpr int B_BYTES = (BN / 2) * 64 * 2;  // this CTA's half of the BN-row B tile
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  // mode 1 (COMM == 1) gives one operand stage to the two 16 KB stages of its copy thread (the 384-wide tile has
  // the room to spare)
  static constexpr int COPY_BYTES = (COMM == 1) ? 2 * 16384 : 0;
  static constexpr int STAGES = (BN == 384) ? 4 : (BN == 256) ? (COMM == 1 ? 5 : 6) : 8 - (COMM == 1 ? 2 : 0);
  static constexpr int ACCS = (BN == 384) ? 1 : 2;  // 384 columns leave no room for a second accumulator
  static constexpr int COPY_OFF = STAGES * STAGE_BYTES + BAR_BYTES + EPI_WARPS * EPI_TILE;
  // with a staging tile per 64 columns of an aux tensor there is one operand stage less
  static constexpr int AUX_TILES = BN / 2 / 64;
  static constexpr int AUX_BYTES = (STAGES - 1) * STAGE_BYTES + EPI_WARPS * AUX_TILES * EPI_TILE;
  static constexpr int PLAIN_BYTES = STAGES * STAGE_BYTES + EPI_WARPS * EPI_TILE + COPY_BYTES;
  static constexpr int SMEM_BYTES = 1024 + BAR_BYTES + (COMM == 0 && AUX_BYTES > PLAIN_BYTES ? AUX_BYTES : PLAIN_BYTES);
};
static_assert(Gemm2Cfg<256, 0>::SMEM_BYTES <= 227 * 1024 && Gemm2Cfg<384, 0>::SMEM_BYTES <= 227 * 1024, "shared memory");
static_assert(Gemm2Cfg<256, 1>::SMEM_BYTES <= 227 * 1024 && Gemm2Cfg<384, 1>::SMEM_BYTES <= 227 * 1024 &&
              Gemm2Cfg<128, 1>::SMEM_BYTES <= 227 * 1024, "mode-1 shared memory");

// Tile order of the tensor-parallel variants: the 256-row blocks are grouped by the rank that owns their rows;
// mode 1 runs the group of this rank first (its operand rows are already here), mode 2 runs it last (the partial
// sums for the peers have the longest way to go). Inside a group the row block index runs fastest, as in the
// plain order, so that neighbouring CTA pairs share a B tile.
template <int COMM>
__device__ __forceinline__ void pair_decode_tile(const GemmParams& p, const TpExt& x, int t, int& mb, int& nb) {
  if (COMM == 0 || x.pair_blocks_per_rank == 0) {
    nb = t / p.num_m_blocks;
    mb = t - nb * p.num_m_blocks;
    return;
  }
  const int bpr = x.pair_blocks_per_rank;
  const int per_group = bpr * p.num_n_blocks;
  const int g = t / per_group;
  const int u = t - g * per_group;
  const int owner = (x.rank + g + (COMM == 2 ? 1 : 0)) % x.tp;
  if (COMM == 1 && g > 0) {  // a peer's rows: row block by row block, the order they arrive in
    const int j = u / p.num_n_blocks;
    nb = u - j * p.num_n_blocks;
    mb = owner * bpr + j;
  } else {
    nb = u / bpr;
    mb = owner * bpr + (u - nb * bpr);
  }
}

// Reduce-scatter side: publish the partial sums this warp stored for its remote tiles. `upto` = first work item
// that is NOT covered (the warp has finished every tile before it). One system-scope fence, then one counter add
// per remote tile: the amount is the number of 32-column chunks the warp wrote, so the consumer's target,
// 4 x ceil(N / 32) per 128-row block and pass, does not depend on the tile width.
template <int BN>
__device__ __forceinline__ void tp_signal_remote_tiles(const GemmParams& p, const TpExt& x, int pair, int num_pairs, int upto,
                                                       uint32_t cta_rank, int half, int lane) {
  __syncwarp();
  if (lane == 0) {
    __threadfence_system();
    for (int work = pair; work < upto; work += num_pairs) {
      int mb, nb;
      pair_decode_tile<2>(p, x, work, mb, nb);
      const int row0 = mb * 256 + (int)cta_rank * 128;
      if (row0 >= p.M) continue;
      const int owner = row0 / x.rows_per_rank;
      if (owner == x.rank) continue;
      const int ncols = (BN == 384) ? 192 : BN / 2;
      const int c0 = nb * BN + half * ncols;
      const int c1 = min(c0 + ncols, p.N);
      if (c1 <= c0) continue;
      red_add_sys(x.arrived[owner] + (row0 - owner * x.rows_per_rank) / 128, (uint32_t)((c1 - c0 + 31) / 32));
    }
  }
  __syncwarp();
}

// Copy warp of mode 1 (one extra warp per CTA, one working thread): send this rank's rows of A to the peers with the
// bulk-copy unit while the tensor core works on the tiles of the rows that are already here. A piece is up to eight
// whole rows inside one 128-row block (at most TP_COPY_STAGE bytes); it is loaded from this rank's buffer into a
// shared-memory stage and stored from there into every peer's buffer (cp.async.bulk both ways, no multicast).
// Pieces are dealt to the CTAs of the grid in row order and each is published as soon as its stores have
// completed, so the row blocks fill up in the order in which the peers' GEMMs ask for them.
#define TP_COPY_WARPS 1
static constexpr int TP_COPY_STAGES = 2;
static constexpr int TP_COPY_STAGE = 16384;
__device__ __forceinline__ void tp_push_rows_bulk(const GemmParams& p, const TpExt& x, uint8_t* stage, uint64_t* bars,
                                                  int cta, int nctas) {
  const uint32_t row_bytes = (uint32_t)p.K * 2u;  // K % 8 == 0 and K * 2 <= TP_COPY_STAGE are checked on the host
  int piece_rows = 8;
  while (piece_rows > 1 && piece_rows * row_bytes > (uint32_t)TP_COPY_STAGE) piece_rows >>= 1;
  if (x.push_ld != p.K) piece_rows = 1;  // padded rows: only one row is contiguous
  const uint32_t bytes = piece_rows * row_bytes;
  const int total = (x.rows_per_rank / 128 - x.push_first_block) * (128 / piece_rows);
  const long long my0 = (long long)x.rank * x.rows_per_rank + (long long)x.push_first_block * 128;
  const int mine = total > cta ? (total - cta + nctas - 1) / nctas : 0;
  auto row_of = [&](int k) { return my0 + (long long)(cta + k * nctas) * piece_rows; };
  auto load = [&](int k) {
    const int s = k % TP_COPY_STAGES;
    mbar_expect_tx(&bars[s], bytes);
    bulk_load_g2s(stage + s * TP_COPY_STAGE, x.push_src + row_of(k) * x.push_ld, bytes, &bars[s]);
  };
  auto publish = [&](int k) {  // the stores of piece k have completed
    __threadfence_system();
    const long long r0 = row_of(k);
    for (int i = 0; i < x.push_n; ++i) red_add_sys(x.push_ready[i] + (r0 >> 7), (uint32_t)piece_rows);
  };
  int issued = 0, done = 0;
  for (; issued < mine && issued < TP_COPY_STAGES; ++issued) load(issued);
  for (int k = 0; k < mine; ++k) {
    const int s = k % TP_COPY_STAGES;
    if (!mbar_wait(&bars[s], (uint32_t)((k / TP_COPY_STAGES) & 1))) {
      if (p.status) atomicOr(p.status, ST_TIMEOUT_PRODUCER);
      break;
    }
    const long long r0 = row_of(k);
    for (int i = 0; i < x.push_n; ++i) bulk_store_s2g(x.push_dst[i] + r0 * x.push_ld, stage + s * TP_COPY_STAGE, bytes);
    bulk_commit_group();
    done = k + 1;
    if (k >= 1) {
      asm volatile("cp.async.bulk.wait_group 1;" ::: "memory");  // piece k - 1 has arrived: its stage is free as well
      publish(k - 1);
      if (issued < mine) load(issued++);
    }
  }
  bulk_wait_group0();
  if (done) publish(done - 1);
  // loads issued but not consumed (only after a time-out): let them land before the block's shared memory goes away
  for (int k = done; k < issued; ++k) mbar_wait(&bars[k % TP_COPY_STAGES], (uint32_t)((k / TP_COPY_STAGES) & 1));
}

template <int BN, int A_MN, int B_MN, int COMM, int KIND>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(64 + 32 * EPI_WARPS + (COMM == 1 ? 32 * TP_COPY_WARPS : 0), 1)
gemm_bf16_tcgen05_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                              const GemmParams p, const __grid_constant__ TpExt tpx, const __grid_constant__ CUtensorMap tmX) {
  using Cfg = Gemm2Cfg<BN, COMM>;
  const int stages = COMM == 0 ? p.stages : Cfg::STAGES;
  const int epi_tiles_each = COMM == 0 ? p.epi_tiles : 1;
  constexpr int HALF = BN / 2;  // B rows (output columns) staged by each CTA
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
  uint8_t* epi_tiles = smem + stages * Cfg::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(epi_tiles + EPI_WARPS * epi_tiles_each * EPI_TILE);
  uint64_t* aux_bars = full + BAR_AUX / 8;  // one per epilogue warp (COMM == 0)
  uint64_t* empty = full + Cfg::STAGES;
  uint64_t* tfull = empty + Cfg::STAGES;
  uint64_t* tempty = tfull + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty + 2);
  volatile uint32_t* abort_flag = tmem_slot + 1;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0: issues the MMAs, 1: partner
  const int pair = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull[a], 1);
      mbar_init(&tempty[a], 2 * EPI_WARPS);
    }
    if (COMM == 0)
      for (int i = 0; i < EPI_WARPS; ++i) mbar_init(&aux_bars[i], 1);
    if (COMM == 1)
      for (int s = 0; s < TP_COPY_STAGES; ++s) mbar_init(&full[24 + s], 1);  // copy thread's stages (byte 192 of the barrier block)
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the partner's barriers and tensor memory exist before anything refers to them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  if (COMM == 0) {  // the tensor-parallel forms wait for other GPUs: plain stream order
    grid_dep_launch();
    grid_dep_wait();
  }

  const int tiles = p.num_m_blocks * p.num_n_blocks;  // in units of 256 x BN
  const int total_work = tiles * p.split_k;

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      const uint32_t a_want = (COMM == 1) ? 128u * *tpx.pass : 0u;
      for (int work = pair; ok && work < total_work; work += num_pairs) {
        const int ks = work / tiles;
        const int t = work - ks * tiles;
        int mb, nb;
        pair_decode_tile<COMM>(p, tpx, t, mb, nb);
        const int row0 = mb * 256 + (int)rank * 128;   // this CTA's rows of A
        const int col0 = nb * BN + (int)rank * HALF;   // this CTA's rows of B (output columns)
        const int kb0 = ks * p.kb_per_split;
        const int kb1 = min(kb0 + p.kb_per_split, p.num_k_blocks);
        if (COMM == 1 && row0 < p.M && row0 / tpx.rows_per_rank != tpx.rank) {
          // rows pushed by their owner: wait until the whole 128-row block has landed, then make the peer's
          // (generic-proxy) stores visible to the TMA reads that follow
          if (!spin_until<true>(tpx.a_ready + (row0 >> 7), a_want)) {
            raise_abort(p.status, abort_flag, ST_TIMEOUT_PEER);
            ok = false;
            break;
          }
          fence_proxy_async_all();
        }
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&empty[stage], phase ^ 1, abort_flag)) {
            raise_abort(p.status, abort_flag, ST_TIMEOUT_PRODUCER);
            ok = false;
            break;
          }
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * Cfg::STAGE_BYTES);
          const uint32_t bar = mapa_shared(smem_u32(&full[stage]), 0);
          uint8_t* a_dst = smem + stage * Cfg::STAGE_BYTES;
          uint8_t* b_dst = a_dst + Cfg::A_BYTES;
          if (A_MN == 0) {
            tma_load_2d_pair(a_dst, &tmA, bar, kb * 64, row0);
          } else {
#pragma unroll
            for (int i = 0; i < 2; ++i) tma_load_2d_pair(a_dst + i * 8192, &tmA, bar, row0 + i * 64, kb * 64);
          }
          if (B_MN == 0) {
            tma_load_2d_pair(b_dst, &tmB, bar, kb * 64, col0);
          } else {
#pragma unroll
            for (int i = 0; i < HALF / 64; ++i) tma_load_2d_pair(b_dst + i * 8192, &tmB, bar, col0 + i * 64, kb * 64);
          }
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(256, BN == 384 ? 256 : BN, A_MN, B_MN);
      constexpr uint32_t idesc_tail = make_idesc_bf16(256, 128, A_MN, B_MN);  // BN == 384 only
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int work = pair; ok && work < total_work; work += num_pairs) {
        const int ks = work / tiles;
        const int kb0 = ks * p.kb_per_split;
        const int kb1 = min(kb0 + p.kb_per_split, p.num_k_blocks);
        if (!wait_or_abort(&tempty[acc], acc_phase ^ 1, abort_flag)) {
          raise_abort(p.status, abort_flag, ST_TIMEOUT_MMA);
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * (BN == 384 ? 0 : BN);
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!wait_or_abort(&full[stage], phase, abort_flag)) {
            raise_abort(p.status, abort_flag, ST_TIMEOUT_MMA);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + stage * Cfg::STAGE_BYTES);
          const uint32_t b_addr = a_addr + Cfg::A_BYTES;
          const uint64_t ad0 = A_MN ? make_smem_desc(a_addr, 8192, 1024) : make_smem_desc(a_addr, 16, 1024);
          const uint64_t bd0 = B_MN ? make_smem_desc(b_addr, 8192, 1024) : make_smem_desc(b_addr, 16, 1024);
          // this CTA's B rows 128..191 (BN == 384 only): two 64-row boxes further when MN-major
          const uint64_t bt0 = B_MN ? make_smem_desc(b_addr + 2 * 8192, 8192, 1024) : make_smem_desc(b_addr + 128 * 128, 16, 1024);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint64_t ad = ad0 + k * (A_MN ? 128 : 2);
            tc_mma_ss_pair(d_tmem, ad, bd0 + k * (B_MN ? 128 : 2), idesc, (kb > kb0 || k > 0) ? 1u : 0u);
            if (BN == 384) tc_mma_ss_pair(d_tmem + 256, ad, bt0 + k * (B_MN ? 128 : 2), idesc_tail, (kb > kb0 || k > 0) ? 1u : 0u);
          }
          tc_commit_pair(&empty[stage], 3);
          if (++stage == stages) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        tc_commit_pair(&tfull[acc], 3);
        if (Cfg::ACCS == 2) acc ^= 1;
        if (acc == 0) acc_phase ^= 1;
      }
    }
  } else if (COMM == 1 && warp >= 10) {
    if (tpx.push_n > 0)
      if (lane == 0) tp_push_rows_bulk(p, tpx, smem + Cfg::COPY_OFF, &full[24], (int)blockIdx.x, (int)gridDim.x);
  } else if (COMM == 0) {
    const int q = warp & 3, half = (warp - 2) >> 2;
    constexpr int WCOLS = BN / (EPI_WARPS / 4);  // columns per warp
    int acc = 0;
    uint32_t acc_phase = 0;
    const uint32_t tempty_remote = mapa_shared(smem_u32(&tempty[0]), 0);  // 8 bytes per accumulator
    EpiWarp ew = {epi_tiles + (warp - 2) * p.epi_tiles * EPI_TILE, aux_bars + (warp - 2), 0};
    auto place = [&](int w, int& row, int& col) {  // rows and columns of this warp in a work item
      const int t = w % tiles;
      const int nb = t / p.num_m_blocks;
      row = (t - nb * p.num_m_blocks) * 256 + (int)rank * 128 + q * 32;
      col = nb * BN + half * WCOLS;
    };
    // tensor memory of this warp's columns; BN == 384: 128 columns of the first product, then 64 of the second
    const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
    constexpr int JUMP = BN == 384 ? 4 : WCOLS / 32;
    const bool lines = KIND != KIND_ANY || p.lines;
    const bool reads = lines && epi_reads_aux<KIND>(p);
    if (reads && lane == 0 && pair < total_work) {
      int row, col;
      place(pair, row, col);
      epi_fetch<WCOLS>(ew, tmX, row, col);
    }
    bool ok = true;
    for (int work = pair; work < total_work; work += num_pairs) {
      int row_base, col_base, next_row = 0, next_col = -1;
      place(work, row_base, col_base);
      if (work + num_pairs < total_work) place(work + num_pairs, next_row, next_col);
      const uint32_t t_addr = t_lane + half * (BN == 384 ? 128 : WCOLS) + acc * (BN == 384 ? 0 : BN);
      const EpiOut eo = {p.D, p.ldd, p.flags};
      const auto release = [&] {
        if (lane == 0) mbar_arrive_cluster(tempty_remote + acc * 8);
      };
      const auto wait_full = [&] { return __all_sync(0xffffffffu, wait_or_abort(&tfull[acc], acc_phase, abort_flag)); };
      ok = lines ? epilogue_lines<WCOLS, KIND>(p, eo, tmX, ew, t_addr, t_lane + 256 + half * 64, JUMP, row_base, col_base, next_row, next_col,
                                           lane, abort_flag, wait_full, release)
                   : epilogue_rows<WCOLS>(p, eo, t_addr, t_lane + 256 + half * 64, JUMP, row_base + lane, col_base, wait_full, release);
      if (!ok) break;
      if (Cfg::ACCS == 2) acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    if (!ok) {
      if (lane == 0) raise_abort(p.status, abort_flag, ST_TIMEOUT_EPILOGUE);
      if (reads) epi_drain(ew, lane);
    }
  } else {
    const int q = warp & 3;
    const int half = (warp - 2) >> 2;
    int acc = 0;
    uint32_t acc_phase = 0;
    const uint32_t tempty_remote = mapa_shared(smem_u32(&tempty[0]), 0);  // 8 bytes per accumulator
    bool unsignalled = false;  // COMM == 2: remote tiles stored but not yet published
    int work = pair;
    for (; work < total_work; work += num_pairs) {
      const int ks = work / tiles;
      const int t = work - ks * tiles;
      int mb, nb;
      pair_decode_tile<COMM>(p, tpx, t, mb, nb);
      const int row_cta = mb * 256 + (int)rank * 128;
      EpiOut eo = {p.D, p.ldd, p.flags};
      if (COMM == 2) {
        const int owner = min(row_cta / tpx.rows_per_rank, tpx.tp - 1);
        const bool remote = owner != tpx.rank;
        if (!remote && unsignalled) {  // the last remote tile of this CTA is behind us
          tp_signal_remote_tiles<BN>(p, tpx, pair, num_pairs, work, rank, half, lane);
          unsignalled = false;
        }
        // block of the owning rank, addressed with the global row index
        eo.D = reinterpret_cast<__nv_bfloat16*>(tpx.out[owner]) - (long long)owner * tpx.rows_per_rank * tpx.ldo;
        eo.ldd = tpx.ldo;
        if (remote) eo.flags = p.flags & ~EPI_BIAS;
        unsignalled = unsignalled || (remote && row_cta < p.M);
      }
      if (!wait_or_abort(&tfull[acc], acc_phase, abort_flag)) {
        if (lane == 0) raise_abort(p.status, abort_flag, ST_TIMEOUT_EPILOGUE);
        break;
      }
      tc_fence_after();
      uint8_t* stage_tile = epi_tiles + (warp - 2) * EPI_TILE;
      const int row_base = row_cta + q * 32;
      if (BN == 384) {
        // warp half h owns output columns [h*192, h*192+192): 128 from the first product, 64 from the second
        const uint32_t t_lane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
        epilogue_warp(p, eo, t_lane + half * 128, 4, row_base, nb * BN + half * 192, lane, stage_tile);
        epilogue_warp(p, eo, t_lane + 256 + half * 64, 2, row_base, nb * BN + half * 192 + 128, lane, stage_tile);
      } else {
        const uint32_t t_addr = tmem_base + acc * BN + (static_cast<uint32_t>(q * 32) << 16) + half * HALF;
        epilogue_warp(p, eo, t_addr, HALF / 32, row_base, nb * BN + half * HALF, lane, stage_tile);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(tempty_remote + acc * 8);
      if (Cfg::ACCS == 2) acc ^= 1;
      if (acc == 0) acc_phase ^= 1;
    }
    // also after an aborted loop: whatever was stored is published, the peers' counters stay consistent
    if (COMM == 2 && unsignalled) tp_signal_remote_tiles<BN>(p, tpx, pair, num_pairs, work, rank, half, lane);
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // no CTA frees tensor memory or exits while its partner may still touch it
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// ------------------------------------------------------------------ host
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

int encode_tmap_bf16(CUtensorMap* m, const void* base, int rank, const uint64_t* dims,
                     const uint64_t* strides_bytes, const uint32_t* box,
                     const uint32_t* elem_strides) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return -1;
  cuuint64_t gdim[5];
  cuuint64_t gstr[5];
  cuuint32_t bx[5];
  cuuint32_t es[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bx[i] = box[i];
    es[i] = elem_strides ? elem_strides[i] : 1;
    if (i > 0) gstr[i - 1] = strides_bytes[i - 1];
  }
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), gdim, gstr,
                  bx, es, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -static_cast<int>(r) - 100;
}

// Same as encode_tmap_bf16 for fp32 elements (128-byte swizzle: the inner box extent is at most 32 elements).
int encode_tmap_f32(CUtensorMap* m, const void* base, int rank, const uint64_t* dims, const uint64_t* strides_bytes,
                    const uint32_t* box) {
  EncodeTiledFn fn = get_encode_fn();
  if (!fn) return -1;
  cuuint64_t gdim[5];
  cuuint64_t gstr[5];
  cuuint32_t bx[5];
  cuuint32_t es[5];
  for (int i = 0; i < rank; ++i) {
    gdim[i] = dims[i];
    bx[i] = box[i];
    es[i] = 1;
    if (i > 0) gstr[i - 1] = strides_bytes[i - 1];
  }
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, rank, const_cast<void*>(base), gdim, gstr, bx, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -static_cast<int>(r) - 100;
}

int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n <= 0) n = 148;
  }
  return n;
}

template <int BN, int A_MN, int B_MN, int KIND, bool BATCHED = false>
static int launch_gemm(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, const CUtensorMap& tx, int grid,
                       cudaStream_t stream) {
  auto kern = gemm_bf16_tcgen05_kernel<BN, A_MN, B_MN, KIND, BATCHED>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         GemmCfg<BN>::SMEM_BYTES);
    if (e != cudaSuccess) return -static_cast<int>(e) - 1000;
    attr_set = true;
  }
  const cudaError_t e = launch_dependent(kern, dim3(grid), dim3(64 + 32 * EPI_WARPS), GemmCfg<BN>::SMEM_BYTES, stream, ta, tb, p, tx);
  return e == cudaSuccess ? 0 : -static_cast<int>(e) - 1000;
}

template <int B_MN, int KIND>
static int launch_gemm_ranges(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, const CUtensorMap& tx, int tiles,
                              cudaStream_t stream) {
  auto kern = gemm_bf16_tcgen05_ranges_kernel<B_MN, KIND>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GemmCfg<128>::SMEM_BYTES);
    if (e != cudaSuccess) return -static_cast<int>(e) - 1000;
    attr_set = true;
  }
  const cudaError_t e = launch_dependent_cluster(kern, p.split_k, dim3(tiles * p.split_k), dim3(64 + 32 * EPI_WARPS),
                                                 GemmCfg<128>::SMEM_BYTES, stream, ta, tb, p, tx);
  return e == cudaSuccess ? 0 : -static_cast<int>(e) - 1000;
}

template <int BN, int A_MN, int B_MN, int KIND, int COMM = 0>
static int launch_gemm_pair(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, const CUtensorMap& tx, int grid,
                            cudaStream_t stream, const TpExt& tpx = TpExt{}) {
  auto kern = gemm_bf16_tcgen05_pair_kernel<BN, A_MN, B_MN, COMM, KIND>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, Gemm2Cfg<BN, COMM>::SMEM_BYTES);
    if (e != cudaSuccess) return -static_cast<int>(e) - 1000;
    attr_set = true;
  }
  cudaError_t e;  // cluster of two through __cluster_dims__
  if (COMM == 0) {
    e = launch_dependent(kern, dim3(grid), dim3(64 + 32 * EPI_WARPS), Gemm2Cfg<BN, COMM>::SMEM_BYTES, stream, ta, tb, p, tpx, tx);
  } else {
    kern<<<grid, COMM == 1 ? 320 + 32 * TP_COPY_WARPS : 320, Gemm2Cfg<BN, COMM>::SMEM_BYTES, stream>>>(ta, tb, p, tpx, tx);
    e = cudaGetLastError();
  }
  return e == cudaSuccess ? 0 : -static_cast<int>(e) - 1000;
}

// Whether epilogue_lines covers this call, and the tensor map of the aux tensor it reads.
static bool epi_lines(const GemmParams& p, CUtensorMap& tx) {
  const bool f32 = (p.flags & (EPI_ATOMIC | EPI_OUT_F32)) != 0;
  const bool dgelu = p.flags & EPI_DGELU, resid = p.flags & EPI_RESID, z = (p.flags & EPI_GELU) && p.aux_out;
  if ((p.flags & EPI_ACCUM) && !f32) return false;
  if (dgelu + resid + z > 1 || (f32 && (dgelu || resid || z))) return false;
  const auto fits = [](const void* base, long long ld, int elem) {
    return (reinterpret_cast<uintptr_t>(base) & 15) == 0 && ld > 0 && (ld * elem) % 16 == 0;
  };
  if (!fits(p.D, p.ldd, f32 ? 4 : 2)) return false;
  if (z) return fits(p.aux_out, p.ld_aux, 2);
  if (dgelu || resid) {
    const void* base = dgelu ? p.aux_in : p.resid;
    const long long ld = resid ? p.ld_res : p.ld_aux;
    const uint64_t dims[2] = {(uint64_t)p.N, (uint64_t)p.M}, pitch[1] = {(uint64_t)ld * 2};
    const uint32_t box[2] = {64, 32};
    return fits(base, ld, 2) && encode_tmap_bf16(&tx, base, 2, dims, pitch, box, nullptr) == 0;
  }
  return true;
}

// The kernel kind with the least code that does what this call asks for.
static int epi_kind(const GemmParams& p) {
  if (!p.lines) return KIND_ANY;
  const int flags = p.flags & EPI_ATOMIC ? p.flags & ~EPI_ACCUM : p.flags;  // what is added with red.add is added anyway
  for (int kind = KIND_PLAIN; kind < KIND_ANY; ++kind)
    if (!(flags & ~kind_flags(kind))) return kind;
  return KIND_ANY;
}

// Kinds are compiled for the operand orders in which layers use them (forward products with a GELU or a tail, data gradients
// with GELU' or a residual); other combinations run as KIND_ANY.
template <int BN>
static int launch_single_kind(int kind, int a_mn, int b_mn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                              const CUtensorMap& tx, int grid, cudaStream_t stream) {
#define TNNB_LAUNCH(AM, BM, K) return launch_gemm<BN, AM, BM, K>(ta, tb, p, tx, grid, stream)
#define TNNB_ORDERS(K)                    \
  do {                                    \
    if (!a_mn && !b_mn) TNNB_LAUNCH(0, 0, K); \
    if (!a_mn && b_mn) TNNB_LAUNCH(0, 1, K);  \
    if (a_mn && !b_mn) TNNB_LAUNCH(1, 0, K);  \
    TNNB_LAUNCH(1, 1, K);                 \
  } while (0)
  if (kind == KIND_PLAIN) TNNB_ORDERS(KIND_PLAIN);
  if constexpr (BN != 256) {
    if (kind == KIND_GELU && !a_mn && !b_mn) TNNB_LAUNCH(0, 0, KIND_GELU);
    if (kind == KIND_DGELU && !a_mn && b_mn) TNNB_LAUNCH(0, 1, KIND_DGELU);
    if (kind == KIND_TAIL && !a_mn && !b_mn) TNNB_LAUNCH(0, 0, KIND_TAIL);
    if (kind == KIND_TAIL && !a_mn && b_mn) TNNB_LAUNCH(0, 1, KIND_TAIL);
  }
  TNNB_ORDERS(KIND_ANY);
#undef TNNB_LAUNCH
}
template <int BN>
static int launch_pair_kind(int kind, int a_mn, int b_mn, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                            const CUtensorMap& tx, int grid, cudaStream_t stream) {
#define TNNB_LAUNCH(AM, BM, K) return launch_gemm_pair<BN, AM, BM, K>(ta, tb, p, tx, grid, stream)
  if (kind == KIND_PLAIN) TNNB_ORDERS(KIND_PLAIN);
  if (kind == KIND_GELU && !a_mn && !b_mn) TNNB_LAUNCH(0, 0, KIND_GELU);
  if (kind == KIND_DGELU && !a_mn && b_mn) TNNB_LAUNCH(0, 1, KIND_DGELU);
  if (kind == KIND_TAIL && !a_mn && b_mn) TNNB_LAUNCH(0, 1, KIND_TAIL);
  if (kind == KIND_TAIL && !a_mn && !b_mn) TNNB_LAUNCH(0, 0, KIND_TAIL);
  TNNB_ORDERS(KIND_ANY);
#undef TNNB_ORDERS
#undef TNNB_LAUNCH
}

// Number of K ranges of a product whose result is added with red.add (weight gradients: few tiles, a long K). At least
// as many as give about two waves of work items (tiles x ranges) on the `units` CTAs or CTA pairs: the tensor core
// truncates as it accumulates, so the error against fp64 grows with the length of a range (768 x 768 x 8192: 4.8e-7 with
// 17 ranges, 1.0e-6 with 8, 9.1e-6 with 1) and is what bounds a range from above. From there on the count whose items
// fill their waves best: a wave costs its K blocks plus about ten more for handing over the accumulators and adding
// them to memory (a K block of a 256 x 256 pair tile takes 0.265 us, a wave's epilogue 2.7 us: sweep over 21 shapes).
// 2304 x 768 x 8192 (27 tiles on 74 pairs): 8 ranges 31.0 us, 6 ranges 34.9; 3072 x 768 x 8192: 6 ranges 36.8 us, 5
// ranges 39.2.
static int pick_split_k(int tiles, int num_k_blocks, int units) {
  const int top = max(num_k_blocks / 4, 1);
  const int least = max(1, min((2 * units + tiles - 1) / tiles, top));
  int best = least;
  long long best_cost = -1;
  for (int s = least; s <= min(top, 2 * least); ++s) {
    const int kbs = (num_k_blocks + s - 1) / s;
    const int ranges = (num_k_blocks + kbs - 1) / kbs;
    const long long waves = ((long long)tiles * ranges + units - 1) / units;
    const long long cost = waves * (kbs + 10);
    if (best_cost < 0 || cost < best_cost) {
      best_cost = cost;
      best = s;
    }
  }
  return best;
}

// Number of K ranges for a product of `tiles` 128 x 128 tiles on the cluster kernel, or 1. The exchange of the partial sums
// and the two cluster barriers cost about as much as eight K blocks (2 ranges) or twelve (4), and more CTAs than SMs would run
// one after the other. Us per launch with 1, 2 and 4 ranges: 69 x 768 x 3072 (48 K blocks) 18.3, 13.9, 11.8; 343 x 512 x 2048
// (32) 14.2, 11.8, 11.0; 999 x 320 x 1280 (20) 10.9, 10.1, 11.3; 1218 x 256 x 1024 (16) 9.7, 9.5, 10.1; 69 x 768 x 768 (12) 8.1,
// 8.6, 9.2; 1024 x 768 x 3072, 48 tiles, 19.6, 15.6, 25.0. Eight ranges are nowhere better than four (69 x 1024 x 4096 13.1, 12.9).
int pick_ranges(long long tiles, int num_k_blocks) {
  const int s = num_k_blocks >= 28 && tiles * 4 <= sm_count() ? 4 : num_k_blocks >= 20 && tiles * 2 <= sm_count() ? 2 : 1;
  const int per = (num_k_blocks + s - 1) / s;
  return (s - 1) * per < num_k_blocks ? s : 1;  // no range is empty
}

}  // namespace tnnb

using namespace tnnb;

static int gemm_dispatch(const void* A, const void* B, void* D, int M, int N, int K, int a_mn,
                         int b_mn, long long lda, long long ldb, long long ldd,
                         const void* bias, const void* aux_in, void* aux_out,
                         long long ld_aux, const void* resid, long long ld_res, int flags,
                         int split_k, int force_bn, int* status, void* stream_, const TpExt* tpx, const ColNorm* norm = nullptr) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0) return -2;
  if ((lda % 8) || (ldb % 8)) return -3;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -4;
  if ((flags & EPI_BIAS) && !bias) return -5;
  if ((flags & EPI_DGELU) && !aux_in) return -5;
  if ((flags & EPI_RESID) && !resid) return -5;
  if ((flags & EPI_NORM) && (!norm || !norm->mean || !norm->var)) return -5;
  if ((flags & EPI_ACCUM) && !(flags & (EPI_ATOMIC | EPI_OUT_F32 | EPI_RESID))) {  // bf16 D += ...: D is its own residual
    flags = (flags & ~EPI_ACCUM) | EPI_RESID;
    resid = D;
    ld_res = ldd;
  }

  GemmParams p;
  p.M = M; p.N = N; p.K = K;
  // 256 x 256 tiles on CTA pairs where the problem has more than 128 rows and columns, but for the small problems named
  // below (force_bn: 512 forces the pair kernel, 64 / 128 / 256 force the single-CTA tile widths)
  int pair_bn = 0;  // force_bn = 1024 + 256 / 384: the pair kernel with that tile width
  int ranges = 0;   // force_bn = 2048 + 2 / 4: the cluster kernel with that many K ranges
  const bool automatic = force_bn == 0 && split_k <= 0;  // split_k = 1 asks for one range
  if (force_bn >= 2048) {
    ranges = force_bn - 2048;
    const int kbs = (K + 63) / 64, per = (kbs + max(ranges, 1) - 1) / max(ranges, 1);
    if ((ranges != 2 && ranges != 4) || a_mn || tpx || (flags & EPI_ATOMIC) || (ranges - 1) * per >= kbs) return -6;
    force_bn = 128;
  } else if (force_bn >= 1024) {
    pair_bn = force_bn - 1024;
    force_bn = 512;
  }
  bool pair = (force_bn == 512) || (force_bn == 0 && M > 128 && N > 128);
  int bn = force_bn;
  // Problems of at most one 128 x 128 tile per SM take single CTAs: the pair kernel's cluster barriers and 512 columns of
  // tensor memory cost about 2 us per launch, which its faster main loop (half the B traffic per SM) does not earn back in
  // one tile. Us per launch, pair and single CTA: 1218 x 768 x 256 7.8 and 5.8, 1024 x 768 x 768 10.5 and 8.5, 343 x 2048 x
  // 512 9.0 and 6.9, 1024 x 768 x 3072 20.7 and 19.6; with more tiles the pair wins (4096 x 3072 x 1024 23.9 and 37.6). One
  // 128 x 256 tile per SM is faster than the pair alone (4096 x 1024 x 1024 11.2 and 12.2) but not among other kernels:
  // GPT-2 medium forward 4361 -> 4612 us. The accumulation order is the same.
  // Added products (red.add) only where both would split K into the same ranges, the shortest allowed (four K blocks).
  if (pair && force_bn == 0 && !tpx) {
    const long long rows = (M + 127) / 128;
    const long long t128 = rows * ((N + 127) / 128);
    if (flags & EPI_ATOMIC) {
      if (split_k <= 0 && t128 <= 36 && K <= 2048) pair = false, bn = 128;
    } else if (t128 <= sm_count()) {
      pair = false, bn = 128;
    }
  }
  p.num_m_blocks = pair ? (M + 255) / 256 : (M + 127) / 128;
  p.num_k_blocks = (K + 63) / 64;
  if (pair) {
    // 256-wide tiles (narrower pair tiles are limited by shared-memory bandwidth: A is re-read per 128
    // columns), or 384-wide ones with a single accumulator when they need clearly fewer waves of CTA pairs
    // (N = 768 with 8192 rows: 64 tiles on 74 pairs instead of 96).
    // With a tensor read beside the output the wider tile has one operand stage less and is still the faster one: 256 and 384 wide with a
    // residual 8192 x 768 x 768 17.6 and 17.0, x 3072 39.2 and 35.6, x 6144 74.4 and 64.2, times GELU' 19.1 and 18.8, 40.9 and 37.4, 84 and 72.
    const int units = sm_count() / 2;
    const long long sk = split_k > 0 ? split_k : 1;
    const long long w256 = ((long long)p.num_m_blocks * ((N + 255) / 256) * sk + units - 1) / units * 256;
    const long long w384 = ((long long)p.num_m_blocks * ((N + 383) / 384) * sk + units - 1) / units * 384;
    bn = ((force_bn == 0 || tpx) && !(flags & EPI_ATOMIC) && w384 * 10 <= w256 * 8) ? 384 : 256;
    if (pair_bn == 256 || pair_bn == 384) bn = pair_bn;
  } else if (bn != 64 && bn != 128 && bn != 256) {
    const int t256 = p.num_m_blocks * ((N + 255) / 256);
    bn = (N > 128 && t256 * (split_k > 0 ? split_k : 1) >= sm_count()) ? 256 : 128;
    if (N > 128 && (flags & EPI_ATOMIC)) bn = 256;
  }
  // 128 x 64 tiles for outputs of up to 64 columns (the second half of a wider tile and its epilogue warps would be idle) and
  // where they fit the SMs once: twice the SMs, three quarters of the operand bytes per K block and CTA. The order of
  // accumulation is the same. Us with 128 and 64 columns: 69 x 768 x 768 7.5 and 7.1, 1218 x 256 x 256 5.3 and 4.7, 1372 x 256 x
  // 1024 9.1 and 8.4, 343 x 2048 x 512 6.8 and 6.3, 802816 x 64 x 256 92.4 and 77.7; past one wave 1218 x 1024 x 256 (160 tiles of
  // 64 columns) 5.6 and 6.5.
  if (force_bn == 0 && !pair && bn == 128 && !(flags & EPI_ATOMIC)) {
    const long long t64 = (long long)p.num_m_blocks * ((N + 63) / 64);
    const bool aligned = (reinterpret_cast<uintptr_t>(D) & 15) == 0 && (ldd * ((flags & EPI_OUT_F32) ? 4 : 2)) % 16 == 0;
    const bool in_ranges = automatic && aligned && !a_mn && pick_ranges((long long)p.num_m_blocks * ((N + 127) / 128), p.num_k_blocks) > 1;
    if (N <= 64 || (t64 <= sm_count() && !in_ranges)) bn = 64;
  }
  p.num_n_blocks = (N + bn - 1) / bn;
  const int tiles = p.num_m_blocks * p.num_n_blocks;
  if (split_k <= 0) {
    split_k = 1;
    if (flags & EPI_ATOMIC) split_k = pick_split_k(tiles, p.num_k_blocks, pair ? sm_count() / 2 : sm_count());
  }
  if (split_k > 1 && !(flags & EPI_ATOMIC)) return -6;
  split_k = min(split_k, p.num_k_blocks);
  p.kb_per_split = (p.num_k_blocks + split_k - 1) / split_k;
  p.split_k = (p.num_k_blocks + p.kb_per_split - 1) / p.kb_per_split;
  p.D = D; p.ldd = ldd;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.aux_in = static_cast<const __nv_bfloat16*>(aux_in);
  p.aux_out = static_cast<__nv_bfloat16*>(aux_out);
  p.ld_aux = ld_aux;
  p.resid = static_cast<const __nv_bfloat16*>(resid);
  p.ld_res = ld_res;
  p.norm = norm ? *norm : ColNorm{};
  p.flags = flags;
  p.status = status;
  p.batch = 1;
  p.a_heads = p.b_heads = p.d_heads = 1;
  p.a_off = p.b_off = p.d_off = 0;
  p.d_stride_h = p.d_stride_b = 0;

  CUtensorMap ta, tb;
  int rc;
  if (!a_mn) {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)M};
    uint64_t str[1] = {(uint64_t)lda * 2};
    uint32_t box[2] = {64, 128};
    rc = encode_tmap_bf16(&ta, A, 2, dims, str, box, nullptr);
  } else {
    uint64_t dims[2] = {(uint64_t)M, (uint64_t)K};
    uint64_t str[1] = {(uint64_t)lda * 2};
    uint32_t box[2] = {64, 64};
    rc = encode_tmap_bf16(&ta, A, 2, dims, str, box, nullptr);
  }
  if (rc) return rc;
  if (!b_mn) {
    uint64_t dims[2] = {(uint64_t)K, (uint64_t)N};
    uint64_t str[1] = {(uint64_t)ldb * 2};
    uint32_t box[2] = {64, pair ? (uint32_t)bn / 2 : (uint32_t)bn};
    rc = encode_tmap_bf16(&tb, B, 2, dims, str, box, nullptr);
  } else {
    uint64_t dims[2] = {(uint64_t)N, (uint64_t)K};
    uint64_t str[1] = {(uint64_t)ldb * 2};
    uint32_t box[2] = {64, 64};
    rc = encode_tmap_bf16(&tb, B, 2, dims, str, box, nullptr);
  }
  if (rc) return rc;

  CUtensorMap tx{};
  p.lines = !tpx && epi_lines(p, tx);
  if ((flags & EPI_NORM) && !p.lines) return -4;
  p.epi_tiles = p.lines && (flags & (EPI_DGELU | EPI_RESID)) ? max(bn / (EPI_WARPS / 4) / 64, 1) : 1;
  p.stages = pair ? (bn == 384 ? Gemm2Cfg<384, 0>::STAGES : Gemm2Cfg<256, 0>::STAGES)
                  : bn == 256 ? GemmCfg<256>::STAGES : bn == 128 ? GemmCfg<128>::STAGES : GemmCfg<64>::STAGES;
  if (p.epi_tiles > 1) --p.stages;
  if (automatic && !pair && bn == 128 && p.lines && !a_mn && !(flags & EPI_ATOMIC)) ranges = pick_ranges(tiles, p.num_k_blocks);
  const int kind = epi_kind(p);
  if (ranges > 1) {
    if (!p.lines) return -4;
    p.split_k = ranges;
    p.kb_per_split = (p.num_k_blocks + ranges - 1) / ranges;
    if (kind == KIND_PLAIN && b_mn) return launch_gemm_ranges<1, KIND_PLAIN>(ta, tb, p, tx, tiles, stream);
    if (kind == KIND_PLAIN) return launch_gemm_ranges<0, KIND_PLAIN>(ta, tb, p, tx, tiles, stream);
    if (kind == KIND_GELU && !b_mn) return launch_gemm_ranges<0, KIND_GELU>(ta, tb, p, tx, tiles, stream);
    if (kind == KIND_TAIL && !b_mn) return launch_gemm_ranges<0, KIND_TAIL>(ta, tb, p, tx, tiles, stream);
    if (kind == KIND_DGELU && b_mn) return launch_gemm_ranges<1, KIND_DGELU>(ta, tb, p, tx, tiles, stream);
    if (b_mn) return launch_gemm_ranges<1, KIND_ANY>(ta, tb, p, tx, tiles, stream);
    return launch_gemm_ranges<0, KIND_ANY>(ta, tb, p, tx, tiles, stream);
  }

  if (pair && tpx) {
    // tensor-parallel variants: A is always K-major, no split-K
    if (a_mn || p.split_k != 1) return -6;
    const int grid2 = 2 * min(tiles, sm_count() / 2);
#define TNNB_TP(BN_, BM_, CM) return launch_gemm_pair<BN_, 0, BM_, KIND_ANY, CM>(ta, tb, p, tx, grid2, stream, *tpx)
    if (tpx->mode == 1) {
      if (bn == 256) { if (b_mn) TNNB_TP(256, 1, 1); TNNB_TP(256, 0, 1); }
      if (b_mn) TNNB_TP(384, 1, 1); TNNB_TP(384, 0, 1);
    } else {
      if (bn == 256) { if (b_mn) TNNB_TP(256, 1, 2); TNNB_TP(256, 0, 2); }
      if (b_mn) TNNB_TP(384, 1, 2); TNNB_TP(384, 0, 2);
    }
#undef TNNB_TP
  }
  if (pair) {
    const int grid2 = 2 * min(tiles * p.split_k, sm_count() / 2);
    if (bn == 256) return launch_pair_kind<256>(kind, a_mn, b_mn, ta, tb, p, tx, grid2, stream);
    return launch_pair_kind<384>(kind, a_mn, b_mn, ta, tb, p, tx, grid2, stream);
  }
  const int grid = min(tiles * p.split_k, sm_count());
  if (bn == 256) return launch_single_kind<256>(kind, a_mn, b_mn, ta, tb, p, tx, grid, stream);
  if (bn == 128) return launch_single_kind<128>(kind, a_mn, b_mn, ta, tb, p, tx, grid, stream);
  return launch_single_kind<64>(kind, a_mn, b_mn, ta, tb, p, tx, grid, stream);
}

extern "C" int tnnb_gemm_bf16(const void* A, const void* B, void* D, int M, int N, int K, int a_mn,
                              int b_mn, long long lda, long long ldb, long long ldd,
                              const void* bias, const void* aux_in, void* aux_out,
                              long long ld_aux, const void* resid, long long ld_res, int flags,
                              int split_k, int force_bn, int* status, void* stream_) {
  return gemm_dispatch(A, B, D, M, N, K, a_mn, b_mn, lda, ldb, ldd, bias, aux_in, aux_out, ld_aux, resid, ld_res, flags,
                       split_k, force_bn, status, stream_, nullptr);
}

// D = relu?(norm(A * B^T [+ bias]) [+ resid]) with a per-column norm from running statistics (inference of a 1 x 1 or patch-matrix
// convolution and the batch norm behind it in one pass): (v - mean) / sqrt(var + eps) * gamma + beta, gamma and beta may be
// null. flags: EPI_BIAS, EPI_RESID, EPI_RELU (before the residual is added) or EPI_RELU_LAST (after). split_k: 1 for one range of K, 0
// for what is fastest.
extern "C" int tnnb_gemm_bf16_norm(const void* A, const void* B, void* D, int M, int N, int K, long long lda, long long ldb, long long ldd,
                                   const void* bias, const void* gamma, const void* beta, const void* mean, const void* var, float eps,
                                   const void* resid, long long ld_res, int flags, int split_k, int* status, void* stream_) {
  if (flags & ~(EPI_BIAS | EPI_RESID | EPI_RELU | EPI_RELU_LAST)) return -6;
  if (N % 8 || ldd % 8 || ((flags & EPI_RESID) && ld_res % 8)) return -3;  // what the norm's own kernels take
  if ((reinterpret_cast<uintptr_t>(D) & 15) || ((flags & EPI_RESID) && (reinterpret_cast<uintptr_t>(resid) & 15))) return -4;
  const ColNorm norm = {static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(beta), static_cast<const float*>(mean),
                        static_cast<const float*>(var), eps};
  return gemm_dispatch(A, B, D, M, N, K, 0, 0, lda, ldb, ldd, bias, nullptr, nullptr, 0, resid, ld_res, flags | EPI_NORM, split_k == 1, 0,
                       status, stream_, nullptr, &norm);
}

// `batch` independent products D[i] = op(A[i]) * op(B[i])^T on the single-CTA kernel. Item i of an operand lies at its base
// + ((i + off) / heads) * stride_b + ((i + off) % heads) * stride_h elements (operands: multiples of 8; D: of its own
// type); an operand holds `heads` x `seqs` items. flags: 0 (bf16 output) or EPI_OUT_F32. Used for attention with head
// sizes other than 64: scores and probabilities of all heads in one launch each, q, k, v and the results in place.
// layout: {heads, seqs, off} of A, B and D in turn; strides: {stride_h, stride_b} likewise.
extern "C" int tnnb_gemm_bf16_heads(const void* A, const void* B, void* D, int M, int N, int K, int a_mn, int b_mn, long long lda,
                                    long long ldb, long long ldd, int batch, const int* layout, const long long* strides, int flags,
                                    int* status, void* stream_) {
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  if (M <= 0 || N <= 0 || K <= 0 || batch <= 0) return -2;
  if (!layout || !strides) return -5;
  for (int o = 0; o < 3; ++o) {
    const int heads = layout[3 * o], seqs = layout[3 * o + 1], off = layout[3 * o + 2];
    if (heads <= 0 || seqs <= 0 || off < 0 || (long long)off + batch > (long long)heads * seqs) return -2;
  }
  if ((lda % 8) || (ldb % 8) || (strides[0] % 8) || (strides[1] % 8) || (strides[2] % 8) || (strides[3] % 8)) return -3;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15)) return -4;
  if (flags & ~EPI_OUT_F32) return -6;
  // the epilogue stores vectors of complete groups of 32 columns where the row pitch allows it: then every item starts on a
  // vector as well
  const int unit = (flags & EPI_OUT_F32) ? 4 : 8;
  if (N >= 32 && ldd % unit == 0 && ((reinterpret_cast<uintptr_t>(D) & 15) || (strides[4] % unit) || (strides[5] % unit))) return -4;
  GemmParams p{};
  p.M = M; p.N = N; p.K = K;
  p.num_m_blocks = (M + 127) / 128;
  p.num_k_blocks = (K + 63) / 64;
  const int bn = (N > 128) ? 256 : 128;
  p.num_n_blocks = (N + bn - 1) / bn;
  p.split_k = 1;
  p.kb_per_split = p.num_k_blocks;
  p.D = D; p.ldd = ldd;
  p.flags = flags;
  p.status = status;
  p.batch = batch;
  p.a_heads = layout[0]; p.a_off = layout[2];
  p.b_heads = layout[3]; p.b_off = layout[5];
  p.d_heads = layout[6]; p.d_off = layout[8];
  p.d_stride_h = strides[4]; p.d_stride_b = strides[5];
  CUtensorMap ta, tb;
  int rc;
  {
    uint64_t dims[4] = {(uint64_t)(a_mn ? M : K), (uint64_t)(a_mn ? K : M), (uint64_t)layout[0], (uint64_t)layout[1]};
    uint64_t str[3] = {(uint64_t)lda * 2, (uint64_t)strides[0] * 2, (uint64_t)strides[1] * 2};
    uint32_t box[4] = {64, (uint32_t)(a_mn ? 64 : 128), 1, 1};
    if ((rc = encode_tmap_bf16(&ta, A, 4, dims, str, box, nullptr))) return rc;
  }
  {
    uint64_t dims[4] = {(uint64_t)(b_mn ? N : K), (uint64_t)(b_mn ? K : N), (uint64_t)layout[3], (uint64_t)layout[4]};
    uint64_t str[3] = {(uint64_t)ldb * 2, (uint64_t)strides[2] * 2, (uint64_t)strides[3] * 2};
    uint32_t box[4] = {64, (uint32_t)(b_mn ? 64 : bn), 1, 1};
    if ((rc = encode_tmap_bf16(&tb, B, 4, dims, str, box, nullptr))) return rc;
  }
  CUtensorMap tx{};
  p.lines = !(strides[4] % unit) && !(strides[5] % unit) && epi_lines(p, tx);
  p.epi_tiles = 1;
  p.stages = bn == 256 ? GemmCfg<256>::STAGES : GemmCfg<128>::STAGES;
  const int grid = min(p.num_m_blocks * p.num_n_blocks * batch, sm_count());
#define TNNB_B(BN_, AM, BM_)                                                                        \
  return p.lines ? launch_gemm<BN_, AM, BM_, KIND_PLAIN, true>(ta, tb, p, tx, grid, stream)        \
                 : launch_gemm<BN_, AM, BM_, KIND_ANY, true>(ta, tb, p, tx, grid, stream)
  if (bn == 256) {
    if (!a_mn && !b_mn) TNNB_B(256, 0, 0);
    if (!a_mn && b_mn) TNNB_B(256, 0, 1);
    if (a_mn && !b_mn) TNNB_B(256, 1, 0);
    TNNB_B(256, 1, 1);
  }
  if (!a_mn && !b_mn) TNNB_B(128, 0, 0);
  if (!a_mn && b_mn) TNNB_B(128, 0, 1);
  if (a_mn && !b_mn) TNNB_B(128, 1, 0);
  TNNB_B(128, 1, 1);
#undef TNNB_B
}

// Tensor-parallel GEMMs on the CTA-pair kernel (protocol: tp_flags.cuh). A is [M, K] K-major.
//   mode 1  Y[M, N] = A * op(B)^T where the rows of A owned by other ranks (row r belongs to rank
//           r / rows_per_rank) are pushed into A by their owners; a_ready = this rank's counters [M / 128].
//   mode 2  partial sums of the rows owned by rank o go to out[o] ([rows_per_rank, ldo], bf16): out[rank] is the
//           local output (bias applied), out[o != rank] this rank's slot in o's inbox; arrived[o] = rank o's
//           counters [rows_per_rank / 128]. D / ldd are ignored.
//           n_push > 0: the kernel also sends this rank's rows of A to n_push peers (push_dst[i] = base of peer i's
//           A buffer, push_ready[i] = peer i's counters), starting at its 128-row block push_first_block - the
//           blocks before it were delivered by the kernel that produced the rows; 0 when that kernel delivered all.
// pass = device word holding the number of passes including this one. out / arrived are arrays of tp pointers.
extern "C" int tnnb_gemm_tp(int mode, const void* A, const void* B, void* D, int M, int N, int K, int b_mn, long long lda,
                            long long ldb, long long ldd, const void* bias, const void* aux_in, void* aux_out, long long ld_aux,
                            int flags, int tp, int rank, int rows_per_rank, const void* pass, const void* a_ready, void** out,
                            long long ldo, void** arrived, int n_push, void** push_dst, void** push_ready, int push_first_block,
                            int force_bn, int* status, void* stream_) {
  if (mode != 1 && mode != 2) return -2;
  if (tp < 1 || tp > TP_MAX || rank < 0 || rank >= tp || !pass) return -2;
  if (rows_per_rank <= 0 || rows_per_rank % 128 || (long long)rows_per_rank * tp != M) return -8;
  if (flags & (EPI_ATOMIC | EPI_OUT_F32 | EPI_ACCUM | EPI_RESID)) return -6;
  TpExt x{};
  x.mode = mode; x.tp = tp; x.rank = rank; x.rows_per_rank = rows_per_rank;
  x.pair_blocks_per_rank = (rows_per_rank % 256 == 0) ? rows_per_rank / 256 : 0;
  x.pass = static_cast<const uint32_t*>(pass);
  x.status = status;
  if (mode == 1) {
    if (!a_ready || !D) return -5;
    x.a_ready = static_cast<const uint32_t*>(a_ready);
    if (n_push < 0 || n_push > TP_MAX - 1) return -2;
    if (n_push > 0) {
      if (!push_dst || !push_ready || (K % 8)) return -5;
      if ((long long)K * 2 > TP_COPY_STAGE) return -3;  // a row must fit one stage of the copy thread
      if (push_first_block < 0 || push_first_block > rows_per_rank / 128) return -3;
      x.push_n = n_push;
      x.push_first_block = push_first_block;
      x.push_src = static_cast<const __nv_bfloat16*>(A);
      x.push_ld = lda;
      for (int i = 0; i < n_push; ++i) {
        if (!push_dst[i] || !push_ready[i] || (reinterpret_cast<uintptr_t>(push_dst[i]) & 15)) return -4;
        x.push_dst[i] = static_cast<__nv_bfloat16*>(push_dst[i]);
        x.push_ready[i] = static_cast<uint32_t*>(push_ready[i]);
      }
    }
  } else {
    if (!out || !arrived || (ldo % 8)) return -5;
    for (int o = 0; o < tp; ++o) {
      if (!out[o] || (o != rank && !arrived[o])) return -5;
      x.out[o] = out[o];
      x.arrived[o] = static_cast<uint32_t*>(arrived[o]);
    }
    x.ldo = ldo;
    D = out[rank];
    ldd = ldo;
  }
  const int fb = (force_bn == 256 || force_bn == 384) ? force_bn + 1024 : 512;  // always the pair kernel
  return gemm_dispatch(A, B, D, M, N, K, 0, b_mn, lda, ldb, ldd, bias, aux_in, aux_out, ld_aux, nullptr, 0, flags, 1, fb,
                       status, stream_, &x);
}
