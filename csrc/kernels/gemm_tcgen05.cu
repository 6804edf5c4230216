// bf16 GEMM on the 5th-generation tensor cores (tcgen05.mma, accumulators in TMEM, operands staged in
// shared memory by TMA, 128-byte swizzle), persistent over output tiles, warp-specialised:
//   warp 0      : TMA producer (one elected lane)
//   warp 1      : TMEM allocator + MMA issuer (one elected lane)
//   warps 2..5  : epilogue (TMEM -> registers -> fused epilogue -> global)
// TMEM holds two accumulator buffers, so the epilogue of tile i overlaps the main loop of tile i+1.
//
// D[M,N] = epilogue( A[M,K] * B[N,K]^T ).  Each operand is either "K-major" (the contraction
// dimension is the contiguous one, i.e. A stored [M,K] / B stored [N,K]) or "MN-major" (stored
// transposed, [K,M] / [K,N]).  The three combinations a linear layer needs are
//   forward  y  = x W^T      : A K-major,  B K-major
//   dgrad    dx = dy W       : A K-major,  B MN-major
//   wgrad    dW = dy^T x     : A MN-major, B MN-major
// so neither activations nor weights are ever transposed in memory.
//
// Replaces the reference's scalar 16x16 tiled matmul (crates/wgpu-backend/src/shaders.wgsl:571),
// its CPU linear (crates/ndarray-backend/src/lib.rs:478) and the fused_linear_bias{,_relu,_gelu}
// op sequences (crates/candle-backend/src/lib.rs:220-312).
#include "gemm_tcgen05.h"

#include "elementwise.h"
#include "gemm_rows.h"

#include <stdlib.h>
#include <string.h>

#include "pairs.cuh"
#include "pdl.cuh"
#include "rb_common.cuh"

namespace rb {

constexpr int kBlockM = 128;
constexpr int kBlockK = 64;   // 64 bf16 = 128 bytes = one swizzle row
constexpr int kUmmaK = 16;
constexpr int kNumEpilogueWarps = 8;   // two groups of four: each group covers all 128 TMEM lanes and half of the columns
constexpr int kNumEpiThreads = kNumEpilogueWarps * 32;
constexpr int kNumThreads = 64 + kNumEpiThreads;

struct EpiParams {
  void* d;
  long long ldd;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  const __nv_bfloat16* aux_in;
  long long ld_aux_in;
  __nv_bfloat16* aux_out;
  long long ld_aux_out;
  int act;
  int out_f32;
  int accumulate;
  float alpha;
  int staged;   // 1: bf16 output goes through a per-warp shared-memory tile and leaves as whole 128/256-byte row segments;
                // 2: 64-column tiles that leave through TMA stores (tensor maps tmD / tmAux; 256- and 128-wide tiles only);
                // 3: fp32 output in 32-column tiles through TMA stores; 4: the same, added to d by TMA reductions
  int side;     // staged == 2: what TMA loads into the tiles before the accumulator is complete: 0 nothing, 1 residual, 2 aux_in
  const float* row_scale;   // fp32 [M] or nullptr: multiplies row i of the accumulator (8-bit operands: per-token scale)
  const float* col_scale;   // fp32 [N] or nullptr: multiplies column j (per-output-channel weight scale)
  float* col_sum;           // fp32 [slabs][M], column sums of A over every col_rows rows; kernels of the EXTRA form with MN-major A only
  int col_rows;
  const __nv_bfloat16* col_src;   // A once more, [K, M] with pitch col_ld: rows of a slab that another part of the contraction loads
  long long col_ld;
  int fp8_b_format;         // 8-bit operands: format of B in the instruction descriptor (0 = e4m3, 1 = e5m2); A is e4m3
};

// Grouped (mixture-of-experts) execution over a permuted token buffer whose expert segments are whole tiles.
//   mode 1: rows of A (and D) belong to experts; the expert of M-tile i is tile_expert[i], the number of M-tiles
//           is read from the device (*num_m_tiles).  B holds all experts stacked: expert e starts b_expert_rows
//           rows further (along N for a K-major B, along K for an MN-major B).
//   mode 2: one output matrix per expert (d + e * d_expert_stride); expert e contracts over the rows
//           [offsets[e], offsets[e+1]) of A and B (both MN-major).  An expert without tokens writes zeros.
struct GroupInfo {
  int mode;
  int num_experts;
  const int* tile_expert;
  const int* num_m_tiles;
  const int* offsets;
  int b_expert_rows;
  long long d_expert_stride;
  const unsigned int* tile_arrived;   // mode 1, optional: rows of A's 128-row tiles stored so far by the dispatching ranks
  const int* tile_expected;           //                    rows each tile has to receive before it may be read
};

// Fusion with tensor-parallel collectives over peer memory (NVLink loads / stores issued by this kernel).
//   mode 1 (all-gather -> GEMM): the A operand [M, K] is sharded by rows over `world` ranks.  This rank's rows are
//           already in a_full; the other ranks' 128-row tiles are copied from their (peer-mapped) shards into a_full by
//           the epilogue warps of all CTAs whenever they have no accumulator to drain, 4 rows at a time, each piece adding one to the tile's
//           counter; the TMA producer waits (bounded) until a remote tile's counter reaches epoch * 32 before loading
//           it.  Local tiles are scheduled first, so the transfer overlaps their math.
//   mode 3 (weight all-gather -> GEMM, the FSDP / ZeRO-3 case): the B operand [N, K] is sharded by rows over the
//           ranks; same pull-and-flag mechanism as mode 1 on 128-row blocks of B, with the tiles visited N-major
//           starting at this rank's own block of output columns.
//   mode 2 (GEMM -> reduce-scatter): the output rows are owned by ranks (rows_per_rank each).  The epilogue stores
//           every tile straight into the OWNER's receive slot for this rank (d_peer[owner] + rank slot), as whole
//           row segments through the staged store; tiles of the next rank come first and this rank's own last, so
//           at any time the ranks send to different peers.  A small kernel on the owner then folds the slots in
//           rank order.
struct PeerInfo {
  int mode, world, rank, rows_per_rank;
  const __nv_bfloat16* a_peer[8];
  __nv_bfloat16* a_full;
  unsigned int* ready;
  unsigned int epoch;
  __nv_bfloat16* d_peer[8];
};

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_gpu(unsigned int* p, unsigned int v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void red_release_gpu_add(unsigned int* p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ unsigned int ld_acquire_sys_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
constexpr int kCopyParts = 32;    // a remote 128-row block is pulled as 32 pieces of 4 rows, by different warps of different CTAs
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

template <int BLOCK_N, int STAGES>
struct SmemLayout {
  static constexpr int kABytes = kBlockM * kBlockK * 2;
  static constexpr int kBBytes = BLOCK_N * kBlockK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kBarOffset = STAGES * kStageBytes;
  // full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], side[warps][2], tmem ptr, abort flag; behind them read[STAGES], summed[STAGES]
  static constexpr int kSumBars = kBarOffset + (2 * STAGES + 4 + 2 * kNumEpilogueWarps) * 8 + 16;
  static constexpr int kTotal = kSumBars + 2 * STAGES * 8;
  // optional output staging (EpiParams::staged): per epilogue warp kSlots tiles of 32 rows x kStageCols bf16 (4 KB: or 32 x 32 fp32)
  static constexpr int kStageCols = (BLOCK_N % 128 == 0) ? 64 : 32;
  static constexpr int kSlots = BLOCK_N == 128 ? 2 : 1;
  static constexpr bool kTma = BLOCK_N % 128 == 0;                 // tiles of 128-byte rows: TMA can move them
  static constexpr bool kSide = kSlots * 64 >= BLOCK_N / 2;        // a tile for each of a warp's column blocks
  static constexpr int kStagingOffset = (kTotal + 1023) & ~1023;   // 1024-byte aligned: the tiles are also TMA-store sources (128B swizzle)
  static constexpr int kStagingBytesPerWarp = kSlots * 32 * kStageCols * 2;
  static constexpr int kTotalStaged = kStagingOffset + kNumEpilogueWarps * kStagingBytesPerWarp;
};

// Epilogue arithmetic on 32 consecutive accumulator columns of one output row (everything but the final store).
// STORE_AUX: write the pre-activation to aux_out from here (one 64-byte piece per thread).  PRE_ONLY: stop after
// the bias, leaving the pre-activation in v (the staged path writes it out itself, coalesced).
template <bool STORE_AUX = true, bool PRE_ONLY = false>
__device__ __forceinline__ void epilogue_math(const EpiParams& ep, uint32_t (&r)[32], long long row, int col0, int N,
                                              float (&v)[32]) {
  const bool full = (col0 + 32 <= N);
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * ep.alpha;

  if (ep.row_scale != nullptr) {
    const float rs = __ldg(ep.row_scale + row);
#pragma unroll
    for (int j = 0; j < 32; ++j) v[j] *= rs;
  }
  if (ep.col_scale != nullptr) {
    if (full) {
      const float4* cp = reinterpret_cast<const float4*>(ep.col_scale + col0);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float4 c = __ldg(cp + q);
        v[q * 4 + 0] *= c.x; v[q * 4 + 1] *= c.y; v[q * 4 + 2] *= c.z; v[q * 4 + 3] *= c.w;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j < N) v[j] *= __ldg(ep.col_scale + col0 + j);
    }
  }

  if (ep.bias != nullptr) {
    if (full) {
      const uint4* bp = reinterpret_cast<const uint4*>(ep.bias + col0);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 b = __ldg(bp + q);
        float2 f0 = unpack_bf16x2(b.x), f1 = unpack_bf16x2(b.y), f2 = unpack_bf16x2(b.z), f3 = unpack_bf16x2(b.w);
        v[q * 8 + 0] += f0.x; v[q * 8 + 1] += f0.y; v[q * 8 + 2] += f1.x; v[q * 8 + 3] += f1.y;
        v[q * 8 + 4] += f2.x; v[q * 8 + 5] += f2.y; v[q * 8 + 6] += f3.x; v[q * 8 + 7] += f3.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j < N) v[j] += __bfloat162float(ep.bias[col0 + j]);
    }
  }

  if (PRE_ONLY) return;

  if (ep.act == RB_ACT_GELU || ep.act == RB_ACT_RELU || ep.act == RB_ACT_SILU || ep.act == RB_ACT_RELU2) {
    if (ep.aux_out != nullptr) {   // keep the pre-activation for the backward pass
      __nv_bfloat16* ap = ep.aux_out + row * ep.ld_aux_out + col0;
      if (!STORE_AUX) {
      } else if (full) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint4 o;
          o.x = pack_bf16x2(v[q * 8 + 0], v[q * 8 + 1]); o.y = pack_bf16x2(v[q * 8 + 2], v[q * 8 + 3]);
          o.z = pack_bf16x2(v[q * 8 + 4], v[q * 8 + 5]); o.w = pack_bf16x2(v[q * 8 + 6], v[q * 8 + 7]);
          reinterpret_cast<uint4*>(ap)[q] = o;
        }
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (col0 + j < N) ap[j] = __float2bfloat16(v[j]);
      }
      // Here the activation is applied to the unrounded fp32 value, while the backward pass differentiates at the bf16-rounded one that it
      // reads back (a relative difference of 2^-9 in the argument).  Results that leave through TMA (`epilogue_tma`) are formed from the
      // rounded value, which their tile holds.
    }
    if (ep.act == RB_ACT_GELU) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = gelu_tanh_fast(v[j]);
    } else if (ep.act == RB_ACT_RELU) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.f);
    } else if (ep.act == RB_ACT_RELU2) {
#pragma unroll
      for (int j = 0; j < 32; ++j) { const float r = fmaxf(v[j], 0.f); v[j] = r * r; }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = silu(v[j]);
    }
  } else if (ep.act == RB_ACT_DGELU || ep.act == RB_ACT_DRELU || ep.act == RB_ACT_DSILU || ep.act == RB_ACT_MUL) {
    // multiply by act'(aux_in) (or by aux_in itself for RB_ACT_MUL)
    const __nv_bfloat16* ap = ep.aux_in + row * ep.ld_aux_in + col0;
    float a[32];
    if (full) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 b = __ldg(reinterpret_cast<const uint4*>(ap) + q);
        float2 f0 = unpack_bf16x2(b.x), f1 = unpack_bf16x2(b.y), f2 = unpack_bf16x2(b.z), f3 = unpack_bf16x2(b.w);
        a[q * 8 + 0] = f0.x; a[q * 8 + 1] = f0.y; a[q * 8 + 2] = f1.x; a[q * 8 + 3] = f1.y;
        a[q * 8 + 4] = f2.x; a[q * 8 + 5] = f2.y; a[q * 8 + 6] = f3.x; a[q * 8 + 7] = f3.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) a[j] = (col0 + j < N) ? __bfloat162float(ap[j]) : 0.f;
    }
    if (ep.act == RB_ACT_DGELU) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] *= gelu_tanh_grad_fast(a[j]);
    } else if (ep.act == RB_ACT_DRELU) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = a[j] > 0.f ? v[j] : 0.f;
    } else if (ep.act == RB_ACT_DSILU) {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] *= silu_grad(a[j]);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] *= a[j];
    }
  }

  if (ep.residual != nullptr) {
    const __nv_bfloat16* rp = ep.residual + row * ep.ldr + col0;
    if (full) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint4 b = __ldg(reinterpret_cast<const uint4*>(rp) + q);
        float2 f0 = unpack_bf16x2(b.x), f1 = unpack_bf16x2(b.y), f2 = unpack_bf16x2(b.z), f3 = unpack_bf16x2(b.w);
        v[q * 8 + 0] += f0.x; v[q * 8 + 1] += f0.y; v[q * 8 + 2] += f1.x; v[q * 8 + 3] += f1.y;
        v[q * 8 + 4] += f2.x; v[q * 8 + 5] += f2.y; v[q * 8 + 6] += f3.x; v[q * 8 + 7] += f3.y;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j < N) v[j] += __bfloat162float(rp[j]);
    }
  }

}

// Stores 32 consecutive columns of one output row from registers.
__device__ __forceinline__ void epilogue_store(const EpiParams& ep, float (&v)[32], long long row, int col0, int N) {
  const bool full = (col0 + 32 <= N);
  if (ep.out_f32) {
    float* dp = reinterpret_cast<float*>(ep.d) + row * ep.ldd + col0;
    if (full) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        float4 o = make_float4(v[q * 4 + 0], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
        if (ep.accumulate) {
          float4 old = reinterpret_cast<float4*>(dp)[q];
          o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
        }
        reinterpret_cast<float4*>(dp)[q] = o;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j < N) dp[j] = ep.accumulate ? dp[j] + v[j] : v[j];
    }
  } else {
    __nv_bfloat16* dp = reinterpret_cast<__nv_bfloat16*>(ep.d) + row * ep.ldd + col0;
    if (full) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (ep.accumulate) {
          uint4 b = reinterpret_cast<uint4*>(dp)[q];
          float2 f0 = unpack_bf16x2(b.x), f1 = unpack_bf16x2(b.y), f2 = unpack_bf16x2(b.z), f3 = unpack_bf16x2(b.w);
          v[q * 8 + 0] += f0.x; v[q * 8 + 1] += f0.y; v[q * 8 + 2] += f1.x; v[q * 8 + 3] += f1.y;
          v[q * 8 + 4] += f2.x; v[q * 8 + 5] += f2.y; v[q * 8 + 6] += f3.x; v[q * 8 + 7] += f3.y;
        }
        uint4 o;
        o.x = pack_bf16x2(v[q * 8 + 0], v[q * 8 + 1]); o.y = pack_bf16x2(v[q * 8 + 2], v[q * 8 + 3]);
        o.z = pack_bf16x2(v[q * 8 + 4], v[q * 8 + 5]); o.w = pack_bf16x2(v[q * 8 + 6], v[q * 8 + 7]);
        reinterpret_cast<uint4*>(dp)[q] = o;
      }
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (col0 + j < N) {
          float o = v[j];
          if (ep.accumulate) o += __bfloat162float(dp[j]);
          dp[j] = __float2bfloat16(o);
        }
    }
  }
}

__device__ __forceinline__ void epilogue_chunk(const EpiParams& ep, uint32_t (&r)[32], long long row, int col0, int N) {
  float v[32];
  epilogue_math(ep, r, row, col0, N, v);
  epilogue_store(ep, v, row, col0, N);
}

__device__ __forceinline__ uint32_t stage_addr(uint32_t slot, int lane, int chunk) {
  return slot + lane * 128 + ((chunk ^ (lane & 7)) << 4);
}
__device__ __forceinline__ void stage_put(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Epilogue of one warp through tiles of 32 rows x 128 bytes in shared memory that TMA moves: bf16 in 64-column blocks (staged 2), fp32 in
// 32-column blocks (3; 4 adds to d: every element is added to by one warp once, so the sum does not depend on any order).  With two tiles
// per warp (SLOTS) one is filled while the other is stored: blocks take them in turn, on into the next output tile (`t` counts those).
// With `side`, TMA has loaded the residual or aux_in into the tiles (`epilogue_side_load`,
// issued before the accumulator is waited for); results replace it in place.  Reading those through the SM's own loads instead, each
// lane 64 bytes of its row, cost more than the products at K = 768: 32768 x 3072 with gelu'(aux_in) 292 us, residual 32768 x 768 61 us.
// `arrive` hands the accumulator back; `row0` is the warp's first row, `col` the first of its COLS columns.
template <int COLS>
__device__ __forceinline__ void epilogue_side_load(const EpiParams& ep, const CUtensorMap* tmSide, uint32_t stg, uint32_t bar_side, int row0,
                                                   int col, int lane) {
  if (lane == 0) {
    tma_store_wait_read<0>();                              // the tiles' last contents have been read out
#pragma unroll
    for (int h = 0; h < COLS / 64; ++h) {
      mbar_arrive_expect_tx(bar_side + 8 * h, 4096);
      tma_load_2d(stg + h * 4096, tmSide, col + h * 64, row0, bar_side + 8 * h);
    }
  }
  __syncwarp();
}

// Pairs of neighbouring columns (pairs.cuh).
__device__ __forceinline__ Pair gelu2(Pair x) {
  constexpr float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const float2 u = floats(mul2(x, fma2(pair_of(k0 * k1, k0 * k1), mul2(x, x), pair_of(k0, k0))));
  const Pair h = mul2(x, pair_of(0.5f, 0.5f));
  return fma2(h, pair_of(tanh_fast(u.x), tanh_fast(u.y)), h);
}
__device__ __forceinline__ Pair gelu_grad2(Pair x) {
  constexpr float k0 = 0.7978845608028654f, k1 = 0.044715f;
  const Pair x2 = mul2(x, x), half = pair_of(0.5f, 0.5f);
  const float2 u = floats(mul2(x, fma2(pair_of(k0 * k1, k0 * k1), x2, pair_of(k0, k0))));
  const Pair t = pair_of(tanh_fast(u.x), tanh_fast(u.y));
  const Pair du = fma2(pair_of(3.f * k0 * k1, 3.f * k0 * k1), x2, pair_of(k0, k0));
  const Pair one_t2 = fma2(mul2(t, pair_of(-1.f, -1.f)), t, pair_of(1.f, 1.f));
  return fma2(mul2(mul2(x, half), one_t2), du, fma2(half, t, half));
}

// Accumulator -> pre-activation of 32 columns (scales, bias).  N is a multiple of 4.
__device__ __forceinline__ void tile_pre(const EpiParams& ep, const uint32_t (&r)[32], long long row, int col0, int N, Pair (&v)[16]) {
  const Pair alpha = pair_of(ep.alpha, ep.alpha);
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = mul2(pair_of(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])), alpha);
  if (ep.row_scale != nullptr) {
    const float rs = __ldg(ep.row_scale + row);
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = mul2(v[j], pair_of(rs, rs));
  }
  if (ep.col_scale != nullptr) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (col0 + 4 * q >= N) break;
      const float4 c = __ldg(reinterpret_cast<const float4*>(ep.col_scale + col0) + q);
      v[2 * q] = mul2(v[2 * q], pair_of(c.x, c.y));
      v[2 * q + 1] = mul2(v[2 * q + 1], pair_of(c.z, c.w));
    }
  }
  if (ep.bias != nullptr) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      if (col0 + 4 * q >= N) break;
      const uint2 b = __ldg(reinterpret_cast<const uint2*>(ep.bias + col0) + q);
      v[2 * q] = add2(v[2 * q], pair_of(b.x));
      v[2 * q + 1] = add2(v[2 * q + 1], pair_of(b.y));
    }
  }
}
__device__ __forceinline__ void tile_act(const EpiParams& ep, const uint32_t (&side)[16], Pair (&v)[16]) {
  if (ep.act == RB_ACT_GELU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = gelu2(v[j]);
  } else if (ep.act == RB_ACT_DGELU) {
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = mul2(v[j], gelu_grad2(pair_of(side[j])));
  } else if (ep.act != RB_ACT_NONE) {
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float2 f = floats(v[j]);
      const float2 a = unpack_bf16x2(side[j]);
      if (ep.act == RB_ACT_SILU) { f.x = silu(f.x); f.y = silu(f.y); }
      else if (ep.act == RB_ACT_MUL) { f.x *= a.x; f.y *= a.y; }
      else if (ep.act == RB_ACT_DSILU) { f.x *= silu_grad(a.x); f.y *= silu_grad(a.y); }
      else if (ep.act == RB_ACT_DRELU) { f.x = a.x > 0.f ? f.x : 0.f; f.y = a.y > 0.f ? f.y : 0.f; }
      else {
        f.x = fmaxf(f.x, 0.f); f.y = fmaxf(f.y, 0.f);
        if (ep.act == RB_ACT_RELU2) { f.x *= f.x; f.y *= f.y; }
      }
      v[j] = pair_of(f.x, f.y);
    }
  }
}

// 32 columns of a side input as packed pairs, by the SM's own loads; N is a multiple of 8.
__device__ __forceinline__ void side_get(const __nv_bfloat16* src, int col0, int N, uint32_t (&side)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint4 u = make_uint4(0u, 0u, 0u, 0u);
    if (col0 + 8 * q < N) u = *reinterpret_cast<const uint4*>(src + col0 + 8 * q);
    side[4 * q] = u.x; side[4 * q + 1] = u.y; side[4 * q + 2] = u.z; side[4 * q + 3] = u.w;
  }
}
__device__ __forceinline__ void tile_get(uint32_t slot, int lane, int half, uint32_t (&v)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v[4 * q]), "=r"(v[4 * q + 1]), "=r"(v[4 * q + 2]), "=r"(v[4 * q + 3])
                 : "r"(stage_addr(slot, lane, half * 4 + q)));
}
__device__ __forceinline__ void tile_put(uint32_t slot, int lane, int half, const Pair (&v)[16]) {
#pragma unroll
  for (int q = 0; q < 4; ++q)
    stage_put(stage_addr(slot, lane, half * 4 + q), packed(v[4 * q]), packed(v[4 * q + 1]), packed(v[4 * q + 2]), packed(v[4 * q + 3]));
}
__device__ __forceinline__ void tile_add(const uint32_t (&r)[16], Pair (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = add2(v[j], pair_of(r[j]));
}

// EXTRA: the forms that the tiles do not suffice for: side inputs beside a second result, two side inputs, and any of them with one tile per
// warp.  What finds no tile is read by the SM's own loads.  Kernels of their own: as branches of the common ones, not taken, these cost 10 % of a
// short contraction and 2.5 of 20 us of a small one.
template <int COLS, int SLOTS, bool EXTRA, class Arrive>
__device__ __forceinline__ void epilogue_tma(const EpiParams& ep, const CUtensorMap* tmD, const CUtensorMap* tmAux, uint32_t stg,
                                             uint32_t bar_side, uint32_t t, uint32_t taddr, int row0, int drow, int col, int M, int N,
                                             int lane, bool empty_k, volatile int* abort_flag, unsigned int* status, Arrive arrive) {
  // rows behind the matrix are computed like the others (on what the accumulator holds for them) and clipped by the stores
  const long long row = min(row0 + lane, M - 1);
  const bool two = ep.aux_out != nullptr && (ep.act == RB_ACT_GELU || ep.act == RB_ACT_RELU || ep.act == RB_ACT_SILU);
  const int cols = ep.staged >= 3 ? 32 : 64;                 // columns of a tile
#pragma unroll 1
  for (int c = 0; c < COLS; c += 32) {
    // 32 columns at a time; `half`: which part of a 64-column tile they are
    const int block = c / cols, half = (c & (cols - 1)) >> 5;
    // The wait below leaves the newest store in flight, so no two blocks in a row may share a tile; a side tile lies where it was loaded to.
    const uint32_t slot = stg + (two ? 0 : (block + (ep.side != 0 ? 0 : t * (COLS / cols))) % SLOTS) * 4096;
    uint32_t r[32];
    tmem_ld_32x32(taddr + c, r);
    uint32_t side[16], residual[16];
    if (EXTRA) {                               // requested before the accumulator is waited for
      if (ep.residual != nullptr && ep.side != 1) side_get(ep.residual + row * ep.ldr, col + c, N, residual);
      if (ep.aux_in != nullptr && ep.side != 2) side_get(ep.aux_in + row * ep.ld_aux_in, col + c, N, side);
    }
    if (ep.side != 0) {
      if (half == 0 && !mbar_wait(bar_side + 8 * block, t & 1, abort_flag, status, 7)) return;
      tile_get(slot, lane, half, side);
    } else if (half == 0) {
      // with two results the first tile may be filled again while the second one, stored later, still leaves
      if (lane == 0) tma_store_wait_read<SLOTS - 1>();
      __syncwarp();
    }
    tmem_ld_wait();
    if (c == COLS - 32) arrive();
    if (empty_k) {
#pragma unroll
      for (int j = 0; j < 32; ++j) r[j] = 0u;
    }
    Pair v[16];
    tile_pre(ep, r, row, col + c, N, v);
    if (ep.staged >= 3) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float2 a = floats(v[2 * q]), b = floats(v[2 * q + 1]);
        stage_put(stage_addr(slot, lane, q), __float_as_uint(a.x), __float_as_uint(a.y), __float_as_uint(b.x), __float_as_uint(b.y));
      }
    } else {
      if (!two) {
        tile_act(ep, side, v);
        if (ep.side == 1) tile_add(side, v);
        else if (EXTRA && ep.residual != nullptr) tile_add(residual, v);
      }
      uint32_t o[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) o[j] = packed(v[j]);
#pragma unroll
      for (int q = 0; q < 4; ++q) stage_put(stage_addr(slot, lane, half * 4 + q), o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
      if (two && SLOTS > 1) {
        // the result is formed from the rounded pre-activation, in the second tile
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = pair_of(o[j]);
        tile_act(ep, side, v);
        if (EXTRA && ep.residual != nullptr) tile_add(residual, v);
        if (half == 0) {
          if (lane == 0) tma_store_wait_read<0>();
          __syncwarp();
        }
        tile_put(slot + 4096, lane, half, v);
      }
      if (half == 0) continue;
    }
    fence_proxy_async_smem();
    __syncwarp();
    if (lane == 0) {
      const int x = col + c - half * 32;
      if (row0 >= M) {}                        // nothing of the matrix; with stacked results these are another one's rows
      else if (ep.staged == 4) tma_reduce_add_2d(tmD, slot, x, drow);
      else tma_store_2d(two ? tmAux : tmD, slot, x, drow);
      tma_store_commit();
      if (two && SLOTS > 1) {
        if (row0 < M) tma_store_2d(tmD, slot + 4096, x, drow);
        tma_store_commit();
      }
    }
    if (EXTRA && SLOTS == 1 && two) {
      // one tile: the result takes the place of the rounded pre-activation when that has been read out, each lane from its own row
      if (lane == 0) tma_store_wait_read<0>();
      __syncwarp();
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        uint32_t o[16];
        tile_get(slot, lane, h, o);
        Pair v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = pair_of(o[j]);
        tile_act(ep, o, v);
        if (ep.residual != nullptr) {
          side_get(ep.residual + row * ep.ldr, col + c - 32 + 32 * h, N, o);
          tile_add(o, v);
        }
        tile_put(slot, lane, h, v);
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        if (row0 < M) tma_store_2d(tmD, slot, col + c - 32, drow);
        tma_store_commit();
      }
    }
  }
}

// Epilogue of one warp of the pair kernel for RB_ACT_SWIGLU: 64 columns of the result from 64 gate columns and the up columns 128 behind
// them.  A kernel of its own read and wrote 1.5 times the products' result again: 149 us of 1600 at 8192 x 14336 x 4096.
template <class Arrive>
__device__ __forceinline__ void epilogue_swiglu(const CUtensorMap* tmD, uint32_t stg, uint32_t t, uint32_t taddr, int row0, int col, int M,
                                                int lane, Arrive arrive) {
  const uint32_t slot = stg + (t & 1) * 4096;
  if (lane == 0) tma_store_wait_read<1>();
  __syncwarp();
#pragma unroll 1
  for (int half = 0; half < 2; ++half) {
    uint32_t g[32], u[32];
    tmem_ld_32x32(taddr + half * 32, g);
    tmem_ld_32x32(taddr + 128 + half * 32, u);
    tmem_ld_wait();
    if (half == 1) arrive();
    uint32_t o[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      float v[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const float x = __uint_as_float(g[2 * j + e]);
        v[e] = __fdividef(x, 1.f + __expf(-x)) * __uint_as_float(u[2 * j + e]);
      }
      o[j] = pack_bf16x2(v[0], v[1]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) stage_put(stage_addr(slot, lane, half * 4 + q), o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
  }
  fence_proxy_async_smem();
  __syncwarp();
  if (lane == 0) {
    if (row0 < M) tma_store_2d(tmD, slot, col, row0);
    tma_store_commit();
  }
}

// Column sums of A beside the products (EpiParams::col_sum): four warps of their own read the A tiles of the first column of output tiles, 16 KB per
// k-block of 64, when the issuer has seen them land (it arrives at bar_read; for a pair of CTAs a commit does, behind the products: an arrival at the
// peer's barrier took the issuer so long that the product took three times as long) and before they are loaded over (bar_summed, for which the
// producer waits).  Warp w sums 32 columns: lane r + 8 c the rows r, r + 8, .. of 8 columns, a swizzle chunk, so that eight lanes read a row of banks.
// The sums are those of `rb_sum_dim0_staged`, bit for bit: its slabs of `col_rows` rows (whole k-blocks), its lanes (every eighth row, one after the other), its order of lanes;
// a slab leaves a row of partial sums, which `rb_sum_dim0_fold` adds up.  A slab belongs to the part of the contraction in which it begins; rows
// of it that the next part loads are read from memory.  (A running sum over a whole part, folded with the parts, needed no second launch, but was
// further from 64 bits from 6000 rows on: of the norm, 32768 rows around zero, 2.2e-7 against 1.3e-7.)  As kernels of its own the sum reads dy once more: 46
// us for 32768 x 3072.
constexpr int kSumWarps = 4;
template <int STAGES>
struct SumProducer {                               // what the TMA producer keeps
  uint32_t used = 0, phase = 0;                    // stages whose present contents are summed; parity of their next bar_summed phase
  __device__ __forceinline__ bool wait(uint32_t s, uint32_t bar_summed, volatile int* abort_flag, unsigned int* status) {
    if (used >> s & 1) {
      if (!mbar_wait(bar_summed + 8 * s, phase >> s & 1, abort_flag, status, 8)) return false;
      phase ^= 1u << s;
      used &= ~(1u << s);
    }
    return true;
  }
};
__device__ __forceinline__ void sum_add(const uint32_t (&u)[4], Pair (&acc)[4]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) acc[j] = add2(acc[j], pair_of(u[j]));
}
// Row `slab` of the partial sums; begins the next one.
__device__ __forceinline__ void sum_store(const EpiParams& ep, int slab, int row0, int M, int w, int lane, Pair (&acc)[4]) {
  float v[8];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float2 f = floats(acc[j]);
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
    acc[j] = pair_of(0.f, 0.f);
  }
  // eight lanes x eight columns, transposed: lane r then has column r of all of them, lane by lane
#pragma unroll
  for (int o = 1; o < 8; o <<= 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      if (i & o) continue;
      const float got = __shfl_xor_sync(0xffffffffu, lane & o ? v[i] : v[i | o], o);
      if (lane & o) v[i] = got;
      else v[i | o] = got;
    }
  }
  float t = 0.f;
#pragma unroll
  for (int y = 0; y < 8; ++y) t += v[y];
  const int m = row0 + 32 * w + lane;
  if (m < M) ep.col_sum[static_cast<long long>(slab) * M + m] = t;
}

// What a warp keeps of the slab that it is in.
struct SumSlab {
  int slab, lo;                                  // lo: its first row
  Pair acc[4];
  __device__ __forceinline__ SumSlab(int kb0, int rows) {
    slab = (kb0 * kBlockK + rows - 1) / rows;    // the first that begins in this part
    lo = slab * rows;
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = pair_of(0.f, 0.f);
  }
  __device__ __forceinline__ void done(const EpiParams& ep, int row0, int M, int w, int lane) {
    sum_store(ep, slab, row0, M, w, lane, acc);
    ++slab;
    lo += ep.col_rows;
  }
  // One k-block in shared memory; rows behind K are zero there (and a sum is never -0).
  __device__ __forceinline__ void block(const EpiParams& ep, uint32_t a_tile, int kb, int K, int row0, int M, int w, int lane) {
    if (lo > kb * kBlockK) return;               // a slab of the part in front
    const int chunk = 4 * w + (lane >> 3), r = lane & 7;
    const uint32_t at = a_tile + (chunk >> 3) * (kBlockK * 128) + r * 128 + (((chunk & 7) ^ r) << 4);
#pragma unroll
    for (int i = 0; i < kBlockK / 8; ++i) {
      uint32_t u[4];
      asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]) : "r"(at + i * 1024));
      sum_add(u, acc);
    }
    if ((kb + 1) * kBlockK >= min(lo + ep.col_rows, K)) done(ep, row0, M, w, lane);
  }
  // Behind the last block of a part: the rest of a slab that has begun in it.
  __device__ __forceinline__ void rest(const EpiParams& ep, int kb1, int K, int row0, int M, int w, int lane) {
    const int from = kb1 * kBlockK, hi = min(lo + ep.col_rows, K), m = row0 + (4 * w + (lane >> 3)) * 8;
    if (lo >= from || hi <= from) return;
    for (int at = from; at < hi; at += 64) {
      const int row = at + (lane & 7);
      uint4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i)
        v[i] = row + 8 * i < hi && m < M ? __ldg(reinterpret_cast<const uint4*>(ep.col_src + (row + 8 * i) * ep.col_ld + m)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t u[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
        sum_add(u, acc);
      }
    }
    done(ep, row0, M, w, lane);
  }
};

// FP8 = 1: both operands hold e4m3 bytes (K-major only).  A 128-byte swizzle row then carries 128 elements, so K, lda
// and ldb arrive halved (in units of two bytes) and only the TMA coordinates, which count elements, are doubled back.
template <int A_MN, int B_MN, int BLOCK_N, int STAGES, int FP8 = 0, bool EXTRA = false>
__global__ void __launch_bounds__(kNumThreads + (EXTRA && A_MN ? 32 * kSumWarps : 0), 1)
gemm_bf16_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                 const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmAux,
                 const __grid_constant__ CUtensorMap tmSide, int M, int N, int K, int group_m, int num_splits, int kb_per_split, long long d_split_stride, EpiParams ep,
                 GroupInfo grp, PeerInfo peer, unsigned int* status) {
  using L = SmemLayout<BLOCK_N, STAGES>;
  extern __shared__ uint8_t smem_raw[];
  // 128-byte swizzle atoms need 1024-byte aligned tiles
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_base = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = smem_u32(bars + STAGES);
  const uint32_t bar_tfull = smem_u32(bars + 2 * STAGES);
  const uint32_t bar_tempty = smem_u32(bars + 2 * STAGES + 2);
  const uint32_t bar_side = smem_u32(bars + 2 * STAGES + 4);
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4 + 2 * kNumEpilogueWarps);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  constexpr bool SUMS = EXTRA && A_MN;             // column sums of A beside the products
  const uint32_t bar_read = smem_u32(smem + L::kSumBars), bar_summed = bar_read + 8 * STAGES;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  // TMEM allocations are powers of two >= 32 columns
  constexpr uint32_t kTmemCols = (2 * BLOCK_N <= 32) ? 32 : (2 * BLOCK_N <= 64) ? 64 : (2 * BLOCK_N <= 128) ? 128
                                 : (2 * BLOCK_N <= 256) ? 256 : 512;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar_tfull + 8 * a, 1);
      mbar_init(bar_tempty + 8 * a, kNumEpilogueWarps);
    }
    for (int w = 0; w < 2 * kNumEpilogueWarps; ++w) mbar_init(bar_side + 8 * w, 1);
    if (SUMS) {
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(bar_read + 8 * s, 1);
        mbar_init(bar_summed + 8 * s, kSumWarps);
      }
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_ptr_smem), kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  // Barriers, TMEM and descriptors were set up under the kernel in front, and so is the first tile's place found where it hangs on nothing in
  // memory: its divisions, in code met for the first time, take a few hundred cycles.  Then every role waits by
  // itself.  One B200, whole passes before / now, us: training steps of 1024 tokens through 2 layers of 256 355 / 347, of 2 k tokens through 6 layers of
  // 384 1122 / 1099, prompts of 2.7 k rows 2721 / 2657.
  bool waited = peer.mode != 0 || grp.mode != 0;
  if (waited) pdl_wait();
  // A kernel that waits for other kernels' stores must not let its successor's blocks take the room that those kernels need.
  if (waited && peer.mode == 0 && grp.tile_arrived == nullptr) pdl_launch();

  int num_m = (M + kBlockM - 1) / kBlockM;
  if (grp.mode == 1) num_m = min(num_m, __ldg(grp.num_m_tiles));
  const int num_n = (N + BLOCK_N - 1) / BLOCK_N;
  const int num_tiles = num_m * num_n;
  const int num_kb_total = (K + kBlockK - 1) / kBlockK;
  const int group_size = group_m * num_n;
  // Work units: (split, tile).  With split-K every unit reduces its own K range into its own fp32 slab
  // d + split * d_split_stride; a second kernel folds the slabs in a fixed order.
  const int num_units = num_tiles * (grp.mode == 2 ? grp.num_experts : num_splits);

  // `outer` is the split index (split-K) or the expert index (grouped mode 2)
  auto decode_tile = [&](int unit, int& m_blk, int& n_blk, int& kb0, int& kb1, int& outer) {
    const int split = unit / num_tiles;
    const int tile = unit - split * num_tiles;
    outer = split;
    if (grp.mode == 2) {
      kb0 = __ldg(grp.offsets + split) / kBlockK;
      kb1 = __ldg(grp.offsets + split + 1) / kBlockK;
    } else {
      kb0 = split * kb_per_split;
      kb1 = min(num_kb_total, kb0 + kb_per_split);
    }
    const int group = tile / group_size;
    const int first_m = group * group_m;
    const int gm = min(group_m, num_m - first_m);
    const int in_group = tile - group * group_size;
    m_blk = first_m + in_group % gm;
    n_blk = in_group / gm;
    if (peer.mode == 1) {          // consumption order starts at this rank's own rows
      m_blk += peer.rank * (peer.rows_per_rank / kBlockM);
      if (m_blk >= num_m) m_blk -= num_m;
    } else if (peer.mode == 3) {   // N-major walk starting at this rank's own columns
      const int n_i = tile / num_m;
      m_blk = tile - n_i * num_m;
      n_blk = n_i + peer.rank * (peer.rows_per_rank / BLOCK_N);
      if (n_blk >= num_n) n_blk -= num_n;
    } else if (peer.mode == 2) {   // rows of the next rank first, this rank's own rows last
      m_blk += ((peer.rank + 1) % peer.world) * (peer.rows_per_rank / kBlockM);
      if (m_blk >= num_m) m_blk -= num_m;
    }
  };

  if (warp == 0) {
    // elect.sync, not lane 0: the compiler then knows that one lane runs this and keeps what it issues in uniform registers
    if (elect_one()) {
      // ------------------------------------------------------------------ TMA producer
      SumProducer<STAGES> sums;
      uint32_t it = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_units && ok; tile += gridDim.x) {
        int m_blk, n_blk, kb0, kb1, outer;
        decode_tile(tile, m_blk, n_blk, kb0, kb1, outer);
        if (!waited) {
          pdl_wait();
          pdl_launch();
          waited = true;
        }
        // grouped mode 1: this M-tile's expert selects the slice of B
        int b_row_off = 0;
        if (grp.mode == 1) {
          const int e = __ldg(grp.tile_expert + m_blk);
          b_row_off = (e < 0 ? 0 : e) * grp.b_expert_rows;
        }
        if (grp.mode == 1 && grp.tile_arrived != nullptr) {
          // expert-parallel dispatch still in flight: this 128-row tile of A is complete once every rank has stored the
          // rows it routes here (counted with system-scope release adds by the dispatch kernels)
          const unsigned int want = static_cast<unsigned int>(__ldg(grp.tile_expected + m_blk));
          const unsigned long long t0 = globaltimer_ns();
          while (ld_acquire_sys_u32(grp.tile_arrived + m_blk) < want) {
            if (*abort_flag || globaltimer_ns() - t0 > kFlagWaitLimitNs) {
              *abort_flag = 1;
              status_set(status, kStatusFlagTimeout, 6);
              ok = false;
              break;
            }
            __nanosleep(100);
          }
          if (!ok) break;
          fence_proxy_async_all();
        }
        if (peer.mode == 1 || peer.mode == 3) {
          // remote 128-row blocks this tile reads: wait until the copy warps have landed all their pieces
          const int blk0 = peer.mode == 1 ? m_blk : n_blk * (BLOCK_N / 128);
          const int nblk = peer.mode == 1 ? 1 : BLOCK_N / 128;
          const unsigned int target = peer.epoch * kCopyParts;
          for (int bi = blk0; bi < blk0 + nblk && ok; ++bi) {
            if ((bi * 128) / peer.rows_per_rank == peer.rank) continue;
            const unsigned long long t0 = globaltimer_ns();
            while (static_cast<int>(ld_acquire_gpu(peer.ready + bi) - target) < 0) {
              if (*abort_flag || globaltimer_ns() - t0 > kFlagWaitLimitNs) {
                *abort_flag = 1;
                status_set(status, kStatusFlagTimeout, 5);
                ok = false;
                break;
              }
              __nanosleep(100);
            }
          }
          if (!ok) break;
          fence_proxy_async_all();     // the rows were written with ordinary stores; TMA reads them through the async proxy
        }
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
          if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, status, 1)) { ok = false; break; }
          if (SUMS) {
            if (!sums.wait(s, bar_summed, abort_flag, status)) { ok = false; break; }
            if (n_blk == 0) sums.used |= 1u << s;
          }
          const uint32_t full = bar_full + 8 * s;
          mbar_arrive_expect_tx(full, L::kStageBytes);
          const uint32_t sa = smem_base + s * L::kStageBytes;
          const uint32_t sb = sa + L::kABytes;
          if (A_MN == 0) {
            tma_load_2d(sa, &tmA, kb * kBlockK * (FP8 ? 2 : 1), m_blk * kBlockM, full);
          } else {
#pragma unroll
            for (int j = 0; j < kBlockM / 64; ++j)
              tma_load_2d(sa + j * (kBlockK * 128), &tmA, m_blk * kBlockM + j * 64, kb * kBlockK, full);
          }
          if (B_MN == 0) {
            tma_load_2d(sb, &tmB, kb * kBlockK * (FP8 ? 2 : 1), b_row_off + n_blk * BLOCK_N, full);
          } else {
#pragma unroll
            for (int j = 0; j < BLOCK_N / 64; ++j)
              tma_load_2d(sb + j * (kBlockK * 128), &tmB, n_blk * BLOCK_N + j * 64, b_row_off + kb * kBlockK, full);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // ------------------------------------------------------------------ MMA issuer
      const uint32_t idesc = FP8 ? (umma_idesc_e4m3(kBlockM, BLOCK_N) | (static_cast<uint32_t>(ep.fp8_b_format) << 10))
                                 : umma_idesc_bf16(kBlockM, BLOCK_N, A_MN, B_MN);
      // K-major: 32 bytes per step of 16 inside the swizzle row, 8-row groups 1024 bytes apart.  MN-major: 16 k-rows of 128 bytes per
      // step, 64-wide MN atoms kBlockK * 128 bytes apart.  An offset of o bytes is o / 16 in the address field.
      const uint64_t desc_a = A_MN ? umma_smem_desc_sw128(smem_base, kBlockK * 128, 1024) : umma_smem_desc_sw128(smem_base, 16, 1024);
      const uint64_t desc_b = B_MN ? umma_smem_desc_sw128(smem_base + L::kABytes, kBlockK * 128, 1024) : umma_smem_desc_sw128(smem_base + L::kABytes, 16, 1024);
      constexpr int kStepA = A_MN ? kUmmaK * 8 : kUmmaK / 8, kStepB = B_MN ? kUmmaK * 8 : kUmmaK / 8;
      uint32_t it = 0, t = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_units && ok; tile += gridDim.x, ++t) {
        int m_blk, n_blk, kb0, kb1, outer;
        decode_tile(tile, m_blk, n_blk, kb0, kb1, outer);
        if (!waited) {
          pdl_wait();                // the limits of its waits count from here
          waited = true;
        }
        const uint32_t acc = t & 1, acc_ph = (t >> 1) & 1;
        if (!mbar_wait(bar_tempty + 8 * acc, acc_ph ^ 1, abort_flag, status, 2)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BLOCK_N;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
          if (!mbar_wait(bar_full + 8 * s, ph, abort_flag, status, 3)) { ok = false; break; }
          if (SUMS && n_blk == 0) mbar_arrive(bar_read + 8 * s);
          tc_fence_after();
          const uint64_t da = desc_a + s * (L::kStageBytes / 16), db = desc_b + s * (L::kStageBytes / 16);
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k) {
            if (FP8) umma_f8_ss(tmem_d, da + k * kStepA, db + k * kStepB, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
            else umma_bf16_ss(tmem_d, da + k * kStepA, db + k * kStepB, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
          }
          umma_commit(bar_empty + 8 * s);   // frees the smem stage once these MMAs have read it
        }
        if (ok) umma_commit(bar_tfull + 8 * acc);   // accumulator complete
      }
    }
  } else if (SUMS && warp >= 2 + kNumEpilogueWarps) {
    // -------------------------------------------------------------------- column sums of A
    if (!waited) pdl_wait();
    const int w = warp - 2 - kNumEpilogueWarps;
    uint32_t it = 0, phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_units && ok; tile += gridDim.x) {
      int m_blk, n_blk, kb0, kb1, outer;
      decode_tile(tile, m_blk, n_blk, kb0, kb1, outer);
      if (n_blk != 0) { it += kb1 - kb0; continue; }
      const int row0 = m_blk * kBlockM;
      SumSlab sum(kb0, ep.col_rows);
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const uint32_t s = it % STAGES;
        if (!mbar_wait(bar_read + 8 * s, phase >> s & 1, abort_flag, status, 9)) { ok = false; break; }
        phase ^= 1u << s;
        sum.block(ep, smem_base + s * L::kStageBytes, kb, K, row0, M, w, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_summed + 8 * s);
      }
      if (ok) sum.rest(ep, kb1, K, row0, M, w, lane);
    }
  } else {
    // -------------------------------------------------------------------- epilogue warps
    if (!waited) pdl_wait();
    const int q = warp & 3;   // TMEM lane quarter this warp may read
    const int ew = warp - 2;  // 0..7
    const int cgrp = ew >> 2; // which half of the tile's columns this warp handles
    // ---- all-gather duty (peer modes 1 and 3): every epilogue warp of every CTA owns a strided share of the 16-row
    // pieces of the remote rows, in the order the tiles consume them.  A warp pulls pieces whenever its next
    // accumulator is not ready yet, and finishes its share after its last tile; nothing a piece needs ever waits.
    const bool gathers = peer.mode == 1 || peer.mode == 3;
    const int tpr = gathers ? peer.rows_per_rank / kBlockM : 0;
    const int num_blk = peer.mode == 1 ? num_m : N / kBlockM;          // 128-row blocks of the gathered operand
    const int remote_items = gathers ? (num_blk - tpr) * kCopyParts : 0;
    const int item_stride = gridDim.x * kNumEpilogueWarps;
    int next_item = blockIdx.x * kNumEpilogueWarps + ew;
    auto copy_one = [&]() {
      const int c = next_item / kCopyParts, part = next_item - c * kCopyParts;
      next_item += item_stride;
      int mt = c + tpr + peer.rank * tpr;                 // consumption order -> global block index
      while (mt >= num_blk) mt -= num_blk;
      const int owner = (mt * kBlockM) / peer.rows_per_rank;
      const long long row0 = static_cast<long long>(mt) * kBlockM + part * (kBlockM / kCopyParts);
      const uint4* src = reinterpret_cast<const uint4*>(peer.a_peer[owner] +
                                                        (row0 - static_cast<long long>(owner) * peer.rows_per_rank) * K);
      uint4* dst = reinterpret_cast<uint4*>(peer.a_full + row0 * K);
      const int total = (kBlockM / kCopyParts) * (K / 8);   // 16-byte chunks per piece
      int i = lane;
      for (; i + 7 * 32 < total; i += 8 * 32) {             // eight peer loads in flight per thread
        uint4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = src[i + u * 32];
#pragma unroll
        for (int u = 0; u < 8; ++u) dst[i + u * 32] = v[u];
      }
      for (; i < total; i += 32) dst[i] = src[i];
      __threadfence();
      __syncwarp();
      if (lane == 0) {
        fence_proxy_async_all();
        red_release_gpu_add(peer.ready + mt, 1u);
      }
      __syncwarp();
    };
    uint32_t t = 0;
    for (int tile = blockIdx.x; tile < num_units; tile += gridDim.x, ++t) {
      int m_blk, n_blk, kb0, kb1, outer;
      decode_tile(tile, m_blk, n_blk, kb0, kb1, outer);
      const bool empty_k = kb1 <= kb0;     // an expert without tokens: the accumulator was never written
      const uint32_t acc = t & 1, acc_ph = (t >> 1) & 1;
      const uint32_t stg = smem_base + L::kStagingOffset + ew * L::kStagingBytesPerWarp;
      const uint32_t side_bars = bar_side + 16 * ew;
      const int row0 = m_blk * kBlockM + q * 32, colg = n_blk * BLOCK_N + cgrp * (BLOCK_N / 2);
      if (L::kSide && ep.side != 0) epilogue_side_load<BLOCK_N / 2>(ep, &tmSide, stg, side_bars, row0, colg, lane);
      while (next_item < remote_items && !mbar_test(bar_tfull + 8 * acc, acc_ph)) copy_one();
      if (!mbar_wait(bar_tfull + 8 * acc, acc_ph, abort_flag, status, 4)) break;
      tc_fence_after();
      const long long row = row0 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BLOCK_N;
      auto arrive = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_tempty + 8 * acc);
      };
      if (L::kTma && ep.staged >= 2) {
        const int drow = num_splits > 1 || grp.mode == 2 ? outer * M + row0 : row0;
        epilogue_tma<BLOCK_N / 2, L::kSlots, EXTRA && !A_MN>(ep, &tmD, &tmAux, stg, side_bars, t, taddr + cgrp * (BLOCK_N / 2), row0, drow, colg, M, N,
                                                    lane, empty_k, abort_flag, status, arrive);
        continue;
      }
      EpiParams epu = ep;
      if (num_splits > 1)
        epu.d = reinterpret_cast<float*>(ep.d) + static_cast<long long>(outer) * d_split_stride;
      if (grp.mode == 2) {
        if (ep.out_f32) epu.d = reinterpret_cast<float*>(ep.d) + static_cast<long long>(outer) * grp.d_expert_stride;
        else epu.d = reinterpret_cast<__nv_bfloat16*>(ep.d) + static_cast<long long>(outer) * grp.d_expert_stride;
      }
      if (peer.mode == 2) {
        // this tile's rows belong to `owner`; write into the owner's receive slot for this rank
        const int owner = (m_blk * kBlockM) / peer.rows_per_rank;
        epu.d = peer.d_peer[owner] + (static_cast<long long>(peer.rank) - owner) * peer.rows_per_rank * ep.ldd;
      }
      if (epu.staged) {
        // registers -> swizzled per-warp tile in shared memory -> whole row segments to global / peer memory
        constexpr int SC = L::kStageCols, CPR = SC / 8;           // staged columns, 16-byte chunks per row
        constexpr int NB = (BLOCK_N / 2) / SC;                    // column blocks per warp group
        const bool two_pass = epu.aux_out != nullptr &&
                              (epu.act == RB_ACT_GELU || epu.act == RB_ACT_RELU || epu.act == RB_ACT_SILU);
        const int num_pass = two_pass ? 2 : 1;
#pragma unroll 1
        for (int hp = 0; hp < NB * num_pass; ++hp) {
          // with a saved pre-activation every column block is read from TMEM twice: first the pre-activation
          // goes out to aux_out, then the activated value to d
          const int h = hp / num_pass;
          const bool pre_pass = two_pass && (hp - h * num_pass) == 0;
          const bool last_pass = hp == NB * num_pass - 1;
          __nv_bfloat16* dbase = pre_pass ? epu.aux_out : reinterpret_cast<__nv_bfloat16*>(epu.d);
          const long long dld = pre_pass ? epu.ld_aux_out : epu.ldd;
#pragma unroll 1
          for (int cc = 0; cc < SC / 32; ++cc) {
            const int c = cgrp * (BLOCK_N / 64) + h * (SC / 32) + cc;
            uint32_t r[32];
            tmem_ld_32x32(taddr + c * 32, r);
            tmem_ld_wait();
            if (last_pass && cc == SC / 32 - 1) arrive();
            const int col0 = n_blk * BLOCK_N + c * 32;
            float v[32];
            if (empty_k) {
#pragma unroll
              for (int j = 0; j < 32; ++j) r[j] = 0u;
            }
            if (row < M && col0 < N) {
              if (pre_pass) epilogue_math<false, true>(epu, r, row, col0, N, v);
              else epilogue_math<false, false>(epu, r, row, col0, N, v);
            } else {
#pragma unroll
              for (int j = 0; j < 32; ++j) v[j] = 0.f;
            }
#pragma unroll
            for (int qq = 0; qq < 4; ++qq) {
              const int chunk = cc * 4 + qq;
              const uint32_t addr = stg + lane * (SC * 2) + ((chunk ^ (lane & (CPR - 1))) << 4);
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr),
                           "r"(pack_bf16x2(v[qq * 8 + 0], v[qq * 8 + 1])), "r"(pack_bf16x2(v[qq * 8 + 2], v[qq * 8 + 3])),
                           "r"(pack_bf16x2(v[qq * 8 + 4], v[qq * 8 + 5])), "r"(pack_bf16x2(v[qq * 8 + 6], v[qq * 8 + 7]))
                           : "memory");
            }
          }
          __syncwarp();
          constexpr int RPI = 32 / CPR;                            // rows written per warp instruction
          const int ch = lane % CPR, rsub = lane / CPR;
          const int colg = n_blk * BLOCK_N + cgrp * (BLOCK_N / 2) + h * SC + ch * 8;
#pragma unroll 4
          for (int r0 = 0; r0 < 32; r0 += RPI) {
            const int rl = r0 + rsub;
            const long long rg = static_cast<long long>(m_blk) * kBlockM + q * 32 + rl;
            uint4 val;
            const uint32_t addr = stg + rl * (SC * 2) + ((ch ^ (rl & (CPR - 1))) << 4);
            asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(val.x), "=r"(val.y), "=r"(val.z), "=r"(val.w) : "r"(addr));
            if (rg < M && colg < N) *reinterpret_cast<uint4*>(dbase + rg * dld + colg) = val;
          }
          __syncwarp();
        }
        continue;
      }
#pragma unroll 1
      for (int c = cgrp * (BLOCK_N / 64); c < (cgrp + 1) * (BLOCK_N / 64); ++c) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + c * 32, r);
        tmem_ld_wait();
        if (empty_k) {
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = 0u;
        }
        // all of this warp's accumulator reads are done: hand the buffer back to the MMA warp
        if (c == (cgrp + 1) * (BLOCK_N / 64) - 1) arrive();
        const int col0 = n_blk * BLOCK_N + c * 32;
        if (row < M && col0 < N) epilogue_chunk(epu, r, row, col0, N);
      }
    }
    while (next_item < remote_items && !*abort_flag) copy_one();
    if (lane == 0) tma_store_wait<0>();      // bulk stores of the last tiles have left shared memory and landed
  }

  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) {
      // give copies and MMAs that are still in flight time to land before TMEM is released
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// ------------------------------------------------------------------------------------------------------------------
// Two-CTA variant (cta_group::2): the two CTAs of a cluster share one 256 x BLOCK_N output tile.  Each CTA loads the
// 128 rows of A it owns and HALF of the B tile (BLOCK_N / 2 rows) into its own shared memory; the even CTA issues
// tcgen05.mma.cta_group::2, which reads both halves of B and writes each CTA's 128 accumulator rows into that CTA's
// TMEM.  Per k-block a CTA moves 16 KB + 16 KB instead of 16 KB + 32 KB through the L2 -> SM fabric, which is what
// bounds the one-CTA kernel on short-K problems.  No TMA multicast: every load targets the loading CTA's own memory
// and reports its bytes to the leader's barrier; tcgen05.commit signals both CTAs' barriers.
// Plain (non-grouped, non-peer) problems only; results leave through TMA (`epilogue_tma`, `epilogue_swiglu`) or, where they cannot, straight
// from registers.
// ------------------------------------------------------------------------------------------------------------------
template <int BLOCK_N, int STAGES>
struct SmemLayoutPair {
  static constexpr int kABytes = kBlockM * kBlockK * 2;
  static constexpr int kBBytes = (BLOCK_N / 2) * kBlockK * 2;
  static constexpr int kStageBytes = kABytes + kBBytes;
  static constexpr int kBarOffset = STAGES * kStageBytes;
  static constexpr int kSumBars = kBarOffset + (2 * STAGES + 4 + 2 * kNumEpilogueWarps) * 8 + 16;
  static constexpr int kTotal = kSumBars + 2 * STAGES * 8;
  static constexpr int kStageCols = 64;
  static constexpr int kSlots = 2;
  static constexpr bool kTma = true, kSide = true;
  static constexpr int kStagingOffset = (kTotal + 1023) & ~1023;   // 1024-byte aligned: the tiles are also TMA-store sources (128B swizzle)
  static constexpr int kStagingBytesPerWarp = kSlots * 32 * kStageCols * 2;
  static constexpr int kTotalStaged = kStagingOffset + kNumEpilogueWarps * kStagingBytesPerWarp;
};

template <int A_MN, int B_MN, int BLOCK_N, int STAGES, int FP8 = 0, bool EXTRA = false>
__global__ void __launch_bounds__(kNumThreads + (EXTRA && A_MN ? 32 * kSumWarps : 0), 1)
gemm_bf16_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                      const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmAux,
                      const __grid_constant__ CUtensorMap tmSide, int M, int N, int K, int group_m, int num_splits, int kb_per_split, long long d_split_stride,
                      const int* expert_offsets, EpiParams ep, unsigned int* status) {
  using L = SmemLayoutPair<BLOCK_N, STAGES>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t smem_base = smem_u32(smem);
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBarOffset);
  const uint32_t bar_full = smem_u32(bars);
  const uint32_t bar_empty = smem_u32(bars + STAGES);
  const uint32_t bar_tfull = smem_u32(bars + 2 * STAGES);
  const uint32_t bar_tempty = smem_u32(bars + 2 * STAGES + 2);
  const uint32_t bar_side = smem_u32(bars + 2 * STAGES + 4);
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 4 + 2 * kNumEpilogueWarps);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);

  constexpr bool SUMS = EXTRA && A_MN;             // column sums of A beside the products
  const uint32_t bar_read = smem_u32(smem + L::kSumBars), bar_summed = bar_read + 8 * STAGES;
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta_rank = cluster_ctarank();       // 0: leader (issues the MMAs), 1: peer
  const int cluster_id = blockIdx.x >> 1;
  const int num_clusters = gridDim.x >> 1;
  constexpr uint32_t kTmemCols = (2 * BLOCK_N <= 64) ? 64 : (2 * BLOCK_N <= 128) ? 128 : (2 * BLOCK_N <= 256) ? 256 : 512;
  constexpr int kPairM = 2 * kBlockM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);                // leader: its own expect_tx arrival (+ both CTAs' bytes)
      mbar_init(bar_empty + 8 * s, 1);               // one multicast commit per use
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(bar_tfull + 8 * a, 1);
      mbar_init(bar_tempty + 8 * a, 2 * kNumEpilogueWarps);   // leader: the epilogue warps of both CTAs
    }
    for (int w = 0; w < 2 * kNumEpilogueWarps; ++w) mbar_init(bar_side + 8 * w, 1);
    if (SUMS) {
      for (int s = 0; s < STAGES; ++s) {
        mbar_init(bar_read + 8 * s, 1);
        mbar_init(bar_summed + 8 * s, kSumWarps);
      }
    }
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc_pair(smem_u32(tmem_ptr_smem), kTmemCols);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                 // the peer's barriers exist before anything signals them
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  bool waited = expert_offsets != nullptr;           // see the one-CTA kernel
  if (waited) {
    pdl_wait();
    pdl_launch();
  }

  const int num_m = (M + kPairM - 1) / kPairM;
  // swiglu: the leader's half of the B tile are 128 gate rows, its peer's the 128 up rows of the same columns, so that both accumulator
  // halves of a CTA belong to one 128-column tile of the result
  const bool glu = ep.act == RB_ACT_SWIGLU;
  const int tile_n = glu ? BLOCK_N / 2 : BLOCK_N;
  const int num_n = (N + tile_n - 1) / tile_n;
  const int num_tiles = num_m * num_n;
  const int num_kb_total = (K + kBlockK - 1) / kBlockK;
  const int group_size = group_m * num_n;
  const int num_units = num_tiles * num_splits;

  auto decode_tile = [&](int unit, int& m_blk, int& n_blk, int& kb0, int& kb1, int& split) {
    split = unit / num_tiles;
    const int tile = unit - split * num_tiles;
    if (A_MN && B_MN && expert_offsets != nullptr) {   // grouped weight gradients: a slab for each expert, from that expert's rows
      kb0 = __ldg(expert_offsets + split) / kBlockK;
      kb1 = __ldg(expert_offsets + split + 1) / kBlockK;
    } else {
      kb0 = split * kb_per_split;
      kb1 = min(num_kb_total, kb0 + kb_per_split);
    }
    const int group = tile / group_size;
    const int first_m = group * group_m;
    const int gm = min(group_m, num_m - first_m);
    const int in_group = tile - group * group_size;
    m_blk = first_m + in_group % gm;
    n_blk = in_group / gm;
  };

  if (warp == 0) {
    if (elect_one()) {
      // ------------------------------------------------------------------ TMA producer (both CTAs)
      SumProducer<STAGES> sums;
      uint32_t it = 0;
      bool ok = true;
      for (int tile = cluster_id; tile < num_units && ok; tile += num_clusters) {
        int m_blk, n_blk, kb0, kb1, split;
        decode_tile(tile, m_blk, n_blk, kb0, kb1, split);
        if (!waited) {
          pdl_wait();
          pdl_launch();
          waited = true;
        }
        const int a_row = m_blk * kPairM + static_cast<int>(cta_rank) * kBlockM;
        const int b_row = n_blk * tile_n + static_cast<int>(cta_rank) * (glu ? N : BLOCK_N / 2);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
          if (!mbar_wait(bar_empty + 8 * s, ph ^ 1, abort_flag, status, 11)) { ok = false; break; }
          if (SUMS) {
            if (!sums.wait(s, bar_summed, abort_flag, status)) { ok = false; break; }
            if (n_blk == 0) sums.used |= 1u << s;
          }
          const uint32_t full_local = bar_full + 8 * s;
          if (cta_rank == 0) mbar_arrive_expect_tx(full_local, 2 * L::kStageBytes);
          const uint32_t full = mapa_shared(full_local, 0);
          const uint32_t sa = smem_base + s * L::kStageBytes;
          const uint32_t sb = sa + L::kABytes;
          if (A_MN == 0) {
            tma_load_2d_pair(sa, &tmA, kb * kBlockK * (FP8 ? 2 : 1), a_row, full);
          } else {
#pragma unroll
            for (int j = 0; j < kBlockM / 64; ++j)
              tma_load_2d_pair(sa + j * (kBlockK * 128), &tmA, a_row + j * 64, kb * kBlockK, full);
          }
          if (B_MN == 0) {
            tma_load_2d_pair(sb, &tmB, kb * kBlockK * (FP8 ? 2 : 1), b_row, full);
          } else {
#pragma unroll
            for (int j = 0; j < BLOCK_N / 2 / 64; ++j)
              tma_load_2d_pair(sb + j * (kBlockK * 128), &tmB, b_row + j * 64, kb * kBlockK, full);
          }
        }
      }
    }
  } else if (warp == 1) {
    if (cta_rank == 0 && elect_one()) {
      // ------------------------------------------------------------------ MMA issuer (leader CTA only)
      const uint32_t idesc = FP8 ? (umma_idesc_e4m3(kPairM, BLOCK_N) | (static_cast<uint32_t>(ep.fp8_b_format) << 10))
                                 : umma_idesc_bf16(kPairM, BLOCK_N, A_MN, B_MN);
      // K-major: 32 bytes per step of 16 inside the swizzle row, 8-row groups 1024 bytes apart.  MN-major: 16 k-rows of 128 bytes per
      // step, 64-wide MN atoms kBlockK * 128 bytes apart.  An offset of o bytes is o / 16 in the address field.
      const uint64_t desc_a = A_MN ? umma_smem_desc_sw128(smem_base, kBlockK * 128, 1024) : umma_smem_desc_sw128(smem_base, 16, 1024);
      const uint64_t desc_b = B_MN ? umma_smem_desc_sw128(smem_base + L::kABytes, kBlockK * 128, 1024) : umma_smem_desc_sw128(smem_base + L::kABytes, 16, 1024);
      constexpr int kStepA = A_MN ? kUmmaK * 8 : kUmmaK / 8, kStepB = B_MN ? kUmmaK * 8 : kUmmaK / 8;
      uint32_t it = 0, t = 0;
      bool ok = true;
      for (int tile = cluster_id; tile < num_units && ok; tile += num_clusters, ++t) {
        int m_blk, n_blk, kb0, kb1, split;
        decode_tile(tile, m_blk, n_blk, kb0, kb1, split);
        if (!waited) {
          pdl_wait();                // the limits of its waits count from here
          waited = true;
        }
        const uint32_t acc = t & 1, acc_ph = (t >> 1) & 1;
        if (!mbar_wait(bar_tempty + 8 * acc, acc_ph ^ 1, abort_flag, status, 12)) { ok = false; break; }
        tc_fence_after();
        const uint32_t tmem_d = tmem_base + acc * BLOCK_N;
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const uint32_t s = it % STAGES, ph = (it / STAGES) & 1;
          if (!mbar_wait(bar_full + 8 * s, ph, abort_flag, status, 13)) { ok = false; break; }
          tc_fence_after();
          const uint64_t da = desc_a + s * (L::kStageBytes / 16), db = desc_b + s * (L::kStageBytes / 16);
#pragma unroll
          for (int k = 0; k < kBlockK / kUmmaK; ++k) {
            if (FP8) umma_f8_ss_pair(tmem_d, da + k * kStepA, db + k * kStepB, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
            else umma_bf16_ss_pair(tmem_d, da + k * kStepA, db + k * kStepB, idesc, (kb != kb0 || k != 0) ? 1u : 0u);
          }
          if (SUMS && n_blk == 0) umma_commit_pair(bar_read + 8 * s, 3);
          umma_commit_pair(bar_empty + 8 * s, 3);     // both CTAs may refill this stage
        }
        if (ok) umma_commit_pair(bar_tfull + 8 * acc, 3);   // both CTAs' accumulator halves are complete
      }
    }
  } else if (SUMS && warp >= 2 + kNumEpilogueWarps) {
    // -------------------------------------------------------------------- column sums of A
    if (!waited) pdl_wait();
    const int w = warp - 2 - kNumEpilogueWarps;
    uint32_t it = 0, phase = 0;
    bool ok = true;
    for (int tile = cluster_id; tile < num_units && ok; tile += num_clusters) {
      int m_blk, n_blk, kb0, kb1, split;
      decode_tile(tile, m_blk, n_blk, kb0, kb1, split);
      if (n_blk != 0) { it += kb1 - kb0; continue; }
      const int row0 = m_blk * kPairM + static_cast<int>(cta_rank) * kBlockM;
      SumSlab sum(kb0, ep.col_rows);
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const uint32_t s = it % STAGES;
        if (!mbar_wait(bar_read + 8 * s, phase >> s & 1, abort_flag, status, 9)) { ok = false; break; }
        phase ^= 1u << s;
        sum.block(ep, smem_base + s * L::kStageBytes, kb, K, row0, M, w, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_summed + 8 * s);
      }
      if (ok) sum.rest(ep, kb1, K, row0, M, w, lane);
    }
  } else {
    // -------------------------------------------------------------------- epilogue warps (both CTAs)
    if (!waited) pdl_wait();
    const int q = warp & 3;
    const int ew = warp - 2;
    const int cgrp = ew >> 2;
    uint32_t t = 0;
    for (int tile = cluster_id; tile < num_units; tile += num_clusters, ++t) {
      int m_blk, n_blk, kb0, kb1, split;
      decode_tile(tile, m_blk, n_blk, kb0, kb1, split);
      const bool empty_k = A_MN && B_MN && kb1 <= kb0;   // an expert without rows: the accumulator was never written
      const uint32_t acc = t & 1, acc_ph = (t >> 1) & 1;
      const uint32_t stg = smem_base + L::kStagingOffset + ew * L::kStagingBytesPerWarp;
      const uint32_t side_bars = bar_side + 16 * ew;
      const int row0 = m_blk * kPairM + static_cast<int>(cta_rank) * kBlockM + q * 32, colg = n_blk * tile_n + cgrp * (tile_n / 2);
      if (ep.side != 0) epilogue_side_load<BLOCK_N / 2>(ep, &tmSide, stg, side_bars, row0, colg, lane);
      if (!mbar_wait(bar_tfull + 8 * acc, acc_ph, abort_flag, status, 14)) break;
      tc_fence_after();
      const long long row = row0 + lane;
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(q * 32) << 16) + acc * BLOCK_N;
      const uint32_t tempty_leader = mapa_shared(bar_tempty + 8 * acc, 0);
      auto arrive = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(tempty_leader);
      };
      if (glu) {
        epilogue_swiglu(&tmD, stg, t, taddr + cgrp * 64, row0, colg, M, lane, arrive);
        continue;
      }
      if (ep.staged >= 2) {
        const int drow = num_splits > 1 ? split * M + row0 : row0;
        epilogue_tma<BLOCK_N / 2, L::kSlots, EXTRA && !A_MN>(ep, &tmD, &tmAux, stg, side_bars, t, taddr + cgrp * (BLOCK_N / 2), row0, drow, colg, M, N,
                                                    lane, empty_k, abort_flag, status, arrive);
        continue;
      }
      EpiParams epu = ep;
      if (num_splits > 1)
        epu.d = static_cast<char*>(ep.d) + static_cast<long long>(split) * d_split_stride * (ep.out_f32 ? 4 : 2);
#pragma unroll 1
      for (int c = cgrp * (BLOCK_N / 64); c < (cgrp + 1) * (BLOCK_N / 64); ++c) {
        uint32_t r[32];
        tmem_ld_32x32(taddr + c * 32, r);
        tmem_ld_wait();
        if (empty_k) {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = 0;
        }
        if (c == (cgrp + 1) * (BLOCK_N / 64) - 1) arrive();
        const int col0 = n_blk * BLOCK_N + c * 32;
        if (row < M && col0 < N) epilogue_chunk(epu, r, row, col0, N);
      }
    }
    if (lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  cluster_sync_all();                                 // the leader's MMAs read this CTA's shared memory until here
  if (warp == 1) {
    if (*abort_flag) {
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols);
  }
}

// d (+)= sum_s ws[s] (+ bias) (+ residual)  (slabs of M*N fp32, dense), s ascending: the order is fixed, so the
// result is reproducible.
__global__ void __launch_bounds__(256)
splitk_reduce_kernel(const float* __restrict__ ws, int splits, long long slab, void* d, long long ldd, int M, int N,
                     int out_f32, int accumulate, const __nv_bfloat16* __restrict__ bias,
                     const __nv_bfloat16* __restrict__ residual, long long ldr) {
  pdl_wait();
  pdl_launch();
  const long long n4 = static_cast<long long>(M) * N / 4;
  const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
    float4 acc = reinterpret_cast<const float4*>(ws)[i];
    for (int s = 1; s < splits; ++s) {
      const float4 v = reinterpret_cast<const float4*>(ws + s * slab)[i];
      acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
    }
    const long long e = i * 4;
    const long long row = e / N;
    const int col = static_cast<int>(e - row * N);
    if (bias != nullptr) {
      const uint2 b = __ldg(reinterpret_cast<const uint2*>(bias + col));
      const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y);
      acc.x += b0.x; acc.y += b0.y; acc.z += b1.x; acc.w += b1.y;
    }
    if (residual != nullptr) {
      const uint2 r = __ldg(reinterpret_cast<const uint2*>(residual + row * ldr + col));
      const float2 r0 = unpack_bf16x2(r.x), r1 = unpack_bf16x2(r.y);
      acc.x += r0.x; acc.y += r0.y; acc.z += r1.x; acc.w += r1.y;
    }
    if (out_f32) {
      float4* dp = reinterpret_cast<float4*>(reinterpret_cast<float*>(d) + row * ldd + col);
      if (accumulate) { const float4 o = *dp; acc.x += o.x; acc.y += o.y; acc.z += o.z; acc.w += o.w; }
      *dp = acc;
    } else {
      uint2* dp = reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(d) + row * ldd + col);
      if (accumulate) {
        const uint2 o = *dp;
        const float2 a = unpack_bf16x2(o.x), b = unpack_bf16x2(o.y);
        acc.x += a.x; acc.y += a.y; acc.z += b.x; acc.w += b.y;
      }
      uint2 o;
      o.x = pack_bf16x2(acc.x, acc.y);
      o.y = pack_bf16x2(acc.z, acc.w);
      *dp = o;
    }
  }
}

}  // namespace rb

// ---------------------------------------------------------------------------------------------
// host launcher
// ---------------------------------------------------------------------------------------------
namespace {

// RUSTRAL_GEMM_STAGED=0/1 turns the shared-memory staged output path off / on for ordinary (non-peer) GEMMs.
bool staged_store_default() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("RUSTRAL_GEMM_STAGED");
    v = (e && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

// Staged 64-column tiles leave through bulk tensor stores (one instruction per tile instead of eight ld.shared /
// st.global pairs per thread); RUSTRAL_GEMM_TMA_STORE=0 keeps the load / store loop.  Measured on one B200, same process:
// bias + GELU + saved pre-activation 32768 x 3072 x 768 224 -> 194 us, QKV shape 99.3 -> 95.3 us, 8192^3 unchanged.
bool tma_store_default() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("RUSTRAL_GEMM_TMA_STORE");
    v = (e && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

// Fills the epilogue's parameters and the tensor maps of what TMA moves for it.  Returns the shared memory to ask for.  `extra` on entry: the
// kernel exists with the EXTRA forms; on return: it has to be that one.
template <class L>
int plan_epilogue(const RbGemmArgs& g, int splits, rb::EpiParams& ep, const CUtensorMap*& td, const CUtensorMap*& tx,
                  const CUtensorMap*& ts, bool& extra) {
  const bool may_extra = extra;
  extra = false;
  ep.d = g.d; ep.ldd = g.ldd;
  ep.bias = reinterpret_cast<const __nv_bfloat16*>(g.bias);
  ep.residual = reinterpret_cast<const __nv_bfloat16*>(g.residual); ep.ldr = g.ldr;
  ep.aux_in = reinterpret_cast<const __nv_bfloat16*>(g.aux_in); ep.ld_aux_in = g.ld_aux_in;
  ep.aux_out = reinterpret_cast<__nv_bfloat16*>(g.aux_out); ep.ld_aux_out = g.ld_aux_out;
  ep.act = g.act; ep.out_f32 = g.out_f32; ep.accumulate = g.accumulate; ep.alpha = g.alpha;
  ep.row_scale = reinterpret_cast<const float*>(g.a_scale);
  ep.col_scale = reinterpret_cast<const float*>(g.b_scale);
  ep.fp8_b_format = g.ab_fp8 == 2 ? 1 : 0;
  ep.staged = 0; ep.side = 0;
  ep.col_sum = g.col_sum; ep.col_rows = g.col_rows;
  ep.col_src = reinterpret_cast<const __nv_bfloat16*>(g.a); ep.col_ld = g.lda;
  if (splits > 1) {
    ep.d = g.workspace; ep.ldd = g.N; ep.out_f32 = 1; ep.accumulate = 0;
    ep.bias = nullptr; ep.residual = nullptr;          // applied once, by the kernel that folds the slabs
  }
  static_assert(L::kTotalStaged + 1024 <= 232448, "the ring and the result tiles share an SM's memory");
  const bool tma = L::kTma && g.peer_mode == 0 && tma_store_default() && staged_store_default();
  // slabs of a split contraction and the experts' results (grouped mode 2) lie below one another: whole 32-row tiles keep each in its own
  const bool stacked = g.M % 32 == 0 && (splits > 1 || (tma && g.d_expert_stride == static_cast<long long>(g.M) * g.ldd));
  const uint64_t stack = splits > 1 ? splits : g.group_mode == 2 ? g.num_experts : 1;
  int err = 0;
  if (!ep.out_f32) {
    if (g.accumulate || (g.N % 8) || (g.group_mode == 2 && !stacked)) return L::kTotal + 1024;
    if (g.peer_mode != 2 && !staged_store_default()) return L::kTotal + 1024;
    ep.staged = 1;
    const bool reads = g.aux_in || g.residual;
    const bool more = L::kSide ? (g.aux_in && g.residual) || (reads && g.aux_out) : reads || g.aux_out;     // than the tiles suffice for
    if (tma && (may_extra || !more)) {
      const uint64_t n = g.N, m = g.M * stack;
      const CUtensorMap* d = rbhost::get_tmap_2d(g.d, 2, n, m, (uint64_t)g.ldd, 64, 32, 1, &err);
      const CUtensorMap* x = g.aux_out ? rbhost::get_tmap_2d(g.aux_out, 2, n, m, (uint64_t)g.ld_aux_out, 64, 32, 1, &err) : d;
      const CUtensorMap* side = nullptr;
      if (L::kSide && !g.aux_out) {            // a second result needs the tiles itself
        if (g.aux_in) side = rbhost::get_tmap_2d(g.aux_in, 2, n, m, (uint64_t)g.ld_aux_in, 64, 32, 1, &err);
        else if (g.residual) side = rbhost::get_tmap_2d(g.residual, 2, n, m, (uint64_t)g.ldr, 64, 32, 1, &err);
      }
      if (d && x && (side || more || !reads)) {
        ep.staged = 2; td = d; tx = x;
        if (side) { ts = side; ep.side = g.aux_in ? 2 : 1; }
        extra = more;
      }
    }
  } else if (tma && (stack == 1 || stacked) && ep.ldd % 4 == 0 && g.N % 4 == 0 && g.act == RB_ACT_NONE &&
             !ep.residual) {
    const CUtensorMap* d = rbhost::get_tmap_2d(ep.d, 4, (uint64_t)g.N, (uint64_t)g.M * stack, (uint64_t)ep.ldd, 32, 32, 1, &err);
    if (d) { ep.staged = ep.accumulate ? 4 : 3; td = d; ep.accumulate = 0; }
  }
  return (ep.staged ? L::kTotalStaged : L::kTotal) + 1024;
}

template <int A_MN, int B_MN, int BLOCK_N, int STAGES, int FP8 = 0>
int launch(const RbGemmArgs& g, const CUtensorMap* ta, const CUtensorMap* tb, int grid, int splits, cudaStream_t stream) {
  using L = rb::SmemLayout<BLOCK_N, STAGES>;
  const int group_m = g.group_m > 0 ? g.group_m : 8;
  const int k_units = FP8 ? (g.K + 1) / 2 : g.K;          // the kernel counts K in two-byte units
  const int num_kb = (k_units + rb::kBlockK - 1) / rb::kBlockK;
  int kb_per = num_kb;
  long long slab = 0;
  if (splits > 1) {
    kb_per = (num_kb + splits - 1) / splits;
    splits = (num_kb + kb_per - 1) / kb_per;   // no split may end up with an empty K range
    slab = static_cast<long long>(g.M) * g.N;
  }
  const CUtensorMap *td = ta, *tx = ta, *ts = ta;         // placeholders unless TMA moves the results
  auto kern = rb::gemm_bf16_kernel<A_MN, B_MN, BLOCK_N, STAGES, FP8>;
  constexpr bool kExtra = (!A_MN && !FP8 && L::kTma) || (A_MN && B_MN);       // forward products and input gradients; weight gradients
  bool extra = kExtra && !A_MN;
  rb::EpiParams ep;
  const int smem = plan_epilogue<L>(g, splits, ep, td, tx, ts, extra);
  if (A_MN) extra = kExtra && g.col_sum != nullptr;
  const int threads = rb::kNumThreads + (A_MN && extra ? 32 * rb::kSumWarps : 0);
  if constexpr (kExtra)
    if (extra) kern = rb::gemm_bf16_kernel<A_MN, B_MN, BLOCK_N, STAGES, FP8, true>;
  if (g.peer_mode == 2 && !ep.staged) return -11;
  static int configured_dev[2][64] = {{0}};   // per instantiation and device: largest size set so far
  int& configured = configured_dev[extra][rbhost::device_slot()];
  if (configured < smem) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = smem;
  }
  rb::GroupInfo grp;
  grp.mode = g.group_mode; grp.num_experts = g.num_experts;
  grp.tile_expert = reinterpret_cast<const int*>(g.tile_expert);
  grp.num_m_tiles = reinterpret_cast<const int*>(g.num_m_tiles);
  grp.offsets = reinterpret_cast<const int*>(g.expert_offsets);
  grp.b_expert_rows = g.b_expert_rows; grp.d_expert_stride = g.d_expert_stride;
  grp.tile_arrived = reinterpret_cast<const unsigned int*>(g.tile_arrived);
  grp.tile_expected = reinterpret_cast<const int*>(g.tile_expected);
  rb::PeerInfo peer;
  memset(&peer, 0, sizeof(peer));
  peer.mode = g.peer_mode; peer.world = g.peer_world; peer.rank = g.peer_rank; peer.rows_per_rank = g.rows_per_rank;
  peer.a_full = reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(g.peer_mode == 3 ? g.b : g.a));
  peer.ready = reinterpret_cast<unsigned int*>(g.ready_flags);
  peer.epoch = g.peer_epoch;
  for (int r = 0; r < 8; ++r) {
    peer.a_peer[r] = reinterpret_cast<const __nv_bfloat16*>(g.peer_ptrs[r]);
    peer.d_peer[r] = reinterpret_cast<__nv_bfloat16*>(const_cast<void*>(g.peer_ptrs[r]));
  }
  rbhost::launch_pdl(kern, dim3(grid), dim3(threads), smem, stream, 1, *ta, *tb, *td, *tx, *ts, g.M, g.N, k_units, group_m, splits, kb_per, slab, ep, grp, peer,
                                                rbhost::status_ptr());
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || splits <= 1) return static_cast<int>(e);
  const long long n4 = slab / 4;
  int rgrid = static_cast<int>((n4 + 255) / 256 < 148 * 8 ? (n4 + 255) / 256 : 148 * 8);
  rbhost::launch_pdl(rb::splitk_reduce_kernel, dim3(rgrid), dim3(256), 0, stream, 1, reinterpret_cast<const float*>(g.workspace), splits, slab, g.d,
                                                      g.ldd, g.M, g.N, g.out_f32, g.accumulate,
                                                      reinterpret_cast<const __nv_bfloat16*>(g.bias),
                                                      reinterpret_cast<const __nv_bfloat16*>(g.residual), g.ldr);
  return static_cast<int>(cudaGetLastError());
}

template <int BLOCK_N, int STAGES>
int dispatch_major(const RbGemmArgs& g, const CUtensorMap* ta, const CUtensorMap* tb, int grid, int splits,
                   cudaStream_t s) {
  if (!g.a_mn_major && !g.b_mn_major) return launch<0, 0, BLOCK_N, STAGES>(g, ta, tb, grid, splits, s);
  if (!g.a_mn_major && g.b_mn_major) return launch<0, 1, BLOCK_N, STAGES>(g, ta, tb, grid, splits, s);
  if (g.a_mn_major && g.b_mn_major) return launch<1, 1, BLOCK_N, STAGES>(g, ta, tb, grid, splits, s);
  return launch<1, 0, BLOCK_N, STAGES>(g, ta, tb, grid, splits, s);
}

// RUSTRAL_GEMM_2CTA=0 keeps every problem on the one-CTA kernel.
bool pair_kernel_enabled() {
  static int v = -1;
  if (v < 0) {
    const char* e = getenv("RUSTRAL_GEMM_2CTA");
    v = (e && e[0] == '0') ? 0 : 1;
  }
  return v == 1;
}

// Problems for the two-CTA kernel (where their tiles are 256 wide).  Of the grouped ones the weight gradients whose experts' results are
// stacked in whole 32-row tiles, so that TMA stores them: every expert has all M x N of its tiles and only the contraction is ragged,
// which costs a pair nothing: eight experts of 16384 x 2048 and 2048 x 8192 over about 750 rows each, forward and backward of the layer
// 2226 us with single CTAs, 2130 with pairs.
// The grouped products over permuted rows stay: an expert's rows come in 128-row tiles, and a pair would leave half a tile idle behind
// every second expert.
bool pair_takes(const RbGemmArgs& g) {
  if (g.peer_mode != 0 || g.M <= 128 || g.max_ctas != 0 || !pair_kernel_enabled()) return false;
  return g.group_mode == 0 || (g.group_mode == 2 && g.M % 32 == 0 && g.d_expert_stride == static_cast<long long>(g.M) * g.ldd);
}

template <int A_MN, int B_MN, int FP8 = 0>
int launch_pair(const RbGemmArgs& g, const CUtensorMap* ta, const CUtensorMap* tb_half, int clusters, int splits,
                cudaStream_t stream) {
  constexpr int BLOCK_N = 256, STAGES = 5;
  using L = rb::SmemLayoutPair<BLOCK_N, STAGES>;
  auto kern = rb::gemm_bf16_pair_kernel<A_MN, B_MN, BLOCK_N, STAGES, FP8>;
  const int group_m = g.group_m > 0 ? g.group_m : 4;      // in 256-row units
  const int k_units = FP8 ? (g.K + 1) / 2 : g.K;
  const int num_kb = (k_units + rb::kBlockK - 1) / rb::kBlockK;
  int kb_per = num_kb;
  long long slab = 0;
  if (splits > 1) {
    kb_per = (num_kb + splits - 1) / splits;
    splits = (num_kb + kb_per - 1) / kb_per;
    slab = static_cast<long long>(g.M) * g.N;
  }
  const bool grouped = g.group_mode == 2;                 // a slab for each expert, not folded
  if (grouped) slab = g.d_expert_stride;
  const CUtensorMap *td = ta, *tx = ta, *ts = ta;
  rb::EpiParams ep;
  constexpr bool kExtra = (!A_MN && !FP8) || (A_MN && B_MN);                  // forward products and input gradients; weight gradients
  bool extra = kExtra && !A_MN;
  int smem = plan_epilogue<L>(g, splits, ep, td, tx, ts, extra);
  if (A_MN) extra = kExtra && g.col_sum != nullptr;
  const int threads = rb::kNumThreads + (A_MN && extra ? 32 * rb::kSumWarps : 0);
  if constexpr (kExtra)
    if (extra) kern = rb::gemm_bf16_pair_kernel<A_MN, B_MN, BLOCK_N, STAGES, FP8, true>;
  if (g.act == RB_ACT_SWIGLU && ep.staged != 2) return -9;
  if (ep.staged == 1) ep.staged = 0, smem = L::kTotal + 1024;       // this kernel stores through TMA or straight from registers
  static int configured_dev[2][64] = {{0}};
  int& configured = configured_dev[extra][rbhost::device_slot()];
  if (configured < smem) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = smem;
  }
  const cudaError_t e = rbhost::launch_pdl(kern, dim3(2 * clusters), dim3(threads), smem, stream, 2, *ta, *tb_half, *td, *tx, *ts, g.M, g.N,
                                           k_units, group_m, grouped ? g.num_experts : splits, kb_per, slab,
                                           grouped ? reinterpret_cast<const int*>(g.expert_offsets) : nullptr, ep, rbhost::status_ptr());
  if (e != cudaSuccess || splits <= 1) return static_cast<int>(e);
  const long long n4 = slab / 4;
  int rgrid = static_cast<int>((n4 + 255) / 256 < 148 * 8 ? (n4 + 255) / 256 : 148 * 8);
  rbhost::launch_pdl(rb::splitk_reduce_kernel, dim3(rgrid), dim3(256), 0, stream, 1, reinterpret_cast<const float*>(g.workspace), splits, slab, g.d,
                                                      g.ldd, g.M, g.N, g.out_f32, g.accumulate,
                                                      reinterpret_cast<const __nv_bfloat16*>(g.bias),
                                                      reinterpret_cast<const __nv_bfloat16*>(g.residual), g.ldr);
  return static_cast<int>(cudaGetLastError());
}

// Relative time of one tile column unit per tile width: narrow tiles re-read the A operand from shared
// memory more often per MMA (measured on B200: 128-wide runs ~1.3x, 64-wide ~2.3x slower than 256-wide).
int width_cost(int bn) { return bn == 256 ? 100 : bn == 192 ? 104 : bn == 128 ? 132 : 235; }

// Microseconds of a plan: waves of tiles at the measured rate (6.5 ns per unit of K for a 128 x 256 tile), the last tile's results, and
// for a split contraction a second launch and the slabs' way through memory.  Leaving the slabs out of the sum had wide results split
// that should not be (measured, split / whole): 2048 x 8192 x 4096 135 / 101 us, 4096 x 2048 x 8192 131 / 98, 2704 x 2048 x 2048 42 / 25.
double plan_cost(int M, int N, int K, int bn, int splits, int experts, int sms, bool pair_ok) {
  const long long tiles = static_cast<long long>((M + 127) / 128) * ((N + bn - 1) / bn) * splits * experts;
  const long long waves = (tiles + sms - 1) / sms;
  // 256-wide plans of plain problems run on the two-CTA kernel, measured about 10 % faster per tile
  const int wc = (bn == 256 && pair_ok) ? 88 : width_cost(bn);
  const double width = bn / 256.0;
  double us = waves * width * (wc / 100.0) * (static_cast<double>(K) / (splits * experts)) * 0.0065 + 1.5 * width;
  if (splits > 1) us += 2.0 + (2.0 * splits + 1.0) * M * static_cast<double>(N) * 4.0 / 5.0e6;
  return us;
}

void pick_plan(const RbGemmArgs& g, int sms, int& bn_out, int& splits_out) {
  const int cands[4] = {256, 192, 128, 64};
  const int split_cands[7] = {1, 2, 3, 4, 6, 8, 12};
  const bool can_split = g.group_mode == 0 && g.peer_mode == 0 && g.workspace != nullptr && g.act == RB_ACT_NONE && !g.aux_out &&
                         !g.a_scale && !g.b_scale && !g.ab_fp8 &&
                         (g.N % 4 == 0) && (static_cast<long long>(g.M) * g.N % 4 == 0) && (!g.residual || (g.ldr % 4 == 0));
  const bool pair_ok = pair_takes(g);
  const int experts = g.group_mode == 2 ? g.num_experts : 1;      // each with tiles of its own and, on average, its part of the contraction
  double best = -1.0;
  bn_out = 128; splits_out = 1;
  for (int c = 0; c < 4; ++c) {
    const int bn = cands[c];
    if (g.block_n && g.block_n != bn) continue;
    if (!g.block_n && bn > 64 && g.N <= bn / 2) continue;
    for (int si = 0; si < 7; ++si) {
      const int sp = split_cands[si];
      if (g.splits > 0 && sp != g.splits) continue;
      if (sp > 1) {
        if (!can_split) continue;
        if (g.splits <= 0 && g.K / sp < 768) continue;
        if (static_cast<long long>(sp) * g.M * g.N * 4 > g.workspace_bytes) continue;
      }
      const double cost = plan_cost(g.M, g.N, g.K, bn, sp, experts, sms, pair_ok);
      if (best < 0.0 || cost < best) { best = cost; bn_out = bn; splits_out = sp; }
    }
  }
}

int gemm_swiglu(const RbGemmArgs& g, cudaStream_t stream) {
  if (g.a_mn_major || g.b_mn_major || g.bias || g.residual || g.aux_in || g.aux_out || g.out_f32 || g.accumulate || g.alpha != 1.f ||
      g.group_mode || g.peer_mode || g.ab_fp8 || g.a_scale || g.b_scale || g.splits > 1 || g.block_n || g.max_ctas || g.group_m || (g.N % 8))
    return -9;
  if (rbhost::gemm_rows_takes(g)) return rbhost::gemm_rows(g, stream);
  if (g.M <= 128 || !pair_kernel_enabled() || !tma_store_default() || !staged_store_default()) return -9;
  // The tiles of this form are 256 x 128 only.  Where they leave most pairs of SMs idle, a product of narrower tiles and a second launch are the
  // faster way, at the shorter contractions less so (us, this form / two launches): 256 x 512 x 4096 24.7 / 12.9, 512 x 512 x 8192 43.5 / 19.1, 256
  // x 2304 x 4096 (18 tiles) 26.2 / 21.3, 256 x 3072 x 4096 (24) 26.8 / 26.2, 300 x 1792 x 4096 (28) 26.1 / 36.6; 256 x 1024 x 1024 (8) 11.0 / 9.5, 1024
  // x 512 x 768 (16) 9.9 / 10.9, 768 x 768 x 768 (18) 10.3 / 10.9.
  const long long tiles = (long long)((g.M + 255) / 256) * ((g.N + 127) / 128);
  const int most = rbhost::device_sm_count() / 2;
  if (tiles * (g.K >= 2048 ? 4 : 5) <= most) return -9;
  int err = 0;
  const CUtensorMap* ta = rbhost::get_tmap_2d(g.a, 2, (uint64_t)g.K, (uint64_t)g.M, (uint64_t)g.lda, 64, 128, 1, &err);
  if (!ta) return err ? err : -5;
  const CUtensorMap* tb = rbhost::get_tmap_2d(g.b, 2, (uint64_t)g.K, 2 * (uint64_t)g.N, (uint64_t)g.ldb, 64, 128, 1, &err);
  if (!tb) return err ? err : -5;
  return launch_pair<0, 0>(g, ta, tb, static_cast<int>(tiles < most ? tiles : most), 1, stream);
}

// 8-bit floating-point operands: byte tensor maps with 128-element boxes, K-major only.
int gemm_fp8(const RbGemmArgs& g, int sms, int bn, int splits, cudaStream_t stream) {
  if (g.a_mn_major || g.b_mn_major || g.peer_mode != 0 || g.group_mode == 2) return -12;
  if ((g.lda & 15) || (g.ldb & 15) || (g.K & 15)) return -2;
  int err = 0;
  const CUtensorMap* ta = rbhost::get_tmap_2d(g.a, 1, (uint64_t)g.K, (uint64_t)g.M, (uint64_t)g.lda, 128, 128, 1, &err);
  if (!ta) return err ? err : -5;
  const uint64_t b_experts = g.group_mode == 1 ? (uint64_t)g.num_experts : 1;
  if (bn == 256 && g.group_mode == 0 && g.M > 128 && g.max_ctas == 0 && pair_kernel_enabled()) {
    const CUtensorMap* tb_half = rbhost::get_tmap_2d(g.b, 1, (uint64_t)g.K, (uint64_t)g.N, (uint64_t)g.ldb, 128, 128, 1, &err);
    if (!tb_half) return err ? err : -5;
    const long long tiles2 = (long long)((g.M + 255) / 256) * ((g.N + 255) / 256) * splits;
    const int max_clusters = sms / 2;
    const int clusters = static_cast<int>(tiles2 < max_clusters ? tiles2 : max_clusters);
    return launch_pair<0, 0, 1>(g, ta, tb_half, clusters, splits, stream);
  }
  const CUtensorMap* tb = rbhost::get_tmap_2d(g.b, 1, (uint64_t)g.K, (uint64_t)g.N * b_experts, (uint64_t)g.ldb, 128, (uint32_t)bn, 1, &err);
  if (!tb) return err ? err : -5;
  const long long tiles = (long long)((g.M + 127) / 128) * ((g.N + bn - 1) / bn) * splits;
  int grid = static_cast<int>(tiles < sms ? tiles : sms);
  if (g.max_ctas > 0 && grid > g.max_ctas) grid = g.max_ctas;
  switch (bn) {
    case 256: return launch<0, 0, 256, 4, 1>(g, ta, tb, grid, splits, stream);
    case 192: return launch<0, 0, 192, 5, 1>(g, ta, tb, grid, splits, stream);
    case 128: return launch<0, 0, 128, 5, 1>(g, ta, tb, grid, splits, stream);
    default: return launch<0, 0, 64, 8, 1>(g, ta, tb, grid, splits, stream);
  }
}

}  // namespace

RB_API long long rb_gemm_workspace(const RbGemmArgs* args, long long most) {
  RbGemmArgs g = *args;
  g.workspace = &g;                           // any address: nothing is launched
  g.workspace_bytes = most;
  if (g.M <= 0 || g.N <= 0 || g.K <= 0 || g.act == RB_ACT_SWIGLU || rbhost::gemm_rows_takes(g)) return 0;
  int bn = 128, splits = 1;
  pick_plan(g, rbhost::device_sm_count(), bn, splits);
  return splits > 1 ? static_cast<long long>(splits) * g.M * g.N * 4 : 0;
}

static int gemm_bf16(const RbGemmArgs& g, cudaStream_t stream) {
  if (g.M <= 0 || g.N <= 0 || g.K <= 0) return -1;
  // TMA needs 16-byte aligned bases and pitches
  if ((reinterpret_cast<uintptr_t>(g.a) & 15) || (reinterpret_cast<uintptr_t>(g.b) & 15)) return -2;
  if (!g.ab_fp8 && ((g.lda & 7) || (g.ldb & 7))) return -2;
  // vector epilogue accesses need 16-byte aligned rows
  const int dalign = g.out_f32 ? 4 : 8;
  if ((g.ldd % dalign) || (reinterpret_cast<uintptr_t>(g.d) & 15)) return -3;
  if (g.residual && ((g.ldr & 7) || (reinterpret_cast<uintptr_t>(g.residual) & 15))) return -3;
  if (g.aux_in && ((g.ld_aux_in & 7) || (reinterpret_cast<uintptr_t>(g.aux_in) & 15))) return -3;
  if (g.aux_out && ((g.ld_aux_out & 7) || (reinterpret_cast<uintptr_t>(g.aux_out) & 15))) return -3;
  if (g.bias && (reinterpret_cast<uintptr_t>(g.bias) & 15)) return -3;
  if (g.a_scale && (reinterpret_cast<uintptr_t>(g.a_scale) & 3)) return -3;
  if (g.b_scale && (reinterpret_cast<uintptr_t>(g.b_scale) & 15)) return -3;
  if ((g.act >= RB_ACT_DGELU && g.act <= RB_ACT_MUL) && !g.aux_in) return -4;
  if (g.act == RB_ACT_RELU2 && g.aux_out) return -4;
  if (g.norm_gamma) {
    if (!rbhost::gemm_rows_norm_takes(g) || !rbhost::gemm_rows_takes(g) || (g.act == RB_ACT_SWIGLU && (g.bias || g.residual || g.out_f32))) return -9;
    if (((reinterpret_cast<uintptr_t>(g.norm_gamma) | reinterpret_cast<uintptr_t>(g.norm_beta)) & 15)) return -3;
    return rbhost::gemm_rows(g, stream);
  }

  if (g.group_mode < 0 || g.group_mode > 2) return -8;
  if (g.group_mode == 1 && (!g.tile_expert || !g.num_m_tiles || g.b_expert_rows <= 0)) return -8;
  if ((g.tile_arrived == nullptr) != (g.tile_expected == nullptr) || (g.tile_arrived && g.group_mode != 1)) return -8;
  if (g.group_mode == 1 && g.b_mn_major && (g.K % 64)) return -8;     // expert K ranges must be whole k-blocks
  if (g.group_mode == 2 && (!g.expert_offsets || g.num_experts <= 0 || !g.a_mn_major || !g.b_mn_major)) return -8;
  if (g.peer_mode < 0 || g.peer_mode > 3) return -11;
  RbGemmArgs forced;
  if (g.peer_mode == 3) {
    // tiles must not straddle two ranks' blocks of B: the tile width divides the rows per rank
    if (g.rows_per_rank <= 0 || (g.rows_per_rank % 128)) return -11;
    const int want = (g.rows_per_rank % 256 == 0) ? 256 : 128;
    if (g.block_n != 0 && g.block_n != 128 && g.block_n != want) return -11;
    if (g.block_n == 0) {
      forced = g;
      forced.block_n = want;
      return gemm_bf16(forced, stream);
    }
  }
  if (g.peer_mode != 0) {
    if (g.peer_world < 2 || g.peer_world > 8 || g.peer_rank < 0 || g.peer_rank >= g.peer_world) return -11;
    if (g.rows_per_rank <= 0 || (g.rows_per_rank % 128) ||
        g.rows_per_rank * g.peer_world != (g.peer_mode == 3 ? g.N : g.M))
      return -11;
    if (g.peer_mode == 3 && (g.b_mn_major || !g.ready_flags || g.ldb != g.K)) return -11;   // b_full is dense [N, K]
    if ((g.peer_mode == 1 && g.a_mn_major) || g.group_mode != 0 || g.out_f32) return -11;
    for (int r = 0; r < g.peer_world; ++r)
      if (!g.peer_ptrs[r] || (reinterpret_cast<uintptr_t>(g.peer_ptrs[r]) & 15)) return -11;
    if (g.peer_mode == 1 && (!g.ready_flags || g.lda != g.K)) return -11;       // a_full is dense [M, K]
  }
  if (g.col_sum && (!g.a_mn_major || !g.b_mn_major || g.group_mode || g.peer_mode || g.ab_fp8 || g.act != RB_ACT_NONE ||
                    (reinterpret_cast<uintptr_t>(g.col_sum) & 3) || !g.col_out || g.col_rows <= 0 || g.col_rows % rb::kBlockK || (g.M & 7)))
    return -9;
  if (g.act == RB_ACT_SWIGLU) return gemm_swiglu(g, stream);
  const int sms = rbhost::device_sm_count();
  if (g.block_n != 0 && g.block_n != 64 && g.block_n != 128 && g.block_n != 192 && g.block_n != 256) return -6;
  if (rbhost::gemm_rows_takes(g)) return rbhost::gemm_rows(g, stream);
  int bn = 128, splits = 1;
  pick_plan(g, sms, bn, splits);
  if (g.splits > 1 && splits != g.splits) return -7;   // a forced split count that cannot be honoured

  if (g.ab_fp8) return gemm_fp8(g, sms, bn, splits, stream);

  int err = 0;
  const CUtensorMap* ta = g.a_mn_major
                              ? rbhost::get_tmap_2d(g.a, 2, (uint64_t)g.M, (uint64_t)g.K, (uint64_t)g.lda, 64, 64, 1, &err)
                              : rbhost::get_tmap_2d(g.a, 2, (uint64_t)g.K, (uint64_t)g.M, (uint64_t)g.lda, 64, 128, 1, &err);
  if (!ta) return err ? err : -5;
  const uint64_t b_experts = g.group_mode == 1 ? (uint64_t)g.num_experts : 1;
  const CUtensorMap* tb = g.b_mn_major
                              ? rbhost::get_tmap_2d(g.b, 2, (uint64_t)g.N, (uint64_t)g.K * b_experts, (uint64_t)g.ldb, 64, 64, 1, &err)
                              : rbhost::get_tmap_2d(g.b, 2, (uint64_t)g.K, (uint64_t)g.N * b_experts, (uint64_t)g.ldb, 64, (uint32_t)bn, 1, &err);
  if (!tb) return err ? err : -5;

  if (bn == 256 && pair_takes(g)) {
    // two-CTA kernel: 256 x 256 tiles per CTA pair, each CTA loads half of the B tile
    const CUtensorMap* tb_half =
        g.b_mn_major ? tb : rbhost::get_tmap_2d(g.b, 2, (uint64_t)g.K, (uint64_t)g.N, (uint64_t)g.ldb, 64, 128, 1, &err);
    if (!tb_half) return err ? err : -5;
    const long long tiles2 = (long long)((g.M + 255) / 256) * ((g.N + 255) / 256) * (g.group_mode == 2 ? g.num_experts : splits);
    const int max_clusters = sms / 2;
    const int clusters = static_cast<int>(tiles2 < max_clusters ? tiles2 : max_clusters);
    if (!g.a_mn_major && !g.b_mn_major) return launch_pair<0, 0>(g, ta, tb_half, clusters, splits, stream);
    if (!g.a_mn_major && g.b_mn_major) return launch_pair<0, 1>(g, ta, tb_half, clusters, splits, stream);
    if (g.a_mn_major && g.b_mn_major) return launch_pair<1, 1>(g, ta, tb_half, clusters, splits, stream);
    return launch_pair<1, 0>(g, ta, tb_half, clusters, splits, stream);
  }
  long long tiles = (long long)((g.M + 127) / 128) * ((g.N + bn - 1) / bn) * splits;
  if (g.group_mode == 2) tiles *= g.num_experts;
  int grid = static_cast<int>(tiles < sms ? tiles : sms);
  if (g.max_ctas > 0 && grid > g.max_ctas) grid = g.max_ctas;
  switch (bn) {
    case 256: return dispatch_major<256, 4>(g, ta, tb, grid, splits, stream);
    case 192: return dispatch_major<192, 5>(g, ta, tb, grid, splits, stream);
    case 128: return dispatch_major<128, 5>(g, ta, tb, grid, splits, stream);
    default: return dispatch_major<64, 8>(g, ta, tb, grid, splits, stream);
  }
}

RB_API int rb_gemm_bf16(const RbGemmArgs* args, void* stream_v) {
  const RbGemmArgs& g = *args;
  if (g.col_out && g.col_rows == 0) {              // slabs that a product cannot form beside itself
    if (!g.a_mn_major || !g.b_mn_major || g.group_mode || g.peer_mode || g.ab_fp8 || !g.col_sum || g.M <= 0 || g.K <= 0) return -9;
    RbGemmArgs plain = g;
    plain.col_sum = plain.col_out = nullptr;
    const int rc = rb_sum_dim0_staged(g.a, g.lda, g.col_out, g.col_sum, g.K, g.M, 1, g.accumulate, stream_v);
    return rc != 0 ? rc : gemm_bf16(plain, reinterpret_cast<cudaStream_t>(stream_v));
  }
  const int rc = gemm_bf16(g, reinterpret_cast<cudaStream_t>(stream_v));
  return rc != 0 || !g.col_sum ? rc : rb_sum_dim0_fold(g.col_sum, (g.K + g.col_rows - 1) / g.col_rows, g.col_out, g.M, g.accumulate, stream_v);
}
