// Matrix products with few rows: D[M, N] = epilogue(alpha * X[M, K] W[N, K]^T) for M <= 96, bf16 operands, fp32 accumulation.
//
// With few rows the product is bound by reading W once, so the kernel is built to have as much of W in flight as the memory wants.
// W takes the 128-row side of tcgen05.mma and the rows of X its N side (rounded up to 16), so nothing is multiplied for padding beyond
// that; 128 rows of W form a tile, and a cluster of up to 8 CTAs shares a tile: each CTA contracts over its part of K with its own ring
// of TMA stages, leaves its partial sums in shared memory, and takes its share of the tile's results, adding the partial sums of all
// CTAs in rank order through distributed shared memory (bit-reproducible, no workspace, no second kernel).  Measured on one B200, one
// row, in a captured chain of one product on weights of their own: 28672 x 4096 41 us = 5.7 TB/s (the tile kernel: 54), 65536 x 4096 6.5
// TB/s, 2048 x 2048 5.4 us (12.0), of which launch, first load, exchange and last store are about 4.
//
// Roles: warp 0 TMA, warp 1 MMA issue and TMEM, warps 2 to 5 accumulator -> shared memory; then all warps the epilogue.
//
// NORM: the rows of X pass through a LayerNorm or RMSNorm on their way in.  For a few rows the norm is no work, only a launch of 4 us in the chain of a
// decoding step; here every CTA reads the whole rows (at most 32 KB, from L2), forms their statistics and puts its part of the normed rows, rounded
// to bf16 as the norm's own kernel does, into the operand tiles itself, while the first stages of W are on their way.  Warps 2 to 5 do that.
// A decoded token of GPT-2 small, 25 norms, with the attention step in one launch 479 -> 392 us on one B200; of 8 Llama style layers of 2048 518 -> 497.
// Lanes and order are those of the norm's kernel; sums over all 128 threads in an order of their own saved 2 % of that (328 / 320 us a token today), but gave a
// sequence other bits beside eight others than beside seven.
//
// A kernel's last barrier across the cluster only keeps shared memory alive: as a release it waited 2000 to 3000 cycles for the results' stores.  Without
// that, with the partial sums of all CTAs asked for at once and the norm's weights under the kernel in front, us per product, before / now, both in one
// chain that is not the one above (their difference counts): 1 row 768 x 3072 6.45 / 5.63, 2048 x 2048 8.1 / 7.1, 2048 x 8192 13.4 / 12.3; 64 rows
// 2048 x 8192 15.8 / 14.1.  In the one above 4.3, 5.4, 10.5 and 12.8; again and again on the same weights 4.4, 4.7, 7.8 and 10.4.
#define RB_INLINE_WAITS
#include "gemm_rows.h"

#include "norm_row.cuh"
#include "pdl.cuh"
#include "rb_common.cuh"

namespace rb {

constexpr int kRowsThreads = 192;
constexpr int kRowsTile = 128;                         // rows of W of a tile
constexpr int kRowsWBytes = kRowsTile * 128;           // one stage of W: 64 columns

constexpr int kNormRows = 8;                           // most rows that NORM takes
constexpr int kNormK = 4096;
constexpr int kNormElements = 16384;                   // most rows x K: every CTA reads them all

struct RowsNorm {
  const __nv_bfloat16* x;
  long long ldx;
  const __nv_bfloat16* gamma;
  const __nv_bfloat16* beta;                           // LayerNorm only, may be NULL
  float eps;
  int rms;
};

struct RowsEpi {
  void* d;
  long long ldd;
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  long long ldr;
  int act, out_f32;
  float alpha;
};

__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}

__device__ __forceinline__ float rows_act(int act, float v) {
  if (act == RB_ACT_GELU) return gelu_tanh_fast(v);
  if (act == RB_ACT_SILU) return silu(v);
  if (act == RB_ACT_RELU || act == RB_ACT_RELU2) {
    v = fmaxf(v, 0.f);
    return act == RB_ACT_RELU ? v : v * v;
  }
  return v;
}

// What warps 2 to 5 do first (NORM: the warps that a row belongs to): statistics of the rows, then the normed columns of k-blocks kb0 .. kb1 into the
// first stages and, for stages that are filled again, into `later`.  Lanes, order and roundings are those of the norm's own kernel, so that a row's bits
// do not hang on how many rows there are.
template <int NORM, int CHUNKS>
__device__ __forceinline__ void rows_norm(const RowsNorm& nm, int M, int K, int kb0, int kb1, int stages, int stage_bytes, uint32_t base,
                                          uint8_t* later, float* red, bool w_constant) {
  constexpr int kRows = 4 / NORM;                // at a time
  const int warp = (threadIdx.x >> 5) - 2, lane = threadIdx.x & 31, wr = warp % NORM;
  const float inv_n = 1.f / static_cast<float>(K);
  auto col = [&](int i) { return norm_col<CHUNKS, NORM>(wr, i, lane); };
  // the norm's weights are the model's like W: asked for before the kernel in front has ended
  uint4 gamma[CHUNKS], beta[CHUNKS];
  if (!w_constant) pdl_wait();
#pragma unroll
  for (int i = 0; i < CHUNKS; ++i) {
    const int c = col(i), kb = c >> 6;
    const bool mine = c < K && kb >= kb0 && kb < kb1 && warp / NORM < M;
    gamma[i] = mine ? *reinterpret_cast<const uint4*>(nm.gamma + c) : make_uint4(0u, 0u, 0u, 0u);
    beta[i] = mine && nm.beta ? *reinterpret_cast<const uint4*>(nm.beta + c) : make_uint4(0u, 0u, 0u, 0u);
  }
  pdl_wait();
  pdl_launch();
  uint4 next[CHUNKS];
  auto fetch = [&](int m) {
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int c = col(i);
      next[i] = m < M && c < K ? *reinterpret_cast<const uint4*>(nm.x + m * nm.ldx + c) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
  auto unpack = [](const uint4& a, float (&v)[8]) {
    const float2 f0 = unpack_bf16x2(a.x), f1 = unpack_bf16x2(a.y), f2 = unpack_bf16x2(a.z), f3 = unpack_bf16x2(a.w);
    v[0] = f0.x; v[1] = f0.y; v[2] = f1.x; v[3] = f1.y; v[4] = f2.x; v[5] = f2.y; v[6] = f3.x; v[7] = f3.y;
  };
  // `at`: 4 floats per row and use
  auto row_sum = [&](float v, float* at) {
    v = warp_sum(v);
    if (NORM == 1) return v;
    if (lane == 0) at[wr] = v;
    asm volatile("bar.sync 1, 128;" ::: "memory");
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < NORM; ++i) s += at[i];
    return s;
  };
  fetch(warp / NORM);
#pragma unroll 1
  for (int m0 = 0; m0 < M; m0 += kRows) {
    const int m = m0 + warp / NORM;              // M or more: nothing is read or written, the barriers are kept
    if (NORM == 1 && m >= M) break;              // (there are none)
    uint4 u[CHUNKS];
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) u[i] = next[i];
    fetch(m + kRows);
    float mean = 0.f;
    if (!nm.rms) {
      float s = 0.f;
#pragma unroll
      for (int i = 0; i < CHUNKS; ++i) {
        float v[8];
        unpack(u[i], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) s += v[j];
      }
      mean = norm_mean(row_sum(s, red + m * 8), inv_n);
    }
    float sq = 0.f;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      if (col(i) < K) {
        float v[8];
        unpack(u[i], v);
#pragma unroll
        for (int j = 0; j < 8; ++j) sq = norm_square(v[j], mean, sq);
      }
    }
    const float rstd = norm_rstd(row_sum(sq, red + m * 8 + 4), inv_n, nm.eps);
    if (m >= M) continue;
#pragma unroll
    for (int i = 0; i < CHUNKS; ++i) {
      const int c = col(i), kb = c >> 6;
      if (kb >= kb0 && kb < kb1) {               // the last block's columns behind the row are zero
        float v[8] = {}, g[8], b[8];
        if (c < K) {
          unpack(u[i], v);
          unpack(gamma[i], g);
          unpack(beta[i], b);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = norm_value(v[j], mean, rstd, g[j], b[j]);     // without beta + 0: the same number
        }
        const uint4 o = make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
        const int it = kb - kb0, chunk = (c & 63) >> 3;
        if (it < stages)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};"
                       ::"r"(base + it * stage_bytes + kRowsWBytes + m * 128 + ((chunk ^ (m & 7)) << 4)), "r"(o.x), "r"(o.y), "r"(o.z), "r"(o.w)
                       : "memory");
        else
          *reinterpret_cast<uint4*>(later + (((it - stages) * M + m) * 8 + chunk) * 16) = o;
      }
    }
  }
  fence_proxy_async_smem();
  asm volatile("bar.sync 1, 128;" ::: "memory");
}

// NORM: 0, or the warps that share a row of the norm (1, 2, 4: K up to 1024, 2048, 4096), CHUNKS: the norm's 16-byte pieces per lane
template <int NORM, int CHUNKS = 4>
__global__ void __launch_bounds__(kRowsThreads)
gemm_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, int M, int N, int K, int mpad,
                 int parts, int stages, int w_constant, const RowsEpi ep, const RowsNorm nm, unsigned int* status) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const uint32_t base = smem_u32(smem);
  const uint32_t stage_bytes = kRowsWBytes + mpad * 128;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + stages * stage_bytes);
  const uint32_t bar_full = smem_u32(bars), bar_empty = bar_full + 8 * stages, bar_acc = bar_empty + 8 * stages;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(bars + 2 * stages + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr + 1);
  float* red = reinterpret_cast<float*>(tmem_ptr + 4);                          // NORM: [kNormRows][2][4], then the rows of later stages
  uint8_t* later = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(red + kNormRows * 8) + 15) & ~uintptr_t(15));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tile = blockIdx.x / parts, part = blockIdx.x - tile * parts;
  const uint32_t tmem_cols = mpad <= 32 ? 32 : mpad <= 64 ? 64 : 128;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2 * stages + 1; ++s) mbar_init(bar_full + 8 * s, NORM != 0 && s < stages ? 2 : 1);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(tmem_ptr), tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_ptr;
  // swiglu: a tile is 64 gate rows and the 64 up rows of the same columns
  const bool glu = ep.act == RB_ACT_SWIGLU;
  const int tile_n = glu ? kRowsTile / 2 : kRowsTile;
  const int num_kb = (K + 63) / 64;
  const int kb0 = static_cast<int>(static_cast<long long>(num_kb) * part / parts);
  const int kb1 = static_cast<int>(static_cast<long long>(num_kb) * (part + 1) / parts);

  if (warp == 0) {
    if (elect_one()) {
      // W of the first stages is on its way before the kernel in front has ended, X follows when it has
      auto load_w = [&](int it, int s) {
        const uint32_t dst = base + s * stage_bytes;
        tma_load_2d(dst, &tmW, (kb0 + it) * 64, tile * tile_n, bar_full + 8 * s);
        if (glu) tma_load_2d(dst + kRowsWBytes / 2, &tmW, (kb0 + it) * 64, N + tile * tile_n, bar_full + 8 * s);
      };
      const int ahead = w_constant ? min(stages, kb1 - kb0) : 0;
      const uint32_t loaded = NORM ? kRowsWBytes : stage_bytes;
      for (int it = 0; it < ahead; ++it) {
        mbar_arrive_expect_tx(bar_full + 8 * it, loaded);
        load_w(it, it);
      }
      pdl_wait();
      for (int it = 0; it < kb1 - kb0; ++it) {
        const int s = it % stages;
        if (it >= ahead) {
          if (!mbar_wait(bar_empty + 8 * s, ((it / stages) & 1) ^ 1, abort_flag, status, 81)) break;
          mbar_arrive_expect_tx(bar_full + 8 * s, loaded);
          load_w(it, s);
        }
        if (!NORM) tma_load_2d(base + s * stage_bytes + kRowsWBytes, &tmX, (kb0 + it) * 64, 0, bar_full + 8 * s);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = umma_idesc_bf16(kRowsTile, mpad, 0, 0);
      bool ok = true;
      for (int kb = kb0; kb < kb1; ++kb) {
        const int it = kb - kb0, s = it % stages;
        if (!mbar_wait(bar_full + 8 * s, (it / stages) & 1, abort_flag, status, 82)) { ok = false; break; }
        tc_fence_after();
        uint64_t dw = umma_smem_desc_sw128(base + s * stage_bytes, 16, 1024);
        uint64_t dx = umma_smem_desc_sw128(base + s * stage_bytes + kRowsWBytes, 16, 1024);
#pragma unroll
        for (int k = 0; k < 4; ++k) umma_bf16_ss(tmem, dw + 2 * k, dx + 2 * k, idesc, (it | k) != 0 ? 1u : 0u);
        umma_commit(bar_empty + 8 * s);
      }
      if (ok) umma_commit(bar_acc);
    }
  } else {
    if constexpr (NORM == 0) {
      pdl_wait();
      pdl_launch();
    } else {
      rows_norm<NORM, CHUNKS>(nm, M, K, kb0, kb1, stages, stage_bytes, base, later, red, w_constant);
      if (warp == 2) {
        if (lane < min(stages, kb1 - kb0)) mbar_arrive(bar_full + 8 * lane);
        for (int it = stages; it < kb1 - kb0; ++it) {
          const int s = it % stages;
          if (!mbar_wait(bar_empty + 8 * s, ((it / stages) & 1) ^ 1, abort_flag, status, 84)) break;
          for (int i = lane; i < M * 8; i += 32) {
            const int m = i >> 3, chunk = i & 7;
            *reinterpret_cast<uint4*>(smem + s * stage_bytes + kRowsWBytes + m * 128 + ((chunk ^ (m & 7)) << 4)) =
                *reinterpret_cast<const uint4*>(later + ((it - stages) * M * 8 + i) * 16);
          }
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_full + 8 * s);
        }
      }
    }
    // Every load of the ring has been consumed when the accumulator is complete: its memory takes the partial sums [M][128].
    if (mbar_wait(bar_acc, 0, abort_flag, status, 83)) {
      tc_fence_after();
      const int q = warp & 3;                            // the quarter of the TMEM lanes that this warp may read
      float* dst = reinterpret_cast<float*>(smem) + q * 32 + lane;
      for (int c = 0; c < mpad; c += 16) {
        uint32_t r[16];
        tmem_ld_32x16(tmem + (static_cast<uint32_t>(q * 32) << 16) + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j)
          if (c + j < M) dst[(c + j) * kRowsTile] = __uint_as_float(r[j]);
      }
      tc_fence_before();
    }
  }
  __syncwarp();
  if (warp < 2) pdl_wait();
  if (parts > 1) cluster_sync_all();
  else __syncthreads();

  // ---- results: four neighbouring columns per item, items dealt to the CTAs of the cluster
  if (!*abort_flag) {
    const int shift = glu ? 4 : 5;                       // of 16 or 32 items in a row
    for (int i = part * kRowsThreads + threadIdx.x; i < M << shift; i += parts * kRowsThreads) {
      const int m = i >> shift, n = (i - (m << shift)) * 4, col = tile * tile_n + n;
      if (col >= N) continue;
      auto sum = [&](int at) {
        if (parts == 1) return *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(smem) + at);
        float4 v[8];                                     // all parts are asked for, then added in rank order
#pragma unroll
        for (int s = 0; s < 8; ++s) v[s] = s < parts ? ld_cluster_f4(mapa_shared(base + at * 4, s)) : make_float4(0.f, 0.f, 0.f, 0.f);
        float4 a = v[0];
#pragma unroll
        for (int s = 1; s < 8; ++s) {
          if (s < parts) { a.x += v[s].x; a.y += v[s].y; a.z += v[s].z; a.w += v[s].w; }
        }
        return a;
      };
      float4 a = sum(m * kRowsTile + n);
      if (glu) {
        const float4 b = sum(m * kRowsTile + tile_n + n);
        a.x = silu(a.x) * b.x; a.y = silu(a.y) * b.y; a.z = silu(a.z) * b.z; a.w = silu(a.w) * b.w;
      }
      float v[4] = {a.x * ep.alpha, a.y * ep.alpha, a.z * ep.alpha, a.w * ep.alpha};
      const bool full = col + 4 <= N;
      if (ep.bias) {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (full || col + j < N) v[j] += __bfloat162float(__ldg(ep.bias + col + j));
      }
      if (ep.act != RB_ACT_NONE && !glu) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] = rows_act(ep.act, v[j]);
      }
      if (ep.residual) {
        const __nv_bfloat16* r = ep.residual + m * ep.ldr + col;
        if (full) {
          const uint2 u = *reinterpret_cast<const uint2*>(r);
          const float2 r0 = unpack_bf16x2(u.x), r1 = unpack_bf16x2(u.y);
          v[0] += r0.x; v[1] += r0.y; v[2] += r1.x; v[3] += r1.y;
        } else {
          for (int j = 0; col + j < N; ++j) v[j] += __bfloat162float(r[j]);
        }
      }
      if (ep.out_f32) {
        float* d = reinterpret_cast<float*>(ep.d) + m * ep.ldd + col;
        if (full) *reinterpret_cast<float4*>(d) = make_float4(v[0], v[1], v[2], v[3]);
        else for (int j = 0; col + j < N; ++j) d[j] = v[j];
      } else {
        __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(ep.d) + m * ep.ldd + col;
        if (full) *reinterpret_cast<uint2*>(d) = make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
        else for (int j = 0; col + j < N; ++j) d[j] = __float2bfloat16(v[j]);
      }
    }
  }
  if (parts > 1) cluster_sync_relaxed();                 // nobody leaves while another CTA still reads its partial sums
  else __syncthreads();
  if (warp == 1) {
    if (*abort_flag) {
      // give copies and MMAs that are still in flight time to land before TMEM is released
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem, tmem_cols);
  }
}

}  // namespace rb

namespace rbhost {

// Up to 96 rows this kernel is the faster one (us per product in a captured chain, tile kernel / this one; 1 row: 768 x 768 8.1 / 3.7,
// 2048 x 2048 12.0 / 5.4, 28672 x 4096 54.0 / 41.3; 96 rows: 8.7 / 6.3, 12.2 / 9.4, 48.1 / 48.9, 65536 x 4096 126 / 100).  With 128 rows the two
// cross (2048 x 8192 16.3 / 17.1).  From 49 rows on a short contraction under many tiles is all results and little reading: 50304 x 768
// with 64 rows 20.8 / 24.8, with 24 rows 21.5 / 20.0.
bool gemm_rows_takes(const RbGemmArgs& g) {
  if (g.M > 96 || (g.M > 48 && g.K < 1024 && g.N > 148 * rb::kRowsTile / (g.act == RB_ACT_SWIGLU ? 2 : 1))) return false;
  return !g.a_mn_major && !g.b_mn_major && !g.accumulate && !g.aux_out && !g.aux_in && g.group_mode == 0 && g.peer_mode == 0 && !g.ab_fp8 &&
         !g.a_scale && !g.b_scale && g.block_n == 0 && g.group_m == 0 && g.max_ctas == 0 && g.splits <= 1;
}

bool gemm_rows_norm_takes(const RbGemmArgs& g) {
  return g.M <= rb::kNormRows && g.K <= rb::kNormK && g.M * g.K <= rb::kNormElements && g.K % 8 == 0 && g.norm_gamma &&
         !(g.norm_rms && g.norm_beta);
}

int gemm_rows(const RbGemmArgs& g, cudaStream_t stream) {
  const bool norm = g.norm_gamma != nullptr;
  const int mpad = (g.M + 15) / 16 * 16;
  const bool glu = g.act == RB_ACT_SWIGLU;
  const int tile_n = glu ? rb::kRowsTile / 2 : rb::kRowsTile;
  const int tiles = (g.N + tile_n - 1) / tile_n, num_kb = (g.K + 63) / 64;
  // About 100 CTAs or more read at the memory's rate; each further part of K costs another CTA's partial sums.  One row, us per product
  // in a captured chain with 1 / 2 / 4 / 8 parts: 768 x 768 5.7 / 4.6 / 4.0 / 3.9, 2048 x 8192 36.9 / 20.6 / 12.5 / 9.6, 16384 x 2048
  // 14.1 / 14.2 / 17.9 / 25.0.
  int parts = 1;
  while (parts < 8 && tiles * parts < 100 && num_kb / (parts + 1) >= 2) ++parts;
  // The ring is kept below half of an SM's shared memory: with one CTA per SM, clusters of 8 no longer all fit side by side (2048 x 2048,
  // 64 rows, 8 parts: 8.1 us with 4 stages, 13.7 with 6).
  const int stage_bytes = rb::kRowsWBytes + mpad * 128;
  int stages = (111 * 1024) / stage_bytes < 6 ? (111 * 1024) / stage_bytes : 6;
  int later = 0;
  if (norm) {
    const int most = (num_kb + parts - 1) / parts;         // k-blocks of a part
    auto kept = [&](int st) { return most > st ? (most - st) * g.M * 128 : 0; };
    while (stages > 1 && stages * stage_bytes + kept(stages) > 111 * 1024) --stages;
    later = kept(stages) + rb::kNormRows * 32 + 32;
  }
  int err = 0;
  const CUtensorMap* tw = get_tmap_2d(g.b, 2, (uint64_t)g.K, (uint64_t)g.N * (glu ? 2 : 1), (uint64_t)g.ldb, 64, (uint32_t)tile_n, 1, &err);
  if (!tw) return err ? err : -5;
  const CUtensorMap* tx = norm ? tw : get_tmap_2d(g.a, 2, (uint64_t)g.K, (uint64_t)g.M, (uint64_t)g.lda, 64, (uint32_t)mpad, 1, &err);
  if (!tx) return err ? err : -5;
  const int smem = stages * stage_bytes + (2 * stages + 1) * 8 + 16 + 1024 + later;
  // the norm's own kernel takes rows of up to 768 in three pieces a lane
  const int form = !norm ? 0 : g.K <= 768 ? 1 : g.K <= 1024 ? 2 : g.K <= 2048 ? 3 : 4;
  auto kern = form == 0   ? rb::gemm_rows_kernel<0>
              : form == 1 ? rb::gemm_rows_kernel<1, 3>
              : form == 2 ? rb::gemm_rows_kernel<1>
              : form == 3 ? rb::gemm_rows_kernel<2>
                          : rb::gemm_rows_kernel<4>;
  static bool configured_dev[5][64] = {{false}};
  bool& configured = configured_dev[form][device_slot()];
  if (!configured) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 114 * 1024);
    if (e != cudaSuccess) return static_cast<int>(e);
    configured = true;
  }
  rb::RowsEpi ep;
  ep.d = g.d; ep.ldd = g.ldd;
  ep.bias = reinterpret_cast<const __nv_bfloat16*>(g.bias);
  ep.residual = reinterpret_cast<const __nv_bfloat16*>(g.residual); ep.ldr = g.ldr;
  ep.act = g.act; ep.out_f32 = g.out_f32; ep.alpha = g.alpha;
  const rb::RowsNorm nm{reinterpret_cast<const __nv_bfloat16*>(g.a), g.lda, reinterpret_cast<const __nv_bfloat16*>(g.norm_gamma),
                        reinterpret_cast<const __nv_bfloat16*>(g.norm_beta), g.norm_eps, g.norm_rms};
  return static_cast<int>(launch_pdl(kern, dim3(tiles * parts), dim3(rb::kRowsThreads), smem, stream, parts, *tw, *tx,
                                     g.M, g.N, g.K, mpad, parts, stages, g.b_constant, ep, nm, status_ptr()));
}

}  // namespace rbhost
