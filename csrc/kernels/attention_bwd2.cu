// Flash attention backward on the 5th-generation tensor cores, second version: P and dS never touch shared memory.
//
// Two kernels from one template, no atomics, bit-reproducible:
//
//   MODE_DQ   a CTA owns 128 queries of one (batch, head) (Q, dO resident in shared memory) and walks over the key
//             tiles they see.  Per step
//                 S  = Q K^T,  dP = dO V^T          tcgen05.mma (SS), accumulators in TMEM (dP double buffered)
//                 dS = exp2(S c - lse) (dP - delta) sixteen warps, query row = TMEM lane; dS goes back to TMEM as packed
//                                                   bf16 over the dP buffer
//                 dQ += dS K                        tcgen05.mma, A operand dS read from TMEM (TS form), K MN-major
//   MODE_DKV  a CTA owns 128 keys of one (batch, kv head) (K, V resident) and walks over the query tiles that see them
//             (all query heads of the group).  The products are formed TRANSPOSED, so that the key is the TMEM lane:
//                 S^T = K Q^T,  dP^T = V dO^T
//                 P^T -> TMEM over S^T,  dV += P^T dO      (TS form, dO MN-major)
//                 dS^T -> TMEM over dP^T, dK += dS^T Q     (TS form, Q MN-major)
//             The log-sum-exp and delta of the step's 128 queries vary along a thread's row here; a warp of their own puts
//             them into shared memory up to two steps ahead, they are read as broadcasts.  With head dim 64 S^T is double buffered.
//
// A step's 128 columns are two halves of 64.  Each has scores, barriers and eight compute warps of its own, and the issuer serves them in
// turn, so the halves run about half a step apart: one is in its exponentials (128 x 128 of them take the special-function units 1024 cycles)
// while the other stores, waits or multiplies.  Because every product that overwrites a TMEM buffer is issued by the one MMA thread after the
// product that last read it, and tcgen05.mma instructions of one thread execute in issue order, no "buffer free" handshake is needed for the
// aliased P / dS operands; the only waits are "operand tile landed", "scores ready", "probabilities written".  The two streamed operands have
// rings of their own, since they are given back at different times: with pairs in two stages (head dim 128) the next pair's way from L2
// was part of every step.  Results leave through the resident operands' memory and TMA: rows of a packed gradient are 3 KB and more apart, and
// stores of 16 bytes per lane took 4200 cycles of an item, two steps' time.
// Measured on one B200, both passes and delta, us, one half, pairs in stages and 16-byte stores / now: 32 x 1024, 12 heads of 64 474 / 353; 4 x 4096,
// 32 (8 KV) heads of 128 2230 / 1883; 2 x 2048, 16 (4) heads of 128 245 / 208.
// Roles: warps 0-15 compute (lane quarter = warp & 3, 32 of the step's 128 columns: warp >> 2), warp 16 TMA producer, warp 17 MMA issuer, warp 18
// statistics.  CTAs are persistent and walk over work items; every wait is bounded.
//
// Same semantics as the other backward kernels (causal alignment to the end of the keys, GQA); replaces the
// reference's dense attention gradient (crates/autodiff/src/lib.rs:645-806 applied to crates/nn/src/attention.rs:640-836).
#include "attention.h"

#include "pairs.cuh"
#include "pdl.cuh"
#include "rb_common.cuh"

namespace rb {

constexpr int kB2Tile = 128;
constexpr int kB2ComputeWarps = 16;
constexpr int kB2Cols = 512 / kB2ComputeWarps;             // columns of a step's 128 that a compute thread takes
constexpr float kB2Log2e = 1.4426950408889634f;
constexpr int B2_DKV = 0;
constexpr int B2_DQ = 1;

struct B2Params {
  const float* lse;
  const float* delta;
  int seq_q, seq_k, heads, kv_heads, causal, batch;
  float scale;
  const int* kv_lens;       // optional [batch]: number of real keys (the rest of seq_k is padding)
};

__device__ __forceinline__ float b2_ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int D, int MODE>
struct B2Smem {
  static constexpr int kThreads = 32 * (kB2ComputeWarps + (MODE == B2_DKV ? 3 : 2));
  static constexpr int kHalf = kB2Tile * 128;                  // 128 rows x 128 B: one 64-column swizzle atom
  static constexpr int kTileBytes = (D / 64) * kHalf;          // one [128, D] operand tile
  static constexpr int kResStages = D == 64 ? 2 : 1;           // owned pair of the next work item prefetched
  static constexpr int kStagesA = D == 64 ? 4 : 3;             // streamed tiles in flight: B2_DKV Q, B2_DQ K
  static constexpr int kStagesB = D == 64 ? 3 : 2;             //                           B2_DKV dO, B2_DQ V
  static constexpr int kRes = 0;
  static constexpr int kRingA = kResStages * 2 * kTileBytes;
  static constexpr int kRingB = kRingA + kStagesA * kTileBytes;
  static constexpr int kStats = kRingB + kStagesB * kTileBytes;         // B2_DKV: [2 steps][lse2 | delta][128] fp32
  static constexpr int kBar = kStats + (MODE == B2_DKV ? 2 * 2 * 128 * 4 : 0);
  // + s_full[2 halves][2], s_empty[2], dp_full[2][2], p_full[2][2], ds_full[2][2], acc_full, acc_empty, stat[2],
  // staged[4]
  static constexpr int kNumBars = 2 * kResStages + 2 * kStagesA + 2 * kStagesB + 26;
  static constexpr int kTotal = kBar + kNumBars * 8 + 16;
  static_assert(kTotal <= 232448, "shared memory of an SM");
  // TMEM columns
  static constexpr int kSBufs = (MODE == B2_DKV && D == 64) ? 2 : 1;    // S (S^T) buffers
  static constexpr int kDpBufs = MODE == B2_DQ ? 2 : 1;                 // dP buffers
  static constexpr int kColS = 0;
  static constexpr int kColDp = kColS + 128 * kSBufs;
  static constexpr int kColAcc0 = kColDp + 128 * kDpBufs;
  static constexpr int kColAcc1 = kColAcc0 + D;
  static_assert(kColAcc0 + (MODE == B2_DKV ? 2 : 1) * D <= 512, "TMEM budget");
};

template <int D, int MODE>
__global__ void __launch_bounds__(B2Smem<D, MODE>::kThreads, 1)
attn_bwd2_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmdO,
                 const __grid_constant__ CUtensorMap tmOut0, const __grid_constant__ CUtensorMap tmOut1, B2Params p,
                 unsigned int* status) {
  pdl_wait();
  pdl_launch();
  using L = B2Smem<D, MODE>;
  constexpr int SA = L::kStagesA, SR = L::kStagesB, RS = L::kResStages, SB = L::kSBufs, DB = L::kDpBufs;
  extern __shared__ __align__(1024) uint8_t smem[];      // swizzle atoms need the alignment; nothing lies in front
  const uint32_t sbase = smem_u32(smem);
  if (sbase & 1023) {
    if (threadIdx.x == 0) status_set(status, kStatusBadArg, 75);
    return;
  }
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + L::kBar);
  const uint32_t b0 = smem_u32(bars);
  const uint32_t bar_res = b0, bar_res_empty = bar_res + 8 * RS, bar_afull = bar_res_empty + 8 * RS, bar_aempty = bar_afull + 8 * SA,
                 bar_bfull = bar_aempty + 8 * SA, bar_bempty = bar_bfull + 8 * SR;
  // [half][2]
  const uint32_t bar_sfull = bar_bempty + 8 * SR, bar_sempty = bar_sfull + 32 /* [half] */, bar_dpfull = bar_sempty + 16,
                 bar_pfull = bar_dpfull + 32, bar_dsfull = bar_pfull + 32, bar_accfull = bar_dsfull + 32, bar_accempty = bar_accfull + 8,
                 bar_stat = bar_accempty + 8 /* [2] */, bar_staged = bar_stat + 16 /* [lane quarter] */;
  static_assert(2 * RS + 2 * SA + 2 * SR + 26 == L::kNumBars, "barrier count");
  uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(bars + L::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_ptr_smem + 1);
  float* stats = reinterpret_cast<float*>(smem + L::kStats);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int group = p.heads / p.kv_heads;
  const int shift = p.seq_k - p.seq_q;
  const int n_q_tiles = (p.seq_q + kB2Tile - 1) / kB2Tile;
  const int n_k_tiles = (p.seq_k + kB2Tile - 1) / kB2Tile;

  // Work items: one owned tile of one (head, batch); a CTA takes items blockIdx.x, + gridDim.x, ...  Long walks first.
  struct Work { int own0, walk_first, walk_count, n_it, head_q0, head_k, b, kv_len; };
  const int n_own = MODE == B2_DKV ? n_k_tiles : n_q_tiles;
  const int ny = MODE == B2_DKV ? p.kv_heads : p.heads;
  const int total_items = n_own * ny * p.batch;
  auto get_work = [&](int item, Work& w) {
    const int per_tile = ny * p.batch;
    const int tw = item / per_tile;
    const int yz = item - tw * per_tile;
    const int y = yz % ny;
    w.b = yz / ny;
    const int blk = (MODE == B2_DKV || !p.causal) ? tw : n_own - 1 - tw;
    w.own0 = blk * kB2Tile;
    w.walk_first = 0;
    // padded keys (positions >= kv_len) are invisible: their dK / dV are zero and no query walks over them
    w.kv_len = p.kv_lens ? max(0, min(p.seq_k, p.kv_lens[w.b])) : p.seq_k;
    if (MODE == B2_DKV) {
      w.head_k = y;
      w.head_q0 = y * group;
      if (p.causal && w.own0 - shift > 0) w.walk_first = (w.own0 - shift) / kB2Tile;
      w.walk_count = n_q_tiles - w.walk_first;
      if (w.walk_count < 0 || w.own0 >= w.kv_len) w.walk_count = 0;
      w.n_it = w.walk_count * group;
    } else {
      w.head_q0 = y;
      w.head_k = y / group;
      w.walk_count = (w.kv_len + kB2Tile - 1) / kB2Tile;
      if (p.causal) {
        const int lim = (w.own0 + kB2Tile - 1 + shift) / kB2Tile + 1;
        if (lim < w.walk_count) w.walk_count = lim;
      }
      w.n_it = w.walk_count;
    }
  };
  auto walk_decode = [&](const Work& w, int it, int& hq, int& q0, int& k0) {
    if (MODE == B2_DKV) {
      const int g = it / w.walk_count;
      hq = w.head_q0 + g;
      q0 = (w.walk_first + it - g * w.walk_count) * kB2Tile;
      k0 = w.own0;
    } else {
      hq = w.head_q0;
      q0 = w.own0;
      k0 = it * kB2Tile;
    }
  };

  if (threadIdx.x == 0) {
    for (int s = 0; s < RS; ++s) { mbar_init(bar_res + 8 * s, 1); mbar_init(bar_res_empty + 8 * s, 4); }
    for (int s = 0; s < SA; ++s) { mbar_init(bar_afull + 8 * s, 1); mbar_init(bar_aempty + 8 * s, 1); }
    for (int s = 0; s < SR; ++s) { mbar_init(bar_bfull + 8 * s, 1); mbar_init(bar_bempty + 8 * s, 1); }
    for (int s = 0; s < 4; ++s) { mbar_init(bar_sfull + 8 * s, 1); mbar_init(bar_dpfull + 8 * s, 1); }
    for (int h = 0; h < 2; ++h) mbar_init(bar_sempty + 8 * h, kB2ComputeWarps / 2);
    // P-ready and dS-ready barriers alternate between two by step: the compute warps can finish step g + 1 (whose
    // scores were issued ahead) before the issuer has looked at step g, and a single barrier would then be two phases
    // ahead of the parity the issuer waits for.  Step g + 2 cannot complete before the issuer has passed step g.
    for (int h = 0; h < 4; ++h) {
      mbar_init(bar_pfull + 8 * h, kB2ComputeWarps / 2);
      mbar_init(bar_dsfull + 8 * h, kB2ComputeWarps / 2);
    }
    for (int h = 0; h < 2; ++h) mbar_init(bar_stat + 8 * h, 1);
    for (int q = 0; q < 4; ++q) mbar_init(bar_staged + 8 * q, kB2ComputeWarps / 4);
    mbar_init(bar_accfull, 1);
    mbar_init(bar_accempty, kB2ComputeWarps);
    *abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmQ);
    tma_prefetch_desc(&tmK);
    tma_prefetch_desc(&tmV);
    tma_prefetch_desc(&tmdO);
  }
  if (warp == kB2ComputeWarps + 1) {
    tmem_alloc(smem_u32(tmem_ptr_smem), 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_ptr_smem;
  const uint32_t sRes = sbase + L::kRes, sRingA = sbase + L::kRingA, sRingB = sbase + L::kRingB;

  if (warp == kB2ComputeWarps) {
    if (elect_one()) {
      // ---------------------------------------------------------------- TMA producer
      uint32_t g = 0, wi = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x, ++wi) {
        Work w;
        get_work(item, w);
        const uint32_t rsl = wi % RS;
        if (!mbar_wait(bar_res_empty + 8 * rsl, ((wi / RS) & 1) ^ 1, abort_flag, status, 60)) break;
        const uint32_t rfull = bar_res + 8 * rsl;
        const uint32_t r0 = sRes + rsl * 2 * L::kTileBytes, r1 = r0 + L::kTileBytes;
        mbar_arrive_expect_tx(rfull, 2 * L::kTileBytes);
#pragma unroll
        for (int hf = 0; hf < D / 64; ++hf) {
          if (MODE == B2_DKV) {
            tma_load_4d(r0 + hf * L::kHalf, &tmK, hf * 64, w.head_k, w.own0, w.b, rfull);
            tma_load_4d(r1 + hf * L::kHalf, &tmV, hf * 64, w.head_k, w.own0, w.b, rfull);
          } else {
            tma_load_4d(r0 + hf * L::kHalf, &tmQ, hf * 64, w.head_q0, w.own0, w.b, rfull);
            tma_load_4d(r1 + hf * L::kHalf, &tmdO, hf * 64, w.head_q0, w.own0, w.b, rfull);
          }
        }
        for (int it = 0; it < w.n_it; ++it, ++g) {
          int hq, q0, k0;
          walk_decode(w, it, hq, q0, k0);
          const int head = MODE == B2_DKV ? hq : w.head_k, row = MODE == B2_DKV ? q0 : k0;
          const uint32_t sa = g % SA, sb = g % SR;
          if (!mbar_wait(bar_aempty + 8 * sa, ((g / SA) & 1) ^ 1, abort_flag, status, 61)) { ok = false; break; }
          mbar_arrive_expect_tx(bar_afull + 8 * sa, L::kTileBytes);
#pragma unroll
          for (int hf = 0; hf < D / 64; ++hf)
            tma_load_4d(sRingA + sa * L::kTileBytes + hf * L::kHalf, MODE == B2_DKV ? &tmQ : &tmK, hf * 64, head, row, w.b, bar_afull + 8 * sa);
          if (!mbar_wait(bar_bempty + 8 * sb, ((g / SR) & 1) ^ 1, abort_flag, status, 76)) { ok = false; break; }
          mbar_arrive_expect_tx(bar_bfull + 8 * sb, L::kTileBytes);
#pragma unroll
          for (int hf = 0; hf < D / 64; ++hf)
            tma_load_4d(sRingB + sb * L::kTileBytes + hf * L::kHalf, MODE == B2_DKV ? &tmdO : &tmV, hf * 64, head, row, w.b, bar_bfull + 8 * sb);
        }
      }
    }
  } else if (warp == kB2ComputeWarps + 1) {
    // elect.sync, not lane 0: the compiler then knows that one lane runs this and keeps descriptors in uniform registers.  Both passes, one
    // B200, us behind `lane == 0` / elect.sync: 4 x 4096, 32 (8 KV) heads of 128 2519 / 2230, 32 x 1024, 12 heads of 64 490 / 474
    if (elect_one()) {
      // ---------------------------------------------------------------- MMA issuer
      constexpr uint32_t idesc_s = umma_idesc_bf16(128, 64, 0, 0);
      constexpr uint32_t idesc_acc = umma_idesc_bf16(128, D, 0, 1);    // A from TMEM (K-major), B MN-major
      uint32_t res_off = 0;
      auto tile_a = [&](uint32_t g) { return sRingA + (g % SA) * L::kTileBytes; };
      auto tile_b = [&](uint32_t g) { return sRingB + (g % SR) * L::kTileBytes; };
      auto wait_a = [&](uint32_t g) { return mbar_wait(bar_afull + 8 * (g % SA), (g / SA) & 1, abort_flag, status, 63); };
      auto wait_b = [&](uint32_t g) { return mbar_wait(bar_bfull + 8 * (g % SR), (g / SR) & 1, abort_flag, status, 66); };
      // half h of S (S^T) and dP (dP^T) of step g: A the resident [128, D] tile, B 64 rows of the streamed one, both K-major
      auto scores = [&](uint32_t dst, uint32_t a, uint32_t bt, uint32_t bar) {
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t off = (ks >> 2) * L::kHalf + (ks & 3) * 32;
          umma_bf16_ss(dst, umma_smem_desc_sw128(a + off, 16, 1024), umma_smem_desc_sw128(bt + off, 16, 1024), idesc_s, ks != 0 ? 1u : 0u);
        }
        umma_commit(bar);
      };
      auto issue_s = [&](uint32_t g, int h) {
        const uint32_t buf = SB == 2 ? (g & 1) : 0;
        scores(tmem_base + L::kColS + buf * 128 + h * 64, sRes + res_off, tile_a(g) + h * 8192, bar_sfull + 16 * h + 8 * buf);
      };
      auto issue_dp = [&](uint32_t g, int h) {
        const uint32_t buf = DB == 2 ? (g & 1) : 0;
        scores(tmem_base + L::kColDp + buf * 128 + h * 64, sRes + res_off + L::kTileBytes, tile_b(g) + h * 8192, bar_dpfull + 16 * h + 8 * buf);
      };
      // acc += A[TMEM, half h, packed bf16: each part of 32 keys / queries at the beginning of its 32 columns] * B[smem tile, MN-major]
      auto issue_acc = [&](uint32_t acc_col, uint32_t a_col, uint32_t b_tile, int h, bool first) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) {
          const uint32_t a_addr = tmem_base + a_col + h * 64 + (ks >> 1) * kB2Cols + (ks & 1) * 8;
          umma_bf16_ts(tmem_base + acc_col, a_addr, umma_smem_desc_sw128(b_tile + (h * 4 + ks) * 2048, L::kHalf, 1024), idesc_acc,
                       (!first || h != 0 || ks != 0) ? 1u : 0u);
        }
      };
      uint32_t g = 0, wi = 0, ai = 0;
      bool ok = true;
      for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x, ++wi) {
        Work w;
        get_work(item, w);
        const uint32_t rsl = wi % RS;
        res_off = rsl * 2 * L::kTileBytes;
        if (!mbar_wait(bar_res + 8 * rsl, (wi / RS) & 1, abort_flag, status, 62)) break;
        if (w.n_it > 0) {
          if (!wait_a(g) || !wait_b(g)) break;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            // B2_DQ: the S buffer is free once the compute warps have loaded the previous step's scores.  (B2_DKV: its last
            // reader is the dV product of an earlier step, issued before this point.)
            if (MODE == B2_DQ && g > 0 && !mbar_wait(bar_sempty + 8 * h, (g - 1) & 1, abort_flag, status, 64)) { ok = false; break; }
            tc_fence_after();
            issue_s(g, h);
            issue_dp(g, h);       // dP buffer of step g: its last reader (step g - DB) was issued long before
          }
          if (!ok) break;
          if (MODE == B2_DQ) umma_commit(bar_bempty + 8 * (g % SR));
          // the compute warps have read out the previous item's accumulators
          if (!mbar_wait(bar_accempty, (ai & 1) ^ 1, abort_flag, status, 65)) break;
          tc_fence_after();
        }
        for (int it = 0; it < w.n_it && ok; ++it, ++g) {
          const bool more = it + 1 < w.n_it;
          if (MODE == B2_DQ) {
            if (more && (!wait_a(g + 1) || !wait_b(g + 1))) { ok = false; break; }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (more) {
                if (!mbar_wait(bar_sempty + 8 * h, g & 1, abort_flag, status, 67)) { ok = false; break; }
                tc_fence_after();
                issue_s(g + 1, h);
                issue_dp(g + 1, h);                              // the other dP buffer: read last by dQ(g - 1), issued
                if (h == 1) umma_commit(bar_bempty + 8 * ((g + 1) % SR));
              }
              if (!mbar_wait(bar_dsfull + 16 * h + 8 * (g & 1), (g >> 1) & 1, abort_flag, status, 68)) { ok = false; break; }
              tc_fence_after();
              issue_acc(L::kColAcc0, L::kColDp + (g & 1) * 128, tile_a(g), h, it == 0);          // dQ += dS K
            }
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              if (more && SB == 2) {                             // other S^T buffer: free since dV(g - 1)
                if (h == 0 && !wait_a(g + 1)) { ok = false; break; }
                tc_fence_after();
                issue_s(g + 1, h);
              }
              if (!mbar_wait(bar_pfull + 16 * h + 8 * (g & 1), (g >> 1) & 1, abort_flag, status, 69)) { ok = false; break; }
              tc_fence_after();
              issue_acc(L::kColAcc1, L::kColS + (SB == 2 ? (g & 1) * 128 : 0), tile_b(g), h, it == 0);   // dV += P^T dO
              if (h == 1) umma_commit(bar_bempty + 8 * (g % SR));                       // dO(g) is not read again
              if (more && SB == 1) {                             // reuses the buffer dV(g) just read
                if (h == 0 && !wait_a(g + 1)) { ok = false; break; }
                tc_fence_after();
                issue_s(g + 1, h);
              }
              if (!mbar_wait(bar_dsfull + 16 * h + 8 * (g & 1), (g >> 1) & 1, abort_flag, status, 68)) { ok = false; break; }
              tc_fence_after();
              issue_acc(L::kColAcc0, L::kColDp, tile_a(g), h, it == 0);                          // dK += dS^T Q
              if (more) {                                        // reuses the buffer dK(g) just read
                if (h == 0 && !wait_b(g + 1)) { ok = false; break; }
                tc_fence_after();
                issue_dp(g + 1, h);
              }
            }
          }
          if (!ok) break;
          umma_commit(bar_aempty + 8 * (g % SA));
        }
        if (!ok) break;
        if (w.n_it > 0) {
          umma_commit(bar_accfull);
          ++ai;
        }
      }
    }
  } else if (warp == kB2ComputeWarps + 2) {
    // ------------------------------------------------------------------ statistics (B2_DKV): one step's 128 queries, four per lane
    uint32_t g = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x) {
      Work w;
      get_work(item, w);
      for (int it = 0; it < w.n_it; ++it, ++g) {
        int hq, q0, k0;
        walk_decode(w, it, hq, q0, k0);
        const int first = q0 + 4 * lane;
        const long long st = (static_cast<long long>(w.b) * p.heads + hq) * p.seq_q + first;
        float l[4], d[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool in = first + j < p.seq_q;
          l[j] = in ? -__ldg(p.lse + st + j) * kB2Log2e : 0.f;
          d[j] = in ? -__ldg(p.delta + st + j) : 0.f;
        }
        // the compute warps have finished step g - 2, whose place this is
        if (g >= 2 && !(mbar_wait(bar_dsfull + 8 * (g & 1), ((g >> 1) - 1) & 1, abort_flag, status, 74) &&
                        mbar_wait(bar_dsfull + 16 + 8 * (g & 1), ((g >> 1) - 1) & 1, abort_flag, status, 74))) {
          ok = false;
          break;
        }
        float4* dst = reinterpret_cast<float4*>(stats + (g & 1) * 256) + lane;
        dst[0] = make_float4(l[0], l[1], l[2], l[3]);
        dst[32] = make_float4(d[0], d[1], d[2], d[3]);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_stat + 8 * (g & 1));
      }
    }
  } else {
    // ------------------------------------------------------------------ compute warps
    const int qtr = warp & 3, cg = warp >> 2;              // TMEM lane quarter, column part
    const int half = cg >> 1;
    const int row = qtr * 32 + lane;                       // TMEM lane: query (B2_DQ) or key (B2_DKV) inside the tile
    const uint32_t lane_off = static_cast<uint32_t>(qtr * 32) << 16;
    const float sl2 = p.scale * kB2Log2e;
    const uint32_t half_sfull = bar_sfull + 16 * half, half_dpfull = bar_dpfull + 16 * half, half_pfull = bar_pfull + 16 * half,
                   half_dsfull = bar_dsfull + 16 * half;
    bool ok = true;
    uint32_t g = 0, ai = 0, wi = 0;
    // B2_DQ: this thread's row statistics (negated), for the whole item.  B2_DKV: one pair of numbers per query of the step, negated too, that
    // the statistics warp has put into shared memory.
    float lse_row = 0.f, dlt_row = 0.f;
    auto row_stats = [&](const Work& v) {
      lse_row = dlt_row = 0.f;
      if (MODE == B2_DQ && v.own0 + row < p.seq_q) {
        const long long st = (static_cast<long long>(v.b) * p.heads + v.head_q0) * p.seq_q + v.own0 + row;
        lse_row = -__ldg(p.lse + st) * kB2Log2e;
        dlt_row = -__ldg(p.delta + st);
      }
    };
    Work w;
    if (static_cast<int>(blockIdx.x) < total_items) {
      get_work(blockIdx.x, w);
      row_stats(w);
    }
    for (int item = blockIdx.x; item < total_items && ok; item += gridDim.x, ++wi) {
      int turn = 0;                                        // tile of the walk (B2_DKV: it starts again for the next head of the group)
      for (int it = 0; it < w.n_it && ok; ++it, ++g) {
        const int walk0 = (w.walk_first + turn) * kB2Tile;
        if (++turn == w.walk_count) turn = 0;
        const float4* st_lse = reinterpret_cast<const float4*>(stats + (g & 1) * 256 + cg * kB2Cols);
        const float4* st_dlt = st_lse + 32;
        // visibility: B2_DQ row = query, columns = keys; B2_DKV row = key, columns = queries
        const int cbase = walk0 + cg * kB2Cols;
        int lim_lo = 0, lim_hi = 0;      // visible columns are [lim_lo, lim_hi]
        if (MODE == B2_DQ) {
          const int q_idx = w.own0 + row;
          lim_hi = q_idx < p.seq_q ? (p.causal ? min(w.kv_len - 1, q_idx + shift) : w.kv_len - 1) : -1;
        } else {
          const int key = w.own0 + row;
          lim_hi = key < w.kv_len ? p.seq_q - 1 : -1;
          lim_lo = p.causal ? max(0, key - shift) : 0;
        }
        const bool need_mask = cbase < lim_lo || cbase + kB2Cols - 1 > lim_hi;
        const uint32_t sb = SB == 2 ? (g & 1) : 0, db = DB == 2 ? (g & 1) : 0;
        const uint32_t t_s = tmem_base + L::kColS + sb * 128 + lane_off + cg * kB2Cols;
        const uint32_t t_dp = tmem_base + L::kColDp + db * 128 + lane_off + cg * kB2Cols;
        if (MODE == B2_DKV && !mbar_wait(bar_stat + 8 * (g & 1), (g >> 1) & 1, abort_flag, status, 73)) { ok = false; break; }
        if (!mbar_wait(half_sfull + 8 * sb, (SB == 2 ? (g >> 1) : g) & 1, abort_flag, status, 70)) { ok = false; break; }
        tc_fence_after();
        // ---- probabilities of this thread's columns (kept in registers as fp32)
        float pr[kB2Cols];
        {
          uint32_t r[2][16];
          tmem_ld_32x16(t_s, r[0]);
          tmem_ld_wait();
          tmem_ld_32x16(t_s + 16, r[1]);
          const Pair sl = pair_of(sl2, sl2), row_l = pair_of(lse_row, lse_row);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (c == 1) {
              tmem_ld_wait();
              if (MODE == B2_DQ) {
                // S is in registers: the next S may overwrite the buffer
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_sempty + 8 * half);
              }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              Pair l0 = row_l, l1 = row_l;
              if (MODE == B2_DKV) {
                const float4 l4 = st_lse[c * 4 + i];
                l0 = pair_of(l4.x, l4.y);
                l1 = pair_of(l4.z, l4.w);
              }
              const float2 x = floats(fma2(pair_of(__uint_as_float(r[c][4 * i]), __uint_as_float(r[c][4 * i + 1])), sl, l0));
              const float2 y = floats(fma2(pair_of(__uint_as_float(r[c][4 * i + 2]), __uint_as_float(r[c][4 * i + 3])), sl, l1));
              pr[c * 16 + 4 * i] = b2_ex2(x.x);
              pr[c * 16 + 4 * i + 1] = b2_ex2(x.y);
              pr[c * 16 + 4 * i + 2] = b2_ex2(y.x);
              pr[c * 16 + 4 * i + 3] = b2_ex2(y.y);
            }
          }
        }
        if (need_mask) {                       // tiles on the diagonal and at the ends only: a loop of its own
#pragma unroll
          for (int i = 0; i < kB2Cols; ++i)
            if (cbase + i < lim_lo || cbase + i > lim_hi) pr[i] = 0.f;
        }
        if (MODE == B2_DKV) {
          // P^T over this thread's own part of S^T: 32 queries -> 16 packed columns at the part's beginning
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(pr[2 * i], pr[2 * i + 1]);
          tmem_st_32x16(t_s, pk);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(half_pfull + 8 * (g & 1));
        }
        // ---- dS = P * (dP - delta) -> packed bf16 over this thread's part of the dP buffer
        if (!mbar_wait(half_dpfull + 8 * db, (DB == 2 ? (g >> 1) : g) & 1, abort_flag, status, 71)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t r[2][16], pk[16];
          tmem_ld_32x16(t_dp, r[0]);
          tmem_ld_32x16(t_dp + 16, r[1]);
          tmem_ld_wait();
          const Pair row_d = pair_of(dlt_row, dlt_row);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int c = i >> 2, e = 4 * (i & 3);
            Pair d0 = row_d, d1 = row_d;
            if (MODE == B2_DKV) {
              const float4 d4 = st_dlt[i];
              d0 = pair_of(d4.x, d4.y);
              d1 = pair_of(d4.z, d4.w);
            }
            const Pair x = add2(pair_of(__uint_as_float(r[c][e]), __uint_as_float(r[c][e + 1])), d0);
            const Pair y = add2(pair_of(__uint_as_float(r[c][e + 2]), __uint_as_float(r[c][e + 3])), d1);
            pk[2 * i] = packed(mul2(pair_of(pr[4 * i], pr[4 * i + 1]), x));
            pk[2 * i + 1] = packed(mul2(pair_of(pr[4 * i + 2], pr[4 * i + 3]), y));
          }
          tmem_st_32x16(t_dp, pk);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(half_dsfull + 8 * (g & 1));
      }
      if (!ok) break;

      // ---- read-out: TMEM lane = key (B2_DKV) or query (B2_DQ) row of the owned tile; this column part's share of D.  The rows go
      // through the memory of the item's resident operands: every product that reads them is complete.
      const Work done = w;
      if (item + static_cast<int>(gridDim.x) < total_items) {      // decoded and requested while the last products run
        get_work(item + gridDim.x, w);
        row_stats(w);
      }
      const bool have = done.n_it > 0;
      if (have) {
        if (!mbar_wait(bar_accfull, ai & 1, abort_flag, status, 72)) { ok = false; break; }
      } else if (!mbar_wait(bar_res + 8 * (wi % RS), (wi / RS) & 1, abort_flag, status, 77)) { ok = false; break; }
      tc_fence_after();
      constexpr int CW = D * kB2Cols / 128;                // output columns per part
      constexpr int kOut = MODE == B2_DKV ? 2 : 1;
      const uint32_t out0 = sRes + (wi % RS) * 2 * L::kTileBytes;
#pragma unroll
      for (int which = 0; which < kOut; ++which) {
        const uint32_t tacc = tmem_base + (which == 0 ? L::kColAcc0 : L::kColAcc1);
        const float mul = which == 0 ? p.scale : 1.f;      // dK and dQ carry the softmax scale, dV does not
        uint32_t r[CW / 16][16];
#pragma unroll
        for (int c = 0; c < CW / 16; ++c) {
          if (have) {
            tmem_ld_32x16(tacc + lane_off + cg * CW + c * 16, r[c]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i) r[c][i] = 0u;
          }
        }
        tmem_ld_wait();
        if (have && which == kOut - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_accempty);
          ++ai;
        }
#pragma unroll
        for (int c = 0; c < CW / 8; ++c) {
          const int col = cg * CW + c * 8;
          const uint32_t* v = &r[c / 2][8 * (c & 1)];
          uint32_t o[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) o[i] = pack_bf16x2(__uint_as_float(v[2 * i]) * mul, __uint_as_float(v[2 * i + 1]) * mul);
          const uint32_t at = out0 + which * L::kTileBytes + (col >> 6) * L::kHalf + row * 128 + ((((col & 63) >> 3) ^ (row & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]) : "memory");
        }
      }
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_staged + 8 * qtr);
      if (cg == 0) {
        // all four parts of these 32 rows are there
        if (!mbar_wait(bar_staged + 8 * qtr, wi & 1, abort_flag, status, 78)) { ok = false; break; }
        if (lane == 0 && done.own0 + qtr * 32 < (MODE == B2_DKV ? p.seq_k : p.seq_q)) {
#pragma unroll
          for (int which = 0; which < kOut; ++which)
#pragma unroll
            for (int hf = 0; hf < D / 64; ++hf)
              tma_store_4d(which == 0 ? &tmOut0 : &tmOut1, out0 + which * L::kTileBytes + hf * L::kHalf + qtr * 4096, hf * 64,
                           MODE == B2_DKV ? done.head_k : done.head_q0, done.own0 + qtr * 32, done.b);
          tma_store_commit();
          tma_store_wait_read<0>();
        }
        if (lane == 0) mbar_arrive(bar_res_empty + 8 * (wi % RS));
        __syncwarp();
      }
    }
    if (cg == 0 && lane == 0) tma_store_wait<0>();
  }

  tc_fence_before();
  __syncthreads();
  if (warp == kB2ComputeWarps + 1) {
    if (*abort_flag) {
      const unsigned long long t0 = globaltimer_ns();
      while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
    }
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace rb

namespace {
// rows: of the box that one copy moves
const CUtensorMap* b2_map(const void* base, const long long* strides, int seq, int heads, int batch, int D, int rows, int* err) {
  long long s[3] = {strides[0] > 0 ? strides[0] : 8, strides[1] > 0 ? strides[1] : D, strides[2] > 0 ? strides[2] : D};
  const uint64_t dims[4] = {(uint64_t)D, (uint64_t)heads, (uint64_t)seq, (uint64_t)batch};
  const uint64_t str[3] = {(uint64_t)s[2] * 2, (uint64_t)s[1] * 2, (uint64_t)s[0] * 2};
  const uint32_t box[4] = {64, 1, (uint32_t)rows, 1};
  return rbhost::get_tmap_4d(base, 2, dims, str, box, 1, err);
}

struct B2Maps {
  const CUtensorMap *q, *k, *v, *d_o;
};

template <int D, int MODE>
int b2_launch(const B2Maps& m, const CUtensorMap* out0, const CUtensorMap* out1, const rb::B2Params& p, dim3 grid, cudaStream_t stream) {
  auto kern = rb::attn_bwd2_kernel<D, MODE>;
  const int smem = rb::B2Smem<D, MODE>::kTotal;
  static bool cfg_dev[64] = {false};
  bool& cfg = cfg_dev[rbhost::device_slot()];
  if (!cfg) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    cfg = true;
  }
  rbhost::launch_pdl(kern, grid, dim3(rb::B2Smem<D, MODE>::kThreads), smem, stream, 1, *m.q, *m.k, *m.v, *m.d_o, *out0, *out1, p,
                     rbhost::status_ptr());
  return static_cast<int>(cudaGetLastError());
}
}  // namespace

// Backward pass, second tcgen05 version (three launches: delta, dK/dV, dQ).  Returns -9 when the problem is outside
// what these kernels take (the caller then uses another backward implementation).
RB_API int rb_attention_bwd_tc2(const RbAttnArgs* a, void* stream_v) {
  if (a->batch <= 0 || a->heads <= 0 || a->kv_heads <= 0 || a->heads % a->kv_heads) return -1;
  if (a->head_dim != 64 && a->head_dim != 128) return -9;
  if (a->seq_q <= 0 || a->seq_k <= 0 || (a->causal && a->seq_q > a->seq_k)) return -1;
  if (!a->lse || !a->delta) return -2;
  const void* ptrs[8] = {a->q, a->k, a->v, a->o, a->d_o, a->dq, a->dk, a->dv};
  for (int i = 0; i < 8; ++i)
    if (!ptrs[i] || (reinterpret_cast<uintptr_t>(ptrs[i]) & 15)) return -9;
  const long long* strs[7] = {a->q_strides, a->k_strides, a->v_strides, a->o_strides, a->dq_strides, a->dk_strides, a->dv_strides};
  for (int i = 0; i < 7; ++i)
    for (int j = 0; j < 3; ++j)
      if (strs[i][j] % 8) return -9;
  const int D = a->head_dim;
  int err = 0;
  B2Maps m;
  m.q = b2_map(a->q, a->q_strides, a->seq_q, a->heads, a->batch, D, rb::kB2Tile, &err);
  m.k = b2_map(a->k, a->k_strides, a->seq_k, a->kv_heads, a->batch, D, rb::kB2Tile, &err);
  m.v = b2_map(a->v, a->v_strides, a->seq_k, a->kv_heads, a->batch, D, rb::kB2Tile, &err);
  m.d_o = b2_map(a->d_o, a->o_strides, a->seq_q, a->heads, a->batch, D, rb::kB2Tile, &err);
  const CUtensorMap* dq = b2_map(a->dq, a->dq_strides, a->seq_q, a->heads, a->batch, D, 32, &err);
  const CUtensorMap* dk = b2_map(a->dk, a->dk_strides, a->seq_k, a->kv_heads, a->batch, D, 32, &err);
  const CUtensorMap* dv = b2_map(a->dv, a->dv_strides, a->seq_k, a->kv_heads, a->batch, D, 32, &err);
  if (!m.q || !m.k || !m.v || !m.d_o || !dq || !dk || !dv) return err ? err : -5;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  int rc = rb_attention_delta_tc(a, stream_v);
  if (rc != 0) return rc;

  rb::B2Params p;
  p.lse = a->lse; p.delta = a->delta;
  p.seq_q = a->seq_q; p.seq_k = a->seq_k; p.heads = a->heads; p.kv_heads = a->kv_heads; p.causal = a->causal;
  p.batch = a->batch;
  p.scale = a->scale;
  p.kv_lens = a->kv_lens;
  const int sms = rbhost::device_sm_count();
  const long long kv_items = static_cast<long long>((a->seq_k + rb::kB2Tile - 1) / rb::kB2Tile) * a->kv_heads * a->batch;
  dim3 kvgrid(static_cast<unsigned>(kv_items < sms ? kv_items : sms));
  rc = D == 64 ? b2_launch<64, rb::B2_DKV>(m, dk, dv, p, kvgrid, stream) : b2_launch<128, rb::B2_DKV>(m, dk, dv, p, kvgrid, stream);
  if (rc != 0) return rc;
  const long long q_items = static_cast<long long>((a->seq_q + rb::kB2Tile - 1) / rb::kB2Tile) * a->heads * a->batch;
  dim3 qgrid(static_cast<unsigned>(q_items < sms ? q_items : sms));
  return D == 64 ? b2_launch<64, rb::B2_DQ>(m, dq, dq, p, qgrid, stream) : b2_launch<128, rb::B2_DQ>(m, dq, dq, p, qgrid, stream);
}
