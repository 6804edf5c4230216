// Attention of one layer of a decoding step of a few sequences, from the packed projection, in one launch: rotation of queries and keys, append of
// the new token, split-KV attention through the block table and the merge of its slices.
//
// With one or a few sequences nothing here takes memory's time; what counts is the chain of latencies between the projection's last store
// and the result.  So everything that does not depend on the projection is done before it ends (programmatic dependent launch): a CTA owns one slice of 256
// cached tokens of a sequence for one KV head, four warps take 32 tokens each and then 32 more, and all their K and V rows are asked for, with
// slots looked up and angles formed, while the projection still runs.  Behind it come the queries and the new token's row, which goes from the
// projection into the tiles and into the cache.  A CTA leaves (max, sum, accumulator) of its slice; the last one of a sequence and KV head to count
// itself in adds up the slices in their order.  Slices, the order inside them and the arithmetic, contractions included, are those of
// `paged_decode_split_kernel` (paged_attention.cu), so a sequence gets the same bits alone as beside many others.
//
// One B200, a layer of a step in a captured chain, us, rotation and append, slices and merge in launches of their own / this kernel: 1 sequence of 2047,
// 4 KV heads of 128 14.4 / 7.2; of 300, 12 heads of 64 9.2 / 5.1.  As a form of `paged_decode_split_kernel` the one launch took 12.8 and 8.5: half of
// that was code met for the first time (200 cycles per hundred instructions), looked-up slots and copies of the second 32 tokens, and a merge by
// one thread per column with its divisions.
#include "paged_attention.h"

#include "pdl.cuh"
#include "rb_common.cuh"
#include "rotary.cuh"
#include "warp_mma.cuh"

namespace rb {

constexpr int kStepWarps = 4;
constexpr int kStepTokens = 256;                 // of a slice: two tiles of 32 per warp
constexpr int kStepGroup = 16;                   // query heads per KV head at most: the rows of the m16n8k16 tile

struct StepParams {
  const __nv_bfloat16* qkv;                      // [batch, (heads + 2 kv_heads) * D], pitch ld
  long long ld;
  __nv_bfloat16* out;
  long long ld_o;
  __nv_bfloat16* k_cache;
  __nv_bfloat16* v_cache;
  const int* block_tables;
  const int* context_lens;
  float* partial;                                // [batch, heads, nsplit][max, sum, D]
  unsigned int* arrived;                         // [batch * kv_heads], zero before and after
  long long num_blocks;
  int max_blocks, block_size, heads, kv_heads, nsplit;
  float scale, log2_theta;                       // log2_theta 0: no rotation
};

template <int D>
struct StepSmem {
  static constexpr int kRow = D + 8;             // padded rows (elements): ldmatrix rows hit distinct banks
  static constexpr int kTile = 32 * kRow;        // one tile of K or V of one warp
  static constexpr int kQ = kStepWarps * 4 * kTile * 2;                  // byte offset of the 16 query rows
  static constexpr int kTurn = kQ + kStepGroup * kRow * 2;               // cosine and sine of the new token's angles
  static constexpr int kFactor = kTurn + (D / 2) * 8;                    // [warps][16] factors and sums of the warps
  static constexpr int kTotal = kFactor + 2 * kStepWarps * kStepGroup * 4;
};

// Sums the n slices of one sequence and KV head, a warp per head; lanes own pairs of neighbouring columns.
template <int D>
__device__ __forceinline__ void step_merge(const float* partial, int n, int nsplit, int group, __nv_bfloat16* out) {
  constexpr int P = D / 64;                      // pairs per lane
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
  for (int g = warp; g < group; g += kStepWarps) {
    const float* base = partial + static_cast<long long>(g) * nsplit * (D + 2);
    float2 ml = lane < n ? __ldcg(reinterpret_cast<const float2*>(base + lane * (D + 2))) : make_float2(-INFINITY, 0.f);
    float mx = ml.x;
    for (int s = lane + 32; s < n; s += 32) mx = fmaxf(mx, __ldcg(base + s * (D + 2)));
    float2 num[P];
    float den = 0.f;
#pragma unroll
    for (int j = 0; j < P; ++j) num[j] = make_float2(0.f, 0.f);
    float factor = 0.f;
#pragma unroll 1
    for (int s0 = 0; s0 < n; s0 += 8) {
      const float* at = base + static_cast<long long>(s0) * (D + 2) + 2 + 2 * lane;
      float2 v[8][P];
#pragma unroll
      for (int s = 0; s < 8; ++s)
#pragma unroll
        for (int j = 0; j < P; ++j)
          v[s][j] = s0 + s < n ? __ldcg(reinterpret_cast<const float2*>(at + s * (D + 2) + j * 64)) : make_float2(0.f, 0.f);
      if ((s0 & 31) == 0) {                      // factors of the next 32 slices, one per lane
        if (s0 == 0) mx = warp_max(mx);
        else ml = s0 + lane < n ? __ldcg(reinterpret_cast<const float2*>(base + (s0 + lane) * (D + 2))) : make_float2(-INFINITY, 0.f);
        factor = ml.x == -INFINITY ? 0.f : __expf(ml.x - mx);
      }
#pragma unroll
      for (int s = 0; s < 8; ++s) {
        const float f = __shfl_sync(0xffffffffu, factor, (s0 + s) & 31), l = __shfl_sync(0xffffffffu, ml.y, (s0 + s) & 31);
        den = __fmaf_rn(l, f, den);
#pragma unroll
        for (int j = 0; j < P; ++j) num[j] = make_float2(__fmaf_rn(v[s][j].x, f, num[j].x), __fmaf_rn(v[s][j].y, f, num[j].y));
      }
    }
#pragma unroll
    for (int j = 0; j < P; ++j)
      *reinterpret_cast<uint32_t*>(out + g * D + 2 * lane + j * 64) =
          den > 0.f ? pack_bf16x2(num[j].x / den, num[j].y / den) : 0u;
  }
}

template <int D>
__global__ void __launch_bounds__(kStepWarps * 32, 1)
paged_step_kernel(const StepParams p RB_BOUNDS_PARAM) {
  using L = StepSmem<D>;
  constexpr int PIECES = D / 8, NT = D / 8, U = D / 16;       // 16-byte pieces of a row; n-tiles of the accumulator; units of eight pairs of a head
  extern __shared__ __align__(16) uint8_t step_smem[];
  const int b = blockIdx.x, hk = blockIdx.y, sp = blockIdx.z;
  const int ctx = p.context_lens[b];
  const int n_slices = max(0, min(p.nsplit, (ctx + kStepTokens - 1) / kStepTokens));
  if (sp >= n_slices) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int gq = lane >> 2, tq = lane & 3;                    // fragment coordinates: row (and row + 8), column pair
  const int group = p.heads / p.kv_heads;
  const int t_end = min(ctx, (sp + 1) * kStepTokens), base = sp * kStepTokens + warp * 32;
  __nv_bfloat16* tiles = reinterpret_cast<__nv_bfloat16*>(step_smem) + warp * 4 * L::kTile;      // K, V of the first 32 tokens, then of the second
  __nv_bfloat16* q_sh = reinterpret_cast<__nv_bfloat16*>(step_smem + L::kQ);
  float2* turn_sh = reinterpret_cast<float2*>(step_smem + L::kTurn);
  float* factor_sh = reinterpret_cast<float*>(step_smem + L::kFactor);
  float* sum_sh = factor_sh + kStepWarps * kStepGroup;
  __shared__ int last_sh;

  // ---- cached tokens.  Lane i knows the slots of tokens base + i and base + 128 + i; -1: past the end, or the new token
  long long place = -1;                                       // of the new token, in the lane that has it
  int slot[2];
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    const int tok = base + t * 128 + lane;
    slot[t] = -1;
    if (tok < t_end) {
      const int blk_idx = tok / p.block_size;
      int blk = blk_idx < p.max_blocks ? p.block_tables[static_cast<long long>(b) * p.max_blocks + blk_idx] : -1;
      const bool bad = blk < 0 || blk >= p.num_blocks;        // corrupt tables read block 0 instead of faulting, and take no new token
      if (bad) RB_BOUNDS_HIT(104);
      const int at = (bad ? 0 : blk) * p.block_size + (tok - blk_idx * p.block_size);
      if (tok < ctx - 1) slot[t] = at;
      else if (!bad) place = static_cast<long long>(at) * p.kv_heads + hk;
    }
  }
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    if (base + t * 128 < t_end) {
#pragma unroll
      for (int kv = 0; kv < 2; ++kv) {
        const __nv_bfloat16* cache = kv ? p.v_cache : p.k_cache;
        const uint32_t dst = smem_u32(tiles + (2 * t + kv) * L::kTile);
#pragma unroll
        for (int i = 0; i < PIECES; ++i) {
          const int idx = i * 32 + lane, r = idx / PIECES, c = (idx - r * PIECES) * 8;
          const int s_r = __shfl_sync(0xffffffffu, slot[t], r);
          wm_cp16(dst + (r * L::kRow + c) * 2, s_r >= 0 ? cache + (static_cast<long long>(s_r) * p.kv_heads + hk) * D + c : cache, s_r >= 0);
        }
      }
    }
  }
  wm_cp_commit();
  if (p.log2_theta != 0.f && threadIdx.x < D / 2) {           // formed like rope_kernel's
    const float inv_freq = exp2f(-p.log2_theta * (2.f * threadIdx.x) / static_cast<float>(D));
    float sn, cs;
    sincosf(static_cast<float>(ctx - 1) * inv_freq, &sn, &cs);
    turn_sh[threadIdx.x] = make_float2(cs, sn);
  }
  __syncthreads();

  // ---- from here on what the projection has written
  pdl_wait();
  pdl_launch();
  auto rotate = [&](int unit, uint4& lo, uint4& hi) {
    if (p.log2_theta != 0.f) rope_unit(lo, hi, [&](int j) { return turn_sh[unit * 8 + j]; });
  };
  const __nv_bfloat16* row = p.qkv + static_cast<long long>(b) * p.ld;
  // the new token belongs to the warp whose tile it lies in: lane u < U holds pairs 8 u .. of its key, lane c < PIECES eight values
  const int fresh = ctx - 1 - base;
  const bool owner = ctx <= t_end && fresh >= 0 && (fresh & 96) == 0;       // in the first 32 tokens of base or base + 128
  uint4 new_lo, new_hi, new_v;
  if (owner) {
    const __nv_bfloat16* k = row + static_cast<long long>(p.heads + hk) * D;
    const __nv_bfloat16* v = row + static_cast<long long>(p.heads + p.kv_heads + hk) * D;
    if (lane < U) {
      new_lo = *reinterpret_cast<const uint4*>(k + lane * 8);
      new_hi = *reinterpret_cast<const uint4*>(k + D / 2 + lane * 8);
    }
    if (lane < PIECES) new_v = *reinterpret_cast<const uint4*>(v + lane * 8);
  }
  for (int i = threadIdx.x; i < kStepGroup * U; i += kStepWarps * 32) {
    const int g = i / U, u = i - g * U;
    uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
    if (g < group) {
      const __nv_bfloat16* src = row + static_cast<long long>(hk * group + g) * D + u * 8;
      lo = *reinterpret_cast<const uint4*>(src);
      hi = *reinterpret_cast<const uint4*>(src + D / 2);
      rotate(u, lo, hi);
    }
    *reinterpret_cast<uint4*>(q_sh + g * L::kRow + u * 8) = lo;
    *reinterpret_cast<uint4*>(q_sh + g * L::kRow + D / 2 + u * 8) = hi;
  }
  wm_cp_wait<0>();
  __syncwarp();                                               // this warp's tiles have landed, zeros in the new token's row
  if (owner) {
    const long long at = __shfl_sync(0xffffffffu, place, fresh & 31);
    __nv_bfloat16* tk = tiles + 2 * (fresh >> 7) * L::kTile + (fresh & 31) * L::kRow;
    if (lane < U) {
      rotate(lane, new_lo, new_hi);
      *reinterpret_cast<uint4*>(tk + lane * 8) = new_lo;
      *reinterpret_cast<uint4*>(tk + D / 2 + lane * 8) = new_hi;
      if (at >= 0) {
        *reinterpret_cast<uint4*>(p.k_cache + at * D + lane * 8) = new_lo;
        *reinterpret_cast<uint4*>(p.k_cache + at * D + D / 2 + lane * 8) = new_hi;
      }
    }
    if (lane < PIECES) {
      *reinterpret_cast<uint4*>(tk + L::kTile + lane * 8) = new_v;
      if (at >= 0) *reinterpret_cast<uint4*>(p.v_cache + at * D + lane * 8) = new_v;
    }
  }
  __syncthreads();

  float m0 = -INFINITY, m1 = -INFINITY, l0 = 0.f, l1 = 0.f;   // rows gq and gq + 8
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  const uint32_t q_u32 = smem_u32(q_sh);
#pragma unroll 1
  for (int t = 0; t < 2; ++t) {
    const int n_tok = min(32, t_end - base - t * 128);
    if (n_tok <= 0) break;
    const uint32_t kt = smem_u32(tiles + 2 * t * L::kTile), vt = kt + L::kTile * 2;
    // ---- S[16 heads, 32 tokens] = Q K^T
    float s[4][4];
#pragma unroll
    for (int n = 0; n < 4; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.f;
#pragma unroll
    for (int k0 = 0; k0 < D; k0 += 16) {
      uint32_t a[4];
      wm_ldsm_x4(wm_a(q_u32, L::kRow, 0, k0, lane), a);
#pragma unroll
      for (int np = 0; np < 2; ++np) {
        uint32_t bfr[4];
        wm_ldsm_x4(wm_b(kt, L::kRow, np * 16, k0, lane), bfr);
        wm_mma(s[2 * np], a, bfr[0], bfr[1]);
        wm_mma(s[2 * np + 1], a, bfr[2], bfr[3]);
      }
    }
    // ---- online softmax over the 32 tokens; this thread holds 8 of them for rows gq and gq + 8
    float mx0 = -INFINITY, mx1 = -INFINITY;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const bool ok = n * 8 + 2 * tq + j < n_tok;
        s[n][j] = ok ? __fmul_rn(s[n][j], p.scale) : -INFINITY;
        s[n][2 + j] = ok ? __fmul_rn(s[n][2 + j], p.scale) : -INFINITY;
        mx0 = fmaxf(mx0, s[n][j]);
        mx1 = fmaxf(mx1, s[n][2 + j]);
      }
    }
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
    mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
    mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
    const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);   // finite: token 0 of the pass is always valid
    const float al0 = (m0 == -INFINITY) ? 0.f : __expf(m0 - mn0);
    const float al1 = (m1 == -INFINITY) ? 0.f : __expf(m1 - mn1);
    float sum0 = 0.f, sum1 = 0.f;
    uint32_t pfr[2][4];                                       // P as the A operand of the two 16-token k-steps
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const float p0 = __expf(s[n][0] - mn0), p1 = __expf(s[n][1] - mn0);
      const float p2 = __expf(s[n][2] - mn1), p3 = __expf(s[n][3] - mn1);
      sum0 += p0 + p1;
      sum1 += p2 + p3;
      pfr[n >> 1][(n & 1) * 2 + 0] = pack_bf16x2(p0, p1);
      pfr[n >> 1][(n & 1) * 2 + 1] = pack_bf16x2(p2, p3);
    }
    sum0 += __shfl_xor_sync(0xffffffffu, sum0, 1);
    sum0 += __shfl_xor_sync(0xffffffffu, sum0, 2);
    sum1 += __shfl_xor_sync(0xffffffffu, sum1, 1);
    sum1 += __shfl_xor_sync(0xffffffffu, sum1, 2);
    l0 = __fmaf_rn(l0, al0, sum0);
    l1 = __fmaf_rn(l1, al1, sum1);
    m0 = mn0;
    m1 = mn1;
#pragma unroll
    for (int n = 0; n < NT; ++n) { acc[n][0] *= al0; acc[n][1] *= al0; acc[n][2] *= al1; acc[n][3] *= al1; }
    // ---- O[16, D] += P[16, 32] V[32, D]
#pragma unroll
    for (int ks = 0; ks < 2; ++ks) {
#pragma unroll
      for (int n2 = 0; n2 < NT / 2; ++n2) {
        uint32_t bfr[4];
        wm_ldsm_x4_t(wm_b_t(vt, L::kRow, n2 * 16, ks * 16, lane), bfr);
        wm_mma(acc[2 * n2], pfr[ks], bfr[0], bfr[1]);
        wm_mma(acc[2 * n2 + 1], pfr[ks], bfr[2], bfr[3]);
      }
    }
  }

  // ---- the warps' results, in the memory of their first tiles
  if (tq == 0) {
    factor_sh[warp * kStepGroup + gq] = m0; sum_sh[warp * kStepGroup + gq] = l0;
    factor_sh[warp * kStepGroup + gq + 8] = m1; sum_sh[warp * kStepGroup + gq + 8] = l1;
  }
  __syncwarp();
  float* mine = reinterpret_cast<float*>(tiles) + gq * L::kRow + 2 * tq;       // [16][D + 8] fp32 where the first K and V tiles were
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    if (gq < group) *reinterpret_cast<float2*>(mine + n * 8) = make_float2(acc[n][0], acc[n][1]);
    if (gq + 8 < group) *reinterpret_cast<float2*>(mine + 8 * L::kRow + n * 8) = make_float2(acc[n][2], acc[n][3]);
  }
  __syncthreads();
  const bool direct = n_slices == 1;
  const float* all = reinterpret_cast<const float*>(step_smem);
  constexpr int kWarpPitch = 2 * L::kTile;                    // floats between two warps' tiles
#pragma unroll 2
  for (int i = threadIdx.x; i < group * D; i += kStepWarps * 32) {
    const int g = i / D, d = i - g * D;
    float mx = -INFINITY;
#pragma unroll
    for (int w = 0; w < kStepWarps; ++w) mx = fmaxf(mx, factor_sh[w * kStepGroup + g]);
    float num = 0.f, den = 0.f;
#pragma unroll
    for (int w = 0; w < kStepWarps; ++w) {
      const float m = factor_sh[w * kStepGroup + g], sc = (m == -INFINITY) ? 0.f : __expf(m - mx);
      num = __fmaf_rn(all[w * kWarpPitch + g * L::kRow + d], sc, num);
      den = __fmaf_rn(sum_sh[w * kStepGroup + g], sc, den);
    }
    if (direct) {
      p.out[b * p.ld_o + static_cast<long long>(hk * group + g) * D + d] = __float2bfloat16(num / den);
    } else {
      float* pp = p.partial + ((static_cast<long long>(b) * p.heads + hk * group + g) * p.nsplit + sp) * (D + 2);
      pp[2 + d] = num;
      if (d == 0) { pp[0] = mx; pp[1] = den; }
    }
  }
  if (direct) return;
  __syncthreads();                                            // all partial results are written
  if (threadIdx.x == 0) {
    __threadfence();                                          // for the whole CTA, behind its barrier; the last arrival brings the counter back to zero
    last_sh = atomicInc(p.arrived + static_cast<long long>(b) * p.kv_heads + hk, n_slices - 1) == static_cast<unsigned>(n_slices - 1);
  }
  __syncthreads();
  if (!last_sh) return;
  __threadfence();
  step_merge<D>(p.partial + (static_cast<long long>(b) * p.heads + hk * group) * p.nsplit * (D + 2), n_slices, p.nsplit, group,
                p.out + b * p.ld_o + static_cast<long long>(hk) * group * D);
}

}  // namespace rb

namespace {
int step_slices(int max_blocks, int block_size) {
  return static_cast<int>((static_cast<long long>(max_blocks) * block_size + rb::kStepTokens - 1) / rb::kStepTokens);
}

template <int D>
int step_launch(const rb::StepParams& p, int batch, cudaStream_t stream) {
  auto kern = rb::paged_step_kernel<D>;
  const int smem = rb::StepSmem<D>::kTotal;
  static bool cfg_dev[64] = {false};
  bool& cfg = cfg_dev[rbhost::device_slot()];
  if (!cfg) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return static_cast<int>(e);
    cfg = true;
  }
  return static_cast<int>(rbhost::launch_pdl(kern, dim3(batch, p.kv_heads, p.nsplit), dim3(rb::kStepWarps * 32), smem, stream, 1, p RB_BOUNDS_ARG));
}
}  // namespace

// Up to six times as many slices as SMs in the tables: the batches and table widths that `paged_decode_split_kernel` works on as a grid of slices.  With
// heads of 64 (75 KB of shared memory) this kernel is faster up to there: 5.8 slices per SM 27.8 us a layer with its projection, three launches
// 29.5.  With heads of 128 (141 KB, one CTA on an SM) it is so up to about two slices per SM that are there: 1.9 22.3 / 25.9, 2.6 30.3 / 28.5, 5.8 57.0 / 42.8; callers
// that know the lengths decide by them, since tables are mostly wider than their sequences.
// Behind it, where slices are dealt as a list to CTAs that stay, counting and summing at a CTA's end cost more than the launches (a list form of this
// kernel, us per layer: 64 sequences of 100 to 4000 tokens 69.2 in three launches, 90.6 in one; 24 of 128 to 2560 42.6, 46.7).
RB_API int rb_paged_attention_step_takes(int batch, int kv_heads, int max_blocks, int block_size) {
  return batch > 0 && kv_heads > 0 && max_blocks > 0 && block_size > 0 &&
         static_cast<long long>(batch) * kv_heads * step_slices(max_blocks, block_size) <= 6ll * rbhost::device_sm_count();
}

RB_API int rb_paged_attention_step(const RbPagedStepArgs* args, void* stream_v) {
  const RbPagedStepArgs& t = *args;
  if (t.batch <= 0) return 0;
  if (t.heads <= 0 || t.kv_heads <= 0 || t.heads % t.kv_heads || t.heads / t.kv_heads > rb::kStepGroup || (t.head_dim != 64 && t.head_dim != 128) ||
      t.block_size <= 0 || t.max_blocks <= 0 || !t.scratch || !t.arrived || t.num_blocks <= 0 || t.num_blocks * t.block_size >= (1ll << 31) ||
      (t.ld_qkv % 8) || (t.ld_o % 2) || t.theta < 0.f)
    return -1;
  if ((reinterpret_cast<uintptr_t>(t.qkv) | reinterpret_cast<uintptr_t>(t.k_cache) | reinterpret_cast<uintptr_t>(t.v_cache)) & 15) return -2;
  if ((reinterpret_cast<uintptr_t>(t.scratch) & 7) || (reinterpret_cast<uintptr_t>(t.out) & 3)) return -2;
  if (!rb_paged_attention_step_takes(t.batch, t.kv_heads, t.max_blocks, t.block_size)) return -9;
  rb::StepParams p;
  p.qkv = reinterpret_cast<const __nv_bfloat16*>(t.qkv); p.ld = t.ld_qkv;
  p.out = reinterpret_cast<__nv_bfloat16*>(t.out); p.ld_o = t.ld_o;
  p.k_cache = reinterpret_cast<__nv_bfloat16*>(t.k_cache);
  p.v_cache = reinterpret_cast<__nv_bfloat16*>(t.v_cache);
  p.block_tables = t.block_tables; p.context_lens = t.context_lens;
  p.partial = t.scratch; p.arrived = t.arrived;
  p.num_blocks = t.num_blocks; p.max_blocks = t.max_blocks; p.block_size = t.block_size;
  p.heads = t.heads; p.kv_heads = t.kv_heads; p.nsplit = step_slices(t.max_blocks, t.block_size);
  p.scale = t.scale;
  p.log2_theta = t.theta > 0.f ? log2f(t.theta) : 0.f;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_v);
  return t.head_dim == 128 ? step_launch<128>(p, t.batch, stream) : step_launch<64>(p, t.batch, stream);
}
