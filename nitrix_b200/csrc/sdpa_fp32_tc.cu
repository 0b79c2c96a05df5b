// fp32 attention on the tcgen05 tensor cores: every fp32 operand is taken apart into three bf16 numbers and every product
// into the six bf16 products that matter.
//
//   x = x0 + x1 + x2 exactly (8 significant bits each, by truncation: x0 the top 16 bits of x, x1 the top 16 of x - x0,
//   x2 the rest; below 2^-103 the last ones are subnormal and flushed, as a TF32 pair's are), and a b = a0 b0 + a0 b1 + a1 b0 + a1 b1 + a0 b2 + a2 b0 but for a1 b2 + a2 b1 + a2 b2, which is below
//   2^-20 |a b| and 2^-22 of it on average; the products are exact and are accumulated in fp32 by the tensor core, the
//   small ones first.
//
// Six products at the bf16 rate cost what three at the tf32 rate would, lose less than a tf32 (hi, lo) pair (2^-20 three
// times over), and need the 16-bit operand layouts only.
//
// split_planes_kernel writes the three planes of q, k, v (and dout) into the workspace as the tiles the MMA reads -- 64 rows
// x 64 columns of bf16 in the 128-byte swizzle, 8 KB, planes of a tile side by side -- so the attention kernels fetch
// them with plain bulk copies, whatever the strides and the length of the operand were: rows past the end are zeros.
#include <math.h>

#include "sdpa_tc_common.cuh"

namespace nb200 {
namespace {

using namespace sm100;
using tc::wait_or_abort;

constexpr int kRows = 64;                 // rows of a split tile, keys of a step
constexpr int kChunkBytes = kRows * 128;  // one plane of 64 columns of a tile

// ---- the split --------------------------------------------------------------------------------------------------
struct SplitOperand {
  const float* x;
  uint8_t* planes;
  int64_t xs[3];      // element strides over (b, h, row)
  int rows, tiles;    // per (b, h)
};
struct SplitArgs {
  SplitOperand op[4];
  int H, bh_begin, D;
};

// eight fp32 as three words of eight bf16 each (see the file's comment)
__device__ __forceinline__ void split8(const float (&x)[8], uint4 (&w)[3]) {
  uint32_t r[8], o[4];
#pragma unroll
  for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(x[i]);
#pragma unroll
  for (int p = 0; p < 3; ++p) {
#pragma unroll
    for (int i = 0; i < 4; ++i) o[i] = __byte_perm(r[2 * i], r[2 * i + 1], 0x7632);
    w[p] = make_uint4(o[0], o[1], o[2], o[3]);
    if (p < 2) {
#pragma unroll
      for (int i = 0; i < 8; ++i) r[i] = __float_as_uint(__uint_as_float(r[i]) - __uint_as_float(r[i] & 0xffff0000u));
    }
  }
}

// Grid (tiles, bh, operands); kCols = the head dim padded to whole 64-column chunks.  Bound by memory traffic (4 bytes in,
// 6 out per element).
template <int kCols>
__global__ void __launch_bounds__(128) split_planes_kernel(SplitArgs a) {
  const SplitOperand op = a.op[blockIdx.z];
  if (int(blockIdx.x) >= op.tiles) return;
  const int bh = a.bh_begin + blockIdx.y, b = bh / a.H, h = bh - b * a.H;
  const float* x = op.x + b * op.xs[0] + h * op.xs[1];
  constexpr int kUnits = kCols / 8;
  uint8_t* tile = op.planes + (int64_t(blockIdx.y) * op.tiles + blockIdx.x) * (3 * (kCols / 64) * kChunkBytes);
  const bool vec = ((reinterpret_cast<uintptr_t>(op.x) & 15) == 0) && ((op.xs[0] | op.xs[1] | op.xs[2]) & 3) == 0;
#pragma unroll 4
  for (int u = threadIdx.x; u < kRows * kUnits; u += 128) {
    const int r = u / kUnits, c = u - r * kUnits, row = blockIdx.x * kRows + r;
    float v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = 0.f;
    if (row < op.rows && c * 8 < a.D) {      // (head dims are multiples of 32)
      const float* src = x + row * op.xs[2] + c * 8;
      if (vec) {
        *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(src);
        *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(src + 4);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = src[i];
      }
    }
    uint4 w[3];
    split8(v, w);
    uint8_t* dst = tile + (c / 8) * kChunkBytes + r * 128 + (((c & 7) ^ (r & 7)) * 16);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(dst + p * (kCols / 64) * kChunkBytes) = w[p];
  }
}

// ---- forward ------------------------------------------------------------------------------------------------------
struct FwdArgs {
  Problem pr;
  const uint8_t *q, *k, *v;     // planes
  int q_tiles, k_tiles;         // 64-row tiles per (b, h)
  int tiles_per_cta;            // 128-row query tiles of a CTA
  int bias_dtype;
  int* status;
};

// the six products, small ones first: (plane of the left operand, plane of the right one)
constexpr int kProducts = 6;
__device__ __forceinline__ constexpr int left_plane(int i) { return i == 0 ? 2 : (i == 1 ? 0 : (i == 2 ? 1 : (i == 3 ? 1 : 0))); }
__device__ __forceinline__ constexpr int right_plane(int i) { return i == 0 ? 0 : (i == 1 ? 2 : (i == 2 ? 1 : (i == 3 ? 0 : (i == 4 ? 1 : 0)))); }

// the addend of a key that the mask drops: a NaN that no arithmetic produces (an -inf bias is a value like any other)
constexpr uint32_t kDropped = 0x7fc0deadu;
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// rows x keys of the bias and the mask that the next step will read, as far as L2: `lane` takes one row of 32 x `keys`
__device__ __forceinline__ void prefetch_addends(const Problem& pr, int bias_size, int64_t b_at, int64_t m_at, int row, int key, int keys) {
  if (row >= pr.S || key >= pr.T) return;
  if (pr.bias && pr.bs[3] == 1) {
    const char* p = static_cast<const char*>(pr.bias) + (b_at + row * pr.bs[2] + key) * bias_size;
    const int bytes = min(keys, pr.T - key) * bias_size;
    for (int i = 0; i < bytes; i += 128) prefetch_l2(p + i);
    prefetch_l2(p + bytes - 1);
  }
  if (pr.mask && pr.ms[3] == 1) prefetch_l2(pr.mask + m_at + row * pr.ms[2] + key);
}
// neither the bias nor the mask has a query axis
__device__ __forceinline__ bool key_only_addends(const Problem& pr) {
  return (!pr.bias || pr.bs[2] == 0) && (!pr.mask || pr.ms[2] == 0);
}
// The soft-max's reference lies kAbove over the last maximum taken, which a later logit may outgrow by up to 2^kAbove: no
// p is above 1, so the un-normalised output overflows for no values of V that it would not overflow for at the maximum.
constexpr float kAbove = 8.f;
constexpr int kAddPitch = 33;   // floats: a row of 32 addends plus one, so that 32 rows fall on distinct banks

template <int kCols, bool kAdd>
struct FwdLayout {
  static constexpr int kChunks = kCols / 64;
  static constexpr int kTiles = kCols == 64 ? 2 : 1;           // 128-row query tiles a CTA has room for
  static constexpr int kStages = kCols == 64 ? 2 : 1;          // of K and of V
  static constexpr int kThreads = (5 * kTiles + 1) * 32;
  static constexpr int kPlane = kChunks * kChunkBytes;         // one plane of a 64-row tile
  static constexpr int kQ = 0;                                 // [kTiles][3][kChunks][128 rows x 128 B]
  static constexpr int kQBytes = 3 * 2 * kPlane;
  static constexpr int kK = kQ + kTiles * kQBytes;             // [kStages][3][kChunks][64 rows x 128 B]
  static constexpr int kV = kK + kStages * 3 * kPlane;
  static constexpr int kAddend = kV + kStages * 3 * kPlane;    // [4 kTiles warps][32 rows][kAddPitch] floats
  static constexpr int kBars = kAddend + (kAdd ? 4 * kTiles * 32 * kAddPitch * 4 : 0);
  static constexpr int kBytes = kBars + 256;
  // TMEM columns of a query tile: scores, the three planes of P, output
  static constexpr int kTmS = 0, kTmP = 64, kTmO = 160, kTmTile = 256, kTmCols = 512;
};
enum FwdBar { K_FULL = 0, K_EMPTY = 2, V_FULL = 4, V_EMPTY = 6, Q_FULL = 8, S_FULL = 10, S_FREE = 12, P_FULL = 14, PV_DONE = 16, kFwdBars = 18 };

// A CTA owns up to kTiles x 128 query rows of one (b, h) and streams the keys in steps of 64.  Warps 0-3 (4-7): a thread
// owns a row of the first (second) 128 -- online soft-max, P into three planes in TMEM; the next warp fetches, the last
// kTiles issue the MMAs of a query tile each: per step 6 x kCols / 16 for Q K^T (both operands in shared memory) and 6 x 4
// for P V.  The scores are read into registers at once, so Q K^T of the next step runs under the soft-max of this one.
// The tensor core truncates every sum it accumulates, which over S / 64 steps of 24 instructions would add up to an
// error proportional to the number of keys (7e-9 per key); so the output is taken out of TMEM into fp32 registers
// (round to nearest) every other step, and wherever a row's maximum has grown by more than 2^8 and it is rescaled.
// kAdd: a bias or a mask; what it adds to the logits is staged coalesced, 32 keys at a time.
// B8 H16 S1024 D64: 603 us on mma.sync (3 x TF32), here 182 + 26 for the planes; 204 with one query tile and single buffers
// for K and V, two CTAs per SM; causal with a bias per (batch, head) 775 -> 390.  Tensor core 65 % of the active cycles (ncu): bound by it and the waits of the two chains.
template <int kCols, bool kAdd>
__global__ void __launch_bounds__(FwdLayout<kCols, kAdd>::kThreads, 1) fwd_fp32_tc_kernel(const __grid_constant__ FwdArgs a) {
  using L = FwdLayout<kCols, kAdd>;
  constexpr int kSoftWarps = 4 * L::kTiles, kStages = L::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  int* abort_flag = reinterpret_cast<int*>(smem + L::kBars + 192);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kBars + 196);
  if (sbase & 1023) {   // (the swizzled tiles need it; the shared-memory window starts on such a boundary)
    if (threadIdx.x == 0) atomicExch(a.status, 300);
    return;
  }
  const Problem& pr = a.pr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh_local = blockIdx.y, bh = pr.bh_begin + bh_local, b = bh / pr.H, h = bh - b * pr.H;
  // (causal: the longest rows first)
  const int qc = pr.causal ? int(gridDim.x) - 1 - int(blockIdx.x) : int(blockIdx.x);
  const int qt0 = qc * a.tiles_per_cta;                        // first 128-row tile
  const int n_tiles = min(a.tiles_per_cta, (pr.S + 127) / 128 - qt0);
  auto steps_of = [&](int g) {
    const int t_end = pr.causal ? min(pr.T, min((qt0 + g + 1) * 128, pr.S)) : pr.T;
    return (t_end + kRows - 1) / kRows;
  };
  const int steps_max = steps_of(n_tiles - 1);
  auto bar = [&](int i) { return sbase + L::kBars + 8 * i; };
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < kFwdBars; ++i) {
      const bool rows = (i >= S_FREE && i < S_FREE + 2) || (i >= P_FULL && i < P_FULL + 2);
      const bool empty = (i >= K_EMPTY && i < K_EMPTY + 2) || (i >= V_EMPTY && i < V_EMPTY + 2);
      mbar_init(bar(i), rows ? 128 : (empty ? n_tiles : 1));
    }
    mbar_init_fence();
  }
  if (warp == kSoftWarps) {
    tmem_alloc(smem_u32(tmem_slot), L::kTmCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = *tmem_slot;

  if (warp == kSoftWarps) {
    if (elect_one()) {
      bool ok = true;
      // Q: up to two 64-row tiles per (plane, chunk), stacked into 128 rows
      for (int g = 0; g < n_tiles; ++g) {
        const int n_q = min(2, a.q_tiles - 2 * (qt0 + g));
        mbar_expect_tx(bar(Q_FULL + g), n_q * 3 * L::kPlane);
        for (int t = 0; t < n_q; ++t) {
          const uint8_t* src = a.q + (int64_t(bh_local) * a.q_tiles + 2 * (qt0 + g) + t) * (3 * L::kPlane);
          for (int i = 0; i < 3 * L::kChunks; ++i)
            bulk_load(sbase + L::kQ + g * L::kQBytes + (2 * i + t) * kChunkBytes, src + i * kChunkBytes, kChunkBytes, bar(Q_FULL + g));
        }
      }
      for (int j = 0; j < steps_max && ok; ++j) {
        const int st = j % kStages;
        const uint32_t ph = ((j / kStages) & 1) ^ 1;
        const int64_t at = (int64_t(bh_local) * a.k_tiles + j) * (3 * L::kPlane);
        ok = wait_or_abort(bar(K_EMPTY + st), ph, abort_flag, a.status, 301);
        if (!ok) break;
        mbar_expect_tx(bar(K_FULL + st), 3 * L::kPlane);
        bulk_load(sbase + L::kK + st * 3 * L::kPlane, a.k + at, 3 * L::kPlane, bar(K_FULL + st));
        ok = wait_or_abort(bar(V_EMPTY + st), ph, abort_flag, a.status, 302);
        if (!ok) break;
        mbar_expect_tx(bar(V_FULL + st), 3 * L::kPlane);
        bulk_load(sbase + L::kV + st * 3 * L::kPlane, a.v + at, 3 * L::kPlane, bar(V_FULL + st));
      }
      if (!ok) tc::drain_after_abort();
    }
  } else if (warp > kSoftWarps) {
    const int g = warp - kSoftWarps - 1;
    if (g < n_tiles && elect_one()) {
      constexpr uint32_t idesc_qk = make_idesc(true, 128, kRows, false, false);
      constexpr uint32_t idesc_pv = make_idesc(true, 128, kCols, false, true);
      const uint64_t qd = make_smem_desc(sbase + L::kQ + g * L::kQBytes, 16, 1024), kd0 = make_smem_desc(sbase + L::kK, 16, 1024);
      const uint64_t vd0 = make_smem_desc(sbase + L::kV, kChunkBytes, 1024);
      const uint32_t tg = tm + g * L::kTmTile;
      const int steps = steps_of(g);
      bool ok = wait_or_abort(bar(Q_FULL + g), 0, abort_flag, a.status, 303);
      // (a tile that is done before the CTA's last one still hands every stage back: one arrival per tile and phase)
      for (int j = 0; j <= steps_max && ok; ++j) {
        if (j < steps_max) {
          const int st = j % kStages;
          ok = wait_or_abort(bar(K_FULL + st), (j / kStages) & 1, abort_flag, a.status, 304);
          if (!ok) break;
          if (j < steps) {
            ok = j == 0 || wait_or_abort(bar(S_FREE + g), (j - 1) & 1, abort_flag, a.status, 305);
            if (!ok) break;
            tc_fence_after_sync();
            const uint64_t kd = kd0 + uint64_t((st * 3 * L::kPlane) >> 4);
#pragma unroll
            for (int i = 0; i < kProducts; ++i)
#pragma unroll
              for (int kk = 0; kk < kCols / 16; ++kk)
                mma_ss(tg + L::kTmS,
                       qd + uint64_t((left_plane(i) * 2 * L::kPlane + (kk / 4) * 2 * kChunkBytes + (kk % 4) * 32) >> 4),
                       kd + uint64_t((right_plane(i) * L::kPlane + (kk / 4) * kChunkBytes + (kk % 4) * 32) >> 4), idesc_qk,
                       i + kk > 0 ? 1u : 0u);
            mma_commit(bar(S_FULL + g));
            mma_commit(bar(K_EMPTY + st));
          } else {
            mbar_arrive(bar(K_EMPTY + st));
          }
        }
        if (j > 0) {
          const int st = (j - 1) % kStages;
          ok = wait_or_abort(bar(V_FULL + st), ((j - 1) / kStages) & 1, abort_flag, a.status, 306);
          if (!ok) break;
          if (j - 1 < steps) {
            ok = wait_or_abort(bar(P_FULL + g), (j - 1) & 1, abort_flag, a.status, 307);
            if (!ok) break;
            tc_fence_after_sync();
            const uint64_t vd = vd0 + uint64_t((st * 3 * L::kPlane) >> 4);
#pragma unroll
            for (int i = 0; i < kProducts; ++i)
#pragma unroll
              for (int kk = 0; kk < 4; ++kk)
                mma_ts(tg + L::kTmO, tg + L::kTmP + left_plane(i) * 32 + kk * 8,
                       vd + uint64_t((right_plane(i) * L::kPlane + kk * 2048) >> 4), idesc_pv, (j > 1 || i + kk > 0) ? 1u : 0u);
            mma_commit(bar(PV_DONE + g));
            mma_commit(bar(V_EMPTY + st));
          } else {
            mbar_arrive(bar(V_EMPTY + st));
          }
        }
      }
    }
  } else if ((warp >> 2) < n_tiles) {
    const int g = warp >> 2, quad = warp & 3;
    const int row0 = (qt0 + g) * 128 + quad * 32, row = row0 + lane;   // the warp's first row, this thread's
    const int steps = steps_of(g);
    const uint32_t tl = tm + g * L::kTmTile + (uint32_t(quad * 32) << 16);
    const float s2scale = pr.scale * kLog2e;
    float m = -INFINITY, l = 0.f;
    float* add = reinterpret_cast<float*>(smem + L::kAddend) + warp * 32 * kAddPitch;
    // what the bias and the mask add to the warp's 32 rows x 32 keys from key k0 on: a lane reads along a key; one row
    // stands for all where neither has a query axis
    const bool key_only = key_only_addends(pr);
    const int add_row = key_only ? 0 : lane * kAddPitch;
    auto stage_addends = [&](int k0) {
      const int key = k0 + lane;
      __syncwarp();
      if (key < pr.T) {
        const int64_t bo = b * pr.bs[0] + h * pr.bs[1] + key * pr.bs[3], mo = b * pr.ms[0] + h * pr.ms[1] + key * pr.ms[3];
        auto rows = [&](auto tag) {
          using BT = decltype(tag);
          auto stage = [&](int r) {
            const int64_t rr = min(row0 + r, pr.S - 1);
            float v = pr.bias ? kLog2e * to_f32<BT>(reinterpret_cast<const BT*>(pr.bias)[bo + rr * pr.bs[2]]) : 0.f;
            if (pr.mask && pr.mask[mo + rr * pr.ms[2]] == 0) v = __uint_as_float(kDropped);
            add[r * kAddPitch + lane] = v;
          };
          if (key_only) {
            stage(0);
          } else {
#pragma unroll
            for (int r = 0; r < 32; ++r) stage(r);
          }
        };
        if (a.bias_dtype == NB200_F32) rows(float{});
        else if (a.bias_dtype == NB200_BF16) rows(__nv_bfloat16{});
        else rows(__half{});
      }
      __syncwarp();
    };
    float o[kCols];
#pragma unroll
    for (int c = 0; c < kCols; ++c) o[c] = 0.f;
    bool ok = true;
    for (int j = 0; j < steps && ok; ++j) {
      const int kt = j * kRows;
      const int last = row < pr.S ? (pr.causal ? min(pr.T - 1, row) : pr.T - 1) - kt : -1;
      if constexpr (kAdd) {   // the first half's while the products run
        stage_addends(kt);
        if (j + 1 < steps && !key_only)
          prefetch_addends(pr, dtype_size(a.bias_dtype), b * pr.bs[0] + h * pr.bs[1], b * pr.ms[0] + h * pr.ms[1], row, kt + kRows, kRows);
      }
      ok = __all_sync(0xffffffffu, wait_or_abort(bar(S_FULL + g), j & 1, abort_flag, a.status, 308));
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t s[2][32];
      tmem_ld32(tl + L::kTmS, s[0]);
      tmem_ld32(tl + L::kTmS + 32, s[1]);
      tmem_wait_ld();
      tc_fence_before_sync();
      mbar_arrive(bar(S_FREE + g));
      // ---- logits in base 2 ----
      float mx = -INFINITY;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        if constexpr (kAdd) {
          // (fetched ahead into registers instead, these cost more in spills than the wait: 390 -> 714 us on the causal case above)
          if (half == 1) stage_addends(kt + 32);
        }
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const bool in = half * 32 + c <= last;
          float x = __uint_as_float(s[half][c]);
          if constexpr (kAdd) {
            const float v = add[add_row + c];   // (of a key past the end: never written)
            x = in && __float_as_uint(v) != kDropped ? fmaf(x, s2scale, v) : -INFINITY;
          } else {
            x = in ? x * s2scale : -INFINITY;
          }
          s[half][c] = __float_as_uint(x);
          mx = fmaxf(mx, x);
        }
      }
      // ---- online soft-max; the reference maximum moves only when some row of the warp has outgrown it by 2^8 ----
      const float m_new = fmaxf(m, mx);
      const bool move = __any_sync(0xffffffffu, m_new > m + kAbove);   // (true for the first kept key: m = -inf)
      float alpha = 1.f;
      if (move) {
        alpha = m_new == -INFINITY ? 1.f : tc::ex2(m - m_new);
        m = m_new;
        l *= alpha;
      }
      const float m_ref = m == -INFINITY ? 0.f : m + kAbove;        // nothing kept so far: every p is 0
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int c = 0; c < 32; ++c) {
          const float p = tc::ex2(__uint_as_float(s[half][c]) - m_ref);
          s[half][c] = __float_as_uint(p);
          sum[c & 3] += p;
        }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      if (j > 0) {
        ok = __all_sync(0xffffffffu, wait_or_abort(bar(PV_DONE + g), (j - 1) & 1, abort_flag, a.status, 309));
        if (!ok) break;
        tc_fence_after_sync();
        if (move || (j & 1) == 0) {
          uint32_t v[32];
#pragma unroll
          for (int c0 = 0; c0 < kCols; c0 += 32) {
            tmem_ld32(tl + L::kTmO + c0, v);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 32; ++c) {
              o[c0 + c] = (o[c0 + c] + __uint_as_float(v[c])) * alpha;
              v[c] = 0u;
            }
            tmem_st32(tl + L::kTmO + c0, v);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < 3; ++p) {
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          uint32_t w[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) w[c] = __byte_perm(s[half][2 * c], s[half][2 * c + 1], 0x7632);
          tmem_st16(tl + L::kTmP + p * 32 + half * 16, w);
          if (p < 2) {
#pragma unroll
            for (int c = 0; c < 32; ++c)
              s[half][c] = __float_as_uint(__uint_as_float(s[half][c]) - __uint_as_float(s[half][c] & 0xffff0000u));
          }
        }
      }
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(bar(P_FULL + g));
    }
    if (ok && steps > 0) {
      ok = __all_sync(0xffffffffu, wait_or_abort(bar(PV_DONE + g), (steps - 1) & 1, abort_flag, a.status, 310));
      tc_fence_after_sync();
    }
    // ---- out = o / l (NaN for a row with no kept key, as the reference's softmax gives), lse ----
    if (ok) {
      const float inv = 1.f / l;
      float* op = reinterpret_cast<float*>(pr.out) + b * pr.os[0] + h * pr.os[1] + int64_t(row) * pr.os[2];
      const bool vec = ((reinterpret_cast<uintptr_t>(pr.out) & 15) == 0) && ((pr.os[0] | pr.os[1] | pr.os[2]) & 3) == 0;
#pragma unroll
      for (int c0 = 0; c0 < kCols; c0 += 32) {
        uint32_t v[32];
        tmem_ld32(tl + L::kTmO + c0, v);
        tmem_wait_ld();
        if (row < pr.S && c0 < pr.Dv) {
#pragma unroll
          for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(l == 0.f ? NAN : (o[c0 + c] + __uint_as_float(v[c])) * inv);
          if (vec) {
#pragma unroll
            for (int c = 0; c < 32; c += 4) *reinterpret_cast<uint4*>(op + c0 + c) = make_uint4(v[c], v[c + 1], v[c + 2], v[c + 3]);
          } else {
#pragma unroll
            for (int c = 0; c < 32; ++c) op[c0 + c] = __uint_as_float(v[c]);
          }
        }
      }
      if (row < pr.S) pr.lse[(int64_t(b) * pr.H + h) * pr.S + row] = m + kAbove + log2f(l);
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == kSoftWarps) tmem_dealloc(tm, L::kTmCols);
}

// ---- backward -----------------------------------------------------------------------------------------------------
// One kernel, two owners.  Query-major (dq, dbias): a CTA owns 128 query rows and streams the keys; key-major (dk, dv): it
// owns 128 keys and streams the queries.  With X0, X1 the owner's rows of (q, dout) or (k, v) and Y0, Y1 a 64-row step of
// the other pair, per step
//     S = X0 Y0^T,  dP = X1 Y1^T,   p = exp2(S scale log2 e + addend - lse),  ds = p (dP - delta),
//     dq += ds Y0     or     dk += ds Y0, dv += p Y1        (p and ds as three planes in TMEM)
// Warps 0-7: element-wise, warps 0-3 the first 32 columns of a step, 4-7 the other 32, a thread per row; warp 8 fetches,
// warp 9 issues the products, warp 10 the accumulates (a step is 72 or 96 MMA instructions, and one thread issuing them
// all would take longer than the tensor core).  S and dP go to registers at once, so the next step's products run under
// this step's arithmetic.  As in the forward the accumulators are emptied every other step into fp32 sums: dq's in
// registers, dk's in shared memory, dv's in TMEM (what each kernel has left).  Those and a dense dbias are summed in a
// fixed order; a broadcast bias' gradient is added by many CTAs with fp32 atomics.
// B8 H16 S1024 D64, both kernels and the planes: 2019 us on mma.sync, here 679 -- query-major 241 (302 with q and dout in
// shared memory), key-major 403 (a step's 48 products at 48 cycles and 48 accumulates at 32 are 224 us).
struct BwdArgs {
  Problem pr;
  const uint8_t *x0, *x1, *y0, *y1;
  int x_tiles, y_tiles;         // 64-row tiles per (b, h)
  int bias_dtype;
  int* status;
};
// The products read their owner operand from TMEM in the query-major kernel (its warps split their own rows of q and dout
// on the way in): a product of two shared-memory operands at N = 64 fetches 6 KB for 32 cycles of the tensor core, which
// shared memory takes 48 cycles to deliver.  The key-major kernel has no TMEM left for that.
template <bool kKeyMajor>
struct BwdLayout {
  static constexpr int kPlane = kChunkBytes;                   // 64 columns
  static constexpr int kStages = kKeyMajor ? 2 : 4;
  static constexpr int kX = 0;                                 // key-major: [K, V][3][128 rows x 128 B]
  static constexpr int kY = kX + (kKeyMajor ? 2 * 3 * 2 * kPlane : 0);   // [kStages][Y0, Y1][3][64 rows x 128 B]
  static constexpr int kStageBytes = 2 * 3 * kPlane;
  // query-major: addends in and ds out, [8 warps][32 rows][kAddPitch]; key-major: lse and delta, [2 stages][2][64], then the
  // sums of dk, [32 columns][256 threads]
  static constexpr int kSide = kY + kStages * kStageBytes;
  static constexpr int kSumDk = kSide + 2 * 2 * 64 * 4;
  static constexpr int kBars = kKeyMajor ? kSumDk + 32 * 256 * 4 : kSide + 8 * 32 * kAddPitch * 4;
  static constexpr int kBytes = kBars + 256;
  // TMEM: S, dP, planes of ds; then key-major: planes of p, accumulators, sum of dv; query-major: planes of q and dout,
  // accumulator
  static constexpr int kTmS = 0, kTmDP = 64, kTmDS = 128, kTmP = 224, kTmX = 224, kTmAcc = kKeyMajor ? 320 : 416;
  static constexpr int kTmAcc2 = 384, kTmSum2 = 448, kTmCols = 512;
};
enum BwdBar { Y_FULL = 0, Y_EMPTY = 4, L_FULL = 8, X_FULL = 10, SP_FULL, SP_FREE, PD_FULL, ACC_DONE, kBwdBars };

template <bool kKeyMajor, bool kAdd>
__global__ void __launch_bounds__(352, 1) bwd_fp32_tc_kernel(const __grid_constant__ BwdArgs a) {
  using L = BwdLayout<kKeyMajor>;
  constexpr int kStages = L::kStages;
  extern __shared__ __align__(1024) uint8_t smem[];
  const uint32_t sbase = smem_u32(smem);
  int* abort_flag = reinterpret_cast<int*>(smem + L::kBars + 192);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::kBars + 196);
  if (sbase & 1023) {
    if (threadIdx.x == 0) atomicExch(a.status, 320);
    return;
  }
  const Problem& pr = a.pr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh_local = blockIdx.y, bh = pr.bh_begin + bh_local, b = bh / pr.H, h = bh - b * pr.H;
  // (causal: the owners with the longest walk first)
  const int xt = (!kKeyMajor && pr.causal) ? int(gridDim.x) - 1 - int(blockIdx.x) : int(blockIdx.x);
  const int x_row0 = xt * 128;
  // steps [j0, j1) of the other operand
  const int j0 = (kKeyMajor && pr.causal) ? min(a.y_tiles, x_row0 / kRows) : 0;
  const int j1 = (!kKeyMajor && pr.causal) ? min(a.y_tiles, (min(x_row0 + 128, pr.S) + kRows - 1) / kRows) : a.y_tiles;
  const int steps = max(0, j1 - j0);
  auto bar = [&](int i) { return sbase + L::kBars + 8 * i; };
  if (threadIdx.x == 0) {
    *abort_flag = 0;
    for (int i = 0; i < kBwdBars; ++i)
      mbar_init(bar(i), i == SP_FREE || i == PD_FULL || (!kKeyMajor && i == X_FULL) ? 256 : (i == L_FULL || i == L_FULL + 1 ? 32 : 1));
    mbar_init_fence();
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(tmem_slot), L::kTmCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tm = *tmem_slot;

  if (warp == 8) {
    bool ok = true;
    if (kKeyMajor && lane == 0 && steps > 0) {
      const int n_x = min(2, a.x_tiles - 2 * xt);
      mbar_expect_tx(bar(X_FULL), n_x * 2 * 3 * L::kPlane);
      for (int w = 0; w < 2; ++w)
        for (int t = 0; t < n_x; ++t) {
          const uint8_t* src = (w ? a.x1 : a.x0) + (int64_t(bh_local) * a.x_tiles + 2 * xt + t) * (3 * L::kPlane);
          for (int i = 0; i < 3; ++i)
            bulk_load(sbase + L::kX + ((w * 3 + i) * 2 + t) * L::kPlane, src + i * L::kPlane, L::kPlane, bar(X_FULL));
        }
    }
    __syncwarp();
    for (int i = 0; i < steps && ok; ++i) {
      const int st = i % kStages, j = j0 + i;
      ok = __all_sync(0xffffffffu, wait_or_abort(bar(Y_EMPTY + st), ((i / kStages) & 1) ^ 1, abort_flag, a.status, 321));
      if (!ok) break;
      if (lane == 0) {
        const int64_t at = (int64_t(bh_local) * a.y_tiles + j) * (3 * L::kPlane);
        mbar_expect_tx(bar(Y_FULL + st), L::kStageBytes);
        bulk_load(sbase + L::kY + st * L::kStageBytes, a.y0 + at, 3 * L::kPlane, bar(Y_FULL + st));
        bulk_load(sbase + L::kY + st * L::kStageBytes + 3 * L::kPlane, a.y1 + at, 3 * L::kPlane, bar(Y_FULL + st));
      }
      if constexpr (kKeyMajor) {
        // (zeros past the last query: those rows of q and dout are zeros as well)
        float* side = reinterpret_cast<float*>(smem + L::kSide) + st * 128;
        for (int q = lane; q < kRows; q += 32) {
          const int row = j * kRows + q;
          const int64_t at = (int64_t(b) * pr.H + h) * pr.S + row;
          side[q] = row < pr.S ? pr.lse[at] : 0.f;
          side[64 + q] = row < pr.S ? pr.delta[at] : 0.f;
        }
        mbar_arrive(bar(L_FULL + st));
      }
    }
    if (!ok) tc::drain_after_abort();
  } else if (warp == 9) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(true, 128, kRows, false, false);
      const uint64_t x0 = make_smem_desc(sbase + L::kX, 16, 1024);
      const uint64_t y0 = make_smem_desc(sbase + L::kY, 16, 1024);
      bool ok = steps == 0 || wait_or_abort(bar(X_FULL), 0, abort_flag, a.status, 323);
      for (int i = 0; i < steps && ok; ++i) {
        const int st = i % kStages;
        ok = wait_or_abort(bar(Y_FULL + st), (i / kStages) & 1, abort_flag, a.status, 324) &&
             (i == 0 || wait_or_abort(bar(SP_FREE), (i - 1) & 1, abort_flag, a.status, 325));
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t ys = y0 + uint64_t((st * L::kStageBytes) >> 4);
#pragma unroll
        for (int w = 0; w < 2; ++w)
#pragma unroll
          for (int t = 0; t < kProducts; ++t)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              if constexpr (kKeyMajor)
                mma_ss(tm + (w ? L::kTmDP : L::kTmS),
                       x0 + uint64_t(((w * 3 + left_plane(t)) * 2 * L::kPlane + kk * 32) >> 4),
                       ys + uint64_t(((w * 3 + right_plane(t)) * L::kPlane + kk * 32) >> 4), idesc, t + kk > 0 ? 1u : 0u);
              else
                mma_ts(tm + (w ? L::kTmDP : L::kTmS), tm + L::kTmX + (w * 3 + left_plane(t)) * 32 + kk * 8,
                       ys + uint64_t(((w * 3 + right_plane(t)) * L::kPlane + kk * 32) >> 4), idesc, t + kk > 0 ? 1u : 0u);
        mma_commit(bar(SP_FULL));
      }
    }
  } else if (warp == 10) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc(true, 128, 64, false, true);
      const uint64_t y0 = make_smem_desc(sbase + L::kY, L::kPlane, 1024);
      bool ok = true;
      for (int i = 0; i < steps && ok; ++i) {
        const int st = i % kStages;
        ok = wait_or_abort(bar(Y_FULL + st), (i / kStages) & 1, abort_flag, a.status, 331) &&
             wait_or_abort(bar(PD_FULL), i & 1, abort_flag, a.status, 326);
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t ys = y0 + uint64_t((st * L::kStageBytes) >> 4);
#pragma unroll
        for (int w = 0; w < (kKeyMajor ? 2 : 1); ++w)      // ds Y0, then p Y1
#pragma unroll
          for (int t = 0; t < kProducts; ++t)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              mma_ts(tm + (w ? L::kTmAcc2 : L::kTmAcc), tm + (w ? L::kTmP : L::kTmDS) + left_plane(t) * 32 + kk * 8,
                     ys + uint64_t(((w * 3 + right_plane(t)) * L::kPlane + kk * 2048) >> 4), idesc,
                     (i > 0 || t + kk > 0) ? 1u : 0u);
        mma_commit(bar(Y_EMPTY + st));
        mma_commit(bar(ACC_DONE));
      }
    }
  } else {
    const int half = warp >> 2, quad = warp & 3;
    const int x_row = x_row0 + quad * 32 + lane;             // this thread's query (query-major) or key
    const uint32_t tl = tm + (uint32_t(quad * 32) << 16);
    const float s2scale = pr.scale * kLog2e;
    const int x_rows = kKeyMajor ? pr.T : pr.S;
    float lse = 0.f, delta = 0.f;
    if (!kKeyMajor && x_row < pr.S) {
      const int64_t at = (int64_t(b) * pr.H + h) * pr.S + x_row;
      lse = pr.lse[at];
      delta = pr.delta[at];
    }
    float* stage = reinterpret_cast<float*>(smem + L::kSide) + warp * 32 * kAddPitch;
    const bool want_db = !kKeyMajor && (pr.dbias != nullptr || pr.dbias_accum != nullptr);
    const bool key_only = key_only_addends(pr);
    const int add_row = key_only ? 0 : lane * kAddPitch;
    const int64_t b_base = b * pr.bs[0] + h * pr.bs[1], m_base = b * pr.ms[0] + h * pr.ms[1];
    const int64_t db_base = b * pr.dbs[0] + h * pr.dbs[1];
    if constexpr (!kKeyMajor) {
      // this thread's row of q (warps 0-3) or dout (4-7), split into TMEM
      const float* xp = reinterpret_cast<const float*>(half ? pr.dout : pr.q);
      const int64_t* xs = half ? pr.dos : pr.qs;
      const bool vec = ((reinterpret_cast<uintptr_t>(xp) & 15) == 0) && ((xs[0] | xs[1] | xs[2]) & 3) == 0;
      xp += b * xs[0] + h * xs[1] + int64_t(x_row) * xs[2];
      uint32_t x[64];
#pragma unroll
      for (int c = 0; c < 64; ++c) x[c] = 0u;
      if (x_row < pr.S) {
#pragma unroll
        for (int c = 0; c < 64; c += 4) {
          if (c >= pr.D) break;
          if (vec) {
            const uint4 v = *reinterpret_cast<const uint4*>(xp + c);
            x[c] = v.x; x[c + 1] = v.y; x[c + 2] = v.z; x[c + 3] = v.w;
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) x[c + e] = __float_as_uint(xp[c + e]);
          }
        }
      }
#pragma unroll
      for (int p = 0; p < 3; ++p) {
        uint32_t o[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) o[c] = __byte_perm(x[2 * c], x[2 * c + 1], 0x7632);
        tmem_st32(tl + L::kTmX + (half * 3 + p) * 32, o);
        if (p < 2) {
#pragma unroll
          for (int c = 0; c < 64; ++c)
            x[c] = __float_as_uint(__uint_as_float(x[c]) - __uint_as_float(x[c] & 0xffff0000u));
        }
      }
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(bar(X_FULL));
    }
    float sum[32];                                           // of dq, this thread's row and 32 columns
    float* sum_dk = reinterpret_cast<float*>(smem + L::kSumDk) + threadIdx.x;   // of dk, a column every 256
#pragma unroll
    for (int c = 0; c < 32; ++c) {
      if constexpr (kKeyMajor) sum_dk[c * 256] = 0.f;
      else sum[c] = 0.f;
    }
    bool ok = true;
    for (int i = 0; i < steps && ok; ++i) {
      const int y_row0 = (j0 + i) * kRows + half * 32;       // first of this warp's 32 columns
      // ---- what bias and mask add to the logits, in flight while the products run ----
      float add[32];
      if constexpr (kAdd) {
        auto fetch = [&](auto tag) {
          using BT = decltype(tag);
          if constexpr (kKeyMajor) {
            // lanes are neighbouring keys: read along a row of the bias / mask
            const int64_t key = min(x_row, pr.T - 1);
            if (key_only) {
              float v = pr.bias ? kLog2e * to_f32<BT>(reinterpret_cast<const BT*>(pr.bias)[b_base + key * pr.bs[3]]) : 0.f;
              if (pr.mask && pr.mask[m_base + key * pr.ms[3]] == 0) v = __uint_as_float(kDropped);
#pragma unroll
              for (int c = 0; c < 32; ++c) add[c] = v;
            } else {
#pragma unroll
              for (int c = 0; c < 32; ++c) {
                const int64_t q = min(y_row0 + c, pr.S - 1);
                add[c] = pr.bias ? kLog2e * to_f32<BT>(reinterpret_cast<const BT*>(pr.bias)[b_base + q * pr.bs[2] + key * pr.bs[3]]) : 0.f;
                if (pr.mask && pr.mask[m_base + q * pr.ms[2] + key * pr.ms[3]] == 0) add[c] = __uint_as_float(kDropped);
              }
            }
          } else {
            // a lane per key here, then a lane per query row through shared memory
            const int64_t key = min(y_row0 + lane, pr.T - 1);
            __syncwarp();
#pragma unroll 16
            for (int r = 0; r < (key_only ? 1 : 32); ++r) {
              const int64_t q = min(x_row0 + quad * 32 + r, pr.S - 1);
              float v = pr.bias ? kLog2e * to_f32<BT>(reinterpret_cast<const BT*>(pr.bias)[b_base + q * pr.bs[2] + key * pr.bs[3]]) : 0.f;
              if (pr.mask && pr.mask[m_base + q * pr.ms[2] + key * pr.ms[3]] == 0) v = __uint_as_float(kDropped);
              stage[r * kAddPitch + lane] = v;
            }
            __syncwarp();
          }
        };
        if (a.bias_dtype == NB200_F32) fetch(float{});
        else if (a.bias_dtype == NB200_BF16) fetch(__nv_bfloat16{});
        else fetch(__half{});
        if (i + 1 < steps && !key_only)
          prefetch_addends(pr, dtype_size(a.bias_dtype), b_base, m_base, kKeyMajor ? y_row0 + kRows + lane : x_row,
                           kKeyMajor ? x_row0 + quad * 32 : y_row0 + kRows, 32);
      }
      ok = __all_sync(0xffffffffu, wait_or_abort(bar(SP_FULL), i & 1, abort_flag, a.status, 327) &&
                                       (!kKeyMajor || wait_or_abort(bar(L_FULL + (i & 1)), (i >> 1) & 1, abort_flag, a.status, 328)));
      if (!ok) break;
      tc_fence_after_sync();
      uint32_t s[32], d[32];
      tmem_ld32(tl + L::kTmS + half * 32, s);
      tmem_ld32(tl + L::kTmDP + half * 32, d);
      tmem_wait_ld();
      tc_fence_before_sync();
      mbar_arrive(bar(SP_FREE));
      const float* side = reinterpret_cast<const float*>(smem + L::kSide) + (i & 1) * 128 + half * 32;
      // columns kept: query-major c <= last; key-major the queries from `first` on, none for a row past the last key
      const int last = x_row < pr.S ? (pr.causal ? min(pr.T - 1, x_row) : pr.T - 1) - y_row0 : -1;
      const int first = x_row < pr.T ? (pr.causal ? x_row - y_row0 : 0) : 64;
#pragma unroll
      for (int c = 0; c < 32; ++c) {
        const bool in = kKeyMajor ? (c >= first && y_row0 + c < pr.S) : c <= last;
        const float ref = kKeyMajor ? side[c] : lse, dl = kKeyMajor ? side[64 + c] : delta;
        float x = __uint_as_float(s[c]);
        bool keep = in;
        if constexpr (kAdd) {
          const float v = kKeyMajor ? add[c] : stage[add_row + c];
          keep = in && __float_as_uint(v) != kDropped;
          x = fmaf(x, s2scale, v) - ref;
        } else {
          x = fmaf(x, s2scale, -ref);
        }
        const float p = keep ? tc::ex2(x) : 0.f;
        s[c] = __float_as_uint(p);
        d[c] = __float_as_uint(p * (__uint_as_float(d[c]) - dl));
      }
      if (want_db) {
        // ds out: a lane per row in, a lane per key out
        __syncwarp();
#pragma unroll
        for (int c = 0; c < 32; ++c) stage[lane * kAddPitch + c] = __uint_as_float(d[c]);
        __syncwarp();
        const int key = y_row0 + lane;
        if (key < pr.T) {
          const int n = min(32, pr.S - (x_row0 + quad * 32));
          const float* from = stage + lane;
          const int64_t at = db_base + int64_t(x_row0 + quad * 32) * pr.dbs[2] + key * pr.dbs[3];
          if (pr.dbias_accum) {
            float* to = pr.dbias_accum + at;
            if (pr.dbs[2] == 0) {                  // summed over the queries: the warp's rows first
              float v = 0.f;
              for (int r = 0; r < n; ++r) v += from[r * kAddPitch];
              if (n > 0) atomicAdd(to, v);
            } else {
#pragma unroll 8
              for (int r = 0; r < n; ++r) atomicAdd(to + r * pr.dbs[2], from[r * kAddPitch]);
            }
          } else if (a.bias_dtype == NB200_F32) {
            float* to = reinterpret_cast<float*>(pr.dbias) + at;
#pragma unroll 8
            for (int r = 0; r < n; ++r) to[r * pr.dbs[2]] = from[r * kAddPitch];
          } else {
            for (int r = 0; r < n; ++r) store_from_f32(pr.dbias, at + r * pr.dbs[2], a.bias_dtype, from[r * kAddPitch]);
          }
        }
      }
      if (i > 0) {
        ok = __all_sync(0xffffffffu, wait_or_abort(bar(ACC_DONE), (i - 1) & 1, abort_flag, a.status, 329));
        if (!ok) break;
        tc_fence_after_sync();
        if ((i & 1) == 0) {
          uint32_t v[32];
          tmem_ld32(tl + L::kTmAcc + half * 32, v);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            if constexpr (kKeyMajor) sum_dk[c * 256] += __uint_as_float(v[c]);
            else sum[c] += __uint_as_float(v[c]);
            v[c] = 0u;
          }
          tmem_st32(tl + L::kTmAcc + half * 32, v);
        } else if (kKeyMajor && i > 1) {
          uint32_t v[32], w[32];
          tmem_ld32(tl + L::kTmAcc2 + half * 32, v);
          if (i > 3) tmem_ld32(tl + L::kTmSum2 + half * 32, w);
          tmem_wait_ld();
#pragma unroll
          for (int c = 0; c < 32; ++c) {
            w[c] = i > 3 ? __float_as_uint(__uint_as_float(w[c]) + __uint_as_float(v[c])) : v[c];
            v[c] = 0u;
          }
          tmem_st32(tl + L::kTmSum2 + half * 32, w);
          tmem_st32(tl + L::kTmAcc2 + half * 32, v);
        }
      }
#pragma unroll
      for (int w = 0; w < (kKeyMajor ? 2 : 1); ++w) {
        uint32_t(&v)[32] = w ? s : d;
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          uint32_t o[16];
#pragma unroll
          for (int c = 0; c < 16; ++c) o[c] = __byte_perm(v[2 * c], v[2 * c + 1], 0x7632);
          tmem_st16(tl + (w ? L::kTmP : L::kTmDS) + p * 32 + half * 16, o);
          if (p < 2) {
#pragma unroll
            for (int c = 0; c < 32; ++c)
              v[c] = __float_as_uint(__uint_as_float(v[c]) - __uint_as_float(v[c] & 0xffff0000u));
          }
        }
      }
      tmem_wait_st();
      tc_fence_before_sync();
      mbar_arrive(bar(PD_FULL));
    }
    if (ok && steps > 0) {
      ok = __all_sync(0xffffffffu, wait_or_abort(bar(ACC_DONE), (steps - 1) & 1, abort_flag, a.status, 330));
      tc_fence_after_sync();
    }
    if (ok && half * 32 < pr.D) {
#pragma unroll
      for (int w = 0; w < (kKeyMajor ? 2 : 1); ++w) {
        void* base = kKeyMajor ? (w ? pr.dv : pr.dk) : pr.dq;
        const int64_t* st3 = kKeyMajor ? (w ? pr.dvs : pr.dks) : pr.dqs;
        const float scale = w ? 1.f : pr.scale;
        uint32_t o[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) o[c] = 0u;
        if (steps > 0) {
          tmem_ld32(tl + (w ? L::kTmAcc2 : L::kTmAcc) + half * 32, o);
          tmem_wait_ld();
          if (w == 0) {
#pragma unroll
            for (int c = 0; c < 32; ++c) o[c] = __float_as_uint((kKeyMajor ? sum_dk[c * 256] : sum[c]) + __uint_as_float(o[c]));
          } else if (steps > 3) {
            uint32_t t[32];
            tmem_ld32(tl + L::kTmSum2 + half * 32, t);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(t[c]) + __uint_as_float(o[c]));
          }
        }
        if (x_row < x_rows) {
          float* op = reinterpret_cast<float*>(base) + b * st3[0] + h * st3[1] + int64_t(x_row) * st3[2] + half * 32;
#pragma unroll
          for (int c = 0; c < 32; ++c) o[c] = __float_as_uint(__uint_as_float(o[c]) * scale);
          if (((reinterpret_cast<uintptr_t>(base) & 15) == 0) && ((st3[0] | st3[1] | st3[2]) & 3) == 0) {
#pragma unroll
            for (int c = 0; c < 32; c += 4) *reinterpret_cast<uint4*>(op + c) = make_uint4(o[c], o[c + 1], o[c + 2], o[c + 3]);
          } else {
#pragma unroll
            for (int c = 0; c < 32; ++c) op[c] = __uint_as_float(o[c]);
          }
        }
      }
    }
    // causal rows never visit keys past the CTA's last row, yet a dense dbias is written everywhere: exact zeros
    if (ok && want_db && !pr.dbias_accum) {
      for (int r = warp; r < min(128, pr.S - x_row0); r += 8)
        for (int key = j1 * kRows + lane; key < pr.T; key += 32)
          store_from_f32(pr.dbias, db_base + int64_t(x_row0 + r) * pr.dbs[2] + key * pr.dbs[3], a.bias_dtype, 0.f);
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (warp == 9) tmem_dealloc(tm, L::kTmCols);
}

int padded_cols(int d) { return d <= 64 ? 64 : 128; }
int64_t tiles_of(int rows) { return (int64_t(rows) + kRows - 1) / kRows; }
size_t plane_bytes(const Problem& pr, int rows) {
  return size_t(pr.bh_count) * tiles_of(rows) * 3 * (padded_cols(pr.D) / 64) * kChunkBytes;
}

// The planes of a large problem are made and used for a range of (b, h) at a time, so that they take 1 GiB at most (or one
// (b, h)): 900 pairs of S = T = 1024, D = 64.  A range is many waves of CTAs.
constexpr size_t kPlanesLimit = size_t(1) << 30;
Problem part_of(const Problem& pr, size_t bytes_per_bh, int done) {
  const size_t fit = kPlanesLimit / bytes_per_bh;
  Problem part = pr;
  part.bh_begin = pr.bh_begin + done;
  const int64_t left = pr.bh_count - done, most = fit > 1 ? int64_t(fit) : 1;
  part.bh_count = int(left < most ? left : most);
  return part;
}
size_t fwd_bytes_per_bh(const Problem& pr) { return (plane_bytes(pr, pr.S) + 2 * plane_bytes(pr, pr.T)) / pr.bh_count; }
size_t bwd_bytes_per_bh(const Problem& pr) { return 2 * (plane_bytes(pr, pr.S) + plane_bytes(pr, pr.T)) / pr.bh_count; }

int launch_split(const Problem& pr, const SplitArgs& sa, int operands, cudaStream_t st) {
  int tiles = 1;
  for (int i = 0; i < operands; ++i) tiles = sa.op[i].tiles > tiles ? sa.op[i].tiles : tiles;
  const dim3 grid(tiles, pr.bh_count, operands);
  if (padded_cols(pr.D) == 64) split_planes_kernel<64><<<grid, 128, 0, st>>>(sa);
  else split_planes_kernel<128><<<grid, 128, 0, st>>>(sa);
  count_launch();
  return check_launch("split_planes_kernel");
}

SplitOperand operand(const void* x, const int64_t* strides, int rows, uint8_t* planes) {
  SplitOperand o{};
  o.x = static_cast<const float*>(x);
  o.planes = planes;
  for (int i = 0; i < 3; ++i) o.xs[i] = strides[i];
  o.rows = rows;
  o.tiles = int(tiles_of(rows));
  return o;
}

template <int kCols, bool kAdd>
int launch_fwd(const FwdArgs& a, cudaStream_t st) {
  using L = FwdLayout<kCols, kAdd>;
  auto kernel = fwd_fp32_tc_kernel<kCols, kAdd>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes) != cudaSuccess) {
    set_error("fwd_fp32_tc_kernel: cudaFuncSetAttribute(%d): %s", L::kBytes, cudaGetErrorString(cudaGetLastError()));
    return NB200_ERR_LAUNCH;
  }
  // two query tiles per CTA, which share the fetched keys, once one per CTA would be more than one wave
  FwdArgs args = a;
  const int tiles = (a.pr.S + 127) / 128;
  args.tiles_per_cta = L::kTiles == 2 && int64_t(tiles) * a.pr.bh_count > tc::sm_count() ? 2 : 1;
  kernel<<<dim3((tiles + args.tiles_per_cta - 1) / args.tiles_per_cta, a.pr.bh_count), L::kThreads, L::kBytes, st>>>(args);
  count_launch();
  return check_launch("fwd_fp32_tc_kernel");
}

template <bool kKeyMajor, bool kAdd>
int launch_bwd(const BwdArgs& a, cudaStream_t st) {
  using L = BwdLayout<kKeyMajor>;
  auto kernel = bwd_fp32_tc_kernel<kKeyMajor, kAdd>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::kBytes) != cudaSuccess) {
    set_error("bwd_fp32_tc_kernel: cudaFuncSetAttribute(%d): %s", L::kBytes, cudaGetErrorString(cudaGetLastError()));
    return NB200_ERR_LAUNCH;
  }
  kernel<<<dim3(((kKeyMajor ? a.pr.T : a.pr.S) + 127) / 128, a.pr.bh_count), 352, L::kBytes, st>>>(a);
  count_launch();
  return check_launch(kKeyMajor ? "bwd_dkv_fp32_tc_kernel" : "bwd_dq_fp32_tc_kernel");
}

}  // namespace

namespace {
bool takes(const Problem& pr) {
  return (pr.D == 32 || pr.D == 64 || pr.D == 128) && pr.D == pr.Dv && pr.S > 0 && pr.T > 0 && pr.bh_count > 0 &&
         pr.bh_count <= 65535;
}
// a bias or a mask that has to be read per query
bool row_addends(const Problem& pr) { return (pr.bias && pr.bs[2] != 0) || (pr.mask && pr.ms[2] != 0); }
int64_t owners_of(int rows) { return (int64_t(rows) + 127) / 128; }
}  // namespace

// Where these kernels win over the mma.sync ones.  A CTA here is 128 rows and has an SM to itself, and a call costs a launch
// for the planes; the others run 64-row CTAs, several to an SM, and split the keys of a small problem over warps or
// clusters.  So: enough tiles for the SMs, enough work behind the start, more with a bias or a mask per query (read by the
// warps that do the soft-max).  Half of the tensor work at head dim 32 is padding to 64, and the others gain most of that
// back unless the addends, which cost them more, are both there.  Forward, us, here / there:
//  D 64: B1 H1 S1536 40 / 26, B1 H4 S1024 31 / 31, the same causal with a key mask 50 / 37, B2 H4 S256 bias, mask 27 / 18,
//   B8 H8 S128 12.6 / 9.4, B64 H8 S64 33 / 17, B32 H16 S64 T512 121 / 93, B8 H16 S17 T1000 78 / 53, B24 H8 S128 24.4 / 22.5
//   <  the line  <  B4 H8 S256 15.4 / 15.7, with key bias and mask 19.9 / 20.1, B8 H8 S192 15 / 23, B4 H6 S344 18 / 21, B16 H8
//   S128 14 / 16, B1 H8 S1024 31 / 45, B16 H8 S200 bias 42 / 74, B8 H8 S300 T700 key bias and mask 56 / 184, B8 H16 S1024 208
//   / 603, the same with a key mask 293 / 810, causal with bias 390 / 775
//  D 32: B4 H8 S512 bias 57 / 46, B24 H8 S192 34 / 22, B16 H8 S100 T1500 75 / 70, B6 H8 S512 T100 30 / 22, B4 H8 S200 bias and
//   mask 1.6 times, causal B32 H8 S344 1.18, B5 H8 S773 T148 bias per query and key mask 45 / 33, B37 H8 S560 mask 430 / 389  <  the line  <  B4 H8 S512 22.5 / 28.9, B4 H8 S344 0.76 times (B12 H8 1.07), B4 H8 S1024 49.6 / 93.8, with bias 0.8 times, B16 H8 S512 bias 0.85
//   times, B12 H8 S256 bias and mask 0.7 times, B4 H8 S1000 T100 bias and mask 0.77, B16 H8 S200 key bias and mask 28.6 / 36.7
//  D 128: B1 H1 S33 T65 5.2 / 5.6; 128 pairs of S40 T80 20.6 / 16.8, S48 T300 41.7 / 36.3, S48 T1000 124.6 / 105.8; B32 H8 S64
//   T64 26 / 19  <  the line  <  32 pairs of S48 T300 0.77 times, 128 with bias 0.97, B1 H1 S128 T1536 84 / 147, B4 H8 S48 T700
//   49 / 71, B1 H4 S512 35 / 53, B2 H8 S1536 184 / 449.
bool fp32_tc_fwd_applies(const Problem& pr) {
  if (!takes(pr) || pr.T <= kRows) return false;
  const bool none = !pr.bias && !pr.mask;
  const int64_t owners = owners_of(pr.S) * pr.bh_count, area = int64_t(pr.S) * pr.T;
  if (pr.D == 128) {
    if (pr.S <= kRows / 2) return false;
    return pr.S > kRows || owners <= 64 || (!none && pr.T >= 256);
  }
  if (pr.S <= kRows) return false;   // (half of a 128-row tile at least would be padding)
  if (pr.D == 32) {
    const int least = pr.S < pr.T ? pr.S : pr.T;
    const bool row = row_addends(pr);
    if (pr.bias && pr.mask) {
      const bool alike = (pr.bs[2] != 0) == (pr.ms[2] != 0);   // (else one of the two costs the others little)
      return (least >= 200 || (alike && (least > 128 || pr.S >= 512))) && area >= 40000 && owners >= (row ? 192 : 96);
    }
    if (row) return least >= 300 && pr.S >= 512 && owners >= 192 && (pr.bias || area >= 500000);
    return least >= 200 && (pr.causal ? area / 2 : area) >= 100000 && owners >= 96;
  }
  const int64_t ctas = tiles_of(pr.S) * pr.bh_count, work = ctas * tiles_of(pr.T);
  if (row_addends(pr)) return ctas >= 192 && work >= 1024;
  if (none && pr.S <= 128 && pr.T <= 128 && pr.bh_count > 148) return false;   // (short CTAs in more than one wave)
  return ctas >= 128 && work >= 512;
}

size_t fp32_tc_fwd_bytes(const Problem& pr) {
  const size_t each = fwd_bytes_per_bh(pr);
  return each * part_of(pr, each, 0).bh_count;
}

namespace {
int forward_part(const Problem& pr, int bias_dtype, void* ws, cudaStream_t st) {
  uint8_t* base = static_cast<uint8_t*>(ws);
  FwdArgs a{};
  a.pr = pr;
  a.bias_dtype = bias_dtype;
  a.q_tiles = int(tiles_of(pr.S));
  a.k_tiles = int(tiles_of(pr.T));
  uint8_t* planes[3] = {base, base + plane_bytes(pr, pr.S), base + plane_bytes(pr, pr.S) + plane_bytes(pr, pr.T)};
  a.q = planes[0];
  a.k = planes[1];
  a.v = planes[2];
  a.status = device_status_word();
  if (!a.status) { set_error("device status word is unavailable"); return NB200_ERR_LAUNCH; }
  SplitArgs sa{};
  sa.H = pr.H;
  sa.bh_begin = pr.bh_begin;
  sa.D = pr.D;
  sa.op[0] = operand(pr.q, pr.qs, pr.S, planes[0]);
  sa.op[1] = operand(pr.k, pr.ks, pr.T, planes[1]);
  sa.op[2] = operand(pr.v, pr.vs, pr.T, planes[2]);
  if (int rc = launch_split(pr, sa, 3, st)) return rc;
  const bool add = pr.bias || pr.mask;
  if (padded_cols(pr.D) == 64) return add ? launch_fwd<64, true>(a, st) : launch_fwd<64, false>(a, st);
  return add ? launch_fwd<128, true>(a, st) : launch_fwd<128, false>(a, st);
}
}  // namespace

int fp32_tc_forward(const Problem& pr, int bias_dtype, void* ws, cudaStream_t st) {
  for (int done = 0; done < pr.bh_count;) {
    const Problem part = part_of(pr, fwd_bytes_per_bh(pr), done);
    if (int rc = forward_part(part, bias_dtype, ws, st)) return rc;
    done += part.bh_count;
  }
  return NB200_OK;
}

// Head dim 128 stays with the other kernels: the planes of an owner's two operands would be 192 KB of shared memory.
// Backward, us, here / there (D 64 unless said): B1 H1 S1536 120 / 67, B2 H4 S256 bias, mask 73 / 33, B64 H8 S64 81 / 60,
//   B4 H8 S65 26 / 23, B4 H8 S128 31 / 29, B4 H8 S256 D32 35 / 33, B2 H8 S512 D32 bias 118 / 89, D32: B12 H8 S192 57 / 42, B24 H8
//   S160 87 / 73, causal B32 H8 S128 56 / 44, B12 H8 S160 mask 74 / 57
//   <  the line  <  B2 H8 S256 38 / 40, B1 H4 S1024 89 / 95, B8 H8 S128 31 / 33, B32 H8 S96 60 / 93, B4 H6 S344 49 / 69, D32:
//   B6 H8 S256 0.76 times, B4 H8 S344 0.68, B8 H8 S192 0.84, B12 H8 S128 bias 0.81; B16 H8 S200 bias 129 / 250, B8 H16 S1024 679 / 2019, the same
//   causal with bias 917 / 2366, B8 H8 S300 T700 key bias 153 / 486.
bool fp32_tc_bwd_applies(const Problem& pr) {
  if (!takes(pr) || pr.D == 128 || pr.T <= kRows || pr.S <= kRows) return false;
  const int64_t ctas = (tiles_of(pr.S) < tiles_of(pr.T) ? tiles_of(pr.S) : tiles_of(pr.T)) * pr.bh_count;
  const bool none = !pr.bias && !pr.mask, one_tile = pr.S <= 128 && pr.T <= 128;
  if (pr.D == 32) {
    // (a small problem that just starts a second wave of CTAs waits for it as long as for the first)
    const int64_t owners = owners_of(pr.S > pr.T ? pr.S : pr.T) * pr.bh_count;
    if (ctas < 192) return false;
    if (int64_t(pr.S) * pr.T >= 40000 || owners <= 148) return true;
    return !none && (!row_addends(pr) || one_tile || owners >= 222);
  }
  return ctas >= (row_addends(pr) ? 192 : (none && one_tile ? 96 : 64));
}

size_t fp32_tc_bwd_bytes(const Problem& pr) {
  const size_t each = bwd_bytes_per_bh(pr);
  return each * part_of(pr, each, 0).bh_count;
}

namespace {
int backward_part(const Problem& pr, int bias_dtype, void* ws, cudaStream_t st) {
  uint8_t* q = static_cast<uint8_t*>(ws);
  uint8_t* g = q + plane_bytes(pr, pr.S);
  uint8_t* k = g + plane_bytes(pr, pr.S);
  uint8_t* v = k + plane_bytes(pr, pr.T);
  int* status = device_status_word();
  if (!status) { set_error("device status word is unavailable"); return NB200_ERR_LAUNCH; }
  SplitArgs sa{};
  sa.H = pr.H;
  sa.bh_begin = pr.bh_begin;
  sa.D = pr.D;
  sa.op[0] = operand(pr.q, pr.qs, pr.S, q);
  sa.op[1] = operand(pr.dout, pr.dos, pr.S, g);
  sa.op[2] = operand(pr.k, pr.ks, pr.T, k);
  sa.op[3] = operand(pr.v, pr.vs, pr.T, v);
  if (int rc = launch_split(pr, sa, 4, st)) return rc;
  BwdArgs a{};
  a.pr = pr;
  a.bias_dtype = bias_dtype;
  a.status = status;
  const bool add = pr.bias || pr.mask;
  a.x0 = q; a.x1 = g; a.y0 = k; a.y1 = v;
  a.x_tiles = int(tiles_of(pr.S));
  a.y_tiles = int(tiles_of(pr.T));
  if (int rc = add ? launch_bwd<false, true>(a, st) : launch_bwd<false, false>(a, st)) return rc;
  a.x0 = k; a.x1 = v; a.y0 = q; a.y1 = g;
  a.x_tiles = int(tiles_of(pr.T));
  a.y_tiles = int(tiles_of(pr.S));
  return add ? launch_bwd<true, true>(a, st) : launch_bwd<true, false>(a, st);
}
}  // namespace

int fp32_tc_backward(const Problem& pr, int bias_dtype, void* ws, cudaStream_t st) {
  for (int done = 0; done < pr.bh_count;) {
    const Problem part = part_of(pr, bwd_bytes_per_bh(pr), done);
    if (int rc = backward_part(part, bias_dtype, ws, st)) return rc;
    done += part.bh_count;
  }
  return NB200_OK;
}

}  // namespace nb200
