// LayerNorm over the trailing axis, forward and backward -- the sibling op of the attention path behind the same
// library (reference src/nitrix/nn/norm/__init__.py:110-176 is the dispatcher, src/nitrix/nn/norm/_reference.py:44-110
// the recipe: biased variance, rsqrt(var + eps), optional per-channel affine, then the constant `out_scale`; a 16-bit
// input is upcast to fp32 for the reductions and the affine transform and the result cast back).
//
//   forward   xhat = (x - mean) rstd,  y = out_scale (xhat w + b);  mean and rstd (fp32 per row) are kept for the
//             backward when the caller passes buffers for them
//   backward  gy = out_scale dy,  dxhat = gy w,  dx = rstd (dxhat - mean(dxhat) - xhat mean(dxhat xhat)),
//             dw = sum_rows gy xhat,  db = sum_rows gy
//
// Rows that are a multiple of 16 bytes (<= 8192 channels, aligned pointers) take the vector kernels below; the rest
// the scalar ones at the end.  The op is bound by HBM traffic (x once in, y once out; the backward x and dy in, dx
// out), so a row is read ONCE with 16-byte loads and held in registers between the reductions and the write: by one
// warp (rows of up to 32 x 16 B x 8) or by one 256-thread CTA (longer rows); the backward see there.  The variance is taken about the mean
// (two passes over the registers, as the reference's `var` does), not as E[x^2] - mean^2.  dw / db: every CTA walks
// rows in a grid-stride loop, keeps its column sums in registers, leaves one partial row per CTA in a
// workspace, and a second kernel adds the partials in a fixed order -- deterministic, no atomics.
#include <math.h>

#include "nitrix_b200_norm.h"
#include "sdpa_common.cuh"

namespace nb200 {
namespace {

constexpr int kThreads = 256;

struct LnArgs {
  const void* x;
  const void* w;
  const void* b;
  void* y;
  float* mean;
  float* rstd;
  const void* dy;
  void* dx;
  float* part;   // [2][grid][C] partial dw, db
  int64_t rows;
  int C;
  float eps, out_scale;
};

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sum over the threads that share a row: the warp, or the whole CTA through shared memory.  `red` holds eight
// floats per use; consecutive uses alternate between buffers (the callers pass red + 8 k), so that ONE barrier per
// reduction is enough: a buffer is rewritten only after a later barrier has shown that every thread has read it.
template <bool kCta>
__device__ __forceinline__ float row_sum(float v, float* red) {
  v = warp_sum_f(v);
  if constexpr (kCta) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red[warp] = v;
    __syncthreads();
    v = 0.f;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) v += red[i];
  }
  return v;
}
// two sums at once (red: 16 floats per use)
template <bool kCta>
__device__ __forceinline__ float2 row_sum2(float a, float b, float* red) {
  a = warp_sum_f(a);
  b = warp_sum_f(b);
  if constexpr (kCta) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
      red[warp] = a;
      red[8 + warp] = b;
    }
    __syncthreads();
    a = b = 0.f;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) {
      a += red[i];
      b += red[8 + i];
    }
  }
  return make_float2(a, b);
}

// The same as pairs: the arithmetic below runs on the packed fp32x2 pipe (one instruction per two elements; each
// lane rounds as the scalar instruction would, so results do not change).  At 16-bit widths the kernels are bound
// by instruction issue as much as by memory.
template <typename T>
__device__ __forceinline__ float2 unpack_pair(uint32_t w);
template <>
__device__ __forceinline__ float2 unpack_pair<__nv_bfloat16>(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
template <>
__device__ __forceinline__ float2 unpack_pair<__half>(uint32_t w) {
  return __half22float2(*reinterpret_cast<const __half2*>(&w));
}
template <typename T>
__device__ __forceinline__ uint32_t pack_pair(float2 v);
template <>
__device__ __forceinline__ uint32_t pack_pair<__nv_bfloat16>(float2 v) {
  const __nv_bfloat162 r = __floats2bfloat162_rn(v.x, v.y);
  return *reinterpret_cast<const uint32_t*>(&r);
}
template <>
__device__ __forceinline__ uint32_t pack_pair<__half>(float2 v) {
  const __half2 r = __floats2half2_rn(v.x, v.y);
  return *reinterpret_cast<const uint32_t*>(&r);
}
template <typename T, int kVec>
__device__ __forceinline__ void load_pairs(const T* p, float2 (&out)[kVec / 2]) {
  const uint4 w = *reinterpret_cast<const uint4*>(p);
  if constexpr (sizeof(T) == 4) {
    out[0] = make_float2(__uint_as_float(w.x), __uint_as_float(w.y));
    out[1] = make_float2(__uint_as_float(w.z), __uint_as_float(w.w));
  } else {
    out[0] = unpack_pair<T>(w.x);
    out[1] = unpack_pair<T>(w.y);
    out[2] = unpack_pair<T>(w.z);
    out[3] = unpack_pair<T>(w.w);
  }
}
template <typename T, int kVec>
__device__ __forceinline__ void store_pairs(T* p, const float2 (&v)[kVec / 2]) {
  uint4 w;
  if constexpr (sizeof(T) == 4) {
    w = make_uint4(__float_as_uint(v[0].x), __float_as_uint(v[0].y), __float_as_uint(v[1].x), __float_as_uint(v[1].y));
  } else {
    w = make_uint4(pack_pair<T>(v[0]), pack_pair<T>(v[1]), pack_pair<T>(v[2]), pack_pair<T>(v[3]));
  }
  *reinterpret_cast<uint4*>(p) = w;
}

// A row is split over kCta ? 256 : 32 threads; a thread holds kPer chunks of kVec = 16 / sizeof(T) elements, chunk p
// at column (p * threads + thread) * kVec.
template <typename T, int kPer, bool kCta>
__global__ void __launch_bounds__(kThreads, kPer <= 4 ? 4 : 2) ln_fwd_kernel(LnArgs a) {
  constexpr int kVec = 16 / int(sizeof(T));
  constexpr int kTpr = kCta ? kThreads : 32;
  __shared__ float red[2 * (kThreads / 32)];
  const int tin = kCta ? threadIdx.x : (threadIdx.x & 31);
  const int64_t row = kCta ? int64_t(blockIdx.x) : int64_t(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5);
  if (row >= a.rows) return;   // (a whole CTA, or a whole warp of a warp-per-row CTA, which never meets a barrier)
  const T* x = reinterpret_cast<const T*>(a.x) + row * a.C;
  constexpr int kPairs = kVec / 2;
  float2 xv[kPer][kPairs];
  float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int p = 0; p < kPer; ++p) {
    const int c0 = (p * kTpr + tin) * kVec;
    if (c0 < a.C) {
      load_pairs<T, kVec>(x + c0, xv[p]);
#pragma unroll
      for (int i = 0; i < kPairs; ++i) s2 = __fadd2_rn(s2, xv[p][i]);
    }
  }
  const float mean = row_sum<kCta>(s2.x + s2.y, red) / float(a.C);
  const float2 nmean = make_float2(-mean, -mean);
  float2 q2 = make_float2(0.f, 0.f);
#pragma unroll
  for (int p = 0; p < kPer; ++p)
    if ((p * kTpr + tin) * kVec < a.C) {
#pragma unroll
      for (int i = 0; i < kPairs; ++i) {
        xv[p][i] = __fadd2_rn(xv[p][i], nmean);      // x - mean, kept
        q2 = __ffma2_rn(xv[p][i], xv[p][i], q2);
      }
    }
  const float rstd = rsqrtf(row_sum<kCta>(q2.x + q2.y, red + 8) / float(a.C) + a.eps);
  if (tin == 0) {
    if (a.mean) a.mean[row] = mean;
    if (a.rstd) a.rstd[row] = rstd;
  }
  T* y = reinterpret_cast<T*>(a.y) + row * a.C;
  const T* w = reinterpret_cast<const T*>(a.w);
  const T* b = reinterpret_cast<const T*>(a.b);
  const float2 rstd2 = make_float2(rstd, rstd), os2 = make_float2(a.out_scale, a.out_scale);
#pragma unroll
  for (int p = 0; p < kPer; ++p) {
    const int c0 = (p * kTpr + tin) * kVec;
    if (c0 < a.C) {
      float2 wv[kPairs], bv[kPairs], out[kPairs];
      if (w) load_pairs<T, kVec>(w + c0, wv);
      if (b) load_pairs<T, kVec>(b + c0, bv);
#pragma unroll
      for (int i = 0; i < kPairs; ++i) {
        float2 v = __fmul2_rn(xv[p][i], rstd2);
        if (w) v = __fmul2_rn(v, wv[i]);
        if (b) v = __fadd2_rn(v, bv[i]);
        out[i] = __fmul2_rn(os2, v);
      }
      store_pairs<T, kVec>(y + c0, out);
    }
  }
}

// Backward.  A CTA is 512 threads = kRowThreads / tpr groups of tpr threads (tpr a power of two); a group takes one row
// at a time, a thread up to kPer 16-byte chunks of it -- always the same columns, so its part of the column sums dw, db
// stays in 2 kPer kVec registers from the first row to the last (16 columns a thread at most).  Every thread copies
// its own chunks of x and dy into its own slots of a shared-memory ring with 16-byte cp.async, several rows ahead: no
// barrier is needed for the data, and 64 to 128 KB per SM are in flight -- HBM needs about 44 KB per SM at its latency.
// kBatch rows share one barrier (the row sums of groups wider than a warp); their x and dy are read from the ring a
// second time behind it, which costs less than the registers that would hold them.
// bf16 (8192, 8192): 142 -> 81 us (4.9 TB/s of x, dy, dx) against the column sums in shared memory without copies ahead;
// 85 us with one row per barrier.
constexpr int kRowThreads = 512;
__device__ __forceinline__ void copy_async16(void* dst, const void* src, bool in) {
  const uint32_t d = uint32_t(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}
template <typename T>
__device__ __forceinline__ void word_pairs(const uint4 w, float2 (&out)[16 / int(sizeof(T)) / 2]) {
  if constexpr (sizeof(T) == 4) {
    out[0] = make_float2(__uint_as_float(w.x), __uint_as_float(w.y));
    out[1] = make_float2(__uint_as_float(w.z), __uint_as_float(w.w));
  } else {
    out[0] = unpack_pair<T>(w.x);
    out[1] = unpack_pair<T>(w.y);
    out[2] = unpack_pair<T>(w.z);
    out[3] = unpack_pair<T>(w.w);
  }
}

template <int kPer>
struct BwdRing {
  static constexpr int kBatch = kPer == 4 ? 1 : 2;             // rows between two barriers
  static constexpr int kAhead = 2;                             // batches in flight
  static constexpr int kStages = kBatch * (kAhead + 1);
  static constexpr size_t kBytes = size_t(kStages) * 2 * kPer * kRowThreads * 16;
};

template <typename T, int kPer>
__global__ void __launch_bounds__(kRowThreads, kPer == 1 ? 2 : 1) ln_bwd_kernel(LnArgs a, int tpr) {
  constexpr int kVec = 16 / int(sizeof(T));
  constexpr int kPairs = kVec / 2;
  constexpr int kBatch = BwdRing<kPer>::kBatch, kAhead = BwdRing<kPer>::kAhead;
  constexpr int kWarps = kRowThreads / 32;
  extern __shared__ __align__(16) uint4 ring[];               // [kStages][x, dy][kPer][kRowThreads]
  __shared__ __align__(16) float2 red[2][kBatch][kWarps];     // the warps' row sums, alternating by batch
  const int tid = threadIdx.x, tin = tid & (tpr - 1), group = tid / tpr, groups = kRowThreads / tpr;
  const int64_t blocks = (a.rows + groups - 1) / groups;      // of `groups` consecutive rows
  const T* x = reinterpret_cast<const T*>(a.x);
  const T* g = reinterpret_cast<const T*>(a.dy);
  auto chunk = [&](int p) { return (p * tpr + tin) * kVec; };  // first column of this thread's chunk p
  const int64_t step = gridDim.x;
  auto slot = [&](int stage, int which, int p) -> uint4* { return ring + ((stage * 2 + which) * kPer + p) * kRowThreads + tid; };
  // batch `it` of this CTA (blocks blockIdx.x + (it kBatch + r) step) into its part of the ring
  auto fetch = [&](int64_t it, int part) {
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      const int64_t blk = blockIdx.x + (it * kBatch + r) * step, row = blk * groups + group;
      const bool in = blk < blocks && row < a.rows;
#pragma unroll
      for (int p = 0; p < kPer; ++p) {
        const bool have = in && chunk(p) < a.C;
        const int64_t at = have ? row * a.C + chunk(p) : 0;
        copy_async16(slot(part * kBatch + r, 0, p), x + at, have);
        copy_async16(slot(part * kBatch + r, 1, p), g + at, have);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float2 w[kPer][kPairs], sw[kPer][kPairs], sb[kPer][kPairs];
#pragma unroll
  for (int p = 0; p < kPer; ++p) {
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      w[p][i] = make_float2(1.f, 1.f);
      sw[p][i] = sb[p][i] = make_float2(0.f, 0.f);
    }
    if (a.w && chunk(p) < a.C) load_pairs<T, kVec>(reinterpret_cast<const T*>(a.w) + chunk(p), w[p]);
  }
#pragma unroll
  for (int i = 0; i < kAhead; ++i) fetch(i, i);
  float nmean[kBatch], nrstd[kBatch];                          // of the batch after this one
  auto fetch_stats = [&](int64_t it) {
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      const int64_t blk = blockIdx.x + (it * kBatch + r) * step, row = blk * groups + group;
      const bool in = blk < blocks && row < a.rows;
      nmean[r] = in ? a.mean[row] : 0.f;
      nrstd[r] = in ? a.rstd[row] : 0.f;
    }
  };
  fetch_stats(0);
  int part = 0, flip = 0;
  const float2 os2 = make_float2(a.out_scale, a.out_scale);
  // (every thread of the CTA runs the same number of iterations: the barriers match; rows past the last are zeros)
  for (int64_t it = 0; blockIdx.x + it * kBatch * step < blocks; ++it) {
    fetch(it + kAhead, part == 0 ? kAhead : part - 1);         // (the slots of the last batch: this thread has read them)
    float2 mean2[kBatch], rstd2[kBatch];
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      mean2[r] = make_float2(-nmean[r], -nmean[r]);
      rstd2[r] = make_float2(nrstd[r], nrstd[r]);
    }
    fetch_stats(it + 1);
    asm volatile("cp.async.wait_group %0;" ::"n"(kAhead) : "memory");
    float t1[kBatch], t2[kBatch];
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      float2 s1 = make_float2(0.f, 0.f), s2 = make_float2(0.f, 0.f);
#pragma unroll
      for (int p = 0; p < kPer; ++p) {
        float2 xh[kPairs], d[kPairs];
        word_pairs<T>(*slot(part * kBatch + r, 0, p), xh);
        word_pairs<T>(*slot(part * kBatch + r, 1, p), d);
        if (chunk(p) < a.C) {
#pragma unroll
          for (int i = 0; i < kPairs; ++i) {
            xh[i] = __fmul2_rn(__fadd2_rn(xh[i], mean2[r]), rstd2[r]);
            const float2 gy = __fmul2_rn(os2, d[i]);
            sw[p][i] = __ffma2_rn(gy, xh[i], sw[p][i]);
            sb[p][i] = __fadd2_rn(sb[p][i], gy);
            const float2 dh = __fmul2_rn(gy, w[p][i]);
            s1 = __fadd2_rn(s1, dh);
            s2 = __ffma2_rn(dh, xh[i], s2);
          }
        }
      }
      t1[r] = s1.x + s1.y;
      t2[r] = s2.x + s2.y;
    }
    for (int o = min(tpr, 32) >> 1; o > 0; o >>= 1) {
#pragma unroll
      for (int r = 0; r < kBatch; ++r) {
        t1[r] += __shfl_xor_sync(0xffffffffu, t1[r], o);
        t2[r] += __shfl_xor_sync(0xffffffffu, t2[r], o);
      }
    }
    if (tpr > 32) {
      // (the buffer is rewritten two batches on, after the next batch's barrier has shown that everyone has read it)
      if ((tid & 31) == 0) {
#pragma unroll
        for (int r = 0; r < kBatch; ++r) red[flip][r][tid >> 5] = make_float2(t1[r], t2[r]);
      }
      __syncthreads();
#pragma unroll
      for (int r = 0; r < kBatch; ++r) {
        t1[r] = t2[r] = 0.f;
        const float4* q = reinterpret_cast<const float4*>(&red[flip][r][group * (tpr >> 5)]);
        for (int k = 0; k < (tpr >> 6); ++k) {
          const float4 v = q[k];
          t1[r] += v.x + v.z;
          t2[r] += v.y + v.w;
        }
      }
      flip ^= 1;
    }
#pragma unroll
    for (int r = 0; r < kBatch; ++r) {
      const int64_t row = (blockIdx.x + (it * kBatch + r) * step) * groups + group;
      if (row >= a.rows) continue;                             // (a block past the last starts past the last row)
      const float c1 = t1[r] / float(a.C), c2 = t2[r] / float(a.C);
      T* dx = reinterpret_cast<T*>(a.dx) + row * a.C;
      const float2 nc1 = make_float2(-c1, -c1), nc2 = make_float2(-c2, -c2);
#pragma unroll
      for (int p = 0; p < kPer; ++p) {
        if (chunk(p) < a.C) {
          float2 xh[kPairs], d[kPairs], out[kPairs];
          word_pairs<T>(*slot(part * kBatch + r, 0, p), xh);
          word_pairs<T>(*slot(part * kBatch + r, 1, p), d);
#pragma unroll
          for (int i = 0; i < kPairs; ++i) {
            xh[i] = __fmul2_rn(__fadd2_rn(xh[i], mean2[r]), rstd2[r]);
            const float2 dh = __fmul2_rn(__fmul2_rn(os2, d[i]), w[p][i]);
            out[i] = __fmul2_rn(rstd2[r], __ffma2_rn(xh[i], nc2, __fadd2_rn(dh, nc1)));
          }
          store_pairs<T, kVec>(dx + chunk(p), out);
        }
      }
    }
    part = part == kAhead ? 0 : part + 1;
  }
  if (!a.part) return;
  // this CTA's partial row: the groups' sums added in group order, through the ring's memory
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  float* all = reinterpret_cast<float*>(ring);                 // [dw, db][groups][C]
  float* mine_w = all + int64_t(group) * a.C;
  float* mine_b = all + int64_t(groups + group) * a.C;
#pragma unroll
  for (int p = 0; p < kPer; ++p) {
    if (chunk(p) < a.C) {
#pragma unroll
      for (int i = 0; i < kPairs; i += 2) {
        *reinterpret_cast<float4*>(mine_w + chunk(p) + 2 * i) = make_float4(sw[p][i].x, sw[p][i].y, sw[p][i + 1].x, sw[p][i + 1].y);
        *reinterpret_cast<float4*>(mine_b + chunk(p) + 2 * i) = make_float4(sb[p][i].x, sb[p][i].y, sb[p][i + 1].x, sb[p][i + 1].y);
      }
    }
  }
  __syncthreads();
  float* pw = a.part + int64_t(blockIdx.x) * a.C;
  float* pb = a.part + (int64_t(gridDim.x) + blockIdx.x) * a.C;
  for (int c = tid; c < a.C; c += kRowThreads) {
    float tw = 0.f, tb = 0.f;
    for (int k = 0; k < groups; ++k) {
      tw += all[int64_t(k) * a.C + c];
      tb += all[int64_t(groups + k) * a.C + c];
    }
    pw[c] = tw;
    pb[c] = tb;
  }
}

// dw[c] = sum over the CTAs' partial rows.  A CTA takes 32 columns (lane = column: 128-byte reads); its eight warps
// take the partial rows in turn, four loads in flight each, and their eight sums are added in warp order -- the
// order of the whole sum is fixed by (grid, column) alone.
template <typename T>
__global__ void __launch_bounds__(kThreads) ln_bwd_finish_kernel(const float* part, int grid, int C, T* dw, T* db) {
  __shared__ float sw[kThreads / 32][32], sb[kThreads / 32][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c = blockIdx.x * 32 + lane;
  float tw[4] = {0.f, 0.f, 0.f, 0.f}, tb[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < C) {
    const float* pw = part + c;
    const float* pb = part + int64_t(grid) * C + c;
    int k = warp;
    for (; k + 3 * (kThreads / 32) < grid; k += 4 * (kThreads / 32)) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        tw[u] += pw[int64_t(k + u * (kThreads / 32)) * C];
        tb[u] += pb[int64_t(k + u * (kThreads / 32)) * C];
      }
    }
    for (; k < grid; k += kThreads / 32) {
      tw[0] += pw[int64_t(k) * C];
      tb[0] += pb[int64_t(k) * C];
    }
  }
  sw[warp][lane] = (tw[0] + tw[1]) + (tw[2] + tw[3]);
  sb[warp][lane] = (tb[0] + tb[1]) + (tb[2] + tb[3]);
  __syncthreads();
  if (warp == 0 && c < C) {
    float a = 0.f, b = 0.f;
#pragma unroll
    for (int i = 0; i < kThreads / 32; ++i) {
      a += sw[i][lane];
      b += sb[i][lane];
    }
    if (dw) dw[c] = from_f32<T>(a);
    if (db) db[c] = from_f32<T>(b);
  }
}

// Any other row (channels not a multiple of 16 bytes, longer than 8192, unaligned pointers): one CTA per row in
// scalar strided passes; the row is re-read from L1 / L2.  dw / db are added to a zeroed [2][C] fp32 workspace with
// atomics (the one place where the order of a sum is not fixed).
template <typename T>
__global__ void __launch_bounds__(kThreads) ln_fwd_generic_kernel(LnArgs a) {
  __shared__ float red[2 * (kThreads / 32)];
  const int64_t row = blockIdx.x;
  const T* x = reinterpret_cast<const T*>(a.x) + row * a.C;
  float s = 0.f;
  for (int c = threadIdx.x; c < a.C; c += kThreads) s += to_f32<T>(x[c]);
  const float mean = row_sum<true>(s, red) / float(a.C);
  float q = 0.f;
  for (int c = threadIdx.x; c < a.C; c += kThreads) {
    const float d = to_f32<T>(x[c]) - mean;
    q = fmaf(d, d, q);
  }
  const float rstd = rsqrtf(row_sum<true>(q, red + 8) / float(a.C) + a.eps);
  if (threadIdx.x == 0) {
    if (a.mean) a.mean[row] = mean;
    if (a.rstd) a.rstd[row] = rstd;
  }
  T* y = reinterpret_cast<T*>(a.y) + row * a.C;
  const T* w = reinterpret_cast<const T*>(a.w);
  const T* b = reinterpret_cast<const T*>(a.b);
  for (int c = threadIdx.x; c < a.C; c += kThreads) {
    float v = (to_f32<T>(x[c]) - mean) * rstd;
    if (w) v *= to_f32<T>(w[c]);
    if (b) v += to_f32<T>(b[c]);
    y[c] = from_f32<T>(a.out_scale * v);
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) ln_bwd_generic_kernel(LnArgs a) {
  __shared__ float red[4 * (kThreads / 32)];
  const T* w = reinterpret_cast<const T*>(a.w);
  int flip = 0;
  for (int64_t row = blockIdx.x; row < a.rows; row += gridDim.x) {
    const T* x = reinterpret_cast<const T*>(a.x) + row * a.C;
    const T* g = reinterpret_cast<const T*>(a.dy) + row * a.C;
    const float mean = a.mean[row], rstd = a.rstd[row];
    float s1 = 0.f, s2 = 0.f;
    for (int c = threadIdx.x; c < a.C; c += kThreads) {
      const float xh = (to_f32<T>(x[c]) - mean) * rstd;
      const float dxh = a.out_scale * to_f32<T>(g[c]) * (w ? to_f32<T>(w[c]) : 1.f);
      s1 += dxh;
      s2 = fmaf(dxh, xh, s2);
    }
    const float2 cs = row_sum2<true>(s1, s2, red + 16 * flip);
    flip ^= 1;
    const float c1 = cs.x / float(a.C), c2 = cs.y / float(a.C);
    T* dx = reinterpret_cast<T*>(a.dx) + row * a.C;
    for (int c = threadIdx.x; c < a.C; c += kThreads) {
      const float xh = (to_f32<T>(x[c]) - mean) * rstd;
      const float gy = a.out_scale * to_f32<T>(g[c]);
      const float dxh = gy * (w ? to_f32<T>(w[c]) : 1.f);
      dx[c] = from_f32<T>(rstd * (dxh - c1 - xh * c2));
      if (a.part) {
        atomicAdd(a.part + c, gy * xh);
        atomicAdd(a.part + a.C + c, gy);
      }
    }
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

struct Shape {
  int vec, per;
  bool cta;
};

// Forward: the smallest per-thread chunk count that covers a row.
bool pick(int C, int dtype, Shape* s) {
  s->vec = dtype == NB200_F32 ? 4 : 8;
  if (C <= 0 || C % s->vec) return false;
  for (int per = 1; per <= 8; per *= 2)
    if (C <= 32 * s->vec * per) { s->per = per; s->cta = false; return true; }
  for (int per = 1; per <= 8; per *= 2)
    if (C <= kThreads * s->vec * per && C <= 8192) { s->per = per; s->cta = true; return true; }
  return false;
}

// Backward: chunks per thread (as few as cover a row with 512 threads: fewer registers, more rows per CTA) and
// threads per row.
struct BwdShape { int per, tpr; };
bool pick_bwd(int C, int dtype, BwdShape* s) {
  const int vec = dtype == NB200_F32 ? 4 : 8;
  if (C <= 0 || C % vec || C > 8192) return false;
  s->per = 1;
  while (C > kRowThreads * vec * s->per) s->per *= 2;
  s->tpr = 1;
  while (s->tpr * vec * s->per < C) s->tpr *= 2;
  return true;
}

// The backward's grid: as many CTAs as are resident at once (`per_sm` from the occupancy calculator; more CTAs only
// add partial rows to sum), at most one per block of rows.  per_sm = 2 bounds it for sizing the workspace.
int bwd_grid(int64_t rows, const BwdShape& s, int per_sm) {
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  const int64_t groups = kRowThreads / s.tpr, units = (rows + groups - 1) / groups;
  const int64_t cap = int64_t(sms) * per_sm;
  return int(units < cap ? (units > 0 ? units : 1) : cap);
}

int check_common(const nb200_layer_norm_params* p, const char* what) {
  if (!p) { set_error("%s: NULL parameter block", what); return NB200_ERR_INVALID; }
  if (p->struct_size != sizeof(nb200_layer_norm_params)) {
    set_error("%s: ABI mismatch: struct_size %zu, library expects %zu", what, size_t(p->struct_size),
              sizeof(nb200_layer_norm_params));
    return NB200_ERR_INVALID;
  }
  if (p->dtype != NB200_F32 && p->dtype != NB200_BF16 && p->dtype != NB200_F16) { set_error("%s: bad dtype", what); return NB200_ERR_INVALID; }
  if (p->rows < 0 || p->channels <= 0) { set_error("%s: bad extents", what); return NB200_ERR_INVALID; }
  return NB200_OK;
}

template <typename T, typename F>
int dispatch(const Shape& s, F&& go) {
  // go(kernel) launches; one instantiation per (chunks, warp / CTA)
  if (!s.cta) {
    switch (s.per) {
      case 1: return go(ln_fwd_kernel<T, 1, false>);
      case 2: return go(ln_fwd_kernel<T, 2, false>);
      case 4: return go(ln_fwd_kernel<T, 4, false>);
      default: return go(ln_fwd_kernel<T, 8, false>);
    }
  }
  switch (s.per) {
    case 1: return go(ln_fwd_kernel<T, 1, true>);
    case 2: return go(ln_fwd_kernel<T, 2, true>);
    case 4: return go(ln_fwd_kernel<T, 4, true>);
    default: return go(ln_fwd_kernel<T, 8, true>);
  }
}

template <typename T>
int fwd_t(const nb200_layer_norm_params* p, const Shape& s, cudaStream_t st) {
  LnArgs a{};
  a.x = p->x; a.w = p->weight; a.b = p->bias; a.y = p->y; a.mean = p->mean; a.rstd = p->rstd;
  a.rows = p->rows; a.C = p->channels; a.eps = p->eps; a.out_scale = p->out_scale;
  const int64_t blocks = s.cta ? p->rows : (p->rows + kThreads / 32 - 1) / (kThreads / 32);
  if (blocks > 0x7fffffff) { set_error("layer_norm: too many rows"); return NB200_ERR_UNSUPPORTED; }
  return dispatch<T>(s, [&](auto kernel) {
    kernel<<<unsigned(blocks), kThreads, 0, st>>>(a);
    count_launch();
    return check_launch("layer_norm_fwd_kernel");
  });
}

template <typename T, int kPer>
int bwd_launch(const LnArgs& a, const BwdShape& s, int* grid, cudaStream_t st) {
  constexpr size_t smem = BwdRing<kPer>::kBytes;
  auto kernel = ln_bwd_kernel<T, kPer>;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) {
    set_error("layer_norm_bwd: cudaFuncSetAttribute(%zu): %s", smem, cudaGetErrorString(cudaGetLastError()));
    return NB200_ERR_LAUNCH;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kRowThreads, smem) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    per_sm = 1;
  }
  *grid = bwd_grid(a.rows, s, per_sm < 2 ? per_sm : 2);
  kernel<<<unsigned(*grid), kRowThreads, smem, st>>>(a, s.tpr);
  count_launch();
  return check_launch("layer_norm_bwd_kernel");
}

template <typename T>
int bwd_t(const nb200_layer_norm_params* p, const BwdShape& s, cudaStream_t st) {
  LnArgs a{};
  a.x = p->x; a.w = p->weight; a.dy = p->dy; a.dx = p->dx; a.mean = p->mean; a.rstd = p->rstd;
  a.rows = p->rows; a.C = p->channels; a.eps = p->eps; a.out_scale = p->out_scale;
  const bool want_params = p->dweight || p->dbias;
  int grid = bwd_grid(p->rows, s, 2);
  if (want_params) {
    const size_t need = sizeof(float) * 2 * size_t(grid) * size_t(p->channels);
    if (!p->workspace || p->workspace_bytes < need) {
      set_error("layer_norm_bwd: workspace of %zu bytes needed (nb200_layer_norm_workspace_bytes), %zu given", need,
                size_t(p->workspace_bytes));
      return NB200_ERR_INVALID;
    }
    a.part = static_cast<float*>(p->workspace);
  }
  int rc;
  if (s.per == 1) {
    rc = bwd_launch<T, 1>(a, s, &grid, st);
  } else if (s.per == 2) {
    rc = bwd_launch<T, 2>(a, s, &grid, st);
  } else {
    rc = bwd_launch<T, sizeof(T) == 4 ? 4 : 2>(a, s, &grid, st);   // (four chunks: fp32 only)
  }
  if (rc || !want_params) return rc;
  ln_bwd_finish_kernel<T><<<(p->channels + 31) / 32, kThreads, 0, st>>>(
      a.part, grid, p->channels, static_cast<T*>(p->dweight), static_cast<T*>(p->dbias));
  count_launch();
  return check_launch("layer_norm_bwd_finish_kernel");
}

template <typename T>
int fwd_generic_t(const nb200_layer_norm_params* p, cudaStream_t st) {
  LnArgs a{};
  a.x = p->x; a.w = p->weight; a.b = p->bias; a.y = p->y; a.mean = p->mean; a.rstd = p->rstd;
  a.rows = p->rows; a.C = p->channels; a.eps = p->eps; a.out_scale = p->out_scale;
  if (p->rows > 0x7fffffff) { set_error("layer_norm: too many rows"); return NB200_ERR_UNSUPPORTED; }
  ln_fwd_generic_kernel<T><<<unsigned(p->rows), kThreads, 0, st>>>(a);
  count_launch();
  return check_launch("layer_norm_fwd_generic_kernel");
}

template <typename T>
int bwd_generic_t(const nb200_layer_norm_params* p, cudaStream_t st) {
  LnArgs a{};
  a.x = p->x; a.w = p->weight; a.dy = p->dy; a.dx = p->dx; a.mean = p->mean; a.rstd = p->rstd;
  a.rows = p->rows; a.C = p->channels; a.eps = p->eps; a.out_scale = p->out_scale;
  const bool want_params = p->dweight || p->dbias;
  if (want_params) {
    const size_t need = sizeof(float) * 2 * size_t(p->channels);
    if (!p->workspace || p->workspace_bytes < need) {
      set_error("layer_norm_bwd: workspace of %zu bytes needed (nb200_layer_norm_workspace_bytes), %zu given", need,
                size_t(p->workspace_bytes));
      return NB200_ERR_INVALID;
    }
    a.part = static_cast<float*>(p->workspace);
    if (cudaMemsetAsync(a.part, 0, need, st) != cudaSuccess) return check_launch("layer_norm_bwd: clearing the workspace");
  }
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t cap = int64_t(sms > 0 ? sms : 148) * 8;
  const int grid = int(p->rows < cap ? (p->rows > 0 ? p->rows : 1) : cap);
  ln_bwd_generic_kernel<T><<<unsigned(grid), kThreads, 0, st>>>(a);
  count_launch();
  if (int rc = check_launch("layer_norm_bwd_generic_kernel")) return rc;
  if (!want_params) return NB200_OK;
  ln_bwd_finish_kernel<T><<<(p->channels + 31) / 32, kThreads, 0, st>>>(
      a.part, 1, p->channels, static_cast<T*>(p->dweight), static_cast<T*>(p->dbias));
  count_launch();
  return check_launch("layer_norm_bwd_finish_kernel");
}

// the vector kernels need 16-byte rows: channels a multiple of 16 bytes (<= 8192) and aligned pointers
bool vector_fwd(const nb200_layer_norm_params* p, Shape* s) {
  return pick(p->channels, p->dtype, s) && aligned16(p->x) && (!p->weight || aligned16(p->weight)) && aligned16(p->y) &&
         (!p->bias || aligned16(p->bias));
}
bool vector_bwd(const nb200_layer_norm_params* p, BwdShape* s) {
  return pick_bwd(p->channels, p->dtype, s) && aligned16(p->x) && (!p->weight || aligned16(p->weight)) &&
         aligned16(p->dy) && aligned16(p->dx);
}

}  // namespace
}  // namespace nb200

using namespace nb200;

extern "C" NB200_API int nb200_layer_norm_workspace_bytes(const nb200_layer_norm_params* p, size_t* bytes) {
  if (!bytes) { set_error("bytes out-pointer is NULL"); return NB200_ERR_INVALID; }
  if (int rc = check_common(p, "layer_norm_workspace_bytes")) return rc;
  // (sized for the vector kernels' per-CTA partial rows, which is never less than the scalar kernels' [2][C])
  BwdShape s;
  const int grid = pick_bwd(p->channels, p->dtype, &s) ? bwd_grid(p->rows, s, 2) : 1;
  *bytes = sizeof(float) * 2 * size_t(grid) * size_t(p->channels);
  return NB200_OK;
}

extern "C" NB200_API int nb200_layer_norm_fwd(const nb200_layer_norm_params* p, void* cuda_stream) {
  if (int rc = check_common(p, "layer_norm_fwd")) return rc;
  if (p->rows == 0) return NB200_OK;
  if (!p->x || !p->y) { set_error("layer_norm_fwd: NULL x or y"); return NB200_ERR_INVALID; }
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  prof_call_begin(st);
  Shape s;
  const bool vec = vector_fwd(p, &s);
  switch (p->dtype) {
    case NB200_F32: return vec ? fwd_t<float>(p, s, st) : fwd_generic_t<float>(p, st);
    case NB200_BF16: return vec ? fwd_t<__nv_bfloat16>(p, s, st) : fwd_generic_t<__nv_bfloat16>(p, st);
    default: return vec ? fwd_t<__half>(p, s, st) : fwd_generic_t<__half>(p, st);
  }
}

extern "C" NB200_API int nb200_layer_norm_bwd(const nb200_layer_norm_params* p, void* cuda_stream) {
  if (int rc = check_common(p, "layer_norm_bwd")) return rc;
  if (p->rows == 0 && !p->dweight && !p->dbias) return NB200_OK;
  if ((p->rows > 0 && (!p->x || !p->dy || !p->dx || !p->mean || !p->rstd))) {
    set_error("layer_norm_bwd: x, dy, dx, mean and rstd are required");
    return NB200_ERR_INVALID;
  }
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  prof_call_begin(st);
  BwdShape s;
  const bool vec = vector_bwd(p, &s);
  switch (p->dtype) {
    case NB200_F32: return vec ? bwd_t<float>(p, s, st) : bwd_generic_t<float>(p, st);
    case NB200_BF16: return vec ? bwd_t<__nv_bfloat16>(p, s, st) : bwd_generic_t<__nv_bfloat16>(p, st);
    default: return vec ? bwd_t<__half>(p, s, st) : bwd_generic_t<__half>(p, st);
  }
}
