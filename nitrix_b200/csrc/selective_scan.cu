// Mamba / S6 selective scan, forward and backward -- the second sibling op behind the same library (reference
// src/nitrix/nn/ssm/__init__.py:127- is the dispatcher, src/nitrix/nn/ssm/_reference.py:60-98 the recipe):
//
//   a_t = exp(delta_t A),  b_t = (delta_t x_t) B_t,  h_t = a_t h_{t-1} + b_t  (h_{-1} = 0),
//   y_t = sum_n C_{t,n} h_{t,n} (+ D x_t)
//
// per batch element, channel d and state n; x, delta (batch, l, d), A (d, n), B, C (batch, l, n), D (d); fp32
// recurrence and readout whatever the storage dtype (reference _reference.py:262-279).
//
// Nothing of size (l, d, n) is materialised.  Forward: four lanes own one channel of one batch element, a quarter of
// its states each, and walk the sequence with them in registers (in segments side by side where there are few channels);
// every eighth step's state goes to a checkpoint array (batch, l / 8, d, n).  Backward, two kernels: ss_adjoint_kernel walks the sequence once more, last step first, with
// the adjoint recurrence g_t = a_{t+1} g_{t+1} + C_t dy_t alone and leaves g at the same eighth steps; with both
// states known at its borders every chunk of eight steps is then independent of all others, and ss_bwd_kernel
// computes the gradients chunk by chunk in parallel.  Its sums over channels (dB_t, dC_t) go through a shared-memory
// tile and 16-byte reductions into fp32 accumulators, those over batch and time (dA, dD) are kept per thread over the
// chunks of a CTA and added once; ss_finish_kernel converts the accumulators to the storage dtype.
#include <cooperative_groups.h>
#include <math.h>

#include "nitrix_b200_scan.h"
#include "sdpa_common.cuh"

namespace nb200 {
namespace {

namespace cg = cooperative_groups;

constexpr int kStep = 8;    // steps per checkpoint interval = chunk of the backward

struct SsArgs {
  const void *x, *delta, *A, *B, *C, *D, *dy;
  void *y, *dx, *ddelta;
  float* ckpt;            // [batch][chunks][Dc][N]: the state after each chunk
  float* gck;             // [batch][chunks][Dc][N]: the adjoint state entering each chunk from the next one
  float *accB, *accC;     // [batch][L][N]
  float *accA, *accD;     // [Dc][N], [Dc]
  int batch, L, Dc, N, chunks;
  int per_cta;            // chunks a CTA of ss_bwd_kernel works through
  int vec;                // groups of four channels of x, delta, y, dy, dx, ddelta can be moved as one word
  int vecn;               // groups of four states of the fp32 arrays can
  // launches of the backward for a range of channels (kRange): the first of them, and how many gck's rows hold (channel 0's
  // states would be at gck)
  int d_first, gD;
  int seg;                // steps of a segment where the walks are split in time (kSplit), a multiple of kStage
};

// a_t = exp(delta_t A) as one multiply and one ex2.approx (relative error 2^-22): A is held pre-multiplied by log2(e)
__device__ __forceinline__ float ex2_ss(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kLog2eSs = 1.4426950408889634f;
__device__ __forceinline__ float2 ex2_ss2(float2 x) { return make_float2(ex2_ss(x.x), ex2_ss(x.y)); }

// four consecutive elements p[0..3], the first `n` of which exist (zeros for the rest); `vec`: n is 0 or 4 and p is
// aligned to the four
template <typename T>
__device__ __forceinline__ float4 load4(const T* p, int n, bool vec) {
  float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec) {
    if (n > 0) {
      if constexpr (sizeof(T) == 4) {
        r = *reinterpret_cast<const float4*>(p);
      } else {
        const uint2 w = *reinterpret_cast<const uint2*>(p);
        const T* e = reinterpret_cast<const T*>(&w);
        r = make_float4(to_f32<T>(e[0]), to_f32<T>(e[1]), to_f32<T>(e[2]), to_f32<T>(e[3]));
      }
    }
  } else {
    if (n > 0) r.x = to_f32<T>(p[0]);
    if (n > 1) r.y = to_f32<T>(p[1]);
    if (n > 2) r.z = to_f32<T>(p[2]);
    if (n > 3) r.w = to_f32<T>(p[3]);
  }
  return r;
}
// The same as loaded, for a prefetch: a conversion behind the load would wait for it on the spot.
template <typename T>
struct Raw4 {
  uint32_t w[4];   // fp32: the four; 16 bits: two words of two (vec) or four of one
  __device__ __forceinline__ void load(const T* p, int n, bool vec) {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = 0u;
    if (vec) {
      if (n > 0) {
        if constexpr (sizeof(T) == 4) {
          const uint4 v = *reinterpret_cast<const uint4*>(p);
          w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
        } else {
          const uint2 v = *reinterpret_cast<const uint2*>(p);
          w[0] = v.x; w[1] = v.y;
        }
      }
    } else {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < n) {
          if constexpr (sizeof(T) == 4) w[i] = reinterpret_cast<const uint32_t*>(p)[i];
          else w[i] = reinterpret_cast<const unsigned short*>(p)[i];
        }
    }
  }
  static __device__ __forceinline__ float f(uint32_t bits) {
    if constexpr (sizeof(T) == 4) {
      return __uint_as_float(bits);
    } else {
      const unsigned short b = static_cast<unsigned short>(bits);
      return to_f32<T>(*reinterpret_cast<const T*>(&b));
    }
  }
  __device__ __forceinline__ float4 get(bool vec) const {
    if constexpr (sizeof(T) == 4) return make_float4(f(w[0]), f(w[1]), f(w[2]), f(w[3]));
    else return vec ? make_float4(f(w[0]), f(w[0] >> 16), f(w[1]), f(w[1] >> 16)) : make_float4(f(w[0]), f(w[1]), f(w[2]), f(w[3]));
  }
};
template <typename T>
__device__ __forceinline__ void store4(T* p, float4 v, int n, bool vec) {
  if (vec) {
    if (n > 0) {
      if constexpr (sizeof(T) == 4) {
        *reinterpret_cast<float4*>(p) = v;
      } else {
        uint2 w;
        T* e = reinterpret_cast<T*>(&w);
        e[0] = from_f32<T>(v.x); e[1] = from_f32<T>(v.y); e[2] = from_f32<T>(v.z); e[3] = from_f32<T>(v.w);
        *reinterpret_cast<uint2*>(p) = w;
      }
    }
  } else {
    if (n > 0) p[0] = from_f32<T>(v.x);
    if (n > 1) p[1] = from_f32<T>(v.y);
    if (n > 2) p[2] = from_f32<T>(v.z);
    if (n > 3) p[3] = from_f32<T>(v.w);
  }
}

// ---- the two sequential walks ------------------------------------------------------------------------------------
// Four adjacent lanes share a channel and hold kQ = kN / 4 of its states each as packed pairs.  A CTA is 16 channels = 64
// threads: small CTAs spread evenly over the SMs (8 x 2048 channels: 7 per SM against an average of 6.9; CTAs of 64
// channels put 2 on some SMs and 1 on the others).  Sixteen steps are staged at a time: a thread fetches four channels
// of one row of each operand with one load, one chunk ahead and kept as loaded (a 16-bit conversion behind the load
// would wait for it), and spreads (delta, delta x) and the B, C rows through shared memory; y goes back the same way.
// A step is 3 shared-memory loads, 8 packed operations and 4 ex2 per 4 states, taken four steps at a time so that no
// operand or exponential waits for the recurrence.  Bounds: the special-function unit (16 ex2 per SM and cycle: 60 us
// for 8 x 1024 x 2048 x 16) and shared memory, which delivers 32 words per cycle however many lanes share them.
// Two channels per thread halve those words, but leave half the warps to cover the latencies: measured slower.
// Forward with checkpoints, f32 (8, 1024, 2048, 16): 288 -> 135 us; bf16 (8, 2048, 2048, 16) without: 931 -> 242 us.
constexpr int kScanCh = 16;
constexpr int kScanThreads = kScanCh * 4;
constexpr int kStage = 16;                       // steps per staged chunk
constexpr int kYPitch = 24;                      // of the staged readouts: four rows x eight channels on distinct banks

// a thread's share of a chunk's [kStage][kN] block of B or C rows: kN / 16 groups of four states
template <typename T, int kN>
struct RowShare {
  static constexpr int kGroups = kStage * (kN / 4);
  static constexpr int kPer = (kGroups + kScanThreads - 1) / kScanThreads;
  Raw4<T> v[kPer];
  __device__ __forceinline__ void load(const T* base, int t0, int L, int N, bool vec, int tid) {
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = tid + kScanThreads * j, s = i / (kN / 4), n0 = (i - s * (kN / 4)) * 4;
      const bool in = i < kGroups && t0 + s < L;
      v[j].load(base + int64_t(t0 + s) * N + n0, in ? min(4, N - n0) : 0, vec);
    }
  }
  __device__ __forceinline__ void store(float* dst, bool vec, int tid) const {
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int i = tid + kScanThreads * j;
      if (i < kGroups) *reinterpret_cast<float4*>(dst + i * 4) = v[j].get(vec);
    }
  }
};

// kQ states of one channel to / from an fp32 [..][N] row
template <int kQ>
__device__ __forceinline__ void store_states(float* p, int n0, int N, bool vec, const float2 (&h)[kQ / 2]) {
  if (vec && kQ % 4 == 0) {
#pragma unroll
    for (int k = 0; k < kQ / 2; k += 2)
      if (n0 + 2 * k < N) *reinterpret_cast<float4*>(p + n0 + 2 * k) = make_float4(h[k].x, h[k].y, h[(k + 1) % (kQ / 2)].x, h[(k + 1) % (kQ / 2)].y);
  } else if (vec) {
    if (n0 < N) *reinterpret_cast<float2*>(p + n0) = h[0];
  } else {
#pragma unroll
    for (int k = 0; k < kQ / 2; ++k) {
      if (n0 + 2 * k < N) p[n0 + 2 * k] = h[k].x;
      if (n0 + 2 * k + 1 < N) p[n0 + 2 * k + 1] = h[k].y;
    }
  }
}

// A's row of a channel, times log2(e), as pairs (zeros for states that do not exist)
template <typename T, int kQ>
__device__ __forceinline__ void load_rates(const SsArgs& a, int d, bool live, int n0, float2 (&Ar)[kQ / 2]) {
  const T* Ap = reinterpret_cast<const T*>(a.A) + int64_t(d) * a.N;
#pragma unroll
  for (int k = 0; k < kQ / 2; ++k) {
    const int n = n0 + 2 * k;
    Ar[k].x = (live && n < a.N) ? kLog2eSs * to_f32<T>(Ap[n]) : 0.f;
    Ar[k].y = (live && n + 1 < a.N) ? kLog2eSs * to_f32<T>(Ap[n + 1]) : 0.f;
  }
}

// two states' row entries from shared memory, kQ / 2 pairs
template <int kQ>
__device__ __forceinline__ void row_pairs(const float* p, float2 (&v)[kQ / 2]) {
  if constexpr (kQ == 2) {
    v[0] = *reinterpret_cast<const float2*>(p);
  } else {
#pragma unroll
    for (int k = 0; k < kQ / 2; k += 2) {
      const float4 w = *reinterpret_cast<const float4*>(p + 2 * k);
      v[k] = make_float2(w.x, w.y);
      v[k + 1] = make_float2(w.z, w.w);
    }
  }
}

// four neighbouring channels' pairs of a step
__device__ __forceinline__ void write_pairs(float2* p, float4 a, float4 b) {
  reinterpret_cast<float4*>(p)[0] = make_float4(a.x, b.x, a.y, b.y);
  reinterpret_cast<float4*>(p)[1] = make_float4(a.z, b.z, a.w, b.w);
}
__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// The walks split in time.  Few channels leave most of the GPU idle while a few CTAs walk a long sequence step by step, a
// step costing its latencies alone (72 ns with one CTA per SM, where seven share one they take 132 ns together).  So a
// cluster of up to eight CTAs takes the sequence in segments: each walks its own from an empty state, keeping its end and
// the sum of its deltas (whose exponential is the segment's whole decay), reads those of the segments before it over
// distributed shared memory, and walks again from the state they give.  About 1.6 times the work, four or eight times the
// SMs (walk_splits has the figures).  Error against 64 bits, f32, norms, mean over (1, 2048, 128, 16), (2, 1024, 96, 8), (1, 1500,
// 64, 32), (2, 600, 40, 64) and (4, 512, 64, 16), each with rates of 0.2 to 1.7 and a hundredth of that, one walk / segments:
// y 1.2e-6 / 7.4e-7, dA 2.4e-6 / 1.4e-6.
template <int kN, bool kUsed>
struct Segment {
  float h[kScanCh][kN];
  float span[kScanCh];   // sum of delta
  // The state behind a segment: end + state * 2^(d rate).  The ends of the range are those of a walk step by step: a state
  // that is zero stays it whatever the decay (no 0 * inf), the factor is applied as two halves where it would leave the range
  // that the product need not leave, and past that (a rate of -inf: no memory) there is no rounding to put back.
  static __device__ __forceinline__ float through(float state, float d, float rate, float end) {
    const float x = __fmul_rn(d, rate);
    const bool wide = fabsf(x) > 126.f;
    const float e = ex2_ss(wide ? 0.5f * x : x);
    // (the exponent of a whole segment is large: its rounding goes back in as a factor 1 + ln 2 * rest)
    const float f = fabsf(x) < 256.f ? fmaf(e * fmaf(d, rate, -x), 0.6931471805599453f, e) : e;
    const float to = fmaf(wide ? state * e : state, f, end);
    return state == 0.f ? end : to;
  }
  // Publishes this segment's end; returns in `state` what enters it, from segments first, first + step .. own - step.
  template <int kPairs>
  __device__ __forceinline__ void join(int first, int own, int step, int ch, int part, float my_span, const float2 (&rate)[kPairs],
                                       float2 (&state)[kPairs]) {
#pragma unroll
    for (int k = 0; k < kPairs; ++k) {
      h[ch][part * 2 * kPairs + 2 * k] = state[k].x;
      h[ch][part * 2 * kPairs + 2 * k + 1] = state[k].y;
      state[k] = make_float2(0.f, 0.f);
    }
    if (part == 0) span[ch] = my_span;
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int s = first; s != own; s += step) {
      const float* rh = cluster.map_shared_rank(&h[ch][part * 2 * kPairs], s);
      const float d = *cluster.map_shared_rank(&span[ch], s);
#pragma unroll
      for (int k = 0; k < kPairs; ++k) {
        state[k].x = through(state[k].x, d, rate[k].x, rh[2 * k]);
        state[k].y = through(state[k].y, d, rate[k].y, rh[2 * k + 1]);
      }
    }
  }
};
template <int kN>
struct Segment<kN, false> {};

// kShort: sequences of up to kStage - 4 steps, one loop over the groups of four that exist (one step of 128 x 2048 channels,
// f32: 31 -> 17 us; an instantiation of its own, since the test costs the others up to a fifth by another order of the
// instructions).
// kSplit: the sequence in segments of a.seg steps, one CTA of a cluster each.
template <typename T, int kN, bool kShort, bool kSplit>
__global__ void __launch_bounds__(kScanThreads) ss_fwd_kernel(SsArgs a) {
  constexpr int kQ = kN / 4;
  __shared__ Segment<kN, kSplit> segment;
  __shared__ __align__(16) float2 du[kStage * kScanCh];    // delta, delta x
  __shared__ __align__(16) float sB[kStage * kN], sC[kStage * kN];
  __shared__ __align__(16) float sy[kStage * kYPitch];
  const int tid = threadIdx.x, part = tid & 3, ch = tid >> 2;
  const int d0 = blockIdx.x * kScanCh, b = blockIdx.y, d = d0 + ch;
  const bool live = d < a.Dc;
  const bool vec = a.vec != 0, vecn = a.vecn != 0;
  // this thread's four channels of one row of a staged chunk
  const int lr = tid >> 2, lc = (tid & 3) * 4, ln = max(0, min(4, a.Dc - (d0 + lc)));
  const int64_t at = int64_t(b) * a.L * a.Dc + d0 + lc;
  const T* xp = reinterpret_cast<const T*>(a.x) + at;
  const T* dp = reinterpret_cast<const T*>(a.delta) + at;
  T* yp = reinterpret_cast<T*>(a.y) + at;
  const T* Bp = reinterpret_cast<const T*>(a.B) + int64_t(b) * a.L * a.N;
  const T* Cp = reinterpret_cast<const T*>(a.C) + int64_t(b) * a.L * a.N;
  const float4 Dd = a.D ? load4<T>(reinterpret_cast<const T*>(a.D) + d0 + lc, ln, false) : make_float4(0.f, 0.f, 0.f, 0.f);
  float2 Ar[kQ / 2], h[kQ / 2];
  load_rates<T, kQ>(a, d, live, part * kQ, Ar);
#pragma unroll
  for (int k = 0; k < kQ / 2; ++k) h[k] = make_float2(0.f, 0.f);
  Raw4<T> nx, nd;
  RowShare<T, kN> nB, nC;
  auto load = [&](int t0) {
    const int n = t0 + lr < a.L ? ln : 0;
    nx.load(xp + int64_t(t0 + lr) * a.Dc, n, vec);
    nd.load(dp + int64_t(t0 + lr) * a.Dc, n, vec);
    nB.load(Bp, t0, a.L, a.N, vecn, tid);
    nC.load(Cp, t0, a.L, a.N, vecn, tid);
  };
  const int t_begin = kSplit ? int(blockIdx.z) * a.seg : 0, t_end = kSplit ? min(a.L, t_begin + a.seg) : a.L;
  if constexpr (kSplit) {
    // the segment from an empty state: nothing but the recurrence (the last segment's end is nobody's start)
    float span = 0.f;
    if (blockIdx.z + 1 < gridDim.z) {
      load(t_begin);
      for (int t0 = t_begin; t0 < t_end; t0 += kStage) {
        const float4 cx = nx.get(vec), dl4 = nd.get(vec);
        __syncthreads();   // (the steps before have been read)
        write_pairs(du + lr * kScanCh + lc, dl4, make_float4(dl4.x * cx.x, dl4.y * cx.y, dl4.z * cx.z, dl4.w * cx.w));
        nB.store(sB, vecn, tid);
        __syncthreads();
        if (t0 + kStage < t_end) load(t0 + kStage);
        float stage_span = 0.f;   // (summed per stage, then over the stages: shorter chains of roundings)
#pragma unroll
        for (int u = 0; u < kStage; ++u) {
          const float2 w = du[u * kScanCh + ch];
          float2 Bv[kQ / 2];
          row_pairs<kQ>(sB + u * kN + part * kQ, Bv);
          stage_span += w.x;
#pragma unroll
          for (int k = 0; k < kQ / 2; ++k)
            h[k] = __ffma2_rn(ex2_ss2(__fmul2_rn(both(w.x), Ar[k])), h[k], __fmul2_rn(both(w.y), Bv[k]));
        }
        span += stage_span;
      }
    }
    segment.join(0, int(blockIdx.z), 1, ch, part, span, Ar, h);
  }
  load(kSplit ? t_begin : 0);
  for (int t0 = kSplit ? t_begin : 0; t0 < (kSplit ? t_end : a.L); t0 += kStage) {
    // (steps past the sequence's end are staged as zeros: the state stays as it is)
    const float4 cx = nx.get(vec), dl4 = nd.get(vec);
    write_pairs(du + lr * kScanCh + lc, dl4, make_float4(dl4.x * cx.x, dl4.y * cx.y, dl4.z * cx.z, dl4.w * cx.w));
    nB.store(sB, vecn, tid);
    nC.store(sC, vecn, tid);
    __syncthreads();
    if (!kShort && t0 + kStage < (kSplit ? t_end : a.L)) load(t0 + kStage);
    // four steps at a time, in three phases: operands and decays (nothing in them depends on the state), then the
    // recurrence, then the sums over the lanes
#pragma unroll
    for (int s0 = 0; s0 < (kShort ? a.L : kStage); s0 += 4) {
      float2 av[4][kQ / 2], bu[4][kQ / 2];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 w = du[(s0 + u) * kScanCh + ch];
        float2 Bv[kQ / 2];
        row_pairs<kQ>(sB + (s0 + u) * kN + part * kQ, Bv);
#pragma unroll
        for (int k = 0; k < kQ / 2; ++k) {
          av[u][k] = ex2_ss2(__fmul2_rn(both(w.x), Ar[k]));
          bu[u][k] = __fmul2_rn(both(w.y), Bv[k]);   // (rows past N are zero)
        }
      }
      float y[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        float2 Cv[kQ / 2], acc = make_float2(0.f, 0.f);
        row_pairs<kQ>(sC + (s0 + u) * kN + part * kQ, Cv);
#pragma unroll
        for (int k = 0; k < kQ / 2; ++k) {
          h[k] = __ffma2_rn(av[u][k], h[k], bu[u][k]);
          acc = k ? __ffma2_rn(Cv[k], h[k], acc) : __fmul2_rn(Cv[k], h[k]);
        }
        y[u] = acc.x + acc.y;
      }
      // the sums over the four lanes, four steps at once: each lane ends with one step
      const bool hi = part & 2, lo = part & 1;
      float k0 = hi ? y[2] : y[0], k1 = hi ? y[3] : y[1];
      k0 += __shfl_xor_sync(0xffffffffu, hi ? y[0] : y[2], 2);
      k1 += __shfl_xor_sync(0xffffffffu, hi ? y[1] : y[3], 2);
      sy[(s0 + part) * kYPitch + ch] = (lo ? k1 : k0) + __shfl_xor_sync(0xffffffffu, lo ? k0 : k1, 1);
      if ((s0 & 4) && a.ckpt) {   // the state after every eighth step (of a chunk that has a successor)
        const int c = (t0 + s0) / kStep;
        if (live && c + 1 < a.chunks)
          store_states<kQ>(a.ckpt + ((int64_t(b) * a.chunks + c) * a.Dc + d) * a.N, part * kQ, a.N, vecn, h);
      }
    }
    __syncthreads();
    float4 v = *reinterpret_cast<const float4*>(sy + lr * kYPitch + lc);
    if (a.D) v = make_float4(fmaf(Dd.x, cx.x, v.x), fmaf(Dd.y, cx.y, v.y), fmaf(Dd.z, cx.z, v.z), fmaf(Dd.w, cx.w, v.w));
    store4<T>(yp + int64_t(t0 + lr) * a.Dc, v, t0 + lr < a.L ? ln : 0, vec);
  }
  if constexpr (kSplit) cg::this_cluster().sync();   // (nobody reads this CTA's shared memory any more)
}

// The adjoint recurrence alone, last step first: leaves for every chunk but the last the g that enters it.
template <typename T, int kN, bool kRange, bool kSplit>
__global__ void __launch_bounds__(kScanThreads) ss_adjoint_kernel(SsArgs a) {
  constexpr int kQ = kN / 4;
  __shared__ Segment<kN, kSplit> segment;
  __shared__ __align__(16) float2 dg[kStage * kScanCh];    // delta, dy
  __shared__ __align__(16) float sC[kStage * kN];
  const int tid = threadIdx.x, part = tid & 3, ch = tid >> 2;
  const int d0 = (kRange ? a.d_first : 0) + blockIdx.x * kScanCh, b = blockIdx.y, d = d0 + ch;
  const bool live = d < a.Dc;
  const bool vec = a.vec != 0, vecn = a.vecn != 0;
  const int lr = tid >> 2, lc = (tid & 3) * 4, ln = max(0, min(4, a.Dc - (d0 + lc)));
  const int64_t at = int64_t(b) * a.L * a.Dc + d0 + lc;
  const T* gp = reinterpret_cast<const T*>(a.dy) + at;
  const T* dp = reinterpret_cast<const T*>(a.delta) + at;
  const T* Cp = reinterpret_cast<const T*>(a.C) + int64_t(b) * a.L * a.N;
  float2 Ar[kQ / 2], g[kQ / 2];
  load_rates<T, kQ>(a, d, live, part * kQ, Ar);
#pragma unroll
  for (int k = 0; k < kQ / 2; ++k) g[k] = make_float2(0.f, 0.f);
  Raw4<T> ng, nd;
  RowShare<T, kN> nC;
  auto load = [&](int t0) {
    const int n = t0 + lr < a.L ? ln : 0;
    ng.load(gp + int64_t(t0 + lr) * a.Dc, n, vec);
    nd.load(dp + int64_t(t0 + lr) * a.Dc, n, vec);
    nC.load(Cp, t0, a.L, a.N, vecn, tid);
  };
  const int first = kSplit ? int(blockIdx.z) * a.seg : 0;
  // (below `first`: an empty segment)
  const int last = kSplit ? min((a.L - 1) / kStage * kStage, first + a.seg - kStage) : (a.L - 1) / kStage * kStage;
  if constexpr (kSplit) {
    float span = 0.f;
    if (blockIdx.z > 0) {   // as in the forward, last segment first
      load(max(last, 0));
      for (int t0 = last; t0 >= first; t0 -= kStage) {
        __syncthreads();
        write_pairs(dg + lr * kScanCh + lc, nd.get(vec), ng.get(vec));
        nC.store(sC, vecn, tid);
        __syncthreads();
        if (t0 > first) load(t0 - kStage);
        float stage_span = 0.f;
#pragma unroll
        for (int u = kStage - 1; u >= 0; --u) {
          const float2 w = dg[u * kScanCh + ch];
          float2 Cv[kQ / 2];
          row_pairs<kQ>(sC + u * kN + part * kQ, Cv);
          stage_span += w.x;
#pragma unroll
          for (int k = 0; k < kQ / 2; ++k)
            g[k] = __fmul2_rn(__ffma2_rn(Cv[k], both(w.y), g[k]), ex2_ss2(__fmul2_rn(both(w.x), Ar[k])));
        }
        span += stage_span;
      }
    }
    segment.join(int(gridDim.z) - 1, int(blockIdx.z), -1, ch, part, span, Ar, g);
  }
  load(kSplit ? max(last, 0) : last);
  for (int t0 = last; t0 >= first; t0 -= kStage) {
    __syncthreads();
    write_pairs(dg + lr * kScanCh + lc, nd.get(vec), ng.get(vec));
    nC.store(sC, vecn, tid);
    __syncthreads();
    if (t0 > first) load(t0 - kStage);
#pragma unroll
    for (int s0 = kStage - 4; s0 >= 0; s0 -= 4) {
      if ((s0 & 4)) {   // the last step of a chunk of eight: what enters it
        const int c = (t0 + s0) / kStep;
        if (live && c + 1 < a.chunks)
          store_states<kQ>(a.gck + ((int64_t(b) * a.chunks + c) * (kRange ? a.gD : a.Dc) + d) * a.N, part * kQ, a.N, vecn, g);
      }
      float2 av[4][kQ / 2], Cv[4][kQ / 2];
      float gy[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float2 w = dg[(s0 + u) * kScanCh + ch];
        row_pairs<kQ>(sC + (s0 + u) * kN + part * kQ, Cv[u]);
        gy[u] = w.y;
#pragma unroll
        for (int k = 0; k < kQ / 2; ++k) av[u][k] = ex2_ss2(__fmul2_rn(both(w.x), Ar[k]));
      }
#pragma unroll
      for (int u = 3; u >= 0; --u)
#pragma unroll
        for (int k = 0; k < kQ / 2; ++k) g[k] = __fmul2_rn(__ffma2_rn(Cv[u][k], both(gy[u]), g[k]), av[u][k]);
    }
  }
  if constexpr (kSplit) cg::this_cluster().sync();
}

// ---- gradients of a chunk ----------------------------------------------------------------------------------------
// A CTA of 128 threads takes 64 channels of one batch element and works through `per_cta` chunks of eight steps, 16
// states at a time.  A thread owns two channels (o and o + 32) and four states of each: both sums over channels (dB,
// dC) start inside the thread, which halves the shared-memory traffic of one channel per thread, and the pairs of the
// packed arithmetic are neighbouring states.  The eight steps are taken as two halves, the second first: the states
// and decays of four steps of eight (channel, state) pairs are 64 registers, those of all eight steps would be 128 and
// leave two warps per scheduler; the first half's steps are run twice for it (1.5 ex2 per step and state).  Bound: shared
// memory (32 words per cycle and SM): per pair and step 3 words of operands, 2 of the dB / dC tile, 1 for the rest; and a chunk's first loads, which
// a prefetch into L2 one chunk ahead shortens.  Backward of f32 (8, 1024, 2048, 16), all kernels: 1123 -> 451 us.
constexpr int kBwdCh = 64;
constexpr int kBwdThreads = 128;
constexpr int kHalf = kStep / 2;
// sums over the states of a chunk, [step][which][channel]: the four lanes that hold (channel, channel + 32) x (two
// sums) of one owner write to banks 8 apart
constexpr int kSumCol = 48 - 32, kSumWhich = 104, kSumStep = 184;

__device__ __forceinline__ void red_add4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}
// up to four sums of a row of N states starting at state n0
__device__ __forceinline__ void add_states(float* row, int n0, int N, bool vec, float4 v) {
  if (vec) {
    if (n0 < N) red_add4(row + n0, v);
  } else {
    if (n0 + 0 < N) atomicAdd(row + n0 + 0, v.x);
    if (n0 + 1 < N) atomicAdd(row + n0 + 1, v.y);
    if (n0 + 2 < N) atomicAdd(row + n0 + 2, v.z);
    if (n0 + 3 < N) atomicAdd(row + n0 + 3, v.w);
  }
}

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// kBlocks: blocks of 16 states (1: the sums of dA stay in registers; more: in shared memory, a slot per thread)
template <typename T, int kBlocks, bool kRange>
__global__ void __launch_bounds__(kBwdThreads, 3) ss_bwd_kernel(SsArgs a) {
  constexpr int kN = 16 * kBlocks;
  extern __shared__ __align__(16) float smem_ss[];
  float4* dxg = reinterpret_cast<float4*>(smem_ss);                // [kStep][kBwdCh]: delta, delta x, dy, x
  float* sB = reinterpret_cast<float*>(dxg + kStep * kBwdCh);      // [kStep][kN]
  float* sC = sB + kStep * kN;
  float* tile = sC + kStep * kN;                                   // [kHalf][32 owners][32]: dB, dC terms of 16 states
  float* sums = tile + kHalf * 32 * 32;                            // [kStep][kSumStep]
  float4* sdA = reinterpret_cast<float4*>(sums + kStep * kSumStep);   // kBlocks > 1: [kBlocks][2][kBwdThreads]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, part = tid & 3, o = tid >> 2;
  const int d0 = (kRange ? a.d_first : 0) + blockIdx.x * kBwdCh, b = blockIdx.z;
  const bool vec = a.vec != 0, vecn = a.vecn != 0;
  const bool hi = part & 2, lo = part & 1;
  // channel ch of dxg: permuted within eight so that both the writers (four channels each) and the readers (eight
  // neighbours per warp) meet distinct banks
  auto place = [](int ch) { return (ch & ~7) | ((ch ^ (ch >> 3)) & 7); };
  const int at0 = place(o), at1 = place(o + 32);
  // this thread's four channels of one step of a chunk
  const int lr = tid >> 4, lc = (tid & 15) * 4, ln = max(0, min(4, a.Dc - (d0 + lc)));
  const int64_t at = int64_t(b) * a.L * a.Dc + d0 + lc;
  float4 dDs = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 Ar[2][2], dA[2][2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    load_rates<T, 4>(a, d0 + o + 32 * j, d0 + o + 32 * j < a.Dc, part * 4, Ar[j]);
    dA[j][0] = dA[j][1] = make_float2(0.f, 0.f);
    if constexpr (kBlocks > 1) {
#pragma unroll
      for (int nb = 0; nb < kBlocks; ++nb) sdA[(nb * 2 + j) * kBwdThreads + tid] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
  }
  const int c_end = min(a.chunks, int(blockIdx.y + 1) * a.per_cta);
  for (int c = blockIdx.y * a.per_cta; c < c_end; ++c) {
    const int t0 = c * kStep;
    const int n = t0 + lr < a.L ? ln : 0;
    const int64_t row = at + int64_t(t0 + lr) * a.Dc;
    const float4 x4 = load4<T>(reinterpret_cast<const T*>(a.x) + row, n, vec);
    const float4 dl4 = load4<T>(reinterpret_cast<const T*>(a.delta) + row, n, vec);
    const float4 gy4 = load4<T>(reinterpret_cast<const T*>(a.dy) + row, n, vec);
    if (c + 1 < c_end) {   // the next chunk's rows and states, as far as L2
      const int64_t next = at + int64_t(min(t0 + kStep + lr, a.L - 1)) * a.Dc;
      if (ln > 0) {
        prefetch_l2(reinterpret_cast<const T*>(a.x) + next);
        prefetch_l2(reinterpret_cast<const T*>(a.delta) + next);
        prefetch_l2(reinterpret_cast<const T*>(a.dy) + next);
      }
      const int64_t st = (int64_t(b) * a.chunks + c) * a.Dc * a.N, n0 = int64_t(d0) * a.N + tid * (kN / 2);
      if (n0 < int64_t(a.Dc) * a.N) {
        prefetch_l2(a.ckpt + st + n0);
        if (!kRange && c + 2 < a.chunks) prefetch_l2(a.gck + st + int64_t(a.Dc) * a.N + n0);
      }
    }
    __syncthreads();   // (the chunk before has been read)
    // (steps past the sequence's end and channels past the last are zeros: they add nothing)
    dxg[lr * kBwdCh + place(lc + 0)] = make_float4(dl4.x, dl4.x * x4.x, gy4.x, x4.x);
    dxg[lr * kBwdCh + place(lc + 1)] = make_float4(dl4.y, dl4.y * x4.y, gy4.y, x4.y);
    dxg[lr * kBwdCh + place(lc + 2)] = make_float4(dl4.z, dl4.z * x4.z, gy4.z, x4.z);
    dxg[lr * kBwdCh + place(lc + 3)] = make_float4(dl4.w, dl4.w * x4.w, gy4.w, x4.w);
    for (int i = tid; i < kStep * kN; i += kBwdThreads) {
      const int s = i / kN, ns = i - s * kN;
      const bool in = ns < a.N && t0 + s < a.L;
      const int64_t bc = (int64_t(b) * a.L + t0 + s) * a.N + ns;
      sB[i] = in ? to_f32<T>(reinterpret_cast<const T*>(a.B)[bc]) : 0.f;
      sC[i] = in ? to_f32<T>(reinterpret_cast<const T*>(a.C)[bc]) : 0.f;
    }
    __syncthreads();
#pragma unroll 1
    for (int nb = 0; nb < kBlocks; ++nb) {
      const int n0 = nb * 16 + part * 4;
      float2 h0[2][2], g[2][2];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int d = d0 + o + 32 * j;
        const int have = d < a.Dc ? max(0, min(4, a.N - n0)) : 0;
        const int64_t st = ((int64_t(b) * a.chunks + c) * a.Dc + d) * a.N + n0;
        const int64_t gt = kRange ? ((int64_t(b) * a.chunks + c) * a.gD + d) * a.N + n0 : st;
        const float4 hv = load4<float>(a.ckpt + st - int64_t(a.Dc) * a.N, c > 0 ? have : 0, vecn);
        const float4 gv = load4<float>(a.gck + gt, c + 1 < a.chunks ? have : 0, vecn);
        h0[j][0] = make_float2(hv.x, hv.y);
        h0[j][1] = make_float2(hv.z, hv.w);
        g[j][0] = make_float2(gv.x, gv.y);
        g[j][1] = make_float2(gv.z, gv.w);
        if constexpr (kBlocks > 1) load_rates<T, 4>(a, d, d < a.Dc, n0, Ar[j]);
      }
#pragma unroll 1
      for (int half = 1; half >= 0; --half) {
        float2 hs[2][2];                        // the state before the half
#pragma unroll
        for (int j = 0; j < 2; ++j) { hs[j][0] = h0[j][0]; hs[j][1] = h0[j][1]; }
        if (half == 1) {
#pragma unroll
          for (int s = 0; s < kHalf; ++s) {
            const float4 Bw = *reinterpret_cast<const float4*>(sB + s * kN + n0);
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const float2 w = *reinterpret_cast<const float2*>(dxg + s * kBwdCh + (j ? at1 : at0));
              const float2 dl = both(w.x), u = both(w.y);
              hs[j][0] = __ffma2_rn(ex2_ss2(__fmul2_rn(dl, Ar[j][0])), hs[j][0], __fmul2_rn(u, make_float2(Bw.x, Bw.y)));
              hs[j][1] = __ffma2_rn(ex2_ss2(__fmul2_rn(dl, Ar[j][1])), hs[j][1], __fmul2_rn(u, make_float2(Bw.z, Bw.w)));
            }
          }
        }
        float2 av[kHalf][2][2], h[kHalf][2][2];
        float4 w[kHalf][2];
        const int sb = half * kHalf;
#pragma unroll
        for (int s = 0; s < kHalf; ++s) {
          const float4 Bw = *reinterpret_cast<const float4*>(sB + (sb + s) * kN + n0);
          const float2 Bv[2] = {make_float2(Bw.x, Bw.y), make_float2(Bw.z, Bw.w)};
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            w[s][j] = dxg[(sb + s) * kBwdCh + (j ? at1 : at0)];
            const float2 dl = both(w[s][j].x), u = both(w[s][j].y);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              av[s][j][k] = ex2_ss2(__fmul2_rn(dl, Ar[j][k]));
              h[s][j][k] = __ffma2_rn(av[s][j][k], s ? h[s - 1][j][k] : hs[j][k], __fmul2_rn(u, Bv[k]));
            }
          }
        }
        __syncthreads();   // (the tile's last sums have been read)
#pragma unroll
        for (int s = kHalf - 1; s >= 0; --s) {
          const float4 Bw = *reinterpret_cast<const float4*>(sB + (sb + s) * kN + n0);
          const float4 Cw = *reinterpret_cast<const float4*>(sC + (sb + s) * kN + n0);
          const float2 Bv[2] = {make_float2(Bw.x, Bw.y), make_float2(Bw.z, Bw.w)};
          const float2 Cv[2] = {make_float2(Cw.x, Cw.y), make_float2(Cw.z, Cw.w)};
          float2 dB[2], dC[2];
          float s1[2], s2[2];
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float2 dl = both(w[s][j].x), u = both(w[s][j].y), gy = both(w[s][j].z);
            float2 e1 = make_float2(0.f, 0.f), e2 = make_float2(0.f, 0.f);
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              const float2 gt = __ffma2_rn(Cv[k], gy, g[j][k]);                                  // dL/dh_t
              const float2 ga = __fmul2_rn(gt, av[s][j][k]);                                     // dL/dh_{t-1} so far
              const float2 da = __fmul2_rn(ga, s ? h[s - 1][j][k] : hs[j][k]);                   // dL/d(delta_t A_n)
              e1 = __ffma2_rn(da, Ar[j][k], e1);
              dA[j][k] = __ffma2_rn(da, dl, dA[j][k]);
              e2 = __ffma2_rn(gt, Bv[k], e2);
              dB[k] = j ? __ffma2_rn(gt, u, dB[k]) : __fmul2_rn(gt, u);
              dC[k] = j ? __ffma2_rn(gy, h[s][j][k], dC[k]) : __fmul2_rn(gy, h[s][j][k]);
              g[j][k] = ga;
            }
            s1[j] = e1.x + e1.y;
            s2[j] = e2.x + e2.y;
          }
          // a row is one owner's 16 dB and 16 dC terms, the halves swapped in every other row (bank conflicts)
          float* tr = tile + (s * 32 + o) * 32;
          *reinterpret_cast<float4*>(tr + part * 4 + (o & 1 ? 16 : 0)) = make_float4(dB[0].x, dB[0].y, dB[1].x, dB[1].y);
          *reinterpret_cast<float4*>(tr + part * 4 + (o & 1 ? 0 : 16)) = make_float4(dC[0].x, dC[0].y, dC[1].x, dC[1].y);
          // sums over the states: over the four lanes, each of which ends with one channel and one of the two sums
          float k1 = hi ? s1[1] : s1[0], k2 = hi ? s2[1] : s2[0];
          k1 += __shfl_xor_sync(0xffffffffu, hi ? s1[0] : s1[1], 2);
          k2 += __shfl_xor_sync(0xffffffffu, hi ? s2[0] : s2[1], 2);
          float r = (lo ? k2 : k1) + __shfl_xor_sync(0xffffffffu, lo ? k1 : k2, 1);
          float* out = sums + (sb + s) * kSumStep + (lo ? kSumWhich : 0) + o + (hi ? 32 + kSumCol : 0);
          if (kBlocks > 1 && nb > 0) r += *out;
          *out = r;
        }
        __syncthreads();
        // column sums of the half's tile: a warp takes one step, a lane four of its 32 columns of eight owners
        {
          const int vg = lane & 7, slot = lane >> 3, t = t0 + sb + warp;
          float2 p0 = make_float2(0.f, 0.f), p1 = make_float2(0.f, 0.f);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 v = *reinterpret_cast<const float4*>(tile + (warp * 32 + slot * 8 + i) * 32 + (vg ^ (i & 1 ? 4 : 0)) * 4);
            p0 = __fadd2_rn(p0, make_float2(v.x, v.y));
            p1 = __fadd2_rn(p1, make_float2(v.z, v.w));
          }
#pragma unroll
          for (int m = 8; m < 32; m <<= 1) {
            p0.x += __shfl_xor_sync(0xffffffffu, p0.x, m);
            p0.y += __shfl_xor_sync(0xffffffffu, p0.y, m);
            p1.x += __shfl_xor_sync(0xffffffffu, p1.x, m);
            p1.y += __shfl_xor_sync(0xffffffffu, p1.y, m);
          }
          if (slot == 0 && t < a.L)
            add_states((vg < 4 ? a.accB : a.accC) + (int64_t(b) * a.L + t) * a.N, nb * 16 + (vg & 3) * 4, a.N, vecn,
                       make_float4(p0.x, p0.y, p1.x, p1.y));
        }
      }
      if constexpr (kBlocks > 1) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float4* slot = sdA + (nb * 2 + j) * kBwdThreads + tid;
          const float4 was = *slot;
          *slot = make_float4(was.x + dA[j][0].x, was.y + dA[j][0].y, was.z + dA[j][1].x, was.w + dA[j][1].y);
          dA[j][0] = dA[j][1] = make_float2(0.f, 0.f);
        }
      }
    }
    // dx_t = delta_t sum_n g B + D dy_t,  ddelta_t = sum_n g h_{t-1} a A + x_t sum_n g B   (the last barrier above
    // stands between these sums and their writers)
    const float* sr = sums + lr * kSumStep + lc + (lc >= 32 ? kSumCol : 0);
    const float4 v1 = *reinterpret_cast<const float4*>(sr), v2 = *reinterpret_cast<const float4*>(sr + kSumWhich);
    const float4* own = dxg + lr * kBwdCh;
    const float4 e0 = own[place(lc)], e1 = own[place(lc + 1)], e2 = own[place(lc + 2)], e3 = own[place(lc + 3)];
    const float4 dl = make_float4(e0.x, e1.x, e2.x, e3.x), gy = make_float4(e0.z, e1.z, e2.z, e3.z), x = make_float4(e0.w, e1.w, e2.w, e3.w);
    constexpr float kLn2 = 1.f / kLog2eSs;
    store4<T>(reinterpret_cast<T*>(a.ddelta) + row,
              make_float4(fmaf(x.x, v2.x, v1.x * kLn2), fmaf(x.y, v2.y, v1.y * kLn2), fmaf(x.z, v2.z, v1.z * kLn2), fmaf(x.w, v2.w, v1.w * kLn2)), n, vec);
    float4 dx = make_float4(dl.x * v2.x, dl.y * v2.y, dl.z * v2.z, dl.w * v2.w);
    if (a.D) {
      const float4 Dd = load4<T>(reinterpret_cast<const T*>(a.D) + d0 + lc, ln, false);
      dx = make_float4(fmaf(Dd.x, gy.x, dx.x), fmaf(Dd.y, gy.y, dx.y), fmaf(Dd.z, gy.z, dx.z), fmaf(Dd.w, gy.w, dx.w));
      dDs = make_float4(fmaf(gy.x, x.x, dDs.x), fmaf(gy.y, x.y, dDs.y), fmaf(gy.z, x.z, dDs.z), fmaf(gy.w, x.w, dDs.w));
    }
    store4<T>(reinterpret_cast<T*>(a.dx) + row, dx, n, vec);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const int d = d0 + o + 32 * j;
    if (d < a.Dc) {
      if constexpr (kBlocks > 1) {
        for (int nb = 0; nb < kBlocks; ++nb)
          add_states(a.accA + int64_t(d) * a.N, nb * 16 + part * 4, a.N, vecn, sdA[(nb * 2 + j) * kBwdThreads + tid]);
      } else {
        add_states(a.accA + int64_t(d) * a.N, part * 4, a.N, vecn, make_float4(dA[j][0].x, dA[j][0].y, dA[j][1].x, dA[j][1].y));
      }
    }
  }
  if (a.accD) {
    // (lanes 16 apart hold two steps of the same channels)
    dDs.x += __shfl_xor_sync(0xffffffffu, dDs.x, 16);
    dDs.y += __shfl_xor_sync(0xffffffffu, dDs.y, 16);
    dDs.z += __shfl_xor_sync(0xffffffffu, dDs.z, 16);
    dDs.w += __shfl_xor_sync(0xffffffffu, dDs.w, 16);
    if (lane < 16) add_states(a.accD + d0 + lc, 0, ln, false, dDs);
  }
}

// The fp32 accumulators in the storage dtype: four arrays in one launch.
struct SsFinish {
  const float* src[4];
  void* dst[4];
  int64_t n[4];
};
template <typename T>
__global__ void __launch_bounds__(256) ss_finish_kernel(SsFinish f) {
  const float* src = f.src[blockIdx.y];
  T* dst = static_cast<T*>(f.dst[blockIdx.y]);
  for (int64_t i = int64_t(blockIdx.x) * 256 + threadIdx.x; i < f.n[blockIdx.y]; i += int64_t(gridDim.x) * 256)
    dst[i] = from_f32<T>(src[i]);
}

int pick_n(int N) { return N <= 8 ? 8 : (N <= 16 ? 16 : (N <= 32 ? 32 : (N <= 64 ? 64 : 0))); }

int check_common(const nb200_selective_scan_params* p, const char* what) {
  if (!p) { set_error("%s: NULL parameter block", what); return NB200_ERR_INVALID; }
  if (p->struct_size != sizeof(nb200_selective_scan_params)) {
    set_error("%s: ABI mismatch: struct_size %zu, library expects %zu", what, size_t(p->struct_size),
              sizeof(nb200_selective_scan_params));
    return NB200_ERR_INVALID;
  }
  if (p->dtype != NB200_F32 && p->dtype != NB200_BF16 && p->dtype != NB200_F16) { set_error("%s: bad dtype", what); return NB200_ERR_INVALID; }
  if (p->batch < 0 || p->length < 0 || p->channels <= 0 || p->states <= 0) { set_error("%s: bad extents", what); return NB200_ERR_INVALID; }
  if (!pick_n(p->states)) { set_error("%s: more than 64 states per channel (%d)", what, p->states); return NB200_ERR_UNSUPPORTED; }
  if (p->batch > 65535) { set_error("%s: more than 65535 batch elements", what); return NB200_ERR_UNSUPPORTED; }
  return NB200_OK;
}

bool aligned(const void* p, size_t to) { return reinterpret_cast<uintptr_t>(p) % to == 0; }

template <typename T>
SsArgs args_of(const nb200_selective_scan_params* p) {
  SsArgs a{};
  a.x = p->x; a.delta = p->delta; a.A = p->A; a.B = p->B; a.C = p->C; a.D = p->D; a.dy = p->dy;
  a.y = p->y; a.dx = p->dx; a.ddelta = p->ddelta; a.ckpt = p->checkpoints;
  a.batch = p->batch; a.L = p->length; a.Dc = p->channels; a.N = p->states;
  a.chunks = p->length / kStep + (p->length % kStep != 0);
  // four channels (states) as one word: every row then starts on that word's boundary, and no group is cut short
  constexpr size_t kWord = 4 * sizeof(T);
  a.vec = p->channels % 4 == 0 && aligned(p->x, kWord) && aligned(p->delta, kWord) && aligned(p->y, kWord) &&
          aligned(p->dy, kWord) && aligned(p->dx, kWord) && aligned(p->ddelta, kWord);
  a.vecn = p->states % 4 == 0 && aligned(p->B, kWord) && aligned(p->C, kWord) && aligned(p->checkpoints, 16) &&
           aligned(p->workspace, 16);
  return a;
}

int segment_steps(int length, int splits) {
  const int stages = (length + kStage - 1) / kStage;
  return (stages + splits - 1) / splits * kStage;
}
// Segments of the walks, 1: not split.  Two give nothing (1.6 times the work: (1, 2048, 2048, 16) 352 -> 341 us, (4, 2048,
// 1024, 16) 446 -> 465), so four or eight.  `load` is the CTAs that they put on an SM.  Up to one wave of clusters a step
// costs its latencies whatever the load, and the segments gain; past it they only add work (f32 forward, N = 16, 296 CTAs of
// one walk, 256 / 2048 steps: 21 / 139 us, in four 28 / 166, in eight 34 / 143; N = 64, 148 CTAs: 40 / 285, in four 68 / 389,
// in eight 173 / 424).  More states hold more registers and shared memory and take longer to join, so the room shrinks and
// the least length, which grows with the load, rises with them.  The lines lie where one walk and segments were level over 2
// to 592 CTAs of one walk and 97 to 2048 steps, N = 8 / 16 / 32 / 64: on 74 CTAs of 2048 steps one walk takes 105 / 132 /
// 167 / 285 us, four 64 / 72 / 105 / 210, eight 40 / 50 / 81 / 243; on 148 of 256 steps 17 / 20 / 25 / 40, 15 / 17 / 26 / 68
// and 17 / 22 / 61 / 173.  As many as left eight CTAs per SM (four from 32 states on) and 24 steps each, as the rule was before,
// made one in ten of these slower than one walk (N = 64, 74 CTAs, 192 steps: 31 -> 84 us).
int walk_splits(int64_t ctas, int64_t length, int states, bool half, bool adjoint) {
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  const float load4 = 4.f * float(ctas) / float(sms), load8 = 2.f * load4, steps = float(length);
  struct Rule { float room8, least8, slope8, room4, slope4; };   // most load; least steps, in all and per load
  const int n = pick_n(states);
  Rule r;
  if (n == 8) r = {7.f, 192.f, 32.f, 7.6f, half && !adjoint ? 16.f : 25.f};
  else if (n == 16) r = adjoint ? Rule{7.f, 192.f, 96.f, 6.f, 50.f} : Rule{7.7f, 192.f, load8 > 7.f ? 120.f : 64.f, 7.6f, 25.f};   // (the wave's end: (4, 927, 550, 16))
  else if (n == 32) r = {5.f, 384.f, 192.f, 5.5f, adjoint ? 100.f : 75.f};
  else if (half && !adjoint) r = {2.f, 768.f, 0.f, 5.5f, 45.f};   // (its one walk is slow: 74 CTAs, 2048 steps 521 us, f32 285)
  else r = {2.f, 768.f, 0.f, 3.f, 150.f};
  if (load8 <= r.room8 && steps >= fmaxf(r.least8, r.slope8 * load8)) return 8;
  if (load4 <= r.room4 && steps >= fmaxf(96.f, r.slope4 * load4)) return 4;
  // 16-bit storage of few states: a little past one wave too (296 CTAs, 2048 steps: N = 8 128 -> 115 us, N = 16 140 -> 136)
  if (half && !adjoint && n <= 16 && load8 <= 20.f && steps >= 128.f * float(n)) return 8;
  return 1;
}

// One of the walks over `grid`, as clusters of `splits` CTAs along z.
template <typename Kernel>
int walk_launch(Kernel kernel, dim3 grid, int splits, const SsArgs& a, cudaStream_t st, const char* what) {
  if (splits == 1) {
    kernel<<<grid, kScanThreads, 0, st>>>(a);
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid.x, grid.y, unsigned(splits));
    cfg.blockDim = dim3(kScanThreads);
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 1;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = unsigned(splits);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, a);
  }
  count_launch();
  return check_launch(what);
}
template <typename T, bool kShort, bool kSplit>
int fwd_launch(const nb200_selective_scan_params* p, const SsArgs& a, int splits, cudaStream_t st) {
  const dim3 grid((p->channels + kScanCh - 1) / kScanCh, p->batch);
  auto kernel = ss_fwd_kernel<T, 64, kShort, kSplit>;
  switch (pick_n(p->states)) {
    case 8: kernel = ss_fwd_kernel<T, 8, kShort, kSplit>; break;
    case 16: kernel = ss_fwd_kernel<T, 16, kShort, kSplit>; break;
    case 32: kernel = ss_fwd_kernel<T, 32, kShort, kSplit>; break;
  }
  return walk_launch(kernel, grid, splits, a, st, "selective_scan_fwd_kernel");
}

template <typename T>
int fwd_t(const nb200_selective_scan_params* p, cudaStream_t st) {
  SsArgs a = args_of<T>(p);
  if (p->length <= kStage - 4) return fwd_launch<T, true, false>(p, a, 1, st);
  const int64_t ctas = int64_t(p->channels + kScanCh - 1) / kScanCh * p->batch;
  const int splits = walk_splits(ctas, p->length, p->states, sizeof(T) == 2, false);
  if (splits == 1) return fwd_launch<T, false, false>(p, a, 1, st);
  a.seg = segment_steps(p->length, splits);
  return fwd_launch<T, false, true>(p, a, splits, st);
}

// workspace of the backward: the fp32 accumulators, then the adjoint states between the chunks
size_t acc_floats(const nb200_selective_scan_params* p) {
  return 2 * size_t(p->batch) * p->length * p->states + size_t(p->channels) * p->states + size_t(p->channels);
}
// The adjoint states take as much again as the checkpoints.  With less workspace the backward runs for a range of batch
// elements, or of one element's channels in whole groups of 64, at a time, each in the same part of it.
struct Range { int batch, channels; };
size_t state_floats(const nb200_selective_scan_params* p, Range r) {
  return size_t(r.batch) * (p->length / kStep + (p->length % kStep != 0)) * p->states * r.channels;
}
Range least_range(const nb200_selective_scan_params* p) { return {p->batch < 1 ? p->batch : 1, p->channels < kBwdCh ? p->channels : kBwdCh}; }
Range range_of(const nb200_selective_scan_params* p, size_t floats) {
  Range r{p->batch, p->channels};
  if (state_floats(p, r) <= floats) return r;
  r.batch = 1;
  const size_t element = state_floats(p, r);
  if (element <= floats) {
    r.batch = int(floats / element);
  } else {
    r.channels = int(floats / (element / p->channels) / kBwdCh) * kBwdCh;   // (an element of one group or less fits)
  }
  return r;
}
size_t acc_bytes(const nb200_selective_scan_params* p) { return (sizeof(float) * acc_floats(p) + 255) / 256 * 256; }

template <typename T, int kBlocks, bool kRange>
int bwd_launch(const SsArgs& a, dim3 grid, cudaStream_t st) {
  constexpr size_t smem = kStep * kBwdCh * sizeof(float4) +
                          sizeof(float) * (2 * kStep * 16 * kBlocks + kHalf * 32 * 32 + kStep * kSumStep) +
                          (kBlocks > 1 ? sizeof(float4) * kBlocks * 2 * kBwdThreads : 0);
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(ss_bwd_kernel<T, kBlocks, kRange>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) != cudaSuccess) {
    set_error("selective_scan_bwd: cudaFuncSetAttribute(%zu): %s", smem, cudaGetErrorString(cudaGetLastError()));
    return NB200_ERR_LAUNCH;
  }
  ss_bwd_kernel<T, kBlocks, kRange><<<grid, kBwdThreads, smem, st>>>(a);
  count_launch();
  return check_launch("selective_scan_bwd_kernel");
}

// Chunks per CTA of the gradients: as many as leave about eight CTAs for every one that the GPU holds at a time (three per
// SM), so that the last wave is short, at most 16 (a CTA's own start and its sums are spread well enough over those); up to
// four such waves are made one; up to six where few channels and many chunks would have more than about 192 CTAs add their
// sums of dA and dD to the same addresses, down to about two CTAs per SM.  us with 1 / 4 / 6 / 16: (256, 64, 64, 16) 191 / 80 / 70 / -, (8, 2048, 128, 16) 285 / 180 /
// 174 / 174, (16, 512, 256, 16) 201 / 102 / 97 / 96, (256, 128, 64, 32) 401 / 194 / 173 / 186, (64, 512, 64, 64) 482 / 354 / 341 / 371, (8, 1024, 512, 16) 236 / 158 / 162 / 183, (8, 1024, 2048, 16) 502 / 451
// / 447 / 448, (8, 128, 2048, 8) 63 / 63 / 64 / 74, (2, 333, 1030, 16) 45 / 42 / 47 / 75.
int chunks_per_cta(int64_t groups, int64_t batch, int64_t chunks) {
  int sms = 0, dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (sms <= 0) sms = 148;
  const int64_t work = groups * batch * chunks, spread = batch * chunks / 192, filled = work / (2 * int64_t(sms));
  const int64_t resident = 3 * int64_t(sms), shared = spread < filled ? spread : filled;
  int64_t per = work / (8 * resident);
  per = per < 1 ? 1 : (per > 16 ? 16 : per);
  const int64_t more = work <= 4 * resident ? (work + resident - 1) / resident : (shared < 6 ? shared : 6);
  per = per < more ? more : per;
  const int64_t least = (chunks + 65534) / 65535;   // (grid.y)
  per = per < least ? least : per;
  return int(per < chunks ? per : chunks);
}

template <typename T, bool kRange, bool kSplit>
int adjoint_launch(const nb200_selective_scan_params* p, const SsArgs& a, dim3 grid, int splits, cudaStream_t st) {
  auto kernel = ss_adjoint_kernel<T, 64, kRange, kSplit>;
  switch (pick_n(p->states)) {
    case 8: kernel = ss_adjoint_kernel<T, 8, kRange, kSplit>; break;
    case 16: kernel = ss_adjoint_kernel<T, 16, kRange, kSplit>; break;
    case 32: kernel = ss_adjoint_kernel<T, 32, kRange, kSplit>; break;
  }
  return walk_launch(kernel, grid, splits, a, st, "selective_scan_adjoint_kernel");
}

// The two kernels of one range: `a` with its batch pointers at the range's first element.
template <typename T, bool kRange>
int bwd_range(const nb200_selective_scan_params* p, const SsArgs& a, Range r, cudaStream_t st) {
  if (a.chunks > 1) {
    const dim3 grid((r.channels + kScanCh - 1) / kScanCh, r.batch);
    const int splits = kRange ? 1 : walk_splits(int64_t(grid.x) * grid.y, p->length, p->states, sizeof(T) == 2, true);
    SsArgs w = a;
    w.seg = segment_steps(p->length, splits);
    if (int rc = splits == 1 ? adjoint_launch<T, kRange, false>(p, w, grid, 1, st) : adjoint_launch<T, false, true>(p, w, grid, splits, st)) return rc;
  }
  const unsigned groups = (r.channels + kBwdCh - 1) / kBwdCh;
  const dim3 grid(groups, unsigned((a.chunks + a.per_cta - 1) / a.per_cta), unsigned(r.batch));
  switch (pick_n(p->states)) {
    case 8:
    case 16: return bwd_launch<T, 1, kRange>(a, grid, st);
    case 32: return bwd_launch<T, 2, kRange>(a, grid, st);
    default: return bwd_launch<T, 4, kRange>(a, grid, st);
  }
}

template <typename T>
int bwd_t(const nb200_selective_scan_params* p, cudaStream_t st) {
  SsArgs a = args_of<T>(p);
  const size_t need = acc_bytes(p) + sizeof(float) * state_floats(p, least_range(p));
  if (!p->workspace || p->workspace_bytes < need) {
    set_error("selective_scan_bwd: workspace of at least %zu bytes needed (nb200_selective_scan_workspace_least_bytes), "
              "%zu given", need, size_t(p->workspace_bytes));
    return NB200_ERR_WORKSPACE;
  }
  float* acc = static_cast<float*>(p->workspace);
  if (cudaMemsetAsync(acc, 0, sizeof(float) * acc_floats(p), st) != cudaSuccess) return check_launch("selective_scan_bwd: clearing the workspace");
  const size_t bln = size_t(p->batch) * p->length * p->states, dn = size_t(p->channels) * p->states;
  a.accB = acc; a.accC = acc + bln; a.accA = acc + 2 * bln; a.accD = p->D ? acc + 2 * bln + dn : nullptr;
  a.gck = reinterpret_cast<float*>(static_cast<char*>(p->workspace) + acc_bytes(p));
  if (p->batch > 0 && p->length > 0) {   // (nothing to walk otherwise: dA and dD are the zeros just written)
    const Range whole = range_of(p, (p->workspace_bytes - acc_bytes(p)) / sizeof(float));
    a.per_cta = chunks_per_cta((whole.channels + kBwdCh - 1) / kBwdCh, whole.batch, a.chunks);
    a.gD = whole.channels;
    for (int b = 0; b < p->batch; b += whole.batch) {
      SsArgs part = a;
      const size_t steps = size_t(b) * p->length, wide = steps * p->channels * sizeof(T), rows = steps * p->states;
      part.x = static_cast<const char*>(a.x) + wide;
      part.delta = static_cast<const char*>(a.delta) + wide;
      part.dy = static_cast<const char*>(a.dy) + wide;
      part.dx = static_cast<char*>(a.dx) + wide;
      part.ddelta = static_cast<char*>(a.ddelta) + wide;
      part.B = static_cast<const char*>(a.B) + rows * sizeof(T);
      part.C = static_cast<const char*>(a.C) + rows * sizeof(T);
      part.accB = a.accB + rows;
      part.accC = a.accC + rows;
      part.ckpt = a.ckpt + state_floats(p, {b, p->channels});
      for (int d = 0; d < p->channels; d += whole.channels) {
        part.d_first = d;
        part.gck = a.gck - int64_t(d) * p->states;
        const Range r{p->batch - b < whole.batch ? p->batch - b : whole.batch,
                      p->channels - d < whole.channels ? p->channels - d : whole.channels};
        if (int rc = whole.channels < p->channels ? bwd_range<T, true>(p, part, r, st) : bwd_range<T, false>(p, part, r, st)) return rc;
      }
    }
  }
  SsFinish f{{a.accB, a.accC, a.accA, acc + 2 * bln + dn}, {p->dB, p->dC, p->dA, p->dD},
             {int64_t(bln), int64_t(bln), int64_t(dn), p->D ? int64_t(p->channels) : 0}};
  int64_t most = 0;
  for (int64_t n : f.n) most = n > most ? n : most;
  const int64_t blocks = (most + 1023) / 1024;
  ss_finish_kernel<T><<<dim3(unsigned(blocks < 4096 ? blocks : 4096), 4), 256, 0, st>>>(f);
  count_launch();
  return check_launch("selective_scan_finish_kernel");
}

}  // namespace
}  // namespace nb200

using namespace nb200;

extern "C" NB200_API int nb200_selective_scan_workspace_bytes(const nb200_selective_scan_params* p, size_t* bytes) {
  if (!bytes) { set_error("bytes out-pointer is NULL"); return NB200_ERR_INVALID; }
  if (int rc = check_common(p, "selective_scan_workspace_bytes")) return rc;
  *bytes = acc_bytes(p) + sizeof(float) * state_floats(p, {p->batch, p->channels});
  return NB200_OK;
}

extern "C" NB200_API int nb200_selective_scan_workspace_least_bytes(const nb200_selective_scan_params* p, size_t* bytes) {
  if (!bytes) { set_error("bytes out-pointer is NULL"); return NB200_ERR_INVALID; }
  if (int rc = check_common(p, "selective_scan_workspace_least_bytes")) return rc;
  *bytes = acc_bytes(p) + sizeof(float) * state_floats(p, least_range(p));
  return NB200_OK;
}

extern "C" NB200_API int nb200_selective_scan_checkpoint_bytes(const nb200_selective_scan_params* p, size_t* bytes) {
  if (!bytes) { set_error("bytes out-pointer is NULL"); return NB200_ERR_INVALID; }
  if (int rc = check_common(p, "selective_scan_checkpoint_bytes")) return rc;
  *bytes = sizeof(float) * state_floats(p, {p->batch, p->channels});
  return NB200_OK;
}

extern "C" NB200_API int nb200_selective_scan_fwd(const nb200_selective_scan_params* p, void* cuda_stream) {
  if (int rc = check_common(p, "selective_scan_fwd")) return rc;
  if (p->batch == 0 || p->length == 0) return NB200_OK;
  if (!p->x || !p->delta || !p->A || !p->B || !p->C || !p->y) { set_error("selective_scan_fwd: NULL operand"); return NB200_ERR_INVALID; }
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  prof_call_begin(st);
  switch (p->dtype) {
    case NB200_F32: return fwd_t<float>(p, st);
    case NB200_BF16: return fwd_t<__nv_bfloat16>(p, st);
    default: return fwd_t<__half>(p, st);
  }
}

extern "C" NB200_API int nb200_selective_scan_bwd(const nb200_selective_scan_params* p, void* cuda_stream) {
  if (int rc = check_common(p, "selective_scan_bwd")) return rc;
  const bool empty = p->batch == 0 || p->length == 0;
  if (!p->dA || (p->D && !p->dD) ||
      (!empty && (!p->x || !p->delta || !p->A || !p->B || !p->C || !p->dy || !p->dx || !p->ddelta || !p->dB || !p->dC ||
                  (p->length > kStep && !p->checkpoints)))) {
    set_error("selective_scan_bwd: NULL operand (x, delta, A, B, C, dy, checkpoints and every gradient are required)");
    return NB200_ERR_INVALID;
  }
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  prof_call_begin(st);
  switch (p->dtype) {
    case NB200_F32: return bwd_t<float>(p, st);
    case NB200_BF16: return bwd_t<__nv_bfloat16>(p, st);
    default: return bwd_t<__half>(p, st);
  }
}
