// RMS normalisation of q and k over the head dim (the `qk_norm=True` pre-op of attention) and its gradient, each as
// ONE launch for both tensors.
//
// The reference applies this outside its fused kernels, as separate element-wise XLA ops whose VJP autodiff chains
// onto the kernels' (reference src/nitrix/nn/attention/__init__.py:184-197; the op itself:
// src/nitrix/nn/attention/_reference.py:52-77, y = x * rsqrt(mean(x^2) + 1e-6), no learnable scale, fp32
// accumulation).  Here the pre-op keeps that place in the call sequence -- so the attention kernels and their
// gradients are untouched -- but costs one read and one write per tensor instead of a chain of element-wise passes:
// 16-byte loads, a row held in registers between the reduction and the scaling.
//
//   forward   y = x r,                       r = rsqrt(mean(x^2) + eps)
//   gradient  dx = r (g - y mean(g y))       (exact, eps included: dr/dx_i = -r^3 x_i / D)
#include <math.h>

#include "sdpa_common.cuh"

namespace nb200 {
namespace {

constexpr float kEps = 1e-6f;

struct NormTensor {
  const void* x;      // [b][h][n][D], last dim contiguous
  const void* g;      // gradient pass: dL/dy, dense [rows][D]
  void* y;            // forward: y; gradient pass: dx -- dense [rows][D]
  int64_t xs[3];      // element strides of x over (b, h, n)
  int H, N;
  int64_t rows;       // B * H * N
  int dense;          // x is dense [rows][D] as well
};

template <typename T>
__device__ __forceinline__ float to_f(T v);
template <>
__device__ __forceinline__ float to_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }
template <>
__device__ __forceinline__ float to_f<__half>(__half v) { return __half2float(v); }
template <typename T>
__device__ __forceinline__ T from_f(float v);
template <>
__device__ __forceinline__ float from_f<float>(float v) { return v; }
template <>
__device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }
template <>
__device__ __forceinline__ __half from_f<__half>(float v) { return __float2half_rn(v); }

// A group of `kLanes` lanes (the power of two that covers a row with kPer words of 16 bytes a lane: two at fp32 and head dims
// above 128) takes kRowsAhead rows, all of whose loads are issued before the first is used; the two tensors
// have their own ranges of CTAs.  Bound by HBM.  One row per warp, whatever its length, left half of the lanes idle at
// bf16 and head dim 128, four 64-bit divisions in front of a single load per lane, and took 40 us for the 85 MB of
// (8, 16, 197 + 1111, 128).
constexpr int kNormThreads = 256;

template <typename T, bool kGrad, int kLanes, int kPer, int kRowsAhead>
__global__ void __launch_bounds__(kNormThreads) qk_rms_norm_kernel(NormTensor a, NormTensor b, int D, unsigned blocks_a) {
  constexpr int kVec = 16 / int(sizeof(T));
  constexpr int kGroups = kNormThreads / kLanes;
  const bool second = blockIdx.x >= blocks_a;
  const NormTensor& t = second ? b : a;
  const int lane = threadIdx.x % kLanes, group = threadIdx.x / kLanes;
  const int64_t row0 = int64_t(blockIdx.x - (second ? blocks_a : 0)) * (kGroups * kRowsAhead) + group;
  uint4 xw[kRowsAhead][kPer], gw[kRowsAhead][kPer];
#pragma unroll
  for (int r = 0; r < kRowsAhead; ++r) {
    const int64_t row = row0 + r * kGroups;
    const T* x = reinterpret_cast<const T*>(t.x);
    if (row < t.rows) {
      if (t.dense) {
        x += row * D;
      } else {
        const int64_t bh = row / t.N, n = row - bh * t.N, bb = bh / t.H, h = bh - bb * t.H;
        x += bb * t.xs[0] + h * t.xs[1] + n * t.xs[2];
      }
    }
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int c0 = (p * kLanes + lane) * kVec;
      const bool in = row < t.rows && c0 < D;
      xw[r][p] = in ? *reinterpret_cast<const uint4*>(x + c0) : make_uint4(0, 0, 0, 0);
      if constexpr (kGrad)
        gw[r][p] = in ? *reinterpret_cast<const uint4*>(reinterpret_cast<const T*>(t.g) + row * D + c0) : make_uint4(0, 0, 0, 0);
    }
  }
#pragma unroll
  for (int r = 0; r < kRowsAhead; ++r) {
    const int64_t row = row0 + r * kGroups;
    float ss = 0.f;
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const T* e = reinterpret_cast<const T*>(&xw[r][p]);
#pragma unroll
      for (int i = 0; i < kVec; ++i) ss = fmaf(to_f<T>(e[i]), to_f<T>(e[i]), ss);
    }
#pragma unroll
    for (int o = kLanes / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    const float rn = rsqrtf(ss / float(D) + kEps);
    float m = 0.f;
    if constexpr (kGrad) {
#pragma unroll
      for (int p = 0; p < kPer; ++p) {
        const T* e = reinterpret_cast<const T*>(&xw[r][p]);
        const T* eg = reinterpret_cast<const T*>(&gw[r][p]);
#pragma unroll
        for (int i = 0; i < kVec; ++i) m = fmaf(to_f<T>(eg[i]), to_f<T>(e[i]) * rn, m);
      }
#pragma unroll
      for (int o = kLanes / 2; o > 0; o >>= 1) m += __shfl_xor_sync(0xffffffffu, m, o);
      m /= float(D);
    }
    if (row >= t.rows) continue;
    T* y = reinterpret_cast<T*>(t.y) + row * D;
#pragma unroll
    for (int p = 0; p < kPer; ++p) {
      const int c0 = (p * kLanes + lane) * kVec;
      if (c0 < D) {
        const T* e = reinterpret_cast<const T*>(&xw[r][p]);
        const T* eg = reinterpret_cast<const T*>(&gw[r][p]);
        uint4 w;
        T* out = reinterpret_cast<T*>(&w);
#pragma unroll
        for (int i = 0; i < kVec; ++i) {
          const float yi = to_f<T>(e[i]) * rn;
          out[i] = from_f<T>(kGrad ? rn * (to_f<T>(eg[i]) - yi * m) : yi);
        }
        *reinterpret_cast<uint4*>(y + c0) = w;
      }
    }
  }
}

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

int check(const nb200_qk_norm_tensor& t, int D, int dtype, bool grad, const char* name, NormTensor* out) {
  const int esz = dtype == NB200_F32 ? 4 : 2;
  const int vec = 16 / esz;
  if (t.B < 0 || t.H <= 0 || t.N < 0) { set_error("qk_rms_norm: bad extents of %s", name); return NB200_ERR_INVALID; }
  out->rows = int64_t(t.B) * t.H * t.N;
  if (out->rows == 0) return NB200_OK;
  if (!t.x || !t.y || (grad && !t.g)) { set_error("qk_rms_norm: NULL pointer in %s", name); return NB200_ERR_INVALID; }
  if (!aligned16(t.x) || !aligned16(t.y) || (grad && !aligned16(t.g)) || t.xs[0] % vec || t.xs[1] % vec || t.xs[2] % vec) {
    set_error("qk_rms_norm: %s needs 16-byte aligned rows (pointer and strides)", name);
    return NB200_ERR_ALIGNMENT;
  }
  out->x = t.x; out->g = t.g; out->y = t.y;
  for (int i = 0; i < 3; ++i) out->xs[i] = t.xs[i];
  out->H = t.H; out->N = t.N;
  // (the stride of an axis of one element says nothing)
  out->dense = (t.N == 1 || t.xs[2] == D) && (t.H == 1 || t.xs[1] == int64_t(t.N) * D) &&
               (t.B == 1 || t.xs[0] == int64_t(t.H) * t.N * D);
  return NB200_OK;
}

template <typename T, bool kGrad, int kLanes, int kPer, int kRowsAhead>
int launch_rows(const NormTensor& a, const NormTensor& b, int D, cudaStream_t st) {
  constexpr int64_t kRows = kNormThreads / kLanes * kRowsAhead;     // rows of a CTA
  const int64_t blocks_a = (a.rows + kRows - 1) / kRows, blocks = blocks_a + (b.rows + kRows - 1) / kRows;
  if (blocks > 0x7fffffff) { set_error("qk_rms_norm: too many rows"); return NB200_ERR_UNSUPPORTED; }
  qk_rms_norm_kernel<T, kGrad, kLanes, kPer, kRowsAhead><<<unsigned(blocks), kNormThreads, 0, st>>>(a, b, D, unsigned(blocks_a));
  count_launch();
  return check_launch(kGrad ? "qk_rms_norm_grad_kernel" : "qk_rms_norm_kernel");
}

// Rows ahead: two; one where that leaves fewer than 512 CTAs, which a call that small waits for one by one; four for a large
// fp32 forward, whose rows are not held up by conversions.  us with 1 / 2 / 4: bf16 D 64, 512 rows 2.2 / 2.3 / 3.4, gradient
// 2.3 / 2.7 / 3.9; bf16 D 128, 167 000 rows 19.9 / 17.7 / 21.0, gradient 25.2 / 26.8 / 34.5; f32 D 128, 167 000 rows 38.5 /
// 35.1 / 32.0, gradient 44.9 / 42.9 / 43.4, 32 000 rows 7.2 / 6.3 / 6.7.
template <typename T, bool kGrad, int kLanes, int kPer = 1>
int launch_lanes(const NormTensor& a, const NormTensor& b, int D, cudaStream_t st) {
  const int64_t ctas = (a.rows + b.rows) / (kNormThreads / kLanes);
  if (ctas < 512) return launch_rows<T, kGrad, kLanes, kPer, 1>(a, b, D, st);
  if constexpr (sizeof(T) == 4 && !kGrad) {
    if (ctas >= 8192) return launch_rows<T, kGrad, kLanes, kPer, 4>(a, b, D, st);
  }
  return launch_rows<T, kGrad, kLanes, kPer, 2>(a, b, D, st);
}

template <typename T, bool kGrad>
int launch_typed(const NormTensor& a, const NormTensor& b, int D, cudaStream_t st) {
  const int words = D / (16 / int(sizeof(T)));
  if (words <= 4) return launch_lanes<T, kGrad, 4>(a, b, D, st);
  if (words <= 8) return launch_lanes<T, kGrad, 8>(a, b, D, st);
  if (words <= 16) return launch_lanes<T, kGrad, 16>(a, b, D, st);
  if constexpr (sizeof(T) == 4) {
    if (words > 32) return launch_lanes<T, kGrad, 32, 2>(a, b, D, st);
  }
  return launch_lanes<T, kGrad, 32>(a, b, D, st);
}

template <bool kGrad>
int launch(const nb200_qk_norm_tensor* q, const nb200_qk_norm_tensor* k, int D, int dtype, void* cuda_stream) {
  if (!q || !k) { set_error("qk_rms_norm: NULL tensor description"); return NB200_ERR_INVALID; }
  if (dtype != NB200_F32 && dtype != NB200_BF16 && dtype != NB200_F16) { set_error("qk_rms_norm: bad dtype"); return NB200_ERR_INVALID; }
  const int vec = dtype == NB200_F32 ? 4 : 8;
  if (D <= 0 || D > 256 || D % vec) {
    set_error("qk_rms_norm: head dim %d must be a multiple of %d and at most 256", D, vec);
    return NB200_ERR_UNSUPPORTED;
  }
  NormTensor a{}, b{};
  if (int rc = check(*q, D, dtype, kGrad, "q", &a)) return rc;
  if (int rc = check(*k, D, dtype, kGrad, "k", &b)) return rc;
  const int64_t rows = a.rows + b.rows;
  if (rows == 0) return NB200_OK;
  cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
  prof_call_begin(st);
  if (dtype == NB200_F32) return launch_typed<float, kGrad>(a, b, D, st);
  if (dtype == NB200_BF16) return launch_typed<__nv_bfloat16, kGrad>(a, b, D, st);
  return launch_typed<__half, kGrad>(a, b, D, st);
}

}  // namespace
}  // namespace nb200

extern "C" NB200_API int nb200_qk_rms_norm(const nb200_qk_norm_tensor* q, const nb200_qk_norm_tensor* k, int head_dim,
                                           int dtype, void* cuda_stream) {
  return nb200::launch<false>(q, k, head_dim, dtype, cuda_stream);
}

extern "C" NB200_API int nb200_qk_rms_norm_grad(const nb200_qk_norm_tensor* q, const nb200_qk_norm_tensor* k, int head_dim,
                                                int dtype, void* cuda_stream) {
  return nb200::launch<true>(q, k, head_dim, dtype, cuda_stream);
}
