// Host side of the tensor-core kernels: coverage gate, workspace plan, tensor
// maps, the mask bit-packing kernel and the launches.
#include <mutex>
#include <stdlib.h>

#include "sdpa_tc_bwd.cuh"
#include "sdpa_tc_common.cuh"
#include "sdpa_tc_fwd.cuh"

namespace nb200 {
namespace tc {

// ---- tensor maps ------------------------------------------------------------
namespace {

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn encode_fn() {
  static EncodeFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeFn>(p);
    else
      cudaGetLastError();
  });
  return fn;
}

}  // namespace

int sm_count() {
  static int cached[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (cached[dev] == 0) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
  }
  return cached[dev];
}

bool tile_map_ok(const void* base, int64_t row_stride, int64_t h_stride, int64_t b_stride, int H, int B,
                 bool allow_broadcast) {
  if (reinterpret_cast<uintptr_t>(base) % 16) return false;
  if (row_stride <= 0 || row_stride % 8) return false;
  // A broadcast (stride 0) head or batch axis is encoded with extent 1, and only the bias loads scale their
  // head / batch coordinate accordingly; q, k, v and dout are addressed by the absolute (b, h), so an expanded
  // view of them is declined here and runs on the CUDA-core family, which indexes by stride.
  if (H > 1 && (h_stride % 8 || h_stride < 0 || (h_stride == 0 && !allow_broadcast))) return false;
  if (B > 1 && (b_stride % 8 || b_stride < 0 || (b_stride == 0 && !allow_broadcast))) return false;
  return true;
}

bool make_tile_map(CUtensorMap* map, const void* base, int rows, int cols, int H, int B, int64_t row_stride,
                   int64_t h_stride, int64_t b_stride, int box_rows, const char** why) {
  EncodeFn fn = encode_fn();
  if (!fn) { if (why) *why = "cuTensorMapEncodeTiled is unavailable"; return false; }
  // broadcast or singleton axes: extent 1 with a harmless natural stride
  const bool h_bc = H <= 1 || h_stride == 0, b_bc = B <= 1 || b_stride == 0;
  const int64_t hs = h_bc ? int64_t(rows) * row_stride : h_stride;
  const int64_t bs = b_bc ? hs * (h_bc ? 1 : H) : b_stride;
  cuuint64_t dims[4] = {cuuint64_t(cols), cuuint64_t(rows), cuuint64_t(h_bc ? 1 : H), cuuint64_t(b_bc ? 1 : B)};
  cuuint64_t strides[3] = {cuuint64_t(row_stride) * 2, cuuint64_t(hs) * 2, cuuint64_t(bs) * 2};
  cuuint32_t box[4] = {cuuint32_t(kSlotCols), cuuint32_t(box_rows), 1, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, const_cast<void*>(base), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) { if (why) *why = "cuTensorMapEncodeTiled rejected the layout"; return false; }
  return true;
}

// ---- mask packing -------------------------------------------------------------
namespace {

// 128 at bit 7 of every non-zero byte, then one dot product gathers four bytes' bits (times 128)
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t v) { return (((v & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | v) & 0x80808080u; }
__device__ __forceinline__ uint32_t keep_bits8(uint32_t lo, uint32_t hi) {
  return __dp4a(nonzero_bytes(hi), 0x80402010u, __dp4a(nonzero_bytes(lo), 0x08040201u, 0u)) >> 7;
}
// keep-bits of kKeys consecutive keys, bit i = key i; keys at or past the `n`th (may be negative) are dropped.
// 16 and 8 keys: one aligned vector load, n either >= kKeys or <= 0; 1: eight single bytes of any stride.  Lanes with
// nothing to read load from `first` (the mask's first element) all the same, so that a row's loads need no branch.
template <int kKeys>
__device__ __forceinline__ uint32_t keep_bits(const uint8_t* p, const uint8_t* first, int64_t st, int n) {
  if (n <= 0) p = first;
  uint32_t bits;
  if constexpr (kKeys == 16) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    bits = keep_bits8(v.x, v.y) | (keep_bits8(v.z, v.w) << 8);
  } else if constexpr (kKeys == 8) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
    bits = keep_bits8(v.x, v.y);
  } else {
    bits = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) bits |= (__ldg(p + (i < n ? i * st : 0)) != 0 && i < n) ? 1u << i : 0u;
  }
  return n > 0 ? bits : 0u;
}
// a 32-key word from the bits of neighbouring lanes (each of them gets it)
template <int kKeys>
__device__ __forceinline__ uint32_t join_bits(uint32_t bits, int lane) {
  constexpr int kLanes = kKeys == 16 ? 2 : 4;   // lanes per word
  uint32_t w = bits << ((32 / kLanes) * (lane & (kLanes - 1)));
  w |= __shfl_xor_sync(0xffffffffu, w, 1);
  if constexpr (kLanes == 4) w |= __shfl_xor_sync(0xffffffffu, w, 2);
  return w;
}

// Mask with a query axis: one CTA packs 64 rows x 256 keys, a warp eight rows, all its loads in flight; a lane takes 16
// keys (rows that are 16-byte aligned and a multiple of 16 long), 8 (the same with 8), or eight single bytes.  The row
// words are kept in shared memory, from which each warp then forms the transposed words of 32 keys: 32 x 32 bits turned
// over in five exchanges between lanes.  Every word of both layouts is written, padding included, so nothing is cleared
// before.  Bound: HBM, the mask once.  32 x 32 tiles of single bytes, or 256 x 256 tiles with a ballot per bit for lengths
// that are multiples of 256, and a memset took (12, 1, 1216, 1216) with the transposed words 58 us, now 7.4; (4, 1, 7424,
// 7424) 108 -> 68, without them 46 -> 47; (3, 1, 1217, 1331) without 15 -> 7; (2, 2, 256, 256) with 7.6 -> 3.1.
// kNarrow: up to 32 keys, one word, 64 x 32 tiles: a lane takes one row's eight keys, where four lanes of a warp would take
// those of eight rows one by one ((1, 8, 3974, 12) with the transposed words 11.2 -> 4.5 us, (4, 16, 1024, 31) 16.8 ->
// 6.5).
template <int kKeys, bool kNarrow>
__global__ void __launch_bounds__(256) mask_pack_kernel(const uint8_t* mask, int64_t sb, int64_t sh, int64_t ss, int64_t st,
                                                        int Hm, int S, int T, uint32_t* rows_out, int words_per_row,
                                                        uint32_t* cols_out, int words_per_col) {
  static_assert(!kNarrow || kKeys != 16, "a load per lane");
  constexpr int kLaneKeys = kKeys == 16 ? 16 : 8, kRowLanes = (kNarrow ? 32 : 256) / kLaneKeys, kLoads = 8 * kRowLanes / 32;
  __shared__ uint32_t sw[64][9];   // [row][key word], padded against bank conflicts
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bm = blockIdx.z / Hm, hm = blockIdx.z - bm * Hm;
  const int key0 = blockIdx.x * 256, row0 = blockIdx.y * 64;
  const int kl = (lane % kRowLanes) * kLaneKeys, key = key0 + kl;
  const int rl0 = warp * 8 + lane / kRowLanes;   // first row of this lane; the next ones 32 / kRowLanes further
  const uint8_t* base = mask + bm * sb + hm * sh + key * st;
  uint32_t bits[kLoads];
  if (row0 + warp * 8 < S) {
#pragma unroll
    for (int i = 0; i < kLoads; ++i) {
      const int row = row0 + rl0 + i * (32 / kRowLanes);
      bits[i] = keep_bits<kKeys>(base + int64_t(row) * ss, mask, st, row < S ? T - key : 0);
    }
  } else {
#pragma unroll
    for (int i = 0; i < kLoads; ++i) bits[i] = 0u;
  }
#pragma unroll
  for (int i = 0; i < kLoads; ++i) {
    const int rl = rl0 + i * (32 / kRowLanes);
    const uint32_t w = join_bits<kKeys>(bits[i], lane);
    if constexpr (kNarrow) {
      // (a row is four words, three of them padding: its four lanes write one each)
      if ((lane & 3) == 0) sw[rl][0] = w;
      if (row0 + rl < S) rows_out[(int64_t(blockIdx.z) * S + row0 + rl) * words_per_row + (lane & 3)] = (lane & 3) ? 0u : w;
    } else if ((kl & 31) == 0) {
      sw[rl][kl >> 5] = w;
      if (row0 + rl < S && (key >> 5) < words_per_row) rows_out[(int64_t(blockIdx.z) * S + row0 + rl) * words_per_row + (key >> 5)] = w;
    }
  }
  if (!cols_out) return;
  __syncthreads();
  if (kNarrow && warp > 0) return;
  uint32_t x[2] = {sw[lane][warp], sw[32 + lane][warp]};   // lane = row
#pragma unroll
  for (int m = 16; m; m >>= 1) {
    const uint32_t low = m == 16 ? 0x0000FFFFu : m == 8 ? 0x00FF00FFu : m == 4 ? 0x0F0F0F0Fu : m == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t y = __shfl_xor_sync(0xffffffffu, x[j], m);
      x[j] = (lane & m) ? (x[j] & ~low) | ((y & ~low) >> m) : (x[j] & low) | ((y & low) << m);
    }
  }
  const int mine = key0 + warp * 32 + lane;   // lane = key now; words_per_col is a multiple of 4
  if (mine < T && (row0 >> 5) < words_per_col)
    *reinterpret_cast<uint2*>(cols_out + (int64_t(blockIdx.z) * T + mine) * words_per_col + (row0 >> 5)) = make_uint2(x[0], x[1]);
}

// Mask without a query axis: one CTA per (batch, head) row packs it and finds 1 + its last kept key.
template <int kKeys>
__global__ void __launch_bounds__(1024) mask_pack_row_kernel(const uint8_t* mask, int64_t sb, int64_t sh, int64_t st, int Hm,
                                                             int T, uint32_t* rows_out, int words_per_row, int* kv_len) {
  static_assert(kKeys != 16, "a warp takes 256 keys");
  __shared__ int last[32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const int bm = blockIdx.x / Hm, hm = blockIdx.x - bm * Hm;
  const uint8_t* base = mask + bm * sb + hm * sh;
  int len = 0;
  for (int word0 = warp * 8; word0 < words_per_row; word0 += warps * 8) {
    const int key = 32 * word0 + 8 * lane, word = key >> 5;
    const uint32_t w = join_bits<kKeys>(keep_bits<kKeys>(base + key * st, mask, st, T - key), lane);
    if (!(lane & 3) && word < words_per_row) rows_out[int64_t(blockIdx.x) * words_per_row + word] = w;
    if (w) len = 32 * word + 32 - __clz(w);   // (words ascend)
  }
  len = __reduce_max_sync(0xffffffffu, len);
  if (lane == 0) last[warp] = len;
  __syncthreads();
  if (warp == 0) {
    len = __reduce_max_sync(0xffffffffu, lane < warps ? last[lane] : 0);
    if (lane == 0) kv_len[blockIdx.x] = len;
  }
}

inline int round_up(int x, int m) { return (x + m - 1) / m * m; }

}  // namespace

// ---- staging ---------------------------------------------------------------------
namespace {

// dst[i0][i1][i2][i3] = src[...] for 16-bit elements, both sides described by element strides.
// Bound: HBM, each element read and written once.  A warp takes one row, or one piece of a row, at a time and a contiguous run
// of them, so an index is divided once per warp and not three times per element in 64 bits; a lane writes aligned words of two
// elements whatever the row's alignment (odd lengths put every other row at an odd element), read as one word where the
// source is aligned like the destination and as two elements otherwise, four words in flight.  One element per thread was
// bound by its divisions: (3, 16, 5158, 5158) 6640 us per copy, now 1070 (2.55 GB each way: 4.8 TB/s); (2, 32, 1223, 6617)
// 2700 -> 580.  Whole rows leave most of the GPU idle where they are few: (1, 8, 4, 65537) 129 us, in pieces 10.
template <bool kSrcUnit, bool kDstUnit>
__global__ void __launch_bounds__(256) copy16_rows_kernel(const uint16_t* __restrict__ src, int64_t s0, int64_t s1, int64_t s2,
                                                          int64_t s3, uint16_t* __restrict__ dst, int64_t d0, int64_t d1,
                                                          int64_t d2, int64_t d3, int64_t e1, int64_t e2, int e3, int piece,
                                                          int pieces, int64_t units, int64_t units_per_warp) {
  const int lane = threadIdx.x & 31;
  const int64_t first = (int64_t(blockIdx.x) * 8 + (threadIdx.x >> 5)) * units_per_warp;
  if (first >= units) return;
  const int64_t last = min(units, first + units_per_warp), row = first / pieces;
  int col = int(first - row * pieces) * piece;
  int64_t i2 = row % e2, i1 = (row / e2) % e1, i0 = row / e2 / e1;
  for (int64_t u = first; u < last; ++u) {
    const uint16_t* sp = src + i0 * s0 + i1 * s1 + i2 * s2 + col * (kSrcUnit ? 1 : s3);
    uint16_t* dp = dst + i0 * d0 + i1 * d1 + i2 * d2 + col * (kDstUnit ? 1 : d3);
    const int n = min(piece, e3 - col);   // >= 1
    col += piece;
    if (col >= e3) {
      col = 0;
      if (++i2 == e2) {
        i2 = 0;
        if (++i1 == e1) { i1 = 0; ++i0; }
      }
    }
    if constexpr (!kDstUnit) {
      for (int w = lane; w < n; w += 32) dp[w * d3] = sp[w * s3];
      continue;
    }
    const int head = int((reinterpret_cast<uintptr_t>(dp) >> 1) & 1);   // elements in front of the first whole word
    const int words = (n - head) >> 1;
    const bool tail = ((n - head) & 1) != 0;
    const uint16_t* se = sp + head * (kSrcUnit ? 1 : s3);
    uint32_t* dw = reinterpret_cast<uint32_t*>(dp + head);
    if (kSrcUnit && (reinterpret_cast<uintptr_t>(se) & 3) == 0) {
      const uint32_t* sw = reinterpret_cast<const uint32_t*>(se);
#pragma unroll 4
      for (int w = lane; w < words; w += 32) dw[w] = __ldg(sw + w);
    } else {
#pragma unroll 4
      for (int w = lane; w < words; w += 32) {
        const uint16_t lo = __ldg(se + (kSrcUnit ? 2 * w : 2 * w * s3)), hi = __ldg(se + (kSrcUnit ? 2 * w + 1 : (2 * w + 1) * s3));
        dw[w] = uint32_t(lo) | (uint32_t(hi) << 16);
      }
    }
    if (lane == 0 && head) dp[0] = sp[0];
    if (lane == 1 && tail) dp[n - 1] = sp[kSrcUnit ? n - 1 : (n - 1) * s3];
  }
}

// The same, an element per thread and turn, for rows that are short or few in all; `I` holds the number of elements.
template <typename I>
__global__ void __launch_bounds__(256) copy16_elements_kernel(const uint16_t* __restrict__ src, int64_t s0, int64_t s1, int64_t s2,
                                                              int64_t s3, uint16_t* __restrict__ dst, int64_t d0, int64_t d1,
                                                              int64_t d2, int64_t d3, I e1, I e2, I e3, I n) {
  for (I i = I(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += I(gridDim.x) * blockDim.x) {
    const I r = i / e3, i3 = i - r * e3, r2 = r / e2, i2 = r - r2 * e2, i0 = r2 / e1, i1 = r2 - i0 * e1;
    dst[i0 * d0 + i1 * d1 + i2 * d2 + i3 * d3] = __ldg(src + i0 * s0 + i1 * s1 + i2 * s2 + i3 * s3);
  }
}

// two (BH, S) fp32 arrays -> (BH, Sp) rows, zero beyond S (one launch for lse and delta)
__global__ void pad_rows_kernel(const float* __restrict__ src0, float* __restrict__ dst0, const float* __restrict__ src1,
                                float* __restrict__ dst1, int S, int Sp, int64_t n) {
  const float* src = blockIdx.y ? src1 : src0;
  float* dst = blockIdx.y ? dst1 : dst0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t bh = i / Sp;
    const int r = int(i - bh * Sp);
    dst[i] = r < S ? src[bh * S + r] : 0.f;
  }
}

inline size_t up256(size_t x) { return (x + 255) / 256 * 256; }
inline bool aligned16(const void* p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

int launch_copy16(const void* src, const int64_t ss[4], void* dst, const int64_t ds[4], const int64_t e[4], cudaStream_t st,
                  const char* what) {
  const int64_t rows = e[0] * e[1] * e[2], n = rows * e[3];
  if (n <= 0) return NB200_OK;
  const uint16_t* s16 = static_cast<const uint16_t*>(src);
  uint16_t* d16 = static_cast<uint16_t*>(dst);
  // By elements below 64 of them a row, where most lanes of a warp per row have nothing to do ((8, 16, 4096, 1) 8 us against
  // 61, 12 keys 27 against 78, 47 keys 82 against 102, 63 level), and up to one element per thread of a full GPU (17680: 6
  // us against 8); from there on by rows ((1, 8, 48, 8191) 12 us against 16, (2, 8, 1000, 1001) 27 against 55).
  if (e[3] < 64 || n <= (int64_t(1) << 19)) {
    const int64_t want = (n + 255) / 256, most = int64_t(sm_count()) * 16;
    const int blocks = int(want < most ? want : most);
    if (n < (int64_t(1) << 31))
      copy16_elements_kernel<uint32_t><<<blocks, 256, 0, st>>>(s16, ss[0], ss[1], ss[2], ss[3], d16, ds[0], ds[1], ds[2], ds[3],
                                                               uint32_t(e[1]), uint32_t(e[2]), uint32_t(e[3]), uint32_t(n));
    else
      copy16_elements_kernel<int64_t><<<blocks, 256, 0, st>>>(s16, ss[0], ss[1], ss[2], ss[3], d16, ds[0], ds[1], ds[2], ds[3],
                                                              e[1], e[2], e[3], n);
    count_launch();
    return check_launch(what);
  }
  // eight CTAs of eight warps per SM; fewer rows than that are cut into pieces of an even length, from 256 elements on
  const int64_t warps = int64_t(sm_count()) * 64;
  const int64_t by_rows = (warps + rows - 1) / rows, by_length = (e[3] + 255) / 256, cut = by_rows < by_length ? by_rows : by_length;
  const int piece = int((e[3] + 2 * cut - 1) / (2 * cut) * 2), pieces = int((e[3] + piece - 1) / piece);
  const int64_t units = rows * pieces, per_warp = (units + warps - 1) / warps;
  const int blocks = int((units + 8 * per_warp - 1) / (8 * per_warp));
  auto kernel = ds[3] != 1 ? copy16_rows_kernel<false, false>
                           : (ss[3] == 1 ? copy16_rows_kernel<true, true> : copy16_rows_kernel<false, true>);
  kernel<<<blocks, 256, 0, st>>>(s16, ss[0], ss[1], ss[2], ss[3], d16, ds[0], ds[1], ds[2], ds[3], e[1], e[2], int(e[3]), piece,
                                 pieces, units, per_warp);
  count_launch();
  return check_launch(what);
}

}  // namespace

Staging plan_staging(const Problem& pr, int pass) {
  Staging sg{};
  sg.Tp = (pr.T + 7) / 8 * 8;
  sg.Sp = (pr.S + kTile / 2 - 1) / (kTile / 2) * (kTile / 2);
  const int64_t full[4] = {pr.B, pr.H, pr.S, pr.T};
  for (int a = 0; a < 4; ++a) sg.extent[a] = (!pr.bias || pr.bs[a] == 0 || full[a] == 1) ? 1 : full[a];
  const bool tile_bias = pr.bias && !(pr.bs[2] == 0 || pr.S == 1);
  if (tile_bias) {
    const bool direct = (pr.T == 1 || pr.bs[3] == 1) && tile_map_ok(pr.bias, pr.bs[2], pr.bs[1], pr.bs[0], pr.H, pr.B, true);
    if (!direct) {
      sg.bias = true;
      sg.bias_bytes = up256(size_t(sg.extent[0] * sg.extent[1] * pr.S) * sg.Tp * 2);
    }
  }
  // a gradient of full extent (no axis of the bias is broadcast) is written by the kernels in 16-byte row segments
  // or by TMA: same layout rules as the bias tiles
  const bool broadcast = (pr.B > 1 && pr.bs[0] == 0) || (pr.H > 1 && pr.bs[1] == 0) || (pr.S > 1 && pr.bs[2] == 0);
  if (pr.bias && pass == NB200_PASS_BWD && pr.want_dbias && !broadcast) {
    const bool direct = pr.T % 8 == 0 && (!pr.dbias || (pr.dbs[3] == 1 && aligned16(pr.dbias) && pr.dbs[0] % 8 == 0 &&
                                                        pr.dbs[1] % 8 == 0 && pr.dbs[2] % 8 == 0));
    if (!direct) {
      sg.dbias = true;
      sg.dbias_bytes = up256(size_t(pr.B) * pr.H * pr.S * sg.Tp * 2);
    }
  }
  if (pass == NB200_PASS_BWD && (pr.S % 4 != 0 || (pr.lse && !aligned16(pr.lse)))) {
    sg.rows = true;
    sg.rows_bytes = up256(sizeof(float) * size_t(pr.B) * pr.H * sg.Sp);
  }
  return sg;
}

Problem staged_view(const Problem& pr, const Staging& sg, void* base) {
  Problem v = pr;
  char* p = base ? static_cast<char*>(base) : reinterpret_cast<char*>(uintptr_t(1) << 20);
  if (sg.bias) {
    v.bias = p;
    // dense over the bias' own extent with rows of Tp keys; broadcast axes keep stride 0
    v.bs[3] = 1;
    v.bs[2] = sg.Tp;
    v.bs[1] = sg.extent[1] == 1 ? 0 : int64_t(pr.S) * sg.Tp;
    v.bs[0] = sg.extent[0] == 1 ? 0 : sg.extent[1] * int64_t(pr.S) * sg.Tp;
    p += sg.bias_bytes;
  }
  if (sg.dbias) {
    v.dbias = p;
    v.dbs[3] = 1;
    v.dbs[2] = sg.Tp;
    v.dbs[1] = int64_t(pr.S) * sg.Tp;
    v.dbs[0] = int64_t(pr.H) * pr.S * sg.Tp;
    p += sg.dbias_bytes;
  }
  if (sg.rows) {
    v.lse = reinterpret_cast<float*>(p);
    v.delta = reinterpret_cast<float*>(p + sg.rows_bytes);
  }
  return v;
}

int stage_in(const Problem& pr, const Problem& v, const Staging& sg, int pass, cudaStream_t stream) {
  if (sg.bias) {
    const int64_t e[4] = {sg.extent[0], sg.extent[1], pr.S, pr.T};
    if (int rc = launch_copy16(pr.bias, pr.bs, const_cast<void*>(v.bias), v.bs, e, stream, "bias_pad_kernel")) return rc;
  }
  if (sg.rows && pass == NB200_PASS_BWD) {
    const int64_t n = int64_t(pr.B) * pr.H * sg.Sp;
    const int blocks = int(((n + 255) / 256) < 148 * 16 ? ((n + 255) / 256) : 148 * 16);
    pad_rows_kernel<<<dim3(blocks, 2), 256, 0, stream>>>(pr.lse, v.lse, pr.delta, v.delta, pr.S, sg.Sp, n);
    count_launch();
    if (int rc = check_launch("pad_rows_kernel")) return rc;
  }
  return NB200_OK;
}

int stage_out(const Problem& pr, const Problem& v, const Staging& sg, cudaStream_t stream) {
  if (!sg.dbias || !pr.dbias) return NB200_OK;
  const int64_t e[4] = {pr.B, pr.H, pr.S, pr.T};
  return launch_copy16(v.dbias, v.dbs, pr.dbias, pr.dbs, e, stream, "dbias_unpad_kernel");
}

bool split_inv_scale(float scale, bool bf16, float* hi, float* lo) {
  *hi = *lo = 0.f;
  if (scale == 0.f || !isfinite(scale) || !isfinite(1.f / scale)) return false;
  const float inv = 1.f / scale;
  const float h = bf16 ? __bfloat162float(__float2bfloat16_rn(inv)) : __half2float(__float2half_rn(inv));
  if (!isfinite(h) || h == 0.f) return false;
  const float rest = inv - h;
  *hi = h;
  *lo = bf16 ? __bfloat162float(__float2bfloat16_rn(rest)) : __half2float(__float2half_rn(rest));
  return true;
}

MaskPackPlan plan_mask_pack(const Problem& pr, bool transposed) {
  MaskPackPlan p{};
  if (!pr.mask) return p;
  const int64_t full[4] = {pr.B, pr.H, pr.S, pr.T};
  for (int a = 0; a < 3; ++a) p.extent[a] = (pr.ms[a] == 0 || full[a] == 1) ? 1 : full[a];
  p.extent[3] = 1;
  p.words_per_row = round_up((pr.T + 31) / 32, 4);
  p.words_per_col = round_up((pr.S + 31) / 32, 4);
  p.rows_bytes = size_t(p.extent[0] * p.extent[1] * p.extent[2]) * p.words_per_row * 4;
  p.rows_bytes = (p.rows_bytes + 255) / 256 * 256;
  p.cols_bytes = transposed ? size_t(p.extent[0] * p.extent[1]) * pr.T * p.words_per_col * 4 : 0;
  p.cols_bytes = (p.cols_bytes + 255) / 256 * 256;
  p.len_bytes = p.extent[2] == 1 ? (size_t(p.extent[0] * p.extent[1]) * 4 + 255) / 256 * 256 : 0;
  return p;
}

bool mask_key_only(const Problem& pr) { return pr.mask && (pr.ms[2] == 0 || pr.S == 1); }

MaskPackPlan mask_plan_for_pass(const Problem& pr, bool backward, size_t* ws_bytes) {
  // a mask without a query axis never needs the transposed copy; a caller-packed mask has the layout it was packed with
  const bool transposed = !mask_key_only(pr) && (pr.mask_packed ? pr.mask_packed == 2 : backward);
  const MaskPackPlan mp = plan_mask_pack(pr, pr.mask && transposed);
  if (ws_bytes) *ws_bytes = pr.mask_packed ? 0 : mp.total();
  return mp;
}

namespace {
// Views into a packed-mask buffer laid out as `plan` says: rows, transposed copy, key lengths.
void mask_views(const Problem& pr, const MaskPackPlan& plan, void* buf, MaskBits* out) {
  uint32_t* rows = static_cast<uint32_t*>(buf);
  uint32_t* cols = plan.cols_bytes ? reinterpret_cast<uint32_t*>(static_cast<char*>(buf) + plan.rows_bytes) : nullptr;
  int* kv_len = plan.len_bytes ? reinterpret_cast<int*>(static_cast<char*>(buf) + plan.rows_bytes + plan.cols_bytes) : nullptr;
  const int Hm = int(plan.extent[1]), Bm = int(plan.extent[0]), Sm = int(plan.extent[2]);
  out->rows = rows;
  out->row_stride = Sm == 1 ? 0 : plan.words_per_row;
  out->h_stride = Hm == 1 ? 0 : int64_t(Sm) * plan.words_per_row;
  out->b_stride = Bm == 1 ? 0 : int64_t(Hm) * Sm * plan.words_per_row;
  out->cols = cols;
  out->tkey_stride = plan.words_per_col;
  out->th_stride = Hm == 1 ? 0 : int64_t(pr.T) * plan.words_per_col;
  out->tb_stride = Bm == 1 ? 0 : int64_t(Hm) * pr.T * plan.words_per_col;
  out->kv_len = kv_len;
  out->len_h_stride = Hm == 1 ? 0 : 1;
  out->len_b_stride = Bm == 1 ? 0 : Hm;
}
}  // namespace

int launch_mask_pack(const Problem& pr, const MaskPackPlan& plan, void* ws, MaskBits* out, cudaStream_t stream) {
  *out = MaskBits{};
  if (!pr.mask) return NB200_OK;
  if (pr.mask_packed) {
    // packed earlier by nb200_mask_pack: nothing to launch
    mask_views(pr, plan, const_cast<uint8_t*>(pr.mask), out);
    return NB200_OK;
  }
  uint32_t* rows = static_cast<uint32_t*>(ws);
  uint32_t* cols = plan.cols_bytes ? reinterpret_cast<uint32_t*>(static_cast<char*>(ws) + plan.rows_bytes) : nullptr;
  const int Bm = int(plan.extent[0]), Hm = int(plan.extent[1]), Sm = int(plan.extent[2]);
  int* kv_len = plan.len_bytes ? reinterpret_cast<int*>(static_cast<char*>(ws) + plan.rows_bytes + plan.cols_bytes) : nullptr;
  // keys per load: rows that start on 16 (8) bytes and hold whole groups of as many
  auto whole = [&](int n) {
    return pr.T % n == 0 && pr.ms[3] == 1 && (Sm == 1 || pr.ms[2] % n == 0) && (Bm == 1 || pr.ms[0] % n == 0) &&
           (Hm == 1 || pr.ms[1] % n == 0) && reinterpret_cast<uintptr_t>(pr.mask) % n == 0;
  };
  const uint8_t* mask = static_cast<const uint8_t*>(pr.mask);
  if (kv_len) {
    auto kernel = whole(8) ? mask_pack_row_kernel<8> : mask_pack_row_kernel<1>;
    const int warps = (plan.words_per_row + 7) / 8;
    kernel<<<Bm * Hm, 32 * (warps < 32 ? warps : 32), 0, stream>>>(mask, pr.ms[0], pr.ms[1], pr.ms[3], Hm, pr.T, rows,
                                                                   plan.words_per_row, kv_len);
  } else {
    auto kernel = pr.T <= 32 ? (whole(8) ? mask_pack_kernel<8, true> : mask_pack_kernel<1, true>)
                  : whole(16) ? mask_pack_kernel<16, false> : (whole(8) ? mask_pack_kernel<8, false> : mask_pack_kernel<1, false>);
    // (with the transposed copy: all of its words, a multiple of 4 per key)
    const dim3 grid((pr.T + 255) / 256, cols ? plan.words_per_col / 2 : (pr.S + 63) / 64, Bm * Hm);
    kernel<<<grid, 256, 0, stream>>>(mask, pr.ms[0], pr.ms[1], pr.ms[2], pr.ms[3], Hm, pr.S, pr.T, rows, plan.words_per_row,
                                     cols, plan.words_per_col);
  }
  count_launch();
  if (int rc = check_launch("mask_pack_kernel")) return rc;
  mask_views(pr, plan, ws, out);
  return NB200_OK;
}

}  // namespace tc

// ---- coverage gate -----------------------------------------------------------
namespace {

struct BiasPlan { int mode; };

bool bias_plan(const Problem& pr, int dtype, int bias_dtype, BiasPlan* bp, const char** why) {
  bp->mode = tc::kBiasNone;
  if (!pr.bias) return true;
  if (bias_dtype != dtype) { *why = "bias dtype differs from q/k/v dtype"; return false; }
  const bool row_bc = pr.bs[2] == 0 || pr.S == 1;
  if (pr.T > 1 && pr.bs[3] != 1) { *why = "bias needs a unit stride over keys"; return false; }
  if (row_bc) {
    // with a positive scale the per-key bias is read element by element (and added by the tensor core); only the
    // path for other scales reads it in 16-byte vectors
    const bool scalar_reads = pr.scale > 0.f && isfinite(1.f / pr.scale);
    if (!scalar_reads && (reinterpret_cast<uintptr_t>(pr.bias) % 16 || pr.bs[0] % 8 || pr.bs[1] % 8 || pr.T % 8)) {
      *why = "per-key bias is not 16-byte aligned";
      return false;
    }
    bp->mode = tc::kBiasKey;
    return true;
  }
  if (!tc::tile_map_ok(pr.bias, pr.bs[2], pr.bs[1], pr.bs[0], pr.H, pr.B, true)) {
    *why = "bias strides / alignment do not fit a TMA descriptor";
    return false;
  }
  bp->mode = tc::kBiasTile;
  return true;
}

}  // namespace

bool tc_supported(const Problem& original, int dtype, int bias_dtype, int pass, const char** why) {
  const char* dummy;
  if (!why) why = &dummy;
  // judged on the problem as the kernels will see it (operands with awkward layouts go through padded copies)
  const tc::Staging sg = tc::plan_staging(original, pass);
  const Problem pr = tc::staged_view(original, sg, nullptr);
  if (dtype != NB200_BF16 && dtype != NB200_F16) { *why = "dtype is not bf16/fp16"; return false; }
  if (pr.D != pr.Dv || (pr.D != 64 && pr.D != 128)) { *why = "head dims must be equal and 64 or 128"; return false; }
  // (the kernels' sums over broadcast axes have one element per key; a bias without a key axis has one per query)
  if (pass == NB200_PASS_BWD && original.bias && original.want_dbias && original.T > 1 && original.bs[3] == 0) {
    *why = "gradient of a bias that is broadcast over the keys";
    return false;
  }
  // Lengths need not fill whole 128-row tiles, nor be multiples of anything: TMA zero-fills rows past the end, the
  // kernels mask keys past T and store only rows below S, and the operands with 16-byte row segments (bias, dbias,
  // lse, delta) are staged through padded copies when the lengths leave those segments ragged.
  if (pr.bh_count > 65535 || int64_t(pr.B) * pr.H > 65535) {
    *why = "more than 65535 (batch, head) pairs (grid limit of the backward and mask-packing launches)";
    return false;
  }
  if (pr.S <= 0 || pr.T <= 0) {
    *why = "query and key lengths must be positive";
    return false;
  }
  if (!tc::tile_map_ok(pr.q, pr.qs[2], pr.qs[1], pr.qs[0], pr.H, pr.B, false) ||
      !tc::tile_map_ok(pr.k, pr.ks[2], pr.ks[1], pr.ks[0], pr.H, pr.B, false) ||
      !tc::tile_map_ok(pr.v, pr.vs[2], pr.vs[1], pr.vs[0], pr.H, pr.B, false)) {
    *why = "q/k/v strides or alignment do not fit a TMA descriptor (expanded views over batch / heads included)";
    return false;
  }
  if (reinterpret_cast<uintptr_t>(pr.out) % 16 || pr.os[0] % 8 || pr.os[1] % 8 || pr.os[2] % 8) {
    *why = "out is not 16-byte aligned";
    return false;
  }
  BiasPlan bp;
  if (!bias_plan(pr, dtype, bias_dtype, &bp, why)) return false;
  if (pass == NB200_PASS_BWD) return tc::bwd_supported(pr, dtype, bias_dtype, why);
  return true;
}

size_t tc_workspace_bytes(const Problem& pr, int dtype, int bias_dtype, int pass) {
  const tc::Staging sg = tc::plan_staging(pr, pass);
  if (pass == NB200_PASS_BWD)
    return (tc::bwd_workspace_bytes(tc::staged_view(pr, sg, nullptr), dtype, bias_dtype) + 255) / 256 * 256 + sg.total();
  size_t bytes = 0;
  tc::mask_plan_for_pass(pr, false, &bytes);
  return (bytes + 255) / 256 * 256 + sg.total();
}

int tc_forward(const Problem& original, int dtype, int bias_dtype, void* ws, size_t ws_bytes, cudaStream_t stream) {
  const char* why = "";
  size_t mask_ws = 0;
  const tc::MaskPackPlan mp = tc::mask_plan_for_pass(original, false, &mask_ws);
  const tc::Staging sg = tc::plan_staging(original, NB200_PASS_FWD);
  const size_t staging_off = (mask_ws + 255) / 256 * 256;
  if (staging_off + sg.total() > ws_bytes || ((mask_ws || sg.total()) && !ws)) {
    set_error("forward needs %zu workspace bytes (mask bits, padded bias)", staging_off + sg.total());
    return NB200_ERR_WORKSPACE;
  }
  const Problem pr = tc::staged_view(original, sg, static_cast<char*>(ws) + staging_off);
  if (int rc = tc::stage_in(original, pr, sg, NB200_PASS_FWD, stream)) return rc;
  BiasPlan bp;
  if (!bias_plan(pr, dtype, bias_dtype, &bp, &why)) { set_error("%s", why); return NB200_ERR_UNSUPPORTED; }
  tc::FwdArgs a{};
  if (int rc = tc::launch_mask_pack(pr, mp, ws, &a.mask, stream)) return rc;
  CUtensorMap tq, tk, tv, tb;
  if (!tc::make_tile_map(&tq, pr.q, pr.S, pr.D, pr.H, pr.B, pr.qs[2], pr.qs[1], pr.qs[0], tc::kTile, &why) ||
      !tc::make_tile_map(&tk, pr.k, pr.T, pr.D, pr.H, pr.B, pr.ks[2], pr.ks[1], pr.ks[0], tc::kTile, &why) ||
      !tc::make_tile_map(&tv, pr.v, pr.T, pr.Dv, pr.H, pr.B, pr.vs[2], pr.vs[1], pr.vs[0], tc::kTile, &why)) {
    set_error("tensor map: %s", why);
    return NB200_ERR_LAUNCH;
  }
  tb = tq;  // placeholder when the bias is not tiled (never dereferenced)
  if (bp.mode == tc::kBiasTile &&
      !tc::make_tile_map(&tb, pr.bias, pr.S, pr.T, pr.H, pr.B, pr.bs[2], pr.bs[1], pr.bs[0], tc::kTile, &why)) {
    set_error("bias tensor map: %s", why);
    return NB200_ERR_LAUNCH;
  }
  a.H = pr.H; a.S = pr.S; a.T = pr.T; a.bh_begin = pr.bh_begin;
  a.causal = pr.causal; a.scale = pr.scale;
  a.bias_mode = bp.mode;
  a.bias_b_mul = (pr.B > 1 && pr.bs[0] != 0) ? 1 : 0;
  a.bias_h_mul = (pr.H > 1 && pr.bs[1] != 0) ? 1 : 0;
  a.bias = pr.bias; a.bias_bs = pr.bs[0]; a.bias_hs = pr.bs[1];
  a.bias_mma = 0;
  if (pr.D == 64 && bp.mode == tc::kBiasTile && pr.scale > 0.f &&
      tc::split_inv_scale(pr.scale, dtype == NB200_BF16, &a.inv_scale_hi, &a.inv_scale_lo))
    a.bias_mma = 1;
  a.key_mma = 0;
  if (bp.mode != tc::kBiasTile && pr.scale > 0.f && isfinite(1.f / pr.scale) &&
      (bp.mode == tc::kBiasKey || a.mask.kv_len != nullptr))
    a.key_mma = 1;
  a.out = pr.out;
  for (int i = 0; i < 3; ++i) a.os[i] = pr.os[i];
  a.out_v8 = reinterpret_cast<uintptr_t>(pr.out) % 32 == 0 && pr.os[0] % 16 == 0 && pr.os[1] % 16 == 0 && pr.os[2] % 16 == 0;
  a.lse = pr.lse;
  a.n_out_peers = pr.n_out_peers;
  for (int i = 0; i < pr.n_out_peers; ++i) {
    a.out_peers[i] = pr.out_peers[i];
    if (reinterpret_cast<uintptr_t>(pr.out_peers[i]) % 32 || pr.os[0] % 16 || pr.os[1] % 16 || pr.os[2] % 16) {
      set_error("fused output all-gather: peer rows must be 32-byte aligned");
      return NB200_ERR_ALIGNMENT;
    }
  }
  a.status = device_status_word();
  if (!a.status) { set_error("device status word is unavailable"); return NB200_ERR_LAUNCH; }
  a.B = pr.B;
  a.bh_count = pr.bh_count;
  a.n_qblocks = (pr.S + 2 * tc::kTile - 1) / (2 * tc::kTile);
  // the whole (batch, head) range: order the items head-major / query block / batch (see decode_item)
  a.head_major = (pr.bh_begin == 0 && pr.bh_count == pr.B * pr.H) ? 1 : 0;
  // causal items differ in length by up to the number of key tiles; with few items per CTA that imbalance costs
  // more than the K / V locality of the head-major order
  if (a.head_major && pr.causal && int64_t(a.n_qblocks) * pr.bh_count <= 16 * int64_t(tc::sm_count())) a.head_major = 2;
  // key padding: items by kept length, longest first (the kernel ranks the batch elements itself)
  if (a.head_major && !pr.causal && a.mask.kv_len && a.mask.len_h_stride == 0 && a.mask.len_b_stride != 0 && pr.B > 1 && pr.B <= tc::kMaxOrder)
    a.head_major = 3;
  return tc::launch_fwd(pr.D, dtype == NB200_BF16, tq, tk, tv, tb, a, stream);
}

size_t tc_mask_pack_bytes(const Problem& pr, bool with_transpose) {
  if (!pr.mask) return 0;
  return tc::plan_mask_pack(pr, with_transpose && !tc::mask_key_only(pr)).total();
}

int tc_mask_pack(const Problem& pr, bool with_transpose, void* packed, size_t packed_bytes, cudaStream_t stream) {
  if (!pr.mask) return NB200_OK;
  if (pr.mask_packed) { set_error("the mask is already packed"); return NB200_ERR_INVALID; }
  const tc::MaskPackPlan mp = tc::plan_mask_pack(pr, with_transpose && !tc::mask_key_only(pr));
  if (!packed || packed_bytes < mp.total()) {
    set_error("the packed mask needs %zu bytes, got %zu", mp.total(), packed ? packed_bytes : size_t(0));
    return NB200_ERR_WORKSPACE;
  }
  if (reinterpret_cast<uintptr_t>(packed) % 256) { set_error("the packed-mask buffer must be 256-byte aligned"); return NB200_ERR_ALIGNMENT; }
  tc::MaskBits unused;
  return tc::launch_mask_pack(pr, mp, packed, &unused, stream);
}

void tc_bwd_dq_region(const Problem& original, int dtype, size_t* offset, size_t* bytes) {
  tc::bwd_dq_region(tc::staged_view(original, tc::plan_staging(original, NB200_PASS_BWD), nullptr), dtype, offset, bytes);
}

int tc_backward(const Problem& original, const TcBwdPrepared& prep, int dtype, int bias_dtype, void* ws, size_t ws_bytes,
                cudaStream_t stream) {
  // padded copies (bias in; lse / delta rows; dbias out) sit behind the kernels' own scratch
  const tc::Staging sg = tc::plan_staging(original, NB200_PASS_BWD);
  const size_t inner = (tc::bwd_workspace_bytes(tc::staged_view(original, sg, nullptr), dtype, bias_dtype) + 255) / 256 * 256;
  if (inner + sg.total() > ws_bytes) {
    set_error("tensor-core backward needs %zu workspace bytes", inner + sg.total());
    return NB200_ERR_WORKSPACE;
  }
  const Problem pr = tc::staged_view(original, sg, static_cast<char*>(ws) + inner);
  if (int rc = tc::stage_in(original, pr, sg, NB200_PASS_BWD, stream)) return rc;
  if (int rc = tc::launch_bwd(pr, prep, dtype, bias_dtype, ws, inner, sg.rows ? sg.Sp : original.S, stream)) return rc;
  return tc::stage_out(original, pr, sg, stream);
}

}  // namespace nb200
