// The differentiable operations of nitrix_b200.nn as C++ autograd functions over the library's C ABI.
//
// A training pass of a small problem is bound by the host.  As Python autograd functions with ctypes calls, a forward and
// backward with 13 us of library calls took 180 us (fp32 attention, 64 x 64; an empty autograd function takes 67), most of
// it filling parameter blocks, allocating through Python and taking the interpreter lock on the engine's device thread;
// here it takes 103, an inference call 16 instead of 38, LayerNorm's pass 81 instead of 131, the scan's 117 instead of 193.
// Nothing is kept between calls: every call asks the library for its plan and its scratch anew (about a microsecond).
//
// The library is the one ctypes has loaded: bind() receives the addresses of its entry points.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/grad_mode.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>

#include "nitrix_b200_attention.h"
#include "nitrix_b200_norm.h"
#include "nitrix_b200_scan.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::tensor_list;
using MaybeTensor = std::optional<Tensor>;

#define NB200_ENTRY_POINTS(X)                                                                                              \
  X(nb200_last_error) X(nb200_sdpa_plan) X(nb200_sdpa_workspace_bytes) X(nb200_sdpa_workspace_least_bytes)                 \
  X(nb200_sdpa_fwd) X(nb200_sdpa_bwd) X(nb200_mask_pack_bytes) X(nb200_mask_pack) X(nb200_qk_rms_norm)                     \
  X(nb200_qk_rms_norm_grad) X(nb200_layer_norm_fwd) X(nb200_layer_norm_bwd) X(nb200_layer_norm_workspace_bytes)            \
  X(nb200_selective_scan_fwd) X(nb200_selective_scan_bwd) X(nb200_selective_scan_checkpoint_bytes)                         \
  X(nb200_selective_scan_workspace_bytes)

struct Library {
#define X(name) decltype(&::name) name = nullptr;
  NB200_ENTRY_POINTS(X)
#undef X
} lib;

void bind(const std::map<std::string, uintptr_t>& addresses) {
#define X(name) lib.name = reinterpret_cast<decltype(&::name)>(addresses.at(#name));
  NB200_ENTRY_POINTS(X)
#undef X
}

std::vector<std::string> entry_points() {
  std::vector<std::string> names;
#define X(name) names.push_back(#name);
  NB200_ENTRY_POINTS(X)
#undef X
  return names;
}

void check(int rc, const char* what) {
  if (rc != NB200_OK) throw std::runtime_error(std::string(what) + " failed (status " + std::to_string(rc) + "): " + lib.nb200_last_error());
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }

Tensor scratch(size_t bytes, const Tensor& like) {
  return at::empty({int64_t(bytes)}, like.options().dtype(at::kByte));
}

int dtype_code(at::ScalarType t) {
  return t == at::kFloat ? NB200_F32 : t == at::kBFloat16 ? NB200_BF16 : t == at::kHalf ? NB200_F16 : -1;
}

bool has_expanded_axis(const Tensor& t) {
  for (int64_t a = 0; a < t.dim(); ++a)
    if (t.stride(a) == 0 && t.size(a) > 1) return true;
  return false;
}

// There are no forward-mode rules.  (torch's own refusal for C++ functions is a RuntimeError, after the kernels have run.)
bool has_tangent(const Tensor& t) { return t._fw_grad(0).defined(); }
bool has_tangent(const MaybeTensor& t) { return t && has_tangent(*t); }
template <typename... T>
void refuse_tangents(const char* what, const T&... operands) {
  TORCH_CHECK_NOT_IMPLEMENTED(!(has_tangent(operands) || ...), what, ": forward-mode differentiation is not implemented");
}

Tensor dense_like(const Tensor& t) { return at::empty(t.sizes(), t.options()); }

void copy_strides(int64_t (&dst)[4], const Tensor& t) {
  for (int a = 0; a < 4; ++a) dst[a] = t.stride(a);
}
// 0 on every axis that t broadcasts over
void copy_strides(int64_t (&dst)[4], const Tensor& t, const int64_t (&full)[4]) {
  for (int a = 0; a < 4; ++a) dst[a] = (t.size(a) == 1 && full[a] != 1) ? 0 : t.stride(a);
}

// ---- attention ---------------------------------------------------------------------------------------------------------
struct Attention {
  Tensor q, k, v;            // (B, H, S, D), (B, H, T, D), (B, H, T, Dv)
  Tensor bias, mask;         // own extent (1 or full) on four axes, or undefined
  Tensor packed;             // the mask's bits as nb200_mask_pack writes them, or undefined
  double scale;
  bool causal;
  int kernel;
  // The mask's strides when it was packed, which are the layout of its bits.  A saved-tensor hook may hand the backward the
  // mask in another layout: an expanded axis, which has no bits of its own, comes back from t.cpu() as a dense one.
  std::vector<int64_t> packed_strides;

  nb200_sdpa_params params() const {
    nb200_sdpa_params p{};
    p.struct_size = sizeof(p);
    p.dtype = dtype_code(q.scalar_type());
    p.B = int32_t(q.size(0)); p.H = int32_t(q.size(1)); p.S = int32_t(q.size(2)); p.D = int32_t(q.size(3));
    p.T = int32_t(k.size(2)); p.Dv = int32_t(v.size(3));
    p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr();
    copy_strides(p.q_stride, q); copy_strides(p.k_stride, k); copy_strides(p.v_stride, v);
    const int64_t full[4] = {p.B, p.H, p.S, p.T};
    if (bias.defined()) {
      p.bias = bias.data_ptr();
      p.bias_dtype = dtype_code(bias.scalar_type());
      copy_strides(p.bias_stride, bias, full);
    }
    if (mask.defined()) {
      p.mask = static_cast<const uint8_t*>(packed.defined() ? packed.data_ptr() : mask.data_ptr());
      if (packed.defined()) std::copy(packed_strides.begin(), packed_strides.end(), p.mask_stride);
      else copy_strides(p.mask_stride, mask, full);
      p.mask_is_bitpacked = packed.defined() ? 2 : 0;
    }
    p.scale = float(scale);
    p.causal = causal;
    p.kernel = kernel;
    p.bh_end = p.B * p.H;
    return p;
  }

  // Kernel family of a pass (no launch; the planner dereferences nothing, q stands in for what does not exist yet)
  int plan(int pass, bool want_dbias) const {
    nb200_sdpa_params p = params();
    p.out = q.data_ptr();
    p.lse = static_cast<float*>(q.data_ptr());
    p.dout = p.dq = p.dk = p.dv = q.data_ptr();
    copy_strides(p.out_stride, q); copy_strides(p.dout_stride, q); copy_strides(p.dq_stride, q);
    copy_strides(p.dk_stride, k); copy_strides(p.dv_stride, v);
    if (want_dbias && pass == NB200_PASS_BWD) {
      p.want_dbias = 1;
      int64_t st = 1;
      for (int a = 3; a >= 0; --a) { p.dbias_stride[a] = st; st *= bias.size(a); }
    }
    int chosen = 0;
    check(lib.nb200_sdpa_plan(&p, pass, &chosen), "nb200_sdpa_plan");
    return chosen;
  }

  // Scratch of a pass; a device without room for all of it gets the least with which the pass runs (the planes of fp32
  // operands take up to 1 GiB that the other kernels do without).
  Tensor workspace(nb200_sdpa_params& p, int pass) const {
    size_t need = 0;
    check(lib.nb200_sdpa_workspace_bytes(&p, pass, &need), "nb200_sdpa_workspace_bytes");
    Tensor ws;
    if (need) {
      try {
        ws = scratch(need, q);
      } catch (const c10::OutOfMemoryError&) {
        size_t least = 0;
        check(lib.nb200_sdpa_workspace_least_bytes(&p, pass, &least), "nb200_sdpa_workspace_least_bytes");
        if (least >= need) throw;
        need = least;
        if (need) ws = scratch(need, q);
      }
    }
    p.workspace = need ? ws.data_ptr() : nullptr;
    p.workspace_bytes = need;
    return ws;
  }

  // The problem as the packing entry points take it, and the bytes its bits take.
  nb200_sdpa_params pack_params(size_t* bytes) const {
    nb200_sdpa_params p = params();
    p.out = q.data_ptr();
    p.lse = static_cast<float*>(q.data_ptr());
    copy_strides(p.out_stride, q);
    p.bias = nullptr;
    p.mask_is_bitpacked = 0;
    check(lib.nb200_mask_pack_bytes(&p, 1, bytes), "nb200_mask_pack_bytes");
    return p;
  }

  void pack_mask() {
    size_t need = 0;
    const nb200_sdpa_params p = pack_params(&need);
    Tensor bits = scratch(need ? need : 1, q);
    check(lib.nb200_mask_pack(&p, 1, bits.data_ptr(), size_t(bits.numel()), stream_of(q)), "nb200_mask_pack");
    packed = bits;
    packed_strides.assign(p.mask_stride, p.mask_stride + 4);
  }

  // Bits of another layout than the one described would be read out of their buffer.
  void check_packed() const {
    if (!packed.defined()) return;
    size_t need = 0;
    pack_params(&need);
    TORCH_CHECK(size_t(packed.numel()) == (need ? need : 1), "scaled_dot_product_attention: the packed mask holds ", packed.numel(),
                " bytes, its layout takes ", need);
  }

  std::pair<Tensor, Tensor> forward() const {
    Tensor out = at::empty({q.size(0), q.size(1), q.size(2), v.size(3)}, q.options());
    Tensor lse = at::empty({q.size(0), q.size(1), q.size(2)}, q.options().dtype(at::kFloat));
    nb200_sdpa_params p = params();
    p.out = out.data_ptr();
    p.lse = lse.data_ptr<float>();
    copy_strides(p.out_stride, out);
    const Tensor ws = workspace(p, NB200_PASS_FWD);   // (same-stream reuse is ordered by the caching allocator)
    check(lib.nb200_sdpa_fwd(&p, stream_of(q)), "nb200_sdpa_fwd");
    return {out, lse};
  }

  tensor_list backward(const Tensor& out, const Tensor& lse, Tensor dout, bool want_dbias) const {
    // (e.g. the cotangent of out.sum() or out.mean(0) arrives as an expanded view)
    if (dout.stride(3) != 1 || has_expanded_axis(dout)) dout = dout.contiguous();
    Tensor dq = dense_like(q), dk = dense_like(k), dv = dense_like(v), dbias;
    nb200_sdpa_params p = params();
    p.out = out.data_ptr();
    p.lse = lse.data_ptr<float>();
    p.dout = dout.data_ptr(); p.dq = dq.data_ptr(); p.dk = dk.data_ptr(); p.dv = dv.data_ptr();
    copy_strides(p.out_stride, out); copy_strides(p.dout_stride, dout); copy_strides(p.dq_stride, dq);
    copy_strides(p.dk_stride, dk); copy_strides(p.dv_stride, dv);
    if (want_dbias) {
      dbias = dense_like(bias);
      p.dbias = dbias.data_ptr();
      copy_strides(p.dbias_stride, dbias);
    }
    check_packed();
    const Tensor ws = workspace(p, NB200_PASS_BWD);
    check(lib.nb200_sdpa_bwd(&p, stream_of(q)), "nb200_sdpa_bwd");
    return {dq, dk, dv, dbias};
  }
};

// Differentiation rule of the fused path (reference src/nitrix/_kernels/cuda/attention.py:661-700): residuals
// (q, k, v, bias, mask, out, lse), cotangents (dq, dk, dv, dbias or none).
struct AttentionRule : torch::autograd::Function<AttentionRule> {
  static tensor_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const MaybeTensor& bias,
                             const MaybeTensor& mask, double scale, bool causal, int64_t kernel, bool tensor_core) {
    Attention a{q, k, v, bias.value_or(Tensor()), mask.value_or(Tensor()), Tensor(), scale, causal, int(kernel), {}};
    const bool want_dbias = bias && bias->requires_grad();
    // (a stride of 0 is a broadcast axis to the library, which has one gradient for it)
    if (want_dbias && has_expanded_axis(a.bias)) a.bias = a.bias.contiguous();
    // On the tensor-core path the mask is bit-packed once, with the key-major copy, and the same bits serve both passes;
    // otherwise each pass reads the byte mask.
    if (tensor_core && mask && a.plan(NB200_PASS_BWD, want_dbias) == NB200_KERNEL_TCGEN05) a.pack_mask();
    auto [out, lse] = a.forward();
    ctx->save_for_backward({q, k, v, a.bias, a.mask, out, lse});
    if (a.packed.defined()) {
      ctx->saved_data["packed"] = a.packed;
      ctx->saved_data["packed_strides"] = a.packed_strides;
    }
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["flags"] = (kernel << 2) | (int64_t(want_dbias) << 1) | int64_t(causal);
    ctx->mark_non_differentiable({lse});
    ctx->set_materialize_grads(false);   // (no zeros for lse's cotangent: an allocation and a launch per backward)
    return {out, lse};
  }
  static tensor_list backward(AutogradContext* ctx, const tensor_list& grads) {
    if (!grads[0].defined()) return tensor_list(9);
    const auto s = ctx->get_saved_variables();
    const int64_t flags = ctx->saved_data["flags"].toInt();
    const auto packed = ctx->saved_data.find("packed");
    const c10::cuda::CUDAGuard guard(s[0].device());
    Attention a{s[0], s[1], s[2], s[3], s[4], Tensor(), ctx->saved_data["scale"].toDouble(), (flags & 1) != 0, int(flags >> 2), {}};
    if (packed != ctx->saved_data.end()) {
      a.packed = packed->second.toTensor();
      a.packed_strides = ctx->saved_data["packed_strides"].toIntVector();
    }
    tensor_list g = a.backward(s[5], s[6], grads[0], (flags & 2) != 0);
    g.resize(9);
    return g;
  }
};

// Operands as the library takes them: four axes, one batch and head count, unit stride on the head dim, nothing expanded
// (the tensor-core kernels address q, k, v by absolute (batch, head)); bias and mask with each axis 1 or full.
bool operands_fit(const Tensor& q, const Tensor& k, const Tensor& v, const MaybeTensor& bias, const MaybeTensor& mask) {
  for (const Tensor* t : {&q, &k, &v})
    if (t->dim() != 4 || !t->is_cuda() || t->device() != q.device() || t->scalar_type() != q.scalar_type() ||
        t->size(0) != q.size(0) || t->size(1) != q.size(1) || t->stride(3) != 1 || has_expanded_axis(*t))
      return false;
  if (dtype_code(q.scalar_type()) < 0 || k.size(2) != v.size(2) || k.size(3) != q.size(3)) return false;
  const int64_t full[4] = {q.size(0), q.size(1), q.size(2), k.size(2)};
  for (const MaybeTensor* t : {&bias, &mask}) {
    if (!*t) continue;
    if ((*t)->dim() != 4 || (*t)->device() != q.device()) return false;
    for (int a = 0; a < 4; ++a)
      if ((*t)->size(a) != 1 && (*t)->size(a) != full[a]) return false;
  }
  if (bias && dtype_code(bias->scalar_type()) < 0) return false;
  return !mask || mask->scalar_type() == at::kBool || mask->scalar_type() == at::kByte;
}

// (out, lse, true); or without tensors: false where the operands have to be brought into shape first, true where the problem
// leaves the tensor-core families and the caller has not allowed that.
using AttentionResult = std::tuple<MaybeTensor, MaybeTensor, bool>;
AttentionResult attention(const Tensor& q, const Tensor& k, const Tensor& v, const MaybeTensor& bias, const MaybeTensor& mask,
                          double scale, bool causal, int64_t kernel, bool any_family) {
  if (!operands_fit(q, k, v, bias, mask)) return {std::nullopt, std::nullopt, false};
  const c10::cuda::CUDAGuard guard(q.device());
  const Attention a{q, k, v, bias.value_or(Tensor()), mask.value_or(Tensor()), Tensor(), scale, causal, int(kernel), {}};
  int family = NB200_KERNEL_SIMT;
  if (kernel == NB200_KERNEL_AUTO) {
    family = a.plan(NB200_PASS_FWD, false);
    if (!any_family && family != NB200_KERNEL_TCGEN05 && family != NB200_KERNEL_MMA_TF32X3) return {std::nullopt, std::nullopt, true};
  }
  if (c10::GradMode::is_enabled() &&
      (q.requires_grad() || k.requires_grad() || v.requires_grad() || (bias && bias->requires_grad()))) {
    refuse_tangents("scaled_dot_product_attention", q, k, v, bias);
    tensor_list r = AttentionRule::apply(q, k, v, bias, mask, scale, causal, kernel, family == NB200_KERNEL_TCGEN05);
    return {r[0], r[1], true};
  }
  auto [out, lse] = a.forward();
  return {out, lse, true};
}

// ---- QK-norm pre-op ------------------------------------------------------------------------------------------------------
// x viewed as (B, H, N, D), leading axes flattened
nb200_qk_norm_tensor norm_desc(const Tensor& x, const Tensor& y, const Tensor& g) {
  const Tensor x4 = x.dim() == 4 ? x : x.reshape({-1, x.size(-3), x.size(-2), x.size(-1)});
  nb200_qk_norm_tensor t{};
  t.x = x4.data_ptr();
  t.y = y.data_ptr();
  t.g = g.defined() ? g.data_ptr() : nullptr;
  for (int a = 0; a < 3; ++a) t.xs[a] = x4.stride(a);
  t.B = int32_t(x4.size(0)); t.H = int32_t(x4.size(1)); t.N = int32_t(x4.size(2));
  return t;
}

struct QkNormRule : torch::autograd::Function<QkNormRule> {
  static tensor_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k) {
    const Tensor qn = dense_like(q), kn = dense_like(k);
    const nb200_qk_norm_tensor dq = norm_desc(q, qn, Tensor()), dk = norm_desc(k, kn, Tensor());
    check(lib.nb200_qk_rms_norm(&dq, &dk, int(q.size(-1)), dtype_code(q.scalar_type()), stream_of(q)), "nb200_qk_rms_norm");
    ctx->save_for_backward({q, k});
    return {qn, kn};
  }
  static tensor_list backward(AutogradContext* ctx, const tensor_list& grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor q = s[0], k = s[1];
    const c10::cuda::CUDAGuard guard(q.device());
    const Tensor gq = grads[0].contiguous().to(q.scalar_type()), gk = grads[1].contiguous().to(k.scalar_type());
    const Tensor dq = dense_like(q), dk = dense_like(k);
    const nb200_qk_norm_tensor tq = norm_desc(q, dq, gq), tk = norm_desc(k, dk, gk);
    check(lib.nb200_qk_rms_norm_grad(&tq, &tk, int(q.size(-1)), dtype_code(q.scalar_type()), stream_of(q)), "nb200_qk_rms_norm_grad");
    return {dq, dk};
  }
};

// The kernel's layout rules: same device, type and head dim, rows of 16-byte words.
bool qk_norm_fits(const Tensor& q, const Tensor& k) {
  if (!q.is_cuda() || !k.is_cuda() || q.device() != k.device() || q.scalar_type() != k.scalar_type() ||
      dtype_code(q.scalar_type()) < 0 || q.dim() < 3 || k.dim() < 3)
    return false;
  const int64_t d = q.size(-1), vec = 16 / int64_t(q.element_size());
  if (k.size(-1) != d || d % vec || d > 256) return false;
  for (const Tensor* z : {&q, &k}) {
    if (z->stride(-1) != 1 || reinterpret_cast<uintptr_t>(z->data_ptr()) % 16 || (z->dim() != 4 && !z->is_contiguous())) return false;
    for (int64_t a = z->dim() - 2; a >= std::max<int64_t>(0, z->dim() - 4); --a)
      if (z->stride(a) % vec) return false;
  }
  return true;
}

std::tuple<Tensor, Tensor> qk_norm(const Tensor& q, const Tensor& k) {
  const c10::cuda::CUDAGuard guard(q.device());
  refuse_tangents("qk_rms_norm", q, k);
  const tensor_list r = QkNormRule::apply(q, k);
  return {r[0], r[1]};
}

// ---- LayerNorm -----------------------------------------------------------------------------------------------------------
nb200_layer_norm_params norm_params(const Tensor& x2, const Tensor& weight, double eps, double out_scale) {
  nb200_layer_norm_params p{};
  p.struct_size = sizeof(p);
  p.rows = x2.size(0);
  p.channels = int32_t(x2.size(1));
  p.dtype = dtype_code(x2.scalar_type());
  p.eps = float(eps);
  p.out_scale = float(out_scale);
  p.x = x2.data_ptr();
  p.weight = weight.defined() ? weight.data_ptr() : nullptr;
  return p;
}

// Saves (x, weight, mean, rstd), returns (dx, dweight, dbias).
struct LayerNormRule : torch::autograd::Function<LayerNormRule> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const MaybeTensor& weight, const MaybeTensor& bias, double eps,
                        double out_scale) {
    const Tensor x2 = x.reshape({-1, x.size(-1)}).contiguous();
    const Tensor w = weight ? weight->to(x.scalar_type()).contiguous() : Tensor();
    const Tensor b = bias ? bias->to(x.scalar_type()).contiguous() : Tensor();
    const Tensor y = dense_like(x2);
    const Tensor mean = at::empty({x2.size(0)}, x.options().dtype(at::kFloat)), rstd = dense_like(mean);
    nb200_layer_norm_params p = norm_params(x2, w, eps, out_scale);
    p.bias = b.defined() ? b.data_ptr() : nullptr;
    p.y = y.data_ptr();
    p.mean = mean.data_ptr<float>();
    p.rstd = rstd.data_ptr<float>();
    check(lib.nb200_layer_norm_fwd(&p, stream_of(x)), "nb200_layer_norm_fwd");
    ctx->save_for_backward({x2, w, mean, rstd});
    ctx->saved_data["eps"] = eps;
    ctx->saved_data["out_scale"] = out_scale;
    ctx->saved_data["shape"] = x.sizes().vec();
    // the types that dweight and dbias leave in; -1: not wanted
    ctx->saved_data["dw"] = weight && weight->requires_grad() ? int64_t(weight->scalar_type()) : int64_t(-1);
    ctx->saved_data["db"] = bias && bias->requires_grad() ? int64_t(bias->scalar_type()) : int64_t(-1);
    return y.reshape(x.sizes());
  }
  static tensor_list backward(AutogradContext* ctx, const tensor_list& grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor x2 = s[0], mean = s[2], rstd = s[3];
    const c10::cuda::CUDAGuard guard(x2.device());
    const Tensor dy2 = grads[0].reshape(x2.sizes()).to(x2.scalar_type()).contiguous();
    const int64_t dw_type = ctx->saved_data["dw"].toInt(), db_type = ctx->saved_data["db"].toInt();
    Tensor dx = dense_like(x2), dw, db, ws;
    nb200_layer_norm_params p = norm_params(x2, s[1], ctx->saved_data["eps"].toDouble(), ctx->saved_data["out_scale"].toDouble());
    p.dy = dy2.data_ptr();
    p.dx = dx.data_ptr();
    p.mean = mean.data_ptr<float>();
    p.rstd = rstd.data_ptr<float>();
    if (dw_type >= 0) dw = at::empty({x2.size(1)}, x2.options());
    if (db_type >= 0) db = at::empty({x2.size(1)}, x2.options());
    if (dw.defined() || db.defined()) {
      size_t need = 0;
      check(lib.nb200_layer_norm_workspace_bytes(&p, &need), "nb200_layer_norm_workspace_bytes");
      ws = scratch(std::max<size_t>(need, 16), x2);
      p.workspace = ws.data_ptr();
      p.workspace_bytes = need;
      p.dweight = dw.defined() ? dw.data_ptr() : nullptr;
      p.dbias = db.defined() ? db.data_ptr() : nullptr;
    }
    check(lib.nb200_layer_norm_bwd(&p, stream_of(x2)), "nb200_layer_norm_bwd");
    if (dw.defined()) dw = dw.to(at::ScalarType(dw_type));
    if (db.defined()) db = db.to(at::ScalarType(db_type));
    return {dx.reshape(ctx->saved_data["shape"].toIntVector()), dw, db, Tensor(), Tensor()};
  }
};

Tensor layer_norm(const Tensor& x, const MaybeTensor& weight, const MaybeTensor& bias, double eps, double out_scale) {
  const c10::cuda::CUDAGuard guard(x.device());
  refuse_tangents("layer_norm", x, weight, bias);
  return LayerNormRule::apply(x, weight, bias, eps, out_scale);
}

// ---- selective scan ------------------------------------------------------------------------------------------------------
nb200_selective_scan_params scan_params(const Tensor& x3, const Tensor& delta3, const Tensor& A, const Tensor& B3, const Tensor& C3,
                                        const Tensor& D) {
  nb200_selective_scan_params p{};
  p.struct_size = sizeof(p);
  p.batch = int32_t(x3.size(0)); p.length = int32_t(x3.size(1)); p.channels = int32_t(x3.size(2)); p.states = int32_t(A.size(1));
  p.dtype = dtype_code(x3.scalar_type());
  p.x = x3.data_ptr(); p.delta = delta3.data_ptr(); p.A = A.data_ptr(); p.B = B3.data_ptr(); p.C = C3.data_ptr();
  p.D = D.defined() ? D.data_ptr() : nullptr;
  return p;
}

// (..., l, n) broadcast over the leading axes of x and dense
Tensor broadcast_rows(const Tensor& t, const Tensor& x) {
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end() - 2);
  shape.push_back(t.size(-2));
  shape.push_back(t.size(-1));
  return t.to(x.scalar_type()).expand(shape).reshape({-1, t.size(-2), t.size(-1)}).contiguous();
}
// gradient of an operand that was broadcast over the leading axes, in that operand's type
Tensor sum_to_operand(const Tensor& g3, at::IntArrayRef lead, at::IntArrayRef shape, int64_t type) {
  std::vector<int64_t> full(lead.begin(), lead.end());
  full.push_back(g3.size(-2));
  full.push_back(g3.size(-1));
  return at::sum_to(g3.reshape(full), shape).to(at::ScalarType(type));
}

// The backward's scratch comes from nitrix_b200.nn.ssm, which decides what a device without room for all of it gets.
PyObject* scan_allocator = nullptr;
// It gets the block with the bytes that are wanted and fills in the workspace.
Tensor scan_workspace(nb200_selective_scan_params& p, const Tensor& like) {
  check(lib.nb200_selective_scan_workspace_bytes(&p, &p.workspace_bytes), "nb200_selective_scan_workspace_bytes");
  py::gil_scoped_acquire gil;
  return py::reinterpret_borrow<py::object>(scan_allocator)(reinterpret_cast<uintptr_t>(&p), int(like.device().index())).cast<Tensor>();
}

// Saves the operands and the forward's checkpoints.
struct ScanRule : torch::autograd::Function<ScanRule> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& delta, const Tensor& A, const Tensor& B,
                        const Tensor& C, const MaybeTensor& D, bool differentiate) {
    const auto dt = x.scalar_type();
    const Tensor x3 = x.reshape({-1, x.size(-2), x.size(-1)}).contiguous();
    const Tensor delta3 = delta.to(dt).reshape(x3.sizes()).contiguous();
    const Tensor B3 = broadcast_rows(B, x), C3 = broadcast_rows(C, x);
    const Tensor A2 = A.to(dt).contiguous(), D1 = D ? D->to(dt).contiguous() : Tensor();
    const Tensor y = dense_like(x3);
    nb200_selective_scan_params p = scan_params(x3, delta3, A2, B3, C3, D1);
    p.y = y.data_ptr();
    Tensor ck;
    if (differentiate) {
      size_t need = 0;
      check(lib.nb200_selective_scan_checkpoint_bytes(&p, &need), "nb200_selective_scan_checkpoint_bytes");
      ck = at::empty({std::max<int64_t>(int64_t(need) / 4, 1)}, x.options().dtype(at::kFloat));
      p.checkpoints = ck.data_ptr<float>();
    }
    check(lib.nb200_selective_scan_fwd(&p, stream_of(x)), "nb200_selective_scan_fwd");
    if (differentiate) {
      ctx->save_for_backward({x3, delta3, A2, B3, C3, D1, ck});
      ctx->saved_data["x"] = x.sizes().vec();
      ctx->saved_data["delta"] = delta.sizes().vec();
      ctx->saved_data["B"] = B.sizes().vec();
      ctx->saved_data["C"] = C.sizes().vec();
      ctx->saved_data["types"] = std::vector<int64_t>{int64_t(delta.scalar_type()), int64_t(A.scalar_type()), int64_t(B.scalar_type()),
                                                      int64_t(C.scalar_type()), D ? int64_t(D->scalar_type()) : int64_t(0)};
    }
    return y.reshape(x.sizes());
  }
  static tensor_list backward(AutogradContext* ctx, const tensor_list& grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor x3 = s[0], D1 = s[5];
    const c10::cuda::CUDAGuard guard(x3.device());
    const Tensor dy3 = grads[0].to(x3.scalar_type()).reshape(x3.sizes()).contiguous();
    const Tensor dx = dense_like(x3), ddelta = dense_like(x3), dA = dense_like(s[2]), dB = dense_like(s[3]), dC = dense_like(s[4]);
    const Tensor dD = D1.defined() ? dense_like(D1) : Tensor();
    nb200_selective_scan_params p = scan_params(x3, s[1], s[2], s[3], s[4], D1);
    p.checkpoints = s[6].data_ptr<float>();
    p.dy = dy3.data_ptr();
    p.dx = dx.data_ptr(); p.ddelta = ddelta.data_ptr(); p.dA = dA.data_ptr(); p.dB = dB.data_ptr(); p.dC = dC.data_ptr();
    p.dD = dD.defined() ? dD.data_ptr() : nullptr;
    const Tensor ws = scan_workspace(p, x3);
    check(lib.nb200_selective_scan_bwd(&p, stream_of(x3)), "nb200_selective_scan_bwd");
    const auto xs = ctx->saved_data["x"].toIntVector(), types = ctx->saved_data["types"].toIntVector();
    const at::IntArrayRef lead(xs.data(), xs.size() - 2);
    return {dx.reshape(xs),
            ddelta.reshape(ctx->saved_data["delta"].toIntVector()).to(at::ScalarType(types[0])),
            dA.to(at::ScalarType(types[1])),
            sum_to_operand(dB, lead, ctx->saved_data["B"].toIntVector(), types[2]),
            sum_to_operand(dC, lead, ctx->saved_data["C"].toIntVector(), types[3]),
            dD.defined() ? dD.to(at::ScalarType(types[4])) : Tensor(),
            Tensor()};
  }
};

Tensor selective_scan(const Tensor& x, const Tensor& delta, const Tensor& A, const Tensor& B, const Tensor& C, const MaybeTensor& D) {
  const c10::cuda::CUDAGuard guard(x.device());
  refuse_tangents("selective_scan", x, delta, A, B, C, D);
  bool differentiate = false;
  if (c10::GradMode::is_enabled()) {
    for (const Tensor* t : {&x, &delta, &A, &B, &C}) differentiate = differentiate || t->requires_grad();
    differentiate = differentiate || (D && D->requires_grad());
  }
  return ScanRule::apply(x, delta, A, B, C, D, differentiate);
}

}  // namespace

PYBIND11_MODULE(_torch_ops, m) {
  m.def("entry_points", &entry_points);
  m.def("bind", &bind);
  // (torch's wrapper: its exception types, and no interpreter lock while the library is called)
  m.def("attention", torch::wrap_pybind_function_no_gil(attention));
  m.def("qk_norm_fits", torch::wrap_pybind_function(qk_norm_fits));
  m.def("qk_norm", torch::wrap_pybind_function_no_gil(qk_norm));
  m.def("layer_norm", torch::wrap_pybind_function_no_gil(layer_norm));
  m.def("set_scan_allocator", [](py::object allocator) { scan_allocator = allocator.release().ptr(); });   // (for good)
  m.def("selective_scan", torch::wrap_pybind_function_no_gil(selective_scan));
}
