// The tensor-level calls of ops.py over the C ABI: check, allocate outputs and workspace, pass pointers and the current
// stream, turn status codes into exceptions.  No arithmetic happens here.
//
// In C++ because the passes of a small model are bound by this code: through ctypes a call of the causal path cost 30 to 40 us
// of interpreter time around kernels of 10 to 20 us (checks, device guard, argument conversion, the status words), here a few.
// The autograd nodes of the path are here for the same reason: with Python ones, whose backward waits for the interpreter on the
// engine's thread, a step of RFA.apply took 88.8 us at 8 heads x 512 tokens, with these 75.2 (a layer's training step 769 and 713).
// Errors keep their Python types: AssertionError for shapes, TypeError for dtypes, ValueError for refused arguments,
// RuntimeError for device trouble.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/extension.h>

#include <algorithm>
#include <atomic>
#include <string>
#include <tuple>

#include "../../include/rfa_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

// The calls run without the interpreter lock (see the module's end); what touches Python objects takes it.
[[noreturn]] void raise(PyObject* type, const std::string& msg) {
  py::gil_scoped_acquire lock;
  PyErr_SetString(type, msg.c_str());
  throw py::error_already_set();
}
std::string attr_name(const Tensor& t, const char* attr) {
  py::gil_scoped_acquire lock;
  return py::str(py::cast(t).attr(attr)).cast<std::string>();
}
std::string dtype_name(const Tensor& t) { return attr_name(t, "dtype"); }
std::string shape_name(const Tensor& t) { return attr_name(t, "shape"); }

void require_cuda(const Tensor& t) {
  if (!t.is_cuda())
    raise(PyExc_RuntimeError, "rfa_b200 kernels take CUDA tensors only (there is no CPU path); got a " + t.device().str() + " tensor");
}
void* ptr(const Tensor& t) {
  require_cuda(t);
  if (!t.is_contiguous()) raise(PyExc_ValueError, "rfa_b200: tensor must be contiguous");
  return t.data_ptr();
}
void* ptr(const OptTensor& t) { return t ? ptr(*t) : nullptr; }
float* fptr(const Tensor& t) { return static_cast<float*>(ptr(t)); }
float* fptr(const OptTensor& t) { return static_cast<float*>(ptr(t)); }
const uint8_t* bptr(const OptTensor& t) { return static_cast<const uint8_t*>(ptr(t)); }

int dtype_code(const Tensor& t) {
  if (t.scalar_type() == at::kHalf) return RFA_F16;
  if (t.scalar_type() == at::kFloat) return RFA_F32;
  raise(PyExc_TypeError, "rfa_b200: unsupported dtype " + dtype_name(t) + " (fp16 and fp32 only)");
}
template <class... T>
void require_half(const T&... ts) {
  for (const Tensor* t : {&ts...})
    if (t->scalar_type() != at::kHalf) raise(PyExc_TypeError, "rfa_b200: this kernel is fp16-only, got " + dtype_name(*t));
}
// A kernel launched on x's device must not be handed another device's addresses.
void require_device(const Tensor& x, std::initializer_list<const Tensor*> others) {
  for (const Tensor* t : others)
    if (t->device() != x.device())
      raise(PyExc_RuntimeError, "rfa_b200: expected all tensors on " + x.device().str() + ", got one on " + t->device().str());
}
void require(bool ok, const std::string& msg = "") {
  if (!ok) raise(PyExc_AssertionError, msg);
}
void rank(const Tensor& t, int64_t n) {
  if (t.dim() != n) raise(PyExc_ValueError, "rfa_b200: expected a tensor of " + std::to_string(n) + " dimensions, got " + shape_name(t));
}
int64_t rows_of(const Tensor& x, int64_t H, int64_t d) {
  if (H * d == 0) raise(PyExc_ZeroDivisionError, "rfa_b200: the matrices are empty");
  return x.numel() / (H * d);
}
std::string shapes(const Tensor& a, const Tensor& b) { return "(" + shape_name(a) + ", " + shape_name(b) + ")"; }

int64_t status_error(int status, const char* what) {
  if (status == 0) {      // a bounded wait of an earlier kernel ran out: synchronise and clear, so that it is reported once
    const int code = rfa_status_peek();
    rfa_debug_status();
    raise(PyExc_RuntimeError, std::string("rfa_b200: a bounded wait inside a kernel launched before or by ") + what + " ran out (site code " +
                                  std::to_string(code) + "); results computed since are invalid");
  }
  raise(status < 0 && status != RFA_EDEVICE ? PyExc_ValueError : PyExc_RuntimeError,
        std::string(what) + " failed with status " + std::to_string(status) + ": " + rfa_last_error());
}
void check(int status, const char* what) {
  if (status != 0 || rfa_status_peek() != 0) status_error(status, what);
}

// Makes the tensor's device current for the call and, on first use of a device, switches on the status mirror.
struct Call {
  c10::cuda::CUDAGuard guard;
  rfa_stream_t stream;
  explicit Call(const Tensor& t) : guard((require_cuda(t), t.device())) {
    static std::atomic<bool> watched[64];
    const int i = t.device().index();
    stream = c10::cuda::getCurrentCUDAStream(i).stream();
    if (i >= 64 || !watched[i].load(std::memory_order_acquire)) {
      const int s = rfa_status_mirror_enable();
      if (s != 0) raise(PyExc_RuntimeError, "rfa_status_mirror_enable failed with status " + std::to_string(s) + ": " + rfa_last_error());
      watched[i].store(true, std::memory_order_release);
    }
  }
};

Tensor fresh(at::IntArrayRef shape, const Tensor& like, at::ScalarType dtype) { return at::empty(shape, like.options().dtype(dtype).requires_grad(false)); }
Tensor fresh_zeros(at::IntArrayRef shape, const Tensor& like) { return at::zeros(shape, like.options().dtype(at::kFloat).requires_grad(false)); }
Tensor fresh_like(const Tensor& t) { return fresh(t.sizes(), t, t.scalar_type()); }
Tensor f32(const Tensor& t) { return t.contiguous().to(at::kFloat); }
OptTensor f32(const OptTensor& t) { return t ? OptTensor(f32(*t)) : t; }

Tensor workspace(int64_t T, int64_t BH, int64_t K, int64_t d, const Tensor& like) {
  const int64_t n = static_cast<int64_t>(rfa_causal_workspace_bytes(T, static_cast<int>(BH), static_cast<int>(K), static_cast<int>(d)));
  return fresh({std::max<int64_t>(n, 256)}, like, at::kByte);
}

// A mask as bytes, non-zero = masked.  Booleans are taken as they are.
OptTensor mask_bytes(const OptTensor& mask, int64_t n, const Tensor& like) {
  if (!mask) return mask;
  Tensor m = mask->to(like.device()).reshape({-1});
  if (m.scalar_type() != at::kBool) m = m.ne(0);
  m = m.contiguous();
  require(m.numel() == n, "(" + std::to_string(m.numel()) + ", " + std::to_string(n) + ")");
  return m;
}

// A padding mask [B, T] (any shape that views as one).
OptTensor pad_bytes(const OptTensor& pad, int64_t B, int64_t T, const Tensor& like) {
  return pad ? mask_bytes(pad->reshape({B, T}), B * T, like) : pad;
}

// ---- feature map ---------------------------------------------------------------------------------------------------------
void check_feature_shapes(const Tensor& x, const Tensor& w) {
  rank(w, 3);
  if (!(x.dim() >= 2 && x.size(-2) == w.size(0) && x.size(-1) == w.size(2))) raise(PyExc_AssertionError, shapes(x, w));
}
Tensor phi_like(const Tensor& x, const Tensor& w, at::ScalarType dtype) {
  auto shape = x.sizes().vec();
  shape.back() = 2 * w.size(1);
  return fresh(shape, x, dtype);
}

Tensor feature_map_fwd(Tensor x, Tensor w, double scale, std::optional<at::ScalarType> out_dtype, const OptTensor& row_mask) {
  check_feature_shapes(x, w);
  x = x.contiguous();
  w = f32(w);
  const int64_t H = w.size(0), D = w.size(1), d = w.size(2), rows = rows_of(x, H, d);
  Tensor phi = phi_like(x, w, out_dtype.value_or(x.scalar_type()));
  const OptTensor m = mask_bytes(row_mask, rows, x);
  Call c(x);
  check(rfa_feature_map_fwd_masked(ptr(x), dtype_code(x), fptr(w), bptr(m), ptr(phi), dtype_code(phi), rows, H, d, D, scale, c.stream),
        "rfa_feature_map_fwd");
  return phi;
}

std::tuple<Tensor, OptTensor> feature_map_bwd(Tensor x, Tensor w, Tensor g_phi, double scale, bool need_gw, const OptTensor& row_mask) {
  rank(w, 3);
  x = x.contiguous();
  w = f32(w);
  g_phi = g_phi.contiguous().to(x.scalar_type());
  const int64_t H = w.size(0), D = w.size(1), d = w.size(2), rows = rows_of(x, H, d);
  Tensor g_x = fresh_like(x);
  OptTensor g_w;
  if (need_gw) g_w = fresh_zeros({H, D, d}, x);
  const OptTensor m = mask_bytes(row_mask, rows, x);
  Call c(x);
  check(rfa_feature_map_bwd_masked(ptr(x), dtype_code(x), fptr(w), bptr(m), ptr(g_phi), dtype_code(g_phi), ptr(g_x), dtype_code(g_x), fptr(g_w),
                                   rows, H, d, D, scale, c.stream),
        "rfa_feature_map_bwd");
  return {g_x, g_w};
}

std::tuple<Tensor, Tensor> feature_map_fwd_pair(Tensor a, Tensor b, Tensor w, double scale, const OptTensor& mask_a, const OptTensor& mask_b) {
  if (a.sizes() != b.sizes()) raise(PyExc_AssertionError, shapes(a, b));
  check_feature_shapes(a, w);
  require_half(a, b);
  a = a.contiguous(); b = b.contiguous();
  w = f32(w);
  const int64_t H = w.size(0), D = w.size(1), d = w.size(2), rows = rows_of(a, H, d);
  Tensor pa = phi_like(a, w, at::kHalf), pb = fresh_like(pa);
  const OptTensor ma = mask_bytes(mask_a, rows, a), mb = mask_bytes(mask_b, rows, a);
  Call c(a);
  check(rfa_feature_map_fwd_pair(ptr(a), ptr(b), fptr(w), bptr(ma), bptr(mb), ptr(pa), ptr(pb), rows, H, d, D, scale, c.stream),
        "rfa_feature_map_fwd_pair");
  return {pa, pb};
}

std::tuple<Tensor, Tensor, OptTensor> feature_map_bwd_pair(Tensor a, Tensor b, Tensor w, Tensor g_a, Tensor g_b, double scale, bool need_gw,
                                                           const OptTensor& mask_a, const OptTensor& mask_b) {
  rank(w, 3);
  require_half(a, b);
  a = a.contiguous(); b = b.contiguous();
  w = f32(w);
  g_a = g_a.contiguous().to(at::kHalf); g_b = g_b.contiguous().to(at::kHalf);
  const int64_t H = w.size(0), D = w.size(1), d = w.size(2), rows = rows_of(a, H, d);
  Tensor gxa = fresh_like(a), gxb = fresh_like(b);
  OptTensor g_w;
  if (need_gw) g_w = fresh_zeros({H, D, d}, a);
  const OptTensor ma = mask_bytes(mask_a, rows, a), mb = mask_bytes(mask_b, rows, a);
  Call c(a);
  check(rfa_feature_map_bwd_pair(ptr(a), ptr(b), fptr(w), bptr(ma), bptr(mb), ptr(g_a), ptr(g_b), ptr(gxa), ptr(gxb), fptr(g_w), rows, H, d, D,
                                 scale, c.stream),
        "rfa_feature_map_bwd_pair");
  return {gxa, gxb, g_w};
}

// ---- causal --------------------------------------------------------------------------------------------------------------
std::tuple<Tensor, OptTensor, OptTensor> causal_fwd(Tensor q, Tensor k, Tensor v, const OptTensor& s_in, const OptTensor& z_in, bool return_state) {
  require_half(q, k, v);
  rank(q, 3);
  require(v.dim() >= 2 && k.sizes() == q.sizes() && v.size(0) == q.size(0) && v.size(1) == q.size(1));
  q = q.contiguous(); k = k.contiguous(); v = v.contiguous();
  const int64_t T = q.size(0), BH = q.size(1), K = q.size(2), d = v.size(-1);
  if (s_in && !z_in) raise(PyExc_ValueError, "rfa_b200: a state is given as the pair (s, z), got s alone");
  Tensor out = fresh({T, BH, d}, q, at::kHalf);
  const OptTensor s = f32(s_in), z = f32(z_in);
  if (T == 0) {      // nothing to launch (empty tensors have no address); the state passes through
    if (!return_state) return {out, std::nullopt, std::nullopt};
    if (!s) return {out, fresh_zeros({BH, K, d}, q), fresh_zeros({BH, K}, q)};
    return {out, s->clone(), z->clone()};
  }
  OptTensor s_out, z_out;
  if (return_state) {
    s_out = fresh({BH, K, d}, q, at::kFloat);
    z_out = fresh({BH, K}, q, at::kFloat);
  }
  Tensor ws = workspace(T, BH, K, d, q);
  Call c(q);
  check(rfa_causal_fwd(ptr(q), ptr(k), ptr(v), ptr(out), fptr(s), fptr(z), fptr(s_out), fptr(z_out), ptr(ws), ws.numel(), T, BH, K, d, c.stream),
        "rfa_causal_fwd");
  return {out, s_out, z_out};
}

std::tuple<Tensor, Tensor> causal_fwd_saved(Tensor q, Tensor k, Tensor v, const OptTensor& s_in, const OptTensor& z_in, const OptTensor& kept,
                                            int ws_has) {
  require_half(q, k, v);
  rank(q, 3);
  q = q.contiguous(); k = k.contiguous(); v = v.contiguous();
  const int64_t T = q.size(0), BH = q.size(1), K = q.size(2), d = v.size(-1);
  Tensor out = fresh({T, BH, d}, q, at::kHalf);
  if (T == 0) return {out, fresh({256}, q, at::kByte)};
  Tensor ws = kept ? *kept : workspace(T, BH, K, d, q);
  Call c(q);
  check(rfa_causal_fwd_staged(ptr(q), ptr(k), ptr(v), ptr(out), fptr(s_in), fptr(z_in), nullptr, nullptr, ptr(ws), ws.numel(), T, BH, K, d,
                              kept ? ws_has & RFA_WS_PARTIALS : 0, 1, c.stream),
        "rfa_causal_fwd_staged");
  return {out, ws};
}

std::tuple<Tensor, Tensor, Tensor> causal_bwd_saved(Tensor q, Tensor k, Tensor v, Tensor g, Tensor out, const Tensor& ws, int ws_has,
                                                    const OptTensor& s_in, const OptTensor& z_in) {
  require_half(q, k, v, g, out);
  rank(q, 3);
  q = q.contiguous(); k = k.contiguous(); v = v.contiguous(); g = g.contiguous(); out = out.contiguous();
  const int64_t T = q.size(0), BH = q.size(1), K = q.size(2), d = v.size(-1);
  Tensor gq = fresh_like(q), gk = fresh_like(k), gv = fresh_like(v);
  if (T == 0) return {gq, gk, gv};
  Call c(q);
  check(rfa_causal_bwd_saved(ptr(q), ptr(k), ptr(v), ptr(g), ptr(out), ptr(gq), ptr(gk), ptr(gv), fptr(s_in), fptr(z_in), nullptr, nullptr,
                             ptr(ws), ws.numel(), T, BH, K, d, ws_has, c.stream),
        "rfa_causal_bwd_saved");
  return {gq, gk, gv};
}

std::tuple<Tensor, OptTensor, OptTensor, OptTensor> causal_fwd_fused(Tensor xq, Tensor xk, Tensor v, Tensor w, double scale, const OptTensor& row_mask,
                                                                     const OptTensor& s_in, const OptTensor& z_in, bool return_state, bool save_den) {
  require_half(xq, xk, v);
  rank(xq, 4);
  xq = xq.contiguous(); xk = xk.contiguous(); v = v.contiguous();
  w = f32(w);
  const int64_t T = xq.size(0), B = xq.size(1), H = xq.size(2), d = xq.size(3), BH = B * H, D = w.size(-2);
  Tensor out = fresh({T, BH, d}, xq, at::kHalf);
  const OptTensor m = mask_bytes(row_mask, T * B, xq);
  OptTensor s_out, z_out, ws;
  if (return_state) {
    s_out = fresh({BH, 2 * D, d}, xq, at::kFloat);
    z_out = fresh({BH, 2 * D}, xq, at::kFloat);
  }
  if (save_den) ws = workspace(std::max<int64_t>(T, 1), BH, 2 * D, d, xq);
  Call c(xq);
  check(rfa_causal_fwd_fused(ptr(xq), ptr(xk), ptr(v), fptr(w), bptr(m), scale, ptr(out), fptr(s_in), fptr(z_in), fptr(s_out), fptr(z_out), ptr(ws),
                             ws ? ws->numel() : 0, T, B, H, d, D, save_den ? 1 : 0, c.stream),
        "rfa_causal_fwd_fused");
  return {out, s_out, z_out, ws};
}

// The same without state or workspace, from the layer's own fp16 matrices (and sigma, tau) and its padding mask [B, T].
Tensor causal_fwd_fused_layer(Tensor xq, Tensor xk, Tensor v, Tensor rm, OptTensor sigma, double tau, double scale, const OptTensor& pad) {
  require_half(xq, xk, v, rm);
  rank(xq, 4);
  rank(rm, 3);
  require_device(xq, {&xk, &v, &rm, sigma ? &*sigma : &xq});
  xq = xq.contiguous(); xk = xk.contiguous(); v = v.contiguous(); rm = rm.contiguous();
  const int64_t T = xq.size(0), B = xq.size(1), H = xq.size(2), d = xq.size(3), D = rm.size(1);
  require(xk.sizes() == xq.sizes() && v.sizes() == xq.sizes() && rm.size(0) == H && rm.size(2) == d);
  if (sigma) {
    require_half(*sigma);
    require(sigma->numel() == H * d);
    sigma = sigma->contiguous();
  }
  Tensor out = fresh({T, B * H, d}, xq, at::kHalf);
  const OptTensor m = pad_bytes(pad, B, T, xq);
  Call c(xq);
  check(rfa_causal_fwd_fused_layer(ptr(xq), ptr(xk), ptr(v), ptr(rm), ptr(sigma), static_cast<float>(1.0 / tau), bptr(m), scale, ptr(out), T, B, H, d,
                                   D, c.stream),
        "rfa_causal_fwd_fused_layer");
  return out;
}

// ---- cross ---------------------------------------------------------------------------------------------------------------
std::tuple<Tensor, Tensor> cross_state_fwd(Tensor phi_k, Tensor v, const OptTensor& pad) {
  require_half(phi_k, v);
  rank(phi_k, 4);
  phi_k = phi_k.contiguous(); v = v.contiguous();
  const int64_t T = phi_k.size(0), B = phi_k.size(1), H = phi_k.size(2), K = phi_k.size(3), d = v.size(-1);
  const OptTensor m = pad_bytes(pad, B, T, phi_k);
  Tensor s = fresh({B, H, K, d}, phi_k, at::kFloat), z = fresh({B, H, K}, phi_k, at::kFloat);
  Call c(phi_k);
  check(rfa_cross_state_fwd(ptr(phi_k), ptr(v), bptr(m), fptr(s), fptr(z), T, B, H, K, d, c.stream), "rfa_cross_state_fwd");
  return {s, z};
}

std::tuple<Tensor, Tensor> cross_state_bwd(Tensor phi_k, Tensor v, const OptTensor& pad, Tensor d_s, Tensor d_z) {
  rank(phi_k, 4);
  phi_k = phi_k.contiguous(); v = v.contiguous();
  d_s = f32(d_s); d_z = f32(d_z);
  const int64_t T = phi_k.size(0), B = phi_k.size(1), H = phi_k.size(2), K = phi_k.size(3), d = v.size(-1);
  const OptTensor m = pad_bytes(pad, B, T, phi_k);
  Tensor g_k = fresh_like(phi_k), g_v = fresh_like(v);
  Call c(phi_k);
  check(rfa_cross_state_bwd(ptr(phi_k), ptr(v), bptr(m), fptr(d_s), fptr(d_z), ptr(g_k), ptr(g_v), T, B, H, K, d, c.stream), "rfa_cross_state_bwd");
  return {g_k, g_v};
}

Tensor cross_query_fwd(Tensor phi_q, Tensor s, Tensor z) {
  require_half(phi_q);
  rank(phi_q, 4);
  phi_q = phi_q.contiguous();
  s = f32(s); z = f32(z);
  const int64_t T = phi_q.size(0), B = phi_q.size(1), H = phi_q.size(2), K = phi_q.size(3), d = s.size(-1);
  Tensor out = fresh({T, B, H, d}, phi_q, at::kHalf);
  Call c(phi_q);
  check(rfa_cross_query_fwd(ptr(phi_q), fptr(s), fptr(z), ptr(out), T, B * H, K, d, c.stream), "rfa_cross_query_fwd");
  return out;
}

std::tuple<Tensor, Tensor, Tensor> cross_query_bwd(Tensor phi_q, Tensor s, Tensor z, Tensor g) {
  require_half(phi_q, g);
  rank(phi_q, 4);
  phi_q = phi_q.contiguous(); g = g.contiguous();
  s = f32(s); z = f32(z);
  const int64_t T = phi_q.size(0), B = phi_q.size(1), H = phi_q.size(2), K = phi_q.size(3), d = s.size(-1);
  Tensor g_q = fresh_like(phi_q), d_s = fresh_like(s), d_z = fresh_like(z);
  Call c(phi_q);
  check(rfa_cross_query_bwd(ptr(phi_q), fptr(s), fptr(z), ptr(g), ptr(g_q), fptr(d_s), fptr(d_z), T, B * H, K, d, c.stream), "rfa_cross_query_bwd");
  return {g_q, d_s, d_z};
}

// ---- decode --------------------------------------------------------------------------------------------------------------
Tensor decode_out(const char* what, const Tensor& v, const OptTensor& out) {
  if (!out) return fresh(v.sizes(), v, v.scalar_type());
  if (out->scalar_type() != v.scalar_type() || !out->is_contiguous())
    raise(PyExc_TypeError, std::string(what) + ": out must be contiguous and of v's dtype");
  return *out;
}
void check_state(const char* what, const char* inputs, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& s, const Tensor& z) {
  if (q.scalar_type() != k.scalar_type() || k.scalar_type() != v.scalar_type() || s.scalar_type() != z.scalar_type())
    raise(PyExc_TypeError, std::string(what) + ": " + inputs + ", v must share a dtype and so must s, z (got " + dtype_name(q) + ", " + dtype_name(k) +
                               ", " + dtype_name(v) + "; " + dtype_name(s) + ", " + dtype_name(z) + ")");
  if (!s.is_contiguous() || !z.is_contiguous())
    raise(PyExc_ValueError, std::string(what) + ": state tensors must be contiguous (they are updated in place)");
}

Tensor decode_step(Tensor phi_q, Tensor phi_k, Tensor v, const Tensor& s, const Tensor& z, const OptTensor& out_) {
  rank(phi_q, 3);
  const int64_t B = phi_q.size(0), H = phi_q.size(1), K = phi_q.size(2), d = v.size(-1);
  phi_q = phi_q.contiguous(); phi_k = phi_k.contiguous(); v = v.contiguous();
  check_state("decode_step", "phi_q, phi_k", phi_q, phi_k, v, s, z);
  Tensor out = out_ ? decode_out("decode_step", v, out_) : fresh({B, H, d}, v, v.scalar_type());
  Call c(v);
  check(rfa_decode_step(ptr(phi_q), ptr(phi_k), ptr(v), dtype_code(v), ptr(s), ptr(z), dtype_code(s), ptr(out), B * H, K, d, c.stream),
        "rfa_decode_step");
  return out;
}

Tensor decode_step_fused(Tensor q, Tensor k, Tensor v, const Tensor& w, double scale, const Tensor& s, const Tensor& z, const OptTensor& out_) {
  rank(q, 3);
  const int64_t B = q.size(0), H = q.size(1), d = q.size(2), D = w.size(1);
  q = q.contiguous(); k = k.contiguous(); v = v.contiguous();
  if (w.scalar_type() != at::kFloat || !w.is_contiguous()) raise(PyExc_ValueError, "decode_step_fused: w must be a contiguous fp32 [H,D,d] tensor");
  check_state("decode_step_fused", "q, k", q, k, v, s, z);
  Tensor out = out_ ? decode_out("decode_step_fused", v, out_) : fresh({B, H, d}, v, v.scalar_type());
  Call c(v);
  check(rfa_decode_step_fused(ptr(q), ptr(k), ptr(v), dtype_code(v), fptr(w), scale, ptr(s), ptr(z), dtype_code(s), ptr(out), B * H, H, D, d, c.stream),
        "rfa_decode_step_fused");
  return out;
}

// The largest batch for which one token through a layer of E features is faster by these kernels than by the library GEMMs module by module, at most 128.
// linear_rows.cu reads x once for every 16 or 32 rows of W and W once for every 64 tokens, so that the products lose as E and the batch grow, while
// the launches that are saved cost 60 us of host time.  us a layer with weights from HBM, here / module by module: E = 1024, 128 rows 48 / 101; 2048, 32, 33, 128
// rows 36 / 98, 55 / 98, 96 / 98; 2560, 48, 64 rows 88 / 99, 101 / 98; 4096, 16, 32 rows 53 / 100, 106 / 100; 8192, 8, 16 rows 115 / 133, 253 / 148.  In a CUDA
// graph only the kernels count: 47.0 / 47.4; 36 / 44, 54 / 44, 95 / 79; 86 / 57, 100 / 62; 52 / 63, 100 / 73; 114 / 121, 215 / 135.
int64_t most_rows(int64_t E, bool captured) {
  if (captured) return E <= 1024 ? 128 : E <= 2048 ? 32 : E <= 4096 ? 16 : 8;
  return E <= 2048 ? 128 : std::clamp<int64_t>((300 << 20) / (E * E), 8, 128);
}
bool capturing(const Tensor& x) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  C10_CUDA_CHECK(cudaStreamIsCapturing(c10::cuda::getCurrentCUDAStream(x.device().index()).stream(), &status));
  return status != cudaStreamCaptureStatusNone;
}

// One token [1, B, E] through a whole self-attention layer: the three projections and the step's random matrices in one launch, the
// decoding step, the output projection.  Null where a launch here would not be what the separate tensor calls do (dtype,
// layout, a broadcast shape, a batch that the library GEMMs serve better): nothing has been done then.
OptTensor layer_decode(const Tensor& x, const Tensor& wq, const OptTensor& bq, const Tensor& wk, const OptTensor& bk, const Tensor& wv,
                       const OptTensor& bv, const Tensor& wo, const OptTensor& bo, const Tensor& rm, const OptTensor& sigma, double tau,
                       double scale, const OptTensor& s, const OptTensor& z, int64_t heads) {
  if (!x.is_cuda() || x.dim() != 3 || x.size(0) != 1 || rm.dim() != 3) return std::nullopt;
  const int64_t B = x.size(1), E = x.size(2), H = rm.size(0), D = rm.size(1), d = rm.size(2);
  const auto plain = [&](const Tensor& t, at::IntArrayRef shape, at::ScalarType type) {
    return t.scalar_type() == type && t.sizes() == shape && t.device() == x.device() && t.layout() == at::kStrided && t.is_contiguous() &&
           !t.is_conj() && !t.is_neg() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  };
  const auto bias = [&](const OptTensor& b) { return !b || plain(*b, {E}, at::kHalf); };
  const bool width = D > 0 && D % 8 == 0 && D <= 128 && (d == 8 || d == 16 || d == 32 || d == 64 || d == 128);
  if (B < 1 || B > most_rows(E, false) || (B > most_rows(E, true) && capturing(x)) || !width || H < 1 || H * d != E || (heads && H != heads) || !plain(x, {1, B, E}, at::kHalf)) return std::nullopt;
  for (const Tensor* w : {&wq, &wk, &wv, &wo})
    if (!plain(*w, {E, E}, at::kHalf)) return std::nullopt;
  if (!bias(bq) || !bias(bk) || !bias(bv) || !bias(bo) || !plain(rm, {H, D, d}, at::kHalf)) return std::nullopt;
  if (sigma && !plain(*sigma, {H, 1, d}, at::kHalf)) return std::nullopt;
  if (!s || !z || !plain(*s, {B, H, 2 * D, d}, s->scalar_type()) || !plain(*z, {B, H, 2 * D}, s->scalar_type())) return std::nullopt;
  if (s->scalar_type() != at::kFloat && s->scalar_type() != at::kHalf) return std::nullopt;
  Tensor qkv = fresh({4, B, E}, x, at::kHalf), w_eff = fresh({H, D, d}, x, at::kFloat), y = fresh({1, B, E}, x, at::kHalf);
  char* base = static_cast<char*>(qkv.data_ptr());
  const int64_t step = B * E * 2;                    // 8 | E: every part is aligned
  const void *w3[3] = {wq.data_ptr(), wk.data_ptr(), wv.data_ptr()}, *b3[3] = {ptr(bq), ptr(bk), ptr(bv)};
  void* y3[3] = {base, base + step, base + 2 * step};
  void* attn = base + 3 * step;
  Call c(x);
  check(rfa_linear_rows(x.data_ptr(), w3, b3, y3, 3, B, E, E, rm.data_ptr(), ptr(sigma), static_cast<float>(1.0 / tau), fptr(w_eff), H, D, d, c.stream),
        "rfa_linear_rows");
  check(rfa_decode_step_fused(y3[0], y3[1], y3[2], RFA_F16, fptr(w_eff), scale, s->data_ptr(), z->data_ptr(), dtype_code(*s), attn, B * H, H, D, d,
                              c.stream),
        "rfa_decode_step_fused");
  const void *wo1[1] = {wo.data_ptr()}, *bo1[1] = {ptr(bo)};
  void* yo1[1] = {y.data_ptr()};
  check(rfa_linear_rows(attn, wo1, bo1, yo1, 1, B, E, E, nullptr, nullptr, 1.f, nullptr, 0, 0, 0, c.stream), "rfa_linear_rows");
  return y;
}

// ---- autograd nodes ------------------------------------------------------------------------------------------------------
// The same graph as the Python functions of one name (rfa.py, utils.py, cross_attention.py) make: what is saved, what a
// backward computes, zeros for an output nothing flows back to.  Who may come here is decided there (``_plain.plain_tensors``).
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

struct RFABackward : torch::autograd::Function<RFABackward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v) {
    if (!(q.requires_grad() || k.requires_grad() || v.requires_grad())) return std::get<0>(causal_fwd(q, k, v, std::nullopt, std::nullopt, false));
    auto [out, ws] = causal_fwd_saved(q, k, v, std::nullopt, std::nullopt, std::nullopt, 0);
    ctx->save_for_backward({q, k, v, out, ws});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const variable_list s = ctx->get_saved_variables();
    const int has = s[0].size(0) ? RFA_WS_STATES | RFA_WS_DEN : 0;
    auto [gq, gk, gv] = causal_bwd_saved(s[0], s[1], s[2], g[0].contiguous().to(s[0].scalar_type()), s[3], s[4], has, std::nullopt, std::nullopt);
    return {gq, gk, gv};
  }
};

Tensor grad_of(const OptTensor& g, const Tensor& like) { return g ? g->to(like.scalar_type()) : Tensor(); }
void keep_mask(AutogradContext* ctx, const char* name, const OptTensor& mask) { if (mask) ctx->saved_data[name] = *mask; }
OptTensor kept_mask(AutogradContext* ctx, const char* name) {
  const auto it = ctx->saved_data.find(name);
  return it == ctx->saved_data.end() ? OptTensor() : OptTensor(it->second.toTensor());
}

struct FeatureMapBackward : torch::autograd::Function<FeatureMapBackward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double scale, const OptTensor& mask) {
    ctx->save_for_backward({x, w});
    ctx->saved_data["scale"] = scale;
    keep_mask(ctx, "mask", mask);
    return feature_map_fwd(x, w, scale, std::nullopt, mask);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const variable_list s = ctx->get_saved_variables();
    auto [gx, gw] = feature_map_bwd(s[0], s[1], g[0], ctx->saved_data["scale"].toDouble(), ctx->needs_input_grad(1), kept_mask(ctx, "mask"));
    return {gx, grad_of(gw, s[1]), Tensor(), Tensor()};
  }
};

struct FeatureMapPairBackward : torch::autograd::Function<FeatureMapPairBackward> {
  static variable_list forward(AutogradContext* ctx, const Tensor& a, const Tensor& b, const Tensor& w, double scale, const OptTensor& mask_a,
                               const OptTensor& mask_b) {
    ctx->save_for_backward({a, b, w});
    ctx->saved_data["scale"] = scale;
    keep_mask(ctx, "mask_a", mask_a);
    keep_mask(ctx, "mask_b", mask_b);
    auto [pa, pb] = feature_map_fwd_pair(a, b, w, scale, mask_a, mask_b);
    return {pa, pb};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const variable_list s = ctx->get_saved_variables();
    auto [ga, gb, gw] = feature_map_bwd_pair(s[0], s[1], s[2], g[0], g[1], ctx->saved_data["scale"].toDouble(), ctx->needs_input_grad(2),
                                             kept_mask(ctx, "mask_a"), kept_mask(ctx, "mask_b"));
    return {ga, gb, grad_of(gw, s[2]), Tensor(), Tensor(), Tensor()};
  }
};

struct CrossStateBackward : torch::autograd::Function<CrossStateBackward> {
  static variable_list forward(AutogradContext* ctx, const Tensor& phi_k, const Tensor& v, const OptTensor& pad) {
    ctx->save_for_backward({phi_k, v});
    keep_mask(ctx, "pad", pad);
    auto [s, z] = cross_state_fwd(phi_k, v, pad);
    return {s, z};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const variable_list s = ctx->get_saved_variables();
    auto [gk, gv] = cross_state_bwd(s[0], s[1], kept_mask(ctx, "pad"), g[0], g[1]);
    return {gk, gv, Tensor()};
  }
};

struct CrossQueryBackward : torch::autograd::Function<CrossQueryBackward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& phi_q, const Tensor& s, const Tensor& z) {
    ctx->save_for_backward({phi_q, s, z});
    return cross_query_fwd(phi_q, s, z);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const variable_list s = ctx->get_saved_variables();
    auto [gq, ds, dz] = cross_query_bwd(s[0], s[1], s[2], g[0].contiguous());
    return {gq, ds.to(s[1].scalar_type()), dz.to(s[2].scalar_type())};
  }
};

// y_m = x W_m^T + b_m for one to three matrices, and their gradients: nn.Linear's graph with one launch for the biases, and with the input's
// gradient summed by the products themselves.  y_m takes `shape`, whatever its view of [rows, out]: no view nodes around it.
struct Shape3 { int64_t n[3]; };                       // (an array of them would be taken for several arguments)
struct ProjectBackward : torch::autograd::Function<ProjectBackward> {
  static Tensor rows(const Tensor& t, int64_t width) { return t.reshape({-1, width}); }
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w0, const OptTensor& w1, const OptTensor& w2, const OptTensor& b0,
                               const OptTensor& b1, const OptTensor& b2, Shape3 shape) {
    const OptTensor w[3] = {w0, w1, w2}, b[3] = {b0, b1, b2};
    const Tensor x2 = x.view({-1, w0.size(1)});
    bool need_x = false;                               // what autograd keeps for nn.Linear: x for W's gradient, W for x's
    variable_list y, keep{Tensor()};
    std::vector<int64_t> bias;
    for (int m = 0; m < 3 && w[m]; ++m) {
      y.push_back(at::_unsafe_view(at::linear(x2, *w[m], b[m]), shape.n));
      keep.push_back(x.requires_grad() ? *w[m] : Tensor());
      need_x |= w[m]->requires_grad();
      bias.push_back(b[m].has_value());
    }
    if (need_x) keep[0] = x;
    ctx->save_for_backward(keep);
    ctx->saved_data["bias"] = bias;
    ctx->saved_data["in"] = w0.size(1);
    ctx->saved_data["out"] = w0.size(0);
    ctx->saved_data["x_shape"] = x.sizes().vec();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const variable_list s = ctx->get_saved_variables();
    const auto bias = ctx->saved_data["bias"].toIntVector();
    const int64_t in = ctx->saved_data["in"].toInt(), out = ctx->saved_data["out"].toInt();
    const int n = static_cast<int>(bias.size());
    const bool recorded = at::GradMode::is_enabled();  // a backward that is itself differentiated: tensor expressions throughout
    variable_list r(8), g2(n);
    for (int m = 0; m < n; ++m) g2[m] = rows(g[m], out);
    if (ctx->needs_input_grad(0)) {
      Tensor gx = at::mm(g2[0], s[1]);
      for (int m = 1; m < n; ++m) recorded ? gx = gx + at::mm(g2[m], s[1 + m]) : gx.addmm_(g2[m], s[1 + m]);
      r[0] = at::_unsafe_view(gx, ctx->saved_data["x_shape"].toIntVector());
    }
    for (int m = 0; m < n; ++m)
      if (ctx->needs_input_grad(1 + m)) r[1 + m] = at::mm(g2[m].t(), rows(s[0], in));
    int edge = 1 + n, count = 0;                       // absent biases have no edge
    const void* from[3];
    void* to[3];
    for (int m = 0; m < n; ++m) {
      if (!bias[m] || !ctx->needs_input_grad(edge++)) continue;
      if (!recorded) g2[m] = g2[m].contiguous();
      if (recorded || out % 8 || reinterpret_cast<uintptr_t>(g2[m].data_ptr()) % 16) {
        r[4 + m] = g2[m].sum(0);
        continue;
      }
      r[4 + m] = fresh({out}, g2[m], at::kHalf);
      from[count] = g2[m].data_ptr();
      to[count++] = r[4 + m].data_ptr();
    }
    if (count) {
      Call c(g2[0]);
      check(rfa_column_sums(from, to, count, g2[0].size(0), out, c.stream), "rfa_column_sums");
    }
    return r;
  }
};

// The layer's random matrices in fp32 from fp16 ones and sigma (build_random_matrices); `mask`, if any, is filled from `pad` on the way.
struct MatricesBackward : torch::autograd::Function<MatricesBackward> {
  static Tensor forward(AutogradContext* ctx, const Tensor& rm, const OptTensor& sigma, double tau, const OptTensor& pad, const OptTensor& mask) {
    const int64_t H = rm.size(0), D = rm.size(1), d = rm.size(2);
    Tensor w = fresh({H, D, d}, rm, at::kFloat);
    ctx->save_for_backward({sigma && sigma->requires_grad() ? rm : Tensor(), sigma && rm.requires_grad() ? *sigma : Tensor()});
    ctx->saved_data["tau"] = tau;
    ctx->saved_data["sigma"] = sigma.has_value();
    Call c(rm);
    check(rfa_layer_matrices(ptr(rm), ptr(sigma), static_cast<float>(1.0 / tau), fptr(w), H, D, d, bptr(pad),
                             mask ? static_cast<uint8_t*>(mask->data_ptr()) : nullptr, pad ? pad->size(1) : 0, pad ? pad->size(0) : 0, c.stream),
          "rfa_layer_matrices");
    return w;
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& g) {
    const variable_list s = ctx->get_saved_variables();
    const double tau = ctx->saved_data["tau"].toDouble();
    const bool sigma = ctx->saved_data["sigma"].toBool(), need_rm = ctx->needs_input_grad(0), need_sigma = sigma && ctx->needs_input_grad(1);
    Tensor g_rm, g_sigma;
    if (at::GradMode::is_enabled()) {
      const Tensor gt = g[0] / tau;
      if (need_rm) g_rm = (sigma ? gt * s[1] : gt).to(at::kHalf);
      if (need_sigma) g_sigma = (gt * s[0]).sum(1, true).to(at::kHalf);
    } else {
      const Tensor gw = g[0].contiguous();
      const int64_t H = gw.size(0), D = gw.size(1), d = gw.size(2);
      if (need_rm) g_rm = fresh({H, D, d}, gw, at::kHalf);
      if (need_sigma) g_sigma = fresh({H, 1, d}, gw, at::kHalf);
      Call c(gw);
      check(rfa_layer_matrices_bwd(fptr(gw), need_sigma ? ptr(s[0]) : nullptr, sigma && need_rm ? ptr(s[1]) : nullptr, static_cast<float>(1.0 / tau),
                                   need_sigma ? ptr(g_sigma) : nullptr, need_rm ? ptr(g_rm) : nullptr, H, D, d, c.stream),
            "rfa_layer_matrices_bwd");
    }
    return {g_rm, g_sigma, Tensor(), Tensor(), Tensor()};
  }
};

// A layer's pass with gradients, x [T, B, E] -> y [T, B, E].  Null, with nothing done, where the nodes are not what the separate calls do.
OptTensor layer_train(const Tensor& x, const Tensor& wq, const OptTensor& bq, const Tensor& wk, const OptTensor& bk, const Tensor& wv,
                      const OptTensor& bv, const Tensor& wo, const OptTensor& bo, const Tensor& rm, const OptTensor& sigma, double tau,
                      double scale, const OptTensor& pad) {
  if (!x.is_cuda() || x.dim() != 3 || rm.dim() != 3 || x.numel() == 0) return std::nullopt;
  const int64_t T = x.size(0), B = x.size(1), E = x.size(2), H = rm.size(0), D = rm.size(1), d = rm.size(2);
  const auto plain = [&](const Tensor& t, at::IntArrayRef shape, at::ScalarType type) {
    return t.scalar_type() == type && t.sizes() == shape && t.device() == x.device() && t.layout() == at::kStrided && t.is_contiguous() &&
           !t.is_conj() && !t.is_neg() && reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
  };
  if (H < 1 || D < 8 || D % 8 || D > 128 || d < 8 || d % 8 || d > 128 || H * d != E || H > 65535 || !plain(x, {T, B, E}, at::kHalf)) return std::nullopt;
  for (const Tensor* w : {&wq, &wk, &wv, &wo})
    if (!plain(*w, {E, E}, at::kHalf)) return std::nullopt;
  for (const OptTensor* b : {&bq, &bk, &bv, &bo})
    if (*b && !plain(**b, {E}, at::kHalf)) return std::nullopt;
  if (!plain(rm, {H, D, d}, at::kHalf) || (sigma && !plain(*sigma, {H, 1, d}, at::kHalf))) return std::nullopt;
  if (pad && !(pad->scalar_type() == at::kBool && pad->sizes() == at::IntArrayRef({B, T}) && pad->device() == x.device() && pad->is_contiguous()))
    return std::nullopt;
  OptTensor mask;
  if (pad) mask = fresh({T, B}, x, at::kBool);
  const variable_list p = ProjectBackward::apply(x, wq, OptTensor(wk), OptTensor(wv), bq, bk, bv, Shape3{{T, B * H, d}});
  const Tensor w = MatricesBackward::apply(rm, sigma, tau, pad, mask);
  variable_list phi;
  const Tensor q = p[0].view({T, B, H, d}), k = p[1].view({T, B, H, d});
  if (D == 64 && d == 64) phi = FeatureMapPairBackward::apply(q, k, w, scale, OptTensor(), mask);
  else phi = {FeatureMapBackward::apply(q, w, scale, OptTensor()), FeatureMapBackward::apply(k, w, scale, mask)};
  const Tensor attn = RFABackward::apply(phi[0].view({T, B * H, 2 * D}), phi[1].view({T, B * H, 2 * D}), p[2]);
  return ProjectBackward::apply(attn, wo, OptTensor(), OptTensor(), bo, OptTensor(), OptTensor(), Shape3{{T, B, E}})[0];
}

Tensor rfa_node(const Tensor& q, const Tensor& k, const Tensor& v) { return RFABackward::apply(q, k, v); }
Tensor feature_map_node(const Tensor& x, const Tensor& w, double scale, const OptTensor& mask) { return FeatureMapBackward::apply(x, w, scale, mask); }
std::tuple<Tensor, Tensor> feature_map_pair_node(const Tensor& a, const Tensor& b, const Tensor& w, double scale, const OptTensor& mask_a,
                                                 const OptTensor& mask_b) {
  const variable_list p = FeatureMapPairBackward::apply(a, b, w, scale, mask_a, mask_b);
  return {p[0], p[1]};
}
std::tuple<Tensor, Tensor> cross_state_node(const Tensor& phi_k, const Tensor& v, const OptTensor& pad) {
  const variable_list r = CrossStateBackward::apply(phi_k, v, pad);
  return {r[0], r[1]};
}
Tensor cross_query_node(const Tensor& phi_q, const Tensor& s, const Tensor& z) { return CrossQueryBackward::apply(phi_q, s, z); }

}  // namespace

// Without the interpreter lock, as the foreign calls before them: an allocation, a launch on a full queue or the synchronisation
// of an error report blocks this thread only.
PYBIND11_MODULE(_native, m) {
  const auto def = [&](const char* name, auto* f) { m.def(name, f, py::call_guard<py::gil_scoped_release>()); };
  def("feature_map_fwd", &feature_map_fwd);
  def("feature_map_bwd", &feature_map_bwd);
  def("feature_map_fwd_pair", &feature_map_fwd_pair);
  def("feature_map_bwd_pair", &feature_map_bwd_pair);
  def("causal_fwd", &causal_fwd);
  def("causal_fwd_saved", &causal_fwd_saved);
  def("causal_bwd_saved", &causal_bwd_saved);
  def("causal_fwd_fused", &causal_fwd_fused);
  def("causal_fwd_fused_layer", &causal_fwd_fused_layer);
  def("cross_state_fwd", &cross_state_fwd);
  def("cross_state_bwd", &cross_state_bwd);
  def("cross_query_fwd", &cross_query_fwd);
  def("cross_query_bwd", &cross_query_bwd);
  def("decode_step", &decode_step);
  def("decode_step_fused", &decode_step_fused);
  def("layer_decode", &layer_decode);
  def("layer_train", &layer_train);
  def("rfa_node", &rfa_node);
  def("feature_map_node", &feature_map_node);
  def("feature_map_pair_node", &feature_map_pair_node);
  def("cross_state_node", &cross_state_node);
  def("cross_query_node", &cross_query_node);
}
