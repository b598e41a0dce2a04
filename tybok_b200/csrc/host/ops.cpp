// Single operations and the two feed-forward hooks of the _native extension.
#include "native.h"

#include <mutex>

namespace tbn {

void raise_status(int rc, const char* what) {
  py::gil_scoped_acquire gil;
  const std::string msg = std::string(what) + " failed with status " + std::to_string(rc) + ": " + tybok_last_error();
  const py::object err = py::module_::import("tybok_b200._lib").attr("TybokError");
  PyErr_SetString(err.ptr(), msg.c_str());
  throw py::error_already_set();
}

void require_cuda(const Tensor& t, const char* what) {
  if (t.is_cuda()) return;
  py::gil_scoped_acquire gil;
  PyErr_SetString(PyExc_NotImplementedError,
                  (std::string("tybok_b200::") + what + " runs on CUDA tensors only: there is no CPU implementation").c_str());
  throw py::error_already_set();
}

static Tensor g_status[64];

static Tensor& status_tensor(int device) {
  static std::mutex mu;
  std::lock_guard<std::mutex> lock(mu);
  Tensor& t = g_status[device & 63];
  if (!t.defined()) t = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, static_cast<c10::DeviceIndex>(device)));
  return t;
}

int* status_ptr(int device) { return static_cast<int*>(status_tensor(device).data_ptr()); }

Tensor rows_of(const Tensor& x) {
  Tensor r = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  return r.stride(-1) == 1 ? r : r.contiguous();
}

Tensor vector_rows_of(const Tensor& x) {
  Tensor r = rows_of(x);
  if (!is_bf16(r)) r = r.to(at::kBFloat16);
  const bool fits = r.stride(0) % 8 == 0 && r.stride(0) >= r.size(1) && !(reinterpret_cast<uintptr_t>(r.data_ptr()) & 15);
  return fits ? r : r.clone(at::MemoryFormat::Contiguous);
}

static void check_w8(const Tensor& w, const char* what) {
  if ((w.scalar_type() != at::kFloat8_e4m3fn && w.scalar_type() != at::kByte) || !w.is_contiguous() || w.dim() != 2)
    type_error(std::string(what) + ": weight must be a contiguous e4m3 (or raw uint8) [N, K] tensor");
}
static void check_scale(const Tensor& s, int64_t rows, const char* what) {
  if (!is_vector(s, at::kFloat, rows))
    type_error(std::string(what) + ": scale must be contiguous fp32 [" + std::to_string(rows) + "] (one per weight row)");
}

W8 w8_of(const py::handle& t, const char* what) {
  const py::tuple u = py::reinterpret_borrow<py::tuple>(t);
  W8 r;
  r.w = u[0].cast<Tensor>();
  r.s = u[1].cast<Tensor>();
  check_w8(r.w, what);
  check_scale(r.s, r.w.size(0), what);
  if (u.size() > 2 && !u[2].is_none()) {
    r.b = u[2].cast<Tensor>();
    if (!is_vector(*r.b, at::kBFloat16, r.w.size(0))) type_error(std::string(what) + ": bias must be contiguous bf16 [N]");
  }
  same_device(r.w.device(), what, {&r.s, opt(r.b)});
  r.n = static_cast<int>(r.w.size(0));
  r.k = static_cast<int>(r.w.size(1));
  return r;
}

// epilogue(x @ (w8 * scale).T + bias) for bf16 x: activation planes, then the GEMM.
static Tensor w8a16_linear(const Tensor& x, const Tensor& w8, const Tensor& scale, const OptTensor& bias, int epilogue,
                           const OptTensor& residual, const OptTensor& gate, int rows_per_gate, int token_tile, int splits, int shift) {
  if (!is_bf16(x)) type_error("split3: x must be bf16");
  check_w8(w8, "w8x3_linear");
  const int64_t n = w8.size(0), k = w8.size(1);
  check_scale(scale, n, "w8x3_linear");
  const Tensor x2 = rows_of(x);
  const int64_t m = x2.size(0);
  if (x2.size(1) != k) value_error("w8x3_linear: planes have K=" + std::to_string(x2.size(1)) + ", weight has K=" + std::to_string(k));
  if (bias && !is_vector(*bias, at::kBFloat16, n)) type_error("w8x3_linear: bias must be contiguous bf16 [N]");
  Tensor res;
  if (residual) {
    res = rows_of(*residual);
    if (res.size(0) != m || res.size(1) != n || !is_bf16(res)) value_error("w8x3_linear: residual must be bf16 [M, N]");
  }
  int gate_bf16 = 0;
  int64_t ldgate = 0;
  if (gate) {
    if ((gate->scalar_type() != at::kFloat && !is_bf16(*gate)) || gate->stride(-1) != 1 || gate->size(-1) != n)
      type_error("w8x3_linear: gate must be fp32 or bf16 [groups, N] with unit inner stride");
    gate_bf16 = is_bf16(*gate);
    ldgate = gate->dim() > 1 ? gate->stride(-2) : n;
    if (epilogue == TYBOK_EPI_RESIDUAL && rows_per_gate > 0 && (gate->dim() > 1 ? gate->size(-2) : 1) * rows_per_gate < m)
      value_error("w8x3_linear: fewer gate rows than groups of rows_per_gate tokens");
  }
  same_device(x.device(), "w8x3_linear", {&w8, &scale, opt(bias), opt(residual), opt(gate)});
  require_cuda(x, "split3");
  const c10::cuda::CUDAGuard guard(x.device());
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = n;
  Tensor y = at::empty(shape, x.options());
  void* st = stream_of(x);
  if (m <= 16 && shift == TYBOK_DEFAULT_X_SHIFT && token_tile <= 0 && splits <= 0) {
    const int rc = tybok_w8a16_linear_direct(ptr(x2), ptr(w8), f32(scale), ptr(bias), ptr(y), m, n, k, x2.stride(0), n, epilogue,
                                             residual ? ptr(res) : nullptr, residual ? res.stride(0) : 0, ptr(gate), ldgate, rows_per_gate,
                                             gate_bf16, status_ptr(x.get_device()), st);
    if (rc != TYBOK_ERR_WORKSPACE) {
      check(rc, "tybok_w8a16_linear");
      return y;
    }
  }
  const Tensor planes = at::empty({3 * m * k}, x.options().dtype(at::kByte));
  check(tybok_split3(ptr(x2), x2.stride(0), ptr(planes), m, k, shift, st), "tybok_split3");
  check(tybok_w8x3_linear(ptr(planes), shift, ptr(w8), f32(scale), ptr(bias), ptr(y), n, nullptr, 0, m, n, k, epilogue,
                          residual ? ptr(res) : nullptr, residual ? res.stride(0) : 0, ptr(gate), ldgate, rows_per_gate, gate_bf16,
                          token_tile, splits, status_ptr(x.get_device()), st),
        "tybok_w8x3_linear");
  return y;
}

static std::tuple<Tensor, Tensor> attention(const Tensor& q, const Tensor& kc, const Tensor& vc, const OptTensor& valid, int tokens,
                                            int keys, double scale, bool out_bf16, bool out_planes, int out_shift) {
  if (kc.dim() != 4) value_error("attention: caches must be [B, G, Lcap, D]");
  const int64_t b = kc.size(0), g = kc.size(1), lcap = kc.size(2), d = kc.size(3);
  if (!is_bf16(kc) || !is_bf16(vc) || !kc.is_contiguous() || !vc.is_contiguous()) type_error("attention: caches must be contiguous bf16");
  if (vc.sizes() != kc.sizes()) value_error("attention: key and value caches differ in shape");
  if (!is_bf16(q) || q.dim() != 2 || !q.is_contiguous() || q.size(0) != b * tokens) type_error("attention: q must be contiguous bf16 [B*L, H*D]");
  const int64_t hd = q.size(1), h = hd / d;
  if (hd != h * d) value_error("attention: the rows of q must hold whole heads");
  if (valid && (valid->scalar_type() != at::kByte || valid->dim() != 2 || valid->size(0) != b || valid->size(1) != keys || !valid->is_contiguous()))
    type_error("attention: key_valid must be contiguous uint8 [B, Lk]");
  if (!out_bf16 && !out_planes) value_error("at least one of out_bf16 / out_planes must be set");
  same_device(q.device(), "attention", {&kc, &vc, opt(valid)});
  require_cuda(q, "attention");
  const c10::cuda::CUDAGuard guard(q.device());
  Tensor y = out_bf16 ? at::empty({b * tokens, h * d}, q.options()) : at::empty({0}, q.options());
  const auto bytes = q.options().dtype(at::kByte);
  Tensor yp = out_planes ? at::empty({3, b * tokens, h * d}, bytes) : at::empty({0}, bytes);
  const size_t need = tybok_attention_workspace_needed(b, tokens, h, g, d, keys);
  Tensor ws;
  if (need) ws = at::empty({static_cast<int64_t>(need)}, bytes);
  check(tybok_attention(ptr(q), ptr(kc), ptr(vc), ptr(valid), out_bf16 ? ptr(y) : nullptr, out_planes ? ptr(yp) : nullptr, out_shift, b,
                        tokens, h, g, d, keys, lcap, scale, need ? ptr(ws) : nullptr, need, status_ptr(q.get_device()), stream_of(q)),
        "tybok_attention");
  return {y, yp};
}

// down(gelu_tanh(gate(x)) * up(x)); gate_up is the interleaved matrix, or gate alone with `up` beside it.
class Mlp {
 public:
  Mlp(const py::tuple& gate_up, const py::object& up, const py::tuple& down) : gu_(w8_of(gate_up, "mlp")), down_(w8_of(down, "mlp")) {
    packed_ = up.is_none();
    if (!packed_) up_ = w8_of(up, "mlp");
    inner_ = packed_ ? gu_.n / 2 : gu_.n;
    if (down_.k != inner_) value_error("mlp: down projection and intermediate width disagree");
    if (!packed_ && !up_.is(gu_.n, gu_.k)) value_error("mlp: gate and up weights differ in shape");
    same_device(gu_.device(), "mlp", {packed_ ? nullptr : &up_.w, &down_.w});
  }
  Tensor forward(const Tensor& x) const {
    same_device(gu_.device(), "mlp", {&x});
    require_cuda(x, "mlp");
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor x2 = vector_rows_of(x);
    if (x2.size(1) != gu_.k) value_error("mlp: input width differs from the weights'");
    const int m = x2.size(0), k = gu_.k, i = inner_;
    std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
    shape.back() = down_.n;
    Tensor y = at::empty(shape, x2.options());
    Arena a;
    const size_t xp = a.add(size_t(3) * m * k), hp = a.add(size_t(3) * m * i);
    a.allocate(x2);
    void* st = stream_of(x);
    int* status = status_ptr(x.get_device());
    bool direct = false;  // few tokens: the gate/up GEMM makes its own planes
    if (m <= 16 && packed_) {
      const int rc = tybok_w8a16_geglu_packed_direct(ptr(x2), x2.stride(0), gu_.wp(), gu_.sp(), a.at(hp), SHIFT_FFN, m, i, k, status, st);
      direct = rc != TYBOK_ERR_WORKSPACE;
      if (direct) check(rc, "tybok_w8a16_geglu_packed");
    }
    if (!direct) {
      check(tybok_split3(ptr(x2), x2.stride(0), a.at(xp), m, k, SHIFT_NORMED, st), "tybok_split3");
      if (packed_)
        check(tybok_w8x3_geglu_packed(a.at(xp), SHIFT_NORMED, gu_.wp(), gu_.sp(), nullptr, i, a.at(hp), SHIFT_FFN, m, i, k, 0, 0, status, st),
              "tybok_w8x3_geglu_packed");
      else
        check(tybok_w8x3_geglu(a.at(xp), SHIFT_NORMED, gu_.wp(), gu_.sp(), up_.wp(), up_.sp(), nullptr, i, a.at(hp), SHIFT_FFN, m, i, k, 0, 0,
                               status, st),
              "tybok_w8x3_geglu");
    }
    check(tybok_w8x3_linear(a.at(hp), SHIFT_FFN, down_.wp(), down_.sp(), nullptr, ptr(y), down_.n, nullptr, 0, m, down_.n, i, TYBOK_EPI_NONE,
                            nullptr, 0, nullptr, 0, 1, 0, 0, 0, status, st),
          "tybok_w8x3_linear");
    return y.scalar_type() == x.scalar_type() ? y : y.to(x.scalar_type());
  }

 private:
  W8 gu_, up_, down_;
  bool packed_ = true;
  int inner_ = 0;
};

// x + gate * down(gelu_tanh(up(modulate(LayerNorm(x), shift, scale)))) of [B, S, H] rows, one modulation row per batch
// element: one chain for the whole batch.
class FfnTail {
 public:
  FfnTail(const py::tuple& up, const py::tuple& down, double eps) : up_(w8_of(up, "ffn_tail")), down_(w8_of(down, "ffn_tail")), eps_(eps) {
    if (!down_.is(up_.k, up_.n)) value_error("ffn_tail: the down weight is not the up weight's shape transposed");
    same_device(up_.device(), "ffn_tail", {&down_.w});
  }
  Tensor forward(const Tensor& x, const Tensor& shift, const Tensor& scale, const Tensor& gate) const {
    same_device(up_.device(), "ffn_tail", {&x, &shift, &scale, &gate});
    require_cuda(x, "ffn_tail");
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t h = x.size(-1), batch = x.dim() == 3 ? x.size(0) : 1;
    if (h != up_.k) value_error("ffn_tail: input width differs from the weights'");
    const Tensor x2 = vector_rows_of(x);
    const int m = x2.size(0), f = up_.n, per = batch ? m / batch : 1;
    Tensor sh = mod_rows(shift, batch, h), sc = mod_rows(scale, batch, h);
    const Tensor gt = mod_rows(gate, batch, h);
    if (sh.size(0) != sc.size(0) || (sh.size(0) > 1 && sh.stride(0) != sc.stride(0))) {  // one stride serves both vectors
      sh = sh.expand({batch, h}).contiguous();
      sc = sc.expand({batch, h}).contiguous();
    }
    const int64_t ldm = sh.size(0) > 1 ? sh.stride(0) : 0;
    Tensor y = at::empty(x.sizes(), x2.options());
    if (m == 0) return y.to(x.scalar_type());
    Arena a;
    const size_t xp = a.add(size_t(3) * m * h), hp = a.add(size_t(3) * m * f);
    a.allocate(x2);
    void* st = stream_of(x);
    int* status = status_ptr(x.get_device());
    check(tybok_layernorm_modulate_groups(ptr(x2), x2.stride(0), ptr(sh), ptr(sc), ldm, per, m, h, eps_, nullptr, h, a.at(xp),
                                          SHIFT_NORMED, st),
          "tybok_layernorm_modulate");
    check(tybok_w8x3_linear(a.at(xp), SHIFT_NORMED, up_.wp(), up_.sp(), up_.bp(), nullptr, f, a.at(hp), SHIFT_FFN, m, f, h, TYBOK_EPI_GELU,
                            nullptr, 0, nullptr, 0, 1, 0, 0, 0, status, st),
          "tybok_w8x3_linear");
    check(tybok_w8x3_linear(a.at(hp), SHIFT_FFN, down_.wp(), down_.sp(), down_.bp(), ptr(y), h, nullptr, 0, m, h, f, TYBOK_EPI_RESIDUAL,
                            ptr(x2), x2.stride(0), ptr(gt), gt.size(0) > 1 ? gt.stride(0) : 0, gt.size(0) > 1 ? per : m, 1, 0, 0, status, st),
          "tybok_w8x3_linear");
    return y.scalar_type() == x.scalar_type() ? y : y.to(x.scalar_type());
  }

 private:
  // [1 or B, H] bf16 rows, 16-byte aligned, of a [B, 1, H], [1, 1, H] or [H] modulation (strided views are taken as they lie;
  // of a table of more rows, the first B).
  static Tensor mod_rows(const Tensor& t, int64_t batch, int64_t h) {
    Tensor r = t.reshape({-1, h});
    if (r.size(0) > batch && batch > 0) r = r.narrow(0, 0, batch);
    if (r.size(0) != 1 && r.size(0) != batch) value_error("ffn_tail: modulation rows must be one, or one per batch element");
    if (!is_bf16(r)) r = r.to(at::kBFloat16);
    if (r.stride(1) != 1 || r.stride(0) % 8 != 0 || (reinterpret_cast<uintptr_t>(r.data_ptr()) & 15)) r = r.contiguous();
    if (reinterpret_cast<uintptr_t>(r.data_ptr()) & 15) r = r.clone();
    return r;
  }
  W8 up_, down_;
  double eps_;
};

void bind_ops(py::module_& m) {
  m.attr("TWO_PLANE_MIN_TOKENS") = TWO_PLANE_MIN_TOKENS;
  m.def("status_word", [](int device) { return status_tensor(device); });
  // `…_op` / `run`: what the registered ops end in.  The others return None where the call is the dispatcher's.
  m.def("w8a16_linear_op", &w8a16_linear, NoGil());
  m.def("attention_op", &attention, NoGil());
  m.def(
      "w8a16_linear",
      [](const Tensor& x, const Tensor& w8, const Tensor& scale, const OptTensor& bias, int epilogue, const OptTensor& residual,
         const OptTensor& gate, int rows_per_gate, int token_tile, int splits, int shift) -> OptTensor {
        if (!plain({&x, &w8, &scale, opt(bias), opt(residual), opt(gate)})) return std::nullopt;
        return w8a16_linear(x, w8, scale, bias, epilogue, residual, gate, rows_per_gate, token_tile, splits, shift);
      },
      NoGil());
  m.def(
      "attention",
      [](const Tensor& q, const Tensor& kc, const Tensor& vc, const OptTensor& valid, int tokens, int keys, double scale, bool out_bf16,
         bool out_planes, int out_shift) -> std::optional<std::tuple<Tensor, Tensor>> {
        if (!plain({&q, &kc, &vc, opt(valid)})) return std::nullopt;
        return attention(q, kc, vc, valid, tokens, keys, scale, out_bf16, out_planes, out_shift);
      },
      NoGil());
  py::class_<Mlp>(m, "Mlp")
      .def(py::init<const py::tuple&, const py::object&, const py::tuple&>())
      .def("run", &Mlp::forward, NoGil())
      .def(
          "forward", [](const Mlp& c, const Tensor& x) -> OptTensor { return plain({&x}) ? OptTensor(c.forward(x)) : std::nullopt; }, NoGil());
  py::class_<FfnTail>(m, "FfnTail")
      .def(py::init<const py::tuple&, const py::tuple&, double>())
      .def("run", &FfnTail::forward, NoGil())
      .def(
          "forward",
          [](const FfnTail& c, const Tensor& x, const Tensor& shift, const Tensor& scale, const Tensor& gate) -> OptTensor {
            return plain({&x, &shift, &scale, &gate}) ? OptTensor(c.forward(x, shift, scale, gate)) : std::nullopt;
          },
          NoGil());
}

}  // namespace tbn

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  tbn::bind_ops(m);
  tbn::bind_dit(m);
  tbn::bind_gemma(m);
}
