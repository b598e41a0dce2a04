// A stack of Gemma decoder layers (VLM prefix, action expert) as a single call on one workspace.
#include "native.h"

#include <cuda_runtime_api.h>

#include <cmath>

#include <algorithm>

namespace tbn {

class GemmaStack {
 public:
  // layers: per layer (qkv paired, o, gate_up packed or gate, up or None, down, input norm weight or None, post norm weight or None).
  GemmaStack(int width, int heads, int kv_heads, int head_dim, const py::list& layers)
      : w_(width), heads_(heads), kv_(kv_heads), hd_(head_dim) {
    for (const py::handle& h : layers) {
      const py::tuple t = py::reinterpret_borrow<py::tuple>(h);
      Layer l;
      l.qkv = w8_of(t[0], "gemma");
      l.o = w8_of(t[1], "gemma");
      l.gate_up = w8_of(t[2], "gemma");
      l.packed = t[3].is_none();
      if (!l.packed) l.up = w8_of(t[3], "gemma");
      l.down = w8_of(t[4], "gemma");
      if (!t[5].is_none()) {
        l.norm_in = t[5].cast<Tensor>();
        l.norm_post = t[6].cast<Tensor>();
      }
      // every layer runs on one workspace, sized by the first one's widths
      const int inner = l.down.k, a = heads_ * hd_;
      if (!l.qkv.is((heads_ + 2 * kv_) * hd_, w_) || !l.o.is(w_, a) || !l.gate_up.is(l.packed ? 2 * inner : inner, w_) ||
          (!l.packed && !l.up.is(inner, w_)) || l.down.n != w_ || (!layers_.empty() && inner != layers_[0].down.k))
        value_error("gemma_stack: the weights' shapes disagree with the stack's widths");
      if (l.norm_in && (!is_vector(*l.norm_in, at::kFloat, w_) || !is_vector(*l.norm_post, at::kFloat, w_)))
        type_error("gemma_stack: norm weights must be contiguous fp32 [W]");
      const at::Device d = layers_.empty() ? l.qkv.device() : layers_[0].qkv.device();
      same_device(d, "gemma_stack", {&l.qkv.w, &l.o.w, &l.gate_up.w, l.packed ? nullptr : &l.up.w, &l.down.w, opt(l.norm_in), opt(l.norm_post)});
      layers_.push_back(l);
    }
  }

  // Layers [first, first + count) on x [B*L, W] bf16.  `mods`: per layer (input, post) AdaRMS rows fp32 [1, 3W], or None
  // for the plain norms.  `fold`: per layer (W shift of the qkv rows, W shift of the gate/up rows), or None; with it, and
  // below the two-plane threshold, every AdaRMS norm after the first one of the call is folded into the GEMMs around it.
  // `wait` / `record`: CUDA events per layer to wait for before it / to record after it.
  Tensor forward(const Tensor& x, int b, int l, const Tensor& pos, const Tensor& cos, const Tensor& sin, const std::vector<Tensor>& kc,
                 const std::vector<Tensor>& vc, int key_off, const Tensor& key_valid, const std::optional<std::vector<std::pair<Tensor, Tensor>>>& mods,
                 const std::optional<std::vector<std::pair<Tensor, Tensor>>>& fold, int first, int count, const std::vector<uint64_t>& wait,
                 const std::vector<uint64_t>& record) const {
    return run(x, b, l, pos, cos, sin, kc, vc, key_off, key_valid, mods, fold, first, count, wait, record, false);
  }
  // The same for the caches alone: a prefix whose output nobody reads ends with its last layer's keys and values.  That layer's
  // attention, output projection and FFN are nearly an eighteenth of the pass (66.3 -> 62.8 ms at batch 32).
  void fill_caches(const Tensor& x, int b, int l, const Tensor& pos, const Tensor& cos, const Tensor& sin, const std::vector<Tensor>& kc,
                   const std::vector<Tensor>& vc, const Tensor& key_valid, const std::vector<uint64_t>& record) const {
    run(x, b, l, pos, cos, sin, kc, vc, 0, key_valid, std::nullopt, std::nullopt, 0, static_cast<int>(layers_.size()), {}, record, true);
  }

 private:
  Tensor run(const Tensor& x, int b, int l, const Tensor& pos, const Tensor& cos, const Tensor& sin, const std::vector<Tensor>& kc,
             const std::vector<Tensor>& vc, int key_off, const Tensor& key_valid, const std::optional<std::vector<std::pair<Tensor, Tensor>>>& mods,
             const std::optional<std::vector<std::pair<Tensor, Tensor>>>& fold, int first, int count, const std::vector<uint64_t>& wait,
             const std::vector<uint64_t>& record, bool caches_only) const {
    const int m = b * l, a = heads_ * hd_, keys = key_off + l;
    const Tensor x0 = rows_of(x);
    if (!is_bf16(x0) || x0.size(0) != m || x0.size(1) != w_) type_error("gemma_stack: x must be bf16 [B*L, W]");
    if (pos.scalar_type() != at::kInt || pos.numel() != m || !pos.is_contiguous()) type_error("gemma_stack: pos must be contiguous int32 [B*L]");
    if (key_valid.scalar_type() != at::kByte || key_valid.dim() != 2 || key_valid.size(0) != b || key_valid.size(1) != keys || !key_valid.is_contiguous())
      type_error("attention: key_valid must be contiguous uint8 [B, Lk]");
    for (const Tensor* t : {&cos, &sin})
      if (!is_bf16(*t) || !t->is_contiguous() || t->size(-1) != hd_) type_error("gemma_stack: cos/sin tables must be contiguous bf16 [max_pos, D]");
    if (cos.sizes() != sin.sizes()) value_error("gemma_stack: cos and sin tables differ in shape");
    const int n = layers_.size();
    if (first < 0 || count <= 0 || first + count > n || static_cast<int>(kc.size()) < n || static_cast<int>(vc.size()) < n ||
        (mods && static_cast<int>(mods->size()) < n) || (fold && static_cast<int>(fold->size()) < n))
      value_error("gemma_stack: one cache pair and one set of modulations per layer");
    if ((!wait.empty() && static_cast<int>(wait.size()) < first + count) || (!record.empty() && static_cast<int>(record.size()) < first + count))
      value_error("gemma_stack: one event per layer");
    const int lcap = kc[0].dim() == 4 ? kc[0].size(2) : -1;
    for (int i = first; i < first + count; ++i)
      for (const Tensor* t : {&kc[i], &vc[i]})
        if (!is_bf16(*t) || !t->is_contiguous() || t->dim() != 4 || t->size(0) != b || t->size(1) != kv_ || t->size(2) != lcap || t->size(3) != hd_)
          type_error("gemma_stack: caches must be contiguous bf16 [B, G, Lcap, D]");
    if (mods)
      for (int i = first; i < first + count; ++i)
        for (const Tensor* t : {&(*mods)[i].first, &(*mods)[i].second})
          if (t->scalar_type() != at::kFloat || !t->is_contiguous() || t->numel() != 3 * w_) type_error("gemma_stack: modulations must be contiguous fp32 [1, 3W]");

    for (int i = first; i < first + count; ++i) {
      if (!mods && !layers_[i].norm_in) value_error("gemma_stack: a layer without norm weights needs its modulations");
      if (fold && (!is_vector((*fold)[i].first, at::kFloat, layers_[i].qkv.n) || !is_vector((*fold)[i].second, at::kFloat, layers_[i].gate_up.n)))
        type_error("gemma_stack: W shift rows must be contiguous fp32 [weight rows]");
    }
    const at::Device dev = layers_[0].qkv.device();
    same_device(dev, "gemma_stack", {&x, &pos, &cos, &sin, &key_valid});
    for (int i = first; i < first + count; ++i) {
      same_device(dev, "gemma_stack", {&kc[i], &vc[i]});
      if (mods) same_device(dev, "gemma_stack", {&(*mods)[i].first, &(*mods)[i].second});
      if (fold) same_device(dev, "gemma_stack", {&(*fold)[i].first, &(*fold)[i].second});
    }
    require_cuda(x, "gemma_stack");
    const c10::cuda::CUDAGuard guard(x.device());

    const int inner = layers_[0].down.k;
    bool packed = true, any_packed = false;
    for (int i = first; i < first + count; ++i) {
      packed = packed && layers_[i].packed;
      any_packed = any_packed || layers_[i].packed;
    }
    const bool folds = mods && fold && m < TWO_PLANE_MIN_TOKENS && any_packed;
    const size_t at_ws = tybok_attention_workspace_needed(b, l, heads_, kv_, hd_, keys);
    const size_t u = folds ? size_t(3) * m * w_ : 0, part = folds ? size_t(4) * m * (w_ / 128 + 1) : 0;
    Arena ar;
    const size_t np = ar.add(size_t(packed && m >= TWO_PLANE_MIN_TOKENS ? 2 : 3) * m * w_), rs = ar.add(size_t(4) * m);
    const size_t q = ar.add(size_t(2) * m * a), ap = ar.add(size_t(3) * m * a), hp = ar.add(size_t(3) * m * inner);
    const size_t x1 = ar.add(size_t(2) * m * w_), xa = ar.add(size_t(2) * m * w_), xb = ar.add(size_t(2) * m * w_), ws = ar.add(at_ws);
    const size_t up0 = ar.add(u), up1 = ar.add(u), part0 = ar.add(part), part1 = ar.add(part);
    ar.allocate(x0);
    Tensor y = at::empty({caches_only ? 0 : m, w_}, x0.options());
    void* st = stream_of(x);
    int* status = status_ptr(x.get_device());
    const float eps = 1e-6f, scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(hd_)));

    const void* cur = ptr(x0);
    int64_t ld = x0.stride(0);
    bool carried = false;  // up1 / part1 hold this layer's normed input in the folded form
    for (int i = first; i < first + count; ++i) {
      const Layer& lay = layers_[i];
      if (!wait.empty() && cudaStreamWaitEvent(static_cast<cudaStream_t>(st), reinterpret_cast<cudaEvent_t>(wait[i]), 0) != cudaSuccess)
        value_error("gemma_stack: cudaStreamWaitEvent failed");
      const bool last = i == first + count - 1;
      const bool folded = mods && fold && m < TWO_PLANE_MIN_TOKENS && lay.packed;
      const bool two = !folded && m >= TWO_PLANE_MIN_TOKENS && lay.packed;
      const float* mi = mods ? f32((*mods)[i].first) : nullptr;
      const float* mp = mods ? f32((*mods)[i].second) : nullptr;
      void* k = ptr(kc[i]);
      void* v = ptr(vc[i]);
      // ---- input norm, q / k / v with rotary embedding and cache store
      if (carried) {
        check(tybok_w8x3_qkv_rope_adarms(ar.at(up1), SHIFT_FOLD, static_cast<float*>(ar.at(part1)), w_ / 128, eps, f32((*fold)[i].first),
                                         lay.qkv.wp(), lay.qkv.sp(), static_cast<const int*>(ptr(pos)), ptr(cos), ptr(sin), ar.at(q), k, v, b, l,
                                         heads_, kv_, hd_, lcap, key_off, w_, 0, 0, status, st),
              "tybok_w8x3_qkv_rope_adarms");
      } else {
        norm(two, cur, ld, lay.norm_in, mi, m, eps, ar.at(np), ar.at(rs), st);
        if (two)
          check(tybok_w8x2_qkv_rope(ar.at(np), static_cast<float*>(ar.at(rs)), lay.qkv.wp(), lay.qkv.sp(), static_cast<const int*>(ptr(pos)),
                                    ptr(cos), ptr(sin), ar.at(q), k, v, b, l, heads_, kv_, hd_, lcap, key_off, w_, 0, 0, status, st),
                "tybok_w8x2_qkv_rope");
        else
          check(tybok_w8x3_qkv_rope(ar.at(np), SHIFT_NORMED, lay.qkv.wp(), lay.qkv.sp(), static_cast<const int*>(ptr(pos)), ptr(cos), ptr(sin),
                                    ar.at(q), k, v, b, l, heads_, kv_, hd_, lcap, key_off, w_, 0, 0, status, st),
                "tybok_w8x3_qkv_rope");
      }
      if (caches_only && last) {
        record_event(record, i, st);
        break;
      }
      check(tybok_attention(ar.at(q), k, v, ptr(key_valid), nullptr, ar.at(ap), SHIFT_ATTN, b, l, heads_, kv_, hd_, keys, lcap, scale, ar.at(ws),
                            at_ws, status, st),
            "tybok_attention");
      void* out = last ? ptr(y) : ar.at((i - first) & 1 ? xb : xa);
      if (folded) {
        check(tybok_w8x3_residual_next_adarms(ar.at(ap), SHIFT_ATTN, lay.o.wp(), lay.o.sp(), ar.at(x1), w_, cur, ld, mi + 2 * w_, mp, ar.at(up0),
                                              SHIFT_FOLD, static_cast<float*>(ar.at(part0)), m, w_, a, 0, 0, status, st),
              "tybok_w8x3_residual_next_adarms");
        check(tybok_w8x3_geglu_packed_adarms(ar.at(up0), SHIFT_FOLD, static_cast<float*>(ar.at(part0)), w_ / 128, eps, f32((*fold)[i].second),
                                             lay.gate_up.wp(), lay.gate_up.sp(), nullptr, inner, ar.at(hp), SHIFT_FFN, m, inner, w_, 0, 0,
                                             status, st),
              "tybok_w8x3_geglu_packed_adarms");
        carried = !last && layers_[i + 1].packed;
        if (carried)
          check(tybok_w8x3_residual_next_adarms(ar.at(hp), SHIFT_FFN, lay.down.wp(), lay.down.sp(), out, w_, ar.at(x1), w_, mp + 2 * w_,
                                                f32((*mods)[i + 1].first), ar.at(up1), SHIFT_FOLD, static_cast<float*>(ar.at(part1)), m, w_, inner,
                                                0, 0, status, st),
                "tybok_w8x3_residual_next_adarms");
        else
          residual(ar.at(hp), SHIFT_FFN, lay.down, out, ar.at(x1), w_, mp + 2 * w_, m, status, st);
      } else {
        residual(ar.at(ap), SHIFT_ATTN, lay.o, ar.at(x1), cur, ld, mi ? mi + 2 * w_ : nullptr, m, status, st);
        norm(two, ar.at(x1), w_, lay.norm_post, mp, m, eps, ar.at(np), ar.at(rs), st);
        if (two)
          check(tybok_w8x2_gemm(ar.at(np), static_cast<float*>(ar.at(rs)), lay.gate_up.wp(), lay.gate_up.sp(), nullptr, nullptr, inner, ar.at(hp),
                                SHIFT_FFN, m, 2 * inner, w_, TYBOK_EPI_GEGLU_PACKED, nullptr, 0, nullptr, 0, 1, 0, 0, 0, status, st),
                "tybok_w8x2_gemm");
        else if (lay.packed)
          check(tybok_w8x3_geglu_packed(ar.at(np), SHIFT_NORMED, lay.gate_up.wp(), lay.gate_up.sp(), nullptr, inner, ar.at(hp), SHIFT_FFN, m,
                                        inner, w_, 0, 0, status, st),
                "tybok_w8x3_geglu_packed");
        else
          check(tybok_w8x3_geglu(ar.at(np), SHIFT_NORMED, lay.gate_up.wp(), lay.gate_up.sp(), lay.up.wp(), lay.up.sp(), nullptr, inner, ar.at(hp),
                                 SHIFT_FFN, m, inner, w_, 0, 0, status, st),
                "tybok_w8x3_geglu");
        residual(ar.at(hp), SHIFT_FFN, lay.down, out, ar.at(x1), w_, mp ? mp + 2 * w_ : nullptr, m, status, st);
        carried = false;
      }
      cur = out;
      ld = w_;
      record_event(record, i, st);
    }
    return y;
  }

  static void record_event(const std::vector<uint64_t>& events, int i, void* st) {
    if (!events.empty() && cudaEventRecord(reinterpret_cast<cudaEvent_t>(events[i]), static_cast<cudaStream_t>(st)) != cudaSuccess)
      value_error("gemma_stack: cudaEventRecord failed");
  }
  struct Layer {
    W8 qkv, o, gate_up, up, down;
    bool packed = true;
    OptTensor norm_in, norm_post;
  };
  void norm(bool two, const void* x, int64_t ld, const OptTensor& weight, const float* mod, int m, float eps, void* planes, void* rs, void* st) const {
    const float* w = mod ? nullptr : f32(*weight);
    if (two)
      check(tybok_norm_planes2(x, ld, mod ? TYBOK_NORM_ADARMS : TYBOK_NORM_RMS, mod ? mod : w, nullptr, mod ? 3 * w_ : 0, m, m, w_, eps, planes,
                               static_cast<float*>(rs), st),
            "tybok_norm_planes2");
    else
      check(tybok_rmsnorm(x, ld, w, mod, mod ? 3 * w_ : 0, m, m, w_, eps, nullptr, w_, planes, SHIFT_NORMED, st), "tybok_rmsnorm");
  }
  static void residual(const void* planes, int shift, const W8& w, void* y, const void* res, int64_t ldres, const float* gate, int m, int* status,
                       void* st) {
    check(tybok_w8x3_linear(planes, shift, w.wp(), w.sp(), nullptr, y, w.n, nullptr, 0, m, w.n, w.k, TYBOK_EPI_RESIDUAL, res, ldres, gate, w.n, m,
                            0, 0, 0, status, st),
          "tybok_w8x3_linear");
  }

  int w_, heads_, kv_, hd_;
  std::vector<Layer> layers_;
};

void bind_gemma(py::module_& m) {
  py::class_<GemmaStack>(m, "GemmaStack")
      .def(py::init<int, int, int, int, const py::list&>())
      .def("forward", &GemmaStack::forward, NoGil())
      .def("fill_caches", &GemmaStack::fill_caches, NoGil());
}

}  // namespace tbn
