// One DiT block as a single call: every launch of DiTBlock.forward (and of its FFN when it is not sharded), on one
// workspace.  Between two kernels the Python form spent 20-25 us on the host; here it is about 3.
#include "native.h"

#include <algorithm>
#include <cmath>

namespace tbn {

class DitBlock {
 public:
  DitBlock(int heads, int head_dim, double eps, const py::tuple& qkv, const py::tuple& o, const py::tuple& cross_q, const py::tuple& cross_o,
           const py::object& up, const py::object& down, const Tensor& norm_q, const Tensor& norm_k, const Tensor& cross_norm_q,
           const Tensor& norm3_w, const Tensor& norm3_b)
      : heads_(heads), hd_(head_dim), eps_(eps), qkv_(w8_of(qkv, "dit")), o_(w8_of(o, "dit")), cq_(w8_of(cross_q, "dit")),
        co_(w8_of(cross_o, "dit")), nq_(norm_q), nk_(norm_k), cnq_(cross_norm_q), n3w_(norm3_w), n3b_(norm3_b) {
    ffn_ = !up.is_none();  // a sharded FFN is finished by the caller (its all-reduce is a collective)
    if (ffn_) {
      up_ = w8_of(up, "dit");
      down_ = w8_of(down, "dit");
    }
    h_ = qkv_.k;
    const int a = heads_ * hd_;
    if (!qkv_.is(3 * a, h_) || !o_.is(h_, a) || !cq_.is(a, h_) || !co_.is(h_, a) || (ffn_ && (up_.k != h_ || !down_.is(h_, up_.n))))
      value_error("DiTBlock: the weights' shapes disagree with heads, head_dim and one another");
    for (const Tensor* t : {&nq_, &nk_, &cnq_})
      if (!is_vector(*t, at::kBFloat16, a)) type_error("DiTBlock: qk-norm weights must be contiguous bf16 [H*D]");
    for (const Tensor* t : {&n3w_, &n3b_})
      if (!is_vector(*t, at::kBFloat16, h_)) type_error("DiTBlock: norm3 must be contiguous bf16 [H]");
    same_device(qkv_.device(), "DiTBlock", {&o_.w, &cq_.w, &co_.w, ffn_ ? &up_.w : nullptr, ffn_ ? &down_.w : nullptr, &nq_, &nk_, &cnq_, &n3w_, &n3b_});
  }

  // x [S, H] bf16.  Keys and values: `k_cache` / `v_cache` [1, heads, Lcap, D] with this block's own appended at key_off;
  // or, with `k_rows` / `v_rows` [Lv, heads*D] (token-major, read in place), a tail cache [heads, cap, D] (finite) that
  // takes the last Lv % 128 rows and this block's own.  Cross keys and values likewise head-major (4-D) or token-major (2-D).
  Tensor forward(const Tensor& x, const Tensor& mods, const Tensor& cos, const Tensor& sin, const Tensor& k_cache, const Tensor& v_cache,
                 int key_off, const OptTensor& k_rows, const OptTensor& v_rows, const OptTensor& cross_k, const OptTensor& cross_v,
                 const OptTensor& ctx_valid) const {
    const Tensor x0 = rows_of(x);
    const int m = x0.size(0), a = heads_ * hd_, h = h_;
    if (!is_bf16(x0) || x0.size(1) != h) type_error("DiTBlock: x must be bf16 [S, H]");
    if (!is_bf16(mods) || mods.size(0) != 6 || mods.numel() != 6 * h) type_error("DiTBlock: mods must be bf16 [6, H]");
    for (const Tensor* t : {&cos, &sin})
      if (t->scalar_type() != at::kFloat || !t->is_contiguous() || t->dim() != 2 || t->size(0) != m || t->size(1) != hd_ / 2)
        type_error("DiTBlock: cos/sin must be contiguous fp32 [S, D/2]");
    // The kernels are told one key count and one capacity per pair of keys and values; both sides must have them.
    const int lk = k_rows ? static_cast<int>(k_rows->size(0)) + m : key_off + m;
    const int lc = ctx_valid ? static_cast<int>(ctx_valid->size(-1)) : cross_k ? static_cast<int>(cross_k->size(-2)) : 0;
    check_pair(k_cache, v_cache, false);
    if (k_rows.has_value() != v_rows.has_value()) value_error("DiTBlock: key rows come with value rows");
    if (k_rows) check_pair(*k_rows, *v_rows, true);
    if (cross_k.has_value() != cross_v.has_value()) value_error("DiTBlock: cross keys come with cross values");
    if (cross_k) {
      check_pair(*cross_k, *cross_v, cross_k->dim() == 2);
      if (cross_k->size(-2) < lc) value_error("DiTBlock: the context mask is longer than the cross keys");
    }
    if (ctx_valid && (ctx_valid->scalar_type() != at::kByte || !ctx_valid->is_contiguous() || ctx_valid->numel() != lc))
      type_error("attention: key_valid must be contiguous uint8 [B, Lk]");
    same_device(qkv_.device(), "DiTBlock", {&x, &mods, &cos, &sin, &k_cache, &v_cache, opt(k_rows), opt(v_rows), opt(cross_k), opt(cross_v), opt(ctx_valid)});
    require_cuda(x, "dit_block");
    const c10::cuda::CUDAGuard guard(x.device());
    const int lcap = k_cache.size(-2);
    void* st = stream_of(x);
    int* status = status_ptr(x.get_device());
    const bool two = m >= TWO_PLANE_MIN_TOKENS;
    const float scale = static_cast<float>(1.0 / std::sqrt(static_cast<double>(hd_)));

    // ---- workspace: normed planes | union of (qkv, q, attention planes) and the FFN's hidden planes | two residual rows
    size_t at_ws = k_rows ? 0 : tybok_attention_workspace_needed(1, m, heads_, heads_, hd_, lk);
    if (cross_k && cross_k->dim() != 2) at_ws = std::max(at_ws, tybok_attention_workspace_needed(1, m, heads_, heads_, hd_, lc));
    Arena ar;
    const size_t np = ar.add(size_t(two ? 2 : 3) * m * h), rs = ar.add(size_t(4) * m);
    const size_t x1 = ar.add(size_t(2) * m * h), x2 = ar.add(size_t(2) * m * h), ws = ar.add(at_ws);
    const size_t qkv = ar.add(size_t(2) * m * 3 * a), q = ar.add(size_t(2) * m * a), ap = ar.add(size_t(3) * m * a);
    const size_t used = size_t(2) * m * 3 * a + size_t(2) * m * a + size_t(3) * m * a;
    if (ffn_ && size_t(3) * m * up_.n > used) ar.add(size_t(3) * m * up_.n - used);
    const size_t hp = qkv;
    ar.allocate(x0);
    Tensor y = at::empty({m, h}, x0.options());
    const Tensor table = mods.contiguous();  // rows that lie apart are gathered
    const char* mod = static_cast<const char*>(table.data_ptr());
    auto mrow = [&](int i) { return static_cast<const void*>(mod + size_t(2) * h * i); };

    // ---- modulated self-attention
    norm_modulate(ptr(x0), x0.stride(0), mrow(0), mrow(1), m, two, ar.at(np), ar.at(rs), st);
    gemm(two, ar.at(np), ar.at(rs), qkv_, ar.at(qkv), nullptr, m, TYBOK_EPI_NONE, status, st);
    int off = key_off;
    if (k_rows) {
      const int lv = k_rows->size(0);
      off = lv % 128;
      if (off)
        check(tybok_kv_rows_to_heads(ptr(*k_rows), ptr(*v_rows), lv - off, off, ptr(k_cache), ptr(v_cache), lcap, heads_, hd_, st),
              "tybok_kv_rows_to_heads");
    }
    check(tybok_qknorm_rope_store(ar.at(qkv), 3 * a, 0, a, 2 * a, ptr(nq_), ptr(nk_), eps_, f32(cos), f32(sin), ar.at(q), ptr(k_cache),
                                  ptr(v_cache), 1, m, heads_, hd_, lcap, off, st),
          "tybok_qknorm_rope_store");
    if (k_rows)
      check(tybok_attention_rows(ar.at(q), ptr(*k_rows), ptr(*v_rows), k_rows->size(0), ptr(k_cache), ptr(v_cache), lcap, nullptr, nullptr,
                                 ar.at(ap), SHIFT_ATTN, m, heads_, hd_, lk, scale, status, st),
            "tybok_attention_rows");
    else
      check(tybok_attention(ar.at(q), ptr(k_cache), ptr(v_cache), nullptr, nullptr, ar.at(ap), SHIFT_ATTN, 1, m, heads_, heads_, hd_, lk, lcap,
                            scale, ar.at(ws), at_ws, status, st),
            "tybok_attention");
    void* cur = (cross_k || ffn_) ? ar.at(x1) : ptr(y);
    residual(ar.at(ap), SHIFT_ATTN, o_, cur, ptr(x0), x0.stride(0), mrow(2), m, status, st);

    // ---- masked cross-attention over the cached context
    if (cross_k) {
      if (two)
        check(tybok_norm_planes2(cur, h, TYBOK_NORM_LN_AFFINE, ptr(n3w_), ptr(n3b_), 0, 1, m, h, eps_, ar.at(np), static_cast<float*>(ar.at(rs)), st),
              "tybok_norm_planes2");
      else
        check(tybok_layernorm_affine(cur, h, ptr(n3w_), ptr(n3b_), m, h, eps_, nullptr, h, ar.at(np), SHIFT_NORMED, st), "tybok_layernorm_affine");
      gemm(two, ar.at(np), ar.at(rs), cq_, ar.at(qkv), nullptr, m, TYBOK_EPI_NONE, status, st);
      check(tybok_qknorm_rope_store(ar.at(qkv), a, 0, -1, -1, ptr(cnq_), nullptr, eps_, nullptr, nullptr, ar.at(q), nullptr, nullptr, 1, m,
                                    heads_, hd_, 0, 0, st),
            "tybok_qknorm_rope_store");
      if (cross_k->dim() == 2) {
        check(tybok_attention_rows(ar.at(q), ptr(*cross_k), ptr(*cross_v), lc, nullptr, nullptr, 0, ptr(ctx_valid), nullptr, ar.at(ap),
                                   SHIFT_ATTN, m, heads_, hd_, lc, scale, status, st),
              "tybok_attention_rows");
      } else {
        check(tybok_attention(ar.at(q), ptr(*cross_k), ptr(*cross_v), ptr(ctx_valid), nullptr, ar.at(ap), SHIFT_ATTN, 1, m, heads_, heads_,
                              hd_, lc, cross_k->size(-2), scale, ar.at(ws), at_ws, status, st),
              "tybok_attention");
      }
      void* next = ffn_ ? ar.at(x2) : ptr(y);
      residual(ar.at(ap), SHIFT_ATTN, co_, next, cur, h, nullptr, m, status, st);
      cur = next;
    }
    if (ffn_) ffn_tail(cur, h, mrow(3), mrow(4), mrow(5), m, two, ar.at(np), ar.at(rs), ar.at(hp), ptr(y), status, st);
    return y;
  }

 private:
  // Keys and values of one shape: head-major [1, heads, Lcap, D] (a tail cache without the 1), or rows [L, heads*D].
  void check_pair(const Tensor& k, const Tensor& v, bool rows) const {
    for (const Tensor* t : {&k, &v}) {
      if (rows && (!is_bf16(*t) || !t->is_contiguous() || t->dim() != 2 || t->size(1) != heads_ * hd_))
        type_error("DiTBlock: key / value rows must be contiguous bf16 [L, heads*D]");
      if (!rows && (!is_bf16(*t) || !t->is_contiguous() || t->dim() < 3 || t->size(-1) != hd_ || t->size(-3) != heads_ ||
                    t->numel() != t->size(-2) * heads_ * hd_))
        type_error("DiTBlock: caches must be contiguous bf16 [1, heads, Lcap, D]");
    }
    if (k.size(-2) != v.size(-2)) value_error("DiTBlock: keys and values differ in length");
  }
  void norm_modulate(const void* x, int64_t ld, const void* shift, const void* scale, int m, bool two, void* planes, void* rs, void* st) const {
    if (two)
      check(tybok_norm_planes2(x, ld, TYBOK_NORM_LN_MODULATE, shift, scale, 0, 1, m, h_, eps_, planes, static_cast<float*>(rs), st), "tybok_norm_planes2");
    else
      check(tybok_layernorm_modulate(x, ld, shift, scale, m, h_, eps_, nullptr, h_, planes, SHIFT_NORMED, st), "tybok_layernorm_modulate");
  }
  static void gemm(bool two, const void* planes, const void* rs, const W8& w, void* y, void* yp, int m, int epi, int* status, void* st) {
    if (two)
      check(tybok_w8x2_gemm(planes, static_cast<const float*>(rs), w.wp(), w.sp(), w.bp(), y, w.n, yp, SHIFT_FFN, m, w.n, w.k, epi, nullptr,
                            0, nullptr, 0, 1, 0, 0, 0, status, st),
            "tybok_w8x2_gemm");
    else
      check(tybok_w8x3_linear(planes, SHIFT_NORMED, w.wp(), w.sp(), w.bp(), y, w.n, yp, SHIFT_FFN, m, w.n, w.k, epi, nullptr, 0, nullptr, 0, 1,
                              0, 0, 0, status, st),
            "tybok_w8x3_linear");
  }
  static void residual(const void* planes, int shift, const W8& w, void* y, const void* res, int64_t ldres, const void* gate, int m, int* status,
                       void* st) {
    check(tybok_w8x3_linear(planes, shift, w.wp(), w.sp(), w.bp(), y, w.n, nullptr, 0, m, w.n, w.k, TYBOK_EPI_RESIDUAL, res, ldres, gate, w.n,
                            m, 1, 0, 0, status, st),
          "tybok_w8x3_linear");
  }
  void ffn_tail(const void* x, int64_t ld, const void* shift, const void* scale, const void* gate, int m, bool two, void* planes, void* rs,
                void* hp, void* y, int* status, void* st) const {
    norm_modulate(x, ld, shift, scale, m, two, planes, rs, st);
    gemm(two, planes, rs, up_, nullptr, hp, m, TYBOK_EPI_GELU, status, st);
    residual(hp, SHIFT_FFN, down_, y, x, ld, gate, m, status, st);
  }

  int heads_, hd_, h_ = 0;
  double eps_;
  bool ffn_ = false;
  W8 qkv_, o_, cq_, co_, up_, down_;
  Tensor nq_, nk_, cnq_, n3w_, n3b_;
};

void bind_dit(py::module_& m) {
  py::class_<DitBlock>(m, "DitBlock")
      .def(py::init<int, int, double, const py::tuple&, const py::tuple&, const py::tuple&, const py::tuple&, const py::object&, const py::object&,
                    const Tensor&, const Tensor&, const Tensor&, const Tensor&, const Tensor&>())
      .def("forward", &DitBlock::forward, NoGil());
}

}  // namespace tbn
