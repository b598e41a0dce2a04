// Shared by the sources of the tybok_b200._native extension: the host path from torch tensors to the C ABI without
// Python or the torch dispatcher in between.  A chain of launches (an FFN, a block, a decoder stack) is one call here.
#pragma once

#include <ATen/ATen.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <initializer_list>
#include <optional>
#include <string>
#include <vector>

#include "../../../include/tybok_b200.h"

namespace tbn {

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

// Exponent shifts of the activation planes per producer (planes hold value * 2^shift).
constexpr int SHIFT_NORMED = 4;  // normalised activations, O(1)
constexpr int SHIFT_ATTN = 6;    // attention outputs: convex combinations of value rows
constexpr int SHIFT_FFN = 4;     // FFN intermediates
constexpr int SHIFT_FOLD = 0;    // residual stream times (1 + scale), not normalised
// From this many token rows a GEMM fed by a norm takes two e4m3 planes with a per-row scale (a third less tensor work, token
// tiles to 128); below it the GEMMs are bound by launch latency and keep the three-plane form.
constexpr int TWO_PLANE_MIN_TOKENS = 128;

// Every call that launches runs without the interpreter lock: a launch waits while the device's queue is full, and other
// threads' Python must go on meanwhile.  What touches Python objects in such a call takes the lock for itself.
using NoGil = py::call_guard<py::gil_scoped_release>;

// Whether a call on these may run as it stands.  Inside a function transform or a dispatch mode, and for tensors that intercept
// torch ops, it has to go through the dispatcher: the Python side then calls the registered op, which ends in the
// unchecked form of the same call.  (Asked here: in Python the question cost a call 1 us.)
inline bool plain(std::initializer_list<const Tensor*> tensors) {
  using K = c10::DispatchKey;
  if (c10::impl::dispatch_mode_enabled() || c10::impl::tls_is_dispatch_key_included(K::FuncTorchDynamicLayerFrontMode)) return false;
  constexpr c10::DispatchKeySet intercepts{K::Python, K::FuncTorchBatched, K::FuncTorchGradWrapper, K::Functionalize};
  for (const Tensor* t : tensors)
    if (t && t->key_set().has_any(intercepts)) return false;
  return true;
}

[[noreturn]] void raise_status(int rc, const char* what);
inline void check(int rc, const char* what) {
  if (rc != 0) raise_status(rc, what);
}
[[noreturn]] inline void type_error(const std::string& m) { throw py::type_error(m); }
[[noreturn]] inline void value_error(const std::string& m) { throw py::value_error(m); }
void require_cuda(const Tensor& t, const char* what);  // NotImplementedError for anything else

int* status_ptr(int device);  // per-device status word (created once, kept)

inline void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
inline void* ptr(const Tensor& t) { return t.data_ptr(); }
inline void* ptr(const OptTensor& t) { return t ? t->data_ptr() : nullptr; }
inline const float* f32(const Tensor& t) { return static_cast<const float*>(t.data_ptr()); }
inline bool is_bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }

// Kernels take plain addresses: a tensor of another device must not get as far as a launch.
inline void same_device(at::Device d, const char* what, std::initializer_list<const Tensor*> tensors) {
  for (const Tensor* t : tensors)
    if (t && t->device() != d) value_error(std::string(what) + ": tensors on " + t->device().str() + " and " + d.str());
}
inline bool is_vector(const Tensor& t, at::ScalarType type, int64_t n) { return t.scalar_type() == type && t.numel() == n && t.is_contiguous(); }
inline const Tensor* opt(const OptTensor& t) { return t ? &*t : nullptr; }

// [rows, width] view of x with unit inner stride.
Tensor rows_of(const Tensor& x);
// The same in bf16 and as the kernels read rows in vectors: 16-byte aligned, row stride a multiple of 8 and at least the
// width.  Anything else (a slice of wider rows, an expanded row, another type) is copied.
Tensor vector_rows_of(const Tensor& x);

// An e4m3 weight [n, k] with its fp32 scale [n] and optional bf16 bias [n].
struct W8 {
  Tensor w, s;
  OptTensor b;
  int n = 0, k = 0;
  const void* wp() const { return w.data_ptr(); }
  const float* sp() const { return f32(s); }
  const void* bp() const { return b ? b->data_ptr() : nullptr; }
  at::Device device() const { return w.device(); }
  bool is(int64_t rows, int64_t cols) const { return n == rows && k == cols; }
};
W8 w8_of(const py::handle& t, const char* what);  // (weight, scale[, bias])

// One allocation per chain, carved into 256-byte aligned pieces; stream-ordered like any torch allocation.
class Arena {
 public:
  size_t add(size_t bytes) {
    const size_t at = size_;
    size_ += (bytes + 255) & ~size_t(255);
    return at;
  }
  void allocate(const Tensor& like) {
    buf_ = at::empty({static_cast<int64_t>(size_ ? size_ : 1)}, like.options().dtype(at::kByte));
    base_ = static_cast<char*>(buf_.data_ptr());
  }
  void* at(size_t offset) const { return base_ + offset; }
  const Tensor& tensor() const { return buf_; }

 private:
  size_t size_ = 0;
  Tensor buf_;
  char* base_ = nullptr;
};

void bind_ops(py::module_& m);
void bind_dit(py::module_& m);
void bind_gemma(py::module_& m);

}  // namespace tbn
