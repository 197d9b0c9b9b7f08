// Host side of the operators as a CPython extension (dlblas_b200/_host.so): argument checks, output and workspace
// allocation, stream lookup and the calls into the C ABI (include/dlblas_b200.h), without a Python frame per tensor.
//
// A small expert layer is some thirty microseconds of kernels.  Through ctypes it spent 140 us on the host: every C call
// converts up to twenty arguments, every torch.empty crosses the dispatcher, and a layer makes seven of the one and a dozen
// of the other.  Here a layer is one call: one workspace for everything that does not leave it, one C++ call per kernel.
//
// The module binds to the C ABI by the addresses that the ctypes loader hands over (bind), so that there is one copy of the
// library however it was located.  Errors of the C ABI become AssertionError (bad arguments, as the reference's
// asserts) or RuntimeError.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>

#include <array>
#include <cctype>
#include <cerrno>
#include <climits>
#include <cmath>
#include <cstdlib>
#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/dlblas_b200.h"

// What this file was compiled for (build.py); _C.host() looks for it before it loads the module.
extern "C" __attribute__((used)) const char dlb_host_built_for[] = DLB_HOST_TAG;

namespace {

using at::Tensor;

// ---- the C ABI by address -----------------------------------------------------------------------------------------
#define ABI_FUNCTIONS(X)                                                                                              \
  X(dlb_last_error_string)                                                                                            \
  X(dlb_sort_by_expert_workspace_size)                                                                                \
  X(dlb_moe_plan)                                                                                                     \
  X(dlb_quant_fp8)                                                                                                    \
  X(dlb_permute_rows)                                                                                                 \
  X(dlb_moe_grouped_gemm)                                                                                             \
  X(dlb_silu_mul_quant)                                                                                               \
  X(dlb_moe_sum_topk)                                                                                                 \
  X(dlb_fp8_gemm)                                                                                                     \
  X(dlb_route_softmax_topk)                                                                                           \
  X(dlb_route_grouped_topk)                                                                                           \
  X(dlb_moe_grouped_gemm_window)                                                                                      \
  X(dlb_ep_gather)                                                                                                    \
  X(dlb_moe_build_tiles_sizes)                                                                                        \
  X(dlb_grouped_gemm_16bit)                                                                                           \
  X(dlb_grouped_gemm_16bit_b_kn)                                                                                      \
  X(dlb_k_grouped_gemm_workspace_bytes)                                                                               \
  X(dlb_k_grouped_gemm_16bit)                                                                                         \
  X(dlb_silu_and_mul)                                                                                                 \
  X(dlb_moe_align_block_size)                                                                                         \
  X(dlb_topk_gating_workspace_size)                                                                                   \
  X(dlb_topk_gating)                                                                                                  \
  X(dlb_topk_gating_bwd)                                                                                              \
  X(dlb_permute_plan)                                                                                                 \
  X(dlb_unpermute)                                                                                                    \
  X(dlb_unpermute_bwd_rows)

struct Abi {
#define X(name) decltype(&::name) name = nullptr;
  ABI_FUNCTIONS(X)
#undef X
} abi;

// ---- errors -------------------------------------------------------------------------------------------------------
struct AssertionFailed : std::runtime_error {
  using std::runtime_error::runtime_error;
};
struct BadValue : std::runtime_error {
  using std::runtime_error::runtime_error;
};
void require(bool ok, const char* msg) {
  if (!ok) throw AssertionFailed(msg);
}
void check(int rc) {
  if (rc == DLB_OK) return;
  const std::string msg = abi.dlb_last_error_string();
  if (rc == DLB_ERR_INVALID) throw AssertionFailed(msg);
  throw std::runtime_error("dlblas_b200 error " + std::to_string(rc) + ": " + msg);
}

// ---- arguments ----------------------------------------------------------------------------------------------------
struct PyFailed {};   // a Python error is already set (thrown with the GIL held only)

// The work of a method, after its arguments are read and before its result is wrapped, runs without the GIL, as torch's own
// operators do: an allocation or a launch into a full queue can wait for the GPU, and other threads go on meanwhile.
template <typename F> auto without_gil(F&& f) {
  struct Released {
    PyThreadState* state = PyEval_SaveThread();
    ~Released() { PyEval_RestoreThread(state); }
  } released;
  return f();
}

const Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "expected a torch.Tensor");
    throw PyFailed{};
  }
  return THPVariable_Unpack(o);
}
std::optional<Tensor> opt_tensor(PyObject* o) {
  if (o == Py_None) return std::nullopt;
  return tensor(o);
}
int64_t integer(PyObject* o) {
  const long long v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PyFailed{};
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw PyFailed{};
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PyFailed{};
  return v != 0;
}
at::ScalarType dtype(PyObject* o) {
  if (!THPDtype_Check(o)) {
    PyErr_SetString(PyExc_TypeError, "expected a torch.dtype");
    throw PyFailed{};
  }
  return reinterpret_cast<THPDtype*>(o)->scalar_type;
}
void need_args(Py_ssize_t n, Py_ssize_t want) {
  if (n != want) {
    PyErr_Format(PyExc_TypeError, "expected %zd arguments, got %zd", want, n);
    throw PyFailed{};
  }
}
PyObject* wrap(const Tensor& t) { return THPVariable_Wrap(t); }
PyObject* wrap_tuple(std::initializer_list<const Tensor*> ts) {
  PyObject* r = PyTuple_New((Py_ssize_t)ts.size());
  Py_ssize_t i = 0;
  for (const Tensor* t : ts) PyTuple_SET_ITEM(r, i++, wrap(*t));
  return r;
}

// Runs the body of a method and turns C++ exceptions into Python ones.
template <typename F> PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const PyFailed&) {
    return nullptr;
  } catch (const AssertionFailed& e) {
    PyErr_SetString(PyExc_AssertionError, e.what());
  } catch (const BadValue& e) {
    PyErr_SetString(PyExc_ValueError, e.what());
  } catch (const c10::OutOfMemoryError& e) {
    // the type that torch's own allocations raise
    PyObject* torch = PyImport_ImportModule("torch");
    PyObject* type = torch != nullptr ? PyObject_GetAttrString(torch, "OutOfMemoryError") : nullptr;
    PyErr_Clear();
    PyErr_SetString(type != nullptr ? type : PyExc_MemoryError, e.what_without_backtrace());
    Py_XDECREF(type);
    Py_XDECREF(torch);
  } catch (python_error& e) {      // of Python code that torch ran on the way, a saved-tensor hook say
    e.restore();
  } catch (const c10::Error& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what_without_backtrace());
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
  }
  return nullptr;
}

// ---- memory, streams ----------------------------------------------------------------------------------------------
// The tensors' device made current, and its current stream.
struct Call {
  c10::cuda::CUDAGuard guard;
  at::Device device;
  cudaStream_t stream;
  explicit Call(const Tensor& t) : guard(t.device()), device(t.device()), stream(at::cuda::getCurrentCUDAStream(t.device().index())) {}
};

void require_cuda(const Tensor& t) {
  if (!t.is_cuda())
    throw std::runtime_error("dlblas_b200 runs on CUDA tensors only (B200, sm_100a); there is no CPU path");
}

// Every tensor whose memory a kernel reads: a host address would fault the device.
void require_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts) require_cuda(*t);
}

// Weights [experts, n, k] of an FP8 layer and one scale per 128 x 128 block: the kernels take the sizes from here, so a
// tensor of another shape would be read past its end.
void require_fp8_weights(const Tensor& w, const Tensor& w_s, int64_t e, int64_t n, int64_t k) {
  require(w.dim() == 3 && w.size(0) == e && w.size(1) == n && w.size(2) == k && w.element_size() == 1,
          "expert weights must be e4m3 [experts, n, k] with matching sizes");
  require(w_s.numel() == e * ((n + 127) / 128) * (k / 128), "one weight scale per 128 x 128 block");
  require(w.is_contiguous() && w_s.is_contiguous(), "weights and scales must be contiguous");
}

Tensor empty(at::IntArrayRef sizes, at::ScalarType dt, const Call& c) {
  return at::detail::empty_cuda(sizes, dt, c.device, std::nullopt);
}

// Pieces of one allocation, each on a 256-byte boundary.
struct Workspace {
  size_t bytes = 0;
  Tensor mem;
  size_t take(size_t n) {
    const size_t at = bytes;
    bytes += (n + 255) / 256 * 256;
    return at;
  }
  void allocate(const Call& c) { mem = empty({(int64_t)std::max<size_t>(bytes, 1)}, at::kByte, c); }
  template <typename T> T* at(size_t off) const { return reinterpret_cast<T*>(static_cast<char*>(mem.data_ptr()) + off); }
};

int code(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return DLB_F32;
    case at::kBFloat16: return DLB_BF16;
    case at::kHalf: return DLB_F16;
    case at::kInt: return DLB_I32;
    case at::kLong: return DLB_I64;
    default: throw AssertionFailed(std::string("dlblas_b200: unsupported dtype ") + c10::toString(t));
  }
}

// Per-device int32 word that the GEMM kernels set when a bounded wait gives up.
Tensor status_word(at::DeviceIndex index) {
  static std::mutex m;
  static Tensor words[64];
  require(index >= 0 && index < 64, "device index out of range");
  std::lock_guard<std::mutex> lock(m);
  if (!words[index].defined())
    words[index] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::kCUDA, index));
  return words[index];
}
int32_t* status_ptr(const Call& c) { return status_word(c.device.index()).data_ptr<int32_t>(); }

// A setting from the environment.  The text is read with the GIL held, which os.environ's writers hold too, and understood
// where it is wanted.
struct Setting {
  const char* name;
  std::optional<std::string> text;
  explicit Setting(const char* n) : name(n) {
    if (const char* v = std::getenv(n)) text = v;
  }
  // a whole number; text that is none is an error, as Python's int() makes it
  int value(int fallback) const {
    if (!text) return fallback;
    const char* v = text->c_str();
    char* end = nullptr;
    errno = 0;
    const long n = std::strtol(v, &end, 10);
    while (end != v && std::isspace((unsigned char)*end)) ++end;
    if (end == v || *end != 0 || errno != 0 || n < INT_MIN || n > INT_MAX)
      throw BadValue(std::string(name) + " must be a whole number, got '" + *text + "'");
    return (int)n;
  }
};
int tile_rows_of(const Setting& setting, int fallback) {
  const int rows = setting.value(fallback);
  if (rows != 128 && rows != 256) throw AssertionFailed(std::string(setting.name) + " must be 128 or 256");
  return rows;
}

// ---- quantisation and the dense GEMM ------------------------------------------------------------------------------
// 1 x group quantisation of the rows of a 2-D tensor; with dst_pos, row t goes to rows dst_pos[t * fanout + j].
std::pair<Tensor, Tensor> quant_fp8(const Tensor& x, int64_t group, int mode, double eps, bool column_major,
                                    const std::optional<Tensor>& dst_pos, int64_t fanout, int64_t rows_out) {
  require_cuda(x);
  require(x.dim() == 2 && x.stride(1) == 1, "x must be 2-D with contiguous rows");
  const int64_t m = x.size(0), k = x.size(1), rows = rows_out < 0 ? m : rows_out;
  require(group > 0, "group_size must be positive");
  if (dst_pos) {
    require_cuda(*dst_pos);
    require(fanout > 0 && dst_pos->numel() >= m * fanout, "dst_pos must have `fanout` entries per row");
  } else {
    require(rows >= m, "fewer rows wanted than there are");
  }
  if (k % group != 0)
    throw AssertionFailed("the last dimension of 'x' " + std::to_string(k) + " must be divisible by 'group_size' " +
                          std::to_string(group));
  Call c(x);
  Tensor q = empty({rows, k}, at::kFloat8_e4m3fn, c);
  Tensor s = column_major ? empty({k / group, rows}, at::kFloat, c).t() : empty({rows, k / group}, at::kFloat, c);
  check(abi.dlb_quant_fp8(x.data_ptr(), code(x.scalar_type()), m, k, x.stride(0), (int)group, mode, (float)eps, q.data_ptr(),
                          s.data_ptr<float>(), s.stride(0), s.stride(1), dst_pos ? dst_pos->data_ptr<int32_t>() : nullptr,
                          (int)fanout, c.stream));
  return {q, s};
}

PyObject* py_quant_fp8(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 8);
    const Tensor& x = tensor(a[0]);
    const int64_t group = integer(a[1]), mode = integer(a[2]), fanout = integer(a[6]), rows_out = integer(a[7]);
    const double eps = real(a[3]);
    const bool column_major = truth(a[4]);
    const std::optional<Tensor> dst_pos = opt_tensor(a[5]);
    auto [q, s] = without_gil([&] { return quant_fp8(x, group, (int)mode, eps, column_major, dst_pos, fanout, rows_out); });
    return wrap_tuple({&q, &s});
  });
}

// per_token_group_quant_fp8: any leading dimensions
std::pair<Tensor, Tensor> group_quant_fp8(const Tensor& x, int64_t group, double eps, bool column_major) {
  require(x.dim() > 0 && x.stride(-1) == 1, "groups must be contiguous");
  if (x.dim() == 2) return quant_fp8(x, group, DLB_QUANT_DIV_EPS, eps, column_major, std::nullopt, 1, -1);
  require(!column_major, "column-major scales need a 2-D input");
  auto [q, s] = quant_fp8(x.reshape({-1, x.size(-1)}), group, DLB_QUANT_DIV_EPS, eps, false, std::nullopt, 1, -1);
  std::vector<int64_t> shape = x.sizes().vec();
  Tensor qv = q.view(shape);
  shape.back() /= group;
  return {qv, s.view(shape)};
}

PyObject* py_group_quant_fp8(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 4);
    const Tensor& x = tensor(a[0]);
    const int64_t group = integer(a[1]);
    const double eps = real(a[2]);
    const bool column_major = truth(a[3]);
    auto [q, s] = without_gil([&] { return group_quant_fp8(x, group, eps, column_major); });
    return wrap_tuple({&q, &s});
  });
}

Tensor fp8_gemm(const Tensor& a, const Tensor& b, const Tensor& a_s, const Tensor& b_s, at::ScalarType out_dtype,
                int tile_rows, const Setting& fp8_tile_rows) {
  for (const Tensor* t : {&a, &b, &a_s, &b_s}) require_cuda(*t);
  if (tile_rows < 0) tile_rows = fp8_tile_rows.value(0);
  if (out_dtype == at::kFloat) tile_rows = 128;
  require(a.is_contiguous() && b.is_contiguous(), "Input tensors must be contiguous");
  require(a_s.is_contiguous() && b_s.is_contiguous(), "Scaling factor tensors must be contiguous");
  require(a.dim() > 0 && a.size(-1) > 0, "a must have a last dimension of at least 128");
  const int64_t k = a.size(-1), m = a.numel() / k, n = b.size(0), kb = k / 128;
  require(b.numel() == n * k, "b must be [n, k]");
  require(a_s.numel() == m * kb && b_s.numel() == (n + 127) / 128 * kb, "scale shapes do not match a / b");
  Call c(a);
  Tensor out;
  if (a.dim() == 2) {
    out = empty({m, n}, out_dtype, c);
  } else {
    std::vector<int64_t> shape = a.sizes().vec();
    shape.back() = n;
    out = empty(shape, out_dtype, c);
  }
  check(abi.dlb_fp8_gemm(a.data_ptr(), b.data_ptr(), a_s.data_ptr<float>(), kb, 1, b_s.data_ptr<float>(), out.data_ptr(),
                         code(out_dtype), m, n, k, tile_rows, status_ptr(c), c.stream));
  return out;
}

PyObject* py_fp8_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 6);
    const Tensor &x = tensor(a[0]), &w = tensor(a[1]), &x_s = tensor(a[2]), &w_s = tensor(a[3]);
    const at::ScalarType out = dtype(a[4]);
    const int64_t tile_rows = integer(a[5]);
    const Setting fp8_tile_rows("DLBLAS_FP8_TILE_ROWS");
    return wrap(without_gil([&] { return fp8_gemm(x, w, x_s, w_s, out, (int)tile_rows, fp8_tile_rows); }));
  });
}

// ---- routing ------------------------------------------------------------------------------------------------------
std::pair<Tensor, Tensor> route_softmax_topk(const Tensor& logits, int64_t top_k, bool renormalize, at::ScalarType ids_dtype) {
  require_cuda(logits);
  require(logits.dim() == 2 && logits.is_contiguous(), "logits must be a contiguous 2-D tensor");
  Call c(logits);
  const int64_t t = logits.size(0);
  Tensor w = empty({t, top_k}, at::kFloat, c), ids = empty({t, top_k}, ids_dtype, c);
  check(abi.dlb_route_softmax_topk(logits.data_ptr(), code(logits.scalar_type()), t, (int)logits.size(1), (int)top_k,
                                   renormalize, w.data_ptr<float>(), ids.data_ptr(), code(ids_dtype), c.stream));
  return {w, ids};
}

PyObject* py_route_softmax_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 4);
    const Tensor& logits = tensor(a[0]);
    const int64_t top_k = integer(a[1]);
    const bool renormalize = truth(a[2]);
    const at::ScalarType ids_dtype = dtype(a[3]);
    auto [w, ids] = without_gil([&] { return route_softmax_topk(logits, top_k, renormalize, ids_dtype); });
    return wrap_tuple({&w, &ids});
  });
}

std::pair<Tensor, Tensor> route_grouped_topk(const Tensor& given, const Tensor& given_bias, int64_t top_k, bool renormalize,
                                             int64_t groups, int64_t topk_group) {
  require_cuda(given);
  require_cuda(given_bias);
  require(given.dim() == 2, "logits must be 2-D");
  Call c(given);
  const Tensor logits = given.is_contiguous() ? given : given.contiguous();
  Tensor bias = given_bias.scalar_type() == at::kFloat ? given_bias : given_bias.to(at::kFloat);
  if (!bias.is_contiguous()) bias = bias.contiguous();
  const int64_t t = logits.size(0), e = logits.size(1);
  require(bias.numel() == e, "the bias must have one entry per expert");
  Tensor w = empty({t, top_k}, at::kFloat, c), ids = empty({t, top_k}, at::kInt, c);
  check(abi.dlb_route_grouped_topk(logits.data_ptr(), code(logits.scalar_type()), bias.data_ptr<float>(), t, (int)e, (int)groups,
                                   (int)topk_group, (int)top_k, renormalize, w.data_ptr<float>(), ids.data_ptr<int32_t>(),
                                   c.stream));
  return {w, ids};
}

PyObject* py_route_grouped_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 6);
    const Tensor &logits = tensor(a[0]), &bias = tensor(a[1]);
    const int64_t top_k = integer(a[2]), groups = integer(a[4]), topk_group = integer(a[5]);
    const bool renormalize = truth(a[3]);
    auto [w, ids] = without_gil([&] { return route_grouped_topk(logits, bias, top_k, renormalize, groups, topk_group); });
    return wrap_tuple({&w, &ids});
  });
}

// ---- the FP8 expert layer -----------------------------------------------------------------------------------------
// plan -> quantise + permute (or permute) -> w13 GEMM with the silu * up + quantise epilogue -> w2 GEMM scattered back to
// (token, slot) order with the routed weight -> sum over the slots.
struct MoeArgs {
  std::optional<Tensor> hidden, x_q, x_s;   // unquantised rows, or quantised ones with their scales
  Tensor w1, w1_s, w2, w2_s, weights, ids;
  int64_t top_k;
  at::ScalarType out_dtype;
  int64_t expert_offset, num_experts;
  int quant_mode;
  bool skip_unrouted, renormalize, fuse_swiglu;
  Setting fp8_tile_rows{"DLBLAS_FP8_TILE_ROWS"};
};

Tensor moe_forward(const MoeArgs& g) {
  const Tensor& x = g.hidden ? *g.hidden : *g.x_q;
  require_cuda({&x, &g.w1, &g.w1_s, &g.w2, &g.w2_s, &g.weights, &g.ids});
  if (g.x_s) require_cuda(*g.x_s);
  require(g.w1.dim() == 3, "w1 must be [experts, 2 * intermediate, hidden]");
  require(g.ids.scalar_type() == at::kInt || g.ids.scalar_type() == at::kLong, "topk_ids must be int32 or int64");
  require(x.dim() == 2 && x.stride(1) == 1, "x must be 2-D with contiguous rows");
  Call c(x);
  const int64_t e_local = g.w1.size(0), n = g.w1.size(1), h = g.w1.size(2), inter = n / 2;
  const int64_t m = x.size(0), slots = m * g.top_k;
  require_fp8_weights(g.w1, g.w1_s, e_local, n, h);
  require_fp8_weights(g.w2, g.w2_s, e_local, h, inter);
  Tensor out = empty({m, h}, g.out_dtype, c);
  if (m == 0) return out;
  require(x.size(1) == h, "hidden size mismatch");
  require(g.ids.numel() == slots && g.weights.numel() == slots, "topk_ids / topk_weights must be [tokens, top_k]");
  const Tensor ids = g.ids.is_contiguous() ? g.ids : g.ids.contiguous();
  Tensor weights = g.weights;
  bool renormalize = g.renormalize;
  if (weights.scalar_type() != at::kFloat || !weights.is_contiguous()) {
    // in the weights' own type, and in the order that torch adds such a layout up
    if (renormalize) weights = weights / weights.sum(-1, true);
    renormalize = false;
    weights = weights.to(at::kFloat);
  }
  if (!weights.is_contiguous()) weights = weights.contiguous();
  int tile_rows = g.fp8_tile_rows.value(0);
  if (tile_rows == 0 || g.out_dtype == at::kFloat) tile_rows = 128;
  require(tile_rows == 128 || tile_rows == 256, "DLBLAS_FP8_TILE_ROWS must be 0, 128 or 256");
  const bool fused = g.fuse_swiglu && n % 256 == 0;
  const int max_tiles = (int)(slots / tile_rows + e_local);
  const size_t out_size = c10::elementSize(g.out_dtype);
  const size_t sort_bytes = abi.dlb_sort_by_expert_workspace_size(slots, (int)g.num_experts);

  Workspace ws;
  const size_t o_sorted = ws.take(slots * 8), o_pos = ws.take(slots * 4), o_tiles = ws.take((max_tiles + 1) * 16),
               o_w = ws.take(renormalize ? slots * 4 : 0), o_sort = ws.take(sort_bytes), o_a = ws.take(slots * h),
               o_as = ws.take(slots * (h / 128) * 4), o_hq = ws.take(slots * inter), o_hs = ws.take(slots * (inter / 128) * 4),
               o_c1 = ws.take(fused ? 0 : slots * n * out_size), o_y = ws.take(slots * h * out_size);
  ws.allocate(c);
  int64_t* sorted_idx = ws.at<int64_t>(o_sorted);
  int32_t* pos = ws.at<int32_t>(o_pos);
  int32_t* tiles = ws.at<int32_t>(o_tiles);
  int32_t* status = status_ptr(c);
  const float* w = renormalize ? ws.at<float>(o_w) : weights.data_ptr<float>();
  check(abi.dlb_moe_plan(ids.data_ptr(), code(ids.scalar_type()), m, (int)g.top_k, (int)g.num_experts, (int)g.expert_offset,
                         (int)e_local, tile_rows, sorted_idx, pos, tiles, max_tiles,
                         renormalize ? weights.data_ptr<float>() : nullptr, renormalize ? ws.at<float>(o_w) : nullptr,
                         ws.at<void>(o_sort), sort_bytes, c.stream));
  if (g.hidden) {
    check(abi.dlb_quant_fp8(x.data_ptr(), code(x.scalar_type()), m, h, x.stride(0), 128, g.quant_mode, 1e-10f,
                            ws.at<void>(o_a), ws.at<float>(o_as), h / 128, 1, pos, (int)g.top_k, c.stream));
  } else {
    require(x.is_contiguous() && x.element_size() == 1, "quantised rows must be contiguous e4m3");
    const Tensor x_s = g.x_s->is_contiguous() ? *g.x_s : g.x_s->contiguous();
    require(x_s.scalar_type() == at::kFloat && x_s.numel() == m * (h / 128), "scales must be fp32 [tokens, hidden / 128]");
    check(abi.dlb_permute_rows(x.data_ptr(), h, x_s.data_ptr<float>(), h / 128, m, pos, (int)g.top_k, ws.at<void>(o_a),
                               ws.at<float>(o_as), c.stream));
  }
  auto gemm = [&](size_t a, size_t a_s, int64_t nn, int64_t kk, const Tensor& b, const Tensor& b_s, int epilogue, size_t dst,
                  size_t q_scale, int64_t ldc) {
    check(abi.dlb_moe_grouped_gemm(ws.at<void>(a), ws.at<float>(a_s), slots, b.data_ptr(), b_s.data_ptr<float>(), (int)e_local,
                                   nn, kk, tiles, max_tiles, tile_rows, epilogue, ws.at<void>(dst), code(g.out_dtype), ldc,
                                   epilogue == DLB_EPI_SWIGLU_QUANT ? ws.at<float>(q_scale) : nullptr, g.quant_mode, 1e-10f,
                                   epilogue == DLB_EPI_SCATTER_WEIGHT ? sorted_idx : nullptr,
                                   epilogue == DLB_EPI_SCATTER_WEIGHT ? w : nullptr, status, c.stream));
  };
  if (fused) {
    gemm(o_a, o_as, n, h, g.w1, g.w1_s, DLB_EPI_SWIGLU_QUANT, o_hq, o_hs, inter);
  } else {
    gemm(o_a, o_as, n, h, g.w1, g.w1_s, DLB_EPI_STORE, o_c1, 0, n);
    check(abi.dlb_silu_mul_quant(ws.at<void>(o_c1), code(g.out_dtype), slots, inter, g.quant_mode, 1e-10f, 0, nullptr, 0,
                                 ws.at<void>(o_hq), ws.at<float>(o_hs), c.stream));
  }
  gemm(o_hq, o_hs, h, inter, g.w2, g.w2_s, DLB_EPI_SCATTER_WEIGHT, o_y, 0, h);
  check(abi.dlb_moe_sum_topk(ws.at<void>(o_y), code(g.out_dtype), m, (int)g.top_k, h, ids.data_ptr(), code(ids.scalar_type()),
                             g.expert_offset, g.expert_offset + e_local, g.skip_unrouted, out.data_ptr(), c.stream));
  return out;
}

PyObject* py_moe_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 17);
    MoeArgs g{opt_tensor(a[0]), opt_tensor(a[1]), opt_tensor(a[2]), tensor(a[3]), tensor(a[4]), tensor(a[5]), tensor(a[6]),
              tensor(a[7]), tensor(a[8]), integer(a[9]), dtype(a[10]), integer(a[11]), integer(a[12]), (int)integer(a[13]),
              truth(a[14]), truth(a[15]), truth(a[16])};
    return wrap(without_gil([&] { return moe_forward(g); }));
  });
}

// The decode step of FusedMoELowLatency on one rank.  Rounding points of the masked-layout path (w13 rows rounded to
// out_dtype, silu rounded before the product, scales max(absmax, eps) / 448, the weights applied in fp32 in the gather), on the
// rows that exist: with a single rank the exchange is a permutation, so the rows go straight into expert order instead of a
// [experts, max tokens, hidden] layout, and the layer is six launches of which two stream the weights.
Tensor low_latency_forward(const Tensor& x, const Tensor& topk_weights, const Tensor& topk_ids, const Tensor& w1,
                           const Tensor& w1_s, const Tensor& w2, const Tensor& w2_s, at::ScalarType out_dtype,
                           const Setting& sm_margin) {
  require_cuda({&x, &w1, &w1_s, &w2, &w2_s, &topk_weights, &topk_ids});
  require(topk_weights.scalar_type() == at::kFloat, "topk_weights must be fp32");
  require(w1.dim() == 3, "w1 must be [experts, 2 * intermediate, hidden]");
  require(topk_ids.dim() == 2, "topk_ids must be [tokens, top_k]");
  require(x.dim() == 2 && x.stride(1) == 1, "hidden states must be 2-D with contiguous rows");
  Call c(x);
  const int64_t e = w1.size(0), n = w1.size(1), h = w1.size(2), inter = n / 2;
  const int64_t m = x.size(0), top_k = topk_ids.size(1), slots = m * top_k;
  require(x.size(1) == h, "hidden size mismatch");
  require(topk_ids.size(0) == m && topk_weights.numel() == slots, "topk_ids / topk_weights must be [tokens, top_k]");
  require_fp8_weights(w1, w1_s, e, n, h);
  require_fp8_weights(w2, w2_s, e, h, inter);
  Tensor out = empty({m, h}, out_dtype, c);
  if (m == 0) return out;
  Tensor ids = topk_ids.scalar_type() == at::kInt || topk_ids.scalar_type() == at::kLong ? topk_ids : topk_ids.to(at::kLong);
  if (!ids.is_contiguous()) ids = ids.contiguous();
  const Tensor weights = topk_weights.is_contiguous() ? topk_weights : topk_weights.contiguous();
  const int max_tiles = (int)(slots / 128 + e);
  const size_t size = c10::elementSize(out_dtype);
  const size_t sort_bytes = abi.dlb_sort_by_expert_workspace_size(slots, (int)e);
  Workspace ws;
  const size_t o_pos = ws.take(slots * 4), o_tiles = ws.take((max_tiles + 1) * 16), o_sort = ws.take(sort_bytes),
               o_a = ws.take(slots * h), o_as = ws.take(slots * (h / 128) * 4), o_c1 = ws.take(slots * n * size),
               o_hq = ws.take(slots * inter), o_hs = ws.take(slots * (inter / 128) * 4), o_y = ws.take(slots * h * size);
  ws.allocate(c);
  int32_t *pos = ws.at<int32_t>(o_pos), *tiles = ws.at<int32_t>(o_tiles), *status = status_ptr(c);
  check(abi.dlb_moe_plan(ids.data_ptr(), code(ids.scalar_type()), m, (int)top_k, (int)e, 0, (int)e, 128, nullptr, pos, tiles,
                         max_tiles, nullptr, nullptr, ws.at<void>(o_sort), sort_bytes, c.stream));
  check(abi.dlb_quant_fp8(x.data_ptr(), code(x.scalar_type()), m, h, x.stride(0), 128, DLB_QUANT_DIV_EPS, 1e-10f,
                          ws.at<void>(o_a), ws.at<float>(o_as), h / 128, 1, pos, (int)top_k, c.stream));
  // SMs left to kernels of other streams (a shared expert's small GEMMs): the weights stream at the memory rate from fewer
  const int margin = sm_margin.value(0);
  auto gemm = [&](size_t a, size_t a_s, int64_t nn, int64_t kk, const Tensor& b, const Tensor& b_s, size_t dst) {
    check(abi.dlb_moe_grouped_gemm_window(ws.at<void>(a), ws.at<float>(a_s), slots, b.data_ptr(), b_s.data_ptr<float>(),
                                          (int)e, nn, kk, tiles, max_tiles, 128, DLB_EPI_STORE, ws.at<void>(dst),
                                          code(out_dtype), nn, nullptr, DLB_QUANT_RECIP_MUL, 1e-10f, nullptr, nullptr, status,
                                          c.stream, 0, nn, margin));
  };
  gemm(o_a, o_as, n, h, w1, w1_s, o_c1);
  check(abi.dlb_silu_mul_quant(ws.at<void>(o_c1), code(out_dtype), slots, inter, DLB_QUANT_DIV_EPS, 1e-10f, 1, nullptr, 0,
                               ws.at<void>(o_hq), ws.at<float>(o_hs), c.stream));
  gemm(o_hq, o_hs, h, inter, w2, w2_s, o_y);
  check(abi.dlb_ep_gather(ws.at<void>(o_y), code(out_dtype), h, pos, pos, DLB_I32, weights.data_ptr<float>(), m, (int)top_k,
                          out.data_ptr(), c.stream));
  return out;
}

PyObject* py_low_latency_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 8);
    const Tensor &x = tensor(a[0]), &weights = tensor(a[1]), &ids = tensor(a[2]), &w1 = tensor(a[3]), &w1_s = tensor(a[4]),
                 &w2 = tensor(a[5]), &w2_s = tensor(a[6]);
    const at::ScalarType out = dtype(a[7]);
    const Setting sm_margin("DLBLAS_DECODE_SM_MARGIN");
    return wrap(without_gil([&] { return low_latency_forward(x, weights, ids, w1, w1_s, w2, w2_s, out, sm_margin); }));
  });
}

// ---- 16-bit grouped GEMMs and the unquantised expert layer --------------------------------------------------------
// pairs of CTAs on 256-row tiles when the groups are large enough to fill them (decided from the shapes, no look at the
// group sizes on the host); DLBLAS_GEMM16_TILE_ROWS = 128 / 256 overrides
struct Gemm16Rows : Setting {
  Gemm16Rows() : Setting("DLBLAS_GEMM16_TILE_ROWS") {}
};
int gemm16_tile_rows(const Gemm16Rows& setting, int64_t rows, int64_t groups) {
  return tile_rows_of(setting, rows >= 512 * groups ? 256 : 128);
}

Tensor group_sizes(const Tensor& sizes) {
  Tensor s = sizes.scalar_type() == at::kInt || sizes.scalar_type() == at::kLong ? sizes : sizes.to(at::kLong);
  return s.is_contiguous() ? s : s.contiguous();
}

Tensor m_grouped_gemm(const Tensor& a_in, const Tensor& b_in, const Tensor& sizes_in, bool trans_b, const Gemm16Rows& setting) {
  require(a_in.dim() == 2, "A must be 2-D");
  require(b_in.dim() == 3, "B must be 3-D");
  for (const Tensor* t : {&a_in, &b_in, &sizes_in}) require_cuda(*t);
  require(a_in.stride(1) == 1, "Please make sure A is K-major");
  require(a_in.scalar_type() == b_in.scalar_type() &&
              (a_in.scalar_type() == at::kBFloat16 || a_in.scalar_type() == at::kHalf),
          "A and B must both be bf16 or fp16");
  Call c(a_in);
  const int64_t m = a_in.size(0), k = a_in.size(1), groups = b_in.size(0);
  const int64_t n = trans_b ? b_in.size(1) : b_in.size(2), bk = trans_b ? b_in.size(2) : b_in.size(1);
  require(bk == k, "K of A should be equal to K of B");
  require(sizes_in.numel() == groups, "one size per group");
  const bool b_kn = !trans_b && k % 64 == 0;
  const Tensor a = a_in.is_contiguous() ? a_in : a_in.contiguous();
  Tensor b = trans_b || b_kn ? b_in : b_in.transpose(1, 2);
  if (!b.is_contiguous()) b = b.contiguous();
  Tensor out = empty({m, n}, a.scalar_type(), c);
  if (m == 0) return out;
  const Tensor sizes = group_sizes(sizes_in);
  const int tile_rows = gemm16_tile_rows(setting, m, groups);
  const int max_tiles = (int)(m / tile_rows + groups);
  Workspace ws;
  ws.take((size_t)(max_tiles + 1) * 16);
  ws.allocate(c);
  int32_t* tiles = ws.at<int32_t>(0);
  check(abi.dlb_moe_build_tiles_sizes(sizes.data_ptr(), code(sizes.scalar_type()), (int)groups, m, tile_rows, tiles, max_tiles,
                                      c.stream));
  auto gemm = b_kn ? abi.dlb_grouped_gemm_16bit_b_kn : abi.dlb_grouped_gemm_16bit;
  check(gemm(a.data_ptr(), b.data_ptr(), code(a.scalar_type()), m, (int)groups, n, k, tiles, max_tiles, tile_rows,
             out.data_ptr(), n, status_ptr(c), c.stream));
  return out;
}

PyObject* py_m_grouped_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 4);
    const Tensor &x = tensor(a[0]), &w = tensor(a[1]), &sizes = tensor(a[2]);
    const bool trans_b = truth(a[3]);
    const Gemm16Rows setting;
    return wrap(without_gil([&] { return m_grouped_gemm(x, w, sizes, trans_b, setting); }));
  });
}

Tensor k_grouped_gemm(const Tensor& a_in, const Tensor& b_in, const Tensor& sizes_in, const Gemm16Rows& setting) {
  require(a_in.dim() == 2, "A must be 2-D");
  require(b_in.dim() == 2, "B must be 2-D");
  for (const Tensor* t : {&a_in, &b_in, &sizes_in}) require_cuda(*t);
  require(a_in.stride(1) == 1, "Please make sure A is K-major");
  require(b_in.stride(1) == 1, "Please make sure B is K-major");
  require(a_in.size(0) == b_in.size(0), "Please make sure that A and B have the same seqlen");
  if (a_in.scalar_type() != b_in.scalar_type() || (a_in.scalar_type() != at::kBFloat16 && a_in.scalar_type() != at::kHalf))
    throw AssertionFailed(std::string("data type ") + c10::toString(a_in.scalar_type()) + " not supported");
  Call c(a_in);
  const Tensor a = a_in.is_contiguous() ? a_in : a_in.contiguous(), b = b_in.is_contiguous() ? b_in : b_in.contiguous();
  const int64_t k = a.size(0), m = a.size(1), n = b.size(1), groups = sizes_in.size(0);
  Tensor out = empty({groups, m, n}, a.scalar_type(), c);
  if (groups == 0 || m == 0 || n == 0) return out;
  Tensor sizes = group_sizes(sizes_in);
  if (sizes.scalar_type() != at::kLong) sizes = sizes.to(at::kLong);
  // pairs of CTAs on 256-row tiles of C unless M is smaller than one; DLBLAS_GEMM16_TILE_ROWS = 128 / 256 overrides
  const int tile_rows = tile_rows_of(setting, m >= 256 ? 256 : 128);
  const int64_t need = abi.dlb_k_grouped_gemm_workspace_bytes(k, m, n, (int)groups, tile_rows);
  require(need > 0, "k_grouped_gemm: bad sizes");
  const Tensor work = empty({need}, at::kByte, c);
  check(abi.dlb_k_grouped_gemm_16bit(a.data_ptr(), b.data_ptr(), code(a.scalar_type()), k, m, n, sizes.data_ptr<int64_t>(),
                                     (int)groups, tile_rows, work.data_ptr(), need, out.data_ptr(), status_ptr(c), c.stream));
  return out;
}

PyObject* py_k_grouped_gemm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 3);
    const Tensor &x = tensor(a[0]), &y = tensor(a[1]), &sizes = tensor(a[2]);
    const Gemm16Rows setting;
    return wrap(without_gil([&] { return k_grouped_gemm(x, y, sizes, setting); }));
  });
}

// rows copied into expert order -> w1 GEMM -> silu(gate) * up -> w2 GEMM -> fp32 weighted sum over the slots
Tensor moe_forward_16bit(const Tensor& x, const Tensor& w1_in, const Tensor& w2_in, const Tensor& weights_in,
                         const Tensor& ids_in, const Gemm16Rows& setting) {
  require(x.scalar_type() == at::kBFloat16 || x.scalar_type() == at::kHalf,
          "the unquantised mode takes bf16 or fp16 activations");
  require(w1_in.scalar_type() == x.scalar_type() && w2_in.scalar_type() == x.scalar_type(),
          "weights must have the activations' type");
  require_cuda({&x, &w1_in, &w2_in, &weights_in, &ids_in});
  require(x.dim() == 2 && x.is_contiguous(), "activations must be contiguous [tokens, hidden]");
  require(w1_in.dim() == 3 && w1_in.size(2) == x.size(1), "w1 must be [E, 2 I, H]");
  require(ids_in.dim() == 2 && ids_in.size(0) == x.size(0) && weights_in.numel() == ids_in.numel(),
          "topk_ids / topk_weights must be [tokens, top_k]");
  Call c(x);
  const int64_t m = x.size(0), h = x.size(1), e = w1_in.size(0), n2 = w1_in.size(1), inter = n2 / 2;
  require(w2_in.dim() == 3 && w2_in.size(0) == e && w2_in.size(1) == h && w2_in.size(2) == inter, "w2 must be [E, H, I]");
  Tensor out = empty({m, h}, x.scalar_type(), c);
  if (m == 0) return out;
  const int64_t top_k = ids_in.size(1), slots = m * top_k;
  require(ids_in.scalar_type() == at::kInt || ids_in.scalar_type() == at::kLong, "topk_ids must be int32 or int64");
  const Tensor ids = ids_in.is_contiguous() ? ids_in : ids_in.contiguous();
  const Tensor w1 = w1_in.is_contiguous() ? w1_in : w1_in.contiguous(), w2 = w2_in.is_contiguous() ? w2_in : w2_in.contiguous();
  Tensor weights = weights_in.scalar_type() == at::kFloat ? weights_in : weights_in.to(at::kFloat);
  if (!weights.is_contiguous()) weights = weights.contiguous();
  const int tile_rows = gemm16_tile_rows(setting, slots, e), max_tiles = (int)(slots / tile_rows + e), dt = code(x.scalar_type());
  const size_t sort_bytes = abi.dlb_sort_by_expert_workspace_size(slots, (int)e);
  Workspace ws;
  const size_t o_pos = ws.take(slots * 4), o_tiles = ws.take((max_tiles + 1) * 16), o_sort = ws.take(sort_bytes),
               o_a = ws.take(slots * h * 2), o_c1 = ws.take(slots * n2 * 2), o_act = ws.take(slots * inter * 2),
               o_y = ws.take(slots * h * 2);
  ws.allocate(c);
  int32_t *pos = ws.at<int32_t>(o_pos), *tiles = ws.at<int32_t>(o_tiles), *status = status_ptr(c);
  check(abi.dlb_moe_plan(ids.data_ptr(), code(ids.scalar_type()), m, (int)top_k, (int)e, 0, (int)e, tile_rows, nullptr, pos,
                         tiles, max_tiles, nullptr, nullptr, ws.at<void>(o_sort), sort_bytes, c.stream));
  check(abi.dlb_permute_rows(x.data_ptr(), 2 * h, nullptr, 0, m, pos, (int)top_k, ws.at<void>(o_a), nullptr, c.stream));
  check(abi.dlb_grouped_gemm_16bit(ws.at<void>(o_a), w1.data_ptr(), dt, slots, (int)e, n2, h, tiles, max_tiles, tile_rows,
                                   ws.at<void>(o_c1), n2, status, c.stream));
  check(abi.dlb_silu_and_mul(ws.at<void>(o_c1), dt, slots, inter, n2, ws.at<void>(o_act), inter, c.stream));
  check(abi.dlb_grouped_gemm_16bit(ws.at<void>(o_act), w2.data_ptr(), dt, slots, (int)e, h, inter, tiles, max_tiles, tile_rows,
                                   ws.at<void>(o_y), h, status, c.stream));
  // slots of other ranks' experts have a negative position and are left out of the sum
  check(abi.dlb_ep_gather(ws.at<void>(o_y), dt, h, pos, pos, DLB_I32, weights.data_ptr<float>(), m, (int)top_k, out.data_ptr(),
                          c.stream));
  return out;
}

PyObject* py_moe_forward_16bit(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 5);
    const Tensor &x = tensor(a[0]), &w1 = tensor(a[1]), &w2 = tensor(a[2]), &weights = tensor(a[3]), &ids = tensor(a[4]);
    const Gemm16Rows setting;
    return wrap(without_gil([&] { return moe_forward_16bit(x, w1, w2, weights, ids, setting); }));
  });
}

// ---- block-aligned token layout -----------------------------------------------------------------------------------
std::array<Tensor, 3> moe_align_block_size(Tensor given, int64_t block, int64_t experts, int64_t local,
                                           const std::optional<Tensor>& expert_map, bool pad) {
  require_cuda(given);
  require(given.scalar_type() == at::kInt || given.scalar_type() == at::kLong, "topk_ids must be int32 or int64");
  require(block > 0 && experts > 0, "block_size and num_experts must be positive");
  Call c(given);
  Tensor ids = given.is_contiguous() ? given : given.contiguous();
  const int64_t slots = ids.numel();
  int64_t padded = slots + experts * (block - 1);
  if (pad) padded = (padded + block - 1) / block * block;
  const int64_t blocks = (padded + block - 1) / block;
  Tensor sorted = empty({padded}, at::kInt, c), owner = empty({blocks}, at::kInt, c), total = empty({1}, at::kInt, c);
  const size_t sort_bytes = abi.dlb_sort_by_expert_workspace_size(slots, (int)experts);
  Workspace ws;
  ws.take(sort_bytes);
  ws.allocate(c);
  check(abi.dlb_moe_align_block_size(ids.data_ptr(), code(ids.scalar_type()), slots, (int)experts, (int)local, (int)block,
                                     sorted.data_ptr<int32_t>(), padded, owner.data_ptr<int32_t>(), (int)blocks,
                                     total.data_ptr<int32_t>(), ws.at<void>(0), sort_bytes, c.stream));
  if (!ids.is_same(given)) given.copy_(ids);      // negative ids are replaced in the caller's tensor
  if (expert_map) owner = expert_map->index({owner.to(at::kLong)});
  return {sorted, owner, total};
}

PyObject* py_moe_align_block_size(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 6);
    const Tensor& ids = tensor(a[0]);
    const int64_t block = integer(a[1]), experts = integer(a[2]), local = integer(a[3]);
    const std::optional<Tensor> expert_map = opt_tensor(a[4]);
    const bool pad = truth(a[5]);
    auto [sorted, owner, total] = without_gil([&] { return moe_align_block_size(ids, block, experts, local, expert_map, pad); });
    return wrap_tuple({&sorted, &owner, &total});
  });
}

// ---- capacity-limited gating --------------------------------------------------------------------------------------
// ceil(T / E * capacity_factor), at least min_capacity, from the single-precision product that the reference forms.  A product
// that is no whole number of slots is an error, as it is for Python's math.ceil.  Needs the GIL.
int64_t gating_capacity(int64_t tokens, int64_t experts, double factor, int64_t min_capacity) {
  require(experts > 0, "logits must have at least one expert");
  const float per_expert = (float)((double)tokens / (double)experts), f = (float)factor;
  const double slots = std::ceil(per_expert * f);
  if (std::isnan(slots) || std::isinf(slots) || slots >= 0x1p63) {
    PyErr_Format(std::isnan(slots) ? PyExc_ValueError : PyExc_OverflowError, "topk_gating: the capacity is not a whole number");
    throw PyFailed{};
  }
  return std::max<int64_t>((int64_t)std::max(slots, -0x1p62), min_capacity);
}

// int(o): a least capacity may be given as a float
int64_t truncated(PyObject* o) {
  PyObject* whole = PyNumber_Long(o);
  if (whole == nullptr) throw PyFailed{};
  const long long v = PyLong_AsLongLong(whole);
  Py_DECREF(whole);
  if (v == -1 && PyErr_Occurred()) throw PyFailed{};
  return v;
}

PyObject* py_gating_capacity(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 4);
    return PyLong_FromLongLong(gating_capacity(integer(a[0]), integer(a[1]), real(a[2]), truncated(a[3])));
  });
}

struct Gating {
  Tensor l_aux, ec_idx, weights, select, ws;
};
Gating gating_forward(const Tensor& given, int64_t k, int64_t capacity) {
  require_cuda(given);
  require(given.dim() == 2, "logits must be 2-D");
  Call c(given);
  const Tensor logits = given.is_contiguous() ? given : given.contiguous();
  const int64_t t = logits.size(0), e = logits.size(1);
  const size_t bytes = abi.dlb_topk_gating_workspace_size(t, (int)e, (int)k);
  Gating g{empty({}, logits.scalar_type(), c), empty({k * t}, at::kInt, c), empty({k * t}, logits.scalar_type(), c),
           empty({e * capacity}, at::kLong, c), empty({(int64_t)std::max<size_t>(bytes, 1)}, at::kByte, c)};
  check(abi.dlb_topk_gating(logits.data_ptr(), code(logits.scalar_type()), t, (int)e, (int)k, capacity, g.l_aux.data_ptr(),
                            g.ec_idx.data_ptr<int32_t>(), g.weights.data_ptr(), g.select.data_ptr<int64_t>(),
                            g.ws.data_ptr(), bytes, c.stream));
  return g;
}

Tensor gating_backward(const Tensor& ws, at::ScalarType dt, int64_t tokens, int64_t experts, int64_t k, int64_t capacity,
                       const Tensor& grad_l_aux, const Tensor& grad_weights) {
  require_cuda(ws);
  Call c(ws);
  auto ready = [&](const Tensor& g) {
    Tensor r = g.scalar_type() == dt ? g : g.to(dt);
    return r.is_contiguous() ? r : r.contiguous();
  };
  const Tensor gl = grad_l_aux.defined() ? ready(grad_l_aux) : at::zeros({}, ws.options().dtype(dt));
  const Tensor gw = grad_weights.defined() ? ready(grad_weights) : Tensor();
  require(gl.numel() >= 1 && (!gw.defined() || gw.numel() >= tokens * k), "gradients smaller than the outputs they belong to");
  Tensor out = empty({tokens, experts}, dt, c);
  check(abi.dlb_topk_gating_bwd(ws.data_ptr(), ws.numel(), code(dt), tokens, (int)experts, (int)k, capacity, gl.data_ptr(),
                                gw.defined() ? gw.data_ptr() : nullptr, out.data_ptr(), c.stream));
  return out;
}

// dlblas/kernels/topk_gating.py:245-285.  The backward differentiates the auxiliary loss (topk_gating_bwd.py:13-68) and,
// with `higher_precision`, the weights too.
struct GatingFunction : torch::autograd::Function<GatingFunction> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& logits, int64_t k,
                                                int64_t capacity, bool higher_precision) {
    Gating g = gating_forward(logits, k, capacity);
    ctx->set_materialize_grads(false);
    ctx->saved_data["k"] = k;
    ctx->saved_data["capacity"] = capacity;
    ctx->saved_data["hp"] = higher_precision;
    ctx->saved_data["t"] = logits.size(0);
    ctx->saved_data["e"] = logits.size(1);
    ctx->saved_data["dtype"] = (int64_t)logits.scalar_type();
    ctx->save_for_backward({g.ws});
    ctx->mark_non_differentiable({g.ec_idx, g.select});
    return {g.l_aux, g.ec_idx, g.weights, g.select};
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    auto& s = ctx->saved_data;
    const Tensor ws = ctx->get_saved_variables()[0];
    return {gating_backward(ws, (at::ScalarType)s["dtype"].toInt(), s["t"].toInt(), s["e"].toInt(), s["k"].toInt(),
                            s["capacity"].toInt(), grads[0], s["hp"].toBool() ? grads[2] : Tensor()),
            Tensor(), Tensor(), Tensor()};
  }
};

// (logits, k, capacity, with workspace) -> (l_aux, ec_idx, weights, select[, workspace])
PyObject* py_gating_forward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 4);
    const Tensor& logits = tensor(a[0]);
    const int64_t k = integer(a[1]), capacity = integer(a[2]);
    Gating g = without_gil([&] { return gating_forward(logits, k, capacity); });
    return truth(a[3]) ? wrap_tuple({&g.l_aux, &g.ec_idx, &g.weights, &g.select, &g.ws})
                       : wrap_tuple({&g.l_aux, &g.ec_idx, &g.weights, &g.select});
  });
}

PyObject* py_gating_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 8);
    const std::optional<Tensor> gw = opt_tensor(a[7]);
    const Tensor &ws = tensor(a[0]), &gl = tensor(a[6]);
    const at::ScalarType dt = dtype(a[1]);
    const int64_t tokens = integer(a[2]), experts = integer(a[3]), k = integer(a[4]), capacity = integer(a[5]);
    return wrap(without_gil([&] { return gating_backward(ws, dt, tokens, experts, k, capacity, gl, gw ? *gw : Tensor()); }));
  });
}

// (logits, k, capacity_factor, min_capacity, higher_precision): differentiable in the logits
PyObject* py_topk_gating(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 5);
    const Tensor& logits = tensor(a[0]);
    const int64_t k = integer(a[1]);
    require(logits.dim() == 2, "logits must be 2-D");
    const int64_t capacity = gating_capacity(logits.size(0), logits.size(1), real(a[2]) * (double)k, truncated(a[3]));
    if (logits.requires_grad() && at::GradMode::is_enabled()) {
      const bool higher_precision = truth(a[4]);
      auto r = without_gil([&] { return GatingFunction::apply(logits, k, capacity, higher_precision); });
      return wrap_tuple({&r[0], &r[1], &r[2], &r[3]});
    }
    Gating g = without_gil([&] { return gating_forward(logits, k, capacity); });
    return wrap_tuple({&g.l_aux, &g.ec_idx, &g.weights, &g.select});
  });
}

// ---- training-side permutation (dlblas/kernels/permute/moe_triton_kernels.py) -------------------------------------
// Ids below this bound are sorted without a look at them on the host.
constexpr int PERMUTE_EXPERTS = 1024;

struct PermutePlan {
  Tensor sorted_idx, dest, row_map;   // sorted flat slots; row of every slot; the same, top_k-major
  int64_t minus_one = 0, negative = 0;
};

// The output of a permutation has as many rows as slots are routed, so one value has to reach the host.  The kernel that
// counts the ids hands their statistics over in pinned memory behind an event; the placement of the rows is queued before
// the host waits for that event, so the GPU works while the host looks.
PermutePlan permute_plan(const Tensor& indices, int64_t dest_limit, bool want_sorted) {
  require_cuda(indices);
  require(indices.dim() == 2, "indices must be [tokens, top_k]");
  require(indices.scalar_type() == at::kInt || indices.scalar_type() == at::kLong, "topk_ids must be int32 or int64");
  Call c(indices);
  const Tensor ids = indices.is_contiguous() ? indices : indices.contiguous();
  const int64_t t = ids.size(0), k = ids.size(1), slots = t * k;
  PermutePlan p;
  if (want_sorted) p.sorted_idx = empty({slots}, at::kLong, c);
  p.dest = empty({slots}, at::kInt, c);
  p.row_map = empty({slots}, at::kInt, c);
  if (t == 0) return p;      // nothing to place
  // one event and twelve bytes per thread and device: both are used up before this function returns
  thread_local at::cuda::CUDAEvent events[16];
  thread_local Tensor stats_mem[16];
  const int dev = c.device.index();
  require(dev < 16, "device index out of range");
  if (!stats_mem[dev].defined()) {
    stats_mem[dev] = at::empty({4}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
    events[dev].record(at::cuda::getCurrentCUDAStream(c.device.index()));   // creates the event
  }
  int32_t* stats = stats_mem[dev].data_ptr<int32_t>();
  auto plan = [&](int64_t experts, bool with_stats) {
    const size_t bytes = abi.dlb_sort_by_expert_workspace_size(slots, (int)experts);
    Workspace ws;
    ws.take(bytes);
    ws.allocate(c);
    check(abi.dlb_permute_plan(ids.data_ptr(), code(ids.scalar_type()), t, (int)k, (int)experts, dest_limit,
                               want_sorted ? p.sorted_idx.data_ptr<int64_t>() : nullptr, p.dest.data_ptr<int32_t>(),
                               p.row_map.data_ptr<int32_t>(), with_stats ? stats : nullptr,
                               with_stats ? (void*)events[dev].event() : nullptr, ws.at<void>(0), bytes, c.stream));
  };
  plan(PERMUTE_EXPERTS, true);
  const cudaError_t waited = cudaEventSynchronize(events[dev].event());
  if (waited != cudaSuccess) throw std::runtime_error(std::string("permute: ") + cudaGetErrorString(waited));
  const int64_t largest = stats[0];
  p.minus_one = stats[1];
  p.negative = stats[2];
  if (largest >= PERMUTE_EXPERTS) plan(largest + 1, false);
  return p;
}

// Copies the rows of x to their places in `out`; rows that no slot fills become zero.
void permute_rows(const Tensor& x, const PermutePlan& p, int64_t k, const Tensor& out) {
  Call c(x);
  const int64_t t = x.size(0), routed = t * k - p.negative, row_bytes = x.size(1) * x.element_size();
  if (out.size(0) > routed) out.narrow(0, routed, out.size(0) - routed).zero_();
  check(abi.dlb_permute_rows(x.data_ptr(), row_bytes, nullptr, 0, t, p.dest.data_ptr<int32_t>(), (int)k, out.data_ptr(),
                             nullptr, c.stream));
}

// moe_permute_topk_op_triton: (indices, rows wanted) -> (sorted_idx, dest, row_id_map, ids equal to -1, ids below 0)
PyObject* py_permute_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 2);
    const Tensor& indices = tensor(a[0]);
    const int64_t dest_limit = integer(a[1]);
    PermutePlan p = without_gil([&] { return permute_plan(indices, dest_limit, true); });
    return Py_BuildValue("(NNNLL)", wrap(p.sorted_idx), wrap(p.dest), wrap(p.row_map), (long long)p.minus_one,
                         (long long)p.negative);
  });
}

Tensor unpermute_rows(const Tensor& x_in, const Tensor& row_map_in, const Tensor& probs_in, int64_t tokens, int64_t k) {
  require_cuda({&x_in, &row_map_in});
  if (probs_in.defined()) require_cuda(probs_in);
  require(row_map_in.numel() >= tokens * k, "the row map must have an entry for every token and slot");
  require(!probs_in.defined() || probs_in.numel() >= tokens * k, "one probability per token and slot");
  Call c(x_in);
  const Tensor x = x_in.is_contiguous() ? x_in : x_in.contiguous();
  const Tensor row_map = row_map_in.is_contiguous() ? row_map_in : row_map_in.contiguous();
  Tensor probs;
  if (probs_in.defined()) {
    probs = probs_in.scalar_type() == at::kFloat ? probs_in : probs_in.to(at::kFloat);
    if (!probs.is_contiguous()) probs = probs.contiguous();
  }
  Tensor out = empty({tokens, x.size(1)}, x.scalar_type(), c);
  check(abi.dlb_unpermute(x.data_ptr(), code(x.scalar_type()), row_map.data_ptr<int32_t>(),
                          probs.defined() ? probs.data_ptr<float>() : nullptr, tokens, (int)k, x.size(1), out.data_ptr(),
                          c.stream));
  return out;
}

PyObject* py_unpermute_rows(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 5);
    const std::optional<Tensor> probs = opt_tensor(a[2]);
    const Tensor &x = tensor(a[0]), &row_map = tensor(a[1]);
    const int64_t tokens = integer(a[3]), k = integer(a[4]);
    return wrap(without_gil([&] { return unpermute_rows(x, row_map, probs ? *probs : Tensor(), tokens, k); }));
  });
}

// (gradient of the rows in act_dtype, gradient of the probabilities in fp32)
std::pair<Tensor, Tensor> unpermute_backward(const Tensor& grad_in, const Tensor& fwd_in, const Tensor& row_map_in,
                                             const Tensor& probs_in, at::ScalarType act_dtype) {
  require_cuda({&grad_in, &fwd_in, &row_map_in, &probs_in});
  Call c(grad_in);
  require(grad_in.scalar_type() == fwd_in.scalar_type(), "gradient and rows must have one type");
  require(probs_in.dim() == 2 && grad_in.dim() == 2 && fwd_in.dim() == 2, "gradient, rows and probabilities must be 2-D");
  require(grad_in.size(0) >= probs_in.size(0) && grad_in.size(1) == fwd_in.size(1), "gradient and rows do not fit together");
  require(row_map_in.numel() >= probs_in.numel(), "the row map must have an entry for every token and slot");
  const int64_t t = probs_in.size(0), k = probs_in.size(1), h = grad_in.size(1), rows = fwd_in.size(0);
  const Tensor grad = grad_in.is_contiguous() ? grad_in : grad_in.contiguous();
  const Tensor fwd = fwd_in.is_contiguous() ? fwd_in : fwd_in.contiguous();
  const Tensor row_map = row_map_in.is_contiguous() ? row_map_in : row_map_in.contiguous();
  Tensor probs = probs_in.scalar_type() == at::kFloat ? probs_in : probs_in.to(at::kFloat);
  if (!probs.is_contiguous()) probs = probs.contiguous();
  Tensor act = empty({rows, fwd.size(1)}, act_dtype, c), prob_grad = empty({t, k}, at::kFloat, c);
  Workspace ws;
  ws.take(rows);
  ws.allocate(c);
  check(abi.dlb_unpermute_bwd_rows(grad.data_ptr(), fwd.data_ptr(), code(grad.scalar_type()), row_map.data_ptr<int32_t>(),
                                   probs.data_ptr<float>(), t, (int)k, h, rows, act.data_ptr(), code(act_dtype),
                                   prob_grad.data_ptr<float>(), ws.at<void>(0), c.stream));
  return {act, prob_grad};
}

PyObject* py_unpermute_backward(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 5);
    const Tensor &grad = tensor(a[0]), &fwd = tensor(a[1]), &row_map = tensor(a[2]), &probs = tensor(a[3]);
    const at::ScalarType act_dtype = dtype(a[4]);
    auto [act, prob] = without_gil([&] { return unpermute_backward(grad, fwd, row_map, probs, act_dtype); });
    return wrap_tuple({&act, &prob});
  });
}

struct PermuteFunction : torch::autograd::Function<PermuteFunction> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& x_in,
                                                const Tensor& indices) {
    const Tensor x = x_in.is_contiguous() ? x_in : x_in.contiguous();
    const int64_t t = x.size(0), k = indices.size(1);
    PermutePlan p = permute_plan(indices, t * k, false);
    Call c(x);
    Tensor out = empty({t * k - p.minus_one, x.size(1)}, x.scalar_type(), c);
    permute_rows(x, p, k, out);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({p.row_map});
    ctx->saved_data["t"] = t;
    ctx->saved_data["k"] = k;
    ctx->saved_data["h"] = x.size(1);
    ctx->saved_data["dtype"] = (int64_t)x.scalar_type();
    ctx->mark_non_differentiable({p.row_map});
    return {out, p.row_map};
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    auto& s = ctx->saved_data;
    const Tensor row_map = ctx->get_saved_variables()[0];
    if (!grads[0].defined())       // the rows' consumer has no gradient for them; zeros for the row map are not wanted
      return {at::zeros({s["t"].toInt(), s["h"].toInt()}, row_map.options().dtype((at::ScalarType)s["dtype"].toInt())), Tensor()};
    if (grads[0].numel() == 0) return {grads[0], Tensor()};
    return {unpermute_rows(grads[0], row_map, Tensor(), s["t"].toInt(), s["k"].toInt()), Tensor()};
  }
};

PyObject* py_permute(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    need_args(n, 2);
    const Tensor& x = tensor(a[0]);
    Tensor indices = tensor(a[1]);
    if (x.numel() == 0) return Py_BuildValue("(NO)", wrap(x), Py_None);
    if (indices.dim() == 1) indices = indices.view({-1, 1});
    if (!x.is_cuda() || !indices.is_cuda()) throw std::runtime_error("permute needs CUDA tensors");
    if (x.size(0) != indices.size(0))
      throw std::runtime_error("token count mismatch: " + std::to_string(x.size(0)) + " vs " + std::to_string(indices.size(0)));
    auto r = without_gil([&] { return PermuteFunction::apply(x, indices); });
    return wrap_tuple({&r[0], &r[1]});
  });
}

struct UnpermuteFunction : torch::autograd::Function<UnpermuteFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& row_map,
                        const std::optional<Tensor>& probs) {
    const int64_t t = probs ? probs->size(0) : row_map.numel(), k = probs ? probs->size(1) : 1;
    ctx->save_for_backward({x, row_map, probs ? *probs : Tensor()});
    ctx->saved_data["with_probs"] = probs.has_value();
    return unpermute_rows(x, row_map, probs ? *probs : Tensor(), t, k);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &row_map = saved[1];
    if (!ctx->saved_data["with_probs"].toBool()) {
      const Tensor ones = at::ones({row_map.numel(), 1}, row_map.options().dtype(at::kFloat));
      return {unpermute_backward(grads[0], x, row_map, ones, x.scalar_type()).first, Tensor(), Tensor()};
    }
    auto [act, prob] = unpermute_backward(grads[0], x, row_map, saved[2], x.scalar_type());
    if (!ctx->needs_input_grad(2)) prob = Tensor();
    else if (prob.scalar_type() != saved[2].scalar_type()) prob = prob.to(saved[2].scalar_type());
    return {act, Tensor(), prob};
  }
};

PyObject* py_unpermute(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&] {
    need_args(n, 3);
    const Tensor& x = tensor(a[0]);
    if (x.numel() == 0) return wrap(x);
    const Tensor& row_map = tensor(a[1]);
    const std::optional<Tensor> probs = opt_tensor(a[2]);
    return wrap(without_gil([&] { return UnpermuteFunction::apply(x, row_map, probs); }));
  });
}

// ---- module -------------------------------------------------------------------------------------------------------
// bind({name: address}): the C ABI to call
PyObject* py_bind(PyObject*, PyObject* arg) {
  return guarded([&]() -> PyObject* {
    auto address = [&](const char* name) -> void* {
      PyObject* v = PyDict_Check(arg) ? PyDict_GetItemString(arg, name) : nullptr;
      if (v == nullptr) throw std::runtime_error(std::string("dlblas_b200: no address for ") + name);
      void* p = PyLong_AsVoidPtr(v);
      if (p == nullptr) throw PyFailed{};
      return p;
    };
#define X(name) abi.name = reinterpret_cast<decltype(abi.name)>(address(#name));
    ABI_FUNCTIONS(X)
#undef X
    Py_RETURN_NONE;
  });
}

PyObject* py_status_word(PyObject*, PyObject* arg) {
  return guarded([&] {
    const int64_t index = integer(arg);
    return wrap(without_gil([&] { return status_word((at::DeviceIndex)index); }));
  });
}

#define FAST(name, fn) {name, (PyCFunction)(void (*)(void))fn, METH_FASTCALL, nullptr}
PyMethodDef methods[] = {
    {"bind", py_bind, METH_O, nullptr},
    {"status_word", py_status_word, METH_O, nullptr},
    FAST("quant_fp8", py_quant_fp8),
    FAST("group_quant_fp8", py_group_quant_fp8),
    FAST("fp8_gemm", py_fp8_gemm),
    FAST("route_softmax_topk", py_route_softmax_topk),
    FAST("route_grouped_topk", py_route_grouped_topk),
    FAST("moe_forward", py_moe_forward),
    FAST("low_latency_forward", py_low_latency_forward),
    FAST("m_grouped_gemm", py_m_grouped_gemm),
    FAST("k_grouped_gemm", py_k_grouped_gemm),
    FAST("moe_forward_16bit", py_moe_forward_16bit),
    FAST("moe_align_block_size", py_moe_align_block_size),
    FAST("gating_capacity", py_gating_capacity),
    FAST("gating_forward", py_gating_forward),
    FAST("gating_backward", py_gating_backward),
    FAST("topk_gating", py_topk_gating),
    FAST("permute_plan", py_permute_plan),
    FAST("unpermute_rows", py_unpermute_rows),
    FAST("unpermute_backward", py_unpermute_backward),
    FAST("permute", py_permute),
    FAST("unpermute", py_unpermute),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit__host(void) { return PyModule_Create(&module); }
