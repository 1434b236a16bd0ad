// CPython module quik_b200._host: the per-call host work of the layer (argument checks, output and workspace allocation,
// the library call) in native code.
//
// A layer of few tokens runs for less time on the GPU (about 10 us) than its two library calls took to issue from Python:
// attribute look-ups, four tensor allocations, device guards and two ctypes calls of 14 and 19 arguments were 49 us per layer,
// so every workload of up to a few hundred tokens was bound by them.  The functions here take the tensors themselves and
// reach the C ABI of libquik_b200.so through the addresses handed to init(); errors become the same RuntimeErrors.
#include <Python.h>
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cstring>
#include <memory>
#include <string>
#include <utility>
#include <vector>

#include "../../include/quik_b200.h"

namespace {

struct Abi {
  decltype(&quik_layer_quantize) quantize = nullptr;
  decltype(&quik_mixed_linear_ld) linear = nullptr;
  decltype(&quik_config_get) config_get = nullptr;
  decltype(&quik_strerror) strerror_ = nullptr;
  decltype(&quik_last_cuda_error) last_cuda_error = nullptr;
  decltype(&quik_rotary_inplace) rotary = nullptr;
} abi;

// attribute and buffer names of the module (interned once)
struct Names {
  PyObject *buffers, *int_weight, *int_indices, *fp_indices, *weights_scales, *reduced_w, *fp_weight, *bias, *int_features_num,
      *out_features, *fp_features_num, *bits;
} names;

void check(int status, const char *what) {
  if (status == QUIK_OK) return;
  std::string msg = std::string(what) + ": " + abi.strerror_(status);
  if (status == QUIK_ERR_CUDA) msg += std::string(" [") + abi.last_cuda_error() + "]";
  throw std::runtime_error(msg);
}

// the conditions of _lib.require_cuda_contiguous
void require(const char *op, const char *name, const at::Tensor &t, const at::Tensor &first) {
  if (!t.is_cuda())
    throw std::runtime_error(std::string(op) + ": expected tensor for argument '" + name + "' to be on a CUDA device");
  if (!t.is_contiguous())
    throw std::runtime_error(std::string(op) + ": expected tensor for argument '" + name + "' to be contiguous");
  if (t.device() != first.device())
    throw std::runtime_error(std::string(op) + ": expected all tensors on the same GPU, got " + first.device().str() + " and " +
                             t.device().str());
}

int dtype_code(at::ScalarType t) {
  if (t == at::kHalf) return QUIK_F16;
  if (t == at::kBFloat16) return QUIK_BF16;
  throw std::runtime_error(std::string("expected a float16 or bfloat16 tensor, got ") + c10::toString(t));
}

void *ptr(const at::Tensor &t) { return t.numel() == 0 ? nullptr : t.data_ptr(); }

const at::Tensor &tensor_arg(PyObject *o) {
  if (!THPVariable_Check(o)) throw std::runtime_error("expected a tensor");
  return THPVariable_Unpack(o);
}
// None -> undefined tensor
at::Tensor optional_arg(PyObject *o) { return o == Py_None ? at::Tensor() : tensor_arg(o); }

void expect(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) throw std::runtime_error("quik_b200._host: wrong number of arguments");
}

// where the quantizer's outputs are (the tensors or the workspace that hold them belong to the caller)
struct Codes {
  void *q, *meta, *fp_x;
};

constexpr int64_t align256(int64_t v) { return (v + 255) & ~(int64_t)255; }

// Checks the arguments of a quantizer call.  Producer 0: none, 1: RMSNorm (aux = weight vector), 2: SiLU(x) * aux.
const char *check_quantize(int producer, const at::Tensor &x, const at::Tensor &aux, const at::Tensor &ids, const at::Tensor &fp_ids,
                           int bits) {
  static const char *const ops[3] = {"quantize", "rmsnorm_quantize", "silu_mul_quantize"};
  const char *op = ops[producer];
  require(op, producer == 2 ? "gate" : (producer == 1 ? "x" : "src"), x, x);
  if (producer) require(op, producer == 1 ? "norm_weight" : "up", aux, x);
  require(op, "int_indices", ids, x);
  require(op, "fp_indices", fp_ids, x);
  if (bits != 4 && bits != 8) throw std::runtime_error("bits argument must be either 4 or 8");
  if (x.dim() != 2) throw std::runtime_error(std::string(op) + ": expected a matrix");
  if (producer == 1 && (aux.numel() != x.size(1) || aux.scalar_type() != x.scalar_type()))
    throw std::runtime_error("rmsnorm_quantize: norm_weight must have one entry per column, of x's dtype");
  if (producer == 2 && (!aux.sizes().equals(x.sizes()) || aux.scalar_type() != x.scalar_type()))
    throw std::runtime_error("silu_mul_quantize: gate and up must have the same shape and dtype");
  return op;
}

void launch_quantize(const char *op, int producer, const at::Tensor &x, const at::Tensor &aux, double eps, const at::Tensor &ids,
                     const at::Tensor &fp_ids, int bits, bool wide, bool settled, const Codes &c) {
  void *st = c10::cuda::getCurrentCUDAStream(x.device().index()).stream();
  check(abi.quantize(producer, ptr(x), producer ? ptr(aux) : nullptr, (float)eps, dtype_code(x.scalar_type()), (int)x.size(0),
                     (int)x.size(1), static_cast<const uint16_t *>(ptr(ids)), (int)ids.numel(),
                     static_cast<const uint16_t *>(ptr(fp_ids)), (int)fp_ids.numel(), bits, wide, settled, c.q, c.meta, c.fp_x, st),
        op);
}

// Operand layouts of a layer of `bits` with k_int integer columns for m tokens, which is to say the engine that the fused launch
// will use (the C side picks it from them, include/quik_b200.h):
//   up to STREAM_M_MAX tokens: weight streaming, the weights stay in their storage format; the tcgen05 streaming engine takes
//     the token codes one per byte, the mma.sync engines (up to SMALL_M_MAX tokens, the default for 4-bit layers) packed
//     like the weights;
//   more tokens: tensor-core GEMM on weight codes one per byte; the quantizer writes the token codes one per byte too,
//     except when the engine with the token operand in tensor memory is selected: it takes 4-bit token codes packed (the
//     reference layout) and widens them on chip.
// (a packed 4-bit row must be a multiple of 16 bytes for these engines; otherwise both operands one per byte)
struct Layouts {
  bool q_packed = false, w_packed = false;
};
Layouts operand_layouts(int bits, int64_t k_int, int64_t m) {
  Layouts r;
  if (bits == 8) return r;
  const bool row_ok = k_int % 32 == 0;
  const int small_m = abi.config_get(QUIK_CFG_SMALL_M);
  if (m <= QUIK_STREAM_M_MAX && small_m != 0 && row_ok) {
    r.w_packed = true;
    r.q_packed = m <= QUIK_SMALL_M_MAX && small_m != 3;
  } else {
    r.q_packed = row_ok && abi.config_get(QUIK_CFG_GEMM_ENGINE) == QUIK_ENGINE_TCGEN05_TS;
  }
  return r;
}

// the layer's own tensors, as the module holds them
struct Layer {
  at::Tensor scales, reduced, fp_w, bias;
  int64_t k_int, n, f;
  int bits;
};

// True at first and after the integer or outlier weights (fp_w may be undefined) were replaced or written in place since the last
// call with this record, by address and version; always for inference tensors, which count no versions.
constexpr size_t kSeenBytes = 4 * sizeof(int64_t);
struct Seen {
  int64_t v[4] = {0, 0, 0, 0};
  bool known = true;
  Seen(const at::Tensor &w, const at::Tensor &fp_w) {
    const at::Tensor *const t[2] = {&w, &fp_w};
    for (int i = 0; i < 2; ++i) {
      if (!t[i]->defined()) continue;
      known = known && !t[i]->is_inference();
      v[2 * i] = (int64_t)(intptr_t)ptr(*t[i]);
      v[2 * i + 1] = known ? (int64_t)t[i]->_version() : 0;
    }
  }
  bool changed(const char *record) const { return !known || std::memcmp(record, v, kSeenBytes) != 0; }
};
char *seen_arg(PyObject *o) {
  if (!PyByteArray_Check(o) || PyByteArray_GET_SIZE(o) != (Py_ssize_t)kSeenBytes) throw std::runtime_error("expected a record of 32 bytes");
  return PyByteArray_AS_STRING(o);
}
// Before a launch for few tokens.  The ring streaming engine loads its first weight tiles before it waits for the stream's earlier
// launches (QUIK_CFG_STREAM_PRELOAD), which may just have written them: after a change of the weights an ordinary launch goes
// first.  It starts when all earlier ones have completed, and the layer's launches start when it has.  Called with the GIL held:
// no other thread takes the weights for settled before that launch is in the stream.
void settle_weights(const at::Tensor &x, const at::Tensor &w, const at::Tensor &fp_w, char *record) {
  const int64_t rows = x.dim() >= 2 ? x.size(-2) : 0;
  if (rows > QUIK_SMALL_M_MAX || !w.is_cuda()) return;
  const Seen now(w, fp_w);
  if (!now.changed(record)) return;
  const c10::cuda::OptionalCUDAGuard guard(w.device());
  at::zeros({1}, w.options());
  std::memcpy(record, now.v, kSeenBytes);
}

// [1, M, N] (or `out_buffer` with that leading dimension added, where the caller gave one)
at::Tensor launch_linear(const at::Tensor &x, const Codes &c, bool q_packed, const void *w, bool w_packed, const Layer &l,
                         const at::Tensor &out_buffer) {
  const int64_t m = x.size(0);
  at::Tensor result = out_buffer.defined() ? out_buffer.unsqueeze(0) : at::empty({1, m, l.n}, x.options());
  const int64_t pitch = out_buffer.defined() ? out_buffer.stride(0) : l.n;
  check(abi.linear(c.q, q_packed, w, w_packed, c.meta, ptr(l.scales), ptr(l.reduced), l.f > 0 ? c.fp_x : nullptr,
                   l.f > 0 ? ptr(l.fp_w) : nullptr, l.bias.defined() ? ptr(l.bias) : nullptr, ptr(result), pitch,
                   dtype_code(x.scalar_type()), (int)m, (int)l.n, (int)l.k_int, (int)l.f, l.bits,
                   c10::cuda::getCurrentCUDAStream(x.device().index()).stream()),
        "MixedQLinear.forward");
  return result;
}

PyObject *py_init(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 6);
  void *p[6];
  for (int i = 0; i < 6; ++i) {
    p[i] = PyLong_AsVoidPtr(a[i]);
    if (p[i] == nullptr) throw std::runtime_error("quik_b200._host.init: a library function is missing");
  }
  abi.quantize = reinterpret_cast<decltype(abi.quantize)>(p[0]);
  abi.linear = reinterpret_cast<decltype(abi.linear)>(p[1]);
  abi.strerror_ = reinterpret_cast<decltype(abi.strerror_)>(p[2]);
  abi.last_cuda_error = reinterpret_cast<decltype(abi.last_cuda_error)>(p[3]);
  abi.config_get = reinterpret_cast<decltype(abi.config_get)>(p[4]);
  abi.rotary = reinterpret_cast<decltype(abi.rotary)>(p[5]);
  const std::pair<PyObject **, const char *> all[] = {
      {&names.buffers, "_buffers"}, {&names.int_weight, "int_weight"}, {&names.int_indices, "int_indices"},
      {&names.fp_indices, "fp_indices"}, {&names.weights_scales, "weights_scales"}, {&names.reduced_w, "reduced_w"},
      {&names.fp_weight, "fp_weight"}, {&names.bias, "bias"}, {&names.int_features_num, "int_features_num"},
      {&names.out_features, "out_features"}, {&names.fp_features_num, "fp_features_num"}, {&names.bits, "bits"}};
  for (auto &a : all)
    if ((*a.first = PyUnicode_InternFromString(a.second)) == nullptr) return nullptr;
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// (producer, x, aux | None, eps, int_ids, fp_ids, bits, wide, ids_settled) -> (codes, meta, fp_x)
PyObject *py_quantize(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 9);
  const int producer = (int)PyLong_AsLong(a[0]), bits = (int)PyLong_AsLong(a[6]);
  const double eps = PyFloat_AsDouble(a[3]);
  const bool wide = PyObject_IsTrue(a[7]) == 1, settled = PyObject_IsTrue(a[8]) == 1;
  if (PyErr_Occurred()) return nullptr;
  if (producer < 0 || producer > 2) throw std::runtime_error("quik_b200._host.quantize: producer");
  const at::Tensor x = tensor_arg(a[1]), aux = optional_arg(a[2]), ids = tensor_arg(a[4]), fp_ids = tensor_arg(a[5]);
  if (producer && !aux.defined()) throw std::runtime_error("expected a tensor");
  at::Tensor q, meta, fp_x;
  {
    py::gil_scoped_release nogil;
    const char *op = check_quantize(producer, x, aux, ids, fp_ids, bits);
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    const int64_t rows = x.size(0), num_int = ids.numel();
    q = bits == 4 && !wide ? at::empty({rows, num_int / 2}, x.options().dtype(at::kByte))
                           : at::empty({rows, num_int}, x.options().dtype(at::kChar));
    meta = at::empty({2 * rows}, x.options());
    fp_x = at::empty({rows, fp_ids.numel()}, x.options());
    launch_quantize(op, producer, x, aux, eps, ids, fp_ids, bits, wide, settled, Codes{ptr(q), ptr(meta), ptr(fp_x)});
  }
  PyObject *r = PyTuple_New(3);
  if (!r) return nullptr;
  PyTuple_SET_ITEM(r, 0, THPVariable_Wrap(std::move(q)));
  PyTuple_SET_ITEM(r, 1, THPVariable_Wrap(std::move(meta)));
  PyTuple_SET_ITEM(r, 2, THPVariable_Wrap(std::move(fp_x)));
  return r;
  END_HANDLE_TH_ERRORS
}

// scales, reduced, fp_w | None, bias | None, k_int, n, f, bits at a[0..7]
bool layer_args(PyObject *const *a, Layer *l) {
  *l = Layer{tensor_arg(a[0]), tensor_arg(a[1]), optional_arg(a[2]), optional_arg(a[3]), PyLong_AsLongLong(a[4]),
             PyLong_AsLongLong(a[5]), PyLong_AsLongLong(a[6]), (int)PyLong_AsLong(a[7])};
  if (PyErr_Occurred()) return false;
  if (l->f > 0 && !l->fp_w.defined()) throw std::runtime_error("expected a tensor");
  return true;
}

// (x, out | None, scales, reduced, fp_w | None, bias | None, k_int, n, f, bits, w, w_packed, codes, q_packed, meta, fp_x, seen):
// the fused launch on a quantized input; x gives the number of tokens, the dtype and the device
PyObject *py_linear(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 17);
  const at::Tensor x = tensor_arg(a[0]), out = optional_arg(a[1]), w = tensor_arg(a[10]), q = tensor_arg(a[12]),
                   meta = tensor_arg(a[14]), fp_x = tensor_arg(a[15]);
  const bool w_packed = PyObject_IsTrue(a[11]) == 1, q_packed = PyObject_IsTrue(a[13]) == 1;
  Layer l;
  if (!layer_args(a + 2, &l)) return nullptr;
  settle_weights(x, w, l.fp_w, seen_arg(a[16]));
  at::Tensor result;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    result = launch_linear(x, Codes{ptr(q), ptr(meta), ptr(fp_x)}, q_packed, ptr(w), w_packed, l, out);
  }
  return THPVariable_Wrap(std::move(result));
  END_HANDLE_TH_ERRORS
}

// Quantizer and fused launch, the quantized input in a workspace that lives as long as the call.  The ids are settled (see
// quik_layer_quantize).  w: the weights in storage format; w8: 4-bit weights one code per byte; an undefined tensor is returned,
// and nothing launched, where the settings ask for them and they were not given.
at::Tensor run_layer(const at::Tensor &given, const at::Tensor &out, const Layer &l, const at::Tensor &w, const at::Tensor &w8,
                     const at::Tensor &ids, const at::Tensor &fp_ids, char *seen) {
  settle_weights(given, w, l.fp_w, seen);
  py::gil_scoped_release nogil;
  const at::Tensor x = given.dim() == 3 ? given.select(0, 0) : given;      // the first matrix of a batch, as ever
  const char *op = check_quantize(0, x, at::Tensor(), ids, fp_ids, l.bits);
  const int64_t m = x.size(0);
  const Layouts lay = operand_layouts(l.bits, l.k_int, m);
  const bool needs_w8 = l.bits == 4 && !lay.w_packed;
  if (needs_w8 && !w8.defined()) return at::Tensor();
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  const int64_t b_q = align256(m * ids.numel()), b_meta = align256(m * 4);
  const at::Tensor ws = at::empty({b_q + b_meta + m * fp_ids.numel() * 2}, x.options().dtype(at::kByte));
  unsigned char *base = static_cast<unsigned char *>(ptr(ws));
  const Codes c{base, base + b_q, base + b_q + b_meta};
  launch_quantize(op, 0, x, at::Tensor(), 0.0, ids, fp_ids, l.bits, !lay.q_packed, true, c);
  return launch_linear(x, c, lay.q_packed, ptr(needs_w8 ? w8 : w), lay.w_packed, l, out);
}

// (x, out | None, scales, reduced, fp_w | None, bias | None, k_int, n, f, bits, w, w8 | None, int_ids, fp_ids, seen): run_layer
PyObject *py_layer(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 15);
  const at::Tensor given = tensor_arg(a[0]), out = optional_arg(a[1]), w = tensor_arg(a[10]), w8 = optional_arg(a[11]),
                   ids = tensor_arg(a[12]), fp_ids = tensor_arg(a[13]);
  Layer l;
  if (!layer_args(a + 2, &l)) return nullptr;
  at::Tensor result = run_layer(given, out, l, w, w8, ids, fp_ids, seen_arg(a[14]));
  if (!result.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(result));
  END_HANDLE_TH_ERRORS
}

// ---- calls by module and plan -----------------------------------------------------------------------------------------------
// A plan is the tuple (int_ids | None, fp_ids | None, w8 | None, sources) of a module's derived operands, where it has derived them; the
// sources say which buffers they were derived from.  The module's buffers and sizes are read on every call; where they are not those of the plan, or something is
// missing, a call returns None having launched nothing, and the module's own path derives them anew.  Reading attributes, comparing
// keys and collecting arguments in Python was 6 us of the 15 us of a call for one token.

// A tensor that something was derived from, at one version of its contents.  Address and version alone do not name it: the allocator
// gives the memory of a tensor that was freed to the next of its size, whose version starts at zero too.  The weak handles keep
// no device memory, but they keep the addresses of the tensor and of its storage object from being given out again.
struct Source {
  c10::weak_intrusive_ptr<at::TensorImpl, at::UndefinedTensorImpl> tensor;
  c10::weak_intrusive_ptr<c10::StorageImpl> storage;
  const void *data;
  int64_t version;
  explicit Source(const at::Tensor &t)
      : tensor(t.getIntrusivePtr()), storage(t.storage().getWeakStorageImpl()), data(ptr(t)), version((int64_t)t._version()) {}
  bool same(const at::Tensor &t) const {
    return t.unsafeGetTensorImpl() == tensor._unsafe_get_target() && t.storage().unsafeGetStorageImpl() == storage._unsafe_get_target() &&
           ptr(t) == data && !t.is_inference() && (int64_t)t._version() == version;
  }
};
using Sources = std::vector<Source>;
constexpr const char *kSourcesName = "quik_b200.sources";
// of the capsule that py_sources made, else nullptr
const Sources *sources_arg(PyObject *o) {
  return PyCapsule_IsValid(o, kSourcesName) ? static_cast<const Sources *>(PyCapsule_GetPointer(o, kSourcesName)) : nullptr;
}

struct Planned {
  Layer l;
  at::Tensor w, w8, ids, fp_ids;
};
// 1: read, 0: not the plan's module any more, -1: Python error
int read_planned(PyObject *module, PyObject *plan, Planned *r) {
  if (!PyTuple_Check(plan) || PyTuple_GET_SIZE(plan) != 4) return 0;
  const Sources *sources = sources_arg(PyTuple_GET_ITEM(plan, 3));
  if (!sources || sources->size() < 3) return 0;
  PyObject *buffers = PyObject_GetAttr(module, names.buffers);
  if (!buffers) return -1;
  bool have = PyDict_Check(buffers);
  auto buffer = [&](PyObject *name, at::Tensor *t, bool may_be_none) {
    PyObject *o = have ? PyDict_GetItemWithError(buffers, name) : nullptr;
    if (o && THPVariable_Check(o)) *t = THPVariable_Unpack(o);
    else if (!(o == Py_None && may_be_none)) have = false;
  };
  auto size = [&](PyObject *name) -> int64_t {
    if (!have) return 0;
    PyObject *o = PyObject_GetAttr(module, name);
    const int64_t v = o ? PyLong_AsLongLong(o) : -1;
    Py_XDECREF(o);
    if (PyErr_Occurred()) have = false;
    return v;
  };
  at::Tensor ids64, fp64;
  buffer(names.int_weight, &r->w, false);
  buffer(names.int_indices, &ids64, false);
  buffer(names.fp_indices, &fp64, false);
  buffer(names.weights_scales, &r->l.scales, false);
  buffer(names.reduced_w, &r->l.reduced, false);
  buffer(names.bias, &r->l.bias, true);
  r->l.k_int = size(names.int_features_num);
  r->l.n = size(names.out_features);
  r->l.f = size(names.fp_features_num);
  r->l.bits = (int)size(names.bits);
  if (have && r->l.f > 0) buffer(names.fp_weight, &r->l.fp_w, false);
  Py_DECREF(buffers);
  if (PyErr_Occurred()) return -1;
  if (!have || r->l.k_int <= 0 || !(*sources)[0].same(ids64) || !(*sources)[1].same(fp64) || !(*sources)[2].same(r->w) ||
      sources->size() != (r->l.f > 0 ? 4u : 3u) || (r->l.f > 0 && !(*sources)[3].same(r->l.fp_w)))
    return 0;
  r->ids = optional_arg(PyTuple_GET_ITEM(plan, 0));
  r->fp_ids = optional_arg(PyTuple_GET_ITEM(plan, 1));
  r->w8 = optional_arg(PyTuple_GET_ITEM(plan, 2));
  return 1;
}
// the device of x becomes the current one, as the module's forward has it
void make_current(const at::Tensor &x) {
  if (c10::cuda::current_device() != x.device().index()) c10::cuda::set_device(x.device().index());
}

// (tensor, ...) -> sources: the tensors and the versions of their contents; RuntimeError where one counts no versions
PyObject *py_sources(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  auto made = std::make_unique<Sources>();
  made->reserve(n);
  for (Py_ssize_t i = 0; i < n; ++i) made->emplace_back(tensor_arg(a[i]));
  PyObject *o = PyCapsule_New(made.get(), kSourcesName, [](PyObject *c) { delete const_cast<Sources *>(sources_arg(c)); });
  if (o) made.release();
  return o;
  END_HANDLE_TH_ERRORS
}

// (sources, tensor, ...) -> whether these are the tensors that the sources were made of, unchanged
PyObject *py_same_sources(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n < 1) expect(n, 1);
  const Sources *sources = sources_arg(a[0]);
  bool same = sources && (Py_ssize_t)sources->size() == n - 1;
  for (Py_ssize_t i = 1; same && i < n; ++i) same = (*sources)[i - 1].same(tensor_arg(a[i]));
  return PyBool_FromLong(same);
  END_HANDLE_TH_ERRORS
}

// (module, plan, seen, x) -> output | None
PyObject *py_forward(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 4);
  Planned r;
  const int ok = read_planned(a[0], a[1], &r);
  if (ok < 0) return nullptr;
  if (ok == 0 || !r.ids.defined() || !r.fp_ids.defined() || !THPVariable_Check(a[3])) Py_RETURN_NONE;
  const at::Tensor x = tensor_arg(a[3]);
  if (!x.is_cuda()) Py_RETURN_NONE;
  make_current(x);
  at::Tensor result = run_layer(x, at::Tensor(), r.l, r.w, r.w8, r.ids, r.fp_ids, seen_arg(a[2]));
  if (!result.defined()) Py_RETURN_NONE;
  return THPVariable_Wrap(std::move(result));
  END_HANDLE_TH_ERRORS
}

// (module, plan, producer, x, aux | None, eps) -> (codes, meta, fp_x, one code per byte) | None; x [1, M, K] or [M, K]
PyObject *py_quantize_for(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 6);
  Planned r;
  const int ok = read_planned(a[0], a[1], &r);
  if (ok < 0) return nullptr;
  const int producer = (int)PyLong_AsLong(a[2]);
  const double eps = PyFloat_AsDouble(a[5]);
  if (PyErr_Occurred()) return nullptr;
  if (ok == 0 || !r.ids.defined() || !r.fp_ids.defined() || producer < 0 || producer > 2 || !THPVariable_Check(a[3])) Py_RETURN_NONE;
  at::Tensor x = tensor_arg(a[3]), aux = optional_arg(a[4]);
  if (!x.is_cuda()) Py_RETURN_NONE;
  if (producer == 0) make_current(x);
  if (producer && !aux.defined()) throw std::runtime_error("expected a tensor");
  at::Tensor q, meta, fp_x;
  bool wide;
  {
    py::gil_scoped_release nogil;
    if (x.dim() == 3) x = x.select(0, 0);
    if (producer) x = x.contiguous();
    if (producer == 2) aux = (aux.dim() == 3 ? aux.select(0, 0) : aux).contiguous();
    const char *op = check_quantize(producer, x, aux, r.ids, r.fp_ids, r.l.bits);
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    const int64_t rows = x.size(0), num_int = r.ids.numel();
    wide = !operand_layouts(r.l.bits, r.l.k_int, rows).q_packed;
    q = r.l.bits == 4 && !wide ? at::empty({rows, num_int / 2}, x.options().dtype(at::kByte))
                               : at::empty({rows, num_int}, x.options().dtype(at::kChar));
    meta = at::empty({2 * rows}, x.options());
    fp_x = at::empty({rows, r.fp_ids.numel()}, x.options());
    launch_quantize(op, producer, x, aux, eps, r.ids, r.fp_ids, r.l.bits, wide, true, Codes{ptr(q), ptr(meta), ptr(fp_x)});
  }
  PyObject *t = PyTuple_New(4);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(q)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(meta)));
  PyTuple_SET_ITEM(t, 2, THPVariable_Wrap(std::move(fp_x)));
  PyTuple_SET_ITEM(t, 3, PyBool_FromLong(wide));
  return t;
  END_HANDLE_TH_ERRORS
}

// (module, plan, seen, x, codes, meta, fp_x, one code per byte) -> output | None: the fused launch on a quantized input
PyObject *py_forward_quantized(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 8);
  Planned r;
  const int ok = read_planned(a[0], a[1], &r);
  if (ok < 0) return nullptr;
  if (ok == 0) Py_RETURN_NONE;
  for (int i = 3; i < 7; ++i)
    if (!THPVariable_Check(a[i])) Py_RETURN_NONE;
  const bool wide = PyObject_IsTrue(a[7]) == 1;
  const at::Tensor given = tensor_arg(a[3]), q = tensor_arg(a[4]), meta = tensor_arg(a[5]), fp_x = tensor_arg(a[6]);
  if (!given.is_cuda() || given.dim() < 1) Py_RETURN_NONE;
  const at::Tensor x = given.dim() == 3 ? given.select(0, 0) : given;
  const Layouts lay = operand_layouts(r.l.bits, r.l.k_int, x.size(0));
  const bool needs_w8 = r.l.bits == 4 && !lay.w_packed;
  if ((r.l.bits == 4 && wide == lay.q_packed) || (needs_w8 && !r.w8.defined())) Py_RETURN_NONE;
  make_current(x);
  settle_weights(x, needs_w8 ? r.w8 : r.w, r.l.fp_w, seen_arg(a[2]));
  at::Tensor result;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::OptionalCUDAGuard guard(x.device());
    result = launch_linear(x, Codes{ptr(q), ptr(meta), ptr(fp_x)}, lay.q_packed, ptr(needs_w8 ? r.w8 : r.w), lay.w_packed, r.l, at::Tensor());
  }
  return THPVariable_Wrap(std::move(result));
  END_HANDLE_TH_ERRORS
}

// (q, k, cos, sin, tokens, q_heads, k_heads, head_dim): rotary embedding in place
PyObject *py_rotary(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 8);
  const at::Tensor q = tensor_arg(a[0]), k = tensor_arg(a[1]), c = tensor_arg(a[2]), s = tensor_arg(a[3]);
  int v[4];
  for (int i = 0; i < 4; ++i) v[i] = (int)PyLong_AsLong(a[4 + i]);
  if (PyErr_Occurred()) return nullptr;
  const c10::cuda::OptionalCUDAGuard guard(q.device());
  check(abi.rotary(ptr(q), ptr(k), ptr(c), ptr(s), dtype_code(q.scalar_type()), v[0], v[1], v[2], v[3],
                   c10::cuda::getCurrentCUDAStream(q.device().index()).stream()),
        "rotary");
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// (bits, k_int, m) -> (token codes packed, weight codes packed)
PyObject *py_operand_layouts(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 3);
  const int bits = (int)PyLong_AsLong(a[0]);
  const int64_t k_int = PyLong_AsLongLong(a[1]), m = PyLong_AsLongLong(a[2]);
  if (PyErr_Occurred()) return nullptr;
  const Layouts r = operand_layouts(bits, k_int, m);
  return PyTuple_Pack(2, r.q_packed ? Py_True : Py_False, r.w_packed ? Py_True : Py_False);
  END_HANDLE_TH_ERRORS
}

// (seen, w, fp_w | None) -> whether the weights differ from the record, which holds them afterwards
PyObject *py_weights_changed(PyObject *, PyObject *const *a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  expect(n, 3);
  char *record = seen_arg(a[0]);
  const Seen now(tensor_arg(a[1]), optional_arg(a[2]));
  const bool changed = now.changed(record);
  std::memcpy(record, now.v, kSeenBytes);
  return PyBool_FromLong(changed);
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"init", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_init)), METH_FASTCALL, "addresses of the C ABI"},
    {"quantize", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_quantize)), METH_FASTCALL, "activation quantizer"},
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_linear)), METH_FASTCALL, "fused launch"},
    {"layer", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_layer)), METH_FASTCALL, "quantizer and fused launch"},
    {"operand_layouts", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_operand_layouts)), METH_FASTCALL,
     "operand layouts for a token count"},
    {"weights_changed", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_weights_changed)), METH_FASTCALL,
     "weights against a record"},
    {"sources", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_sources)), METH_FASTCALL, "tensors at their versions"},
    {"same_sources", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_same_sources)), METH_FASTCALL,
     "tensors against sources"},
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_forward)), METH_FASTCALL, "a module's forward by its plan"},
    {"quantize_for", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_quantize_for)), METH_FASTCALL,
     "activation quantizer for a module by its plan"},
    {"forward_quantized", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_forward_quantized)), METH_FASTCALL,
     "fused launch of a module by its plan"},
    {"rotary", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_rotary)), METH_FASTCALL, "rotary embedding in place"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "native host path of the layer", -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) { return PyModule_Create(&module); }
