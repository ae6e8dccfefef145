// Host side of the operators as a CPython extension: argument checks, output allocation, workspace lookup and the
// C-ABI calls of one operator in one native call. Through ctypes a quantise + GEMM pair cost 40 us of interpreter
// time on the calling thread (20 arguments marshalled twice, three tensors allocated from Python), more than the
// two kernels run for at decode and short-prompt sizes.
//
// Every function here handles the regular case only and returns None for anything else (another layout, dtype or
// device, a tensor subclass, an unsupported shape): the Python wrapper then takes its general path, which also
// raises the errors. Nothing is kept from one call to the next except the scratch buffers below.
//
// The interpreter lock is given back while a function allocates and launches: a launch waits when the stream's queue is
// full, for as long as the work ahead of it takes, and that work may include a host callback that needs the lock.
#include <dlfcn.h>

#include <atomic>
#include <list>
#include <mutex>
#include <vector>

#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/b200_blockfp8.h"

namespace {

using at::Tensor;

// The library is the one the ctypes binding loaded (possibly another build of it), so its functions are looked up
// there instead of being linked.
struct Abi {
  decltype(&b200_status_string) status_string;
  decltype(&b200_last_error_detail) last_error_detail;
  decltype(&b200_get_tuning) get_tuning;
  decltype(&b200_per_token_group_quant_fp8) quant;
  decltype(&b200_per_token_group_quant_fp8_ue8m0) quant_ue8m0;
  decltype(&b200_w8a8_block_fp8_gemm_workspace_bytes) gemm_ws;
  decltype(&b200_w8a8_block_fp8_gemm) gemm;
  decltype(&b200_w8a8_block_fp8_gemm_packed_workspace_bytes) packed_ws;
  decltype(&b200_w8a8_block_fp8_gemm_packed) packed;
  decltype(&b200_w8a8_block_fp8_linear_workspace_bytes) linear_ws;
  decltype(&b200_w8a8_block_fp8_linear) linear;
  decltype(&b200_fused_experts_fp8_workspace_bytes) experts_ws;
  decltype(&b200_fused_experts_fp8) experts;
  decltype(&b200_route_topk) route;
} abi;

PyObject* fail(int status, const char* what) {
  PyObject* type = status == B200_E_BAD_ARG       ? PyExc_AssertionError
                   : status == B200_E_UNSUPPORTED ? PyExc_NotImplementedError
                                                  : PyExc_RuntimeError;
  return PyErr_Format(type, "%s: %s: %s", what, abi.status_string(status), abi.last_error_detail());
}

// Other Python threads run while one of these is alive: no Python object is touched in its scope.
struct WithoutInterpreterLock {
  PyThreadState* state = PyEval_SaveThread();
  WithoutInterpreterLock() = default;
  WithoutInterpreterLock(const WithoutInterpreterLock&) = delete;
  ~WithoutInterpreterLock() { PyEval_RestoreThread(state); }
};

// ------------------------------------------------------------------------------ scratch buffers
// One grow-only scratch buffer per (device, stream); work on one stream is ordered, so the next call may reuse it.
// Threads may share a stream: a call keeps the buffer's lock until its last kernel is launched, so that another call's
// kernels cannot come between them. The lock is only ever waited for without the interpreter lock.
// A CUDA graph bakes the buffer's address into its nodes: once a call has been seen under capture, a buffer that has to
// grow is kept alive instead of being given back to the allocator.
struct Scratch {
  int device;
  void* stream;
  std::mutex busy;  // guards the members below
  Tensor buf;
  std::vector<Tensor> retired;
};
// never destroyed: the process may end after the CUDA context
std::mutex& scratch_list_lock = *new std::mutex;
std::list<Scratch>& scratch = *new std::list<Scratch>;
std::atomic<bool> capture_seen{false};

Tensor empty_on(int device, at::IntArrayRef size, at::ScalarType dtype) {
  return Tensor(at::detail::empty_cuda(size, dtype, c10::Device(c10::kCUDA, (c10::DeviceIndex)device), std::nullopt));
}

Scratch& scratch_of(int device, void* stream) {
  std::lock_guard<std::mutex> guard(scratch_list_lock);
  for (auto& s : scratch)
    if (s.device == device && s.stream == stream) return s;
  Scratch& s = scratch.emplace_back();  // a list: the references of other threads stay valid
  s.device = device;
  s.stream = stream;
  return s;
}

// At least `bytes` bytes; s.busy is held.
void grow(Scratch& s, size_t bytes) {
  if (c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None) capture_seen = true;
  const size_t have = s.buf.defined() ? (size_t)s.buf.numel() : 0;
  if (have >= bytes) return;
  if (have && capture_seen) s.retired.push_back(s.buf);
  const size_t want = bytes > have + have / 2 ? bytes : have + have / 2;
  s.buf = Tensor();  // back to the allocator first: the larger block may take its place
  s.buf = empty_on(s.device, {(int64_t)want}, at::kByte);
}

// A stream's scratch for the kernels of one call: nothing when no bytes are needed.
struct Lease {
  std::unique_lock<std::mutex> lock;
  void* ptr = nullptr;
  Lease() = default;
  Lease(int device, void* stream, size_t bytes) {
    if (bytes == 0) return;
    Scratch& s = scratch_of(device, stream);
    lock = std::unique_lock<std::mutex>(s.busy);
    grow(s, bytes);
    ptr = s.buf.data_ptr();
  }
};

// ------------------------------------------------------------------------------------ arguments
// A plain CUDA tensor on the current device, or null.
const Tensor* plain(PyObject* o, int device) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided && t.get_device() == device ? &t : nullptr;
}
const Tensor* plain(PyObject* o, int device, at::ScalarType dtype) {  // and contiguous, of one type
  const Tensor* t = plain(o, device);
  return t && t->scalar_type() == dtype && t->is_contiguous() ? t : nullptr;
}
bool is_2d(const Tensor& t, int64_t rows, int64_t cols) { return t.dim() == 2 && t.size(0) == rows && t.size(1) == cols; }
int dtype_code(at::ScalarType t) {
  return t == at::kBFloat16 ? B200_BF16 : t == at::kHalf ? B200_F16 : t == at::kFloat ? B200_F32 : -1;
}
at::ScalarType dtype_of_code(long code) {
  return code == B200_BF16 ? at::kBFloat16 : code == B200_F16 ? at::kHalf : at::kFloat;
}
int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }
void* stream_of(int device) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)device).stream(); }
constexpr auto kFp8 = at::kFloat8_e4m3fn;
constexpr size_t kKeptScratch = 32u << 20;

// linear(x, weight, weight_scale): quantise per 1x128 group, block-FP8 GEMM, result of x's type.
PyObject* linear(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  const Tensor* x = plain(args[0], dev);
  const Tensor* w = plain(args[1], dev, kFp8);
  const Tensor* ws = plain(args[2], dev, at::kFloat);
  if (!x || !w || !ws || x->dim() < 1 || w->dim() != 2 || !x->is_contiguous()) Py_RETURN_NONE;
  const auto type = x->scalar_type();
  const int code = dtype_code(type);
  const int64_t K = x->size(-1), N = w->size(0);
  if ((code != B200_BF16 && code != B200_F16) || w->size(1) != K || K == 0 || K % 128 || N == 0 || N % 8) Py_RETURN_NONE;
  const int64_t M = x->numel() / K;
  if (M == 0 || !is_2d(*ws, cdiv(N, 128), K / 128)) Py_RETURN_NONE;
  c10::SmallVector<int64_t, 4> shape(x->sizes().begin(), x->sizes().end());
  shape.back() = N;
  Tensor out;
  int rc;
  {
    WithoutInterpreterLock unlocked;
    out = empty_on(dev, shape, type);
    void* st = stream_of(dev);
    const size_t need = abi.linear_ws(M, N, K);
    // a large scratch (long prefill) is worth a block of the caching allocator, which other work can use in between
    const bool kept = need <= kKeptScratch;
    const Lease lease = kept ? Lease(dev, st, need) : Lease();
    const Tensor own = kept ? Tensor() : empty_on(dev, {(int64_t)need}, at::kByte);
    rc = abi.linear(x->data_ptr(), code, w->data_ptr(), ws->data_ptr<float>(), out.data_ptr(), M, N, K,
                    kept ? lease.ptr : own.data_ptr(), need, st);
  }
  if (rc) return fail(rc, "w8a8_block_fp8_linear");
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// [a][b] storage seen as [rows, a], row index contiguous: the sizes of the fresh tensor are set in place (a view through the
// dispatcher costs two microseconds).
Tensor& row_contiguous(Tensor& t, int64_t rows, int64_t cols, int64_t pitch) {
  t.unsafeGetTensorImpl()->set_sizes_and_strides(at::IntArrayRef({rows, cols}), at::IntArrayRef({1, pitch}));
  return t;
}

PyObject* pair(Tensor a, Tensor b) {
  PyObject* t = PyTuple_New(2);
  if (!t) return nullptr;
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(a)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(b)));
  return t;
}

// quant(x, group, column_major, tma_aligned, ue8m0, formula, eps) of a 2-D input -> (x_q, x_s)
PyObject* quant(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 7) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  const Tensor* x = plain(args[0], dev);
  const long group = PyLong_AsLong(args[1]);
  const bool col = args[2] == Py_True, aligned = args[3] == Py_True, ue8m0 = args[4] == Py_True;
  const long formula = PyLong_AsLong(args[5]);
  const double eps = PyFloat_AsDouble(args[6]);
  if (!x || PyErr_Occurred() || x->dim() != 2 || !x->is_contiguous() || group <= 0) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const int code = dtype_code(x->scalar_type());
  const int64_t M = x->size(0), K = x->size(1);
  if (code < 0 || M == 0 || K == 0 || K % group || (ue8m0 && !(col && aligned))) Py_RETURN_NONE;
  const int64_t groups = K / group, padded = cdiv(M, 4) * 4;
  Tensor q, s;
  int rc;
  if (ue8m0) {  // four exponent bytes per word, row index contiguous, rows padded to 4
    {
      WithoutInterpreterLock unlocked;
      q = empty_on(dev, {M, K}, kFp8);
      s = empty_on(dev, {cdiv(groups, 4), padded}, at::kInt);
      rc = abi.quant_ue8m0(x->data_ptr(), code, q.data_ptr(), s.data_ptr(), M, K, (int)group, padded, 0, nullptr, 1,
                           stream_of(dev));
    }
    if (rc) return fail(rc, "per_token_group_quant_fp8 (UE8M0)");
    return pair(std::move(q), row_contiguous(s, M, cdiv(groups, 4), padded));
  }
  const int64_t ld = aligned ? padded : M;
  {
    WithoutInterpreterLock unlocked;
    q = empty_on(dev, {M, K}, kFp8);
    s = col ? empty_on(dev, {groups, ld}, at::kFloat) : empty_on(dev, {M, groups}, at::kFloat);
    rc = abi.quant(x->data_ptr(), code, q.data_ptr(), s.data_ptr<float>(), M, K, (int)group, col ? 1 : groups, col ? ld : 1,
                   (float)eps, (int)formula, stream_of(dev));
  }
  if (rc) return fail(rc, "per_token_group_quant_fp8");
  return pair(std::move(q), col ? row_contiguous(s, M, groups, ld) : s);
  END_HANDLE_TH_ERRORS
}

// matmul(A, B, As, Bs, out_dtype_code): 2-D operands, fp32 scales
PyObject* matmul(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  const Tensor *A = plain(args[0], dev, kFp8), *B = plain(args[1], dev, kFp8);
  const Tensor *As = plain(args[2], dev), *Bs = plain(args[3], dev, at::kFloat);
  const long code = PyLong_AsLong(args[4]);
  if (!A || !B || !As || !Bs || A->dim() != 2 || B->dim() != 2 || As->scalar_type() != at::kFloat) Py_RETURN_NONE;
  const int64_t M = A->size(0), K = A->size(1), N = B->size(0);
  if (M == 0 || N == 0 || K == 0 || B->size(1) != K || !is_2d(*As, M, cdiv(K, 128)) ||
      !is_2d(*Bs, cdiv(N, 128), cdiv(K, 128)) || code < B200_BF16 || code > B200_F32)
    Py_RETURN_NONE;
  Tensor out;
  int rc;
  {
    WithoutInterpreterLock unlocked;
    out = empty_on(dev, {M, N}, dtype_of_code(code));
    void* st = stream_of(dev);
    const size_t need = abi.gemm_ws(M, N, K);
    const Lease lease(dev, st, need);
    rc = abi.gemm(A->data_ptr(), As->data_ptr<float>(), As->stride(0), As->stride(1), B->data_ptr(), Bs->data_ptr<float>(),
                  out.data_ptr(), (int)code, M, N, K, lease.ptr, need, st);
  }
  if (rc) return fail(rc, "w8a8_block_fp8_matmul");
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// matmul_ue8m0(A, B, As, Bs, out_dtype_code): both scales packed exponent words, row index contiguous
PyObject* matmul_ue8m0(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  long knob = -1;
  abi.get_tuning("gemm_ue8m0", &knob);
  if (nargs != 5 || knob == 0) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  const Tensor *A = plain(args[0], dev, kFp8), *B = plain(args[1], dev, kFp8);
  const Tensor *As = plain(args[2], dev), *Bs = plain(args[3], dev);
  const long code = PyLong_AsLong(args[4]);
  if (!A || !B || !As || !Bs || A->dim() != 2 || B->dim() != 2 || As->scalar_type() != at::kInt || Bs->scalar_type() != at::kInt)
    Py_RETURN_NONE;
  const int64_t M = A->size(0), K = A->size(1), N = B->size(0), words = cdiv(K, 512);
  auto mn_major = [&](const Tensor& s, int64_t rows) {
    return s.dim() == 2 && s.size(0) == rows && s.size(1) >= words && (s.stride(0) == 1 || rows == 1) &&
           (s.size(1) == 1 || s.stride(1) >= rows);
  };
  if (M == 0 || N == 0 || K == 0 || K % 16 || N % 8 || B->size(1) != K || !mn_major(*As, M) || code < B200_BF16 || code > B200_F32)
    Py_RETURN_NONE;
  const int rows_per_word = mn_major(*Bs, N) ? 1 : mn_major(*Bs, cdiv(N, 128)) ? 128 : 0;
  if (!rows_per_word) Py_RETURN_NONE;
  auto pitch = [](const Tensor& s) { return s.size(1) > 1 ? s.stride(1) : s.size(0); };
  Tensor out;
  int rc;
  {
    WithoutInterpreterLock unlocked;
    out = empty_on(dev, {M, N}, dtype_of_code(code));
    void* st = stream_of(dev);
    const size_t need = abi.packed_ws(M, N, K);
    const Lease lease(dev, st, need);
    rc = abi.packed(A->data_ptr(), As->data_ptr<int>(), pitch(*As), B->data_ptr(), Bs->data_ptr<int>(), pitch(*Bs),
                    rows_per_word, out.data_ptr(), (int)code, M, N, K, lease.ptr, need, st);
  }
  if (rc) return fail(rc, "w8a8_block_fp8_matmul (UE8M0)");
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// experts(hidden, w1, w2, topk_weights, topk_ids, w1_scale, w2_scale, inplace, no_combine, weight_on_input, scale)
PyObject* experts(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 11) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  const Tensor* x = plain(args[0], dev);
  const Tensor *w1 = plain(args[1], dev, kFp8), *w2 = plain(args[2], dev, kFp8);
  const Tensor *tw = plain(args[3], dev, at::kFloat), *ti = plain(args[4], dev, at::kInt);
  const Tensor *s1 = plain(args[5], dev, at::kFloat), *s2 = plain(args[6], dev, at::kFloat);
  const bool inplace = args[7] == Py_True, no_combine = args[8] == Py_True, on_input = args[9] == Py_True;
  const double scale = args[10] == Py_None ? 1.0 : PyFloat_AsDouble(args[10]);
  if (PyErr_Occurred()) PyErr_Clear();
  else if (x && w1 && w2 && tw && ti && s1 && s2 && x->dim() == 2 && x->is_contiguous() && w1->dim() == 3 && w2->dim() == 3 &&
           ti->dim() == 2) {
    const int code = dtype_code(x->scalar_type());
    const int64_t T = x->size(0), H = x->size(1), E = w1->size(0), I = w1->size(1) / 2, k = ti->size(1);
    auto is_3d = [](const Tensor& t, int64_t a, int64_t b, int64_t c) {
      return t.dim() == 3 && t.size(0) == a && t.size(1) == b && t.size(2) == c;
    };
    if ((code == B200_BF16 || code == B200_F16) && T > 0 && k > 0 && ti->size(0) == T && is_2d(*tw, T, k) &&
        w1->size(2) == H && is_3d(*w2, E, H, I) && is_3d(*s1, E, cdiv(2 * I, 128), cdiv(H, 128)) &&
        is_3d(*s2, E, cdiv(H, 128), cdiv(I, 128)) && !(inplace && no_combine) && (!on_input || k == 1)) {
      Tensor out;
      if (inplace) out = *x;
      int rc;
      {
        WithoutInterpreterLock unlocked;
        if (!inplace) out = no_combine ? empty_on(dev, {T, k, H}, x->scalar_type()) : empty_on(dev, {T, H}, x->scalar_type());
        void* st = stream_of(dev);
        const size_t need = abi.experts_ws(T, (int)k, (int)E, H, I);
        const Lease lease(dev, st, need);
        rc = abi.experts(x->data_ptr(), nullptr, code, w1->data_ptr(), w2->data_ptr(), s1->data_ptr<float>(),
                         s2->data_ptr<float>(), tw->data_ptr<float>(), ti->data_ptr<int>(), out.data_ptr(), T, (int)k, (int)E, H,
                         I, no_combine, on_input, (float)scale, lease.ptr, need, st);
      }
      if (rc) return fail(rc, "fused_experts");
      return THPVariable_Wrap(std::move(out));
    }
  }
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// route(logits, bias or None, topk, scoring, groups, topk_group, group_score, renormalize, scale) -> (weights, ids)
PyObject* route(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 9) Py_RETURN_NONE;
  const int dev = c10::cuda::current_device();
  const Tensor* x = plain(args[0], dev);
  const bool biased = args[1] != Py_None;
  const Tensor* bias = biased ? plain(args[1], dev, at::kFloat) : nullptr;
  long v[5];
  for (int i = 0; i < 5; ++i) v[i] = args[2 + i] == Py_None ? 0 : PyLong_AsLong(args[2 + i]);
  const bool renormalize = args[7] == Py_True;
  const double scale = PyFloat_AsDouble(args[8]);
  if (PyErr_Occurred() || !x || x->dim() != 2 || !x->is_contiguous() || v[0] <= 0 || x->size(0) == 0 ||
      dtype_code(x->scalar_type()) < 0 || (biased && (!bias || bias->numel() != x->size(1)))) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  const int64_t T = x->size(0);
  Tensor w, ids;
  int rc;
  {
    WithoutInterpreterLock unlocked;
    w = empty_on(dev, {T, v[0]}, at::kFloat);
    ids = empty_on(dev, {T, v[0]}, at::kInt);
    rc = abi.route(x->data_ptr(), dtype_code(x->scalar_type()), bias ? bias->data_ptr<float>() : nullptr, T, (int)x->size(1),
                   (int)v[0], (int)v[1], (int)v[2], (int)v[3], (int)v[4], renormalize, (float)scale, nullptr,
                   w.data_ptr<float>(), ids.data_ptr<int>(), stream_of(dev));
  }
  if (rc) return fail(rc, "route_topk");
  return pair(std::move(w), std::move(ids));
  END_HANDLE_TH_ERRORS
}

// scratch(device, bytes): the current stream's scratch buffer as a uint8 tensor of at least that size
PyObject* scratch_tensor(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 2) return PyErr_Format(PyExc_TypeError, "scratch(device, bytes)");
  const long dev = PyLong_AsLong(args[0]);
  const size_t bytes = PyLong_AsSize_t(args[1]);
  if (PyErr_Occurred()) return nullptr;
  Tensor buf;
  {
    WithoutInterpreterLock unlocked;
    Scratch& s = scratch_of((int)dev, stream_of((int)dev));
    std::lock_guard<std::mutex> guard(s.busy);
    grow(s, bytes);
    buf = s.buf;
  }
  return THPVariable_Wrap(std::move(buf));
  END_HANDLE_TH_ERRORS
}

// acquire(device, bytes): the same, kept from every other call that uses this scratch until release(device)
PyObject* acquire(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 2) return PyErr_Format(PyExc_TypeError, "acquire(device, bytes)");
  const long dev = PyLong_AsLong(args[0]);
  const size_t bytes = PyLong_AsSize_t(args[1]);
  if (PyErr_Occurred()) return nullptr;
  Tensor buf;
  {
    WithoutInterpreterLock unlocked;
    Scratch& s = scratch_of((int)dev, stream_of((int)dev));
    std::unique_lock<std::mutex> lock(s.busy);
    grow(s, bytes);
    buf = s.buf;
    lock.release();  // stays locked
  }
  return THPVariable_Wrap(std::move(buf));
  END_HANDLE_TH_ERRORS
}
PyObject* release(PyObject*, PyObject* arg) {
  HANDLE_TH_ERRORS
  const long dev = PyLong_AsLong(arg);
  if (PyErr_Occurred()) return nullptr;
  scratch_of((int)dev, stream_of((int)dev)).busy.unlock();
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

// bind(path of the C-ABI library)
PyObject* bind(PyObject*, PyObject* arg) {
  const char* path = PyUnicode_AsUTF8(arg);
  if (!path) return nullptr;
  void* lib = dlopen(path, RTLD_NOW | RTLD_LOCAL);
  if (!lib) return PyErr_Format(PyExc_ImportError, "%s", dlerror());
  bool ok = true;
  auto get = [&](auto& fn, const char* name) {
    fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(lib, name));
    ok = ok && fn != nullptr;
  };
  get(abi.status_string, "b200_status_string");
  get(abi.last_error_detail, "b200_last_error_detail");
  get(abi.get_tuning, "b200_get_tuning");
  get(abi.quant, "b200_per_token_group_quant_fp8");
  get(abi.quant_ue8m0, "b200_per_token_group_quant_fp8_ue8m0");
  get(abi.gemm_ws, "b200_w8a8_block_fp8_gemm_workspace_bytes");
  get(abi.gemm, "b200_w8a8_block_fp8_gemm");
  get(abi.packed_ws, "b200_w8a8_block_fp8_gemm_packed_workspace_bytes");
  get(abi.packed, "b200_w8a8_block_fp8_gemm_packed");
  get(abi.linear_ws, "b200_w8a8_block_fp8_linear_workspace_bytes");
  get(abi.linear, "b200_w8a8_block_fp8_linear");
  get(abi.experts_ws, "b200_fused_experts_fp8_workspace_bytes");
  get(abi.experts, "b200_fused_experts_fp8");
  get(abi.route, "b200_route_topk");
  if (!ok) return PyErr_Format(PyExc_ImportError, "%s lacks a symbol of its header", path);
  Py_RETURN_NONE;
}

#define FAST(fn) reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(fn)), METH_FASTCALL
PyMethodDef methods[] = {
    {"bind", bind, METH_O, nullptr},          {"linear", FAST(linear), nullptr},
    {"quant", FAST(quant), nullptr},          {"matmul", FAST(matmul), nullptr},
    {"matmul_ue8m0", FAST(matmul_ue8m0), nullptr}, {"experts", FAST(experts), nullptr},
    {"route", FAST(route), nullptr},          {"scratch", FAST(scratch_tensor), nullptr},
    {"acquire", FAST(acquire), nullptr},      {"release", release, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", "Native host path of the block-FP8 operators.", -1, methods,
                      nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host() { return PyModule_Create(&module); }
