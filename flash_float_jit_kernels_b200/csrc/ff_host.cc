// Host path of the public operators: argument checks, output allocation, workspace lookup and the call
// into the C ABI, in one native function per operator.
//
// Why: a decode-step select takes about 10 us on the GPU, and the same steps written in Python
// (some forty tensor attribute reads, torch.empty, a 17-argument ctypes call) took 15-20 us per call, so
// eager calls were bound by the host.  Here they take about 4 us, of which about half is the launch.
//
// Every function returns None when an argument is not of the plain, valid kind it handles; the Python
// layer then runs the full checks, which raise the documented errors (or handle the rare kinds,
// such as tensor subclasses).  C++ exceptions leave as the Python ones torch maps them to (an allocation that does
// not fit is torch.OutOfMemoryError).  The C ABI functions are bound by address (bind()), so that this module
// uses the very library instance ctypes has loaded, whatever its build knobs.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <limits>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

#include "../../include/ff_indexer_logits.h"
#include "../../include/ff_topk.h"

namespace {

decltype(&ff_topk_launch_typed) p_typed = nullptr;
decltype(&ff_topk_launch_handover) p_handover = nullptr;
decltype(&ff_topk_transform_launch) p_transform = nullptr;
decltype(&ff_topk_workspace_bytes) p_workspace_bytes = nullptr;
decltype(&ff_indexer_logits_launch_fresh) p_logits = nullptr;
PyObject* g_on_error = nullptr;   // Python callable (return code, operator name): raises

using at::Tensor;

// The tensor behind `o` if it is a plain CUDA tensor.
inline const Tensor* cuda_tensor(PyObject* o) {
  if (!THPVariable_CheckExact(o)) return nullptr;
  const Tensor& t = THPVariable_Unpack(o);
  return t.is_cuda() && t.layout() == at::kStrided ? &t : nullptr;
}
inline bool is_none(PyObject* o) { return o == Py_None; }

// A contiguous vector of n elements of `type` on `dev`.
inline const Tensor* vector_of(PyObject* o, int64_t n, at::ScalarType type, c10::Device dev) {
  const Tensor* t = cuda_tensor(o);
  if (t == nullptr || t->dim() != 1 || t->size(0) != n || t->scalar_type() != type || t->device() != dev ||
      !t->is_contiguous())
    return nullptr;
  return t;
}

// ---- zero-filled scratch of split rows ----
// The kernels leave it zeroed, and no two launches that may overlap on the GPU share it:
//   * a call in plain stream order takes the buffer of its (device, stream), grown on demand; the number of streams
//     bounds the map, and a buffer that was replaced is reused in stream order;
//   * a call under stream capture takes a buffer of its (capture, stream), filled at once on a stream of its own, because
//     a fill that were only recorded would not have run for another graph or an eager call, and its own, because graphs
//     captured one after the other on one stream may be replayed side by side on two.  When the graph goes is not known
//     here, so the buffers of the first captures, 64 MiB of them per device, are kept; those of later ones are handed to
//     the graph, which returns them with its end but takes 6 us longer per replay (24 selects of 1 Mi columns: 12.61 instead
//     of 12.36 us each).
constexpr int64_t kKeptForCaptures = 64 << 20;
std::mutex g_returned_mutex;
std::vector<Tensor*>& g_returned = *new std::vector<Tensor*>();   // of destroyed graphs, given back by the next call

// Called by the CUDA runtime when the last graph that holds the buffer is gone (no CUDA call is allowed here).
void CUDART_CB return_scratch(void* t) {
  const std::lock_guard<std::mutex> lock(g_returned_mutex);
  g_returned.push_back(static_cast<Tensor*>(t));
}

Tensor zeroed(int64_t bytes, c10::Device dev, cudaStream_t stream) {
  Tensor t = at::empty({bytes}, at::TensorOptions().dtype(at::kByte).device(dev));
  C10_CUDA_CHECK(cudaMemsetAsync(t.data_ptr(), 0, static_cast<size_t>(bytes), stream));
  return t;
}

// A buffer that is zero when this returns and belongs to no capture, whatever the calling thread is capturing.
Tensor zeroed_outside_capture(int64_t bytes, c10::Device dev) {
  const c10::cuda::CUDAStreamCaptureModeGuard relaxed(cudaStreamCaptureModeRelaxed);
  static auto& streams = *new std::map<int, cudaStream_t>();   // one per device; guarded by the GIL
  cudaStream_t& side = streams[dev.index()];
  if (side == nullptr) C10_CUDA_CHECK(cudaStreamCreateWithFlags(&side, cudaStreamNonBlocking));
  const c10::cuda::CUDAStreamGuard guard(c10::cuda::getStreamFromExternal(side, dev.index()));
  Tensor t = zeroed(bytes, dev, side);
  C10_CUDA_CHECK(cudaStreamSynchronize(side));
  return t;
}

// `dev` is the current device.
Tensor scratch_for(c10::Device dev, cudaStream_t stream, int64_t need) {
  {
    std::vector<Tensor*> returned;
    {
      const std::lock_guard<std::mutex> lock(g_returned_mutex);
      returned.swap(g_returned);
    }
    for (Tensor* t : returned) delete t;
  }
  const std::pair<int, cudaStream_t> key{dev.index(), stream};
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo(stream, &status, &id, &graph) != cudaSuccess) {
    (void)cudaGetLastError();   // (the legacy stream beside a capture on a blocking one: the launch will say so)
    status = cudaStreamCaptureStatusNone;
  }
  if (status == cudaStreamCaptureStatusActive) {
    struct Captured {
      unsigned long long id = 0;    // ids are not used twice
      Tensor* scratch = nullptr;    // kept, or the graph's and valid while `id` is being captured
    };
    static auto& captured = *new std::map<std::pair<int, cudaStream_t>, Captured>();   // guarded by the GIL
    Captured& c = captured[key];
    if (c.scratch != nullptr && c.id == id && c.scratch->numel() >= need) return *c.scratch;
    Tensor* scratch = new Tensor(zeroed_outside_capture(need, dev));
    static auto& kept_bytes = *new std::map<int, int64_t>();   // by device; guarded by the GIL
    if (kept_bytes[dev.index()] + need <= kKeptForCaptures) {
      kept_bytes[dev.index()] += need;
    } else {
      cudaUserObject_t object;
      const cudaError_t e = cudaUserObjectCreate(&object, scratch, return_scratch, 1, cudaUserObjectNoDestructorSync);
      if (e != cudaSuccess) delete scratch;
      C10_CUDA_CHECK(e);
      C10_CUDA_CHECK(cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove));
    }
    c = {id, scratch};
    return *scratch;
  }
  static auto& kept = *new std::map<std::pair<int, cudaStream_t>, Tensor>();   // guarded by the GIL
  Tensor& t = kept[key];
  if (!t.defined() || t.numel() < need) t = zeroed(need, dev, stream);
  return t;
}

struct Workspace {
  void* ptr = nullptr;
  size_t bytes = 0;
  Tensor keep;   // holds the memory while the launch is enqueued without the GIL
};

void workspace_for(c10::Device dev, cudaStream_t stream, int64_t B, int64_t L, int64_t k, Workspace& ws) {
  const size_t need = p_workspace_bytes(static_cast<int32_t>(B), L, static_cast<int32_t>(k));
  if (need == 0) return;
  ws.keep = scratch_for(dev, stream, static_cast<int64_t>(need));
  ws.ptr = ws.keep.data_ptr();
  ws.bytes = static_cast<size_t>(ws.keep.numel());
}

PyObject* report(int rc, const char* what) {
  PyObject* r = PyObject_CallFunction(g_on_error, "is", rc, what);
  if (r != nullptr) {
    Py_DECREF(r);
    PyErr_SetString(PyExc_RuntimeError, what);
  }
  return nullptr;
}

inline int score_type(at::ScalarType t) {
  return t == at::kFloat ? FF_DTYPE_F32 : t == at::kBFloat16 ? FF_DTYPE_BF16 : t == at::kHalf ? FF_DTYPE_F16 : -1;
}

struct Scores {
  const Tensor* score = nullptr;
  const Tensor* lengths = nullptr;
  const Tensor* row_starts = nullptr;
  int64_t B = 0, L = 0, row_stride = 0;
};

// The arguments all selects share; false: not of the plain valid kind.
bool take_scores(PyObject* score, PyObject* lengths, PyObject* row_starts, int64_t k, Scores& s) {
  if (k < 1 || k > FF_TOPK_MAX_K) return false;
  s.score = cuda_tensor(score);
  if (s.score == nullptr || s.score->dim() != 2) return false;
  s.B = s.score->size(0);
  s.L = s.score->size(1);
  if (s.B < 1 || s.L < 1 || s.B > std::numeric_limits<int32_t>::max() || s.score->stride(1) != 1) return false;
  const c10::Device dev = s.score->device();
  s.lengths = vector_of(lengths, s.B, at::kInt, dev);
  if (s.lengths == nullptr) return false;
  if (!is_none(row_starts)) {
    s.row_starts = vector_of(row_starts, s.B, at::kInt, dev);
    if (s.row_starts == nullptr) return false;
  }
  s.row_stride = s.score->stride(0);
  if (s.B == 1 && s.row_stride < s.L) s.row_stride = s.L;
  return true;
}

// status word: the Python layer passes its address on unchecked, so any CUDA tensor with room for it will do
inline bool take_status(PyObject* o, int32_t*& p) {
  p = nullptr;
  if (is_none(o)) return true;
  const Tensor* t = cuda_tensor(o);
  if (t == nullptr) return false;
  p = static_cast<int32_t*>(t->data_ptr());
  return true;
}

template <typename F>
int without_gil(F&& f) {
  int rc;
  Py_BEGIN_ALLOW_THREADS;
  rc = f();
  Py_END_ALLOW_THREADS;
  return rc;
}

// select(): the launch behind fast_topk_v3 and the second half of indexer_topk.  Returns a new
// reference to the result, None when the arguments need the Python layer, nullptr on error.
PyObject* select(PyObject* py_score, PyObject* py_lengths, int64_t k, PyObject* py_row_starts, PyObject* py_out,
                 PyObject* py_status, PyObject* py_hint, PyObject* py_index_dtype, PyObject* py_handover,
                 const char* what) {
  Scores s;
  if (!take_scores(py_score, py_lengths, py_row_starts, k, s)) Py_RETURN_NONE;
  const c10::Device dev = s.score->device();
  const int dtype = score_type(s.score->scalar_type());
  if (dtype < 0) Py_RETURN_NONE;
  int32_t* status;
  if (!take_status(py_status, status)) Py_RETURN_NONE;
  float* hint = nullptr;
  if (!is_none(py_hint)) {
    const Tensor* t = vector_of(py_hint, s.B, at::kFloat, dev);
    if (t == nullptr) Py_RETURN_NONE;
    hint = static_cast<float*>(t->data_ptr());
  }
  Tensor fresh;
  const Tensor* out;
  if (is_none(py_out)) {
    if (!THPDtype_Check(py_index_dtype)) Py_RETURN_NONE;
    const at::ScalarType it = reinterpret_cast<THPDtype*>(py_index_dtype)->scalar_type;
    if (it != at::kInt && it != at::kLong) Py_RETURN_NONE;
    fresh = at::empty({s.B, k}, at::TensorOptions().dtype(it).device(dev));
    out = &fresh;
  } else {
    out = cuda_tensor(py_out);
    if (out == nullptr || out->dim() != 2 || out->size(0) != s.B || out->size(1) != k || out->device() != dev ||
        !out->is_contiguous() || (out->scalar_type() != at::kInt && out->scalar_type() != at::kLong))
      Py_RETURN_NONE;
  }
  const int index_bits = out->scalar_type() == at::kLong ? 64 : 32;
  void* handover = nullptr;
  if (!is_none(py_handover)) {
    const Tensor* t = cuda_tensor(py_handover);
    if (t == nullptr || hint == nullptr || dtype != FF_DTYPE_F32 || index_bits != 32 || t->scalar_type() != at::kByte ||
        t->device() != dev || !t->is_contiguous() || t->numel() < s.B * FF_TOPK_HANDOVER_ROW_BYTES)
      Py_RETURN_NONE;
    handover = t->data_ptr();
  }
  const c10::cuda::OptionalCUDAGuard guard(dev);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  Workspace ws;
  workspace_for(dev, stream, s.B, s.L, k, ws);
  const int32_t* row_starts = s.row_starts == nullptr ? nullptr : static_cast<const int32_t*>(s.row_starts->data_ptr());
  const void* scores = s.score->data_ptr();
  const int32_t* lengths = static_cast<const int32_t*>(s.lengths->data_ptr());
  void* out_ptr = out->data_ptr();
  const int rc = without_gil([&] {
    if (handover != nullptr)
      return p_handover(static_cast<const float*>(scores), s.row_stride, lengths, row_starts, static_cast<int32_t*>(out_ptr),
                        static_cast<int32_t>(s.B), s.L, static_cast<int32_t>(k), hint, hint, handover, ws.ptr, ws.bytes,
                        status, stream);
    return p_typed(scores, dtype, s.row_stride, lengths, row_starts, out_ptr, index_bits, static_cast<int32_t>(s.B), s.L,
                   static_cast<int32_t>(k), hint, hint, ws.ptr, ws.bytes, status, stream);
  });
  if (rc != 0) return report(rc, what);
  if (out == &fresh) return THPVariable_Wrap(std::move(fresh));
  Py_INCREF(py_out);
  return py_out;
}

bool take_k(PyObject* o, int64_t& k) {
  if (!PyLong_Check(o)) return false;
  int overflow = 0;
  k = PyLong_AsLongLongAndOverflow(o, &overflow);
  return overflow == 0;
}

// topk(score, lengths, topk, row_starts, out, status, threshold_hint, index_dtype, handover)
PyObject* py_topk(PyObject*, PyObject* const* a, Py_ssize_t n) {
  int64_t k;
  if (n != 9 || !take_k(a[2], k)) Py_RETURN_NONE;
  HANDLE_TH_ERRORS
  return select(a[0], a[1], k, a[3], a[4], a[5], a[6], a[7], a[8], "fast_topk_v3");
  END_HANDLE_TH_ERRORS
}

// transform(score, lengths, out, row_starts, table, cu_seqlens, offset): table and cu_seqlens for the
// page-table gather, offset for the per-row offset; True when launched
PyObject* py_transform(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 7) Py_RETURN_NONE;
  HANDLE_TH_ERRORS
  const Tensor* out = cuda_tensor(a[2]);
  if (out == nullptr || out->dim() != 2 || !out->is_contiguous() || out->scalar_type() != at::kInt) Py_RETURN_NONE;
  const int64_t k = out->size(1);
  Scores s;
  if (!take_scores(a[0], a[1], a[3], k, s) || s.score->scalar_type() != at::kFloat || out->size(0) != s.B) Py_RETURN_NONE;
  const c10::Device dev = s.score->device();
  if (out->device() != dev) Py_RETURN_NONE;
  const bool pages = !is_none(a[4]);
  const int32_t *table = nullptr, *cu = nullptr, *offsets = nullptr;
  int64_t table_stride = 0, requests = 0;
  if (pages) {
    const Tensor* t = cuda_tensor(a[4]);
    const Tensor* c = cuda_tensor(a[5]);
    if (t == nullptr || c == nullptr || t->dim() != 2 || t->scalar_type() != at::kInt || t->stride(1) != 1 ||
        t->device() != dev || c->dim() != 1)
      Py_RETURN_NONE;
    requests = c->size(0) - 1;
    if (vector_of(a[5], requests + 1, at::kInt, dev) == nullptr || t->size(0) != requests || requests > s.B || requests < 1)
      Py_RETURN_NONE;
    table = static_cast<const int32_t*>(t->data_ptr());
    table_stride = t->stride(0);
    if (!(s.row_starts == nullptr && requests == s.B)) cu = static_cast<const int32_t*>(c->data_ptr());
  } else {
    const Tensor* o = vector_of(a[6], s.B, at::kInt, dev);
    if (o == nullptr) Py_RETURN_NONE;
    offsets = static_cast<const int32_t*>(o->data_ptr());
  }
  const c10::cuda::OptionalCUDAGuard guard(dev);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  Workspace ws;
  workspace_for(dev, stream, s.B, s.L, k, ws);
  const float* scores = static_cast<const float*>(s.score->data_ptr());
  const int32_t* lengths = static_cast<const int32_t*>(s.lengths->data_ptr());
  const int32_t* row_starts = s.row_starts == nullptr ? nullptr : static_cast<const int32_t*>(s.row_starts->data_ptr());
  int32_t* out_ptr = static_cast<int32_t*>(out->data_ptr());
  const int rc = without_gil([&] {
    return p_transform(scores, s.row_stride, lengths, row_starts, out_ptr, static_cast<int32_t>(s.B), s.L,
                       static_cast<int32_t>(k), pages ? FF_EPILOGUE_PAGE_TABLE : FF_EPILOGUE_ADD_OFFSET, table,
                       table_stride, cu, static_cast<int32_t>(pages ? requests : 0), offsets, ws.ptr, ws.bytes, nullptr,
                       stream);
  });
  if (rc != 0) return report(rc, pages ? "fast_topk_transform_fused" : "fast_topk_transform_ragged_fused");
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// The logits launch; returns a new reference like select().
PyObject* logits(PyObject* py_q, PyObject* py_k, PyObject* py_w, PyObject* py_lengths, PyObject* py_out,
                 PyObject* py_status, int64_t ctas_per_row, PyObject* py_hint, PyObject* py_handover) {
  constexpr int64_t kHeads = 64, kDim = 128;
  const Tensor *q = cuda_tensor(py_q), *keys = cuda_tensor(py_k), *w = cuda_tensor(py_w);
  if (q == nullptr || keys == nullptr || w == nullptr) Py_RETURN_NONE;
  if (q->dim() != 3 || keys->dim() != 3 || w->dim() != 2 || q->element_size() != 1 || keys->element_size() != 1) Py_RETURN_NONE;
  const int64_t B = q->size(0), L = keys->size(1);
  const c10::Device dev = q->device();
  if (B < 1 || L < 1 || q->size(1) != kHeads || q->size(2) != kDim || !q->is_contiguous() || keys->size(0) != B ||
      keys->size(2) != kDim || keys->stride(2) != 1 || keys->stride(1) != kDim || keys->device() != dev ||
      w->size(0) != B || w->size(1) != kHeads || w->scalar_type() != at::kFloat || !w->is_contiguous() || w->device() != dev ||
      B > std::numeric_limits<int32_t>::max() || L > std::numeric_limits<int32_t>::max())
    Py_RETURN_NONE;
  const Tensor* lengths = vector_of(py_lengths, B, at::kInt, dev);
  int32_t* status;
  if (lengths == nullptr || !take_status(py_status, status)) Py_RETURN_NONE;
  const float* hint = nullptr;
  void* handover = nullptr;
  if (!is_none(py_handover)) {
    const Tensor* h = vector_of(py_hint, B, at::kFloat, dev);
    const Tensor* t = cuda_tensor(py_handover);
    if (h == nullptr || t == nullptr || t->scalar_type() != at::kByte || t->device() != dev || !t->is_contiguous() ||
        t->numel() < B * FF_TOPK_HANDOVER_ROW_BYTES)
      Py_RETURN_NONE;
    hint = static_cast<const float*>(h->data_ptr());
    handover = t->data_ptr();
  }
  Tensor fresh;
  const Tensor* out;
  bool fill = false;
  if (is_none(py_out)) {
    // the kernel writes the -inf behind the rows' ends itself where it can (a fill kernel of its own: 5 us for 64 x 128 Ki)
    const auto options = at::TensorOptions().dtype(at::kFloat).device(dev);
    fill = ctas_per_row == 0 && B <= FF_INDEXER_MAX_FILL_ROWS && (B == 1 || keys->stride(0) < (int64_t{1} << 40));
    fresh = fill ? at::empty({B, L}, options) : at::full({B, L}, -std::numeric_limits<float>::infinity(), options);
    out = &fresh;
  } else {
    out = cuda_tensor(py_out);
    if (out == nullptr || out->dim() != 2 || out->size(0) != B || out->size(1) != L || out->scalar_type() != at::kFloat ||
        out->stride(1) != 1 || out->device() != dev)
      Py_RETURN_NONE;
  }
  const c10::cuda::OptionalCUDAGuard guard(dev);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const int64_t k_stride = B > 1 ? keys->stride(0) : std::max(keys->stride(0), L * kDim);
  const int64_t out_stride = B > 1 ? out->stride(0) : std::max(out->stride(0), L);
  const void *q_ptr = q->data_ptr(), *k_ptr = keys->data_ptr();
  const float* w_ptr = static_cast<const float*>(w->data_ptr());
  const int32_t* len_ptr = static_cast<const int32_t*>(lengths->data_ptr());
  float* out_ptr = static_cast<float*>(out->data_ptr());
  const int rc = without_gil([&] {
    return p_logits(q_ptr, k_ptr, k_stride, w_ptr, len_ptr, out_ptr, out_stride, static_cast<int32_t>(B),
                    static_cast<int32_t>(L), static_cast<int32_t>(ctas_per_row), fill ? 1 : 0, hint, handover, status, stream);
  });
  if (rc != 0) return report(rc, "indexer_logits_fp8");
  if (out == &fresh) return THPVariable_Wrap(std::move(fresh));
  Py_INCREF(py_out);
  return py_out;
}

// logits(q, k, w, lengths, out, status, ctas_per_row, threshold_hint, handover)
PyObject* py_logits(PyObject*, PyObject* const* a, Py_ssize_t n) {
  int64_t ctas;
  if (n != 9 || !take_k(a[6], ctas) || ctas > 65535 || ctas < -65535) Py_RETURN_NONE;
  HANDLE_TH_ERRORS
  return logits(a[0], a[1], a[2], a[3], a[4], a[5], ctas, a[7], a[8]);
  END_HANDLE_TH_ERRORS
}

// scratch(device index, bytes): zero-filled scratch for a launch on the device's current stream
PyObject* py_scratch(PyObject*, PyObject* const* a, Py_ssize_t n) {
  int64_t device, bytes;
  if (n != 2 || !take_k(a[0], device) || !take_k(a[1], bytes) || device < 0 || device > 127 || bytes < 1) {
    PyErr_SetString(PyExc_TypeError, "scratch(device index, bytes)");
    return nullptr;
  }
  HANDLE_TH_ERRORS
  const c10::Device dev(c10::kCUDA, static_cast<c10::DeviceIndex>(device));
  const c10::cuda::OptionalCUDAGuard guard(dev);
  return THPVariable_Wrap(scratch_for(dev, c10::cuda::getCurrentCUDAStream(dev.index()).stream(), bytes));
  END_HANDLE_TH_ERRORS
}

// bind(name, address): the C ABI functions of the loaded libraries; bind("on_error", callable)
PyObject* py_bind(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != 2 || !PyUnicode_Check(a[0])) {
    PyErr_SetString(PyExc_TypeError, "bind(name, address)");
    return nullptr;
  }
  const char* name = PyUnicode_AsUTF8(a[0]);
  if (strcmp(name, "on_error") == 0) {
    Py_INCREF(a[1]);
    Py_XSETREF(g_on_error, a[1]);
    Py_RETURN_NONE;
  }
  void* p = PyLong_AsVoidPtr(a[1]);
  if (p == nullptr) {
    if (!PyErr_Occurred()) PyErr_SetString(PyExc_ValueError, "bind: null address");
    return nullptr;
  }
  if (strcmp(name, "ff_topk_launch_typed") == 0) p_typed = reinterpret_cast<decltype(p_typed)>(p);
  else if (strcmp(name, "ff_topk_launch_handover") == 0) p_handover = reinterpret_cast<decltype(p_handover)>(p);
  else if (strcmp(name, "ff_topk_transform_launch") == 0) p_transform = reinterpret_cast<decltype(p_transform)>(p);
  else if (strcmp(name, "ff_topk_workspace_bytes") == 0) p_workspace_bytes = reinterpret_cast<decltype(p_workspace_bytes)>(p);
  else if (strcmp(name, "ff_indexer_logits_launch_fresh") == 0) p_logits = reinterpret_cast<decltype(p_logits)>(p);
  else {
    PyErr_SetString(PyExc_ValueError, "bind: unknown name");
    return nullptr;
  }
  Py_RETURN_NONE;
}

PyMethodDef kMethods[] = {
    {"bind", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_bind)), METH_FASTCALL, nullptr},
    {"scratch", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_scratch)), METH_FASTCALL, nullptr},
    {"topk", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_topk)), METH_FASTCALL, nullptr},
    {"transform", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_transform)), METH_FASTCALL, nullptr},
    {"logits", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_logits)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "ff_host", nullptr, -1, kMethods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit_ff_host(void) { return PyModule_Create(&kModule); }
