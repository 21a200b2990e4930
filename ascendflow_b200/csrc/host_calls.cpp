// The host side of a call in native code: what `ops.sparse_mla`, `neighbours.topk_indices`,
// `neighbours.cache_append` and the registered torch op do between the user's call and the launch.
//
// The checks of the Python front end (runtime/signature.py) on thirteen tensors cost 60-70 us per
// call, more than a decode step's kernel takes. Here the same conditions are tested on the tensors'
// C++ objects (about 2 us with the launch). A call that passes is launched through the C ABI; for
// one that does not, the functions return None without having enqueued anything, and the caller goes
// through the Python front end, which finds the violated rule again and raises its error. So
// nothing here words an error, and nothing is accepted that the front end would refuse.

#include <Python.h>

#include <ATen/FuncTorchTLS.h>
#include <ATen/core/Tensor.h>
#include <ATen/core/grad_mode.h>
#include <ATen/ops/empty.h>
#include <ATen/ops/zeros.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/VariableTypeUtils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include <cuda_runtime_api.h>

#include <algorithm>
#include <array>
#include <mutex>
#include <utility>
#include <vector>

#include "../../include/sparse_mla.h"

namespace {

constexpr int kTensors = SPARSE_MLA_TENSORS;
using Tensors = std::array<const at::Tensor*, kTensors>;
enum Argument { kQ, kOriKv, kCmpKv, kIndices, kOriTable, kCmpTable, kCu, kSeqOri, kSeqCmp, kResidual, kTopkLength, kSinks, kOut };

using LaunchAttention = decltype(&launch_sparse_mla_kept_status);
using LaunchSelect = decltype(&launch_sparse_mla_topk_indices);
using LaunchAppend = decltype(&launch_sparse_mla_cache_append_flagged);

// Entry points of the kernel library (loaded, and its hash verified, by the Python side).
LaunchAttention launch_attention = nullptr;
LaunchSelect launch_select = nullptr;
LaunchAppend launch_append = nullptr;
PyObject* checked_attention = nullptr;  // the Python front end's call, for arguments refused here

PyObject* raise_launch_status(int status) {
  PyErr_Format(PyExc_RuntimeError, "kernel launch failed with status %d; device retries are disabled", status);
  return nullptr;
}

// A plain strided, contiguous CUDA tensor of one type on one device.
bool plain(const at::Tensor& t, at::ScalarType type, int device) {
  return t.defined() && t.layout() == at::kStrided && t.is_cuda() && t.device().index() == device && t.scalar_type() == type &&
         t.is_contiguous();
}

bool shaped(const at::Tensor& t, std::initializer_list<int64_t> sizes) {
  return t.dim() == int64_t(sizes.size()) && std::equal(sizes.begin(), sizes.end(), t.sizes().begin());
}

struct Sizes {
  int64_t batches, tokens, pages, ori_blocks, cmp_blocks, cmp_page;
};

// The conditions of the operator's signature: types, placement, shapes, disjoint memory.
bool accepted(const Tensors& t, int device, Sizes* s) {
  const at::Tensor& q = *t[kQ];
  if (!q.defined() || q.dim() != 3) return false;
  const at::ScalarType type = q.scalar_type();
  if (type != at::kBFloat16 && type != at::kHalf) return false;
  for (int i = 0; i < kTensors; ++i) {
    const bool stored = i == kQ || i == kOriKv || i == kCmpKv || i == kOut;
    if (!plain(*t[i], stored ? type : i == kSinks ? at::kFloat : at::kInt, device)) return false;
  }
  if (t[kOriTable]->dim() != 2 || t[kOriKv]->dim() != 4 || t[kCmpKv]->dim() != 4) return false;
  *s = {t[kOriTable]->size(0), q.size(0), t[kOriTable]->size(1), t[kOriKv]->size(0), t[kCmpKv]->size(0), t[kCmpKv]->size(1)};
  if (s->batches < 1 || s->tokens < 1 || s->pages < 1 || s->ori_blocks < 1 || s->cmp_blocks < 1 || s->cmp_page < 64 ||
      s->cmp_page % 64 != 0)
    return false;
  const bool shapes = shaped(q, {s->tokens, 64, 512}) && shaped(*t[kOut], {s->tokens, 64, 512}) &&
                      shaped(*t[kOriKv], {s->ori_blocks, 128, 1, 512}) && shaped(*t[kCmpKv], {s->cmp_blocks, s->cmp_page, 1, 512}) &&
                      shaped(*t[kIndices], {s->tokens, 1, 512}) && shaped(*t[kCmpTable], {s->batches, s->pages}) &&
                      shaped(*t[kCu], {s->batches + 1}) && shaped(*t[kSeqOri], {s->batches}) && shaped(*t[kSeqCmp], {s->batches}) &&
                      shaped(*t[kResidual], {s->batches}) && shaped(*t[kTopkLength], {s->tokens, 1}) && shaped(*t[kSinks], {64});
  if (!shapes) return false;
  std::array<std::pair<uintptr_t, uintptr_t>, kTensors> spans;
  for (int i = 0; i < kTensors; ++i) {
    const uintptr_t begin = reinterpret_cast<uintptr_t>(t[i]->const_data_ptr());
    spans[i] = {begin, begin + t[i]->nbytes()};
  }
  std::sort(spans.begin(), spans.end());
  for (int i = 1; i < kTensors; ++i)
    if (spans[i].first < spans[i - 1].second) return false;
  return true;
}

// Allocations in a call that may run while another thread (or this one) captures a stream.
struct RelaxedCapture {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
};

// One status block per device and stream, kept (and zero: no call clears it, `read_status` does). At most
// kMostWorkspaces of them: a program that makes streams without end gets the oldest one's memory back for the
// newest (the allocator holds freed memory until its stream is done with it).
constexpr size_t kWorkspaceBytes = 1024, kMostWorkspaces = 64;
struct Workspace {
  int device;
  cudaStream_t stream;
  at::Tensor memory;
};
std::mutex workspace_mutex;
std::vector<Workspace>* workspaces = new std::vector<Workspace>;  // never destroyed: outlives the CUDA context

// (A copy, so that the memory of a block pushed out meanwhile lives until the launch is enqueued.)
at::Tensor workspace_for(const c10::cuda::CUDAStream& stream) {
  std::lock_guard<std::mutex> lock(workspace_mutex);
  for (const Workspace& w : *workspaces)
    if (w.device == stream.device_index() && w.stream == stream.stream()) return w.memory;
  at::Tensor memory = at::zeros({int64_t(kWorkspaceBytes)}, at::TensorOptions(at::kByte).device(at::kCUDA, stream.device_index()));
  c10::cuda::CUDACachingAllocator::recordStream(memory.storage().data_ptr(), stream);
  if (workspaces->size() >= kMostWorkspaces) workspaces->erase(workspaces->begin());
  workspaces->push_back({stream.device_index(), stream.stream(), memory});
  return memory;
}

// A captured launch runs whenever its graph is replayed, on any stream, for as long as the graph lives. All
// captured launches of a device share one block (its first report counts, as everywhere), which is
// allocated and cleared outside of the capture and never given back.
constexpr int kMostDevices = 64;
std::array<void*, kMostDevices> captured_blocks = {};

cudaError_t captured_block(int device, void** block) {
  if (device < 0 || device >= kMostDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(workspace_mutex);
  cudaError_t error = cudaSuccess;
  if (captured_blocks[device] == nullptr) {
    const RelaxedCapture relaxed;
    cudaStream_t aside = nullptr;  // not the capturing one, and none that waits for it
    void* memory = nullptr;
    error = cudaStreamCreateWithFlags(&aside, cudaStreamNonBlocking);
    if (error == cudaSuccess) error = cudaMalloc(&memory, kWorkspaceBytes);
    if (error == cudaSuccess) error = cudaMemsetAsync(memory, 0, kWorkspaceBytes, aside);
    if (error == cudaSuccess) error = cudaStreamSynchronize(aside);
    if (aside != nullptr) cudaStreamDestroy(aside);
    if (error == cudaSuccess) captured_blocks[device] = memory;
    else if (memory != nullptr) cudaFree(memory);
  }
  *block = captured_blocks[device];
  return error;
}

cudaError_t is_capturing(cudaStream_t stream, bool* capturing) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  const cudaError_t error = cudaStreamIsCapturing(stream, &status);
  *capturing = status != cudaStreamCaptureStatusNone;
  return error;
}

// Launches an accepted call on the current stream. -1000: not accepted, nothing enqueued.
constexpr int kRefused = -1000;
int attention(const Tensors& t) {
  // (Nothing is asked of the CUDA runtime for tensors that are elsewhere: there may be no device.)
  if (launch_attention == nullptr || !t[kQ]->defined() || !t[kQ]->is_cuda()) return kRefused;
  const c10::DeviceIndex device = c10::cuda::current_device();
  Sizes s;
  if (!accepted(t, device, &s)) return kRefused;
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream(device);
  // Arguments allocated on another stream: their memory must not be recycled before this stream is
  // done with it. (Their contents being ready is the caller's business.)
  for (const at::Tensor* tensor : t) c10::cuda::CUDACachingAllocator::recordStream(tensor->storage().data_ptr(), stream);
  void* p[kTensors];
  for (int i = 0; i < kTensors; ++i) p[i] = const_cast<void*>(t[i]->const_data_ptr());
  bool capturing = false;
  if (const cudaError_t error = is_capturing(stream.stream(), &capturing)) return int(error);
  at::Tensor kept;
  void* workspace = nullptr;
  if (!capturing) workspace = (kept = workspace_for(stream)).mutable_data_ptr();
  else if (const cudaError_t error = captured_block(device, &workspace)) return int(error);
  return launch_attention(stream.stream(), t[kQ]->scalar_type() == at::kHalf, p, workspace, s.batches, s.tokens, s.pages, s.ori_blocks,
                          s.cmp_blocks, s.cmp_page);
}

// ---- the registered op -----------------------------------------------------------------------------

void sparse_mla_op(const at::Tensor& q, const at::Tensor& ori_kv, const at::Tensor& cmp_kv, const at::Tensor& indices,
                   const at::Tensor& ori_table, const at::Tensor& cmp_table, const at::Tensor& cu, const at::Tensor& seq_ori,
                   const at::Tensor& seq_cmp, const at::Tensor& residual, const at::Tensor& topk_length,
                   const at::Tensor& sinks, at::Tensor& out) {
  const Tensors tensors = {&q, &ori_kv, &cmp_kv, &indices, &ori_table, &cmp_table, &cu, &seq_ori, &seq_cmp, &residual, &topk_length,
                           &sinks, &out};
  const int status = attention(tensors);
  if (status == 0) return;
  pybind11::gil_scoped_acquire gil;
  PyObject* result = nullptr;
  if (status == kRefused && checked_attention != nullptr) {
    PyObject* arguments = PyTuple_New(kTensors);
    for (int i = 0; i < kTensors; ++i) PyTuple_SET_ITEM(arguments, i, THPVariable_Wrap(*tensors[i]));
    result = PyObject_CallObject(checked_attention, arguments);
    Py_DECREF(arguments);
  } else {
    raise_launch_status(status);
  }
  if (result == nullptr) {
    python_error error;
    error.persist();
    throw error;
  }
  Py_DECREF(result);
}

// The output is written in place: its version counts up, as for any in-place operation (a tensor made in
// inference mode has none). The op has no gradient. Plain autograd leaves the output without one, but
// functorch's transforms would take what they track for a constant and return zeros: refused.
void sparse_mla_mutates(const at::Tensor& q, const at::Tensor& ori_kv, const at::Tensor& cmp_kv, const at::Tensor& indices,
                        const at::Tensor& ori_table, const at::Tensor& cmp_table, const at::Tensor& cu, const at::Tensor& seq_ori,
                        const at::Tensor& seq_cmp, const at::Tensor& residual, const at::Tensor& topk_length,
                        const at::Tensor& sinks, at::Tensor& out) {
  static const auto op =
      c10::Dispatcher::singleton().findSchemaOrThrow("ascendflow_b200::sparse_mla", "").typed<decltype(sparse_mla_op)>();
  if (const auto& functorch = at::functorch::functorchTLSAccessor(); functorch != nullptr && at::GradMode::is_enabled())
    for (const at::Tensor* tensor : std::initializer_list<const at::Tensor*>{&q, &ori_kv, &cmp_kv, &indices, &ori_table, &cmp_table, &cu,
                                                                             &seq_ori, &seq_cmp, &residual, &topk_length, &sinks, &out})
      if (tensor->defined() && tensor->requires_grad()) functorch->checkSupportsCppAutogradFunction();  // throws inside a transform
  {
    at::AutoDispatchBelowADInplaceOrView below;
    op.call(q, ori_kv, cmp_kv, indices, ori_table, cmp_table, cu, seq_ori, seq_cmp, residual, topk_length, sinks, out);
  }
  if (out.defined() && !out.is_inference()) torch::autograd::increment_version(out);
}

TORCH_LIBRARY(ascendflow_b200, m) {
  m.def("sparse_mla(Tensor q, Tensor ori_kv, Tensor cmp_kv, Tensor cmp_sparse_indices, Tensor ori_block_table, "
        "Tensor cmp_block_table, Tensor cu_seqlens_q, Tensor seqused_ori_kv, Tensor seqused_cmp_kv, Tensor cmp_residual_kv, "
        "Tensor ori_topk_length, Tensor sinks, Tensor(a12!) attention_out) -> ()",
        {at::Tag::pt2_compliant_tag});
}
TORCH_LIBRARY_IMPL(ascendflow_b200, CUDA, m) { m.impl("sparse_mla", sparse_mla_op); }
TORCH_LIBRARY_IMPL(ascendflow_b200, ADInplaceOrView, m) { m.impl("sparse_mla", sparse_mla_mutates); }
// No gradient: the output never requires one.
TORCH_LIBRARY_IMPL(ascendflow_b200, Autograd, m) { m.impl("sparse_mla", torch::CppFunction::makeFallthrough()); }

// ---- Python functions --------------------------------------------------------------------------------

// The C++ tensor of an argument; nullptr for anything but a plain torch.Tensor (subclasses may hold
// no memory).
const at::Tensor* tensor_of(PyObject* object) { return THPVariable_CheckExact(object) ? &THPVariable_Unpack(object) : nullptr; }

template <size_t N>
bool tensors_of(PyObject* const* arguments, std::array<const at::Tensor*, N>* tensors) {
  for (size_t i = 0; i < N; ++i)
    if (((*tensors)[i] = tensor_of(arguments[i])) == nullptr) return false;
  return true;
}

PyObject* call_attention(PyObject*, PyObject* const* arguments, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  Tensors tensors;
  if (count != kTensors || !tensors_of(arguments, &tensors)) Py_RETURN_FALSE;
  int status;
  {
    pybind11::gil_scoped_release no_gil;  // the caller holds references to all of them
    status = attention(tensors);
  }
  if (status == kRefused) Py_RETURN_FALSE;
  if (status != 0) return raise_launch_status(status);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// (scores, cu_seqlens_q, seqused_cmp_kv, cmp_residual_kv, ratio, out or None) -> out, or None if refused
PyObject* call_select(PyObject*, PyObject* const* arguments, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  std::array<const at::Tensor*, 4> t;
  if (count != 6 || launch_select == nullptr || !tensors_of(arguments, &t) || !PyLong_CheckExact(arguments[4])) Py_RETURN_NONE;
  int overflow = 0;
  const long ratio = PyLong_AsLongAndOverflow(arguments[4], &overflow);
  if (overflow != 0 || !t[0]->is_cuda()) Py_RETURN_NONE;
  const c10::DeviceIndex device = c10::cuda::current_device();
  if ((ratio != 1 && ratio != 2) || !plain(*t[0], at::kFloat, device) || t[0]->dim() != 2) Py_RETURN_NONE;
  for (int i = 1; i < 4; ++i)
    if (!plain(*t[i], at::kInt, device)) Py_RETURN_NONE;
  const int64_t tokens = t[0]->size(0), span = t[0]->size(1);
  if (t[1]->dim() < 1 || t[2]->dim() < 1) Py_RETURN_NONE;
  const int64_t batches = t[2]->size(0);
  if (t[1]->size(0) != batches + 1) Py_RETURN_NONE;
  at::Tensor out;
  if (arguments[5] == Py_None) {
    out = at::empty({tokens, 1, 512}, t[0]->options().dtype(at::kInt).requires_grad(false));
  } else {
    const at::Tensor* given = tensor_of(arguments[5]);
    if (given == nullptr || !plain(*given, at::kInt, device) || !shaped(*given, {tokens, 1, 512})) Py_RETURN_NONE;
    out = *given;
  }
  int status;
  {
    pybind11::gil_scoped_release no_gil;
    auto pointer = [](const at::Tensor& tensor) { return const_cast<void*>(tensor.const_data_ptr()); };
    status = launch_select(c10::cuda::getCurrentCUDAStream(device).stream(), pointer(*t[0]), pointer(*t[1]), pointer(*t[2]),
                           pointer(*t[3]), pointer(out), batches, tokens, span, 128 / ratio);
  }
  if (status != 0) return raise_launch_status(status);
  if (arguments[5] != Py_None) return Py_NewRef(arguments[5]);
  return THPVariable_Wrap(out);
  END_HANDLE_TH_ERRORS
}

// What one running append needs: the kernel's status block (device, all zero between calls) and a
// word of host memory that the kernel sets when it has written one. A call holds a pair until its
// stream has been waited for, so there are as many as calls run at the same time, at most kMostWorkspaces of
// them kept. Blocks are cleared on the stream of the call that has them, and that stream is waited for before
// another call gets them: a plain cudaMemset runs on the default stream, for which others do not wait.
struct AppendStatus {
  int device;
  int32_t* words;        // device
  volatile int32_t* flag;  // host, mapped
  int32_t* flag_on_device;
};
std::mutex append_mutex;
std::vector<AppendStatus>* append_pool = new std::vector<AppendStatus>;

cudaError_t take_append_status(int device, cudaStream_t stream, AppendStatus* s) {
  {
    std::lock_guard<std::mutex> lock(append_mutex);
    for (size_t i = 0; i < append_pool->size(); ++i)
      if ((*append_pool)[i].device == device) {
        *s = (*append_pool)[i];
        append_pool->erase(append_pool->begin() + i);
        return cudaSuccess;
      }
  }
  const RelaxedCapture relaxed;
  void *words = nullptr, *flag = nullptr, *flag_on_device = nullptr;
  cudaError_t error = cudaMalloc(&words, kWorkspaceBytes);
  if (error == cudaSuccess) error = cudaMemsetAsync(words, 0, kWorkspaceBytes, stream);
  if (error == cudaSuccess) error = cudaHostAlloc(&flag, 64, cudaHostAllocMapped | cudaHostAllocPortable);
  if (error == cudaSuccess) error = cudaHostGetDevicePointer(&flag_on_device, flag, 0);
  if (error != cudaSuccess) {
    if (words != nullptr) cudaFree(words);
    if (flag != nullptr) cudaFreeHost(flag);
    return error;
  }
  *s = {device, static_cast<int32_t*>(words), static_cast<volatile int32_t*>(flag), static_cast<int32_t*>(flag_on_device)};
  *s->flag = 0;
  return cudaSuccess;
}

void free_append_status(const AppendStatus& s) {
  const RelaxedCapture relaxed;
  cudaFree(s.words);
  cudaFreeHost(const_cast<int32_t*>(s.flag));
}

// Launch, wait for the stream, read the status: the status block only travels when there is one.
int append_and_wait(int device, cudaStream_t stream, void* const (&p)[5], int64_t batches, int64_t tokens, int64_t pages,
                    int64_t blocks, int64_t page_rows, int32_t (&words)[SPARSE_MLA_STATUS_WORDS]) {
  AppendStatus s;
  if (cudaError_t error = take_append_status(device, stream, &s)) return int(error);
  std::fill(std::begin(words), std::end(words), 0);
  const int status = launch_append(stream, p[0], p[1], p[2], p[3], p[4], s.words, s.flag_on_device, batches, tokens, pages, blocks, page_rows);
  cudaError_t error = cudaStreamSynchronize(stream);
  if (error == cudaSuccess && *s.flag != 0) {
    error = cudaMemcpyAsync(words, s.words, sizeof(words), cudaMemcpyDeviceToHost, stream);
    if (error == cudaSuccess) error = cudaMemsetAsync(s.words, 0, kWorkspaceBytes, stream);
    if (error == cudaSuccess) error = cudaStreamSynchronize(stream);
    *s.flag = 0;
  }
  if (error == cudaSuccess) {  // (after an error the pair is left alone)
    std::unique_lock<std::mutex> lock(append_mutex);
    const bool kept = append_pool->size() < kMostWorkspaces;
    if (kept) append_pool->push_back(s);
    lock.unlock();
    if (!kept) free_append_status(s);
  }
  return status != 0 ? status : int(error);
}

// (new_rows, cache, block_table, cu_seqlens_q, seqused_kv) -> the status block, or None if refused
PyObject* call_append(PyObject*, PyObject* const* arguments, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  std::array<const at::Tensor*, 5> t;
  if (count != 5 || launch_append == nullptr || !tensors_of(arguments, &t) || !t[0]->is_cuda()) Py_RETURN_NONE;
  const c10::DeviceIndex device = c10::cuda::current_device();
  const at::ScalarType type = t[0]->scalar_type();
  if ((type != at::kBFloat16 && type != at::kHalf) || !plain(*t[0], type, device) || !plain(*t[1], type, device)) Py_RETURN_NONE;
  for (int i = 2; i < 5; ++i)
    if (!plain(*t[i], at::kInt, device)) Py_RETURN_NONE;
  if (t[0]->dim() != 2 || t[0]->size(1) != 512 || t[1]->dim() != 4 || t[1]->size(2) != 1 || t[1]->size(3) != 512 || t[2]->dim() != 2)
    Py_RETURN_NONE;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(device).stream();
  void* p[5];
  for (int i = 0; i < 5; ++i) p[i] = const_cast<void*>(t[i]->const_data_ptr());
  int32_t words[SPARSE_MLA_STATUS_WORDS];
  int status;
  {
    pybind11::gil_scoped_release no_gil;
    status = append_and_wait(device, stream, p, t[2]->size(0), t[0]->size(0), t[2]->size(1), t[1]->size(0), t[1]->size(1), words);
  }
  if (status != 0) return raise_launch_status(status);
  PyObject* result = PyTuple_New(SPARSE_MLA_STATUS_WORDS);
  for (int i = 0; i < SPARSE_MLA_STATUS_WORDS; ++i) PyTuple_SET_ITEM(result, i, PyLong_FromLong(words[i]));
  return result;
  END_HANDLE_TH_ERRORS
}

// (launch_sparse_mla_kept_status, ..._topk_indices, ..._cache_append_flagged: addresses; the front end's call)
PyObject* configure(PyObject*, PyObject* arguments) {
  unsigned long long attention, select, append;
  PyObject* fallback;
  if (!PyArg_ParseTuple(arguments, "KKKO", &attention, &select, &append, &fallback)) return nullptr;
  launch_attention = reinterpret_cast<LaunchAttention>(attention);
  launch_select = reinterpret_cast<LaunchSelect>(select);
  launch_append = reinterpret_cast<LaunchAppend>(append);
  Py_XSETREF(checked_attention, Py_NewRef(fallback));
  Py_RETURN_NONE;
}

// The first report of the calls on the current stream since it was last read, or else of the device's captured launches:
// waits for the stream, and leaves what it has read zero.
int take_report(cudaStream_t stream, void* block, int32_t (&words)[SPARSE_MLA_STATUS_WORDS]) {
  cudaError_t error = cudaMemcpyAsync(words, block, sizeof(words), cudaMemcpyDeviceToHost, stream);
  if (error == cudaSuccess) error = cudaStreamSynchronize(stream);
  if (error == cudaSuccess && words[0] != 0) {
    error = cudaMemsetAsync(block, 0, kWorkspaceBytes, stream);
    if (error == cudaSuccess) error = cudaStreamSynchronize(stream);
  }
  return int(error);
}

PyObject* read_status(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  int32_t words[SPARSE_MLA_STATUS_WORDS] = {};
  const c10::cuda::CUDAStream stream = c10::cuda::getCurrentCUDAStream();
  at::Tensor own;
  void* captured = nullptr;
  {
    std::lock_guard<std::mutex> lock(workspace_mutex);
    for (const Workspace& w : *workspaces)
      if (w.device == stream.device_index() && w.stream == stream.stream()) own = w.memory;
    if (stream.device_index() < kMostDevices) captured = captured_blocks[stream.device_index()];
  }
  int status = 0;
  {
    pybind11::gil_scoped_release no_gil;
    if (own.defined()) status = take_report(stream.stream(), own.mutable_data_ptr(), words);
    if (status == 0 && words[0] == 0 && captured != nullptr) status = take_report(stream.stream(), captured, words);
  }
  if (status != 0) {
    PyErr_Format(PyExc_RuntimeError, "status read failed with CUDA error %d; device retries are disabled", status);
    return nullptr;
  }
  PyObject* result = PyTuple_New(SPARSE_MLA_STATUS_WORDS);
  for (int i = 0; i < SPARSE_MLA_STATUS_WORDS; ++i) PyTuple_SET_ITEM(result, i, PyLong_FromLong(words[i]));
  return result;
  END_HANDLE_TH_ERRORS
}

PyObject* release_workspaces(PyObject*, PyObject*) {
  {
    std::lock_guard<std::mutex> lock(workspace_mutex);
    workspaces->clear();
  }
  std::vector<AppendStatus> unused;
  {
    std::lock_guard<std::mutex> lock(append_mutex);
    unused.swap(*append_pool);
  }
  for (const AppendStatus& s : unused) free_append_status(s);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"configure", configure, METH_VARARGS, nullptr},
    {"sparse_mla", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_attention)), METH_FASTCALL, nullptr},
    {"topk_indices", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_select)), METH_FASTCALL, nullptr},
    {"cache_append", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(call_append)), METH_FASTCALL, nullptr},
    {"read_status", read_status, METH_NOARGS, nullptr},
    {"release_workspaces", release_workspaces, METH_NOARGS, nullptr},
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_calls() { return PyModule_Create(&module); }
