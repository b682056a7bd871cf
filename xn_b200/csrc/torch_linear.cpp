// The torch side of a linear's call, in C++: what QCudaTensor.matmul_t and QCudaLinear.forward do for the ordinary case (float rows on the
// weight's device, which is the current one, no `out`).
//
// A one-row call is bound by the host, not by its kernel (Q4_0 4096 x 4096: the kernel takes 3.3 us). In Python, with the library called through
// ctypes, it took 10.5 us: some 25 attribute reads and comparisons, a tensor made through the dispatcher, twelve arguments converted one by one, and
// the launch. Everything that is not ordinary returns None, and the Python code takes the call; nothing is kept from one call for the next but
// scratch, by stream.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDACachingAllocator.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <mutex>

namespace {

using MatmulFn = int (*)(const void *, const void *, int, int64_t, int64_t, const void *, void *, int, int64_t, void *, size_t, void *);
using MatvecFn = int (*)(const void *, const void *, int, const void *, void *, int, void *);
using WorkspaceFn = size_t (*)(const void *, int64_t);
MatmulFn g_matmul = nullptr;         // xnq_matmul_t_bias
MatvecFn g_matvec = nullptr;         // xnq_matvec
WorkspaceFn g_workspace_bytes = nullptr; // xnq_matmul_workspace_bytes
PyObject *g_check = nullptr;         // raises the error of a status

struct Weight { // what a call needs of a weight; owned by the capsule that the Python weight keeps
  const void *handle;
  int64_t n, k;
  c10::DeviceIndex device; // -1: the weight was put on "cuda", without an index
  int64_t ws_rows; // rows asked for last and the scratch they need: a program calls a linear with the same few row counts
  size_t ws_bytes;
  bool row_without_scratch; // until xnq_matvec has said that it does not serve this weight
};
constexpr int UNSUPPORTED = -8; // XNQ_ERR_UNSUPPORTED
constexpr const char *NAME = "xnq.weight";

// Scratch (the quantized activations, the tickets and partial sums of split tiles): one buffer for all calls of a device was overwritten by calls on
// another stream, by another thread's call between a call's kernels, and by graphs replayed side by side. So a call gets a block of its own from torch's
// caching allocator, which gives it out again in the order of the stream that it was allocated for, or within the graph that is being captured. That
// costs a call 0.4 us (two rows of Q4_1 512 x 512, which the host bounds: 6.35 us, with the one buffer 5.85), so that rows that need no scratch get none,
// and up to four MiB, all that such small calls ask for, are taken from a slab of the stream (5.9 us): whoever enqueues a call's kernels holds the slab's
// lock, and the stream keeps them in order. Not under capture: a graph may be replayed on another stream. At most SLABS streams have one; the slabs are given
// back with the last weight. (Not from the caching allocator, whose block might belong to a pool of the program's.)
struct Slab {
  c10::DeviceIndex device;
  cudaStream_t stream;
  void *p;
  std::mutex lock;
};
constexpr size_t SLAB = 4 << 20; // the integer kernel's parts of split tiles take 2.4 MB with up to 16 rows
constexpr int SLABS = 16;
Slab g_slabs[SLABS]; // they and the counts: under the interpreter's lock
int g_num_slabs = 0;
int64_t g_weights = 0;

struct RelaxedCapture { // (a graph that another thread is capturing does not mind what this one allocates or frees)
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
  ~RelaxedCapture() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};
// the slab of a stream of the current device, or null: the call takes a block of its own
Slab *slab_for(c10::DeviceIndex device, cudaStream_t stream, size_t bytes) {
  if (bytes > SLAB) return nullptr;
  cudaStreamCaptureStatus capture;
  if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  if (capture != cudaStreamCaptureStatusNone) return nullptr;
  for (int i = 0; i < g_num_slabs; i++)
    if (g_slabs[i].stream == stream && g_slabs[i].device == device) return &g_slabs[i];
  if (g_num_slabs == SLABS) return nullptr;
  Slab &s = g_slabs[g_num_slabs];
  const RelaxedCapture relaxed;
  if (cudaMalloc(&s.p, SLAB) != cudaSuccess) {
    (void)cudaGetLastError();
    return nullptr;
  }
  s.device = device, s.stream = stream;
  g_num_slabs++;
  return &s;
}
void free_weight(PyObject *capsule) {
  delete static_cast<Weight *>(PyCapsule_GetPointer(capsule, NAME));
  if (--g_weights > 0) return;
  const RelaxedCapture relaxed;
  for (; g_num_slabs > 0; g_num_slabs--) (void)cudaFree(g_slabs[g_num_slabs - 1].p); // (waits for the kernels that use it; fails where the process is ending)
  (void)cudaGetLastError();
}

size_t scratch_bytes(Weight *w, int64_t rows) {
  if (w->ws_rows != rows) w->ws_rows = rows, w->ws_bytes = std::max<size_t>(g_workspace_bytes(w->handle, rows), 256);
  return w->ws_bytes;
}

int xnq_dtype(at::ScalarType t) { // F32 0, F16 1, BF16 30: the ggml ids
  return t == at::kFloat ? 0 : (t == at::kHalf ? 1 : (t == at::kBFloat16 ? 30 : -1));
}
// an ordinary dense CUDA tensor: no subclass, no wrapper of a transform
bool plain(PyObject *o) {
  if (!THPVariable_CheckExact(o)) return false;
  constexpr c10::DispatchKeySet allowed({c10::DispatchKey::CUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::AutocastCUDA});
  const c10::DispatchKeySet ks = THPVariable_Unpack(o).key_set();
  return (ks.raw_repr() & ~allowed.raw_repr()) == 0 && ks.has(c10::DispatchKey::CUDA);
}
// Something of torch looks at operators or replaces them: a function or dispatch mode, a transform of torch.func (whatever tensors it has wrapped), a tracer.
bool observed() {
  constexpr c10::DispatchKeySet ordinary({c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView});
  return (c10::impl::tls_local_dispatch_key_set().included_.raw_repr() & ~ordinary.raw_repr()) != 0 || c10::impl::TorchDispatchModeTLS::any_modes_set() ||
         at::impl::torch_function_mode_enabled();
}

PyObject *py_observed(PyObject *, PyObject *) { return PyBool_FromLong(observed()); }

// linear(weight capsule, x, bias or None) -> y, or None where the general code has to take the call
PyObject *linear(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3) {
    PyErr_SetString(PyExc_TypeError, "linear(weight, x, bias)");
    return nullptr;
  }
  Weight *w = static_cast<Weight *>(PyCapsule_GetPointer(args[0], NAME));
  if (!w) return nullptr;
  if (!plain(args[1]) || observed()) Py_RETURN_NONE;
  const at::Tensor &x = THPVariable_Unpack(args[1]);
  const int xt = xnq_dtype(x.scalar_type());
  const int64_t dims = x.dim();
  if (xt < 0 || dims < 2 || x.size(dims - 1) != w->k || x.device().index() != w->device || c10::cuda::current_device() != w->device) Py_RETURN_NONE;
  const int64_t m = x.numel() / w->k;
  int64_t ldx = w->k;
  if (!x.is_contiguous()) {
    if (dims != 2 || x.stride(1) != 1 || (m > 1 && x.stride(0) < w->k)) Py_RETURN_NONE;
    if (m > 1) ldx = x.stride(0);
  }
  const void *bias = nullptr;
  if (args[2] != Py_None) {
    if (!plain(args[2])) Py_RETURN_NONE;
    const at::Tensor &b = THPVariable_Unpack(args[2]);
    if (b.dim() != 1 || b.size(0) != w->n || b.scalar_type() != x.scalar_type() || b.device() != x.device() || !b.is_contiguous() ||
        (b.requires_grad() && c10::GradMode::is_enabled()) || b._fw_grad(0).defined())
      Py_RETURN_NONE;
    bias = b.const_data_ptr();
  }
  c10::SmallVector<int64_t, 6> shape(x.sizes().begin(), x.sizes().end());
  shape[dims - 1] = w->n;
  // (what empty_cuda does behind its look for the device, which is the current one here)
  at::Tensor y = at::Tensor(at::detail::empty_generic(shape, c10::cuda::CUDACachingAllocator::get(), c10::DispatchKeySet(c10::DispatchKey::CUDA), x.scalar_type(), std::nullopt));
  void *const yp = y.mutable_data_ptr();
  const void *const xp = x.const_data_ptr();
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(w->device).stream();
  int rc = UNSUPPORTED;
  if (m == 1 && w->row_without_scratch) {
    Py_BEGIN_ALLOW_THREADS // a launch may block while the device's queue is full
    rc = g_matvec(w->handle, xp, xt, bias, yp, xt, stream);
    Py_END_ALLOW_THREADS
    if (rc == UNSUPPORTED) w->row_without_scratch = false;
  }
  if (rc == UNSUPPORTED) {
    const size_t wsb = scratch_bytes(w, m);
    Slab *const slab = slab_for(w->device, stream, wsb);
    c10::DataPtr block;
    if (!slab) block = c10::cuda::CUDACachingAllocator::get()->allocate(wsb); // for the current device and stream, where the call launches
    void *const ws = slab ? slab->p : block.get();
    Py_BEGIN_ALLOW_THREADS
    if (slab) slab->lock.lock();
    rc = g_matmul(w->handle, xp, xt, m, ldx, bias, yp, xt, w->n, ws, wsb, stream);
    if (slab) slab->lock.unlock();
    Py_END_ALLOW_THREADS
  }
  if (rc != 0) return PyObject_CallFunction(g_check, "i", rc);
  return THPVariable_Wrap(std::move(y));
  END_HANDLE_TH_ERRORS
}

// workspace(weight capsule, rows) -> scratch for one call of that many rows
PyObject *workspace(PyObject *, PyObject *args) {
  HANDLE_TH_ERRORS
  PyObject *capsule;
  long long m;
  if (!PyArg_ParseTuple(args, "OL", &capsule, &m)) return nullptr;
  Weight *w = static_cast<Weight *>(PyCapsule_GetPointer(capsule, NAME));
  if (!w) return nullptr;
  const at::Device device(at::kCUDA, w->device < 0 ? c10::cuda::current_device() : w->device);
  return THPVariable_Wrap(at::Tensor(at::detail::empty_cuda({(int64_t)scratch_bytes(w, m)}, at::kByte, device, std::nullopt)));
  END_HANDLE_TH_ERRORS
}

// weight(handle, n, k, device index) -> capsule
PyObject *weight(PyObject *, PyObject *args) {
  unsigned long long handle;
  long long n, k;
  int device;
  if (!PyArg_ParseTuple(args, "KLLi", &handle, &n, &k, &device)) return nullptr;
  PyObject *capsule = PyCapsule_New(new Weight{reinterpret_cast<const void *>(handle), n, k, (c10::DeviceIndex)device, -1, 0, true}, NAME, free_weight);
  if (capsule) g_weights++;
  return capsule;
}

// bind(xnq_matmul_t_bias, xnq_matvec, xnq_matmul_workspace_bytes, check): the library that ctypes has loaded
PyObject *bind(PyObject *, PyObject *args) {
  unsigned long long matmul, matvec, ws;
  PyObject *check;
  if (!PyArg_ParseTuple(args, "KKKO", &matmul, &matvec, &ws, &check)) return nullptr;
  g_matmul = reinterpret_cast<MatmulFn>(matmul), g_matvec = reinterpret_cast<MatvecFn>(matvec), g_workspace_bytes = reinterpret_cast<WorkspaceFn>(ws);
  Py_INCREF(check);
  Py_XSETREF(g_check, check);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"linear", reinterpret_cast<PyCFunction>(reinterpret_cast<void *>(linear)), METH_FASTCALL, "linear(weight, x, bias) -> y or None"},
    {"workspace", workspace, METH_VARARGS, "workspace(weight, rows) -> scratch"},
    {"weight", weight, METH_VARARGS, "weight(handle, n, k, device index) -> capsule"},
    {"observed", py_observed, METH_NOARGS, "observed() -> whether a mode, a transform or a tracer looks at torch's operators"},
    {"bind", bind, METH_VARARGS, "bind(matmul, matvec, workspace_bytes, check)"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_xnq_torch", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

} // namespace

PyMODINIT_FUNC PyInit__xnq_torch() { return PyModule_Create(&module_def); }
