// The common call of the whole path without Python in between: argument checks, plan lookup, result tensor, library call and the
// deferred status check of prefill.py, for plain CUDA tensors that the kernels can read in place and the default options.  Whatever it
// does not cover it leaves, untouched, to the Python code (returns None), which also raises all errors.
// A call of 187 tokens keeps the GPU busy for 14 us, and its Python took 36: here 14 (calls back to back 36.7 -> 21.5 us).
#include <Python.h>

#include <torch/csrc/autograd/python_variable.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/ops/empty_like.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/DynamicTypes.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/object_ptr.h>

#include <cstdlib>
#include <vector>

#include "../../include/pbs_b200.h"

namespace {

constexpr int kSlots = 16;             // calls whose status words may be in flight to the host at once
constexpr const char* kName = "pbs_attn_b200.call";
const cudaStream_t kNoStream = reinterpret_cast<cudaStream_t>(~uintptr_t{0});

using PrefillFn = decltype(&pbs_prefill_fwd);
using ExportFn = decltype(&pbs_export_status);

// What a plan's calls share; the pointers are the plan's own buffers and structs, which live as long as it does, and so does this.
struct Call {
  const pbs_shape_t* shape;
  const pbs_scratch_t* scratch;
  int32_t* ring;                       // pinned, kSlots x 8, from the pool below
  int device;
  PrefillFn prefill;
  ExportFn export_status;
  cudaEvent_t landed[kSlots];
  int made, first, count, next;        // events created; pending slots: first .. first + count - 1
  int told;                            // so many of these, the oldest, are no longer looked at: an error among them has been raised
  cudaStream_t last;                   // stream of the last call (kNoStream: none yet); its event is the latest pending one, if any is
  PyThread_type_lock turn;             // held while a call is enqueued
  bool unwatched;                      // words are on their way to the ring that no event tells of
};

Call* get(PyObject* capsule) { return static_cast<Call*>(PyCapsule_GetPointer(capsule, kName)); }

// Rings of calls that are gone, and calls whose plan is gone while the device may still write to their rings.  The interpreter's lock guards
// both; there are never more of them than there were plans at a time and plans that left with calls in flight.
std::vector<int32_t*> free_rings;
std::vector<Call*> leaving;

// Recycles what has left and landed.
void sweep() {
  size_t kept = 0;
  for (Call* c : leaving) {
    while (c->count > 0 && cudaEventQuery(c->landed[c->first]) != cudaErrorNotReady) {
      c->first = (c->first + 1) % kSlots;
      --c->count;
    }
    if (c->count > 0) {
      leaving[kept++] = c;
      continue;
    }
    for (int i = 0; i < c->made; ++i) (void)cudaEventDestroy(c->landed[i]);
    if (!c->unwatched) free_rings.push_back(c->ring);
    PyThread_free_lock(c->turn);
    delete c;
  }
  leaving.resize(kept);
}

void destroy(PyObject* capsule) { leaving.push_back(static_cast<Call*>(PyCapsule_GetPointer(capsule, kName))); }

bool capturing(cudaStream_t st) {
  cudaStreamCaptureStatus s;
  return cudaStreamIsCapturing(st, &s) != cudaSuccess || s != cudaStreamCaptureStatusNone;
}

// Sends the status words of the call just enqueued to its slot of the ring.  Not those of a captured call: it is replayed at times unknown
// here, perhaps after the plan is gone (check_status reads the device's words).  by_copy: for calls that go through Python, the
// host-tensor call's among them, whose own copies out it queues with (16384 tokens 4.95 ms so, 5.19 with the kernel); for all others the
// kernel is ahead (pbs_api.cu has the figures).
cudaError_t queue_status(Call* c, cudaStream_t st, bool by_copy) {
  if (capturing(st)) return cudaSuccess;
  const int slot = c->next;
  const int32_t* words = static_cast<const int32_t*>(c->scratch->status);
  cudaError_t e = cudaSuccess;
  while (c->made <= slot) {
    if ((e = cudaEventCreateWithFlags(&c->landed[c->made], cudaEventDisableTiming)) != cudaSuccess) return e;
    ++c->made;
  }
  if (by_copy) e = cudaMemcpyAsync(c->ring + 8 * slot, words, 8 * sizeof(int32_t), cudaMemcpyDeviceToHost, st);
  else if (c->export_status(words, c->ring + 8 * slot, st) != PBS_OK) e = cudaErrorLaunchFailure;
  if (e != cudaSuccess) return e;
  if ((e = cudaEventRecord(c->landed[slot], st)) != cudaSuccess) {
    c->unwatched = true;
    return e;
  }
  c->last = st;
  c->next = (slot + 1) % kSlots;
  ++c->count;
  return cudaSuccess;
}

// Drops the pending slots that have landed (all of them if wait_all, the oldest in any case if the ring is full) up to one that reports an
// error: its number, or -1.  That slot stays, the caller decides.
int landed_error(Call* c, bool wait_all) {
  while (c->count > 0) {
    cudaEvent_t ev = c->landed[c->first];
    if (wait_all || c->count >= kSlots) {
      const int slot = c->first;
      Py_BEGIN_ALLOW_THREADS
      (void)cudaEventSynchronize(ev);
      Py_END_ALLOW_THREADS
      if (c->count == 0 || c->first != slot) continue;     // another thread has been here
    } else if (cudaEventQuery(ev) != cudaSuccess) {
      break;                                               // not there yet; an error of the device shows at the next library call
    }
    if (c->told > 0) --c->told;
    else if (*const_cast<volatile int32_t*>(c->ring + 8 * c->first) != 0) return c->first;
    c->first = (c->first + 1) % kSlots;
    --c->count;
  }
  return -1;
}

// A plan may be made while its stream is captured: what is done here belongs to no graph and must not end the capture.
struct Relaxed {
  cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
  Relaxed() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
  ~Relaxed() { (void)cudaThreadExchangeStreamCaptureMode(&mode); }
};

PyObject* py_attach(PyObject*, PyObject* args) {
  HANDLE_TH_ERRORS
  unsigned long long shape, scratch, fn, fn2;
  int device;
  if (!PyArg_ParseTuple(args, "KKiKK", &shape, &scratch, &device, &fn, &fn2)) return nullptr;
  const c10::cuda::CUDAGuard guard(static_cast<c10::DeviceIndex>(device));   // pinned memory brings up the current device, which may be another one
  const Relaxed relaxed;
  sweep();
  const PyThread_type_lock turn = PyThread_allocate_lock();
  if (!turn) return PyErr_NoMemory();
  int32_t* ring = nullptr;
  if (free_rings.empty()) {
    const cudaError_t e = cudaHostAlloc(reinterpret_cast<void**>(&ring), kSlots * 8 * sizeof(int32_t), cudaHostAllocPortable);
    if (e != cudaSuccess) {
      PyThread_free_lock(turn);
      return PyErr_Format(PyExc_RuntimeError, "pinned memory for the status words: %s", cudaGetErrorString(e));
    }
  } else {
    ring = free_rings.back();
    free_rings.pop_back();
  }
  Call* c = new Call{reinterpret_cast<const pbs_shape_t*>(shape), reinterpret_cast<const pbs_scratch_t*>(scratch), ring,
                     device, reinterpret_cast<PrefillFn>(fn), reinterpret_cast<ExportFn>(fn2), {}, 0, 0, 0, 0, 0, kNoStream, turn, false};
  return PyCapsule_New(c, kName, destroy);
  END_HANDLE_TH_ERRORS
}

// inspect(call, wait_all): None, or the status words of a call that failed (what all pending ones report is then not looked at any more; their
// slots stay taken until the words have landed)
PyObject* py_inspect(PyObject*, PyObject* args) {
  PyObject* capsule;
  int wait_all;
  if (!PyArg_ParseTuple(args, "Op", &capsule, &wait_all)) return nullptr;
  Call* c = get(capsule);
  if (!c) return nullptr;
  if (!wait_all && capturing(c10::cuda::getCurrentCUDAStream(c->device).stream())) Py_RETURN_NONE;   // an event query would end the capture
  const int slot = landed_error(c, wait_all != 0);
  if (slot < 0) Py_RETURN_NONE;
  c->told = c->count;
  PyObject* words = PyList_New(8);
  for (int i = 0; words && i < 8; ++i) PyList_SET_ITEM(words, i, PyLong_FromLong(c->ring[8 * slot + i]));
  return words;
}

// enter(call), leave(call): take and give back the turn
PyObject* py_enter(PyObject*, PyObject* capsule) {
  Call* c = get(capsule);
  if (!c) return nullptr;
  Py_BEGIN_ALLOW_THREADS
  PyThread_acquire_lock(c->turn, WAIT_LOCK);
  Py_END_ALLOW_THREADS
  Py_RETURN_NONE;
}

PyObject* py_leave(PyObject*, PyObject* capsule) {
  Call* c = get(capsule);
  if (!c) return nullptr;
  PyThread_release_lock(c->turn);
  Py_RETURN_NONE;
}

// follow(call, stream): the next call, on this stream, comes after the last one.  The plan's device is current.
PyObject* py_follow(PyObject*, PyObject* args) {
  PyObject* capsule;
  unsigned long long stream;
  if (!PyArg_ParseTuple(args, "OK", &capsule, &stream)) return nullptr;
  Call* c = get(capsule);
  if (!c) return nullptr;
  const cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (c->count == 0 || st == c->last || capturing(st)) Py_RETURN_NONE;   // (a capture cannot wait for work outside)
  const cudaError_t e = cudaStreamWaitEvent(st, c->landed[(c->next + kSlots - 1) % kSlots], 0);
  if (e != cudaSuccess) return PyErr_Format(PyExc_RuntimeError, "wait for the last call of the plan: %s", cudaGetErrorString(e));
  Py_RETURN_NONE;
}

// queue(call, stream): the plan's device is current
PyObject* py_queue(PyObject*, PyObject* args) {
  PyObject* capsule;
  unsigned long long stream;
  if (!PyArg_ParseTuple(args, "OK", &capsule, &stream)) return nullptr;
  Call* c = get(capsule);
  if (!c) return nullptr;
  const cudaError_t e = queue_status(c, reinterpret_cast<cudaStream_t>(stream), true);
  if (e != cudaSuccess) return PyErr_Format(PyExc_RuntimeError, "copy of the status words: %s", cudaGetErrorString(e));
  Py_RETURN_NONE;
}

bool plain_int(PyObject* o, int64_t* v) {
  if (!PyLong_CheckExact(o)) return false;
  int over = 0;
  *v = PyLong_AsLongLongAndOverflow(o, &over);
  return !over && *v > 0 && *v < (1ll << 31);
}

// prefill.py's _readable
bool readable(const at::Tensor& t, bool distinct_heads) {
  const auto st = t.strides(), sz = t.sizes();
  if (st[3] != 1 || st[2] <= 0 || st[0] < 0 || st[1] < 0) return false;
  if (((st[0] | st[1] | st[2]) * t.element_size()) % 16 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16) return false;
  return !distinct_heads || ((st[0] > 0 || sz[0] == 1) && (st[1] > 0 || sz[1] == 1));
}

// A call's turn for as long as this lives, if nobody has it.
struct TryTurn {
  Call* c;
  const bool held;
  explicit TryTurn(Call* call) : c(call), held(PyThread_acquire_lock(call->turn, NOWAIT_LOCK)) {}
  ~TryTurn() {
    if (held) PyThread_release_lock(c->turn);
  }
};

enum Flags { kForceFirst = 1, kMeanPooling = 2, kNoOwnSegment = 4 };

// call(plans, q, k, v, block_size, segment_size, threshold, flags): the result, or None
PyObject* py_call(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  if (n != 8) { PyErr_SetString(PyExc_TypeError, "call takes 8 arguments"); return nullptr; }
  for (int i = 1; i <= 3; ++i)
    if (!THPVariable_CheckExact(a[i])) Py_RETURN_NONE;
  const at::Tensor &q = THPVariable_Unpack(a[1]), &k = THPVariable_Unpack(a[2]), &v = THPVariable_Unpack(a[3]);
  int64_t bs, seg;
  if (!PyFloat_CheckExact(a[6]) || !plain_int(a[4], &bs) || !plain_int(a[5], &seg) || seg % bs) Py_RETURN_NONE;
  if (at::impl::torch_function_mode_enabled() || !q.is_cuda() || q.dim() != 4 || k.dim() != 4) Py_RETURN_NONE;
  const auto qz = q.sizes(), kz = k.sizes();
  if (kz[0] != qz[0] || kz[2] != qz[2] || kz[3] != qz[3] || kz[1] < 1 || qz[1] % kz[1] || v.sizes() != kz) Py_RETURN_NONE;
  if (k.device() != q.device() || v.device() != q.device() || k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) Py_RETURN_NONE;
  if (q.numel() == 0 || q.layout() != at::kStrided || k.layout() != at::kStrided || v.layout() != at::kStrided) Py_RETURN_NONE;
  if (!readable(q, true) || !readable(k, false) || !readable(v, false)) Py_RETURN_NONE;
  const char* check = std::getenv("PBS_B200_CHECK_STATUS");
  if (check && check[0] == '1' && !check[1]) Py_RETURN_NONE;
  const long flags = PyLong_AsLong(a[7]);

  // the plan, by the key of prefill.get_plan
  const auto device = q.device();
  THPObjectPtr key(Py_BuildValue("(LLLLLLLOi)", (long long)qz[0], (long long)qz[1], (long long)kz[1], (long long)qz[2], (long long)qz[3], (long long)bs,
                                 (long long)seg, (PyObject*)torch::getTHPDtype(q.scalar_type()), (int)device.index()));
  if (!key) return nullptr;
  PyObject* plan = PyDict_GetItemWithError(a[0], key.get());
  if (!plan) {
    if (PyErr_Occurred()) return nullptr;
    Py_RETURN_NONE;
  }
  Py_INCREF(plan);
  THPObjectPtr plan_owner(plan), capsule(PyObject_GetAttrString(plan, "_native"));
  if (!capsule) return nullptr;
  if (!PyCapsule_IsValid(capsule.get(), kName)) Py_RETURN_NONE;
  Call* c = get(capsule.get());
  const TryTurn turn(c);                                   // the scratch serves one call at a time: Python waits for its turn
  if (!turn.held) Py_RETURN_NONE;
  const c10::cuda::CUDAGuard guard(device);
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(device.index()).stream();
  // (another stream than last time has to wait, and the scratch's memory to be told of it)
  if (capturing(st) || st != c->last || landed_error(c, false) >= 0) Py_RETURN_NONE;   // (or an earlier call failed)
  at::Tensor out = at::empty_like(q);
  if (!readable(out, false)) Py_RETURN_NONE;
  pbs_options_t opt = {};
  opt.threshold = (float)PyFloat_AS_DOUBLE(a[6]);
  opt.force_select_first_block = (flags & kForceFirst) != 0;
  opt.query_pool_mode = opt.key_pool_mode = PBS_POOL_MEAN;
  opt.attn_impl = PBS_ATTN_AUTO;
  opt.no_permutation = opt.diagonal_candidates = (flags & kMeanPooling) != 0;
  opt.no_own_segment = (flags & kNoOwnSegment) != 0;
  opt.kv_in_place = 1;
  const bool in_place = (opt.no_permutation || qz[2] <= seg) && q.scalar_type() != at::kFloat;
  int rc;
  cudaError_t e = cudaSuccess;
  Py_BEGIN_ALLOW_THREADS
  rc = c->prefill(c->shape, q.data_ptr(), q.strides().data(), k.data_ptr(), k.strides().data(), v.data_ptr(), v.strides().data(), out.data_ptr(),
                  out.strides().data(), &opt, c->scratch, st);
  Py_END_ALLOW_THREADS
  if (rc != PBS_OK) Py_RETURN_NONE;                        // refused before anything was enqueued: Python says why
  if (PyObject_SetAttrString(plan, "_kv_left_out", in_place ? Py_True : Py_False) < 0) return nullptr;
  e = queue_status(c, st, false);
  if (e != cudaSuccess) return PyErr_Format(PyExc_RuntimeError, "copy of the status words: %s", cudaGetErrorString(e));
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"attach", py_attach, METH_VARARGS, "attach(shape, scratch, device, prefill, export_status): addresses of a plan's buffers -> its call object"},
    {"inspect", py_inspect, METH_VARARGS, "inspect(call, wait_all): None or the status words of a failed call"},
    {"enter", py_enter, METH_O, "enter(call): wait for the call's turn and take it"},
    {"leave", py_leave, METH_O, "leave(call): give the turn back"},
    {"follow", py_follow, METH_VARARGS, "follow(call, stream): let the stream wait for the last call if that was on another one"},
    {"queue", py_queue, METH_VARARGS, "queue(call, stream): send the status words of the call just enqueued"},
    {"call", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_call)), METH_FASTCALL,
     "call(plans, q, k, v, block_size, segment_size, threshold, flags): the result, or None where Python has to do it"},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "pbs_host", nullptr, -1, methods};

}  // namespace

PyMODINIT_FUNC PyInit_pbs_host(void) { return PyModule_Create(&module); }
