// Python binding of the calls that a time-stepping loop makes: the sort, the sort with its payload
// and the collision stage.  It checks the arguments, allocates the results and calls the C ABI.
//
// Small calls are bound by the host: through ctypes, a sort of 5000 particles took 22.4 us a call (13 on the
// device), 100,000 particles with payload 35.3, a step of 200,003 46.5; through this 19.1, 26.0 and 38.6.
//
// The functions take the plain form of a call only (dense contiguous tensors on the current device,
// Python numbers, a workspace that is there already) and return None for any other: the Python code
// around them then does the call, and raises what there is to raise.
#include <Python.h>

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <cmath>

#include "../../include/aether_sort.h"

namespace {

// Entry points of the library that ctypes loaded (bind).
decltype(&AetherSortWorkspaceBytes) workspace_bytes = nullptr;
decltype(&AetherSortParticlesByCell) sort_entry = nullptr;
decltype(&AetherSortAndGatherParticlesZeroPadded) gather_entry = nullptr;
decltype(&AetherPushSortAndGatherParticlesZeroPadded) push_entry = nullptr;
decltype(&AetherDsmcCollideTma) collide_entry = nullptr;
PyTypeObject* grid_type = nullptr;  // CellGrid

constexpr int64_t kMostCells = int64_t{1} << 25;  // keys of 32 bits
constexpr int64_t kMostParticles = (int64_t{1} << 30) - 1;

// Nothing that wants to see the operations of a call: a mode, a function transform, a tracer.
bool unwatched() {
  constexpr auto usual = c10::DispatchKeySet({c10::DispatchKey::BackendSelect, c10::DispatchKey::ADInplaceOrView,
                                              c10::DispatchKey::AutocastCUDA});
  const auto included = c10::impl::tls_local_dispatch_key_set().included_;
  return (included.raw_repr() & ~usual.raw_repr()) == 0 && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         !at::impl::torch_function_mode_enabled();
}

// The tensor behind `object` if it is an ordinary dense CUDA tensor of that type, else null.
const at::Tensor* dense(PyObject* object, at::ScalarType type) {
  if (!THPVariable_CheckExact(object)) return nullptr;
  const at::Tensor& t = THPVariable_Unpack(object);
  constexpr auto usual = c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA,
                                              c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutocastCUDA});
  if (!t.defined() || !t.is_cuda() || (t.key_set().raw_repr() & ~usual.raw_repr()) != 0 || t.scalar_type() != type)
    return nullptr;
  return &t;
}

// A vector of n elements on `device`; n < 0: any length.
const at::Tensor* vector_of(PyObject* object, at::ScalarType type, int64_t n, int device) {
  const at::Tensor* t = dense(object, type);
  if (!t || t->dim() != 1 || !t->is_contiguous() || (n >= 0 && t->numel() != n) || t->get_device() != device)
    return nullptr;
  return t;
}

bool number(PyObject* object, double* out) {
  if (PyFloat_CheckExact(object)) {
    *out = PyFloat_AS_DOUBLE(object);
    return true;
  }
  if (!PyLong_CheckExact(object)) return false;
  int overflow = 0;
  const long long v = PyLong_AsLongLongAndOverflow(object, &overflow);
  *out = static_cast<double>(v);
  return overflow == 0 && v > -(1ll << 53) && v < (1ll << 53);
}

bool word64(PyObject* object, uint64_t* out) {
  if (!PyLong_CheckExact(object)) return false;
  *out = PyLong_AsUnsignedLongLongMask(object);
  return true;
}

// Three numbers in a tuple or list.
bool three(PyObject* object, double out[3]) {
  const bool tuple = PyTuple_Check(object);
  if ((!tuple && !PyList_CheckExact(object)) || PySequence_Fast_GET_SIZE(object) != 3) return false;
  for (int k = 0; k < 3; ++k)
    if (!number(PySequence_Fast_GET_ITEM(object, k), &out[k])) return false;
  return true;
}

// A CellGrid, which is a tuple (lo, hi, cells).  The inverse spacing is a quotient of doubles, as
// native_grid has it.
bool whole_grid(PyObject* object, AetherGrid* g, int64_t* cells) {
  double lo[3], hi[3], count[3];
  if (Py_TYPE(object) != grid_type || PyTuple_GET_SIZE(object) != 3 || !three(PyTuple_GET_ITEM(object, 0), lo) ||
      !three(PyTuple_GET_ITEM(object, 1), hi))
    return false;
  PyObject* numbers = PyTuple_GET_ITEM(object, 2);
  if (!three(numbers, count)) return false;
  for (int k = 0; k < 3; ++k)
    if (!PyLong_CheckExact(PySequence_Fast_GET_ITEM(numbers, k)) || !(count[k] >= 1) ||
        count[k] > static_cast<double>(kMostCells) || !(hi[k] - lo[k] > 0) || !std::isfinite(hi[k] - lo[k]))
      return false;
  const double total = count[0] * count[1] * count[2];
  if (total > static_cast<double>(kMostCells)) return false;
  *cells = static_cast<int64_t>(total);
  g->x0 = static_cast<float>(lo[0]);
  g->y0 = static_cast<float>(lo[1]);
  g->z0 = static_cast<float>(lo[2]);
  g->inv_dx = static_cast<float>(count[0] / (hi[0] - lo[0]));
  g->inv_dy = static_cast<float>(count[1] / (hi[1] - lo[1]));
  g->inv_dz = static_cast<float>(count[2] / (hi[2] - lo[2]));
  g->nx = static_cast<int32_t>(count[0]);
  g->ny = static_cast<int32_t>(count[1]);
  g->nz = static_cast<int32_t>(count[2]);
  g->ix_offset = 0;
  g->nx_local = g->nx;
  return true;
}

// What every sort begins with.
struct SortCall {
  const at::Tensor* c[3];
  int64_t n, cells;
  int device;
  AetherGrid grid;
  uint64_t seed;
  at::Tensor workspace;  // held: another thread may replace it
  cudaStream_t stream;

  bool plain(PyObject* const* positions, PyObject* grid_object, PyObject* seed_object, PyObject* workspaces,
             int payload) {
    if (!unwatched()) return false;
    c[0] = dense(positions[0], at::kFloat);
    if (!c[0] || c[0]->dim() != 1 || !c[0]->is_contiguous()) return false;
    n = c[0]->numel();
    device = c[0]->get_device();
    if (n < 1 || n > kMostParticles || device != c10::cuda::current_device()) return false;
    for (int k = 1; k < 3; ++k) {
      c[k] = vector_of(positions[k], at::kFloat, n, device);
      if (!c[k]) return false;
    }
    if (!whole_grid(grid_object, &grid, &cells) || !word64(seed_object, &seed) || !PyDict_CheckExact(workspaces))
      return false;
    stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
    PyObject* key = Py_BuildValue("(iN)", device, PyLong_FromVoidPtr(stream));
    if (!key) {
      PyErr_Clear();
      return false;
    }
    PyObject* held = PyDict_GetItem(workspaces, key);
    Py_DECREF(key);
    if (!held || !THPVariable_CheckExact(held)) return false;
    workspace = THPVariable_Unpack(held);
    return static_cast<size_t>(workspace.numel()) >= workspace_bytes(n, cells, payload);
  }
};

at::Tensor fresh(at::IntArrayRef sizes, at::ScalarType type, int device) {
  return at::empty(sizes, at::TensorOptions().dtype(type).device(c10::Device(c10::kCUDA, static_cast<c10::DeviceIndex>(device))));
}

template <class T>
T* at_start(const at::Tensor& t) { return static_cast<T*>(t.data_ptr()); }

// None, with the error the Python code raises for a status.
PyObject* failed(const char* what, int status) {
  PyErr_Format(PyExc_RuntimeError, "%s failed with cudaError %d", what, status);
  return nullptr;
}

// sort(x, y, z, grid, seed, workspaces) -> (keys, index, counts, start) or None
PyObject* sort(PyObject*, PyObject* const* args, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  SortCall s;
  if (count != 6 || !s.plain(args, args[3], args[4], args[5], 0)) Py_RETURN_NONE;
  const at::Tensor out[4] = {fresh({s.n}, at::kInt, s.device), fresh({s.n}, at::kInt, s.device),
                             fresh({s.cells}, at::kInt, s.device), fresh({s.cells + 1}, at::kInt, s.device)};
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = sort_entry(at_start<float>(*s.c[0]), at_start<float>(*s.c[1]), at_start<float>(*s.c[2]), s.n, &s.grid,
                      s.seed, at_start<uint32_t>(out[0]), at_start<int32_t>(out[1]), at_start<int32_t>(out[2]),
                      at_start<int32_t>(out[3]), s.workspace.data_ptr(), static_cast<size_t>(s.workspace.numel()),
                      s.stream);
  Py_END_ALLOW_THREADS
  if (status != 0) return failed("AetherSortParticlesByCell", status);
  PyObject* result = PyTuple_New(4);
  if (!result) return nullptr;
  for (int k = 0; k < 4; ++k) PyTuple_SET_ITEM(result, k, THPVariable_Wrap(out[k]));
  return result;
  END_HANDLE_TH_ERRORS
}

// gather(x, y, z, velocity, grid, seed, path, padded_out, out, push, workspaces)
//   -> (keys, index, counts, start, x, y, z, velocity), those of `out` if it is given, or None
PyObject* gather(PyObject*, PyObject* const* args, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  SortCall s;
  if (count != 11 || !PyLong_CheckExact(args[6])) Py_RETURN_NONE;
  const long path = PyLong_AsLong(args[6]);
  if (path < 0 || path > 2) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  if (!s.plain(args, args[4], args[5], args[10], 1)) Py_RETURN_NONE;
  const at::Tensor* velocity = dense(args[3], at::kFloat);
  if (!velocity || velocity->dim() != 2 || velocity->size(0) != 3 || velocity->size(1) < s.n ||
      velocity->stride(1) != 1 || velocity->stride(0) < s.n || velocity->get_device() != s.device)
    Py_RETURN_NONE;
  const int64_t padded = velocity->stride(0);
  int64_t padded_sorted = padded;
  if (args[7] != Py_None) {
    if (!PyLong_CheckExact(args[7])) Py_RETURN_NONE;
    padded_sorted = PyLong_AsLongLong(args[7]);
    if (padded_sorted < s.n || padded_sorted > 4 * kMostParticles) {
      PyErr_Clear();
      Py_RETURN_NONE;
    }
  }
  double dt = 0, lo[3], hi[3];
  const bool push = args[9] != Py_None;
  if (push) {
    PyObject* spec = args[9];
    if (!PyTuple_Check(spec) || PyTuple_GET_SIZE(spec) != 3 || !number(PyTuple_GET_ITEM(spec, 0), &dt) ||
        !three(PyTuple_GET_ITEM(spec, 1), lo) || !three(PyTuple_GET_ITEM(spec, 2), hi))
      Py_RETURN_NONE;
  }
  at::Tensor out[8];
  PyObject* given[8] = {};
  if (args[8] != Py_None) {
    PyObject* o = args[8];
    if (!PyTuple_Check(o) || PyTuple_GET_SIZE(o) != 3) Py_RETURN_NONE;
    PyObject *order = PyTuple_GET_ITEM(o, 0), *positions = PyTuple_GET_ITEM(o, 1);
    if (!PyTuple_Check(order) || PyTuple_GET_SIZE(order) != 4 || !PyTuple_Check(positions) ||
        PyTuple_GET_SIZE(positions) != 3)
      Py_RETURN_NONE;
    for (int k = 0; k < 4; ++k) given[k] = PyTuple_GET_ITEM(order, k);
    for (int k = 0; k < 3; ++k) given[4 + k] = PyTuple_GET_ITEM(positions, k);
    given[7] = PyTuple_GET_ITEM(o, 2);
    const int64_t length[7] = {s.n, s.n, s.cells, s.cells + 1, s.n, s.n, s.n};
    for (int k = 0; k < 7; ++k) {
      const at::Tensor* t = vector_of(given[k], k < 4 ? at::kInt : at::kFloat, length[k], s.device);
      if (!t) Py_RETURN_NONE;
      out[k] = *t;
    }
    const at::Tensor* v = dense(given[7], at::kFloat);
    if (!v || v->dim() != 2 || v->size(0) != 3 || v->size(1) != padded_sorted || !v->is_contiguous() ||
        v->get_device() != s.device)
      Py_RETURN_NONE;
    out[7] = *v;
  } else {
    out[0] = fresh({s.n}, at::kInt, s.device);
    out[1] = fresh({s.n}, at::kInt, s.device);
    out[2] = fresh({s.cells}, at::kInt, s.device);
    out[3] = fresh({s.cells + 1}, at::kInt, s.device);
    for (int k = 4; k < 7; ++k) out[k] = fresh({s.n}, at::kFloat, s.device);
    out[7] = fresh({3, padded_sorted}, at::kFloat, s.device);
  }
  // The library zeroes the padding columns.  A given tensor that PyTorch would not let be written to, or that it counts
  // the writes to, is treated as by its own operation.
  if (padded_sorted > s.n && given[7]) {
    if (out[7].requires_grad() || out[7].is_inference()) out[7].narrow(1, s.n, padded_sorted - s.n).zero_();
    else out[7].unsafeGetTensorImpl()->bump_version();
  }
  const float flo[3] = {static_cast<float>(lo[0]), static_cast<float>(lo[1]), static_cast<float>(lo[2])};
  const float fhi[3] = {static_cast<float>(hi[0]), static_cast<float>(hi[1]), static_cast<float>(hi[2])};
  const float *x = at_start<float>(*s.c[0]), *y = at_start<float>(*s.c[1]), *z = at_start<float>(*s.c[2]),
              *v = at_start<float>(*velocity);
  auto *keys = at_start<uint32_t>(out[0]);
  auto *index = at_start<int32_t>(out[1]), *counts = at_start<int32_t>(out[2]), *start = at_start<int32_t>(out[3]);
  auto *xs = at_start<float>(out[4]), *ys = at_start<float>(out[5]), *zs = at_start<float>(out[6]),
       *vs = at_start<float>(out[7]);
  void* workspace = s.workspace.data_ptr();
  const size_t bytes = static_cast<size_t>(s.workspace.numel());
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = push ? push_entry(x, y, z, v, padded, s.n, static_cast<float>(dt), flo, fhi, &s.grid, s.seed, keys, index,
                             counts, start, xs, ys, zs, vs, padded_sorted, static_cast<int>(path), workspace, bytes,
                             s.stream)
                : gather_entry(x, y, z, v, padded, s.n, &s.grid, s.seed, keys, index, counts, start, xs, ys, zs, vs,
                               padded_sorted, static_cast<int>(path), workspace, bytes, s.stream);
  Py_END_ALLOW_THREADS
  if (status != 0) return failed(push ? "AetherPushSortAndGatherParticles" : "AetherSortAndGatherParticles", status);
  PyObject* result = PyTuple_New(8);
  if (!result) return nullptr;
  for (int k = 0; k < 8; ++k) {
    if (given[k]) Py_INCREF(given[k]);
    PyTuple_SET_ITEM(result, k, given[k] ? given[k] : THPVariable_Wrap(out[k]));
  }
  return result;
  END_HANDLE_TH_ERRORS
}

// collide(velocity, cell_start, sigma_g_max, collisions, num_particles, selection_factor,
//         vhs_coefficient, vhs_exponent, seed, step) -> True or None
PyObject* collide(PyObject*, PyObject* const* args, Py_ssize_t count) {
  HANDLE_TH_ERRORS
  if (count != 10 || !unwatched()) Py_RETURN_NONE;
  const at::Tensor* velocity = dense(args[0], at::kFloat);
  if (!velocity || velocity->dim() != 2 || velocity->size(0) != 3 || !velocity->is_contiguous()) Py_RETURN_NONE;
  const int device = velocity->get_device();
  const at::Tensor* start = vector_of(args[1], at::kInt, -1, device);
  const at::Tensor* sigma = vector_of(args[2], at::kFloat, -1, device);
  const at::Tensor* collisions = vector_of(args[3], at::kInt, -1, device);
  double factor, coefficient, exponent;
  uint64_t seed, step;
  if (!start || !sigma || !collisions || device != c10::cuda::current_device() || !PyLong_CheckExact(args[4]) ||
      !number(args[5], &factor) || !number(args[6], &coefficient) || !number(args[7], &exponent) ||
      !word64(args[8], &seed) || !word64(args[9], &step))
    Py_RETURN_NONE;
  const long long n = PyLong_AsLongLong(args[4]);
  if (n < 0 || n > velocity->size(1) || velocity->size(1) > kMostParticles || sigma->numel() > kMostCells) {
    PyErr_Clear();
    Py_RETURN_NONE;
  }
  float* v = at_start<float>(*velocity);
  const int* first = at_start<int>(*start);
  float* majorant = at_start<float>(*sigma);
  int* accepted = at_start<int>(*collisions);
  const int padded = static_cast<int>(velocity->size(1)), cells = static_cast<int>(sigma->numel());
  void* stream = c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(device)).stream();
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = collide_entry(v, first, majorant, accepted, static_cast<int>(n), padded, cells, static_cast<float>(factor),
                         static_cast<float>(coefficient), static_cast<float>(exponent), seed, step, stream);
  Py_END_ALLOW_THREADS
  if (status != 0) return failed("AetherDsmcCollideTma", status);
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// bind(CellGrid, address, ...): the class of grids, a tuple, and the library's entry points in the order below
PyObject* bind(PyObject*, PyObject* const* args, Py_ssize_t count) {
  void* p[5];
  if (count != 6 || !PyType_Check(args[0]) ||
      !PyType_IsSubtype(reinterpret_cast<PyTypeObject*>(args[0]), &PyTuple_Type)) {
    PyErr_SetString(PyExc_TypeError, "bind takes the class of grids and five addresses");
    return nullptr;
  }
  for (int k = 0; k < 5; ++k) {
    p[k] = PyLong_AsVoidPtr(args[k + 1]);
    if (PyErr_Occurred()) return nullptr;
  }
  Py_INCREF(args[0]);
  grid_type = reinterpret_cast<PyTypeObject*>(args[0]);
  workspace_bytes = reinterpret_cast<decltype(workspace_bytes)>(p[0]);
  sort_entry = reinterpret_cast<decltype(sort_entry)>(p[1]);
  gather_entry = reinterpret_cast<decltype(gather_entry)>(p[2]);
  push_entry = reinterpret_cast<decltype(push_entry)>(p[3]);
  collide_entry = reinterpret_cast<decltype(collide_entry)>(p[4]);
  Py_RETURN_NONE;
}

PyMethodDef methods[] = {
    {"bind", reinterpret_cast<PyCFunction>(bind), METH_FASTCALL, nullptr},
    {"sort", reinterpret_cast<PyCFunction>(sort), METH_FASTCALL, nullptr},
    {"gather", reinterpret_cast<PyCFunction>(gather), METH_FASTCALL, nullptr},
    {"collide", reinterpret_cast<PyCFunction>(collide), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_binding", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

// What the build compiled this against; another PyTorch or Python has other internals (see _native.py).
PyMODINIT_FUNC PyInit__binding() {
  PyObject* made = PyModule_Create(&module);
  if (made && PyModule_AddStringConstant(made, "built_for", AETHER_BUILT_FOR) != 0) Py_CLEAR(made);
  return made;
}
