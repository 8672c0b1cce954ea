// Host path of the evaluators in C++: argument checks, descriptor tables, uploads, launches and result views.
//
// A pass of a small batch is bounded by the host: reading the attributes of a few hundred tensors, filling
// the descriptor tables with numpy and making result views took 120-900 us in Python where the GPU works
// 40-400 us. Each function here takes the whole step for plain arguments: lists or tuples of ordinary
// contiguous tensors of the usual types on the current device, with no dispatch mode or transform active.
// For anything else it returns None before it has changed or launched anything, and the caller takes the
// general Python path, which converts what can be converted and raises what has to be raised. Both fill the
// same tables. Instance and joint updates differ in their launches: here gathering, sorting, sampling and
// clearing are one (pe_inst_begin), masks may be streamed and an unchecked update matches from the pixel
// counts; the Python path gathers, sorts, contracts and prepares by a launch each. The results are the same.
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/ops/cat.h>
#include <ATen/ops/empty.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <initializer_list>
#include <optional>
#include <vector>

#include "pe_fields.h"
#include "pe_gb300.h"

namespace {

using at::Tensor;
using namespace pe;

// ---- the C ABI, bound to the addresses of the library that the Python layer loaded ------------------

#define PE_HOST_API(X)                                                                              \
  X(pe_update) X(pe_zero) X(pe_compute) X(pe_reward_pq) X(pe_pack) X(pe_pack_rgb) X(pe_contract_maps)          \
  X(pe_contract_blocks) X(pe_inst_begin) X(pe_seg_sort) X(pe_seg_sort_workspace)                   \
  X(pe_inst_counts) X(pe_inst_match) X(pe_stream_limit) X(pe_inst_prepare) X(pe_seg_match) X(pe_instance_accumulate)                  \
  X(pe_instance_accumulate_workspace) X(pe_seg_pass) X(pe_seg_score) X(pe_prefix)

struct Api {
#define X(name) decltype(&::name) name = nullptr;
  PE_HOST_API(X)
#undef X
} api;

// ---- small helpers ----------------------------------------------------------------------------------

struct Ref {
  PyObject* p;
  explicit Ref(PyObject* o = nullptr) : p(o) {}
  Ref(Ref&& o) noexcept : p(o.p) { o.p = nullptr; }
  Ref(const Ref&) = delete;
  Ref& operator=(const Ref&) = delete;
  ~Ref() { Py_XDECREF(p); }
  bool is_none() const { return p == Py_None; }
  explicit operator bool() const { return p != nullptr; }
};

struct ReleaseGil {
  PyThreadState* state = PyEval_SaveThread();
  ~ReleaseGil() { PyEval_RestoreThread(state); }
};

// Attribute names, interned once.
#define PE_HOST_NAMES(X)                                                                                       \
  X(segment_map) X(classes) X(crowd) X(lookup_ids) X(lookup_slots) X(tp) X(fp) X(fn) X(iou_sum) X(confusion)    \
  X(isthing) X(num_classes) X(validate) X(_scratch) X(_default_crowd) X(_validation_error) X(_state) X(masks)   \
  X(scores) X(areas) X(_store) X(_counts) X(_arena) X(n) X(capacity) X(ranks) X(flags) X(reserve) X(instance)   \
  X(panoptic) X(_isthing_u8) X(_side) X(cuda_stream) X(desc) X(descs) X(d_off) X(g_off) X(pair_off)             \
  X(total_chunks) X(id) X(category_id) X(iscrowd) X(flat) X(_layout)

struct Names {
#define X(name) PyObject* name = nullptr;
  PE_HOST_NAMES(X)
#undef X
} names;

Ref attr(PyObject* o, PyObject* name) {
  PyObject* v = PyObject_GetAttr(o, name);
  if (!v) PyErr_Clear();
  return Ref(v);
}

PyObject* attr_steal(PyObject* o, PyObject* name) {
  Ref r = attr(o, name);
  PyObject* p = r.p;
  r.p = nullptr;
  return p;
}

std::optional<int64_t> integer(const Ref& r) {
  if (!r || !PyLong_Check(r.p)) return std::nullopt;
  int overflow = 0;
  const long long v = PyLong_AsLongLongAndOverflow(r.p, &overflow);
  if (overflow) return std::nullopt;
  return (int64_t)v;
}

// No dispatch mode, functorch transform or other interception: torch calls made here and in Python agree.
bool ordinary() {
  if (c10::impl::TorchDispatchModeTLS::any_modes_set()) return false;
  return !c10::impl::tls_local_dispatch_key_set().included_.has(c10::DispatchKey::FuncTorchDynamicLayerFrontMode);
}

constexpr int kHostOnly = -2;  // tables over CPU tensors, for comparison with the general path's

// An ordinary contiguous tensor on CUDA device `index`, or nothing.
std::optional<Tensor> plain(PyObject* o, int index) {
  if (!o || !THPVariable_CheckExact(o)) return std::nullopt;
  const Tensor& t = THPVariable_Unpack(o);
  if (!t.defined() || t.layout() != at::kStrided || !t.is_contiguous() || t.is_neg()) return std::nullopt;
  if (t.unsafeGetTensorImpl()->is_python_dispatch() || !t.has_storage()) return std::nullopt;
  if (index == kHostOnly ? !t.is_cpu() : (!t.is_cuda() || t.get_device() != index)) return std::nullopt;
  return t;
}

std::optional<Tensor> plain(const Ref& r, int index) { return r ? plain(r.p, index) : std::nullopt; }

bool is(const Tensor& t, at::ScalarType type, std::initializer_list<int64_t> sizes) {
  return t.scalar_type() == type && t.sizes() == at::IntArrayRef(sizes.begin(), sizes.size());
}

// Tensors of a list or tuple (held while their pointers are in use), all of them ordinary and on `index`.
bool tensors(PyObject* seq, int index, std::vector<Tensor>& out) {
  if (!PyList_CheckExact(seq) && !PyTuple_CheckExact(seq)) return false;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
  PyObject** items = PySequence_Fast_ITEMS(seq);
  out.reserve(n);
  for (Py_ssize_t i = 0; i < n; ++i) {
    auto t = plain(items[i], index);
    if (!t) return false;
    out.push_back(std::move(*t));
  }
  return true;
}

at::TensorOptions on(int index, at::ScalarType type) { return at::device(at::Device(at::kCUDA, index)).dtype(type); }

// Upload buffer: pinned (freed buffers are reused once the copies from them are done).
Tensor staging(int64_t bytes, int index) {
  return at::empty({std::max<int64_t>(bytes, 1)}, at::TensorOptions().dtype(at::kByte).pinned_memory(index >= 0));
}

// A contiguous view of a fresh allocation's bytes, without the dispatcher (a result has up to 40 of them).
PyObject* view(const Tensor& base, int64_t byte_offset, at::ScalarType type, at::IntArrayRef sizes) {
  Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::TensorImpl::VIEW, c10::Storage(base.storage()),
                                                      base.key_set(), c10::scalarTypeToTypeMeta(type));
  auto* impl = t.unsafeGetTensorImpl();
  impl->set_storage_offset(byte_offset / (int64_t)c10::elementSize(type));
  impl->set_sizes_contiguous(sizes);
  return THPVariable_Wrap(t);
}

int64_t round_up(int64_t n, int64_t a) { return (n + a - 1) / a * a; }
int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }
int64_t address(const Tensor& t) { return reinterpret_cast<int64_t>(t.data_ptr()); }
template <typename T>
T* at_address(int64_t p) { return reinterpret_cast<T*>(p); }
template <typename T>
T* data(const Tensor& t) { return reinterpret_cast<T*>(t.data_ptr()); }

cudaStream_t current_stream(int index) { return c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)index).stream(); }

int sm_count(int index) {
  static int counts[64] = {0};
  if (index == kHostOnly) return 152;
  if (index < 0 || index >= 64) return 1;
  if (!counts[index]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, index) != cudaSuccess || n <= 0) return 1;
    counts[index] = n;
  }
  return counts[index];
}

// Offsets of 256-byte-aligned parts of one device buffer.
struct Layout {
  int64_t size = 0;
  int64_t add(int64_t bytes) {
    const int64_t off = size;
    size = round_up(size + std::max<int64_t>(bytes, 1), 256);
    return off;
  }
};

// The evaluator's scratch buffer of at least `bytes`, kept between calls as the general path keeps its own.
Tensor arena(PyObject* self, int index, int64_t bytes) {
  auto held = plain(attr(self, names._arena), index);
  if (held && held->scalar_type() == at::kByte && held->numel() >= bytes) return *held;
  Tensor fresh = at::empty({held ? bytes + bytes / 4 : bytes}, on(index, at::kByte));
  Ref object(THPVariable_Wrap(fresh));
  if (!object || PyObject_SetAttr(self, names._arena, object.p) < 0) throw python_error();
  return fresh;
}

PyObject* none() { Py_RETURN_NONE; }

bool set(PyObject* dict, const char* key, PyObject* value) {  // steals value
  if (!value) return false;
  const bool ok = PyDict_SetItemString(dict, key, value) == 0;
  Py_DECREF(value);
  return ok;
}

// ---- panoptic -----------------------------------------------------------------------------------------

struct Maps {
  Tensor maps, classes;
  int64_t images() const { return maps.size(0); }
  int64_t slots() const { return classes.size(1); }
};

// A compact PanopticBatch: B x H x W and B x S int32 on one device.
bool read_maps(PyObject* batch, int index, Maps& out) {
  if (!attr(batch, names.lookup_ids).is_none() || !attr(batch, names.lookup_slots).is_none()) return false;
  auto maps = plain(attr(batch, names.segment_map), index);
  auto classes = plain(attr(batch, names.classes), index);
  if (!maps || !classes || maps->dim() != 3 || classes->dim() != 2 || maps->scalar_type() != at::kInt ||
      classes->scalar_type() != at::kInt || classes->size(0) != maps->size(0) || classes->size(1) < 1)
    return false;
  out.maps = *maps;
  out.classes = *classes;
  return true;
}

// The batch's crowd flags (B x S bool); `missing` when it has none.
bool read_crowd(PyObject* batch, const Maps& m, int index, std::optional<Tensor>& crowd, bool& missing) {
  Ref r = attr(batch, names.crowd);
  if (!r) return false;
  missing = r.is_none();
  if (missing) return true;
  crowd = plain(r, index);
  return crowd && is(*crowd, at::kBool, {m.images(), m.slots()});
}

struct PanopticState {
  Tensor tp, fp, fn, iou_sum, confusion;
  int64_t C = 0;
};

bool read_state(PyObject* self, int index, PanopticState& s) {
  const auto C = integer(attr(self, names.num_classes));
  auto tp = plain(attr(self, names.tp), index), fp = plain(attr(self, names.fp), index);
  auto fn = plain(attr(self, names.fn), index), sums = plain(attr(self, names.iou_sum), index);
  auto confusion = plain(attr(self, names.confusion), index);
  if (!C || !tp || !fp || !fn || !sums || !confusion) return false;
  if (!is(*tp, at::kLong, {*C}) || !is(*fp, at::kLong, {*C}) || !is(*fn, at::kLong, {*C}) ||
      !is(*sums, at::kDouble, {*C}) || !is(*confusion, at::kLong, {*C, *C + 1}))
    return false;
  s = {*tp, *fp, *fn, *sums, *confusion, *C};
  return true;
}

// PanopticEvaluator.update of compact maps: the status of pe_update, or None.
PyObject* panoptic_update(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3 || !ordinary()) return none();
  PyObject* self = args[0];
  const int index = c10::cuda::current_device();
  Maps pred, gt;
  std::optional<Tensor> crowd;
  bool missing = false;
  PanopticState s;
  if (!read_maps(args[1], index, pred) || !read_maps(args[2], index, gt) || pred.maps.sizes() != gt.maps.sizes() ||
      !read_crowd(args[2], gt, index, crowd, missing) || !read_state(self, index, s))
    return none();
  const int64_t B = gt.images(), G = gt.slots(), P = pred.slots();
  if (missing) {
    crowd = plain(attr(self, names._default_crowd), index);
    if (!crowd || !is(*crowd, at::kBool, {B, G})) return none();
  }
  auto error = plain(attr(self, names._validation_error), index);
  Ref validate = attr(self, names.validate), scratch = attr(self, names._scratch);
  if (!error || !is(*error, at::kInt, {1}) || !validate || !scratch) return none();
  std::vector<Tensor> work;
  if (scratch.is_none() || !tensors(scratch.p, index, work) || work.size() != 3 || !is(work[0], at::kLong, {B, G, P})) {
    work = {at::empty({B, G, P}, on(index, at::kLong)), at::empty({B, G + P}, on(index, at::kLong)),
            at::empty({B, G}, on(index, at::kInt))};
    Ref fresh(PyTuple_Pack(3, Ref(THPVariable_Wrap(work[0])).p, Ref(THPVariable_Wrap(work[1])).p,
                           Ref(THPVariable_Wrap(work[2])).p));
    if (!fresh || PyObject_SetAttr(self, names._scratch, fresh.p) < 0) return nullptr;
  }
  const int check = PyObject_IsTrue(validate.p);
  if (check < 0) return nullptr;
  const cudaStream_t stream = current_stream(index);
  int code;
  {
    ReleaseGil released;
    code = api.pe_update(gt.maps.data_ptr(), 0, pred.maps.data_ptr(), 0, B, gt.maps.size(1) * gt.maps.size(2),
                         data<int32_t>(gt.classes), data<int32_t>(pred.classes), data<uint8_t>(*crowd), G, P, s.C,
                         data<int64_t>(work[0]), data<int64_t>(work[1]), data<int32_t>(work[2]), data<int64_t>(s.tp),
                         data<int64_t>(s.fp), data<int64_t>(s.fn), data<double>(s.iou_sum), data<int64_t>(s.confusion),
                         nullptr, nullptr, nullptr, nullptr, data<int32_t>(*error), check, 0, stream);
  }
  return PyLong_FromLong(code);
  END_HANDLE_TH_ERRORS
}

// Outputs of pe_compute for one row, laid out as _cuda_evaluator.compute_one lays them out.
struct ComputeOut {
  Tensor f64, i64;
};

ComputeOut compute_outputs(int index, int64_t C) {
  return {at::empty({5 * C + 10}, on(index, at::kDouble)), at::empty({3 + 3 * C + C * (C + 1)}, on(index, at::kLong))};
}

int launch_compute(const PanopticState& s, const Tensor& things, const ComputeOut& o, cudaStream_t stream) {
  const int64_t C = s.C;
  double* f = data<double>(o.f64);
  int64_t* conf = data<int64_t>(o.i64);
  int64_t* tail = conf + C * (C + 1);
  return api.pe_compute(data<int64_t>(s.tp), data<int64_t>(s.fp), data<int64_t>(s.fn), data<double>(s.iou_sum),
                        data<int64_t>(s.confusion), data<uint8_t>(things), 1, C, f, f + 4 * C, tail + 3 * C,
                        f + 4 * C + 9, tail, tail + C, tail + 2 * C, f + 4 * C + 10, conf, stream);
}

PyObject* compute_dict(const ComputeOut& o, int64_t C) {
  Ref result(PyDict_New()), classes(PyDict_New());
  if (!result || !classes) return nullptr;
  const int64_t tail = 8 * C * (C + 1);
  auto f64 = [&](int64_t k, at::IntArrayRef sizes) { return view(o.f64, 8 * k, at::kDouble, sizes); };
  auto i64 = [&](int64_t off, at::IntArrayRef sizes) { return view(o.i64, off, at::kLong, sizes); };
  const char* groups[3] = {"All", "Things", "Stuff"};
  const char* metrics[4] = {"pq", "sq", "rq", "iou"};
  for (int g = 0; g < 3; ++g) {
    Ref group(PyDict_New());
    if (!group) return nullptr;
    for (int m = 0; m < 3; ++m)
      if (!set(group.p, metrics[m], f64(4 * C + 3 * g + m, {}))) return nullptr;
    if (!set(group.p, "n", i64(tail + 8 * (3 * C + g), {}))) return nullptr;
    if (PyDict_SetItemString(result.p, groups[g], group.p) < 0) return nullptr;
  }
  for (int m = 0; m < 4; ++m)
    if (!set(classes.p, metrics[m], f64(m * C, {C}))) return nullptr;
  if (PyDict_SetItemString(result.p, "per_class", classes.p) < 0 || !set(result.p, "miou", f64(4 * C + 9, {})) ||
      !set(result.p, "tp", i64(tail, {C})) || !set(result.p, "fp", i64(tail + 8 * C, {C})) ||
      !set(result.p, "fn", i64(tail + 16 * C, {C})) || !set(result.p, "iou_sum", f64(4 * C + 10, {C})) ||
      !set(result.p, "confusion", i64(0, {C, C + 1})))
    return nullptr;
  PyObject* out = result.p;
  result.p = nullptr;
  return out;
}

bool read_things(PyObject* self, int index, int64_t C, std::optional<Tensor>& things) {
  things = plain(attr(self, names.isthing), index);
  return things && is(*things, at::kBool, {C});
}

// PanopticEvaluator.compute: (status, result dict), or None.
PyObject* panoptic_compute(PyObject*, PyObject* self) {
  HANDLE_TH_ERRORS
  if (!ordinary()) return none();
  const int index = c10::cuda::current_device();
  PanopticState s;
  std::optional<Tensor> things;
  if (!read_state(self, index, s) || !read_things(self, index, s.C, things)) return none();
  const ComputeOut o = compute_outputs(index, s.C);
  const int code = launch_compute(s, *things, o, current_stream(index));
  Ref result(code < 0 ? (Py_INCREF(Py_None), Py_None) : compute_dict(o, s.C));
  if (!result) return nullptr;
  return Py_BuildValue("(iO)", code, result.p);
  END_HANDLE_TH_ERRORS
}

// Zeroes an ordinary tensor on the current stream: True, or None.
PyObject* zero(PyObject*, PyObject* object) {
  HANDLE_TH_ERRORS
  if (!ordinary()) return none();
  const int index = c10::cuda::current_device();
  auto t = plain(object, index);
  if (!t) return none();
  if (api.pe_zero(t->data_ptr(), (int64_t)t->nbytes(), current_stream(index)) != 0) {
    PyErr_SetString(PyExc_RuntimeError, "clearing the accumulators failed");
    return nullptr;
  }
  Py_RETURN_TRUE;
  END_HANDLE_TH_ERRORS
}

// panoptic_quality of compact maps: (status, [B] scores), or None.
PyObject* reward(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4 || !ordinary()) return none();
  const int index = c10::cuda::current_device();
  Maps pred, gt;
  std::optional<Tensor> crowd;
  bool missing = false;
  int64_t C = PyLong_AsLongLong(args[2]);
  if (C <= 0) {
    PyErr_Clear();
    return none();
  }
  const int validate = PyObject_IsTrue(args[3]);
  if (validate < 0) return nullptr;
  if (!read_maps(args[0], index, pred) || !read_maps(args[1], index, gt) || pred.maps.sizes() != gt.maps.sizes() ||
      !read_crowd(args[1], gt, index, crowd, missing))
    return none();
  const int64_t B = gt.images(), G = gt.slots(), P = pred.slots();
  // pairs, areas, matched and error; then the [4, B, C] statistics and absent crowd flags, zeroed together.
  const int64_t longs = B * (G * P + G + P), ints = (B * G) / 2 + 1, rows = 4 * B * C;
  const int64_t zeroed = 8 * rows + (missing ? B * G : 0);
  Tensor work = at::empty({longs + ints + rows + (missing ? (B * G + 7) / 8 : 0)}, on(index, at::kLong));
  Tensor scores = at::empty({B}, on(index, at::kDouble));
  int64_t* pairs = data<int64_t>(work);
  int32_t* matched = reinterpret_cast<int32_t*>(pairs + longs);
  int64_t* stats = pairs + longs + ints;
  const uint8_t* flags = missing ? reinterpret_cast<uint8_t*>(stats + rows) : data<uint8_t>(*crowd);
  double* sums = reinterpret_cast<double*>(stats + 3 * B * C);
  const cudaStream_t stream = current_stream(index);
  int code = 0;
  {
    ReleaseGil released;
    code = api.pe_zero(stats, zeroed, stream);
    if (!code)
      code = api.pe_update(gt.maps.data_ptr(), 0, pred.maps.data_ptr(), 0, B, gt.maps.size(1) * gt.maps.size(2),
                           data<int32_t>(gt.classes), data<int32_t>(pred.classes), flags, G, P, C, pairs,
                           pairs + B * G * P, matched, stats, stats + B * C, stats + 2 * B * C, sums, nullptr, nullptr,
                           nullptr, nullptr, nullptr, matched + B * G, validate, 1, stream);
    if (!code)
      code = api.pe_reward_pq(stats, stats + B * C, stats + 2 * B * C, sums, B, C, data<double>(scores), nullptr,
                              nullptr, nullptr, nullptr, stream);
  }
  Ref out(THPVariable_Wrap(scores));
  return out ? Py_BuildValue("(iO)", code, out.p) : nullptr;
  END_HANDLE_TH_ERRORS
}

// Reads one device error word (GIL released while the stream drains); negative when the copy fails.
int read_error(const int32_t* error, cudaStream_t stream) {
  int code = 0;
  ReleaseGil released;
  if (cudaMemcpyAsync(&code, error, sizeof(int), cudaMemcpyDeviceToHost, stream) != cudaSuccess ||
      cudaStreamSynchronize(stream) != cudaSuccess)
    return -2;
  return code;
}

// PanopticBatch.from_coco(compact=True): (status, slot maps, classes, crowd), or None. Tables are those of
// evaluator.PanopticBatch.from_coco; anything its checks refuse goes there.
PyObject* coco_slots(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 3 || !ordinary()) return none();
  const int index = c10::cuda::current_device();
  auto maps = plain(args[0], index);
  if (!maps) return none();
  const bool rgb = maps->dim() == 4 && maps->size(3) == 3 && maps->scalar_type() == at::kByte;
  const bool wide = maps->scalar_type() == at::kLong;
  if (!rgb && !(maps->dim() == 3 && (wide || maps->scalar_type() == at::kInt))) return none();
  const int64_t B = maps->size(0), pixels = maps->size(1) * maps->size(2);
  if (B < 1) return none();
  if (!PyList_CheckExact(args[1]) && !PyTuple_CheckExact(args[1])) return none();
  if (PySequence_Fast_GET_SIZE(args[1]) != B) return none();
  if (!PyList_CheckExact(args[2]) && !PyTuple_CheckExact(args[2]) && !PyRange_Check(args[2])) return none();
  Ref categories(PySequence_Fast(args[2], "")), lookup(PyDict_New());
  if (!categories || !lookup) {
    PyErr_Clear();
    return none();
  }
  const Py_ssize_t n_categories = PySequence_Fast_GET_SIZE(categories.p);
  for (Py_ssize_t i = 0; i < n_categories; ++i) {
    Ref position(PyLong_FromSsize_t(i));
    if (!position || PyDict_SetItem(lookup.p, PySequence_Fast_GET_ITEM(categories.p, i), position.p) < 0) {
      PyErr_Clear();
      return none();
    }
  }
  if (PyDict_GET_SIZE(lookup.p) != n_categories) return none();
  PyObject** infos = PySequence_Fast_ITEMS(args[1]);
  Py_ssize_t most = 0;
  for (int64_t b = 0; b < B; ++b) {
    if (!PyList_CheckExact(infos[b]) && !PyTuple_CheckExact(infos[b])) return none();
    most = std::max(most, PySequence_Fast_GET_SIZE(infos[b]));
  }
  const int64_t S = most + 1, cells = B * S;
  Tensor host = staging(17 * cells, index);
  int64_t* ids = data<int64_t>(host);
  int32_t* slots = reinterpret_cast<int32_t*>(ids + cells);
  int32_t* classes = slots + cells;
  uint8_t* crowd = reinterpret_cast<uint8_t*>(classes + cells);
  std::fill(ids, ids + cells, INT64_MAX);
  std::fill(slots, slots + cells, 0);
  std::fill(classes, classes + cells, -1);
  std::fill(crowd, crowd + cells, 0);
  std::vector<std::pair<int64_t, int32_t>> order;
  for (int64_t b = 0; b < B; ++b) {
    const Py_ssize_t n = PySequence_Fast_GET_SIZE(infos[b]);
    order.clear();
    for (Py_ssize_t i = 0; i < n; ++i) {
      PyObject* entry = PySequence_Fast_GET_ITEM(infos[b], i);
      if (!PyDict_CheckExact(entry)) return none();
      PyObject* id = PyDict_GetItemWithError(entry, names.id);
      PyObject* category = PyDict_GetItemWithError(entry, names.category_id);
      PyObject* position = category ? PyDict_GetItemWithError(lookup.p, category) : nullptr;
      int overflow = 0;
      const long long value = id && PyLong_CheckExact(id) ? PyLong_AsLongLongAndOverflow(id, &overflow) : 0;
      if (!position || overflow || value <= 0 || value >= INT64_MAX) {
        PyErr_Clear();
        return none();
      }
      PyObject* flag = PyDict_GetItemWithError(entry, names.iscrowd);
      const int is_crowd = flag ? PyObject_IsTrue(flag) : 0;
      if (is_crowd < 0 || PyErr_Occurred()) {
        PyErr_Clear();
        return none();
      }
      classes[b * S + 1 + i] = (int32_t)PyLong_AsLong(position);
      crowd[b * S + 1 + i] = (uint8_t)is_crowd;
      order.emplace_back((int64_t)value, (int32_t)(i + 1));
    }
    std::sort(order.begin(), order.end());
    ids[b * S] = 0;
    for (Py_ssize_t i = 0; i < n; ++i) {
      if (i && order[i].first == order[i - 1].first) return none();
      ids[b * S + 1 + i] = order[i].first;
      slots[b * S + 1 + i] = order[i].second;
    }
  }
  // Tables (one upload) and the error word of the lookup, in one allocation.
  const int64_t error_at = round_up(17 * cells, 16);
  Tensor tables = at::empty({error_at + 16}, on(index, at::kByte));
  Tensor packed = at::empty({B, maps->size(1), maps->size(2)}, on(index, at::kInt));
  tables.narrow(0, 0, 17 * cells).copy_(host.narrow(0, 0, 17 * cells), /*non_blocking=*/true);
  const int64_t base = address(tables);
  const cudaStream_t stream = current_stream(index);
  int32_t* error = at_address<int32_t>(base + error_at);
  int code = rgb ? api.pe_pack_rgb(data<uint8_t>(*maps), B, pixels, at_address<int64_t>(base),
                                   at_address<int32_t>(base + 8 * cells), S, data<int32_t>(packed), error, stream)
                 : api.pe_pack(maps->data_ptr(), wide, B, pixels, at_address<int64_t>(base),
                               at_address<int32_t>(base + 8 * cells), S, data<int32_t>(packed), error, stream);
  if (!code) code = read_error(error, stream);
  Ref out(THPVariable_Wrap(packed)), labels(view(tables, 12 * cells, at::kInt, {B, S}));
  Ref flags(view(tables, 16 * cells, at::kBool, {B, S}));
  if (!out || !labels || !flags) return nullptr;
  return Py_BuildValue("(iOOO)", code, out.p, labels.p, flags.p);
  END_HANDLE_TH_ERRORS
}

// ---- instances ----------------------------------------------------------------------------------------

constexpr int kChains = 40;
constexpr int64_t kMaxImagePixels = (int64_t(1) << 32) - 1;

// The record store's tail for `extra` more records.
struct Tail {
  int64_t n = 0;
  double* scores = nullptr;
  int32_t* classes = nullptr;
  int32_t* ranks = nullptr;
  int8_t* flags = nullptr;
  std::vector<Tensor> held;
};

bool record_tail(PyObject* store, int index, int64_t extra, Tail& t) {
  const auto n = integer(attr(store, names.n));
  auto capacity = integer(attr(store, names.capacity));
  if (!n || !capacity) return false;
  if (*n + extra > *capacity) {
    Ref amount(PyLong_FromLongLong(extra));
    Ref grown(PyObject_CallMethodOneArg(store, names.reserve, amount.p));
    if (!grown) throw python_error();
    capacity = integer(attr(store, names.capacity));
  }
  auto scores = plain(attr(store, names.scores), index), classes = plain(attr(store, names.classes), index);
  auto ranks = plain(attr(store, names.ranks), index), flags = plain(attr(store, names.flags), index);
  if (!capacity || !scores || !classes || !ranks || !flags || !is(*scores, at::kDouble, {*capacity}) ||
      !is(*classes, at::kInt, {*capacity}) || !is(*ranks, at::kInt, {*capacity}) ||
      !is(*flags, at::kChar, {*capacity, kChains}))
    return false;
  t.n = *n;
  t.scores = data<double>(*scores) + *n;
  t.classes = data<int32_t>(*classes) + *n;
  t.ranks = data<int32_t>(*ranks) + *n;
  t.flags = data<int8_t>(*flags) + *n * kChains;
  t.held = {*scores, *classes, *ranks, *flags};
  return true;
}

bool store_count(PyObject* store, int64_t n) {
  Ref value(PyLong_FromLongLong(n));
  return value && PyObject_SetAttr(store, names.n, value.p) == 0;
}

struct Metadata {  // one per-image field: its tensors and, per image, whether it has the wider type
  std::vector<Tensor> held;
  bool wide(size_t b, at::ScalarType type) const { return held[b].scalar_type() == type; }
};

// Field of per-image vectors of `sizes` elements in one of two types; absent when the attribute is None.
bool read_field(PyObject* batch, PyObject* name, int index, const std::vector<int64_t>& sizes, at::ScalarType narrow,
                at::ScalarType wide, bool optional, Metadata& out) {
  Ref r = attr(batch, name);
  if (!r) return false;
  if (r.is_none()) return optional;
  if (!tensors(r.p, index, out.held) || out.held.size() != sizes.size()) return false;
  for (size_t b = 0; b < sizes.size(); ++b) {
    const Tensor& t = out.held[b];
    if (t.dim() != 1 || t.size(0) != sizes[b] || (t.scalar_type() != narrow && t.scalar_type() != wide)) return false;
  }
  return true;
}

// The masks of a batch: N x H x W bool per image, in place.
bool read_masks(PyObject* batch, int index, std::vector<Tensor>& masks, std::vector<int64_t>& counts) {
  Ref r = attr(batch, names.masks);
  if (!r || !tensors(r.p, index, masks)) return false;
  for (const Tensor& m : masks) {
    if (m.dim() != 3 || m.scalar_type() != at::kBool || m.size(1) <= 0 || m.size(2) <= 0) return false;
    if (m.size(1) * m.size(2) > kMaxImagePixels) return false;
    counts.push_back(m.size(0));
  }
  return true;
}

// Offsets that follow the descriptors in an upload: d_off [B + 1], g_off [B + 1], pair_off [B].
int64_t table_words(int64_t B) { return B * kDescFields + 3 * B + 2; }

void fill_offsets(int64_t* words, int64_t B) {
  int64_t* d_off = words + B * kDescFields;
  int64_t* g_off = d_off + B + 1;
  int64_t* pair_off = g_off + B + 1;
  d_off[0] = g_off[0] = 0;
  for (int64_t b = 0; b < B; ++b) {
    const int64_t* d = words + b * kDescFields;
    d_off[b + 1] = d_off[b] + d[kD];
    g_off[b + 1] = g_off[b] + d[kG];
    pair_off[b] = d[kDPairBegin];
  }
}

struct InstancePlan {
  std::vector<Tensor> pm, gm;
  std::vector<int64_t> dets, gts;
  Metadata pc, scores, gc, crowd, areas;
  int64_t B = 0, total_d = 0, total_g = 0, pairs = 0, max_g = 1;
  int64_t n_blocks = 0, total_chunks = 0, ranges = 0, chunks = 0, stream_limit = 0;
  int64_t bounds_at = 0, blocks_at = 0, maps_at = -1, rows_at = 0, words = 0;
  Tensor host;
};

// Checks and tables of InstanceEvaluator.update (the general path's DescTable, contract_plan and gather_rows),
// in one pinned buffer: descriptors, offsets, contraction bounds, blocks, tensor maps, field rows.
bool plan_instances(PyObject* prediction, PyObject* target, int index, PyObject* costs, double default_cost,
                    InstancePlan& p) {
  constexpr int64_t kRowsA = 127, kRowsB = 63, kChunk = 4096;
  if (!read_masks(prediction, index, p.pm, p.dets) || !read_masks(target, index, p.gm, p.gts)) return false;
  p.B = (int64_t)p.pm.size();
  const int64_t B = p.B;
  if (B == 0 || (int64_t)p.gm.size() != B) return false;
  Metadata unused;
  if (!read_field(prediction, names.classes, index, p.dets, at::kInt, at::kLong, false, p.pc) ||
      !read_field(prediction, names.scores, index, p.dets, at::kFloat, at::kDouble, false, p.scores) ||
      !read_field(prediction, names.crowd, index, p.dets, at::kBool, at::kBool, true, unused) ||
      !read_field(target, names.classes, index, p.gts, at::kInt, at::kLong, false, p.gc) ||
      !read_field(target, names.crowd, index, p.gts, at::kBool, at::kBool, true, p.crowd) ||
      !read_field(target, names.areas, index, p.gts, at::kFloat, at::kDouble, true, p.areas))
    return false;
  if (!attr(prediction, names.areas).is_none() || !attr(target, names.scores).is_none()) return false;
  std::vector<int64_t> pixels(B), table(B * kDescFields, 0);
  std::vector<uint8_t> tma(B);
  int64_t cap = 0, chunks = 0;
  for (int64_t b = 0; b < B; ++b) {
    if (p.pm[b].size(1) != p.gm[b].size(1) || p.pm[b].size(2) != p.gm[b].size(2)) return false;
    pixels[b] = p.pm[b].size(1) * p.pm[b].size(2);
    int64_t* d = table.data() + b * kDescFields;
    const int64_t pm = address(p.pm[b]), gm = address(p.gm[b]), D = p.dets[b], G = p.gts[b];
    d[kPixels] = d[kMaskStride] = pixels[b];
    d[kMasks] = pm;
    d[kTarget] = gm;
    d[kD] = D;
    d[kG] = G;
    d[kDetBegin] = p.total_d;
    d[kSlotBegin] = p.total_g;
    d[kDPairBegin] = p.pairs;
    d[kChunkBegin] = chunks;
    d[kFlags] = (pm | gm | pixels[b]) % 16 == 0 ? 2 : 0;
    p.total_d += D;
    p.total_g += G;
    p.pairs += D * G;
    p.max_g = std::max(p.max_g, G);
    chunks += ceil_div(pixels[b], kChunk);
    cap += (ceil_div(D, kRowsA) + 1) * (ceil_div(G, kRowsB) + 1);
  }
  const int64_t ctas = sm_count(index);
  p.bounds_at = table_words(B);
  p.blocks_at = p.bounds_at + ctas + 1;
  const int64_t maps_at = round_up(p.blocks_at + 4 * cap, 8);
  p.rows_at = maps_at + 32 * B;
  p.words = p.rows_at + 6 * B;
  p.host = staging(8 * p.words, index);
  int64_t* words = data<int64_t>(p.host);
  if (reinterpret_cast<uintptr_t>(words) % 64) return false;  // allocators give 64 bytes and more
  const int given = api.pe_contract_maps(table.data(), B, words + maps_at);
  if (given < 0) return false;
  p.maps_at = given ? maps_at : -1;
  double cost = default_cost;
  if (given) {
    int64_t loaded = 0, bytes = 0;
    for (int64_t b = 0; b < B; ++b) {
      tma[b] = (table[b * kDescFields + kFlags] & 4) != 0;
      const int64_t n = (p.dets[b] + p.gts[b]) * pixels[b];
      bytes += n;
      loaded += tma[b] ? n : 0;
    }
    Ref bucket(PyLong_FromLongLong(bytes ? 10 * loaded / bytes : 0));
    PyObject* tuned = bucket ? PyDict_GetItemWithError(costs, bucket.p) : nullptr;
    if (tuned) cost = PyFloat_AsDouble(tuned);
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
  }
  p.n_blocks = api.pe_contract_blocks(p.dets.data(), p.gts.data(), pixels.data(), given ? tma.data() : nullptr, B, cost,
                                      ctas, words + p.blocks_at, cap, words + p.bounds_at, &p.total_chunks, &p.ranges);
  if (p.n_blocks < 0) return false;
  p.chunks = chunks;
  p.stream_limit = api.pe_stream_limit(p.dets.data(), p.gts.data(), pixels.data(), given ? tma.data() : nullptr, B, ctas);
  if (p.stream_limit < 0) return false;
  std::memcpy(words, table.data(), 8 * B * kDescFields);
  fill_offsets(words, B);
  for (int64_t b = 0; b < B; ++b) {
    int64_t* r = words + p.rows_at + 6 * b;
    r[0] = address(p.pc.held[b]);
    r[1] = address(p.scores.held[b]);
    r[2] = address(p.gc.held[b]);
    r[3] = p.crowd.held.empty() ? 0 : address(p.crowd.held[b]);
    r[4] = p.areas.held.empty() ? 0 : address(p.areas.held[b]);
    r[5] = (p.pc.wide(b, at::kLong) ? 1 : 0) | (p.scores.wide(b, at::kDouble) ? 2 : 0) |
           (p.gc.wide(b, at::kLong) ? 4 : 0) | (!p.areas.held.empty() && p.areas.wide(b, at::kDouble) ? 16 : 0);
  }
  return true;
}

// The words plan_instances uploads for CPU tensors, and where its parts start: (bytes, bounds, blocks, maps or -1, rows, number of blocks, chunks, ranges), or None.
PyObject* instance_tables(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4 || !ordinary()) return none();
  InstancePlan p;
  if (!plan_instances(args[0], args[1], kHostOnly, args[2], PyFloat_AsDouble(args[3]), p)) return none();
  Ref bytes(PyBytes_FromStringAndSize(data<char>(p.host), 8 * p.words));
  if (!bytes) return nullptr;
  return Py_BuildValue("(OLLLLLLL)", bytes.p, (long long)p.bounds_at, (long long)p.blocks_at, (long long)p.maps_at,
                       (long long)p.rows_at, (long long)p.n_blocks, (long long)p.total_chunks, (long long)p.ranges);
  END_HANDLE_TH_ERRORS
}

// InstanceEvaluator.update (self, prediction, target, tuned costs, default cost): the error bits (negative: a
// failed call), or None. The records are counted only when no bit is set.
PyObject* instance_update(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 5 || !ordinary()) return none();
  PyObject* self = args[0];
  const int index = c10::cuda::current_device();
  const auto C = integer(attr(self, names.num_classes));
  Ref validate = attr(self, names.validate), store = attr(self, names._store);
  auto counts = plain(attr(self, names._counts), index);
  if (!C || !validate || !store || !counts || !is(*counts, at::kLong, {*C, 4})) return none();
  const int check = PyObject_IsTrue(validate.p);
  if (check < 0) return nullptr;
  InstancePlan p;
  if (!plan_instances(args[1], args[2], index, args[3], PyFloat_AsDouble(args[4]), p)) return none();
  Tail tail;
  if (!record_tail(store.p, index, p.total_d, tail)) return none();
  const int64_t B = p.B, D = p.total_d, G = p.total_g;
  const int64_t sort_bytes = api.pe_seg_sort_workspace(D);
  Layout l;
  const int64_t table_at = l.add(8 * p.words), pc_at = l.add(4 * D), scores_at = l.add(8 * D), gc_at = l.add(4 * G);
  const int64_t crowd_at = l.add(G), ann_in_at = l.add(8 * G), order_at = l.add(8 * D), sort_at = l.add(sort_bytes);
  const int64_t pa_d_at = l.add(8 * D), ga_d_at = l.add(8 * G), ann_at = l.add(8 * G);
  const int64_t bits_at = l.add(4 * B * ((*C + 31) / 32)), stream_at = l.add(8 * (8 * B + 1));
  // Intersections, the error word, then both area counters, without gaps: pe_inst_begin clears them at once.
  const int64_t inter_len = round_up(p.pairs, 2) + 2, counts_at = l.add(4 * inter_len + 8 * (D + G));
  Tensor work = arena(self, index, l.size);
  work.narrow(0, table_at, 8 * p.words).copy_(p.host.narrow(0, 0, 8 * p.words), /*non_blocking=*/true);
  const int64_t base = address(work), table = base + table_at;
  const int64_t* descs = at_address<int64_t>(table);
  const int64_t* d_off = descs + B * kDescFields;
  uint32_t* inter = at_address<uint32_t>(base + counts_at);
  int32_t* error = reinterpret_cast<int32_t*>(inter + inter_len - 2);
  uint64_t* pa = reinterpret_cast<uint64_t*>(inter + inter_len);
  double* ann_in = p.areas.held.empty() ? nullptr : at_address<double>(base + ann_in_at);
  int32_t* pc = at_address<int32_t>(base + pc_at);
  int32_t* gc = at_address<int32_t>(base + gc_at);
  double* scores = at_address<double>(base + scores_at);
  uint8_t* crowd = at_address<uint8_t>(base + crowd_at);
  int64_t* order = at_address<int64_t>(base + order_at);
  double* pa_d = at_address<double>(base + pa_d_at);
  double* ga_d = at_address<double>(base + ga_d_at);
  double* ann = at_address<double>(base + ann_at);
  uint32_t* bits = at_address<uint32_t>(base + bits_at);
  const cudaStream_t stream = current_stream(index);
  int code = 0;
  {
    ReleaseGil released;
    uint64_t* sample = at_address<uint64_t>(base + stream_at);
    code = api.pe_inst_begin(descs, descs + p.rows_at, B, pc, scores, gc, crowd, ann_in, D, order, tail.scores,
                             tail.classes, at_address<void>(base + sort_at), sort_bytes, inter, inter_len, pa, D,
                             pa + D, G, p.stream_limit, sample, *C, check ? nullptr : bits, stream);
    const int64_t* blocks = p.total_chunks ? descs + p.blocks_at : nullptr;
    const int64_t* bounds = p.total_chunks ? descs + p.bounds_at : nullptr;
    const int64_t* maps = p.maps_at >= 0 && p.total_chunks ? descs + p.maps_at : nullptr;
    if (!code)
      code = api.pe_inst_counts(descs, B, p.chunks, blocks, p.n_blocks, p.total_chunks, bounds, p.ranges, order, inter,
                                pa, pa + D, maps, p.stream_limit, sample, error, stream);
    if (!code && check) {
      code = api.pe_inst_prepare(descs, B, pa, pa + D, pa_d, ga_d, tail.classes, gc, tail.scores, ann_in, ann, *C, check,
                                 bits, error, stream);
      if (!code)
        code = api.pe_seg_match(inter, d_off + 2 * B + 2, d_off, d_off + B + 1, B, tail.classes, pa_d, gc, ga_d, crowd,
                                ann, *C, p.max_g, tail.flags, 1, kChains, tail.ranks, data<int64_t>(*counts), error,
                                bits, stream);
    } else if (!code) {
      code = api.pe_inst_match(inter, d_off + 2 * B + 2, d_off, d_off + B + 1, B, tail.classes, pa, gc, pa + D, crowd,
                               ann_in, *C, p.max_g, tail.flags, 1, kChains, tail.ranks, data<int64_t>(*counts), error,
                               bits, stream);
    }
  }
  if (!code && check) code = read_error(error, stream);
  if (!code && !store_count(store.p, tail.n + D)) return nullptr;
  return PyLong_FromLong(code);
  END_HANDLE_TH_ERRORS
}

struct Accumulation {
  Tensor out, work;
  int64_t C = 0, n = 0;
  Tail records;
  Tensor counts;
};

bool plan_accumulation(PyObject* self, int index, Accumulation& a) {
  const auto C = integer(attr(self, names.num_classes));
  Ref store = attr(self, names._store);
  auto counts = plain(attr(self, names._counts), index);
  if (!C || !store || !counts || !is(*counts, at::kLong, {*C, 4}) || !record_tail(store.p, index, 0, a.records))
    return false;
  a.C = *C;
  a.n = a.records.n;
  a.counts = *counts;
  const int64_t bytes = api.pe_instance_accumulate_workspace(a.n, a.C);
  a.out = at::empty({10 * 102 * a.C * 12 + 12}, on(index, at::kDouble));
  a.work = arena(self, index, bytes);
  return true;
}

int launch_accumulation(const Accumulation& a, cudaStream_t stream) {
  double* precision = data<double>(a.out);
  double* recall = precision + 10 * 101 * a.C * 12;
  return api.pe_instance_accumulate(a.records.classes - a.n, a.records.ranks - a.n, a.records.flags - a.n * kChains, 1,
                                    kChains, a.records.scores - a.n, a.n, data<int64_t>(a.counts), a.C,
                                    a.work.data_ptr(), a.work.numel(), precision, recall, recall + 10 * a.C * 12,
                                    stream);
}

PyObject* accumulation_dict(const Accumulation& a) {
  static const char* keys[12] = {"ap", "ap50", "ap75", "ap_small", "ar_small", "ap_medium",
                                 "ar_medium", "ap_large", "ar_large", "ar1", "ar10", "ar100"};
  Ref result(PyDict_New());
  if (!result) return nullptr;
  const int64_t recall = 10 * 101 * a.C * 12, summary = recall + 10 * a.C * 12;
  for (int k = 0; k < 12; ++k)
    if (!set(result.p, keys[k], view(a.out, 8 * (summary + k), at::kDouble, {}))) return nullptr;
  if (!set(result.p, "precision", view(a.out, 0, at::kDouble, {10, 101, a.C, 4, 3})) ||
      !set(result.p, "recall", view(a.out, 8 * recall, at::kDouble, {10, a.C, 4, 3})))
    return nullptr;
  PyObject* out = result.p;
  result.p = nullptr;
  return out;
}

// InstanceEvaluator.compute: (status, result dict), or None.
PyObject* instance_compute(PyObject*, PyObject* self) {
  HANDLE_TH_ERRORS
  if (!ordinary()) return none();
  const int index = c10::cuda::current_device();
  Accumulation a;
  if (!plan_accumulation(self, index, a)) return none();
  const int code = launch_accumulation(a, current_stream(index));
  Ref result(code < 0 ? (Py_INCREF(Py_None), Py_None) : accumulation_dict(a));
  return result ? Py_BuildValue("(iO)", code, result.p) : nullptr;
  END_HANDLE_TH_ERRORS
}

// ---- combined -----------------------------------------------------------------------------------------

// Sizes of a batch of the fused pass, from its host descriptors.
struct SegSizes {
  int64_t B = 0, D = 0, slots = 0, pslots = 0, pairs = 0, dpairs = 0, max_g = 1, max_p = 1, pan_cap = 0, det_cap = 0;
  bool rows16 = true;

  void add(const int64_t* d) {
    const int64_t n = d[kD], g = d[kG], p = d[kP];
    ++B;
    D += n;
    slots += g;
    pslots += p;
    pairs += g * p;
    dpairs += n * g;
    max_g = std::max(max_g, g);
    max_p = std::max(max_p, p);
    pan_cap = std::max(pan_cap, g * p);
    det_cap = std::max(det_cap, n * g);
    rows16 = rows16 && (d[kFlags] & 2);
  }
};

struct SegInputs {
  const int64_t* descs = nullptr;     // device: descriptors, then d_off, g_off, pair_off
  const int64_t* d_off = nullptr;
  const int64_t* g_off = nullptr;
  const int64_t* pair_off = nullptr;
  int64_t total_chunks = 0;
  const int32_t* gc = nullptr;
  const int32_t* pc = nullptr;
  const uint8_t* crowd = nullptr;
  const int32_t* det_classes = nullptr;
  const double* det_scores = nullptr;
  const double* areas = nullptr;
  // With fields still to gather (pe_inst_gather's rows): the arrays they go to.
  const int64_t* rows = nullptr;
  int32_t* rows_classes = nullptr;
  double* rows_scores = nullptr;
  int32_t* rows_gc = nullptr;
  uint8_t* rows_crowd = nullptr;
};

struct SegEvaluator {
  PanopticState pan;
  Tensor counts, things;
  Tail tail;
  Ref store;
  int64_t C = 0;
  int validate = 0;
};

// State of a SegmentationEvaluator with room for `detections` more records.
bool read_segmentation(PyObject* self, int index, int64_t detections, SegEvaluator& ev) {
  Ref instance = attr(self, names.instance), panoptic = attr(self, names.panoptic), validate = attr(self, names.validate);
  const auto C = integer(attr(self, names.num_classes));
  if (!instance || !panoptic || !validate || !C) return false;
  auto counts = plain(attr(instance.p, names._counts), index);
  auto things = plain(attr(self, names._isthing_u8), index);
  if (!counts || !things || !is(*counts, at::kLong, {*C, 4}) || !is(*things, at::kByte, {*C}) ||
      !read_state(panoptic.p, index, ev.pan) || ev.pan.C != *C)
    return false;
  ev.store.p = attr_steal(instance.p, names._store);
  if (!ev.store || !record_tail(ev.store.p, index, detections, ev.tail)) return false;
  ev.counts = *counts;
  ev.things = *things;
  ev.C = *C;
  ev.validate = PyObject_IsTrue(validate.p);
  return ev.validate >= 0;
}

// Scratch of the fused pass and what follows it; the counts, the error word and the chunk counter have no
// gaps between them, so the pass clears them as one span.
struct SegScratch {
  Layout layout;
  int64_t order, sort, sort_bytes, areas, matched, det_pa, slot_ga, slot_class, ann, bits, counted, dpairs_len;

  SegScratch(const SegSizes& z, int64_t C) {
    order = layout.add(8 * z.D);
    sort_bytes = api.pe_seg_sort_workspace(z.D);
    sort = layout.add(sort_bytes);
    areas = layout.add(8 * (z.slots + z.pslots));
    matched = layout.add(4 * z.slots);
    det_pa = layout.add(8 * z.D);
    slot_ga = layout.add(8 * z.slots);
    slot_class = layout.add(4 * z.slots);
    ann = layout.add(8 * z.slots);
    bits = layout.add(4 * z.B * ((C + 31) / 32));
    dpairs_len = round_up(z.pairs + z.dpairs + 1, 2) - z.pairs;  // the error word is the last of them
    counted = layout.add(4 * (z.pairs + dpairs_len) + 8);
  }
};

int launch_seg(const SegSizes& z, const SegInputs& in, const SegScratch& w, SegEvaluator& ev, int64_t base,
               int32_t*& error, cudaStream_t stream) {
  int64_t* order = at_address<int64_t>(base + w.order);
  uint32_t* pairs = at_address<uint32_t>(base + w.counted);
  uint32_t* dpairs = pairs + z.pairs;
  error = reinterpret_cast<int32_t*>(dpairs + w.dpairs_len - 1);
  double* det_pa = at_address<double>(base + w.det_pa);
  double* slot_ga = at_address<double>(base + w.slot_ga);
  double* ann = at_address<double>(base + w.ann);
  int32_t* slot_class = at_address<int32_t>(base + w.slot_class);
  uint32_t* bits = at_address<uint32_t>(base + w.bits);
  void* sort = at_address<void>(base + w.sort);
  int code = in.rows ? api.pe_inst_begin(in.descs, in.rows, z.B, in.rows_classes, in.rows_scores, in.rows_gc,
                                         in.rows_crowd, nullptr, z.D, order, ev.tail.scores, ev.tail.classes, sort,
                                         w.sort_bytes, nullptr, 0, nullptr, 0, nullptr, 0, 0, nullptr, 0, nullptr, stream)
                     : api.pe_seg_sort(in.descs, z.B, in.det_scores, in.det_classes, z.D, order, ev.tail.scores,
                                       ev.tail.classes, sort, w.sort_bytes, stream);
  if (!code)
    code = api.pe_seg_pass(in.descs, z.B, in.total_chunks, order, pairs, z.pairs, dpairs, w.dpairs_len, z.pan_cap,
                           z.det_cap, z.rows16 ? 1 : 2, nullptr, 0, reinterpret_cast<uint64_t*>(dpairs + w.dpairs_len),
                           error, stream);
  if (!code)
    code = api.pe_seg_score(in.descs, z.B, z.max_p, z.pan_cap, pairs, dpairs, in.gc, in.pc, in.crowd,
                            at_address<int64_t>(base + w.areas), at_address<int32_t>(base + w.matched),
                            data<int64_t>(ev.pan.tp), data<int64_t>(ev.pan.fp), data<int64_t>(ev.pan.fn),
                            data<double>(ev.pan.iou_sum), data<int64_t>(ev.pan.confusion), ev.C,
                            data<uint8_t>(ev.things), ev.tail.classes, ev.tail.scores, det_pa, slot_ga, slot_class,
                            in.areas, ann, ev.validate, 0, bits, error, stream);
  if (!code)
    code = api.pe_seg_match(dpairs, in.pair_off, in.d_off, in.g_off, z.B, ev.tail.classes, det_pa, slot_class, slot_ga,
                            in.crowd, ann, ev.C, z.max_g, ev.tail.flags, 1, kChains, ev.tail.ranks,
                            data<int64_t>(ev.counts), error, bits, stream);
  return code;
}

PyObject* finish_seg(SegEvaluator& ev, const SegSizes& z, int code, const int32_t* error, cudaStream_t stream) {
  if (!code && ev.validate) code = read_error(error, stream);
  if (!code && !store_count(ev.store.p, ev.tail.n + z.D)) return nullptr;
  return PyLong_FromLong(code);
}

struct CombinedPlan {
  Maps gt, pred;
  Tensor crowd;
  std::vector<Tensor> masks;
  std::vector<int64_t> dets;
  Metadata classes, scores;
  SegSizes sizes;
  int64_t total_chunks = 0, rows_at = 0, words = 0;
  Tensor host;
};

// Checks and tables of SegmentationEvaluator.update (combined.run_batch): descriptors, offsets, field rows.
bool plan_combined(PyObject* prediction, PyObject* detections, PyObject* target, int index, CombinedPlan& p) {
  constexpr int64_t kChunk = 8192;
  std::optional<Tensor> crowd;
  bool missing = false;
  if (!read_maps(target, index, p.gt) || !read_maps(prediction, index, p.pred) ||
      p.gt.maps.sizes() != p.pred.maps.sizes() || !read_crowd(target, p.gt, index, crowd, missing) || missing ||
      !read_masks(detections, index, p.masks, p.dets))
    return false;
  const int64_t B = p.gt.images(), S = p.gt.slots(), P = p.pred.slots();
  if (B == 0 || (int64_t)p.masks.size() != B || !attr(detections, names.crowd).is_none() ||
      !attr(detections, names.areas).is_none() ||
      !read_field(detections, names.classes, index, p.dets, at::kInt, at::kLong, false, p.classes) ||
      !read_field(detections, names.scores, index, p.dets, at::kFloat, at::kDouble, false, p.scores))
    return false;
  p.crowd = *crowd;
  const int64_t pixels = p.gt.maps.size(1) * p.gt.maps.size(2), chunks = ceil_div(pixels, kChunk);
  const int64_t target_ptr = address(p.gt.maps), pred_ptr = address(p.pred.maps), classes_ptr = address(p.gt.classes);
  const int64_t maps16 = (target_ptr | pred_ptr) % 16 == 0 && pixels % 4 == 0 ? 1 : 0;
  p.rows_at = table_words(B);
  p.words = p.rows_at + 6 * B;
  p.host = staging(8 * p.words, index);
  int64_t* words = data<int64_t>(p.host);
  std::fill(words, words + p.words, 0);
  for (int64_t b = 0; b < B; ++b) {
    if (p.masks[b].size(1) != p.gt.maps.size(1) || p.masks[b].size(2) != p.gt.maps.size(2)) return false;
    int64_t* d = words + b * kDescFields;
    const int64_t masks = address(p.masks[b]);
    d[kTarget] = target_ptr + 4 * b * pixels;
    d[kPred] = pred_ptr + 4 * b * pixels;
    d[kMasks] = masks;
    d[kPixels] = d[kMaskStride] = pixels;
    d[kChunkBegin] = b * chunks;
    d[kDetBegin] = p.sizes.D;
    d[kSlotBegin] = b * S;
    d[kPSlotBegin] = b * P;
    d[kPairBegin] = b * S * P;
    d[kDPairBegin] = p.sizes.dpairs;
    d[kD] = p.dets[b];
    d[kG] = S;
    d[kP] = P;
    d[kFlags] = maps16 | ((masks | pixels) % 16 == 0 ? 2 : 0);
    p.sizes.add(d);
    int64_t* r = words + p.rows_at + 6 * b;
    r[0] = address(p.classes.held[b]);
    r[1] = address(p.scores.held[b]);
    r[2] = classes_ptr + 4 * b * S;  // the target columns are gathered too (and not read)
    r[5] = (p.classes.wide(b, at::kLong) ? 1 : 0) | (p.scores.wide(b, at::kDouble) ? 2 : 0);
  }
  fill_offsets(words, B);
  p.total_chunks = B * chunks;
  return true;
}

// The words plan_combined uploads for CPU tensors (descriptors, offsets, field rows) and the chunk count, or None.
PyObject* combined_tables(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  CombinedPlan p;
  if (nargs != 3 || !ordinary() || !plan_combined(args[0], args[1], args[2], kHostOnly, p)) return none();
  Ref bytes(PyBytes_FromStringAndSize(data<char>(p.host), 8 * p.words));
  return bytes ? Py_BuildValue("(OL)", bytes.p, (long long)p.total_chunks) : nullptr;
  END_HANDLE_TH_ERRORS
}

// SegmentationEvaluator.update (self, prediction, detections, target): the error bits, or None.
PyObject* combined_update(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4 || !ordinary()) return none();
  const int index = c10::cuda::current_device();
  CombinedPlan p;
  SegEvaluator ev;
  if (!plan_combined(args[1], args[2], args[3], index, p) || !read_segmentation(args[0], index, p.sizes.D, ev))
    return none();
  Ref instance = attr(args[0], names.instance);
  SegScratch w(p.sizes, ev.C);
  const int64_t table_at = w.layout.add(8 * p.words), classes_at = w.layout.add(4 * p.sizes.D);
  const int64_t scores_at = w.layout.add(8 * p.sizes.D), gc_at = w.layout.add(4 * p.sizes.slots);
  const int64_t crowd_at = w.layout.add(p.sizes.slots);
  Tensor work = arena(instance.p, index, w.layout.size);
  work.narrow(0, table_at, 8 * p.words).copy_(p.host.narrow(0, 0, 8 * p.words), /*non_blocking=*/true);
  const int64_t base = address(work), B = p.sizes.B;
  SegInputs in;
  in.descs = at_address<int64_t>(base + table_at);
  in.d_off = in.descs + B * kDescFields;
  in.g_off = in.d_off + B + 1;
  in.pair_off = in.g_off + B + 1;
  in.total_chunks = p.total_chunks;
  in.gc = data<int32_t>(p.gt.classes);
  in.pc = data<int32_t>(p.pred.classes);
  in.crowd = data<uint8_t>(p.crowd);
  if (p.sizes.D) in.rows = in.descs + p.rows_at;
  in.det_classes = in.rows_classes = at_address<int32_t>(base + classes_at);
  in.det_scores = in.rows_scores = at_address<double>(base + scores_at);
  in.rows_gc = at_address<int32_t>(base + gc_at);
  in.rows_crowd = at_address<uint8_t>(base + crowd_at);
  const cudaStream_t stream = current_stream(index);
  int32_t* error = nullptr;
  int code = 0;
  {
    ReleaseGil released;
    code = launch_seg(p.sizes, in, w, ev, base, error, stream);
  }
  return finish_seg(ev, p.sizes, code, error, stream);
  END_HANDLE_TH_ERRORS
}

// SegmentationEvaluator.update_images (self, table, arena tensor, field offsets): the error bits, or None.
// `offsets`: byte offsets in the arena of the target classes, crowd flags, prediction classes, detection classes,
// scores and annotation areas (-1: none).
PyObject* images_update(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 4 || !ordinary() || !PyTuple_CheckExact(args[3]) || PyTuple_GET_SIZE(args[3]) != 6) return none();
  const int index = c10::cuda::current_device();
  auto device = plain(args[2], index);
  auto descs = plain(attr(args[1], names.descs), index), d_off = plain(attr(args[1], names.d_off), index);
  auto g_off = plain(attr(args[1], names.g_off), index), pair_off = plain(attr(args[1], names.pair_off), index);
  const auto chunks = integer(attr(args[1], names.total_chunks));
  Ref table = attr(args[1], names.desc);
  if (!device || !descs || !d_off || !g_off || !pair_off || !chunks || !table || device->scalar_type() != at::kByte)
    return none();
  SegSizes sizes;
  {
    Py_buffer rows;
    if (PyObject_GetBuffer(table.p, &rows, PyBUF_C_CONTIGUOUS) < 0) {
      PyErr_Clear();
      return none();
    }
    const bool fits = rows.itemsize == 8 && rows.len == 8 * descs->numel() && rows.len % (8 * kDescFields) == 0;
    if (fits)
      for (int64_t b = 0; b < rows.len / (8 * kDescFields); ++b)
        sizes.add(static_cast<const int64_t*>(rows.buf) + b * kDescFields);
    PyBuffer_Release(&rows);
    if (!fits || !sizes.B) return none();
  }
  int64_t offsets[6];
  for (int k = 0; k < 6; ++k) {
    offsets[k] = PyLong_AsLongLong(PyTuple_GET_ITEM(args[3], k));
    if (PyErr_Occurred()) return nullptr;
  }
  SegEvaluator ev;
  if (!read_segmentation(args[0], index, sizes.D, ev)) return none();
  Ref instance = attr(args[0], names.instance);
  SegScratch w(sizes, ev.C);
  Tensor work = arena(instance.p, index, w.layout.size);
  const int64_t fields = address(*device), base = address(work);
  SegInputs in;
  in.descs = data<int64_t>(*descs);
  in.d_off = data<int64_t>(*d_off);
  in.g_off = data<int64_t>(*g_off);
  in.pair_off = data<int64_t>(*pair_off);
  in.total_chunks = *chunks;
  in.gc = at_address<int32_t>(fields + offsets[0]);
  in.crowd = at_address<uint8_t>(fields + offsets[1]);
  in.pc = at_address<int32_t>(fields + offsets[2]);
  in.det_classes = at_address<int32_t>(fields + offsets[3]);
  in.det_scores = at_address<double>(fields + offsets[4]);
  in.areas = offsets[5] < 0 ? nullptr : at_address<double>(fields + offsets[5]);
  const cudaStream_t stream = current_stream(index);
  int32_t* error = nullptr;
  int code;
  {
    ReleaseGil released;
    code = launch_seg(sizes, in, w, ev, base, error, stream);
  }
  return finish_seg(ev, sizes, code, error, stream);
  END_HANDLE_TH_ERRORS
}

// SegmentationEvaluator.compute: (status, result dict), or None. The panoptic summary runs on the side stream
// between an event of the current stream and one that the current stream waits for; its outputs come from
// the current stream's memory pool, which is not reused before that wait.
PyObject* combined_compute(PyObject*, PyObject* self) {
  HANDLE_TH_ERRORS
  if (!ordinary()) return none();
  const int index = c10::cuda::current_device();
  Ref instance = attr(self, names.instance), panoptic = attr(self, names.panoptic), side_object = attr(self, names._side);
  if (!instance || !panoptic || !side_object || side_object.is_none()) return none();
  Ref handle = attr(side_object.p, names.cuda_stream);
  if (!handle || !PyLong_Check(handle.p)) return none();
  PanopticState s;
  std::optional<Tensor> things;
  Accumulation a;
  if (!read_state(panoptic.p, index, s) || !read_things(panoptic.p, index, s.C, things) ||
      !plan_accumulation(instance.p, index, a))
    return none();
  const ComputeOut o = compute_outputs(index, s.C);
  const cudaStream_t stream = current_stream(index);
  const cudaStream_t side = reinterpret_cast<cudaStream_t>(PyLong_AsVoidPtr(handle.p));
  cudaEvent_t fork = nullptr, join = nullptr;
  int code = 0;
  bool ok = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming) == cudaSuccess &&
            cudaEventCreateWithFlags(&join, cudaEventDisableTiming) == cudaSuccess &&
            cudaEventRecord(fork, stream) == cudaSuccess && cudaStreamWaitEvent(side, fork, 0) == cudaSuccess;
  if (ok) {
    code = launch_compute(s, *things, o, side);
    if (!code) code = launch_accumulation(a, stream);
    // Joined whatever the launches answered: a capture must not keep an open branch.
    ok = cudaEventRecord(join, side) == cudaSuccess && cudaStreamWaitEvent(stream, join, 0) == cudaSuccess;
  }
  if (fork) cudaEventDestroy(fork);
  if (join) cudaEventDestroy(join);
  if (!ok) {
    PyErr_SetString(PyExc_RuntimeError, "the summaries' streams could not be joined");
    return nullptr;
  }
  if (code < 0) return Py_BuildValue("(iO)", code, Py_None);
  Ref result(compute_dict(o, s.C)), inner(accumulation_dict(a));
  if (!result || !inner || PyDict_SetItemString(result.p, "instance", inner.p) < 0) return nullptr;
  return Py_BuildValue("(iO)", code, result.p);
  END_HANDLE_TH_ERRORS
}

// ---- prefixes -----------------------------------------------------------------------------------------

struct PrefixPlan {
  Maps gt;
  Tensor crowd;
  std::vector<Tensor> masks;
  std::vector<int64_t> counts;
  Metadata classes;
  int64_t total_masks = 0, max_masks = 0, rows = 0, chunks = 0, cells = 0, T = 0;
  int64_t descs_at = 0, steps_at = 0, bytes = 0;  // byte offsets in the upload
  Tensor host;
};

// Checks and tables of segmentation_prefixes (prefix.run_prefixes): thresholds, descriptors, step table.
// `points`: the checkpoints of every image, or None for every prefix.
bool plan_prefixes(PyObject* prediction, PyObject* target, int64_t C, PyObject* thresholds, PyObject* points, int index,
                   PrefixPlan& p) {
  constexpr int64_t kChunk = 4096;
  std::optional<Tensor> crowd;
  bool missing = false;
  if (!read_maps(target, index, p.gt) || !read_crowd(target, p.gt, index, crowd, missing) || missing ||
      !read_masks(prediction, index, p.masks, p.counts) ||
      !read_field(prediction, names.classes, index, p.counts, at::kInt, at::kLong, false, p.classes) ||
      !PyTuple_CheckExact(thresholds) || (points != Py_None && !PyTuple_CheckExact(points)))
    return false;
  const int64_t B = p.gt.images(), S = p.gt.slots();
  if (B == 0 || (int64_t)p.masks.size() != B) return false;
  p.crowd = *crowd;
  p.T = PyTuple_GET_SIZE(thresholds);
  std::vector<int64_t> shared;
  if (points != Py_None)
    for (Py_ssize_t k = 0; k < PyTuple_GET_SIZE(points); ++k) {
      shared.push_back(PyLong_AsLongLong(PyTuple_GET_ITEM(points, k)));
      if (PyErr_Occurred()) {
        PyErr_Clear();
        return false;
      }
    }
  const int64_t pixels = p.gt.maps.size(1) * p.gt.maps.size(2), chunks = ceil_div(pixels, kChunk);
  int64_t steps = 0;
  for (int64_t b = 0; b < B; ++b) {
    if (p.masks[b].size(1) != p.gt.maps.size(1) || p.masks[b].size(2) != p.gt.maps.size(2)) return false;
    if (!shared.empty() && shared.back() > p.counts[b]) return false;
    p.total_masks += p.counts[b];
    p.max_masks = std::max(p.max_masks, p.counts[b]);
    steps += p.counts[b] + 1;
  }
  p.descs_at = 8 * p.T;
  p.steps_at = p.descs_at + 8 * B * kPrefixFields;
  p.bytes = p.steps_at + 4 * steps + 8;
  p.host = staging(p.bytes, index);
  char* bytes = data<char>(p.host);
  for (int64_t t = 0; t < p.T; ++t) {
    const double v = PyFloat_AsDouble(PyTuple_GET_ITEM(thresholds, t));
    if (PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
    std::memcpy(bytes + 8 * t, &v, 8);
  }
  int64_t* descs = reinterpret_cast<int64_t*>(bytes + p.descs_at);
  int32_t* step = reinterpret_cast<int32_t*>(bytes + p.steps_at);
  std::fill(step, step + steps + 2, -1);
  const int64_t target_ptr = address(p.gt.maps);
  const int64_t maps16 = target_ptr % 16 == 0 && pixels % 4 == 0 ? 1 : 0;
  int64_t masks = 0, raw = 0, at = 0;
  for (int64_t b = 0; b < B; ++b) {
    int64_t* d = descs + b * kPrefixFields;
    const int64_t n = p.counts[b], ptr = address(p.masks[b]);
    // Without requested checkpoints: every prefix 1..n, or the empty one.
    const int64_t q = points != Py_None ? (int64_t)shared.size() : std::max<int64_t>(n, 1);
    d[kPrefixTarget] = target_ptr + 4 * b * pixels;
    d[kPrefixMasks] = ptr;
    d[kPrefixPixels] = d[kPrefixStride] = pixels;
    d[kPrefixChunkBegin] = b * chunks;
    d[kPrefixN] = n;
    d[kPrefixG] = S;
    d[kPrefixDetBegin] = masks;
    d[kPrefixSlotBegin] = b * S;
    d[kPrefixQBegin] = p.rows;
    d[kPrefixQ] = q;
    d[kPrefixPairBegin] = p.cells;
    d[kPrefixRawBegin] = raw;
    d[kPrefixFlags] = maps16 | ((ptr | pixels) % 16 == 0 ? 2 : 0);
    d[kPrefixStepBegin] = at;
    d[kPrefixCountBegin] = b * p.T * C * 2;
    if (points != Py_None)
      for (size_t k = 0; k < shared.size(); ++k) step[at + shared[k]] = (int32_t)k;
    else if (n == 0)
      step[at] = 0;
    else
      for (int64_t k = 1; k <= n; ++k) step[at + k] = (int32_t)(k - 1);
    masks += n;
    raw += n * S;
    at += n + 1;
    p.rows += q;
    p.cells += q * S * (n + 1);
  }
  p.chunks = B * chunks;
  return true;
}

// The bytes plan_prefixes uploads for CPU tensors, the descriptors' and step table's byte offsets and the row count, or None.
PyObject* prefix_tables(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  PrefixPlan p;
  if (nargs != 5 || !ordinary() ||
      !plan_prefixes(args[0], args[1], PyLong_AsLongLong(args[2]), args[3], args[4], kHostOnly, p))
    return none();
  Ref bytes(PyBytes_FromStringAndSize(data<char>(p.host), p.bytes));
  if (!bytes) return nullptr;
  return Py_BuildValue("(OLLL)", bytes.p, (long long)p.descs_at, (long long)p.steps_at, (long long)p.rows);
  END_HANDLE_TH_ERRORS
}

// segmentation_prefixes (prediction, target, classes, thing flags, thresholds, checkpoints or None, validate):
// (status, packed outputs, thresholds tensor), or None. Outputs are packed as prefix._output_layout says.
PyObject* prefixes(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs != 7 || !ordinary()) return none();
  const int index = c10::cuda::current_device();
  const int64_t C = PyLong_AsLongLong(args[2]);
  auto things = plain(args[3], index);
  const int validate = PyObject_IsTrue(args[6]);
  PrefixPlan p;
  if (C <= 0 || validate < 0 || !things || !is(*things, at::kByte, {C}) ||
      !plan_prefixes(args[0], args[1], C, args[4], args[5], index, p)) {
    PyErr_Clear();
    return none();
  }
  const int64_t B = p.gt.images(), S = p.gt.slots(), T = p.T, R = p.rows;
  Tensor classes = p.total_masks == 0 ? at::empty({0}, on(index, at::kInt))
                   : B == 1           ? p.classes.held[0]
                                      : at::cat(p.classes.held);
  if (classes.scalar_type() != at::kInt) classes = classes.to(at::kInt);
  Tensor table = at::empty({p.bytes}, on(index, at::kByte));
  table.copy_(p.host.narrow(0, 0, p.bytes), /*non_blocking=*/true);
  // Output fields in order, 8-byte elements; the last element is the owner pass's chunk counter.
  const int64_t sizes[14] = {R * C, R * C, R * C, R * C, R * C * (C + 1), R * T * C, R * T * C, R * T * C,
                             R * T * C, R * T * C, R * 4 * C, R * 9, R * 3, R};
  int64_t* out[15];
  int64_t total = 0;
  for (int64_t n : sizes) total += n;
  Tensor flat = at::empty({total + 1}, on(index, at::kLong));
  out[0] = data<int64_t>(flat);
  for (int k = 0; k < 14; ++k) out[k + 1] = out[k] + sizes[k];
  auto f64 = [&](int k) { return reinterpret_cast<double*>(out[k]); };
  // int32 workspaces back to back: ga, raw, pairs, counters (reserved), error (zeroed by the call).
  const int64_t raw_len = S * p.total_masks, counters_len = B * T * C * 2;
  Tensor work = at::empty({B * S + raw_len + p.cells + counters_len + 1}, on(index, at::kInt));
  uint32_t* ga = data<uint32_t>(work);
  uint32_t* raw = ga + B * S;
  int32_t* pairs = reinterpret_cast<int32_t*>(raw + raw_len);
  int32_t* counters = pairs + p.cells;
  const char* base = data<char>(table);
  const cudaStream_t stream = current_stream(index);
  int code;
  {
    ReleaseGil released;
    code = api.pe_prefix(reinterpret_cast<const int64_t*>(base + p.descs_at), B, p.chunks, R, S, p.max_masks + 1,
                         S * (p.max_masks + 1), reinterpret_cast<const int32_t*>(base + p.steps_at),
                         data<int32_t>(classes), data<int32_t>(p.gt.classes), data<uint8_t>(p.crowd),
                         data<uint8_t>(*things), reinterpret_cast<const double*>(base), T, C, ga, B * S, raw, raw_len,
                         pairs, p.cells, counters, counters_len, out[0], out[1], out[2], f64(3), out[4], out[5],
                         out[6], out[7], f64(8), f64(9), f64(10), f64(11), out[12], f64(13), validate, 1,
                         reinterpret_cast<uint64_t*>(out[14]), counters + counters_len, stream);
  }
  Ref packed(THPVariable_Wrap(flat)), levels(view(table, 0, at::kDouble, {T}));
  if (!packed || !levels) return nullptr;
  return Py_BuildValue("(iOO)", code, packed.p, levels.p);
  END_HANDLE_TH_ERRORS
}

// prefix._part of PackedOutputs (outputs, row, field, further indices ...): a view like those of the other results.
PyObject* part(PyObject*, PyObject* const* args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  if (nargs < 3) {
    PyErr_SetString(PyExc_TypeError, "part(outputs, row, field, *index)");
    return nullptr;
  }
  Ref flat = attr(args[0], names.flat), layout = attr(args[0], names._layout);
  PyObject* entry = layout && PyDict_CheckExact(layout.p) ? PyDict_GetItemWithError(layout.p, args[2]) : nullptr;
  PyObject* shape = entry && PyTuple_CheckExact(entry) && PyTuple_GET_SIZE(entry) == 3 ? PyTuple_GET_ITEM(entry, 1) : nullptr;
  const Py_ssize_t leading = nargs - 2, dims = shape && PyTuple_CheckExact(shape) ? PyTuple_GET_SIZE(shape) : 0;
  constexpr Py_ssize_t kMost = 4;
  if (flat && THPVariable_CheckExact(flat.p) && leading <= dims && dims <= kMost && ordinary() &&
      THPDtype_Check(PyTuple_GET_ITEM(entry, 2))) {
    const Tensor& base = THPVariable_Unpack(flat.p);
    int64_t offset = PyLong_AsLongLong(PyTuple_GET_ITEM(entry, 0)), numel = 1, count = 1, sizes[kMost];
    bool inside = offset >= 0;
    for (Py_ssize_t k = dims - 1; k >= 0; --k) {
      sizes[k] = PyLong_AsLongLong(PyTuple_GET_ITEM(shape, k));
      if (k < leading) {
        const int64_t i = PyLong_AsLongLong(k ? args[k + 2] : args[1]);
        inside = inside && i >= 0 && i < sizes[k];
        offset += i * numel;
      } else {
        count *= sizes[k];
      }
      numel *= sizes[k];
    }
    const at::ScalarType type = reinterpret_cast<THPDtype*>(PyTuple_GET_ITEM(entry, 2))->scalar_type;
    if (!PyErr_Occurred() && inside && count >= 0 && plain(flat.p, base.is_cuda() ? base.get_device() : kHostOnly) &&
        base.scalar_type() == at::kLong && base.storage_offset() == 0 && offset + count <= base.numel() &&
        (type == at::kLong || type == at::kDouble))
      return view(base, 8 * offset, type, at::IntArrayRef(sizes + leading, dims - leading));
  }
  PyErr_Clear();
  // Anything else: outputs[field][row, index ...].
  Ref field(PyObject_GetItem(args[0], args[2])), index(PyTuple_New(leading));
  if (!field || !index) return nullptr;
  for (Py_ssize_t k = 0; k < leading; ++k) {
    PyObject* i = k ? args[k + 2] : args[1];
    Py_INCREF(i);
    PyTuple_SET_ITEM(index.p, k, i);
  }
  return PyObject_GetItem(field.p, index.p);
  END_HANDLE_TH_ERRORS
}

// ---- module -------------------------------------------------------------------------------------------

// bind({name: address}): entry points of the loaded library.
PyObject* bind(PyObject*, PyObject* table) {
  Api bound;
#define X(name)                                                                    \
  {                                                                                \
    PyObject* address = PyDict_GetItemString(table, #name);                       \
    if (!address) {                                                                \
      PyErr_SetString(PyExc_KeyError, #name);                                      \
      return nullptr;                                                              \
    }                                                                              \
    bound.name = reinterpret_cast<decltype(bound.name)>(PyLong_AsVoidPtr(address)); \
    if (PyErr_Occurred()) return nullptr;                                          \
  }
  PE_HOST_API(X)
#undef X
  api = bound;
  Py_RETURN_NONE;
}

#define FAST(name, function) \
  {name, reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(function)), METH_FASTCALL, nullptr}

PyMethodDef methods[] = {
    {"bind", bind, METH_O, nullptr},
    {"zero", zero, METH_O, nullptr},
    {"panoptic_compute", panoptic_compute, METH_O, nullptr},
    {"instance_compute", instance_compute, METH_O, nullptr},
    {"combined_compute", combined_compute, METH_O, nullptr},
    FAST("panoptic_update", panoptic_update),
    FAST("reward", reward),
    FAST("coco_slots", coco_slots),
    FAST("instance_update", instance_update),
    FAST("instance_tables", instance_tables),
    FAST("combined_update", combined_update),
    FAST("combined_tables", combined_tables),
    FAST("images_update", images_update),
    FAST("prefixes", prefixes),
    FAST("prefix_tables", prefix_tables),
    FAST("part", part),
    {nullptr, nullptr, 0, nullptr},
};

PyModuleDef module = {PyModuleDef_HEAD_INIT, "_host", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host(void) {
#define X(name)                                              \
  names.name = PyUnicode_InternFromString(#name);            \
  if (!names.name) return nullptr;
  PE_HOST_NAMES(X)
#undef X
  return PyModule_Create(&module);
}
