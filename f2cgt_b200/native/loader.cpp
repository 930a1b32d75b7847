// One step of the sampling loader (f2cgt_b200/sage.py, GPUSamplingDataloader): wait for the minibatch built during the previous
// step, queue the next one on the loader's own stream, hand the finished one out as views of its buffers.  The same in Python
// is about thirty tensor and event operations, 80 us of a training step.
#include "native.h"

#include <c10/core/TensorImpl.h>

namespace f2c_native {
namespace {

struct Set {
  f2c_minibatch args{};
  at::Tensor indptr, indices, ws, node_map, header, unique, seeds;
  std::vector<at::Tensor> sub_indptr, ids, local;
  cudaEvent_t built = nullptr, consumed = nullptr;
  bool lent = false;  // handed out before: its last user must be through before it is overwritten
  ~Set() {
    // A minibatch may still be under construction on the loader's stream, in memory that other streams (and, for the header, the
    // host) would get next.
    if (built != nullptr) (void)cudaEventSynchronize(built);
    if (built != nullptr) (void)cudaEventDestroy(built);
    if (consumed != nullptr) (void)cudaEventDestroy(consumed);
  }
};

constexpr const char* kCapsule = "f2cgt_b200.minibatch_set";

Set& set_of(PyObject* o) {
  Set* s = (Set*)PyCapsule_GetPointer(o, kCapsule);
  if (s == nullptr) throw PythonError{};
  return *s;
}

// first n elements of a contiguous tensor from `offset` on, as a tensor of its own
at::Tensor view(const at::Tensor& base, int64_t offset, int64_t n) {
  auto impl = c10::make_intrusive<c10::TensorImpl>(c10::Storage(base.storage()), base.key_set(), base.dtype());
  impl->set_storage_offset(base.storage_offset() + offset);
  impl->set_sizes_contiguous({n});
  return at::Tensor(std::move(impl));
}

// indptr, indices, workspace (zeroed), node words, header (pinned), unique, sub_indptr list, ids list, local list, picks list
PyObject* minibatch_new(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("minibatch_new", n, 10);
    auto s = std::make_unique<Set>();
    s->indptr = tensor(a[0], "indptr", kIndex);
    const unsigned same = bit(dtype_tag(s->indptr.scalar_type()));
    s->indices = tensor(a[1], "indices", same);
    s->ws = tensor(a[2], "workspace", bit(F2C_U8));
    s->node_map = tensor(a[3], "node_map", bit(F2C_I64));
    if (!THPVariable_Check(a[4])) fail(PyExc_TypeError, "header must be a torch.Tensor");
    s->header = THPVariable_Unpack(a[4]);
    s->unique = tensor(a[5], "unique", same);
    const Py_ssize_t hops = PyList_Check(a[9]) ? PyList_GET_SIZE(a[9]) : 0;
    if (hops < 1 || hops > F2C_MAX_HOPS || !s->header.is_pinned() || s->header.scalar_type() != at::kLong || s->header.numel() != 2 * hops + 1)
      fail(PyExc_RuntimeError, "minibatch_new: bad arguments");
    f2c_minibatch& m = s->args;
    m.indptr = s->indptr.data_ptr(); m.indices = s->indices.data_ptr(); m.n_nodes = s->indptr.numel() - 1;
    m.index_dtype = dtype_tag(s->indptr.scalar_type()); m.n_hops = (int)hops;
    m.unique = s->unique.data_ptr(); m.node_map = s->node_map.data_ptr(); m.header = (int64_t*)s->header.data_ptr();
    m.workspace = s->ws.data_ptr(); m.workspace_bytes = s->ws.numel();
    for (Py_ssize_t h = 0; h < hops; ++h) {
      for (int k = 6; k < 9; ++k)
        if (!PyList_Check(a[k]) || PyList_GET_SIZE(a[k]) != hops) fail(PyExc_TypeError, "minibatch_new: one tensor per hop");
      s->sub_indptr.push_back(tensor(PyList_GET_ITEM(a[6], h), "sub_indptr", same));
      s->ids.push_back(tensor(PyList_GET_ITEM(a[7], h), "ids", same));
      s->local.push_back(tensor(PyList_GET_ITEM(a[8], h), "local", same));
      m.sub_indptr[h] = s->sub_indptr[h].data_ptr(); m.ids[h] = s->ids[h].data_ptr(); m.local[h] = s->local[h].data_ptr();
      m.num_pick[h] = (int)integer(PyList_GET_ITEM(a[9], h));
    }
    c10::cuda::CUDAGuard guard(s->indptr.device());
    C10_CUDA_CHECK(cudaEventCreateWithFlags(&s->built, cudaEventDisableTiming));
    C10_CUDA_CHECK(cudaEventCreateWithFlags(&s->consumed, cudaEventDisableTiming));
    PyObject* cap = PyCapsule_New(s.get(), kCapsule, [](PyObject* o) { delete (Set*)PyCapsule_GetPointer(o, kCapsule); });
    if (cap == nullptr) throw PythonError{};
    s.release();
    return cap;
  });
}

void launch(Set& s, const at::Tensor& order, int64_t first, int64_t count, int64_t epoch, uint64_t rng_seed, uint64_t rng_offset, cudaStream_t st) {
  s.seeds = view(order, first, count);
  s.args.seeds = s.seeds.data_ptr(); s.args.n_seeds = count; s.args.epoch = (uint32_t)epoch;
  s.args.rng_seed = rng_seed; s.args.rng_offset = rng_offset;
  check_status(unlocked([&] {
    const int rc = f2c_sample_minibatch(&s.args, st);
    if (rc == F2C_OK) C10_CUDA_CHECK(cudaEventRecord(s.built, st));
    return rc;
  }));
}

uint64_t bits64(PyObject* o) {
  const unsigned long long v = PyLong_AsUnsignedLongLongMask(o);
  if (v == (unsigned long long)-1 && PyErr_Occurred()) throw PythonError{};
  return v;
}

cudaStream_t handle(PyObject* o) { return (cudaStream_t)(uintptr_t)bits64(o); }

const at::Tensor& order_of(const Set& s, PyObject* o, int64_t first, int64_t count) {
  const at::Tensor& order = tensor(o, "seeds", bit(s.args.index_dtype));
  if (order.dim() != 1 || first < 0 || count < 1 || first + count > order.numel()) fail(PyExc_RuntimeError, "sample_minibatch: bad seed range");
  return order;
}

// set, seeds, first, count, epoch, rng_seed, rng_offset, stream handle
PyObject* minibatch_launch(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("minibatch_launch", n, 8);
    Set& s = set_of(a[0]);
    const int64_t first = integer(a[2]), count = integer(a[3]);
    const at::Tensor& order = order_of(s, a[1], first, count);
    c10::cuda::CUDAGuard guard(s.indptr.device());
    launch(s, order, first, count, integer(a[4]), bits64(a[5]), bits64(a[6]), handle(a[7]));
    Py_RETURN_NONE;
  });
}

void put(PyObject* dict, PyObject* key, PyObject* value) {  // steals value
  if (value == nullptr || PyDict_SetItem(dict, key, value) != 0) { Py_XDECREF(value); throw PythonError{}; }
  Py_DECREF(value);
}

// (input_nodes, output_nodes, blocks), blocks outermost hop first
PyObject* hand_out(Set& s) {
  static PyObject* keys[6] = {PyUnicode_InternFromString("dst_nodes"), PyUnicode_InternFromString("src_nodes"), PyUnicode_InternFromString("indptr"),
                              PyUnicode_InternFromString("indices_global"), PyUnicode_InternFromString("indices_local"),
                              PyUnicode_InternFromString("n_edges")};
  const int64_t* h = (const int64_t*)s.header.data_ptr();
  const int hops = s.args.n_hops;
  if (h[2 * hops] != 0)
    fail(PyExc_RuntimeError, h[2 * hops] == 2 ? "sample_minibatch: negative id in the graph or the seeds"
                                              : "sample_minibatch: id beyond the graph's nodes in the graph or the seeds");
  struct Owned { PyObject* o; ~Owned() { Py_XDECREF(o); } PyObject* release() { return std::exchange(o, nullptr); } };
  Owned blocks{PyList_New(hops)};
  if (blocks.o == nullptr) throw PythonError{};
  PyObject* frontier = THPVariable_Wrap(s.seeds);
  Owned first{Py_XNewRef(frontier)}, keep{frontier};
  int64_t rows = s.args.n_seeds;
  for (int i = 0; i < hops; ++i) {
    Owned d{PyDict_New()};
    if (d.o == nullptr || keep.o == nullptr) throw PythonError{};
    Owned src{THPVariable_Wrap(view(s.unique, 0, h[2 * i + 1]))};
    put(d.o, keys[0], Py_NewRef(keep.o));
    put(d.o, keys[1], Py_XNewRef(src.o));
    put(d.o, keys[2], THPVariable_Wrap(view(s.sub_indptr[i], 0, rows + 1)));
    put(d.o, keys[3], THPVariable_Wrap(view(s.ids[i], 0, h[2 * i])));
    put(d.o, keys[4], THPVariable_Wrap(view(s.local[i], 0, h[2 * i])));
    put(d.o, keys[5], PyLong_FromLongLong(h[2 * i]));
    PyList_SET_ITEM(blocks.o, hops - 1 - i, d.release());
    rows = h[2 * i + 1];
    std::swap(keep.o, src.o);
  }
  return PyTuple_Pack(3, keep.o, first.o, blocks.o);
}

// Wait on the host for what was launched in `set` and hand it out.
PyObject* minibatch_take(PyObject*, PyObject* o) {
  return guarded([&]() -> PyObject* {
    Set& s = set_of(o);
    C10_CUDA_CHECK(unlocked([&] { return cudaEventSynchronize(s.built); }));
    return hand_out(s);
  });
}

// built set, set to build next (None at the end), seeds, first, count, epoch, rng_seed, rng_offset, stream handle
PyObject* minibatch_next(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("minibatch_next", n, 9);
    Set& s = set_of(a[0]);
    c10::cuda::CUDAGuard guard(s.indptr.device());
    C10_CUDA_CHECK(unlocked([&] { return cudaEventSynchronize(s.built); }));
    if (a[1] != Py_None) {
      Set& next = set_of(a[1]);
      const int64_t first = integer(a[3]), count = integer(a[4]);
      const at::Tensor& order = order_of(next, a[2], first, count);
      if (next.lent) {
        // Everything queued on the current stream so far belongs to earlier minibatches: once it has run, the minibatch that
        // was handed out of this set may be overwritten.
        const cudaStream_t side = handle(a[8]);
        unlocked([&] {
          C10_CUDA_CHECK(cudaEventRecord(next.consumed, stream_of(s.indptr)));
          C10_CUDA_CHECK(cudaStreamWaitEvent(side, next.consumed, 0));
        });
      }
      launch(next, order, first, count, integer(a[5]), bits64(a[6]), bits64(a[7]), handle(a[8]));
    }
    s.lent = true;
    return hand_out(s);
  });
}

}  // namespace

PyMethodDef g_loader_methods[] = {{"minibatch_new", (PyCFunction)(void*)minibatch_new, METH_FASTCALL, nullptr},
                                  {"minibatch_launch", (PyCFunction)(void*)minibatch_launch, METH_FASTCALL, nullptr},
                                  {"minibatch_take", minibatch_take, METH_O, nullptr},
                                  {"minibatch_next", (PyCFunction)(void*)minibatch_next, METH_FASTCALL, nullptr},
                                  {nullptr, nullptr, 0, nullptr}};

}  // namespace f2c_native
