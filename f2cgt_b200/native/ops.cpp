// The per-call part of f2cgt_b200/ops.py for the decoders and the aggregations: argument checks, output allocation, stream
// lookup and the library call.  In Python these cost 10-14 us per call, several times the launch itself; here 3-4 us.
#include "native.h"

namespace f2c_native {

PyObject* g_error_class = nullptr;

void arguments(const char* name, Py_ssize_t got, Py_ssize_t want) {
  if (got != want) fail(PyExc_TypeError, "%s: expected %zd arguments, got %zd", name, want, got);
}

namespace {

struct Csc { const at::Tensor &indptr, &indices; int64_t n_dst; int tag; };

Csc csc(PyObject* ip, PyObject* ix) {
  const at::Tensor& indptr = tensor(ip, "indptr", kIndex);
  const at::Tensor& indices = tensor(ix, "indices", kIndex);
  if (indptr.scalar_type() != indices.scalar_type()) fail(PyExc_RuntimeError, "indptr and indices must have the same dtype");
  if (indptr.dim() != 1 || indptr.numel() < 1) fail(PyExc_RuntimeError, "indptr must be 1-D with at least one element");
  return Csc{indptr, indices, indptr.numel() - 1, dtype_tag(indptr.scalar_type())};
}

// Rows asked for by out_rows (None: the block's own), and the width checked: what block_out() needs of Python.
int64_t asked_rows(int64_t n_dst, int64_t width, PyObject* out_rows) {
  if (width < 0) fail(PyExc_RuntimeError, "negative width");
  return out_rows == Py_None ? n_dst : integer(out_rows);
}

// [max(n_dst, |asked|), width]; rows behind n_dst are zero, or - asked negative - left as they are
at::Tensor block_out(int64_t n_dst, int64_t asked, int64_t width, at::ScalarType dtype, const at::Device& device, cudaStream_t st) {
  const int64_t rows = std::max(n_dst, std::abs(asked));
  at::Tensor out = empty({rows, width}, dtype, device);
  if (rows > n_dst && asked > 0) {
    const size_t row = (size_t)width * out.element_size();
    C10_CUDA_CHECK(cudaMemsetAsync((char*)out.data_ptr() + (size_t)n_dst * row, 0, (size_t)(rows - n_dst) * row, st));
  }
  return out;
}

// dropout: None or a mapping with p, seed, offset, training, scale; kernel: an f2c_kernel value
struct Options {
  f2c_epilogue e{};
  bool set = false;
  const f2c_epilogue* get() const { return set ? &e : nullptr; }
};

Options options(PyObject* dropout, PyObject* kernel) {
  Options o;
  o.e.kernel = (int)integer(kernel);
  o.set = o.e.kernel != 0;
  if (dropout == Py_None) return o;
  o.set = true;
  PyObject* d = PyDict_Check(dropout) ? Py_NewRef(dropout) : PyObject_CallOneArg((PyObject*)&PyDict_Type, dropout);
  if (d == nullptr) throw PythonError{};
  struct Drop { PyObject* o; ~Drop() { Py_DECREF(o); } } keep{d};
  auto item = [&](const char* k) -> PyObject* { return PyDict_GetItemString(d, k); };
  PyObject* p = item("p");
  if (p == nullptr) fail(PyExc_KeyError, "p");
  o.e.p = (float)real(p);
  auto whole = [&](const char* k, int64_t otherwise) -> int64_t {
    PyObject* v = item(k);
    if (v == nullptr) return otherwise;
    if (PyLong_Check(v)) {
      const unsigned long long u = PyLong_AsUnsignedLongLongMask(v);
      if (u == (unsigned long long)-1 && PyErr_Occurred()) throw PythonError{};
      return (int64_t)u;
    }
    return integer(v);
  };
  o.e.training = item("training") ? (PyObject_IsTrue(item("training")) ? 1 : 0) : 1;
  o.e.scale = item("scale") ? (PyObject_IsTrue(item("scale")) ? 1 : 0) : 0;
  o.e.seed = (uint64_t)whole("seed", 0);
  o.e.offset = (uint64_t)whole("offset", 0);
  return o;
}

PyObject* sq_decompress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("sq_decompress", n, 5);
    const at::Tensor& codes = tensor(a[0], "compress_data", kCodes);
    const at::Tensor& cb = tensor(a[1], "codebooks", kF32);
    if (codes.dim() != 2) fail(PyExc_RuntimeError, "compress_data must be 2-D");
    const int64_t bits = integer(a[2]), cs = integer(a[3]), dim = integer(a[4]);
    const int64_t rows = asked_rows(codes.size(0), dim, Py_None);
    at::Tensor out;
    check_status(unlocked([&] {
      c10::cuda::CUDAGuard guard(codes.device());
      cudaStream_t st = stream_of(codes);
      out = block_out(rows, rows, dim, at::kFloat, codes.device(), st);
      return f2c_sq_decompress(codes.data_ptr(), dtype_tag(codes.scalar_type()), cb.const_data_ptr<float>(), cb.size(0),
                               out.mutable_data_ptr<float>(), codes.size(0), codes.size(1), dim, (int)bits, cs, st);
    }));
    return THPVariable_Wrap(std::move(out));
  });
}

PyObject* vq_decompress(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("vq_decompress", n, 3);
    const at::Tensor& codes = tensor(a[0], "index_tensor", kCodes);
    const at::Tensor& cb = tensor(a[1], "codebooks", kF32 | bit(F2C_F16));
    if (codes.dim() != 2 || cb.dim() != 3 || codes.size(1) != cb.size(0))
      fail(PyExc_RuntimeError, "index_tensor must be [rows, n_codebooks] and codebooks [n_codebooks, length, column_slice]");
    const int64_t dim = integer(a[2]);
    const int64_t rows = asked_rows(codes.size(0), dim, Py_None);
    at::Tensor out;
    check_status(unlocked([&] {
      c10::cuda::CUDAGuard guard(codes.device());
      cudaStream_t st = stream_of(codes);
      out = block_out(rows, rows, dim, at::kFloat, codes.device(), st);
      return f2c_vq_decompress(codes.data_ptr(), dtype_tag(codes.scalar_type()), cb.data_ptr(), dtype_tag(cb.scalar_type()),
                               out.mutable_data_ptr<float>(), codes.size(0), cb.size(0), cb.size(1), cb.size(2), dim, st);
    }));
    return THPVariable_Wrap(std::move(out));
  });
}

PyObject* spmm(PyObject*, PyObject* const* a, Py_ssize_t n) {  // feat, indptr, indices, reduce, out_rows
  return guarded([&]() -> PyObject* {
    arguments("spmm", n, 5);
    const at::Tensor& feat = tensor(a[0], "feat", kF32 | bit(F2C_F16) | bit(F2C_F64));
    const Csc c = csc(a[1], a[2]);
    if (feat.dim() != 2) fail(PyExc_RuntimeError, "feat must be 2-D");
    const int64_t rows = asked_rows(c.n_dst, feat.size(1), a[4]);
    const int reduce = (int)integer(a[3]);
    at::Tensor out;
    check_status(unlocked([&] {
      c10::cuda::CUDAGuard guard(feat.device());
      cudaStream_t st = stream_of(feat);
      out = block_out(c.n_dst, rows, feat.size(1), feat.scalar_type(), feat.device(), st);
      return f2c_spmm_csr(feat.data_ptr(), dtype_tag(feat.scalar_type()), c.indptr.data_ptr(), c.indices.data_ptr(), c.tag, out.data_ptr(),
                          c.n_dst, feat.size(1), reduce, st);
    }));
    return THPVariable_Wrap(std::move(out));
  });
}

// codes, codebooks, indptr, indices, bits, column_slice, feat_dim, reduce, dropout, kernel, out_rows
PyObject* sq_spmm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("sq_spmm", n, 11);
    const at::Tensor& codes = tensor(a[0], "compress_feat", kCodes);
    const at::Tensor& cb = tensor(a[1], "codebooks", kF32);
    const Csc c = csc(a[2], a[3]);
    if (codes.dim() != 2) fail(PyExc_RuntimeError, "compress_feat must be 2-D");
    const int64_t bits = integer(a[4]), cs = integer(a[5]), dim = integer(a[6]);
    const Options o = options(a[8], a[9]);
    const int64_t rows = asked_rows(c.n_dst, dim, a[10]);
    const int reduce = (int)integer(a[7]);
    at::Tensor out;
    check_status(unlocked([&] {
      c10::cuda::CUDAGuard guard(codes.device());
      cudaStream_t st = stream_of(codes);
      out = block_out(c.n_dst, rows, dim, at::kFloat, codes.device(), st);
      return f2c_sq_spmm_csr(codes.data_ptr(), dtype_tag(codes.scalar_type()), cb.const_data_ptr<float>(), cb.size(0), c.indptr.data_ptr(),
                             c.indices.data_ptr(), c.tag, out.mutable_data_ptr<float>(), c.n_dst, codes.size(0), codes.size(1), dim,
                             (int)bits, cs, reduce, o.get(), st);
    }));
    return THPVariable_Wrap(std::move(out));
  });
}

// codes, codebooks, indptr, indices, feat_dim, reduce, dropout, kernel, out_rows
PyObject* vq_spmm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("vq_spmm", n, 9);
    const at::Tensor& codes = tensor(a[0], "compress_feat", kCodes);
    const at::Tensor& cb = tensor(a[1], "codebooks", kF32);
    const Csc c = csc(a[2], a[3]);
    if (codes.dim() != 2 || cb.dim() != 3 || codes.size(1) != cb.size(0))
      fail(PyExc_RuntimeError, "compress_feat must be [rows, n_codebooks] and codebooks [n_codebooks, length, column_slice]");
    const int64_t dim = integer(a[4]);
    const Options o = options(a[6], a[7]);
    const int64_t rows = asked_rows(c.n_dst, dim, a[8]);
    const int reduce = (int)integer(a[5]);
    at::Tensor out;
    check_status(unlocked([&] {
      c10::cuda::CUDAGuard guard(codes.device());
      cudaStream_t st = stream_of(codes);
      out = block_out(c.n_dst, rows, dim, at::kFloat, codes.device(), st);
      return f2c_vq_spmm_csr(codes.data_ptr(), dtype_tag(codes.scalar_type()), cb.const_data_ptr<float>(), c.indptr.data_ptr(),
                             c.indices.data_ptr(), c.tag, out.mutable_data_ptr<float>(), c.n_dst, cb.size(0), cb.size(1), cb.size(2), dim,
                             reduce, o.get(), st);
    }));
    return THPVariable_Wrap(std::move(out));
  });
}

// sq codes, sq codebooks, bits, column_slice, vq codes, vq codebooks, slot, indptr, indices, feat_dim, reduce, dropout, kernel, out_rows
PyObject* two_level_spmm(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("two_level_spmm", n, 14);
    const at::Tensor& sq = tensor(a[0], "sq_data", kCodes);
    const at::Tensor& sq_cb = tensor(a[1], "sq_codebooks", kF32);
    const at::Tensor& vq = tensor(a[4], "vq_data", kCodes);
    const at::Tensor& vq_cb = tensor(a[5], "vq_codebooks", kF32);
    const int32_t* slot = a[6] == Py_None ? nullptr : tensor(a[6], "slot", bit(F2C_I32)).const_data_ptr<int32_t>();
    const Csc c = csc(a[7], a[8]);
    if (vq_cb.dim() != 3 || sq.dim() != 2 || vq.dim() != 2) fail(PyExc_RuntimeError, "sq_data and vq_data must be 2-D and vq_codebooks 3-D");
    const int64_t dim = integer(a[9]);
    const Options o = options(a[11], a[12]);
    const int64_t rows = asked_rows(c.n_dst, dim, a[13]);
    const int64_t bits = integer(a[2]), cs = integer(a[3]);
    const int reduce = (int)integer(a[10]);
    at::Tensor out;
    check_status(unlocked([&] {
      c10::cuda::CUDAGuard guard(vq.device());
      cudaStream_t st = stream_of(vq);
      out = block_out(c.n_dst, rows, dim, at::kFloat, vq.device(), st);
      return f2c_hybrid_spmm_csr(sq.data_ptr(), dtype_tag(sq.scalar_type()), sq_cb.const_data_ptr<float>(), sq_cb.size(0), (int)bits, cs, sq.size(1),
                                 vq.data_ptr(), dtype_tag(vq.scalar_type()), vq_cb.const_data_ptr<float>(), vq_cb.size(0), vq_cb.size(1),
                                 vq_cb.size(2), slot, sq.size(0), c.indptr.data_ptr(), c.indices.data_ptr(), c.tag, out.mutable_data_ptr<float>(),
                                 c.n_dst, dim, reduce, o.get(), st);
    }));
    return THPVariable_Wrap(std::move(out));
  });
}

PyObject* kmeans_assign(PyObject*, PyObject* const* a, Py_ssize_t n) {  // x, centers, metric and scorer flags -> labels, [undecided, error]
  return guarded([&]() -> PyObject* {
    arguments("kmeans_assign", n, 3);
    const at::Tensor& x = tensor(a[0], "data", kF32);
    const at::Tensor& centers = tensor(a[1], "centers", kF32);
    if (x.dim() != 2 || centers.dim() != 2 || x.size(1) != centers.size(1)) fail(PyExc_RuntimeError, "data must be [n, d] and centers [k, d]");
    const int metric = (int)integer(a[2]);
    const int64_t rows = x.size(0), k = centers.size(0), d = x.size(1);
    at::Tensor labels, head;  // the workspace starts with what the second result is
    check_status(unlocked([&] {
      c10::cuda::CUDAGuard guard(x.device());
      const cudaStream_t st = stream_of(x);
      labels = empty({rows}, at::kLong, x.device());
      const int64_t bytes = f2c_kmeans_assign_workspace(rows, k, d);
      head = empty({std::max(bytes, (int64_t)8) / 4}, at::kInt, x.device());
      if (bytes == 0) C10_CUDA_CHECK(cudaMemsetAsync(head.data_ptr(), 0, 8, st));
      return f2c_kmeans_assign(x.const_data_ptr<float>(), centers.const_data_ptr<float>(), labels.mutable_data_ptr<int64_t>(), rows, k, d, metric,
                               bytes > 0 ? head.data_ptr() : nullptr, st);
    }));
    PyObject* l = THPVariable_Wrap(std::move(labels));
    PyObject* h = THPVariable_Wrap(std::move(head));
    PyObject* r = PyTuple_Pack(2, l, h);
    Py_DECREF(l); Py_DECREF(h);
    return r;
  });
}

PyObject* set_error_class(PyObject*, PyObject* cls) {
  Py_XSETREF(g_error_class, Py_NewRef(cls));
  Py_RETURN_NONE;
}

PyMethodDef g_methods[] = {
    {"sq_decompress", (PyCFunction)(void*)sq_decompress, METH_FASTCALL, nullptr},
    {"vq_decompress", (PyCFunction)(void*)vq_decompress, METH_FASTCALL, nullptr},
    {"spmm", (PyCFunction)(void*)spmm, METH_FASTCALL, nullptr},
    {"sq_spmm", (PyCFunction)(void*)sq_spmm, METH_FASTCALL, nullptr},
    {"vq_spmm", (PyCFunction)(void*)vq_spmm, METH_FASTCALL, nullptr},
    {"two_level_spmm", (PyCFunction)(void*)two_level_spmm, METH_FASTCALL, nullptr},
    {"kmeans_assign", (PyCFunction)(void*)kmeans_assign, METH_FASTCALL, nullptr},
    {"set_error_class", set_error_class, METH_O, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef g_module = {PyModuleDef_HEAD_INIT, "_native", nullptr, -1, g_methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace
}  // namespace f2c_native

PyMODINIT_FUNC PyInit__native(void) {
  PyObject* m = PyModule_Create(&f2c_native::g_module);
  for (PyMethodDef* more : {f2c_native::g_sage_methods, f2c_native::g_loader_methods})
    if (m != nullptr && PyModule_AddFunctions(m, more) != 0) Py_CLEAR(m);
  return m;
}
