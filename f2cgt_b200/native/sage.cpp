// A GraphSAGE network over a minibatch's blocks as ONE autograd node: what f2cgt_b200/sage.py's layers do (products, bias, ReLU,
// dropout, mean aggregation over the hidden layers), forward and backward, without an interpreter or an autograd node in
// between.  A training step was bound by the host: about seventy launches, each behind 10-20 us of Python and dispatcher.
//
// The forward products are the library's kernel where products may use tf32 (csrc/sage_gemm.cu: both products of a layer, bias
// and ReLU in one launch, the same sums as the two library products it replaces, see use_own()).  All other products are
// torch's, on row counts padded by sage._bucket as in the Python layers: their sums over 10^3 .. 10^5 rows depend on how they
// are split, and a weight gradient that differs by 10^-5 is enough for Adam's first steps to go the other way on a weight whose
// gradient is nearly zero.  What changes there is the time around them: the mask of ReLU and dropout, with the bias gradient, is
// one pass (csrc/sage_mask.cu), and the weight gradients, which cuBLAS gives to a few CTAs each, run on a second stream
// beside the input gradients and each other.  Dropout is torch's own, over the padded rows, so that masks are the ones
// torch.nn.Dropout would draw.
#include "native.h"

#include <array>
#include <atomic>

#include <ATen/cuda/CUDAEvent.h>
#include <cublas_v2.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>

namespace f2c_native {
namespace {

using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

struct Layer {
  int64_t rows = 0, padded = 0;       // destination rows of the block, and the row count dropout sees
  at::Tensor indptr, indices;         // hidden layers: the block over the previous layer's rows
};

struct Net {
  std::vector<Layer> layers;
  double p = 0.0;                     // dropout between the layers (0 outside training)
  bool tf32 = false;                  // forward products may be the library's
  c10::optional<at::ScalarType> cast; // operand type of torch's products (backward pass: the type in force then)
  double scale() const { return p < 1.0 ? 1.0 / (1.0 - p) : 0.0; }
};

// Operand type of torch's products in force (sage.products_in): a scalar type, or -1.
std::atomic<int> g_product_type{-1};

struct Status {  // library status inside a node (no Python exception there)
  void operator=(int rc) const { TORCH_CHECK(rc == F2C_OK, "f2cgt_b200: ", f2c_last_error()); }
};
constexpr Status checked{};

// Kernels run behind the host, so a bounded wait that ran out in one of them shows at a later call: here, without a wait of its own.
void check_reported() {
  int32_t code = 0;
  if (f2c_device_status_seen(&code) == F2C_OK && code != 0)
    TORCH_CHECK(false, "f2cgt_b200: a bounded wait ran out inside an earlier kernel of this device (code ", code,
                "): results of that call are unfinished (device_status() reports and clears this)");
}

float* f32(const at::Tensor& t) { return (float*)t.data_ptr(); }

at::Tensor mm(const Net& net, const at::Tensor& a, const at::Tensor& b) {
  return net.cast ? at::mm(a.to(*net.cast), b.to(*net.cast)).to(at::kFloat) : at::mm(a, b);
}
void addmm_(const Net& net, at::Tensor& y, const at::Tensor& a, const at::Tensor& b) {
  if (net.cast) y.add_(mm(net, a, b)); else y.addmm_(a, b);
}

// Whether a layer's forward product is the library's kernel.  Both sides round operands to tf32 (2.9e-4 off in float64 terms for either)
// except for one column or one row, where cuBLAS takes a matrix-vector product in fp32 (1e-7): those stay there.  Under a training run
// (record) the result has to be the two library products' bit for bit (see above).  It is for k % 32 == 0 from 2 rows on, for k % 8 == 0
// (checked for k = 8 .. 512, n = 4 .. 300, 2 .. 73,728 rows), and for k % 8 == 4, where cuBLAS adds in another order for few rows and for
// few columns or odd numbers of them, from 32,768 rows of 64 columns on (k = 20 .. 300, n = 64 .. 256 in fours, to 102,400 rows; at 64 columns
// 28,672 rows still differ).  k % 8 == 0 below 16,384 rows is left to cuBLAS, where a step has been timed that way only.
// tests/test_gpu_sage.py compares both sides over this range: with another cuBLAS it tells whether the rule still holds.
bool use_own(const Net& net, const at::Tensor& x1, const at::Tensor& x2, const at::Tensor& w1, const at::Tensor& w2, int64_t rows, bool record) {
  const int64_t n = w1.size(0), k = w1.size(1);
  if (!net.tf32 || k % 4 != 0 || k > 65536 || n < 2 || n > 65536 || rows < 2) return false;
  for (const at::Tensor* t : {&x1, &x2, &w1, &w2})  // parameters may be views into a flat buffer
    if ((reinterpret_cast<uintptr_t>(t->data_ptr()) & 15) != 0) return false;
  if (!record) return true;
  if (n < 4) return false;  // (two columns of k = 512: another order)
  return k % 32 == 0 || (k % 8 == 0 && rows >= 16384) || (n % 4 == 0 && n >= 64 && rows >= 32768);
}

// Ranges to be set to zero, as many in one launch as it takes: a memset each costs the host as much as a kernel.
struct Zeros {
  static constexpr int kMost = 32;  // of f2c_zero_ranges
  explicit Zeros(cudaStream_t stream) : st(stream) {}
  cudaStream_t st;
  void* at[kMost];
  int64_t bytes[kMost];
  int count = 0;
  void add(void* p, int64_t n) {
    if (n <= 0) return;
    if (count == kMost) run();
    at[count] = p;
    bytes[count++] = n;
  }
  void tail(const at::Tensor& t, int64_t rows) { add(f32(t) + rows * t.size(1), (t.size(0) - rows) * t.size(1) * 4); }
  void run() {
    checked = f2c_zero_ranges(at, bytes, count, st);
    count = 0;
  }
};

// Products of the backward pass as at::mm computes them (same library call, same operands), without its dispatch: out is
// [a.size(1), b.size(1)] = a^T (first rows of b), or - plain - [a.size(0), b.size(1)] = a b, added to what out holds when add.
void product(const Net& net, at::Tensor& out, const at::Tensor& a, bool a_turned, const at::Tensor& b, bool add) {
  const int64_t inner = a_turned ? a.size(0) : b.size(0), rows = out.size(0), cols = out.size(1);
  if (net.cast) {
    const at::Tensor r = mm(net, a_turned ? a.t() : a, b.narrow(0, 0, inner));
    if (add) out.add_(r); else out.copy_(r);
    return;
  }
  const float one = 1.0f, beta = add ? 1.0f : 0.0f;
  const cublasStatus_t rc = cublasSgemm(at::cuda::getCurrentCUDABlasHandle(), CUBLAS_OP_N, a_turned ? CUBLAS_OP_T : CUBLAS_OP_N, (int)cols,
                                        (int)rows, (int)inner, &one, f32(b), (int)cols, f32(a), (int)(a_turned ? rows : inner), &beta, f32(out),
                                        (int)cols);
  TORCH_CHECK(rc == CUBLAS_STATUS_SUCCESS, "cublasSgemm failed with status ", (int)rc);
}

// y of one layer (before dropout), `padded` rows
at::Tensor layer_forward(const Net& net, const at::Tensor& x1, const at::Tensor& x2, const at::Tensor* w, const Layer& l, bool relu, bool record,
                         cudaStream_t st) {
  const at::Tensor &w1 = w[0], &w2 = w[1], &bias = w[2];
  if (use_own(net, x1, x2, w1, w2, l.rows, record)) {
    at::Tensor y = empty({l.padded, w1.size(0)}, at::kFloat, x1.device());
    checked = f2c_sage_forward(f32(x1), f32(x2), f32(w1), f32(w2), bias.defined() ? f32(bias) : nullptr, f32(y), l.rows, w1.size(0), w1.size(1),
                               relu ? 1 : 0, st);
    return y;
  }
  const at::Tensor a = x1.narrow(0, 0, l.padded), b = x2.narrow(0, 0, l.padded);
  at::Tensor y;
  if (bias.defined() && !net.cast) {
    y = at::addmm(bias, a, w1.t());
  } else {
    y = mm(net, a, w1.t());
    if (bias.defined()) y.add_(bias);
  }
  addmm_(net, y, b, w2.t());
  if (relu) y.relu_();
  return y;
}

// The stream beside the caller's on which weight gradients run, and the events that tie the two; one set per thread and device.
struct Beside {
  c10::optional<c10::cuda::CUDAStream> stream;
  at::cuda::CUDAEvent fork{cudaEventDisableTiming}, join{cudaEventDisableTiming};
};
Beside& beside(c10::DeviceIndex device) {
  // never freed: at thread exit the CUDA context may be gone before the events
  static thread_local std::array<Beside*, 64> all{};
  Beside*& b = all[(size_t)device & 63];
  if (b == nullptr) {
    b = new Beside();
    b->stream = c10::cuda::getStreamFromPool(false, device);
  }
  return *b;
}
constexpr int64_t kBesideRows = 4096;  // fewer rows: a product is shorter than the calls that would move it

// Stands behind gradients that were asked for with a graph (create_graph) and have none.
struct NotTwice : public torch::autograd::Node {
  std::string name() const override { return "SageNotTwiceDifferentiable"; }
  variable_list apply(variable_list&&) override {
    TORCH_CHECK(false, "a SAGE network of several layers cannot be differentiated twice: its aggregations have no second derivative here");
  }
};

// A tensor kept for the backward pass, and what it has to be when it comes back: saved-tensor hooks (offloading, checkpointing) see
// it like any other saved tensor, and may give back another one.
class Kept {
 public:
  explicit Kept(const at::Tensor& t) : saved_(t, false) {
    if (!t.defined()) return;
    sizes_ = t.sizes();
    dtype_ = t.scalar_type();
    device_ = t.device();
  }
  at::Tensor get(const std::shared_ptr<torch::autograd::Node>& node) const {
    at::Tensor t = saved_.unpack(node);
    if (!t.defined()) return t;
    TORCH_CHECK(t.sizes() == sizes_ && t.scalar_type() == dtype_ && t.device() == device_,
                "sage_net: a saved-tensor hook gave back a tensor of another shape, type or device");
    return t.contiguous();
  }

 private:
  SavedVariable saved_;
  c10::DimVector sizes_;
  at::ScalarType dtype_ = at::kFloat;
  at::Device device_ = at::kCPU;
};

// One layer of what the backward pass needs: inputs of the products (x1 is also the previous layer's output), what the ReLU gave and
// dropout's mask (undefined in the last layer and without dropout), the block (not in the first layer).
template <typename T>
struct PerLayer { T x1, x2, active, keep, indptr, indices; };

struct SageBackward : public torch::autograd::Node {
  Net net;
  std::vector<Kept> weights;            // per layer: self, neigh, bias
  std::vector<PerLayer<Kept>> layers;
  bool released = false;

  std::string name() const override { return "SageBackward"; }
  void release_variables() override {
    released = true;
    weights.clear(); layers.clear();
  }

  variable_list apply(variable_list&& grads) override {
    TORCH_CHECK(!released, "Trying to backward through the graph a second time: its saved tensors have been freed");
    if (!grads[0].defined()) return variable_list(3 * net.layers.size());
    const int type = g_product_type.load();
    net.cast = type < 0 ? c10::nullopt : c10::make_optional((at::ScalarType)type);
    if (!at::GradMode::is_enabled()) return gradients(grads[0]);
    // create_graph: the gradients are to be differentiable themselves
    if (net.layers.size() == 1) return one_layer_with_graph(grads[0]);
    variable_list result = gradients(grads[0]), from = {grads[0]};
    auto self = shared_from_this();
    for (const Kept& w : weights) from.push_back(w.get(self));
    if (!torch::autograd::compute_requires_grad(from)) return result;
    auto node = std::shared_ptr<NotTwice>(new NotTwice(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(from));
    for (at::Tensor& r : result) {
      if (!r.defined()) continue;
      {
        at::NoGradGuard no_grad;
        r = r.clone();  // two of them share memory
      }
      torch::autograd::set_history(r, node);
    }
    return result;
  }

  // A single layer is linear in the gradient that it is given, so torch's own products make the graph.
  variable_list one_layer_with_graph(const at::Tensor& given) {
    const at::Tensor dy = given.to(at::kFloat), turned = dy.t();
    auto self = shared_from_this();
    const at::Tensor x1 = layers[0].x1.get(self).narrow(0, 0, dy.size(0)), x2 = layers[0].x2.get(self).narrow(0, 0, dy.size(0));
    auto of = [&](size_t i, auto&& make) { return task_should_compute_output(i) ? make() : at::Tensor(); };
    const bool bias = weights[2].get(self).defined();
    return {of(0, [&] { return mm(net, turned, x1); }), of(1, [&] { return mm(net, turned, x2); }),
            of(2, [&] { return bias ? dy.sum(0) : at::Tensor(); })};
  }

  variable_list gradients(const at::Tensor& grad_output) {
    const size_t L = net.layers.size();
    variable_list result(3 * L);
    at::NoGradGuard no_grad;
    const at::Tensor given = grad_output.to(at::kFloat);
    c10::cuda::CUDAGuard guard(given.device());
    check_reported();
    const c10::cuda::CUDAStream main = at::cuda::getCurrentCUDAStream(given.device().index());
    cudaStream_t st = main.stream();
    auto self = shared_from_this();
    std::vector<at::Tensor> w(3 * L);
    int64_t biases = 0;
    for (size_t i = 0; i < 3 * L; ++i) {
      w[i] = weights[i].get(self);
      if (i % 3 == 2 && w[i].defined()) biases += (w[i].numel() + 63) / 64 * 64;
    }
    std::vector<PerLayer<at::Tensor>> of;
    for (const PerLayer<Kept>& l : layers)
      of.push_back({l.x1.get(self), l.x2.get(self), l.active.get(self), l.keep.get(self), l.indptr.get(self), l.indices.get(self)});
    at::Tensor bias_grads = empty({biases}, at::kFloat, given.device());  // the mask kernel adds to it
    // The weight gradients' products run over padded rows, where the gradients are zero; what they meet there must be finite.
    Zeros zeros(st);
    zeros.add(bias_grads.data_ptr(), biases * 4);
    for (size_t i = 0; i < L; ++i) {
      zeros.tail(of[i].x1, net.layers[i == 0 ? 0 : i - 1].rows);
      zeros.tail(of[i].x2, net.layers[i].rows);
    }

    // gradient of the last layer's output on its padded rows
    at::Tensor g = given.contiguous();
    if (net.layers[L - 1].padded > g.size(0)) {
      at::Tensor padded = empty({net.layers[L - 1].padded, g.size(1)}, at::kFloat, g.device());
      C10_CUDA_CHECK(cudaMemcpyAsync(padded.data_ptr(), g.data_ptr(), (size_t)g.numel() * 4, cudaMemcpyDeviceToDevice, st));
      zeros.tail(padded, g.size(0));
      g = padded;
    }
    zeros.run();
    Beside& side = beside(given.device().index());
    std::vector<at::Tensor> read_beside;  // what the side stream reads, until the streams have joined
    // Joins the streams again, also when something below throws (out of memory): until then what the other stream reads and writes must
    // not serve anybody else.
    struct Join {
      Beside& side;
      const c10::cuda::CUDAStream& main;
      bool forked = false;
      void now() {
        if (!std::exchange(forked, false)) return;
        side.join.record(*side.stream);
        side.join.block(main);
      }
      ~Join() {
        try { now(); } catch (...) {}
      }
    } join{side, main};
    int64_t bias_at = 0;
    for (size_t i = L; i-- > 0;) {
      const Layer& l = net.layers[i];
      const at::Tensor* wi = &w[3 * i];
      const int64_t n = wi[0].size(0), k = wi[0].size(1), m = g.size(0);
      at::Tensor db;
      if (wi[2].defined()) {
        db = bias_grads.narrow(0, bias_at, n);
        bias_at += (n + 63) / 64 * 64;
      }
      at::Tensor dy = g;
      if (i + 1 < L) {
        dy = empty({m, n}, at::kFloat, g.device());
        const at::Tensor &active = of[i].active, &keep = of[i].keep;
        checked = f2c_sage_mask_dropout(f32(g), f32(of[i + 1].x1), active.defined() ? f32(active) : nullptr,
                                        keep.defined() ? (const uint8_t*)keep.data_ptr() : nullptr, (float)net.scale(), f32(dy),
                                        db.defined() ? f32(db) : nullptr, m, n, st);
      } else if (db.defined()) {
        checked = f2c_sage_mask(f32(dy), nullptr, 1.0f, nullptr, f32(db), m, n, st);
      }
      result[3 * i + 2] = db;
      at::Tensor both = empty({2, n, k}, at::kFloat, g.device());
      at::Tensor d_self = result[3 * i] = both.select(0, 0), d_nb = result[3 * i + 1] = both.select(0, 1);
      if (m >= kBesideRows) {
        side.fork.record(main);
        side.fork.block(*side.stream);
        join.forked = true;
        c10::cuda::CUDAStreamGuard on_side(*side.stream);
        product(net, d_nb, dy, true, of[i].x2, false);
        if (i > 0) product(net, d_self, dy, true, of[i].x1, false);
        read_beside.push_back(dy);
      } else {
        product(net, d_nb, dy, true, of[i].x2, false);
        if (i > 0) product(net, d_self, dy, true, of[i].x1, false);
      }
      if (i == 0) product(net, d_self, dy, true, of[i].x1, false);
      if (i > 0) {
        at::Tensor dh = empty({net.layers[i - 1].padded, k}, at::kFloat, g.device());  // gradient of the previous layer's output
        at::Tensor d_rows = empty({m, k}, at::kFloat, g.device());
        product(net, d_rows, dy, false, wi[1], false);
        checked = f2c_spmm_csr_backward(f32(d_rows), of[i].indptr.data_ptr(), of[i].indices.data_ptr(), dtype_tag(of[i].indptr.scalar_type()), f32(dh),
                                        l.rows, dh.size(0), k, F2C_MEAN, st);
        at::Tensor head = dh.narrow(0, 0, m);
        product(net, head, dy, false, wi[0], true);
        g = dh;
      }
    }
    join.now();
    for (size_t i = 0; i < 3 * L; ++i)
      if (!task_should_compute_output(i)) result[i] = at::Tensor();
    return result;
  }
};

// h_self, h_neigh, indptrs (list, layers 1..), indices (list), rows (list), padded (list), weights (list of 3 L, None = no bias),
// dropout p, tf32 products allowed (bool), operand type of torch's products (torch.dtype or None)
PyObject* sage_net(PyObject*, PyObject* const* a, Py_ssize_t n) {
  return guarded([&]() -> PyObject* {
    arguments("sage_net", n, 10);
    const at::Tensor& h_self = tensor(a[0], "h_self", kF32);
    const at::Tensor& h_neigh = tensor(a[1], "h_neigh", kF32);
    auto list = [](PyObject* o, Py_ssize_t want) {
      if (!PyList_Check(o) || (want >= 0 && PyList_GET_SIZE(o) != want)) fail(PyExc_TypeError, "sage_net: lists of matching lengths are wanted");
      return PyList_GET_SIZE(o);
    };
    const Py_ssize_t L = list(a[4], -1);
    list(a[2], L - 1); list(a[3], L - 1); list(a[5], L); list(a[6], 3 * L);
    Net net;
    net.layers.resize(L);
    std::vector<at::Tensor> w(3 * L);
    for (Py_ssize_t i = 0; i < L; ++i) {
      Layer& l = net.layers[i];
      l.rows = integer(PyList_GET_ITEM(a[4], i));
      l.padded = integer(PyList_GET_ITEM(a[5], i));
      if (l.rows < 0 || l.padded < l.rows) fail(PyExc_RuntimeError, "sage_net: bad row counts");
      if (i > 0) {
        l.indptr = tensor(PyList_GET_ITEM(a[2], i - 1), "indptr", kIndex);
        l.indices = tensor(PyList_GET_ITEM(a[3], i - 1), "indices", kIndex);
        if (l.indptr.scalar_type() != l.indices.scalar_type()) fail(PyExc_RuntimeError, "indptr and indices must have the same dtype");
        if (l.indptr.numel() != l.rows + 1 || l.rows > net.layers[i - 1].rows || l.padded > net.layers[i - 1].padded) fail(PyExc_RuntimeError, "sage_net: blocks do not fit together");
      }
      for (int j = 0; j < 3; ++j) {
        PyObject* o = PyList_GET_ITEM(a[6], 3 * i + j);
        if (j == 2 && o == Py_None) continue;
        w[3 * i + j] = tensor(o, "weight", kF32);
      }
      const at::Tensor &w1 = w[3 * i], &w2 = w[3 * i + 1];
      const int64_t in = i == 0 ? h_self.size(1) : w[3 * i - 3].size(0);
      if (w1.dim() != 2 || w1.sizes() != w2.sizes() || w1.size(1) != in || (w[3 * i + 2].defined() && w[3 * i + 2].numel() != w1.size(0)))
        fail(PyExc_RuntimeError, "sage_net: weights do not fit together");
    }
    net.p = real(a[7]);
    net.tf32 = PyObject_IsTrue(a[8]) == 1;
    if (a[9] != Py_None) net.cast = reinterpret_cast<THPDtype*>(a[9])->scalar_type;
    if (h_self.dim() != 2 || h_self.sizes() != h_neigh.sizes() || h_self.size(0) < net.layers[0].padded) fail(PyExc_RuntimeError, "sage_net: bad inputs");
    auto elsewhere = [&](const at::Tensor& t) { return t.defined() && t.device() != h_self.device(); };
    bool apart = elsewhere(h_neigh);
    for (const at::Tensor& t : w) apart = apart || elsewhere(t);
    for (const Layer& l : net.layers) apart = apart || elsewhere(l.indptr) || elsewhere(l.indices);
    if (apart) fail(PyExc_RuntimeError, "sage_net: expected all tensors on the same device");
    const bool record = at::GradMode::is_enabled() && torch::autograd::compute_requires_grad(w);
    at::Tensor result = unlocked([&] {
      c10::cuda::CUDAGuard guard(h_self.device());
      check_reported();
      cudaStream_t st = stream_of(h_self);
      std::shared_ptr<SageBackward> node;
      if (record) {
        node = std::shared_ptr<SageBackward>(new SageBackward(), torch::autograd::deleteNode);
        node->set_next_edges(torch::autograd::collect_next_edges(w));
      }
      at::Tensor h;
      std::vector<PerLayer<at::Tensor>> of;
      of.reserve(L);
      {
        at::AutoDispatchBelowADInplaceOrView below;
        at::Tensor x1 = h_self, x2 = h_neigh;
        for (Py_ssize_t i = 0; i < L; ++i) {
          const Layer& l = net.layers[i];
          const bool last = i + 1 == L;
          if (i > 0) {
            x1 = h;
            x2 = empty({l.padded, h.size(1)}, at::kFloat, h.device());
            checked = f2c_spmm_csr(h.data_ptr(), F2C_F32, l.indptr.data_ptr(), l.indices.data_ptr(), dtype_tag(l.indptr.scalar_type()), x2.data_ptr(),
                                   l.rows, h.size(1), F2C_MEAN, st);
          }
          h = layer_forward(net, x1, x2, &w[3 * i], l, !last, record, st);
          const at::Tensor active = h;
          at::Tensor keep;
          if (!last && net.p > 0) {
            if (net.p < 1 && h.numel() > 0) std::tie(h, keep) = at::native_dropout(h, net.p, true);
            else h = at::dropout(h, net.p, true);
          }
          if (record) of.push_back({x1, x2, last || net.p <= 0 ? at::Tensor() : active, keep, l.indptr, l.indices});
        }
        if (h.size(0) > net.layers[L - 1].rows) h = h.narrow(0, 0, net.layers[L - 1].rows);
      }
      if (record) {
        node->weights.reserve(w.size());
        node->layers.reserve(of.size());
        for (const at::Tensor& t : w) node->weights.emplace_back(t);
        for (const PerLayer<at::Tensor>& l : of)
          node->layers.push_back({Kept(l.x1), Kept(l.x2), Kept(l.active), Kept(l.keep), Kept(l.indptr), Kept(l.indices)});
        for (Layer& l : net.layers) l.indptr = l.indices = at::Tensor();
        node->net = std::move(net);
        torch::autograd::set_history(h, node);
      }
      return h;
    });
    return THPVariable_Wrap(std::move(result));
  });
}

PyObject* product_type(PyObject*, PyObject* o) {  // torch.dtype or None
  return guarded([&]() -> PyObject* {
    if (o != Py_None && !THPDtype_Check(o)) fail(PyExc_TypeError, "product_type: a torch.dtype or None");
    g_product_type = o == Py_None ? -1 : (int)reinterpret_cast<THPDtype*>(o)->scalar_type;
    Py_RETURN_NONE;
  });
}

}  // namespace

PyMethodDef g_sage_methods[] = {{"sage_net", (PyCFunction)(void*)sage_net, METH_FASTCALL, nullptr},
                                {"product_type", product_type, METH_O, nullptr},
                                {nullptr, nullptr, 0, nullptr}};

}  // namespace f2c_native
