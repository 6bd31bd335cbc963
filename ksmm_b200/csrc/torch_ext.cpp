// Thin PyTorch C++ extension over the C ABI of libksmm_cu.so.
//
// Same module surface as the reference's extension
// (src/ksmm_py/layer/kronecker_sparse/kernel.cpp:25-50): forward(input, factor,
// bs_last, a, b, c, d, dtype, vsize) -> output tensor on the input's device and
// current stream.  `dtype` and `vsize` are accepted for signature compatibility;
// the element type is the input tensor's and vector widths are chosen by the
// library.  chain_forward runs all factors of one KSLinear in one call.
//
// The package's own layers go through layer_forward, layer_train, factor_forward, fp8_forward and
// grouped_forward below, which hold everything between Python and the C ABI (argument checks, output and
// workspace allocation, stream): two factors (384 -> 1536, fp16) on 16 rows 48 -> 20 us against the same calls
// through ctypes, a training step of that layer 241 -> 151 us.  They return None where an
// argument is not what the call takes; the Python wrappers then run the same call through ctypes and raise
// what is wrong with it.  A status other than KSMM_OK comes back as that number; inside the autograd node of
// layer_train it raises what the wrappers raise for it.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <string>
#include <vector>

#include "../../include/ksmm_cu.h"

namespace {

int dtype_code(const torch::Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return KSMM_F32;
    case at::kHalf: return KSMM_F16;
    case at::kBFloat16: return KSMM_BF16;
    default: TORCH_CHECK(false, "ksmm: unsupported tensor type ", t.scalar_type());
  }
  return -1;
}

void check_input(const torch::Tensor& x, const char* name) {
  TORCH_CHECK(x.device().is_cuda(), name, " must be a CUDA tensor");
  TORCH_CHECK(x.is_contiguous(), name, " must be contiguous");
}

void check_status(int st) { TORCH_CHECK(st == KSMM_OK, "libksmm_cu: ", ksmm_cu_last_error()); }

torch::Tensor forward(torch::Tensor input, torch::Tensor factor, int64_t bs_last, int64_t a, int64_t b,
                      int64_t c, int64_t d, const std::string& /*dtype*/, int64_t /*vsize*/) {
  check_input(input, "input");
  check_input(factor, "factor");
  TORCH_CHECK(input.dim() == 2 && factor.dim() == 2, "input and factor are 2-D");
  TORCH_CHECK(input.size(bs_last ? 0 : 1) == a * c * d, "input has ", input.size(bs_last ? 0 : 1),
              " features, the pattern expects ", a * c * d);
  TORCH_CHECK(factor.size(0) == a * d * c && factor.size(1) == b, "factor must be (a*d*c, b)");
  TORCH_CHECK(factor.scalar_type() == input.scalar_type() && factor.device() == input.device(),
              "factor and input must share type and device");
  const c10::cuda::CUDAGuard guard(input.device());
  const int64_t batch = input.size(bs_last ? 1 : 0);
  auto out = bs_last ? torch::empty({a * b * d, batch}, input.options())
                     : torch::empty({batch, a * b * d}, input.options());
  ksmm_forward_desc_t f = {};
  f.input = input.data_ptr();
  f.values = factor.data_ptr();
  f.output = out.data_ptr();
  f.batch = batch;
  f.a = static_cast<int>(a); f.b = static_cast<int>(b); f.c = static_cast<int>(c); f.d = static_cast<int>(d);
  f.in_dtype = f.out_dtype = dtype_code(input);
  f.bs_last = bs_last ? 1 : 0;
  f.algo = KSMM_ALGO_AUTO;
  f.config = -1;
  f.alpha = 1.f;
  torch::Tensor scratch;
  if (const size_t need = ksmm_cu_layout_scratch_bytes(&f)) {
    scratch = torch::empty({static_cast<int64_t>(need)}, input.options().dtype(at::kByte));
    f.scratch = scratch.data_ptr();
    f.scratch_bytes = need;
  }
  check_status(ksmm_cu_forward_ex(&f, at::cuda::getCurrentCUDAStream().stream()));
  return out;
}

torch::Tensor chain_forward(torch::Tensor input, std::vector<torch::Tensor> factors,
                            std::vector<std::vector<int64_t>> patterns, int64_t bs_last,
                            c10::optional<torch::Tensor> bias, int64_t activation) {
  check_input(input, "input");
  TORCH_CHECK(input.dim() == 2, "input is 2-D: (features, batch) batch-last, (batch, features) batch-first");
  TORCH_CHECK(!patterns.empty() && patterns.size() == factors.size(), "one factor per pattern");
  std::vector<int32_t> flat;
  std::vector<const void*> vals;
  int64_t feats = input.size(bs_last ? 0 : 1);  // features entering the next factor
  for (size_t f = 0; f < patterns.size(); ++f) {
    TORCH_CHECK(patterns[f].size() == 4, "a pattern is (a, b, c, d)");
    for (int64_t v : patterns[f])
      TORCH_CHECK(v > 0 && v <= 0x7fffffffLL, "pattern values are positive 32-bit integers, got ", v);
    const int64_t a = patterns[f][0], b = patterns[f][1], c = patterns[f][2], d = patterns[f][3];
    TORCH_CHECK(a * c * d == feats, "factor ", f, " expects ", a * c * d, " features but receives ", feats);
    check_input(factors[f], "factor");
    TORCH_CHECK(factors[f].dim() == 2 && factors[f].size(0) == a * d * c && factors[f].size(1) == b,
                "factor ", f, " must have shape (a*d*c, b) = (", a * d * c, ", ", b, ")");
    TORCH_CHECK(factors[f].scalar_type() == input.scalar_type(), "factors share the input's type");
    TORCH_CHECK(factors[f].device() == input.device(), "factors live on the input's device");
    for (int64_t v : patterns[f]) flat.push_back(static_cast<int32_t>(v));
    vals.push_back(factors[f].data_ptr());
    feats = a * b * d;
  }
  const c10::cuda::CUDAGuard guard(input.device());
  const int64_t batch = input.size(bs_last ? 1 : 0);
  const auto& pl = patterns.back();
  const int64_t n_out = pl[0] * pl[1] * pl[3];
  auto out = bs_last ? torch::empty({n_out, batch}, input.options())
                     : torch::empty({batch, n_out}, input.options());
  const int code = dtype_code(input);
  const size_t need = ksmm_cu_chain_workspace_bytes_ex(static_cast<int>(patterns.size()), flat.data(), batch,
                                                       code, bs_last ? 1 : 0);
  torch::Tensor ws;
  if (need > 0) ws = torch::empty({static_cast<int64_t>(need)}, input.options().dtype(at::kByte));
  const void* bptr = nullptr;
  if (bias.has_value()) {
    check_input(*bias, "bias");
    TORCH_CHECK(bias->numel() == n_out && bias->scalar_type() == input.scalar_type() &&
                    bias->device() == input.device(),
                "bias must hold out_size elements of the input's type on the input's device");
    bptr = bias->data_ptr();
  }
  check_status(ksmm_cu_chain_forward_act(input.data_ptr(), vals.data(), out.data_ptr(), bptr,
                                         need > 0 ? ws.data_ptr() : nullptr, need, batch,
                                         static_cast<int>(patterns.size()), flat.data(), code,
                                         bs_last ? 1 : 0, static_cast<int>(activation),
                                         at::cuda::getCurrentCUDAStream().stream()));
  return out;
}


// ---------------------------------------------------------------------------
// the package's own calls
// ---------------------------------------------------------------------------
struct Patterns {
  std::vector<int32_t> flat;
  int n = 0;
  int64_t in(int f) const { return static_cast<int64_t>(flat[4 * f]) * flat[4 * f + 2] * flat[4 * f + 3]; }
  int64_t out(int f) const { return static_cast<int64_t>(flat[4 * f]) * flat[4 * f + 1] * flat[4 * f + 3]; }
};

// a list of 4-tuples of positive ints; false for anything else
bool read_patterns(const py::handle& h, Patterns* p) {
  PyObject* seq = h.ptr();
  if (!PyList_Check(seq) && !PyTuple_Check(seq)) return false;
  const Py_ssize_t n = PySequence_Fast_GET_SIZE(seq);
  if (n < 1 || n > 1024) return false;
  p->n = static_cast<int>(n);
  p->flat.reserve(4 * n);
  for (Py_ssize_t f = 0; f < n; ++f) {
    PyObject* q = PySequence_Fast_GET_ITEM(seq, f);
    if ((!PyList_Check(q) && !PyTuple_Check(q)) || PySequence_Fast_GET_SIZE(q) != 4) return false;
    for (int e = 0; e < 4; ++e) {
      PyObject* v = PySequence_Fast_GET_ITEM(q, e);
      if (!PyLong_Check(v)) return false;
      int overflow = 0;
      const long long x = PyLong_AsLongLongAndOverflow(v, &overflow);
      if (overflow || x <= 0 || x > 0x7fffffffLL) return false;
      p->flat.push_back(static_cast<int32_t>(x));
    }
  }
  return true;
}

bool plain_dtype(const at::Tensor& t) {
  return t.scalar_type() == at::kFloat || t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16;
}

// a plain strided CUDA tensor whose memory may be handed to the library
bool usable(const at::Tensor& t) {
  return t.defined() && t.is_cuda() && t.layout() == at::kStrided && t.is_contiguous() && !t.is_neg() && !t.is_conj();
}

// does the chain take these tensors?  groups: weights of several chains, one after the other
bool chain_fits(const at::Tensor& x, const std::vector<at::Tensor>& w, const Patterns& p, bool last, at::ScalarType wtype,
                int64_t groups = 1) {
  if (static_cast<int>(w.size()) != p.n || !usable(x) || x.dim() != 2 || x.size(last ? 0 : 1) != p.in(0)) return false;
  for (int f = 0; f < p.n; ++f) {
    if (!usable(w[f]) || w[f].dim() != 2 || w[f].scalar_type() != wtype || w[f].device() != x.device()) return false;
    if (w[f].size(0) != groups * p.flat[4 * f] * static_cast<int64_t>(p.flat[4 * f + 3]) * p.flat[4 * f + 2] ||
        w[f].size(1) != p.flat[4 * f + 1])
      return false;
    if (f > 0 && p.in(f) != p.out(f - 1)) return false;
  }
  return true;
}

bool bias_fits(const c10::optional<at::Tensor>& b, const at::Tensor& x, int64_t n, at::ScalarType type) {
  return !b.has_value() || (usable(*b) && b->numel() == n && b->scalar_type() == type && b->device() == x.device());
}

const void* ptr_or_null(const c10::optional<at::Tensor>& t) { return t.has_value() ? t->data_ptr() : nullptr; }

at::Tensor new_tensor(int64_t feats, int64_t batch, bool last, const at::TensorOptions& o) {
  return last ? at::empty({feats, batch}, o) : at::empty({batch, feats}, o);
}
at::Tensor new_bytes(size_t n, const at::Tensor& like) {
  return at::empty({static_cast<int64_t>(n)}, like.options().dtype(at::kByte));
}
void* stream_of(const at::Tensor& x) { return at::cuda::getCurrentCUDAStream(x.get_device()).stream(); }

std::vector<const void*> pointers(const std::vector<at::Tensor>& w) {
  std::vector<const void*> v(w.size());
  for (size_t f = 0; f < w.size(); ++f) v[f] = w[f].data_ptr();
  return v;
}

bool wants_grad(const at::Tensor& x, const std::vector<at::Tensor>& w, const c10::optional<at::Tensor>& b) {
  if (!at::GradMode::is_enabled()) return false;
  if (x.requires_grad() || (b.has_value() && b->requires_grad())) return true;
  for (const auto& t : w)
    if (t.requires_grad()) return true;
  return false;
}

py::object result(int st, const at::Tensor& out) { return st == KSMM_OK ? py::cast(out) : py::cast(st); }

// KSLinear without gradients: every factor, bias, activation and residual in one call
py::object layer_forward(const at::Tensor& x, const std::vector<at::Tensor>& factors, const py::handle& patterns, bool last,
                         bool out_last, const c10::optional<at::Tensor>& bias, int activation,
                         const c10::optional<at::Tensor>& residual) {
  Patterns p;
  if (!read_patterns(patterns, &p) || !usable(x) || !plain_dtype(x) || wants_grad(x, factors, bias) ||
      !chain_fits(x, factors, p, last, x.scalar_type()) || !bias_fits(bias, x, p.out(p.n - 1), x.scalar_type()))
    return py::none();
  const int64_t batch = x.size(last ? 1 : 0), n_out = p.out(p.n - 1);
  if (residual.has_value() && (!usable(*residual) || residual->scalar_type() != x.scalar_type() || residual->dim() != 2 ||
                               residual->size(out_last ? 0 : 1) != n_out || residual->size(out_last ? 1 : 0) != batch ||
                               residual->device() != x.device()))
    return py::none();
  int st;
  at::Tensor out;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(x.device());
    const int code = dtype_code(x);
    out = new_tensor(n_out, batch, out_last, x.options());
    const size_t need = ksmm_cu_chain_workspace_bytes_layouts(p.n, p.flat.data(), batch, code, last, out_last);
    at::Tensor ws;
    if (need) ws = new_bytes(need, x);
    const auto vals = pointers(factors);
    ksmm_chain_desc_t d = {};
    d.input = x.data_ptr();
    d.values = vals.data();
    d.output = out.data_ptr();
    d.bias = ptr_or_null(bias);
    d.residual = ptr_or_null(residual);
    d.workspace = need ? ws.data_ptr() : nullptr;
    d.workspace_bytes = need;
    d.batch = batch;
    d.nfactors = p.n;
    d.patterns = p.flat.data();
    d.dtype = code;
    d.bs_last = last;
    d.out_layout = out_last ? 2 : 1;
    d.activation = activation;
    st = ksmm_cu_chain_forward_desc(&d, stream_of(x));
  }
  return result(st, out);
}

// Kernel.forward: one factor
py::object factor_forward(const at::Tensor& x, const at::Tensor& w, bool last, int64_t a, int64_t b, int64_t c, int64_t d) {
  if (a <= 0 || b <= 0 || c <= 0 || d <= 0 || a > 0x7fffffff || b > 0x7fffffff || c > 0x7fffffff || d > 0x7fffffff ||
      !usable(x) || !usable(w) || !plain_dtype(x) || x.dim() != 2 || w.dim() != 2 || w.scalar_type() != x.scalar_type() ||
      w.device() != x.device() || x.size(last ? 0 : 1) != a * c * d || w.size(0) != a * c * d || w.size(1) != b)
    return py::none();
  int st;
  at::Tensor out;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t batch = x.size(last ? 1 : 0);
    out = new_tensor(a * b * d, batch, last, x.options().requires_grad(false));
    ksmm_forward_desc_t f = {};
    f.input = x.data_ptr();
    f.values = w.data_ptr();
    f.output = out.data_ptr();
    f.batch = batch;
    f.a = static_cast<int>(a); f.b = static_cast<int>(b); f.c = static_cast<int>(c); f.d = static_cast<int>(d);
    f.in_dtype = f.out_dtype = dtype_code(x);
    f.bs_last = last;
    f.algo = KSMM_ALGO_AUTO;
    f.config = -1;
    f.alpha = 1.f;
    const size_t need = ksmm_cu_layout_scratch_bytes(&f);
    at::Tensor scratch;
    if (need) {
      scratch = new_bytes(need, x);
      f.scratch = scratch.data_ptr();
      f.scratch_bytes = need;
    }
    st = ksmm_cu_forward_ex(&f, stream_of(x));
  }
  return result(st, out);
}

// the factors of an fp8 layer
py::object fp8_forward(const at::Tensor& x, const std::vector<at::Tensor>& factors, const std::vector<float>& scales,
                       const py::handle& patterns, bool last, const c10::optional<at::Tensor>& bias) {
  Patterns p;
  if (!read_patterns(patterns, &p) || !usable(x) || !plain_dtype(x) || scales.size() != factors.size() ||
      !chain_fits(x, factors, p, last, at::kFloat8_e4m3fn) || !bias_fits(bias, x, p.out(p.n - 1), at::kBFloat16))
    return py::none();
  int st;
  at::Tensor out;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t batch = x.size(last ? 1 : 0);
    const int code = dtype_code(x);
    out = new_tensor(p.out(p.n - 1), batch, last, x.options().dtype(at::kBFloat16).requires_grad(false));
    const size_t need = ksmm_cu_chain_fp8_workspace_bytes(p.n, p.flat.data(), batch, code, last);
    const at::Tensor ws = new_bytes(need, x);
    const auto vals = pointers(factors);
    st = ksmm_cu_chain_forward_fp8(x.data_ptr(), code, vals.data(), scales.data(), out.data_ptr(), ptr_or_null(bias),
                                   ws.data_ptr(), need, batch, p.n, p.flat.data(), last, stream_of(x));
  }
  return result(st, out);
}

// several chains on one input, weights and bias stacked
py::object grouped_forward(const at::Tensor& x, const std::vector<at::Tensor>& factors, const py::handle& patterns, bool last,
                           int64_t groups, const c10::optional<at::Tensor>& bias) {
  Patterns p;
  if (groups < 1 || groups > 65535 || !read_patterns(patterns, &p) || !usable(x) || !plain_dtype(x) ||
      !chain_fits(x, factors, p, last, x.scalar_type(), groups) ||
      !bias_fits(bias, x, groups * p.out(p.n - 1), x.scalar_type()))
    return py::none();
  int st;
  at::Tensor out;
  {
    py::gil_scoped_release nogil;
    const c10::cuda::CUDAGuard guard(x.device());
    const int64_t batch = x.size(last ? 1 : 0), n_out = p.out(p.n - 1);
    const int code = dtype_code(x);
    const auto o = x.options().requires_grad(false);
    out = last ? at::empty({groups, n_out, batch}, o) : at::empty({groups, batch, n_out}, o);
    const size_t need = groups * ksmm_cu_chain_workspace_bytes_ex(p.n, p.flat.data(), batch, code, last);
    at::Tensor ws;
    if (need) ws = new_bytes(need, x);
    const auto vals = pointers(factors);
    st = ksmm_cu_grouped_chain_forward(x.data_ptr(), vals.data(), out.data_ptr(), ptr_or_null(bias),
                                       need ? ws.data_ptr() : nullptr, need, batch, p.n, p.flat.data(), code, last,
                                       static_cast<int>(groups), stream_of(x));
  }
  return result(st, out);
}

// Raises ksmm_b200.KsmmError for a status, on whichever thread autograd runs (with or without the GIL).
void raise_status(int st) {
  if (st == KSMM_OK) return;
  py::gil_scoped_acquire gil;
  py::module_::import("ksmm_b200._lib").attr("check")(st);
}

// A trainable layer as one autograd node: ksmm_b200.kernel.ChainFunction without Python in its backward.
at::Tensor aligned(const at::Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 ? t.clone() : t; }

struct ChainNode : torch::autograd::Function<ChainNode> {
  static at::Tensor forward(torch::autograd::AutogradContext* ctx, const at::Tensor& x_in, const c10::optional<at::Tensor>& bias,
                            at::TensorList factors, std::vector<int64_t> patterns, bool last) {
    const at::Tensor x = aligned(x_in);
    const c10::cuda::CUDAGuard guard(x.device());
    const int n = static_cast<int>(factors.size());
    std::vector<int32_t> flat(patterns.begin(), patterns.end());
    const int32_t* pl = flat.data() + 4 * (n - 1);
    const int64_t batch = x.size(last ? 1 : 0), n_out = static_cast<int64_t>(pl[0]) * pl[1] * pl[3];
    const int code = dtype_code(x);
    size_t bytes[3];
    raise_status(ksmm_cu_chain_train_bytes(n, flat.data(), batch, code, last, &bytes[0], &bytes[1], &bytes[2]));
    at::Tensor out = new_tensor(n_out, batch, last, x.options());
    const at::Tensor saved = new_bytes(bytes[0], x), scratch = new_bytes(bytes[1], x);
    std::vector<const void*> vals(n);
    for (int f = 0; f < n; ++f) vals[f] = factors[f].data_ptr();
    int32_t layouts[16] = {};
    raise_status(ksmm_cu_chain_train_forward(x.data_ptr(), vals.data(), out.data_ptr(), ptr_or_null(bias), saved.data_ptr(),
                                             bytes[0], scratch.data_ptr(), bytes[1], batch, n, flat.data(), code, last, layouts,
                                             stream_of(x)));
    torch::autograd::variable_list keep{x, saved};
    keep.insert(keep.end(), factors.begin(), factors.end());
    ctx->save_for_backward(std::move(keep));
    // number of factors, layout, bytes of the backward, patterns, layouts, the bias's shape
    std::vector<int64_t> meta{n, last, static_cast<int64_t>(bytes[2])};
    meta.insert(meta.end(), patterns.begin(), patterns.end());
    for (int f = 0; f + 1 < n; ++f) meta.push_back(layouts[f]);
    meta.push_back(bias.has_value());
    if (bias.has_value()) meta.insert(meta.end(), bias->sizes().begin(), bias->sizes().end());
    ctx->saved_data["chain"] = std::move(meta);
    return out;
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    const auto kept = ctx->get_saved_variables();
    const std::vector<int64_t> meta = ctx->saved_data["chain"].toIntVector();
    const int n = static_cast<int>(meta[0]);
    const bool last = meta[1] != 0;
    const size_t need = static_cast<size_t>(meta[2]);
    const std::vector<int32_t> flat(meta.begin() + 3, meta.begin() + 3 + 4 * n);
    std::vector<int32_t> layouts(meta.begin() + 3 + 4 * n, meta.begin() + 3 + 4 * n + n - 1);
    const bool has_bias = meta[3 + 4 * n + n - 1] != 0;
    layouts.push_back(0);
    const at::Tensor& x = kept[0];
    const at::Tensor& saved = kept[1];
    const c10::cuda::CUDAGuard guard(x.device());
    const at::Tensor g = aligned(grads[0].contiguous());
    // edges of the graph: the input, the bias if there is one, the factors
    at::Tensor gx, gb;
    if (ctx->needs_input_grad(0)) gx = at::empty(x.sizes(), x.options());
    if (has_bias && ctx->needs_input_grad(1))
      gb = at::empty(at::IntArrayRef(meta.data() + 3 + 4 * n + n, meta.size() - (3 + 4 * n + n)), x.options());
    std::vector<at::Tensor> gw(n);
    std::vector<const void*> vals(n);
    std::vector<void*> outs(n, nullptr);
    for (int f = 0; f < n; ++f) {
      const at::Tensor& w = kept[2 + f];
      vals[f] = w.data_ptr();
      if (ctx->needs_input_grad(1 + has_bias + f)) {
        gw[f] = at::empty(w.sizes(), w.options());
        outs[f] = gw[f].data_ptr();
      }
    }
    const at::Tensor ws = new_bytes(need, x);
    raise_status(ksmm_cu_chain_backward(x.data_ptr(), vals.data(), saved.data_ptr(), layouts.data(), g.data_ptr(),
                                        gx.defined() ? gx.data_ptr() : nullptr, outs.data(),
                                        gb.defined() ? gb.data_ptr() : nullptr, ws.data_ptr(), need, x.size(last ? 1 : 0), n,
                                        flat.data(), dtype_code(x), last, stream_of(x)));
    torch::autograd::variable_list r{gx, gb};
    r.insert(r.end(), gw.begin(), gw.end());
    r.emplace_back();  // patterns
    r.emplace_back();  // layout
    return r;
  }
};

py::object layer_train(const at::Tensor& x, const std::vector<at::Tensor>& factors, const py::handle& patterns, bool last,
                       const c10::optional<at::Tensor>& bias) {
  Patterns p;
  if (!read_patterns(patterns, &p) || p.n > 16 || !usable(x) || !plain_dtype(x) ||
      !chain_fits(x, factors, p, last, x.scalar_type()) || !bias_fits(bias, x, p.out(p.n - 1), x.scalar_type()))
    return py::none();
  at::Tensor out;
  {
    py::gil_scoped_release nogil;
    out = ChainNode::apply(x, bias, at::TensorList(factors), std::vector<int64_t>(p.flat.begin(), p.flat.end()), last);
  }
  return py::cast(out);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("forward", &forward, "One Kronecker-sparse factor (CUDA, libksmm_cu)");
  m.def("chain_forward", &chain_forward, "All factors of a KSLinear in one call (CUDA, libksmm_cu)",
        py::arg("input"), py::arg("factors"), py::arg("patterns"), py::arg("bs_last"),
        py::arg("bias") = py::none(), py::arg("activation") = 0);
  m.def("layer_forward", &layer_forward, "A KSLinear without gradients");
  m.def("layer_train", &layer_train, "A trainable KSLinear as one autograd node");
  m.def("factor_forward", &factor_forward, "One factor in its input's type");
  m.def("fp8_forward", &fp8_forward, "The factors of an fp8 KSLinear");
  m.def("grouped_forward", &grouped_forward, "Several chains on one input");
}
