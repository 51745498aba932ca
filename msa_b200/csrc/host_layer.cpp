// The host side of a decoder layer of the memory model in bf16 inference, in native code.
//
// A decode token of two layers (32 sequences), then 34 launches of 300 us in all, took 714 us through the modules: what bounded it was Python
// between them (module calls, attribute look-ups through nn.Module.__getattr__, ctypes).  The same launches took 371 us from here (30 of
// them 350, since the one that appends a token advances the lengths), 16 questions of 96 tokens 1361 us instead of 1566.  A layer is two
// calls around the attention of its stage:
// `front` (residual add and norm, q / k / v, head norm and rotation) and `back` (output product, residual add and norm, gated
// feed-forward), and a third for the attention of a single token.  Products are the library calls
// that nn.Linear comes to.
//
// Nothing is kept between calls.  `layers` reads the modules anew each time and answers None where anything is not what it steps
// over: another class, a hook, a forward of its own, a bias, a subclass of Tensor, another device or type; every other function
// answers None for operands that it does not take.  The caller then goes the way through the modules.
#include <dlfcn.h>

#include <ATen/PythonTorchFunctionTLS.h>
#include <ATen/autocast_mode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <array>

#include "../../include/msa_b200.h"

namespace {

using at::Tensor;
namespace py = pybind11;

#define MSA_FUNCTIONS(F) \
  F(msa_last_error) F(msa_add_rmsnorm) F(msa_heads_norm_rope) F(msa_silu_mul_parts) F(msa_rope_table) F(msa_decode_workspace_bytes) F(msa_sparse_decode_attn_next)
struct Library {
#define MSA_MEMBER(name) decltype(&::name) name = nullptr;
  MSA_FUNCTIONS(MSA_MEMBER)
#undef MSA_MEMBER
} lib;

void bind(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(h, "cannot load ", path, ": ", dlerror());
  Library l;
#define MSA_LOAD(name)                                              \
  l.name = reinterpret_cast<decltype(l.name)>(dlsym(h, #name));     \
  TORCH_CHECK(l.name, path, " lacks " #name);
  MSA_FUNCTIONS(MSA_LOAD)
#undef MSA_LOAD
  lib = l;
}
void check(int rc, const char* what) { TORCH_CHECK(rc == 0, what, " failed (", rc, "): ", lib.msa_last_error()); }

// ---- what the fused calls take
bool plain_key_set(const Tensor& t) {             // no wrapper of a transformation, no negative or conjugate view
  const c10::DispatchKeySet known({c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView, c10::DispatchKey::AutocastCUDA,
                                   c10::DispatchKey::CUDA});
  return t.is_cuda() && (t.key_set().raw_repr() & ~known.raw_repr() & ~c10::full_backend_mask) == 0;
}
bool takes(const Tensor& t, at::ScalarType type, c10::Device device) {
  return t.defined() && plain_key_set(t) && t.scalar_type() == type && t.device() == device && t.is_contiguous() &&
         reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0;
}
bool bf16(const Tensor& t, c10::Device device) { return takes(t, at::kBFloat16, device); }
bool quiet() {                                     // no gradient to keep, nobody who watches or changes calls
  return !at::GradMode::is_enabled() && !at::autocast::is_autocast_enabled(at::kCUDA) && !c10::impl::dispatch_mode_enabled() &&
         !at::impl::torch_function_mode_enabled() && lib.msa_last_error;
}
// Allocations, products and launches, which may block (a full launch queue, a device that is asked for memory): Python's other threads go on.
template <typename F> auto unlocked(const F& work) {
  const py::gil_scoped_release release;
  return work();
}
PyTypeObject *tensor_type = nullptr, *parameter_type = nullptr;
bool exact(PyObject* o) { return o && (Py_TYPE(o) == tensor_type || Py_TYPE(o) == parameter_type); }
// The tensor behind an object that is exactly a Tensor or a Parameter; undefined otherwise.
Tensor tensor_of(PyObject* o) { return exact(o) ? THPVariable_Unpack(o) : Tensor(); }
Tensor tensor_of(const py::handle& o) { return tensor_of(o.ptr()); }

// ---- modules
struct Names {
  PyObject *forward, *hooks[4], *modules, *parameters, *weight, *bias, *training, *eps;
  static PyObject* of(const char* s) { return PyUnicode_InternFromString(s); }
  Names()
      : forward(of("forward")), hooks{of("_forward_hooks"), of("_forward_pre_hooks"), of("_backward_hooks"), of("_backward_pre_hooks")},
        modules(of("_modules")), parameters(of("_parameters")), weight(of("weight")), bias(of("bias")), training(of("training")),
        eps(of("variance_epsilon")) {}
};
const Names& names() {
  static const Names n;
  return n;
}
// The attributes of a module that is exactly of a class, has that class's forward and no hook of its own; null otherwise (borrowed).
PyObject* untouched(PyObject* m, PyObject* cls) {
  if (!m || reinterpret_cast<PyObject*>(Py_TYPE(m)) != cls) return nullptr;
  py::object dict = py::reinterpret_steal<py::object>(PyObject_GenericGetDict(m, nullptr));
  if (!dict || !PyDict_Check(dict.ptr())) { PyErr_Clear(); return nullptr; }
  PyObject* d = dict.ptr();                        // the module holds it
  if (PyDict_GetItem(d, names().forward)) return nullptr;
  for (PyObject* h : names().hooks) {
    PyObject* v = PyDict_GetItem(d, h);
    if (!v || !PyDict_Check(v) || PyDict_Size(v) != 0) return nullptr;
  }
  return d;
}
PyObject* item(PyObject* attributes, PyObject* table, const char* name) {
  PyObject* t = attributes ? PyDict_GetItem(attributes, table) : nullptr;
  return t && PyDict_Check(t) ? PyDict_GetItemString(t, name) : nullptr;
}
PyObject* child(PyObject* attributes, const char* name) { return item(attributes, names().modules, name); }
Tensor weight_of(PyObject* attributes) { return tensor_of(item(attributes, names().parameters, "weight")); }
Tensor linear_weight(PyObject* m, PyObject* cls) {
  PyObject* d = untouched(m, cls);
  if (!d || item(d, names().parameters, "bias") != Py_None) return Tensor();
  return weight_of(d);
}

struct Norm { Tensor w; double eps = 0.0; };
Norm norm_of(PyObject* m, PyObject* cls) {
  Norm n;
  PyObject* d = untouched(m, cls);
  PyObject* e = d ? PyDict_GetItem(d, names().eps) : nullptr;
  if (!e || !PyFloat_Check(e)) return n;
  n.eps = PyFloat_AsDouble(e);
  n.w = weight_of(d);
  return n;
}

struct Layer {
  Norm in, post, q_norm, k_norm;
  Tensor q, k, v, o, gate, up, down;
  int64_t hidden = 0;
};
constexpr int64_t kHead = 128, kMaxHidden = 12288;

bool matrix(const Tensor& w, int64_t rows, int64_t cols, c10::Device dev) {
  return bf16(w, dev) && w.dim() == 2 && (rows < 0 ? w.size(0) > 0 : w.size(0) == rows) && w.size(1) == cols;
}
bool vector(const Norm& n, int64_t size, c10::Device dev) { return bf16(n.w, dev) && n.w.dim() == 1 && n.w.size(0) == size; }

// `classes`: decoder layer, attention, feed-forward, activation, norm, linear.
py::object layers(const py::tuple& modules, const py::tuple& classes) {
  if (!quiet() || classes.size() != 6) return py::none();
  PyObject* cls[6];
  for (int i = 0; i < 6; ++i) cls[i] = PyTuple_GET_ITEM(classes.ptr(), i);
  py::list out;
  for (const py::handle& m : modules) {
    PyObject* d = untouched(m.ptr(), cls[0]);
    PyObject* attn = d ? untouched(child(d, "self_attn"), cls[1]) : nullptr;
    PyObject* mlp = d ? untouched(child(d, "mlp"), cls[2]) : nullptr;
    if (!attn || !mlp || PyDict_GetItem(attn, names().training) != Py_False || !untouched(child(mlp, "act_fn"), cls[3])) return py::none();
    auto l = std::make_shared<Layer>();
    l->in = norm_of(child(d, "input_layernorm"), cls[4]);
    l->post = norm_of(child(d, "post_attention_layernorm"), cls[4]);
    l->q_norm = norm_of(child(attn, "q_norm"), cls[4]);
    l->k_norm = norm_of(child(attn, "k_norm"), cls[4]);
    if (!l->in.w.defined() || l->in.w.dim() != 1 || !l->in.w.is_cuda() || l->q_norm.eps != l->k_norm.eps) return py::none();
    const c10::Device dev = l->in.w.device();
    const int64_t hidden = l->hidden = l->in.w.size(0);
    l->q = linear_weight(child(attn, "q_proj"), cls[5]);
    l->k = linear_weight(child(attn, "k_proj"), cls[5]);
    l->v = linear_weight(child(attn, "v_proj"), cls[5]);
    l->o = linear_weight(child(attn, "o_proj"), cls[5]);
    l->gate = linear_weight(child(mlp, "gate_proj"), cls[5]);
    l->up = linear_weight(child(mlp, "up_proj"), cls[5]);
    l->down = linear_weight(child(mlp, "down_proj"), cls[5]);
    if (hidden <= 0 || hidden % 2 || hidden > kMaxHidden || !vector(l->in, hidden, dev) || !vector(l->post, hidden, dev) ||
        !vector(l->q_norm, kHead, dev) || !vector(l->k_norm, kHead, dev) || !matrix(l->q, -1, hidden, dev) || !matrix(l->k, -1, hidden, dev) ||
        !matrix(l->gate, -1, hidden, dev))
      return py::none();
    const int64_t heads = l->q.size(0), kv = l->k.size(0), ffn = l->gate.size(0);
    if (heads % kHead || kv % kHead || ffn % 2 || !matrix(l->v, kv, hidden, dev) || !matrix(l->o, hidden, heads, dev) ||
        !matrix(l->up, ffn, hidden, dev) || !matrix(l->down, hidden, ffn, dev))
      return py::none();
    out.append(py::cast(l));
  }
  return std::move(out);
}

// ---- launches
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
bool rows_fit(const Tensor& x) { return x.dim() == 3 && x.numel() > 0 && x.size(0) * x.size(1) < (1ll << 31); }

// x w^T for rows [batch, tokens, features]: the product that at::linear comes to, without its detour over shapes (6.5 -> 4 us a call)
Tensor product(const Tensor& x, const Tensor& w) {
  const int64_t b = x.size(0), s = x.size(1);
  return at::mm(x.view({b * s, x.size(2)}), w.t()).view({b, s, w.size(0)});
}

// (x + branch, norm(x + branch))
std::pair<Tensor, Tensor> add_norm_of(const Tensor& x, const Tensor& branch, const Norm& n) {
  const int64_t hidden = x.size(-1);
  Tensor x_new = branch.defined() ? at::empty_like(x) : x, h = at::empty_like(x);
  check(lib.msa_add_rmsnorm(x.const_data_ptr(), branch.defined() ? branch.const_data_ptr() : nullptr, n.w.const_data_ptr(), (float)n.eps,
                            (int32_t)(x.numel() / hidden), (int32_t)hidden, branch.defined() ? x_new.data_ptr() : nullptr, h.data_ptr(), stream_of(x)),
        "msa_add_rmsnorm");
  return {x_new, h};
}
// operand of a fused call: None is allowed where `optional`
bool operand(const py::handle& o, c10::Device dev, const Tensor& like, bool optional, Tensor& out) {
  if (optional && o.is_none()) return true;
  out = tensor_of(o);
  return bf16(out, dev) && out.sizes() == like.sizes();
}

py::object add_norm(const py::object& x_, const py::object& branch_, const py::object& norm, const py::object& cls) {
  const Norm n = norm_of(norm.ptr(), cls.ptr());
  const Tensor x = tensor_of(x_);
  Tensor branch;
  if (!quiet() || !x.defined() || !x.is_cuda() || !bf16(x, x.device()) || !rows_fit(x) || x.size(2) % 2 || x.size(2) > kMaxHidden ||
      !operand(branch_, x.device(), x, true, branch) || !vector(n, x.size(2), x.device()))
    return py::none();
  const auto r = unlocked([&] {
    const c10::cuda::CUDAGuard guard(x.device());
    return add_norm_of(x, branch, n);
  });
  return py::make_tuple(r.first, r.second);
}

// (stream, normed rows, q, k, v): rows [batch, tokens, features], q and k normed and turned, all three as [batch, heads, tokens, 128]
py::object front(const Layer& l, const py::object& x_, const py::object& branch_, const py::object& cos_, const py::object& sin_) {
  const Tensor x = tensor_of(x_), cos = tensor_of(cos_), sin = tensor_of(sin_);
  const c10::Device dev = l.q.device();
  Tensor branch;
  if (!quiet() || !bf16(x, dev) || !rows_fit(x) || x.size(2) != l.hidden || !operand(branch_, dev, x, true, branch) || !bf16(cos, dev) || !bf16(sin, dev) ||
      cos.sizes() != sin.sizes() || cos.dim() != 3 || cos.size(2) != kHead || cos.size(1) != x.size(1) || (cos.size(0) != x.size(0) && cos.size(0) != 1))
    return py::none();
  const auto r = unlocked([&] {
    const c10::cuda::CUDAGuard guard(dev);
    auto [x_new, h] = add_norm_of(x, branch, l.in);
    const Tensor q0 = product(h, l.q), k0 = product(h, l.k), v = product(h, l.v);
    Tensor q = at::empty_like(q0), k = at::empty_like(k0);
    const int64_t heads = l.q.size(0), kv = l.k.size(0);
    check(lib.msa_heads_norm_rope(q0.const_data_ptr(), heads, k0.const_data_ptr(), kv, (int32_t)(x.size(0) * x.size(1)), (int32_t)(heads / kHead),
                                  (int32_t)(kv / kHead), (int32_t)kHead, l.q_norm.w.const_data_ptr(), l.k_norm.w.const_data_ptr(), (float)l.q_norm.eps,
                                  cos.const_data_ptr(), sin.const_data_ptr(), (int32_t)(cos.size(0) * cos.size(1)), q.data_ptr(), k.data_ptr(), stream_of(x)),
          "msa_heads_norm_rope");
    auto heads_of = [&](const Tensor& t) { return t.view({x.size(0), x.size(1), -1, kHead}).transpose(1, 2); };
    return std::array<Tensor, 5>{x_new, h, heads_of(q), heads_of(k), heads_of(v)};
  });
  return py::make_tuple(r[0], r[1], r[2], r[3], r[4]);
}

// (stream with the attention's branch, the feed-forward's branch)
py::object back(const Layer& l, const py::object& x_, const py::object& attn_) {
  const Tensor x = tensor_of(x_), attn = tensor_of(attn_);
  const c10::Device dev = l.q.device();
  if (!quiet() || !bf16(x, dev) || !rows_fit(x) || x.size(2) != l.hidden || !bf16(attn, dev) || attn.dim() != 3 || attn.size(0) != x.size(0) ||
      attn.size(1) != x.size(1) || attn.size(2) != l.o.size(1))
    return py::none();
  const auto r = unlocked([&] {
    const c10::cuda::CUDAGuard guard(dev);
    auto [x_new, h] = add_norm_of(x, product(attn, l.o), l.post);
    const Tensor gate = product(h, l.gate), up = product(h, l.up);
    Tensor act = at::empty_like(gate);
    const int64_t ffn = l.gate.size(0);
    check(lib.msa_silu_mul_parts(gate.const_data_ptr(), ffn, up.const_data_ptr(), ffn, (int32_t)(x.size(0) * x.size(1)), (int32_t)ffn, act.data_ptr(),
                                 stream_of(x)),
          "msa_silu_mul_parts");
    return std::pair<Tensor, Tensor>{x_new, product(act, l.down)};
  });
  return py::make_tuple(r.first, r.second);
}

// cos and sin of positions [batch, tokens] (int64): bf16 [batch, tokens, 2 * frequencies]
py::object angles(const py::object& positions_, const py::object& inv_freq_, double scaling) {
  const Tensor pos = tensor_of(positions_), freq = tensor_of(inv_freq_);
  if (!quiet() || !pos.defined() || !pos.is_cuda() || !takes(pos, at::kLong, pos.device()) || !takes(freq, at::kFloat, pos.device()) || pos.dim() != 2 ||
      freq.dim() != 1 || pos.numel() == 0 || pos.numel() >= (1ll << 31))
    return py::none();
  const auto r = unlocked([&] {
    const c10::cuda::CUDAGuard guard(pos.device());
    const Tensor both = at::empty({2, pos.size(0), pos.size(1), 2 * freq.size(0)}, pos.options().dtype(at::kBFloat16));
    Tensor cos = both.select(0, 0), sin = both.select(0, 1);
    check(lib.msa_rope_table(static_cast<const int64_t*>(pos.const_data_ptr()), static_cast<const float*>(freq.const_data_ptr()), (int32_t)pos.numel(),
                             (int32_t)freq.size(0), (float)scaling, cos.data_ptr(), sin.data_ptr(), stream_of(pos)),
          "msa_rope_table");
    return std::pair<Tensor, Tensor>{cos, sin};
  });
  return py::make_tuple(r.first, r.second);
}

// The attention of one token per sequence over its compact cache, which takes the token in: q, k, v [batch, heads, 1, 128].
// (rows [batch, 1, features], entries per sequence, the caller's lengths), both one more.
py::object decode(const py::object& q_, const py::object& k_, const py::object& v_, const py::object& k_store_, const py::object& v_store_,
                  const py::object& start_, const py::object& len_, const py::object& lengths_, int64_t n_splits) {
  const Tensor q4 = tensor_of(q_), k4 = tensor_of(k_), v4 = tensor_of(v_), ks = tensor_of(k_store_), vs = tensor_of(v_store_), start = tensor_of(start_),
               len = tensor_of(len_), lengths = tensor_of(lengths_);
  if (!quiet() || !q4.defined() || !q4.is_cuda() || q4.dim() != 4 || q4.size(2) != 1 || !k4.defined() || !v4.defined() || k4.dim() != 4 || v4.dim() != 4)
    return py::none();
  const c10::Device dev = q4.device();
  const Tensor q = q4.select(2, 0), k = k4.select(2, 0), v = v4.select(2, 0);
  const int64_t b = q.size(0), hq = q.size(1), d = q.size(2), hkv = k.size(1);
  if (!bf16(q, dev) || !bf16(k, dev) || !bf16(v, dev) || !bf16(ks, dev) || !bf16(vs, dev) || d != kHead || b == 0 || hkv == 0 || hq % hkv ||
      k.sizes() != v.sizes() || k.size(0) != b || k.size(2) != d || k4.size(2) != 1 || ks.dim() != 4 || ks.sizes() != vs.sizes() || ks.size(0) != b ||
      ks.size(1) != hkv || ks.size(3) != d || !takes(start, at::kInt, dev) || !takes(len, at::kInt, dev) || start.numel() != b || len.numel() != b ||
      !lengths.defined() || !plain_key_set(lengths) || lengths.device() != dev || n_splits < 1)
    return py::none();
  const auto r = unlocked([&] {
    const c10::cuda::CUDAGuard guard(dev);
    Tensor out = at::empty({b, 1, hq * d}, q.options()), space;
    const int64_t need = lib.msa_decode_workspace_bytes((int32_t)b, (int32_t)hq, (int32_t)d, (int32_t)n_splits);
    if (need > 0) space = at::empty({need / 4}, q.options().dtype(at::kFloat));
    const bool counts = takes(lengths, at::kLong, dev) && lengths.numel() == b && lengths.dim() == 1 && len.dim() == 1;
    const Tensor next_len = counts ? at::empty_like(len) : Tensor(), next_lengths = counts ? at::empty_like(lengths) : Tensor();
    check(lib.msa_sparse_decode_attn_next(q.const_data_ptr(), MSA_BF16, ks.data_ptr(), vs.data_ptr(), ks.stride(0), ks.stride(1),
                                     static_cast<const int32_t*>(start.const_data_ptr()), static_cast<const int32_t*>(len.const_data_ptr()),
                                     k.const_data_ptr(), v.const_data_ptr(), (int32_t)b, (int32_t)hq, (int32_t)hkv, (int32_t)d,
                                     (float)(1.0 / std::sqrt((double)d)), out.data_ptr(), need > 0 ? space.data_ptr() : nullptr, need > 0 ? need : 0,
                                     (int32_t)n_splits, counts ? static_cast<const int64_t*>(lengths.const_data_ptr()) : nullptr,
                                     counts ? static_cast<int32_t*>(next_len.data_ptr()) : nullptr,
                                     counts ? static_cast<int64_t*>(next_lengths.data_ptr()) : nullptr, stream_of(q)),
          "msa_sparse_decode_attn");
    return counts ? std::array<Tensor, 3>{out, next_len, next_lengths} : std::array<Tensor, 3>{out, len.add(1), lengths.add(1)};
  });
  return py::make_tuple(r[0], r[1], r[2]);
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  tensor_type = reinterpret_cast<PyTypeObject*>(THPVariableClass);
  py::object parameter = py::module_::import("torch.nn.parameter").attr("Parameter");
  parameter_type = reinterpret_cast<PyTypeObject*>(parameter.release().ptr());
  py::class_<Layer, std::shared_ptr<Layer>>(m, "Layer");
  m.def("bind", &bind);
  m.def("layers", &layers);
  m.def("add_norm", &add_norm);
  m.def("front", &front);
  m.def("back", &back);
  m.def("angles", &angles);
  m.def("decode", &decode);
}
