// Autograd functions of the bf16 operators, in C++ over the C entry points of libsavanna_b200.so.
//
// A training step of a small model is a few hundred launches of a few microseconds each; with the functions in Python (argument checks,
// ctypes calls, an autograd.Function forward and backward per operator) the host needed 80 to 150 us for a forward and backward whose
// kernels take 50.  Here the same allocations and the same entry points are called from one C++ frame, the backward runs in the engine
// without the interpreter lock, and a gated MLP or a norm with its projection is one node instead of four or two.
// Forward and backward, us, Python -> here: gated Hyena-MR [3 x 777 x 512] 120 -> 77 (an operator that does nothing costs 53 through the engine),
// gated MLP [999 x 1024] 329 -> 130, a step of a four-operator model, 2 x 1024 tokens of 256 channels, 4181 -> 2200.
// Python keeps what decides (ops/cuda_ops.py: shapes, types, which operator), and the oracle.
//
// Nothing is cached between calls but the entry points (entries.h) and the address of the per-device status word.
#include <dlfcn.h>

#include <atomic>
#include <mutex>
#include <sstream>

#include <c10/cuda/CUDAException.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <nvtx3/nvToolsExt.h>
#include <torch/csrc/autograd/graph_task.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/extension.h>

#include "entries.h"

namespace {

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
typedef std::optional<Tensor> OptTensor;

constexpr auto BF16 = at::kBFloat16;
constexpr auto F32 = at::kFloat;

// ------------------------------------------------------------------------------------ the library's entry points
#define SB_ENTRIES(X) \
  X(sb_gemm_bf16) X(sb_gemm_last_error_detail) X(sb_attn_last_encode_result) X(sb_colsum) X(sb_rmsnorm_fwd) X(sb_rmsnorm_bwd_blocks) \
  X(sb_rmsnorm_bwd) X(sb_glu_fwd) X(sb_glu_bwd) X(sb_ce_fwd) X(sb_ce_bwd) X(sb_dwconv_fwd) X(sb_dwconv_fwd_taps) X(sb_dwconv_bwd) \
  X(sb_se_fwd) X(sb_se_fwd_taps) X(sb_se_bwd) X(sb_mr_fwd) X(sb_mr_bwd) X(sb_mr_tc_fwd) X(sb_mr_tc_bwd) X(sb_mr_umma_fwd) X(sb_mr_umma_bwd) \
  X(sb_li_fwd_tiled) \
  X(sb_li_bwd_tiled_chunk) X(sb_li_bwd_tiled) X(sb_attn_fwd) X(sb_attn_bwd) X(sb_attn_rope)

struct {
#define SB_DECLARE(name) decltype(&::name) name = nullptr;
  SB_ENTRIES(SB_DECLARE)
#undef SB_DECLARE
} L;

PyObject* g_ops = nullptr;                 // ops.cuda_ops: guarded allocations and status words
std::atomic<long long> g_launches{0};
std::atomic<bool> g_guarded{false}, g_nvtx{false};

void load(const std::string& path, py::object ops) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw std::runtime_error(std::string("cannot load ") + path + ": " + dlerror());
#define SB_RESOLVE(name)                                          \
  *reinterpret_cast<void**>(&L.name) = dlsym(h, #name);           \
  if (!L.name) throw std::runtime_error("no entry point " #name " in " + path);
  SB_ENTRIES(SB_RESOLVE)
#undef SB_RESOLVE
  g_ops = ops.release().ptr();             // lives as long as the process
}

// What was handed to an entry point that refused it: name, shape, strides, address.
std::string layouts(std::initializer_list<std::pair<const char*, const Tensor*>> ts) {
  std::ostringstream s;
  for (const auto& [name, t] : ts) {
    s << (s.tellp() > 0 ? ", " : "") << name;
    if (t->defined()) s << t->sizes() << '/' << t->strides() << " at " << t->const_data_ptr();
    else s << " none";
  }
  return s.str();
}
// One call of an entry point: NVTX range while the profiler wants one, launch count; its error code.
template <class... A, class... B>
int run(const char* name, int launches, int (*fn)(A...), B... args) {
  const bool mark = g_nvtx.load(std::memory_order_relaxed);
  if (mark) nvtxRangePushA(name);
  const int rc = fn(args...);
  if (mark) nvtxRangePop();
  if (rc == 0) g_launches.fetch_add(launches, std::memory_order_relaxed);
  return rc;
}
#define SB_RUN(name, launches, ...) run(#name, launches, L.name, __VA_ARGS__)
#define SB_CALL(name, launches, ...)                                                                                     \
  do {                                                                                                                   \
    const int rc_ = SB_RUN(name, launches, __VA_ARGS__);                                                                 \
    TORCH_CHECK(rc_ == 0, "savanna_b200 kernel `", #name + 3, "` rejected its arguments or failed to launch (code ", rc_, ")"); \
  } while (0)

cudaStream_t stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

// ------------------------------------------------------------------------------------ tensors
Tensor alloc(at::IntArrayRef shape, at::ScalarType dtype, at::Device device) {
  if (g_guarded.load(std::memory_order_relaxed)) {         // debug aid: the buffer inside a larger one with margins
    py::gil_scoped_acquire gil;
    py::tuple s(shape.size());
    for (size_t i = 0; i < shape.size(); ++i) s[i] = shape[i];
    py::object t = py::handle(g_ops).attr("_alloc")(s, py::arg("dtype") = py::cast(dtype), py::arg("device") = py::cast(device));
    return t.cast<Tensor>();
  }
  return at::empty(shape, at::TensorOptions().dtype(dtype).device(device));
}
Tensor alloc_like(const Tensor& t) { return alloc(t.sizes(), t.scalar_type(), t.device()); }

const void* ptr(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }
void* out(const Tensor& t) { return t.defined() ? t.mutable_data_ptr() : nullptr; }
const long long* i64(const Tensor& t) { return static_cast<const long long*>(ptr(t)); }
const float* f32(const Tensor& t) { return static_cast<const float*>(ptr(t)); }
float* f32o(const Tensor& t) { return static_cast<float*>(out(t)); }
// Zeros of a whole buffer on the current stream: a memset instead of a fill kernel by way of the dispatcher (a backward of Hyena-MR has
// two, one of a small four-operator model thirteen).
Tensor cleared(Tensor t) {
  if (t.numel() > 0) C10_CUDA_CHECK(cudaMemsetAsync(out(t), 0, t.nbytes(), stream()));
  return t;
}
Tensor zeros(at::IntArrayRef shape, at::ScalarType dtype, at::Device device) { return cleared(alloc(shape, dtype, device)); }
// Operands that may be absent reach Function::apply as empty optionals (it refuses undefined tensors) and have no edge then: the edges
// behind them move up.
Tensor opt(const OptTensor& t) { return t.has_value() ? *t : Tensor(); }

Tensor contiguous(const Tensor& t) { return t.is_contiguous() ? t : t.contiguous(); }
bool on16(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.const_data_ptr()) % 16 == 0; }
// contiguous and on a 16-byte boundary (a view into the middle of another tensor need not be)
Tensor aligned(const Tensor& t) {
  Tensor c = contiguous(t);
  return on16(c) ? c : c.clone();
}
Tensor aligned(const OptTensor& t) { return t.has_value() ? aligned(*t) : Tensor(); }
Tensor f32c(const Tensor& t) {
  Tensor d = t.detach();
  if (d.scalar_type() != F32) d = d.to(F32);
  return contiguous(d);
}
// [.., N] -> [rows, N] as the GEMM reads it: unit inner stride, rows on 16-byte boundaries
Tensor rows(const Tensor& x) {
  Tensor r = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  if (r.stride(1) != 1 || r.stride(0) % 8 || !on16(r)) r = r.contiguous();
  return r;
}
Tensor rows_contiguous(const Tensor& x) { return contiguous(x.dim() == 2 ? x : x.reshape({-1, x.size(-1)})); }
std::vector<int64_t> with_last(at::IntArrayRef shape, int64_t n) {
  std::vector<int64_t> s(shape.begin(), shape.end());
  s.back() = n;
  return s;
}

unsigned int* status_word(at::Device device) {
  static std::mutex m;
  static unsigned int* word[64] = {nullptr};
  const int i = device.index() < 0 ? 0 : device.index();
  TORCH_CHECK(i < 64, "device index ", i);
  {
    std::lock_guard<std::mutex> lock(m);
    if (word[i]) return word[i];
  }
  py::gil_scoped_acquire gil;
  void* t = py::handle(g_ops).attr("status_word")(py::cast(device)).cast<Tensor>().mutable_data_ptr();    // kept by cuda_ops
  unsigned int* p = static_cast<unsigned int*>(t);
  std::lock_guard<std::mutex> lock(m);
  return word[i] = p;
}

// The functions of this file know nothing of functorch's wrappers (forward-mode tangents are refused by Function::apply itself).
void no_transforms() {
  TORCH_CHECK(!c10::impl::tls_is_dispatch_key_included(c10::DispatchKey::FuncTorchDynamicLayerFrontMode),
              "the CUDA operators of savanna_b200 do not support functorch transforms (vmap, grad, jvp)");
}

// ------------------------------------------------------------------------------------ GEMM
// o[M,N] = A B^T (+bias) (+residual) (+o); a_mn / b_mn: the operand is stored transposed
void gemm(const Tensor& a, const Tensor& b, const Tensor& o, bool a_mn, bool b_mn, const Tensor& bias = Tensor(), bool accumulate = false,
          const Tensor& residual = Tensor()) {
  const int M = o.size(0), N = o.size(1), K = a_mn ? a.size(0) : a.size(1);
  for (const Tensor* t : {&a, &b, &o})
    TORCH_CHECK_VALUE(t->dim() == 2 && t->stride(1) == 1 && t->scalar_type() == BF16, "gemm operands must be 2-D bf16 with unit inner stride");
  TORCH_CHECK_VALUE(!residual.defined() || (residual.dim() == 2 && residual.stride(1) == 1 && residual.scalar_type() == BF16 &&
                                            residual.size(0) == M && residual.size(1) == N),
                    "gemm residual must be a [M, N] bf16 matrix with unit inner stride");
  const int rc = SB_RUN(sb_gemm_bf16, 1, ptr(a), ptr(b), out(o), ptr(bias), ptr(residual), M, N, K, (int)a.stride(0), (int)b.stride(0),
                        (int)o.stride(0), residual.defined() ? (int)residual.stride(0) : 0, (int)a_mn, (int)b_mn, (int)accumulate,
                        status_word(o.device()), 0, stream());
  if (rc) {
    const int detail = L.sb_gemm_last_error_detail();
    TORCH_CHECK(false, "gemm_bf16 failed (code ", rc, ", operand ", detail >> 16, ", driver result ", detail & 0xffff, "): M=", M, " N=", N, " K=", K,
                " a_mn=", a_mn, " b_mn=", b_mn, " ", layouts({{"a", &a}, {"b", &b}, {"out", &o}, {"residual", &residual}}));
  }
}

Tensor colsum(const Tensor& g2, at::ScalarType dtype) {
  if (g2.size(1) % 8) return g2.to(F32).sum(0).to(dtype);
  Tensor o = zeros({g2.size(1)}, F32, g2.device());
  SB_CALL(sb_colsum, 1, ptr(g2), f32o(o), (int)g2.size(0), (int)g2.size(1), stream());
  return o.to(dtype);
}

// dW = dY^T X; added by the GEMM's epilogue straight into the parameter's gradient where that lives in a persistent flat buffer
// (`sink`: the parameter, marked _fuse_grad_accum), else returned
Tensor weight_grad(const Tensor& g2, const Tensor& x2, const Tensor& w, const Tensor& sink) {
  if (sink.defined()) {
    const Tensor& tgt = sink.grad();
    if (tgt.defined() && tgt.scalar_type() == BF16 && tgt.is_contiguous() && tgt.sizes() == w.sizes()) {
      gemm(g2, x2, tgt, true, true, Tensor(), true);
      return Tensor();
    }
  }
  Tensor gw = alloc(w.sizes(), BF16, w.device());
  gemm(g2, x2, gw, true, true);
  return gw;
}
Tensor input_grad(const Tensor& g2, const Tensor& w) {
  Tensor gx = alloc({g2.size(0), w.size(1)}, BF16, g2.device());
  gemm(g2, w, gx, false, true);
  return gx;
}
Tensor sink(AutogradContext* ctx, const char* key) {
  auto it = ctx->saved_data.find(key);
  return it == ctx->saved_data.end() ? Tensor() : it->second.toTensor();
}

// Intermediate results of a node that joins several operators.  What save_for_backward keeps lives until the whole node has run; these
// are let go one by one, at their last use in the backward, as they would be between nodes of their own (unless the graph is kept).
// Hooks and version checks are those of any saved tensor.  Only made when there will be a backward (`train`).
struct Kept : torch::CustomClassHolder { std::vector<torch::autograd::SavedVariable> v; };
void keep(AutogradContext* ctx, bool train, std::initializer_list<Tensor> ts) {
  if (!train) return;
  auto k = c10::make_intrusive<Kept>();
  for (const Tensor& t : ts) k->v.emplace_back(t, /*is_output=*/false);
  ctx->saved_data["kept"] = c10::IValue::make_capsule(std::move(k));
}
struct Taker {
  Kept* k;
  bool hold = torch::autograd::get_current_graph_task_keep_graph();
  explicit Taker(AutogradContext* ctx) : k(static_cast<Kept*>(ctx->saved_data["kept"].toCapsule().get())) {}
  ~Taker() { for (size_t i = 0; !hold && i < k->v.size(); ++i) k->v[i].reset_data(); }
  Tensor operator()(int i) {
    Tensor t = k->v[i].unpack();
    if (!hold) k->v[i].reset_data();
    return t;
  }
};
bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t && t->requires_grad()) return true;
  return false;
}
const Tensor* given(const OptTensor& t) { return t.has_value() ? &*t : nullptr; }

struct Linear : Function<Linear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& bias, const OptTensor& residual, bool fuse) {
    Tensor x2 = rows(x), o = alloc({x2.size(0), w.size(0)}, BF16, x.device());
    gemm(x2, w, o, false, false, opt(bias), false, residual.has_value() ? rows(*residual) : Tensor());
    ctx->save_for_backward({x2, w});
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->saved_data["bias"] = bias.has_value();
    ctx->saved_data["res"] = residual.has_value();
    if (fuse) ctx->saved_data["sink"] = w;
    return o.view(with_last(x.sizes(), w.size(0)));
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &w = s[1], &gy = g[0];
    const bool bias = ctx->saved_data["bias"].toBool();
    Tensor g2 = rows(gy), gx, gw, gb, gr;
    if (ctx->needs_input_grad(0)) gx = input_grad(g2, w).view(ctx->saved_data["shape"].toIntVector());
    if (ctx->needs_input_grad(1)) gw = weight_grad(g2, x2, w, sink(ctx, "sink"));
    if (bias && ctx->needs_input_grad(2)) gb = colsum(g2, gy.scalar_type());
    if (ctx->saved_data["res"].toBool() && ctx->needs_input_grad(2 + bias)) gr = gy;
    return {gx, gw, gb, gr, Tensor()};
  }
};

// ------------------------------------------------------------------------------------ RMSNorm
struct Norm { Tensor x2, w, a, y; };
Norm norm_fwd(const Tensor& x, const Tensor& w, double eps, int64_t form) {
  Norm n;
  n.x2 = rows_contiguous(x);
  n.w = contiguous(w);
  n.y = alloc_like(n.x2);
  n.a = alloc({n.x2.size(0)}, F32, x.device());
  SB_CALL(sb_rmsnorm_fwd, 1, ptr(n.x2), ptr(n.w), out(n.y), f32o(n.a), (int)n.x2.size(0), (int)n.x2.size(1), (float)eps, (int)form, stream());
  return n;
}
std::pair<Tensor, Tensor> norm_bwd(const Tensor& x2, const Tensor& w, const Tensor& a, const Tensor& gy, const Tensor& gres, double eps,
                                   int64_t form) {
  const int T = x2.size(0), D = x2.size(1);
  Tensor g2 = contiguous(gy.reshape({T, D})), r2 = gres.defined() ? contiguous(gres.reshape({T, D})) : Tensor();
  Tensor dx = alloc_like(x2), dw = alloc({D}, BF16, x2.device()),
         partial = alloc({(int64_t)L.sb_rmsnorm_bwd_blocks(T, D) * D}, F32, x2.device());
  SB_CALL(sb_rmsnorm_bwd, 2, ptr(x2), ptr(w), ptr(g2), f32(a), ptr(r2), out(dx), out(dw), f32o(partial), T, D, (float)eps, (int)form, stream());
  return {dx, dw};
}
void save_norm(AutogradContext* ctx, const Tensor& x, double eps, int64_t form) {
  ctx->saved_data["eps"] = eps;
  ctx->saved_data["form"] = form;
  ctx->saved_data["shape"] = x.sizes().vec();
}
// (dx in the input's shape, dw)
std::pair<Tensor, Tensor> saved_norm_bwd(AutogradContext* ctx, const Tensor& x2, const Tensor& w, const Tensor& a, const Tensor& gy,
                                         const Tensor& gres) {
  auto d = norm_bwd(x2, w, a, gy, gres, ctx->saved_data["eps"].toDouble(), ctx->saved_data["form"].toInt());
  return {d.first.view(ctx->saved_data["shape"].toIntVector()), d.second};
}

struct RmsNorm : Function<RmsNorm> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps, int64_t form) {
    Norm n = norm_fwd(x, w, eps, form);
    ctx->save_for_backward({n.x2, n.w, n.a});
    save_norm(ctx, x, eps, form);
    return n.y.view(x.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    auto d = saved_norm_bwd(ctx, s[0], s[1], s[2], g[0], Tensor());
    return {d.first, d.second, Tensor(), Tensor()};
  }
};

// (norm(x), x): the second output carries x down the residual branch; the gradient arriving there is added inside the norm's backward
// kernel instead of by a separate accumulation kernel.
struct RmsNormResidual : Function<RmsNormResidual> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, double eps, int64_t form) {
    Norm n = norm_fwd(x, w, eps, form);
    ctx->save_for_backward({n.x2, n.w, n.a});
    save_norm(ctx, x, eps, form);
    ctx->set_materialize_grads(false);
    return {n.y.view(x.sizes()), x.view_as(x)};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    if (!g[0].defined()) return {g[1], Tensor(), Tensor(), Tensor()};
    const variable_list s = ctx->get_saved_variables();
    auto d = saved_norm_bwd(ctx, s[0], s[1], s[2], g[0], g[1]);
    return {d.first, d.second, Tensor(), Tensor()};
  }
};

// (linear(norm(x)), x) as one node
struct NormLinear : Function<NormLinear> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wn, double eps, int64_t form, const Tensor& w,
                               const OptTensor& bias, bool fuse, bool train) {
    Norm n = norm_fwd(x, wn, eps, form);
    Tensor y2 = rows(n.y), o = alloc({y2.size(0), w.size(0)}, BF16, x.device());
    gemm(y2, w, o, false, false, opt(bias));
    ctx->save_for_backward({n.x2, n.w, n.a, w});
    keep(ctx, train, {y2});
    save_norm(ctx, x, eps, form);
    ctx->saved_data["bias"] = bias.has_value();
    if (fuse) ctx->saved_data["sink"] = w;
    ctx->set_materialize_grads(false);
    return {o.view(with_last(x.sizes(), w.size(0))), x.view_as(x)};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    Taker kept(ctx);
    if (!g[0].defined()) return {g[1], Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor(), Tensor()};
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &wn = s[1], &a = s[2], &w = s[3];
    Tensor y2 = kept(0), g2 = rows(g[0]), gx, gwn, gw, gb;
    if (ctx->needs_input_grad(2)) gw = weight_grad(g2, y2, w, sink(ctx, "sink"));
    y2.reset();
    if (ctx->needs_input_grad(0) || ctx->needs_input_grad(1)) std::tie(gx, gwn) = saved_norm_bwd(ctx, x2, wn, a, input_grad(g2, w), g[1]);
    if (ctx->saved_data["bias"].toBool() && ctx->needs_input_grad(3)) gb = colsum(g2, g[0].scalar_type());
    return {gx, gwn, Tensor(), Tensor(), gw, gb, Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------ gated activation, gated MLP
struct Glu : Function<Glu> {
  static Tensor forward(AutogradContext* ctx, const Tensor& ab, int64_t act) {
    Tensor ab2 = rows_contiguous(ab);
    const int64_t T = ab2.size(0), F = ab2.size(1) / 2;
    Tensor h = alloc({T, F}, BF16, ab.device());
    SB_CALL(sb_glu_fwd, 1, ptr(ab2), out(h), (long long)T, (int)F, (int)act, stream());
    ctx->save_for_backward({ab2});
    ctx->saved_data["act"] = act;
    ctx->saved_data["shape"] = ab.sizes().vec();
    return h.view(with_last(ab.sizes(), F));
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor& ab2 = s[0];
    const int64_t T = ab2.size(0), F = ab2.size(1) / 2;
    Tensor g2 = contiguous(g[0].reshape({T, F})), dab = alloc_like(ab2);
    SB_CALL(sb_glu_bwd, 1, ptr(ab2), ptr(g2), out(dab), (long long)T, (int)F, (int)ctx->saved_data["act"].toInt(), stream());
    return {dab.view(ctx->saved_data["shape"].toIntVector()), Tensor()};
  }
};

// x + w3(act(a) * b) + b3 with [a | b] = w12(norm(x)) as one node.  The same kernels on the same values as the four functions one by
// one; the residual's gradient is added in the norm's backward kernel.
struct MlpGated : Function<MlpGated> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& wn, double eps, int64_t form, const Tensor& w12, const Tensor& w3,
                        const OptTensor& b3, int64_t act, bool fuse12, bool fuse3, bool train) {
    Norm n = norm_fwd(x, wn, eps, form);
    const int64_t T = n.x2.size(0), F = w12.size(0) / 2;
    Tensor y2 = rows(n.y), ab = alloc({T, 2 * F}, BF16, x.device()), h = alloc({T, F}, BF16, x.device());
    gemm(y2, w12, ab, false, false);
    SB_CALL(sb_glu_fwd, 1, ptr(ab), out(h), (long long)T, (int)F, (int)act, stream());
    Tensor h2 = rows(h), o = alloc({T, w3.size(0)}, BF16, x.device());
    gemm(h2, w3, o, false, false, opt(b3), false, rows(n.x2));
    ctx->save_for_backward({n.x2, n.w, n.a, w12, w3});
    keep(ctx, train, {y2, ab, h2});
    save_norm(ctx, x, eps, form);
    ctx->saved_data["act"] = act;
    ctx->saved_data["b3"] = b3.has_value();
    if (fuse12) ctx->saved_data["sink12"] = w12;
    if (fuse3) ctx->saved_data["sink3"] = w3;
    return o.view(x.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &x2 = s[0], &wn = s[1], &a = s[2], &w12 = s[3], &w3 = s[4];
    Taker kept(ctx);
    Tensor g2 = rows(g[0]), gx, gwn, gw12, gw3, gb3;
    // edges: x, norm weight, w12, w3, b3.  Alive at most: the gate's inputs, their gradients and the gradient of its output.
    const bool stem = ctx->needs_input_grad(0) || ctx->needs_input_grad(1), need12 = ctx->needs_input_grad(2);
    Tensor h2 = kept(2);
    if (ctx->needs_input_grad(3)) gw3 = weight_grad(g2, h2, w3, sink(ctx, "sink3"));
    h2.reset();
    if (stem || need12) {
      Tensor gh = input_grad(g2, w3), ab = kept(1), dab = alloc_like(ab);
      SB_CALL(sb_glu_bwd, 1, ptr(ab), ptr(gh), out(dab), (long long)ab.size(0), (int)(ab.size(1) / 2), (int)ctx->saved_data["act"].toInt(), stream());
      gh.reset(); ab.reset();
      Tensor y2 = kept(0), gy;
      if (need12) gw12 = weight_grad(dab, y2, w12, sink(ctx, "sink12"));
      y2.reset();
      if (stem) gy = input_grad(dab, w12);
      dab.reset();
      if (stem) std::tie(gx, gwn) = saved_norm_bwd(ctx, x2, wn, a, gy, g[0]);
    }
    if (ctx->saved_data["b3"].toBool() && ctx->needs_input_grad(4)) gb3 = colsum(g2, g[0].scalar_type());
    return {gx, gwn, Tensor(), Tensor(), gw12, gw3, gb3, Tensor(), Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------ cross entropy
struct CrossEntropy : Function<CrossEntropy> {
  static Tensor forward(AutogradContext* ctx, const Tensor& logits, const Tensor& labels) {
    const int64_t V = logits.size(-1);
    Tensor l2 = contiguous(logits.reshape({-1, V})), lab = contiguous(labels.reshape({-1}));
    const int64_t T = l2.size(0);
    Tensor loss = alloc({T}, F32, logits.device()), lse = alloc({T}, F32, logits.device());
    SB_CALL(sb_ce_fwd, 1, ptr(l2), i64(lab), f32o(loss), f32o(lse), (long long)T, (int)V, stream());
    ctx->save_for_backward({l2, lab, lse});
    ctx->saved_data["shape"] = logits.sizes().vec();
    return loss.view(labels.sizes());
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &l2 = s[0], &lab = s[1], &lse = s[2];
    Tensor gc = g[0].reshape({-1});
    if (gc.scalar_type() != F32) gc = gc.to(F32);
    gc = contiguous(gc);
    Tensor dl = alloc_like(l2);
    SB_CALL(sb_ce_bwd, 1, ptr(l2), i64(lab), f32(lse), f32(gc), out(dl), (long long)l2.size(0), (int)l2.size(1), stream());
    return {dl.view(ctx->saved_data["shape"].toIntVector()), Tensor()};
  }
};

// ------------------------------------------------------------------------------------ short convolutions
// The taps as the forward kernel reads them and the fp32 copy that the backward will: a bf16 parameter is converted by the kernel that
// reads it, not by a launch of its own.
struct Taps { Tensor in, f32; int bf16; };
Taps taps(const Tensor& w) {
  if (w.scalar_type() != BF16) { Tensor f = f32c(w); return {f, f, 0}; }
  return {contiguous(w.detach()), alloc(w.sizes(), F32, w.device()), 1};
}
at::ScalarType saved_type(AutogradContext* ctx, const char* key) { return (at::ScalarType)ctx->saved_data[key].toInt(); }

struct DwConv : Function<DwConv> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w, const OptTensor& halo, bool fast) {
    const int B = x.size(0), Ln = x.size(1), C = x.size(2), K = w.size(-1);
    Tensor xc = aligned(x), hc = aligned(halo), y = alloc_like(xc), wf;
    if (fast) {
      Taps t = taps(w);
      wf = t.f32;
      SB_CALL(sb_dwconv_fwd_taps, 1, ptr(xc), ptr(hc), ptr(t.in), t.bf16, t.bf16 ? f32o(wf) : (float*)nullptr, out(y), B, Ln, C, K, stream());
    } else {
      wf = f32c(w);
      SB_CALL(sb_dwconv_fwd, 1, ptr(xc), ptr(hc), f32(wf), out(y), B, Ln, C, K, stream());
    }
    ctx->save_for_backward({xc, wf, hc});
    ctx->saved_data["wtype"] = (int64_t)w.scalar_type();
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &xc = s[0], &wf = s[1], &hc = s[2];
    Tensor gc = aligned(g[0]), dx = alloc_like(xc), dh = hc.defined() ? alloc_like(hc) : Tensor(), dw = zeros(wf.sizes(), F32, wf.device());
    SB_CALL(sb_dwconv_bwd, 1, ptr(xc), ptr(hc), f32(wf), ptr(gc), out(dx), out(dh), f32o(dw), (int)xc.size(0), (int)xc.size(1), (int)xc.size(2),
            (int)wf.size(-1), stream());
    return {dx, dw.to(saved_type(ctx, "wtype")), dh, Tensor()};
  }
};

struct HyenaSE : Function<HyenaSE> {
  static Tensor forward(AutogradContext* ctx, const Tensor& feat, const Tensor& w, const OptTensor& halo, bool pre, bool post, bool fast) {
    const int B = feat.size(0), Ln = feat.size(1), D = feat.size(2) / 3, G = w.size(0), K = w.size(1);
    Tensor fc = aligned(feat), hc = aligned(halo), z = alloc({B, Ln, D}, BF16, feat.device()), wf;
    if (fast) {
      Taps t = taps(w);
      wf = t.f32;
      SB_CALL(sb_se_fwd_taps, 1, ptr(fc), ptr(hc), ptr(t.in), t.bf16, t.bf16 ? f32o(wf) : (float*)nullptr, out(z), B, Ln, D, G, K, (int)pre, (int)post,
              stream());
    } else {
      wf = f32c(w);
      SB_CALL(sb_se_fwd, 1, ptr(fc), ptr(hc), f32(wf), out(z), B, Ln, D, G, K, (int)pre, (int)post, stream());
    }
    ctx->save_for_backward({fc, wf, hc});
    ctx->saved_data["wtype"] = (int64_t)w.scalar_type();
    ctx->saved_data["gates"] = (int64_t)(2 * pre + post);
    return z;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &fc = s[0], &wf = s[1], &hc = s[2];
    const int gates = ctx->saved_data["gates"].toInt();
    Tensor gc = aligned(g[0]), df = alloc_like(fc), dh = hc.defined() ? alloc_like(hc) : Tensor(), dw = zeros(wf.sizes(), F32, wf.device());
    SB_CALL(sb_se_bwd, 1, ptr(fc), ptr(hc), f32(wf), ptr(gc), out(df), out(dh), f32o(dw), (int)fc.size(0), (int)fc.size(1), (int)fc.size(2) / 3,
            (int)wf.size(0), (int)wf.size(1), gates >> 1, gates & 1, stream());
    return {df, dw.to(saved_type(ctx, "wtype")), dh, Tensor(), Tensor(), Tensor()};
  }
};

// Tensor-core kernels when a 16-channel slab shares one filter (mr_conv_umma.cu, with halo rows mr_conv_tc.cu), else the CUDA-core
// kernels (mr_conv.cu), whose backward wants the convolution itself (kept when `train`).
//
// A forward without halo rows stays with mr_conv_tc.cu where that is faster: its products grow with the filter in steps of 16 taps, those of
// mr_conv_umma.cu are 256 taps whatever K is.  us, mr_conv_tc.cu / mr_conv_umma.cu: K = 16 8192 x 1024 16.9 / 19.5, 2 x 1237 x 1024 8.9 / 10.0,
// 300 x 4096 7.6 / 8.1, 600 x 1024 6.9 / 6.4; K = 31 17.5 / 19.4, 9.3 / 10.1, 7.9 / 8.1, 7.3 / 6.5, 1237 x 1024 8.0 / 7.4; K = 40 18.6 / 19.4, 10.4 /
// 10.1, 9.0 / 8.1; one row of 256 3.9 / 4.7 (K = 3).  The backward is faster on mr_conv_umma.cu at every size measured (K = 3, one row 12.7 -> 10.4).
bool short_filter(int64_t B, int64_t Ln, int64_t D, int64_t K) {
  return K <= 32 && B <= 65535 && (Ln <= 32 || B * Ln * D >= 65536 * std::max<int64_t>(K, 16));
}
struct HyenaMR : Function<HyenaMR> {
  static Tensor forward(AutogradContext* ctx, const Tensor& feat, const Tensor& h, const Tensor& bias, const OptTensor& halo, bool train) {
    const int B = feat.size(0), Ln = feat.size(1), D = feat.size(2) / 3, G = h.size(0), K = h.size(1);
    Tensor fc = aligned(feat), hc = aligned(halo), hf = f32c(h), bf = f32c(bias), z = alloc({B, Ln, D}, BF16, feat.device()), y;
    const bool tc = (D / G) % 16 == 0 && D % 8 == 0;
    if (tc && !hc.defined() && !short_filter(B, Ln, D, K)) {
      SB_CALL(sb_mr_umma_fwd, 1, ptr(fc), f32(hf), f32(bf), out(z), B, Ln, D, G, K, status_word(feat.device()), stream());
    } else if (tc) {
      SB_CALL(sb_mr_tc_fwd, 1, ptr(fc), ptr(hc), f32(hf), f32(bf), out(z), B, Ln, D, G, K, stream());
    } else {
      if (train) y = alloc_like(z);
      SB_CALL(sb_mr_fwd, 1, ptr(fc), ptr(hc), f32(hf), f32(bf), out(z), out(y), B, Ln, D, G, K, stream());
    }
    ctx->save_for_backward({fc, hf, bf, y, hc});
    ctx->saved_data["tc"] = tc;
    ctx->saved_data["htype"] = (int64_t)h.scalar_type();
    ctx->saved_data["btype"] = (int64_t)bias.scalar_type();
    return z;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &fc = s[0], &hf = s[1], &bf = s[2], &y = s[3], &hc = s[4];
    const int B = fc.size(0), Ln = fc.size(1), D = fc.size(2) / 3, G = hf.size(0), K = hf.size(1);
    Tensor gc = aligned(g[0]), df = alloc_like(fc), dhalo = hc.defined() ? cleared(alloc_like(hc)) : Tensor(),
           dh = zeros(hf.sizes(), F32, hf.device()), db = zeros(bf.sizes(), F32, bf.device());
    const bool tc = ctx->saved_data["tc"].toBool();
    if (tc && !hc.defined()) {
      const Tensor ba = aligned(bf);       // read in 16-byte vectors; a parameter may lie anywhere in a flat buffer
      SB_CALL(sb_mr_umma_bwd, 1, ptr(fc), f32(hf), f32(ba), ptr(gc), out(df), f32o(dh), f32o(db), B, Ln, D, G, K, status_word(fc.device()), stream());
    } else if (tc) {
      SB_CALL(sb_mr_tc_bwd, 1, ptr(fc), ptr(hc), f32(hf), f32(bf), ptr(gc), out(df), out(dhalo), f32o(dh), f32o(db), B, Ln, D, G, K, stream());
    } else {
      SB_CALL(sb_mr_bwd, 2, ptr(fc), ptr(hc), f32(hf), f32(bf), ptr(gc), ptr(y), out(df), out(dhalo), f32o(dh), f32o(db), B, Ln, D, G, K, stream());
    }
    return {df, dh.to(saved_type(ctx, "htype")), db.to(saved_type(ctx, "btype")), dhalo, Tensor()};
  }
};

// ------------------------------------------------------------------------------------ Hyena-LI
// The shared-memory tiled scan (li_scan.cu): D % 8 == 0.  The filter is prepared by the forward's first kernel and handed to the
// backward; the filter gradients come finished out of the backward's last one.  `tc`: chunk length of the forward.
constexpr int64_t LI_ORDER = 16;
struct HyenaLI : Function<HyenaLI> {
  static variable_list forward(AutogradContext* ctx, const Tensor& feat, const Tensor& gamma, const Tensor& R, const Tensor& p, const Tensor& bias,
                               const OptTensor& state_in, bool want_state, int64_t tc) {
    const int64_t B = feat.size(0), Ln = feat.size(1), D = feat.size(2) / 3, O = gamma.size(1);
    const at::Device dev = feat.device();
    Tensor fc = aligned(feat), bf = f32c(bias), sin = state_in.has_value() ? f32c(*state_in) : Tensor();
    // the backward reads the entering state: the caller may go on with its own buffer
    if (sin.defined() && sin.const_data_ptr() == state_in->const_data_ptr()) sin = sin.clone();
    Tensor modal = alloc({4 * D, LI_ORDER}, F32, dev), S = alloc({B, (Ln + tc - 1) / tc, D, LI_ORDER}, F32, dev),
           sout = want_state ? alloc({B, D, O}, F32, dev) : Tensor(), z = alloc({B, Ln, D}, BF16, dev), gf = f32c(gamma), pf = f32c(p), Rf = f32c(R);
    SB_CALL(sb_li_fwd_tiled, 4, ptr(fc), f32(gf), f32(pf), f32(Rf), f32(bf), f32(sin), f32o(sout), f32o(modal), f32o(S), out(z), (int)B, (int)Ln,
            (int)D, (int)O, (int)tc, stream());
    ctx->save_for_backward({fc, modal, bf, sin});
    ctx->saved_data["meta"] = std::vector<int64_t>{O, (int64_t)gamma.scalar_type(), (int64_t)R.scalar_type(), (int64_t)p.scalar_type(),
                                                   (int64_t)bias.scalar_type()};
    ctx->set_materialize_grads(false);
    if (want_state) return {z, sout};
    return {z};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &fc = s[0], &modal = s[1], &bf = s[2], &sin = s[3];
    const std::vector<int64_t> m = ctx->saved_data["meta"].toIntVector();
    const int64_t O = m[0], B = fc.size(0), Ln = fc.size(1), D = fc.size(2) / 3;
    const at::Device dev = fc.device();
    const int64_t tc = L.sb_li_bwd_tiled_chunk(), NC = (Ln + tc - 1) / tc;
    Tensor gc = g[0].defined() ? aligned(g[0]) : at::zeros({B, Ln, D}, fc.options());
    Tensor S = alloc({B, NC, D, LI_ORDER}, F32, dev), A = alloc({B, NC, D, LI_ORDER}, F32, dev), dRp = alloc({B, NC, D, LI_ORDER}, F32, dev),
           dBp = alloc({B, NC, D}, F32, dev), df = alloc_like(fc), dR = alloc({D, O}, F32, dev), dll = alloc({D, O}, F32, dev),
           db = alloc({D}, F32, dev), dsi = sin.defined() ? alloc({B, D, O}, F32, dev) : Tensor(),
           dso = g.size() > 1 && g[1].defined() ? f32c(g[1]) : Tensor();
    SB_CALL(sb_li_bwd_tiled, 4, ptr(fc), ptr(gc), f32(modal), f32(bf), f32(sin), f32(dso), f32o(S), f32o(A), f32o(dRp), f32o(dBp), out(df), f32o(dR),
            f32o(dll), f32o(db), f32o(dsi), (int)B, (int)Ln, (int)D, (int)O, stream());
    const auto type = [&](int i) { return (at::ScalarType)m[i]; };
    // gamma and p get gradients of their own storage
    Tensor dp = type(3) != F32 ? dll.to(type(3)) : ctx->needs_input_grad(3) ? dll.clone() : Tensor();
    return {df, dll.to(type(1)), dR.to(type(2)), dp, db.to(type(4)), dsi, Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------ attention on the packed projection
struct Strides { long long s[3]; explicit Strides(const Tensor& t) : s{t.stride(0), t.stride(1), t.stride(2)} {} };

// rotary embedding of two tensors in one launch: (source, destination) pairs [B, L, H, 128], sources bf16 or fp32
void rope2(const Tensor& s0, const Tensor& d0, const Tensor& s1, const Tensor& d1, const Tensor& cos, const Tensor& sin, bool inverse) {
  const void* src[2] = {ptr(s0), ptr(s1)};
  void* dst[2] = {out(d0), out(d1)};
  const Strides a(s0), b(s1), c(d0), d(d1);
  const long long ss[6] = {a.s[0], a.s[1], a.s[2], b.s[0], b.s[1], b.s[2]}, ds[6] = {c.s[0], c.s[1], c.s[2], d.s[0], d.s[1], d.s[2]};
  const int wide[2] = {s0.scalar_type() == F32, s1.scalar_type() == F32};
  const int rc = SB_RUN(sb_attn_rope, 1, src, dst, ss, ds, wide, 2, f32(cos), f32(sin), (int)s0.size(0), (int)s0.size(1), (int)s0.size(2),
                        (int)cos.size(-1), (int)inverse, stream());
  TORCH_CHECK(rc == 0, "rotary embedding failed (code ", rc, "): ", layouts({{"cos", &cos}, {"from", &s0}, {"to", &d0}, {"from", &s1}, {"to", &d1}}));
}
bool packed_rows(const Tensor& t) {        // what the kernels read in place: unit inner stride, the others on 16-byte boundaries
  return t.dim() == 4 && t.scalar_type() == BF16 && t.size(3) == 128 && t.stride(3) == 1 && t.stride(0) % 8 == 0 && t.stride(1) % 8 == 0 &&
         t.stride(2) % 8 == 0 && on16(t);
}

// Attention on qkv [B, L, H, 3 * 128] (per head: q, k, v) with rotary embedding of q and k inside.  The backward writes dq, dk, dv
// straight into one packed gradient buffer; with rotary embedding the query gradient is rotated back out of its fp32 accumulator.
struct FlashPacked : Function<FlashPacked> {
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, const OptTensor& cos_, const OptTensor& sin_, bool causal) {
    const Tensor cos = opt(cos_), sin = opt(sin_);
    const int64_t B = qkv.size(0), Ln = qkv.size(1), H = qkv.size(2);
    const at::Device dev = qkv.device();
    Tensor q = qkv.slice(3, 0, 128), k = qkv.slice(3, 128, 256), v = qkv.slice(3, 256, 384), qr, kr;
    if (cos.defined()) {
      qr = alloc({B, Ln, H, 128}, BF16, dev);
      kr = alloc({B, Ln, H, 128}, BF16, dev);
      rope2(q, qr, k, kr, cos, sin, false);
      q = qr; k = kr;
    }
    Tensor o = alloc({B, Ln, H, 128}, BF16, dev), lse = alloc({B, H, Ln}, F32, dev);
    const Strides qs(q), ks(k), vs(v), os(o);
    const int rc = SB_RUN(sb_attn_fwd, 1, ptr(q), ptr(k), ptr(v), out(o), f32o(lse), (int)B, (int)H, (int)Ln, (int)Ln, qs.s, ks.s, vs.s, os.s,
                          (int)causal, 0.08838834764831845f, status_word(dev), stream());
    TORCH_CHECK(rc == 0, "attention forward failed (code ", rc, ", encode ", L.sb_attn_last_encode_result(), "): ", layouts({{"q", &q}, {"k", &k}, {"v", &v}}));
    ctx->save_for_backward({qkv, qr, kr, o, lse, cos, sin});
    ctx->saved_data["causal"] = causal;
    return o;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const variable_list s = ctx->get_saved_variables();
    const Tensor &qkv = s[0], &o = s[3], &lse = s[4], &cos = s[5], &sin = s[6];
    const bool rot = cos.defined();
    const int64_t B = qkv.size(0), Ln = qkv.size(1), H = qkv.size(2);
    const at::Device dev = qkv.device();
    Tensor q = rot ? s[1] : qkv.slice(3, 0, 128), k = rot ? s[2] : qkv.slice(3, 128, 256), v = qkv.slice(3, 256, 384);
    Tensor go = packed_rows(g[0]) ? g[0] : g[0].contiguous();
    Tensor dqkv = alloc(qkv.sizes(), BF16, dev), dq = dqkv.slice(3, 0, 128), dk = dqkv.slice(3, 128, 256), dv = dqkv.slice(3, 256, 384);
    Tensor acc = zeros({B, Ln, H, 128}, F32, dev), stats = alloc({2 * B * H * ((Ln + 63) / 64 * 64)}, F32, dev);
    const Strides gs(go), qs(q), ks(k), vs(v), os(o), dqs(rot ? o : dq), dks(dk), dvs(dv);
    const int rc = SB_RUN(sb_attn_bwd, 3, ptr(go), ptr(q), ptr(k), ptr(v), ptr(o), f32(lse), (const float*)nullptr, f32o(stats), f32o(acc),
                          rot ? (void*)nullptr : out(dq), out(dk), (int)B, (int)H, (int)Ln, (int)Ln, out(dv), gs.s, qs.s, ks.s, vs.s, os.s, dqs.s,
                          dks.s, dvs.s, (int)ctx->saved_data["causal"].toBool(), 0.08838834764831845f, status_word(dev), stream());
    TORCH_CHECK(rc == 0, "attention backward failed (code ", rc, ", encode ", L.sb_attn_last_encode_result(), "): ",
                layouts({{"dout", &go}, {"q", &q}, {"k", &k}, {"v", &v}}));
    if (rot) rope2(acc, dq, dk, dk, cos, sin, true);
    return {dqkv, Tensor(), Tensor(), Tensor()};
  }
};

// ------------------------------------------------------------------------------------ what Python calls
bool fused(const py::handle& w) {          // the parameter's gradient lives in a persistent flat buffer (set by the ZeRO optimizers)
  PyObject* v = PyObject_GetAttrString(w.ptr(), "_fuse_grad_accum");
  if (!v) { PyErr_Clear(); return false; }
  const int yes = PyObject_IsTrue(v);
  Py_DECREF(v);
  return yes == 1;
}
OptTensor table(const OptTensor& t) { return t.has_value() ? OptTensor(aligned(t->to(F32))) : t; }

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("load", &load);
  m.def("launches", [] { return g_launches.load(); });
  m.def("set_guarded", [](bool on) { g_guarded = on; });
  m.def("set_nvtx", [](bool on) { g_nvtx = on; });
  m.def("linear", [](const Tensor& x, const py::object& w, const OptTensor& bias, const OptTensor& residual) {
    no_transforms();
    return Linear::apply(x, w.cast<Tensor>(), bias, residual, fused(w));
  });
  m.def("rmsnorm", [](const Tensor& x, const Tensor& w, double eps, int64_t form) { no_transforms(); return RmsNorm::apply(x, w, eps, form); });
  m.def("rmsnorm_residual", [](const Tensor& x, const Tensor& w, double eps, int64_t form) {
    no_transforms();
    variable_list r = RmsNormResidual::apply(x, w, eps, form);
    return std::make_tuple(r[0], r[1]);
  });
  m.def("norm_linear", [](const Tensor& x, const Tensor& wn, double eps, int64_t form, const py::object& w, const OptTensor& bias) {
    no_transforms();
    const Tensor wt = w.cast<Tensor>();
    variable_list r = NormLinear::apply(x, wn, eps, form, wt, bias, fused(w), wants_grad({&x, &wn, &wt, given(bias)}));
    return std::make_tuple(r[0], r[1]);
  });
  m.def("glu", [](const Tensor& ab, int64_t act) { no_transforms(); return Glu::apply(ab, act); });
  m.def("mlp_gated", [](const Tensor& x, const Tensor& wn, double eps, int64_t form, const py::object& w12, const py::object& w3, const OptTensor& b3,
                        int64_t act) {
    no_transforms();
    const Tensor a = w12.cast<Tensor>(), b = w3.cast<Tensor>();
    return MlpGated::apply(x, wn, eps, form, a, b, b3, act, fused(w12), fused(w3), wants_grad({&x, &wn, &a, &b, given(b3)}));
  });
  m.def("cross_entropy", [](const Tensor& logits, const Tensor& labels) { no_transforms(); return CrossEntropy::apply(logits, labels); });
  m.def("dwconv", [](const Tensor& x, const Tensor& w, const OptTensor& halo, bool fast) { no_transforms(); return DwConv::apply(x, w, halo, fast); });
  m.def("hyena_se", [](const Tensor& feat, const Tensor& w, const OptTensor& halo, bool pre, bool post, bool fast) {
    no_transforms();
    return HyenaSE::apply(feat, w, halo, pre, post, fast);
  });
  m.def("hyena_mr", [](const Tensor& feat, const Tensor& h, const Tensor& bias, const OptTensor& halo) {
    no_transforms();
    return HyenaMR::apply(feat, h, bias, halo, wants_grad({&feat, &h, &bias, given(halo)}));
  });
  m.def("hyena_li", [](const Tensor& feat, const Tensor& gamma, const Tensor& R, const Tensor& p, const Tensor& bias, const OptTensor& state_in,
                       bool want_state, int64_t tc) {
    no_transforms();
    variable_list r = HyenaLI::apply(feat, gamma, R, p, bias, state_in, want_state, tc);
    return std::make_tuple(r[0], want_state ? OptTensor(r[1]) : OptTensor());
  });
  m.def("attention_packed", [](const Tensor& qkv, const OptTensor& cos, const OptTensor& sin, bool causal) {
    no_transforms();
    return FlashPacked::apply(qkv, table(cos), table(sin), causal);
  });
}
