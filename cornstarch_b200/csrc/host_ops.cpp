// Host side of the hot calls: shapes, strides, output allocation and the launch of one operator without coming back to Python
// in between.
//
// What it replaces is Python around the same entry points of libcornstarch_b200.so: three to ten tensor methods and allocations
// and one ctypes call of up to 45 arguments per operator, 20 to 45 us of host time where the kernels of a layer of a few thousand
// tokens take 3 to 40 us.  The autograd functions stay in Python (hooks, saved tensors, transforms and buffers see the same
// tensors as before); they hand their tensors over here.  A function answers None for a form that it does not take (activations
// take all that Python sends them): the Python statement of the operator decides what happens then (another route, a copy, an
// error).
//
// What allocates or launches runs without the GIL (60 ns a call), as calls through ctypes do: a launch waits while the stream's
// queue is full, an allocation may wait for the device, and the threads that watch over a hanging step are Python threads.  What is
// Python (arguments, results, the one look-up of a status word) is done before, after, or with the GIL taken back for it.
//
// The kernels' entry points are looked up once in the library that ctypes has loaded (bind), so there is one library per process
// whichever file it came from.
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/types.h>

#include <atomic>
#include <optional>
#include <stdexcept>
#include <string>
#include <tuple>
#include <unordered_map>
#include <vector>

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;
using Tensor2 = std::tuple<Tensor, Tensor>;  // (undefined tensors become None)
using Tensor3 = std::tuple<Tensor, Tensor, Tensor>;
using Tensor5 = std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor>;

namespace {

std::atomic<long> g_launches{0};
py::object* g_status_word = nullptr;  // Python: device index -> address of its status word
constexpr int MAX_DEVICES = 64;
std::atomic<int*> g_status[MAX_DEVICES];

// One exported function of the library; counted like a call through ctypes.
struct EntryPoint {
  const char* name;
  std::atomic<void*> address{nullptr};  // set by bind, read without the GIL
  explicit EntryPoint(const char* n) : name(n) { all().push_back(this); }
  static std::vector<EntryPoint*>& all() {
    static std::vector<EntryPoint*> list;
    return list;
  }
};
template <typename F>
struct Entry : EntryPoint {
  using EntryPoint::EntryPoint;
  F get() {
    void* p = address.load();
    if (p == nullptr) throw std::runtime_error(std::string("host_ops: no entry point ") + name);
    return reinterpret_cast<F>(p);
  }
};
void check(int code, const char* what) {
  if (code != 0)
    throw std::runtime_error(std::string("cornstarch_b200 native call ") + what + " failed with code " + std::to_string(code));
}

void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

int* status_word(const Tensor& t) {
  const int i = t.device().index();
  if (i < 0 || i >= MAX_DEVICES) throw std::runtime_error("host_ops: device index");
  int* p = g_status[i].load();
  if (p == nullptr) {
    py::gil_scoped_acquire gil;
    p = reinterpret_cast<int*>((*g_status_word)(i).cast<uintptr_t>());
    g_status[i].store(p);
  }
  return p;
}

void* ptr(const OptTensor& t) { return t.has_value() ? t->data_ptr() : nullptr; }
bool on_grid(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
bool bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }
bool grad_type(const Tensor& t) { return bf16(t) || t.scalar_type() == at::kFloat; }
bool is_fp32(const Tensor& t) { return t.scalar_type() == at::kFloat; }
bool fits_int(int64_t v) { return v >= 0 && v <= 0x7fffffff; }
// Contiguous and on the 16-byte grid of the kernels' vector loads.
Tensor dense(const Tensor& t) {
  if (!t.is_contiguous()) return t.contiguous();
  return on_grid(t) ? t : t.clone();
}

Tensor as_2d(const Tensor& x) {
  Tensor x2 = x.dim() == 2 ? x : x.reshape({-1, x.size(-1)});
  if (x2.stride(1) != 1 || (x2.stride(0) % 8) || !on_grid(x2)) x2 = x2.contiguous();
  return x2;
}

// Tensors one behind the other in one storage as one (dims = 2: rows of equal width; 1: vectors); none otherwise.
OptTensor fuse_adjacent(const std::vector<Tensor>& ts, int dims) {
  const Tensor& t0 = ts[0];
  int64_t n = 0;
  const char* end = static_cast<const char*>(t0.data_ptr());
  for (const Tensor& t : ts) {
    if (dims == 2 && (t.dim() != 2 || !t.is_contiguous() || t.size(1) != t0.size(1) || t.scalar_type() != t0.scalar_type())) return std::nullopt;
    if (static_cast<const char*>(t.data_ptr()) != end || t.storage().data() != t0.storage().data()) return std::nullopt;
    end += t.numel() * t.element_size();
    n += dims == 2 ? t.size(0) : t.numel();
  }
  return dims == 2 ? t0.as_strided({n, t0.size(1)}, {t0.size(1), 1}, t0.storage_offset()) : t0.as_strided({n}, {1}, t0.storage_offset());
}

// ---------------------------------------------------------------------------------------------------------------- GEMM
using GemmFn = int (*)(const void*, const void*, void*, const void*, int, int, int, int, int, int, int, int, int, int, int, int, int, int*, void*);
Entry<GemmFn> e_gemm("csb_gemm_bf16");

bool gemm_operand(const Tensor& t) {
  return t.is_cuda() && bf16(t) && t.dim() == 2 && t.stride(1) == 1 && t.stride(0) % 8 == 0 && on_grid(t) && fits_int(t.stride(0)) &&
         fits_int(t.size(0)) && fits_int(t.size(1));
}
void launch_gemm(const Tensor& a, const Tensor& b, void* out, const void* bias, int64_t M, int64_t N, int64_t K, int64_t ldc, bool a_mn, bool b_mn,
                 bool fp32, bool acc, int act, int tile_n, int max_ctas) {
  ++g_launches;
  check(e_gemm.get()(a.data_ptr(), b.data_ptr(), out, bias, (int)M, (int)N, (int)K, (int)a.stride(0), (int)b.stride(0), (int)ldc, a_mn, b_mn,
                     fp32, acc, act, tile_n, max_ctas, status_word(a), stream()),
        "csb_gemm_bf16");
}
OptTensor gemm(const Tensor& a, const Tensor& b, bool a_mn, bool b_mn, const OptTensor& bias, int act, const OptTensor& out_, bool acc, int tile_n,
                int max_ctas) {
  if (!gemm_operand(a) || !gemm_operand(b)) return std::nullopt;
  const int64_t M = a.size(a_mn ? 1 : 0), K = a.size(a_mn ? 0 : 1), N = b.size(b_mn ? 1 : 0);
  if (b.size(b_mn ? 0 : 1) != K || M == 0 || N == 0 || K == 0) return std::nullopt;
  if (bias && (!bf16(*bias) || !bias->is_contiguous() || bias->numel() != N)) return std::nullopt;
  Tensor out;
  if (out_) {
    out = *out_;
    if (out.dim() != 2 || out.size(0) != M || out.size(1) != N || out.stride(1) != 1 || !grad_type(out) || !fits_int(out.stride(0))) return std::nullopt;
  } else {
    out = at::empty({M, N}, a.options());
    acc = false;
  }
  launch_gemm(a, b, out.data_ptr(), ptr(bias), M, N, K, out.stride(0), a_mn, b_mn, is_fp32(out), acc, act, tile_n, max_ctas);
  return out;
}

// ------------------------------------------------------------------------------------------------------- linear layers
using ColsFn = int (*)(const void*, const void* const*, const void* const*, const int*, int, void*, int, int, int, int, int, int*, void*);
Entry<ColsFn> e_gemm_cols("csb_gemm_cols_bf16");
constexpr int MAX_COL_GROUPS = 4, ERR_NO_FIT = -5;

// Weights that are not adjacent as one launch; false where the library has no tile for them.
bool cols_gemm(const Tensor& x2, const std::vector<Tensor>& ws, const std::vector<Tensor>& biases, void* out, int64_t T, int64_t N, int64_t K) {
  if (ws.size() > MAX_COL_GROUPS || (reinterpret_cast<uintptr_t>(out) & 15) || N % 8) return false;
  const void* b[MAX_COL_GROUPS];
  const void* bias[MAX_COL_GROUPS];
  int widths[MAX_COL_GROUPS];
  for (size_t i = 0; i < ws.size(); ++i) {
    if (ws[i].stride(0) != ws[0].stride(0)) return false;
    b[i] = ws[i].data_ptr();
    bias[i] = biases.empty() ? nullptr : biases[i].data_ptr();
    widths[i] = (int)ws[i].size(0);
  }
  const int r = e_gemm_cols.get()(x2.data_ptr(), b, biases.empty() ? nullptr : bias, widths, (int)ws.size(), out, (int)T, (int)K, (int)x2.stride(0),
                                  (int)ws[0].stride(0), (int)N, status_word(x2), stream());
  if (r == ERR_NO_FIT) return false;
  ++g_launches;
  check(r, "csb_gemm_cols_bf16");
  return true;
}

// (out, x as 2-D): the concatenated projections of x; one GEMM where the weights (and biases) are adjacent, else one each.
std::optional<Tensor2> linear_fwd(const Tensor& x, const std::vector<Tensor>& ws, const std::vector<OptTensor>& bs) {
  if (!x.is_cuda() || !bf16(x) || x.dim() < 1 || x.numel() == 0) return std::nullopt;
  const int64_t K = x.size(-1);
  int64_t N = 0;
  for (const Tensor& w : ws) {
    if (!gemm_operand(w) || w.size(1) != K || w.size(0) == 0) return std::nullopt;
    N += w.size(0);
  }
  const bool has_bias = bs[0].has_value();
  std::vector<Tensor> biases;
  for (size_t i = 0; i < ws.size(); ++i) {
    if (bs[i].has_value() != has_bias) return std::nullopt;
    if (has_bias) {
      if (!bf16(*bs[i]) || !bs[i]->is_contiguous() || bs[i]->numel() != ws[i].size(0)) return std::nullopt;
      biases.push_back(*bs[i]);
    }
  }
  Tensor x2 = as_2d(x);
  if (!gemm_operand(x2)) return std::nullopt;
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = N;
  Tensor out = at::empty(shape, x.options());
  const int64_t T = x2.size(0);
  OptTensor w, b;
  if (ws.size() == 1) {
    w = ws[0];
    if (has_bias) b = biases[0];
  } else {
    w = fuse_adjacent(ws, 2);
    if (has_bias) b = fuse_adjacent(biases, 1);
  }
  if (w && (!has_bias || b)) {
    launch_gemm(x2, *w, out.data_ptr(), ptr(b), T, N, K, N, false, false, false, false, 0, 0, 0);
  } else if (!cols_gemm(x2, ws, biases, out.data_ptr(), T, N, K)) {
    char* o = static_cast<char*>(out.data_ptr());
    for (size_t i = 0; i < ws.size(); ++i) {
      launch_gemm(x2, ws[i], o, has_bias ? biases[i].data_ptr() : nullptr, T, ws[i].size(0), K, N, false, false, false, false, 0, 0, 0);
      o += ws[i].size(0) * 2;
    }
  }
  return Tensor2(out, x2);
}

using LinearBwdFn = int (*)(const void*, const void*, const void*, void*, void*, void*, float*, int, int, int, int, int, int, int, int, int, int,
                            int, int*, void*);
using PartsFn = int (*)(int);
Entry<LinearBwdFn> e_linear_bwd("csb_linear_bwd");
Entry<PartsFn> e_colsum_parts("csb_colsum_parts");

// (dx or None, dW, db or None) of a linear layer whose operands the caller has looked over; w_main / b_main: the buffers that dW and
// db are added to.
std::optional<Tensor3> linear_bwd(const Tensor& dy2, const Tensor& x2, const Tensor& w, bool need_x, const OptTensor& w_main, bool has_bias, const OptTensor& b_main) {
  if (!gemm_operand(dy2) || !gemm_operand(x2) || !gemm_operand(w)) return std::nullopt;
  const int64_t T = dy2.size(0), N = w.size(0), K = w.size(1);
  if (T == 0 || N % 8 || K % 8 || N == 0 || K == 0) return std::nullopt;
  Tensor dW = w_main ? *w_main : at::empty({N, K}, dy2.options()), db, scratch, dx;
  if (has_bias) {
    scratch = at::empty({e_colsum_parts.get()((int)T) * N}, dy2.options().dtype(at::kFloat));
    db = b_main ? *b_main : at::empty({N}, dy2.options());
  }
  if (need_x) dx = at::empty({T, K}, dy2.options());
  ++g_launches;
  check(e_linear_bwd.get()(dy2.data_ptr(), x2.data_ptr(), w.data_ptr(), need_x ? dx.data_ptr() : nullptr, dW.data_ptr(),
                           has_bias ? db.data_ptr() : nullptr, has_bias ? static_cast<float*>(scratch.data_ptr()) : nullptr, (int)T, (int)N,
                           (int)K, (int)dy2.stride(0), (int)x2.stride(0), (int)w.stride(0), (int)dW.stride(0), is_fp32(dW), w_main.has_value(),
                           has_bias && is_fp32(db), b_main.has_value(), status_word(dy2), stream()),
        "csb_linear_bwd");
  return Tensor3(dx, dW, db);
}

// --------------------------------------------------------------------------------------------------------------- norms
using NormFwdFn = int (*)(int, const void*, const void*, const void*, const void*, void*, void*, float*, float*, int, int, float, float, void*);
using NormBwdFn = int (*)(int, const void*, const void*, const void*, const float*, const float*, const void*, void*, float*, float*, void*, void*,
                          int, int, int, int, float, void*);
Entry<NormFwdFn> e_norm_fwd("csb_norm_fwd");
Entry<NormBwdFn> e_norm_bwd("csb_norm_bwd");
Entry<PartsFn> e_norm_parts("csb_norm_bwd_parts");

// (y, h or None, what the backward normalises, mean or None, rstd)
std::optional<Tensor5> norm_fwd(const Tensor& x, const OptTensor& res, const Tensor& w, const OptTensor& b, double eps, bool is_ln, double w_offset) {
  const int64_t H = x.size(-1);
  if (x.numel() == 0) return std::nullopt;
  const Tensor x2 = dense(x.reshape({-1, H}));
  const int64_t rows = x2.size(0);
  Tensor r2, h, mean;
  if (res) {
    r2 = dense(res->reshape({-1, H}));
    h = at::empty_like(x2);
  }
  Tensor y = at::empty_like(x2), rstd = at::empty({rows}, x.options().dtype(at::kFloat));
  if (is_ln) mean = at::empty({rows}, rstd.options());
  const Tensor wd = dense(w);
  OptTensor bd;
  if (b) bd = dense(*b);
  ++g_launches;
  check(e_norm_fwd.get()(is_ln, x2.data_ptr(), res ? r2.data_ptr() : nullptr, wd.data_ptr(), ptr(bd), y.data_ptr(), res ? h.data_ptr() : nullptr,
                         is_ln ? static_cast<float*>(mean.data_ptr()) : nullptr, static_cast<float*>(rstd.data_ptr()), (int)rows, (int)H, (float)eps,
                         (float)w_offset, stream()),
        "csb_norm_fwd");
  return Tensor5(y.view(x.sizes()), res ? h.view(x.sizes()) : Tensor(), res ? h : x2, mean, rstd);
}
// (dx, dw, db or None); w_main / b_main: buffers to add to instead of new gradients
std::optional<Tensor3> norm_bwd(const Tensor& dy, const OptTensor& dh, const Tensor& hs, const Tensor& w, const OptTensor& mean, const Tensor& rstd, bool is_ln,
                    bool has_b, double w_offset, const OptTensor& w_main, const OptTensor& b_main) {
  const int64_t rows = hs.size(0), H = hs.size(1);
  if (rows == 0) return std::nullopt;
  const Tensor dy2 = dense(dy.reshape({-1, H})), wd = dense(w);
  Tensor dres, dbp, dw, db;
  if (dh) dres = dense(dh->reshape({-1, H}));
  Tensor dx = at::empty_like(hs);
  const auto f32 = hs.options().dtype(at::kFloat);
  const int64_t parts = e_norm_parts.get()((int)rows);
  Tensor dwp = at::empty({parts * H}, f32);
  const bool bias = is_ln && has_b, main = w_main.has_value();
  if (bias) dbp = at::empty({parts * H}, f32);
  dw = main ? *w_main : at::empty({H}, hs.options());
  if (main ? b_main.has_value() : bias) db = main ? *b_main : at::empty({H}, hs.options());
  ++g_launches;
  check(e_norm_bwd.get()(is_ln, dy2.data_ptr(), hs.data_ptr(), wd.data_ptr(), mean ? static_cast<const float*>(mean->data_ptr()) : nullptr,
                         static_cast<const float*>(rstd.data_ptr()), dh ? dres.data_ptr() : nullptr, dx.data_ptr(), static_cast<float*>(dwp.data_ptr()),
                         bias ? static_cast<float*>(dbp.data_ptr()) : nullptr, dw.data_ptr(), db.defined() ? db.data_ptr() : nullptr, is_fp32(dw), main,
                         (int)rows, (int)H, (float)w_offset, stream()),
        "csb_norm_bwd");
  return Tensor3(dx, dw, db);
}

// ---------------------------------------------------------------------------------------------------------- activations
using ActFwdFn = int (*)(const void*, void*, long, int, void*);
using ActBwdFn = int (*)(const void*, const void*, void*, long, int, void*);
using GluFwdFn = int (*)(const void*, void*, long, int, int, void*);
using GluBwdFn = int (*)(const void*, const void*, void*, long, int, int, void*);
Entry<ActFwdFn> e_act_fwd("csb_act_fwd");
Entry<ActBwdFn> e_act_bwd("csb_act_bwd");
Entry<GluFwdFn> e_glu_fwd("csb_glu_fwd");
Entry<GluBwdFn> e_glu_bwd("csb_glu_bwd");

Tensor2 act_fwd(const Tensor& x, int kind) {
  const Tensor xc = dense(x);
  Tensor y = at::empty_like(xc);
  ++g_launches;
  check(e_act_fwd.get()(xc.data_ptr(), y.data_ptr(), xc.numel(), kind, stream()), "csb_act_fwd");
  return {y, xc};
}
Tensor act_bwd(const Tensor& xc, const Tensor& dy, int kind) {
  const Tensor d = dense(dy);
  Tensor dx = at::empty_like(xc);
  ++g_launches;
  check(e_act_bwd.get()(xc.data_ptr(), d.data_ptr(), dx.data_ptr(), xc.numel(), kind, stream()), "csb_act_bwd");
  return dx;
}
Tensor2 glu_fwd(const Tensor& gu, int act) {
  const int64_t I = gu.size(-1) / 2;
  const Tensor g2 = dense(gu.reshape({-1, 2 * I}));
  std::vector<int64_t> shape(gu.sizes().begin(), gu.sizes().end());
  shape.back() = I;
  Tensor y = at::empty(shape, gu.options());
  ++g_launches;
  check(e_glu_fwd.get()(g2.data_ptr(), y.data_ptr(), g2.size(0), (int)I, act, stream()), "csb_glu_fwd");
  return {y, g2};
}
Tensor glu_bwd(const Tensor& g2, const Tensor& dy, int act) {
  const int64_t I = g2.size(1) / 2;
  const Tensor d2 = dense(dy.reshape({-1, I}));
  Tensor dgu = at::empty_like(g2);
  ++g_launches;
  check(e_glu_bwd.get()(g2.data_ptr(), d2.data_ptr(), dgu.data_ptr(), g2.size(0), (int)I, act, stream()), "csb_glu_bwd");
  return dgu;
}

// ------------------------------------------------------------------------------------------------------------ attention
using AttnFwdFn = int (*)(const void*, const void*, const void*, void*, float*, int, int, int, int, int, int, long, long, long, long, long, long, long,
                          long, float, int, const void*, const void*, const void*, const void*, const void*, int*, void*);
using AttnBwdFn = int (*)(const void*, const void*, const void*, const void*, const void*, const float*, float*, float*, void*, void*, void*, int, int,
                          int, int, int, int, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, long, float,
                          int, const void*, const void*, const void*, const void*, const void*, int*, void*, float*, int);
using SplitsFn = int (*)(int, int, int, int, int, int);
Entry<AttnFwdFn> e_attn_fwd("csb_attn_fwd");
Entry<AttnBwdFn> e_attn_bwd("csb_attn_bwd");
Entry<SplitsFn> e_attn_splits("csb_attn_bwd_splits");

bool attn_layout(const Tensor& t) {
  return t.dim() == 4 && t.stride(3) == 1 && t.stride(2) == t.size(3) && t.stride(1) % 8 == 0 && on_grid(t) && t.is_cuda() && bf16(t);
}
// (out, lse); the mask is a mode with optional per-token bits and positions ([B, S], dense) and its class map
std::optional<Tensor2> attn_fwd(const Tensor& q, const Tensor& k, const Tensor& v, double scale, int mode, const OptTensor& qb, const OptTensor& kb,
                    const OptTensor& qp, const OptTensor& kp, const OptTensor& cls) {
  if (!attn_layout(q) || !attn_layout(k) || !attn_layout(v)) return std::nullopt;
  const int64_t B = q.size(0), Sq = q.size(1), Hq = q.size(2), D = q.size(3), Sk = k.size(1), Hk = k.size(2);
  if (k.size(0) != B || k.size(3) != D || v.sizes() != k.sizes() || q.numel() == 0 || k.numel() == 0) return std::nullopt;
  Tensor out = at::empty({B, Sq, Hq, D}, q.options()), lse = at::empty({B, Hq, Sq}, q.options().dtype(at::kFloat));
  ++g_launches;
  check(e_attn_fwd.get()(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), static_cast<float*>(lse.data_ptr()), (int)B, (int)Sq, (int)Sk,
                         (int)Hq, (int)Hk, (int)D, q.stride(1), q.stride(0), k.stride(1), k.stride(0), v.stride(1), v.stride(0), out.stride(1),
                         out.stride(0), (float)scale, mode, ptr(qb), ptr(kb), ptr(qp), ptr(kp), ptr(cls), status_word(q), stream()),
        "csb_attn_fwd");
  return Tensor2(out, lse);
}
std::optional<Tensor3> attn_bwd(const Tensor& do_, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Tensor& lse, const Tensor& acc, double scale,
                    int mode, const OptTensor& qb, const OptTensor& kb, const OptTensor& qp, const OptTensor& kp, const OptTensor& cls, const OptTensor& dq_,
                    const OptTensor& dk_, const OptTensor& dv_) {
  const int64_t B = q.size(0), Sq = q.size(1), Hq = q.size(2), D = q.size(3), Sk = k.size(1), Hk = k.size(2);
  if (q.numel() == 0 || k.numel() == 0) return std::nullopt;
  const Tensor dout = do_.stride(3) != 1 || do_.stride(2) != D || do_.stride(1) % 8 ? do_.contiguous() : do_;
  const auto f32 = q.options().dtype(at::kFloat);
  Tensor dq = dq_ ? *dq_ : at::empty({B, Sq, Hq, D}, q.options()), dk = dk_ ? *dk_ : at::empty({B, Sk, Hk, D}, q.options()),
         dv = dv_ ? *dv_ : at::empty({B, Sk, Hk, D}, q.options());
  Tensor delta = at::empty({B, Hq, Sq}, f32), part;
  const int splits = e_attn_splits.get()(mode, (int)B, (int)Sq, (int)Sk, (int)Hq, (int)Hk);
  if (splits > 1) part = at::empty({2 * splits * B * Sk * Hk * D}, f32);
  ++g_launches;
  check(e_attn_bwd.get()(q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr(), dout.data_ptr(), static_cast<const float*>(lse.data_ptr()),
                         static_cast<float*>(delta.data_ptr()), static_cast<float*>(acc.data_ptr()), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(),
                         (int)B, (int)Sq, (int)Sk, (int)Hq, (int)Hk, (int)D, q.stride(1), q.stride(0), k.stride(1), k.stride(0), v.stride(1),
                         v.stride(0), out.stride(1), out.stride(0), dout.stride(1), dout.stride(0), dq.stride(1), dq.stride(0), dk.stride(1),
                         dk.stride(0), dv.stride(1), dv.stride(0), (float)scale, mode, ptr(qb), ptr(kb), ptr(qp), ptr(kp), ptr(cls), status_word(q),
                         stream(), splits > 1 ? static_cast<float*>(part.data_ptr()) : nullptr, splits),
        "csb_attn_bwd");
  return Tensor3(dq, dk, dv);
}

}  // namespace

PYBIND11_MODULE(_host_ops, m) {
  m.def("bind", [](const std::unordered_map<std::string, uintptr_t>& entries, py::object status) {
    for (EntryPoint* e : EntryPoint::all()) {
      const auto it = entries.find(e->name);
      if (it != entries.end()) e->address.store(reinterpret_cast<void*>(it->second));
    }
    g_status_word = new py::object(std::move(status));  // kept for the life of the process
  });
  m.def("launches", [] { return g_launches.load(); });
  const auto no_gil = py::call_guard<py::gil_scoped_release>();
  m.def("as_2d", &as_2d, no_gil);
  m.def("fuse_adjacent", [](const std::vector<Tensor>& ts) { return fuse_adjacent(ts, 2); });
  m.def("gemm", &gemm, no_gil);
  m.def("linear_fwd", &linear_fwd, no_gil);
  m.def("linear_bwd", &linear_bwd, no_gil);
  m.def("norm_fwd", &norm_fwd, no_gil);
  m.def("norm_bwd", &norm_bwd, no_gil);
  m.def("act_fwd", &act_fwd, no_gil);
  m.def("act_bwd", &act_bwd, no_gil);
  m.def("glu_fwd", &glu_fwd, no_gil);
  m.def("glu_bwd", &glu_bwd, no_gil);
  m.def("attn_fwd", &attn_fwd, no_gil);
  m.def("attn_bwd", &attn_bwd, no_gil);
}
