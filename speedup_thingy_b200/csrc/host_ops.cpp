// The operator table and the sparse-FFN modules as native autograd operators over the C ABI (kernels.py, cluster_pool.py,
// svd_ffn.py hold the public functions, their argument checks and what they mean).
//
// A launch through ctypes costs the host 15-20 us with its tensors and argument struct, several times what most of these
// kernels run: the attention half of a block on 256 tokens took 330 us for 46 us of device time.  Here an operator's
// allocations, launches and saved tensors are C++: 6 us or so per call (Python entry, autograd node, output tensors) and 3
// to 4 per launch -- RMSNorm 10 us, rotary embedding 11, attention 13 with its two launches, the three projections and the
// output projection with its gather 17 each; the attention half takes 84 us of host time for ten launches, 23 us of device
// time.  Products write the type the caller gets (fp32
// straight from the accumulators), type conversions of an operator's inputs share one launch, views are read with their
// strides.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <map>
#include <mutex>
#include <tuple>

#include "rte_b200.h"

namespace {

using torch::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;
using OptTensor = std::optional<Tensor>;

constexpr auto BF = torch::kBFloat16;
constexpr auto F32 = torch::kFloat32;

// Per device: the status word of the launch table (a device tensor kernels.py hands over once).
std::array<Tensor, 64> g_status;

void bind_status(const Tensor& status) { g_status.at(status.get_device()) = status; }

struct Dev {                                 // makes the tensor's device current for the operator's launches
  c10::cuda::CUDAGuard guard;
  rte_stream_t st;
  int32_t* status;
  explicit Dev(const Tensor& t, const Tensor& status_word = {})
      : guard(t.device()), st(at::cuda::getCurrentCUDAStream(t.get_device()).stream()) {
    const Tensor& s = status_word.defined() ? status_word : g_status.at(t.get_device());
    TORCH_CHECK(s.defined(), "rte_b200: the launch table of this device has not been created");
    status = s.data_ptr<int32_t>();
  }
};

// A refused launch raises what the ctypes binding raises for it, also out of a backward on an autograd thread.
void check(int rc, const char* what) {
  if (rc == 0) return;
  pybind11::gil_scoped_acquire gil;
  const auto type = pybind11::module_::import("speedup_thingy_b200._abi").attr("RteError");
  PyErr_SetString(type.ptr(), c10::str(what, " failed: ", rte_status_string(rc), " (code ", rc, ")").c_str());
  throw pybind11::error_already_set();
}

Tensor empty(std::initializer_list<int64_t> shape, at::ScalarType dt, const Tensor& like) {
  return at::empty(c10::IntArrayRef(shape.begin(), shape.size()), like.options().dtype(dt));
}
Tensor empty_as(const Tensor& t, at::ScalarType dt) { return at::empty(t.sizes(), t.options().dtype(dt)); }
float* f32(const Tensor& t) { return t.defined() ? static_cast<float*>(t.data_ptr()) : nullptr; }
int32_t* i32(const Tensor& t) { return static_cast<int32_t*>(t.data_ptr()); }
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }

// bf16 copies of up to four tensors: what already is bf16 and contiguous is taken as it is, dense fp32 goes through one launch.
std::vector<Tensor> to_bf16(const Dev& dev, std::initializer_list<Tensor> tensors) {
  std::vector<Tensor> out;
  const float* src[4];
  void* dst[4];
  int64_t n[4];
  int count = 0;
  for (const Tensor& t : tensors) {
    if (t.scalar_type() == F32 && t.is_contiguous() && t.numel() > 0) {
      out.push_back(empty_as(t, BF));
      src[count] = f32(t);
      dst[count] = out.back().data_ptr();
      n[count++] = t.numel();
    } else if (t.scalar_type() == BF && t.is_contiguous()) {
      out.push_back(t);
    } else {                                  // one pass whatever the type and the strides
      out.push_back(empty_as(t, BF).copy_(t));
    }
  }
  if (count) check(rte_cast_many_f32_bf16(src, dst, n, count, dev.st), "rte_cast_many_f32_bf16");
  return out;
}

struct Gemm {
  rte_gemm_args a{};
  const Dev& dev;
  Gemm(const Dev& d, const void* A, int64_t lda, bool a_mn, const void* B, int64_t ldb, bool b_mn, void* C, int64_t ldc, int64_t M, int64_t N, int64_t K,
       int epilogue)
      : dev(d) {
    a.M = M; a.N = N; a.K = K;
    a.A = A; a.lda = lda; a.a_mn_major = a_mn;
    a.B = B; a.ldb = ldb; a.b_mn_major = b_mn;
    a.epilogue = epilogue;
    a.C = C; a.ldc = ldc;
    a.splits = 1;
    a.status = d.status;
  }
  Gemm& residual(const void* R, int64_t ldr) { a.R = R; a.ldr = ldr; return *this; }
  Gemm& pair(void* C2, int64_t ldc2, int64_t F) { a.C2 = C2; a.ldc2 = ldc2; a.b_pair_offset = F; return *this; }
  Gemm& groups(const Tensor& tile_group, int64_t n, int64_t stride) { a.tile_group = i32(tile_group); a.n_groups = n; a.b_group_stride = stride; return *this; }
  Gemm& split(int64_t splits, int64_t stride, const int32_t* kblocks) { a.splits = splits; a.split_stride = stride; a.split_kblocks = kblocks; return *this; }
  void run() { check(rte_gemm_bf16(&a, dev.st), "rte_gemm_bf16"); }
};

int epi_of(const Tensor& out) { return out.scalar_type() == F32 ? RTE_EPI_F32 : RTE_EPI_BF16; }
bool direct(at::ScalarType t) { return t == F32 || t == BF; }            // types a product can write itself

// out[M,N] = x[M,K] @ w[K,N]   (weight stored input-major)
void mm_io(const Dev& dev, const Tensor& x16, const Tensor& w16, const Tensor& out) {
  const auto M = x16.size(0), K = x16.size(1), N = w16.size(1);
  if (M > 0) Gemm(dev, ptr(x16), K, false, ptr(w16), N, true, ptr(out), N, M, N, K, epi_of(out)).run();
}
// out[M,N] = x[M,K] @ w[N,K]^T
void mm_oi(const Dev& dev, const Tensor& x16, const Tensor& w16, const Tensor& out) {
  const auto M = x16.size(0), K = x16.size(1), N = w16.size(0);
  if (M > 0) Gemm(dev, ptr(x16), K, false, ptr(w16), K, false, ptr(out), N, M, N, K, epi_of(out)).run();
}

// out f32 [M,N] = a[K,M]^T @ b[K,N], the reduction over K rows cut into partials where that is faster
void wgrad(const Dev& dev, const Tensor& a, const Tensor& b, float* out, int64_t M, int64_t N, int64_t K) {
  Gemm g(dev, ptr(a), a.stride(0), true, ptr(b), b.stride(0), true, out, N, M, N, K, RTE_EPI_F32);
  static std::mutex lock;
  static std::map<std::tuple<int64_t, int64_t, int64_t>, int> known;       // (the rule costs more than a launch)
  int splits;
  {
    std::lock_guard<std::mutex> hold(lock);
    auto it = known.find({M, N, K});
    if (it == known.end()) {
      if (known.size() > 4096) known.clear();
      it = known.emplace(std::make_tuple(M, N, K), rte_gemm_wgrad_splits(&g.a, 16)).first;
    }
    splits = it->second;
  }
  if (splits <= 1) return g.run();
  const Tensor ws = empty({splits, M, N}, F32, a);
  g.a.C = ptr(ws);
  g.split(splits, M * N, nullptr).run();
  check(rte_reduce_splits(f32(ws), splits, M * N, M * N, out, 0, dev.st), "rte_reduce_splits");
}
Tensor wgrad_new(const Dev& dev, const Tensor& a, const Tensor& b, int64_t M, int64_t N, int64_t K, at::ScalarType dt) {
  const Tensor out = empty({M, N}, F32, a);
  if (K > 0) wgrad(dev, a, b, f32(out), M, N, K);
  else out.zero_();
  return dt == F32 ? out : out.to(dt);
}

void dims8(std::initializer_list<int64_t> dims) {
  for (auto v : dims) TORCH_CHECK_VALUE(v % 8 == 0, "rte_b200 GEMM operands need dimensions that are multiples of 8, got ", v);
}
Tensor flat2(const Tensor& t) { return t.view({-1, t.size(-1)}); }
std::vector<int64_t> with_last(c10::IntArrayRef sizes, int64_t n) {
  std::vector<int64_t> s(sizes.begin(), sizes.end());
  s.back() = n;
  return s;
}

// Kernels that take 16 bytes at a time: a contiguous tensor on a 16-byte boundary (a view into the middle of a buffer is
// copied; torch's own allocations start on 512).
Tensor on16(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 ? t.clone() : t; }

// --------------------------------------------------------------------------- RMSNorm
struct RmsNorm : Function<RmsNorm> {
  static Tensor plain(const Tensor& t) {       // contiguous bf16 or fp32 on a 16-byte boundary
    const Tensor u = t.contiguous();
    return on16(direct(u.scalar_type()) ? u : u.to(F32));
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, const OptTensor& residual, double eps) {
    Dev dev(x);
    TORCH_CHECK_VALUE(x.dim() > 0 && x.size(-1) > 0, "k_fused_rmsnorm: rows without columns, got ", x.sizes());
    const Tensor xc = plain(x), wc = plain(weight), rc = residual ? plain(residual->expand(x.sizes())) : Tensor();
    const auto d = x.size(-1), rows = x.numel() / d;
    const auto out_t = at::result_type(x, weight), sum_t = residual ? at::result_type(x, *residual) : x.scalar_type();
    Tensor out = empty_as(xc, direct(out_t) ? out_t : F32), sum = residual ? empty_as(xc, direct(sum_t) ? sum_t : F32) : Tensor();
    const Tensor rstd = empty({rows}, F32, x);
    // what backward needs: the fp32 rows (the inputs themselves where they are that) and the fp32 weight
    const bool need_y = xc.scalar_type() != F32 || residual.has_value(), need_w = wc.scalar_type() != F32;
    const Tensor y = need_y ? empty_as(xc, F32) : xc, w = need_w ? empty_as(wc, F32) : wc;
    if (rows > 0)
      check(rte_rmsnorm_op_fwd(ptr(xc), xc.scalar_type() == BF, ptr(rc), rc.defined() && rc.scalar_type() == BF, ptr(wc), wc.scalar_type() == BF,
                               need_y ? f32(y) : nullptr, ptr(out), out.scalar_type() == BF, ptr(sum), sum.defined() && sum.scalar_type() == BF, f32(rstd),
                               need_w ? f32(w) : nullptr, rows, d, eps, dev.st),
            "rte_rmsnorm_op_fwd");
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({y, w, rstd});
    ctx->saved_data["types"] = std::vector<int64_t>{int64_t(x.scalar_type()), int64_t(weight.scalar_type()), residual ? int64_t(residual->scalar_type()) : -1};
    if (out.scalar_type() != out_t) out = out.to(out_t);
    if (!residual) return {out};
    return {out, sum.scalar_type() == sum_t ? sum : sum.to(sum_t)};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &y = saved[0], &w = saved[1], &rstd = saved[2];
    Dev dev(y);
    const auto types = ctx->saved_data["types"].toIntVector();
    const bool has_res = types[2] >= 0;
    const auto d = y.size(-1), rows = y.numel() / d;
    const Tensor dy = grads[0].defined() ? plain(grads[0]) : torch::zeros_like(y);
    const Tensor dres = has_res && grads.size() > 1 && grads[1].defined() ? plain(grads[1].to(F32)) : Tensor();
    const auto x_t = at::ScalarType(types[0]);
    const bool x16 = x_t == BF;
    const bool need_f32 = !x16 || (has_res && at::ScalarType(types[2]) != BF);
    const Tensor dx32 = need_f32 ? empty_as(y, F32) : Tensor(), dx16 = x16 ? empty_as(y, BF) : Tensor();
    const int parts = 8 * rte_device_sm_count();
    const Tensor partial = empty({parts, d}, F32, y), dw = empty_as(w, F32);
    int32_t n_part = 0;
    auto as = [&](int64_t t) { return at::ScalarType(t) == BF ? (dx16.defined() ? dx16 : dx32.to(BF)) : dx32.to(at::ScalarType(t)); };
    if (rows == 0) return {as(types[0]), dw.zero_().to(at::ScalarType(types[1])), has_res ? as(types[2]) : Tensor(), Tensor()};
    check(rte_rmsnorm_bwd(f32(y), f32(w), nullptr, f32(rstd), dy.scalar_type() == BF ? ptr(dy) : nullptr, dy.scalar_type() == F32 ? f32(dy) : nullptr, f32(dres),
                          f32(dx32), ptr(dx16), f32(partial), nullptr, nullptr, rows, d, parts, &n_part, dev.st),
          "rte_rmsnorm_bwd");
    check(rte_colsum_partials(f32(partial), n_part, d, f32(dw), 0, dev.st), "rte_colsum_partials");
    return {as(types[0]), dw.to(at::ScalarType(types[1])), has_res ? as(types[2]) : Tensor(), Tensor()};
  }
};
std::tuple<Tensor, OptTensor> rmsnorm(const Tensor& x, const Tensor& w, const OptTensor& residual, double eps) {
  auto out = RmsNorm::apply(x, w, residual, eps);
  return {out[0], out.size() > 1 ? OptTensor(out[1]) : OptTensor()};
}

// --------------------------------------------------------------------------- rotary embedding
struct Bhs {                                  // a [..., S, hd] tensor as a [B, H, S, hd] view
  Tensor t;
  int64_t B, H, S, hd, strides[3];
  explicit Bhs(const Tensor& x) {
    t = x.dim() == 4 && x.stride(3) == 1 ? x : x.dim() == 3 && x.stride(2) == 1 ? x : x.contiguous();
    S = t.size(-2); hd = t.size(-1);
    if (t.dim() == 4) { B = t.size(0); H = t.size(1); strides[0] = t.stride(0); strides[1] = t.stride(1); strides[2] = t.stride(2); }
    else if (t.dim() == 3) { B = 1; H = t.size(0); strides[0] = 0; strides[1] = t.stride(0); strides[2] = t.stride(1); }
    else { t = t.contiguous(); B = 1; H = t.numel() / (S * hd); strides[0] = 0; strides[1] = S * hd; strides[2] = hd; }
  }
};
variable_list rotate(const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin, bool adjoint) {
  Dev dev(q);
  TORCH_CHECK_VALUE(q.size(-2) > 0 && q.size(-1) > 0, "k_rope_apply: no positions or no head columns, got ", q.sizes());
  auto plain = [](const Tensor& t) { return direct(t.scalar_type()) ? t : t.to(F32); };
  Tensor in[2] = {plain(q), plain(k)}, out[2];
  if (in[0].sizes() == in[1].sizes() && in[0].scalar_type() == in[1].scalar_type()) {
    const Bhs a(in[0]), b(in[1]);
    out[0] = empty_as(a.t, a.t.scalar_type()); out[1] = empty_as(b.t, b.t.scalar_type());
    const Bhs oa(out[0]), ob(out[1]);
    if (q.numel() > 0)
      check(rte_rope_views(ptr(a.t), a.strides, ptr(b.t), b.strides, ptr(oa.t), oa.strides, ptr(ob.t), ob.strides, f32(cos), f32(sin), a.B, a.H, a.S, a.hd,
                           in[0].scalar_type() == BF, adjoint, dev.st),
            "rte_rope_views");
  } else {                                    // (different head counts or types: one after the other)
    for (int i = 0; i < 2; ++i) {
      const Tensor x = in[i].contiguous();
      out[i] = empty_as(x, x.scalar_type());
      check(rte_rope_apply(ptr(x), f32(cos), f32(sin), ptr(out[i]), x.numel() / (x.size(-2) * x.size(-1)), x.size(-2), x.size(-1), x.scalar_type() == BF, adjoint,
                           dev.st),
            "rte_rope_apply");
    }
  }
  return {out[0].to(q.scalar_type()), out[1].to(k.scalar_type())};
}
struct Rope : Function<Rope> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin) {
    ctx->set_materialize_grads(false);
    const auto S = q.size(-2), hd = q.size(-1);
    const Tensor c = cos.to(F32).contiguous().view({S, hd}), s = sin.to(F32).contiguous().view({S, hd});
    ctx->save_for_backward({c, s});
    if (q.sizes() != k.sizes() || q.scalar_type() != k.scalar_type()) {      // (what backward cannot tell from the other gradient)
      ctx->saved_data["q"] = q.sizes().vec();
      ctx->saved_data["k"] = k.sizes().vec();
      ctx->saved_data["types"] = std::vector<int64_t>{int64_t(q.scalar_type()), int64_t(k.scalar_type())};
    }
    return rotate(q, k, c, s, false);
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    // (an output that no loss used: zeros of its own shape and type; q and k may differ in both)
    auto grad = [&](int i, const char* shape) {
      if (g[i].defined()) return g[i];
      if (!ctx->saved_data.count(shape)) return torch::zeros_like(g[1 - i]);
      return torch::zeros(ctx->saved_data[shape].toIntVector(), saved[0].options().dtype(at::ScalarType(ctx->saved_data["types"].toIntVector()[i])));
    };
    auto out = rotate(grad(0, "q"), grad(1, "k"), saved[0], saved[1], true);
    return {out[0], out[1], Tensor(), Tensor()};
  }
};
std::tuple<Tensor, Tensor> rope(const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin) {
  auto out = Rope::apply(q, k, cos, sin);
  return {out[0], out[1]};
}

// --------------------------------------------------------------------------- causal attention
struct Attention : Function<Attention> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& identity) {
    Dev dev(q);
    const auto B = q.size(0), H = q.size(1), S = q.size(2), hd = q.size(3);
    const bool same = q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type() && direct(q.scalar_type());
    const Bhs a(same ? q : q.to(BF)), b(same ? k : k.to(BF)), c(same ? v : v.to(BF));
    const Tensor qkv = empty({B * S, 3 * H * hd}, BF, q), y = empty({B * S, H * hd}, BF, q), lse = empty({B * H * S}, F32, q);
    check(rte_pack_qkv(ptr(a.t), a.strides, ptr(b.t), b.strides, ptr(c.t), c.strides, ptr(qkv), B, H, S, hd, a.t.scalar_type() == BF, dev.st), "rte_pack_qkv");
    check(rte_attn_fwd(ptr(qkv), 3 * H * hd, H * hd, ptr(y), H * hd, f32(lse), f32(identity), B, S, H, hd, dev.st), "rte_attn_fwd");
    ctx->save_for_backward({qkv, y, lse, identity});
    ctx->saved_data["dims"] = std::vector<int64_t>{B, H, S, hd, int64_t(q.scalar_type())};
    return {y.view({B, S, H, hd}).permute({0, 2, 1, 3}).to(q.scalar_type())};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &qkv = saved[0], &y = saved[1], &lse = saved[2];
    Dev dev(qkv);
    const auto dims = ctx->saved_data["dims"].toIntVector();
    const auto B = dims[0], H = dims[1], S = dims[2], hd = dims[3];
    Tensor dy = g[0].permute({0, 2, 1, 3});
    dy = on16(to_bf16(dev, {dy})[0]).view({B * S, H * hd});
    const Tensor dqkv = at::empty_like(qkv);
    check(rte_attn_bwd(ptr(qkv), 3 * H * hd, H * hd, ptr(y), ptr(dy), H * hd, f32(lse), ptr(dqkv), f32(saved[3]), B, S, H, hd, dev.st), "rte_attn_bwd");
    const Tensor all = dqkv.view({B, S, 3, H, hd}).permute({2, 0, 3, 1, 4}).to(at::ScalarType(dims[4]));
    return {all[0], all[1], all[2], Tensor()};
  }
};
Tensor attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& identity) { return Attention::apply(q, k, v, identity)[0]; }

// --------------------------------------------------------------------------- products
// y_i = x @ w_i, w_i [in, out_i]: one or three products that share their input (and its gradient)
struct MatmulIO : Function<MatmulIO> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w0, const OptTensor& w1, const OptTensor& w2) {
    Dev dev(x);
    const bool three = w1.has_value();
    const std::vector<Tensor> w = three ? std::vector<Tensor>{w0, *w1, *w2} : std::vector<Tensor>{w0};
    const std::vector<Tensor> conv = three ? to_bf16(dev, {x, w0, *w1, *w2}) : to_bf16(dev, {x, w0});
    ctx->set_materialize_grads(false);
    const Tensor x16 = flat2(conv[0]);
    variable_list out, saved = {x16};
    std::vector<int64_t> types = {int64_t(x.scalar_type())};
    for (size_t i = 0; i < w.size(); ++i) {
      dims8({x16.size(1), w[i].size(1)});
      const auto dt = direct(x.scalar_type()) ? x.scalar_type() : F32;
      const Tensor y = empty({x16.size(0), w[i].size(1)}, dt, x);
      mm_io(dev, x16, conv[1 + i], y);
      out.push_back(y.to(x.scalar_type()).view(with_last(x.sizes(), w[i].size(1))));
      saved.push_back(conv[1 + i]);
      types.push_back(int64_t(w[i].scalar_type()));
    }
    ctx->save_for_backward(saved);
    ctx->saved_data["types"] = types;
    ctx->saved_data["shape"] = x.sizes().vec();
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor& x16 = saved[0];
    Dev dev(x16);
    const auto types = ctx->saved_data["types"].toIntVector(), shape = ctx->saved_data["shape"].toIntVector();
    const auto M = x16.size(0), K = x16.size(1);
    const size_t n = saved.size() - 1;
    variable_list grads(4);
    // d x = sum_i dy_i @ w_i^T; with several products the sum runs in fp32 through the epilogue's residual
    const auto x_t = at::ScalarType(types[0]);
    const Tensor dx = empty({M, K}, n == 1 && direct(x_t) ? x_t : F32, x16);
    bool first = true;
    for (size_t i = 0; i < n; ++i) {
      if (!g[i].defined()) continue;
      const Tensor& w16 = saved[1 + i];
      const auto N = w16.size(1);
      const Tensor dy = to_bf16(dev, {g[i]})[0].view({M, N});
      if (M > 0) {
        Gemm p(dev, ptr(dy), N, false, ptr(w16), N, false, ptr(dx), K, M, K, N, epi_of(dx));
        if (!first) p.residual(ptr(dx), K);
        p.run();
      }
      first = false;
      grads[1 + i] = wgrad_new(dev, x16, dy, K, N, M, at::ScalarType(types[1 + i]));
    }
    if (!first) grads[0] = dx.to(x_t).view(shape);
    return grads;
  }
};
Tensor matmul_io(const Tensor& x, const Tensor& w) { return MatmulIO::apply(x, w, OptTensor(), OptTensor())[0]; }
std::tuple<Tensor, Tensor, Tensor> qkv_dense(const Tensor& x, const Tensor& wq, const Tensor& wk, const Tensor& wv) {
  auto out = MatmulIO::apply(x, wq, OptTensor(wk), OptTensor(wv));
  return {out[0], out[1], out[2]};
}

// y = x @ w^T, w [out, in]
struct MatmulOI : Function<MatmulOI> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& w) {
    Dev dev(x);
    const auto conv = to_bf16(dev, {x, w});
    const Tensor x16 = flat2(conv[0]);
    dims8({x16.size(1)});
    const auto dt = direct(x.scalar_type()) ? x.scalar_type() : F32;
    const Tensor y = empty({x16.size(0), w.size(0)}, dt, x);
    mm_oi(dev, x16, conv[1], y);
    ctx->save_for_backward({x16, conv[1]});
    ctx->saved_data["types"] = std::vector<int64_t>{int64_t(x.scalar_type()), int64_t(w.scalar_type())};
    ctx->saved_data["shape"] = x.sizes().vec();
    return {y.to(x.scalar_type()).view(with_last(x.sizes(), w.size(0)))};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x16 = saved[0], &w16 = saved[1];
    Dev dev(x16);
    const auto types = ctx->saved_data["types"].toIntVector();
    const auto M = x16.size(0), K = x16.size(1), N = w16.size(0);
    dims8({N});
    const Tensor dy = to_bf16(dev, {g[0]})[0].view({M, N});
    const auto x_t = at::ScalarType(types[0]);
    const Tensor dx = empty({M, K}, direct(x_t) ? x_t : F32, x16);
    mm_io(dev, dy, w16, dx);                                           // dy [M, out] . w [out, in]
    return {dx.to(x_t).view(ctx->saved_data["shape"].toIntVector()), wgrad_new(dev, dy, x16, N, K, M, at::ScalarType(types[1]))};
  }
};
Tensor matmul_oi(const Tensor& x, const Tensor& w) { return MatmulOI::apply(x, w)[0]; }

// x @ wo[row_indices, :]
struct OutProj : Function<OutProj> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wo, const Tensor& rows) {
    Dev dev(x);
    const Tensor idx = rows.to(torch::kInt32).contiguous();
    const auto n = idx.numel(), dout = wo.size(1);
    dims8({n, dout});
    const auto conv = to_bf16(dev, {x, wo});
    const Tensor x16 = conv[0].view({-1, n}), sel = empty({n, dout}, BF, x);
    check(rte_gather_rows(ptr(conv[1]), i32(idx), ptr(sel), n, dout * 2, dev.st), "rte_gather_rows");
    const auto dt = direct(x.scalar_type()) ? x.scalar_type() : F32;
    const Tensor y = empty({x16.size(0), dout}, dt, x);
    mm_io(dev, x16, sel, y);
    ctx->save_for_backward({x16, sel, idx});
    ctx->saved_data["types"] = std::vector<int64_t>{int64_t(x.scalar_type()), int64_t(wo.scalar_type())};
    ctx->saved_data["shape"] = x.sizes().vec();
    ctx->saved_data["wshape"] = wo.sizes().vec();
    return {y.to(x.scalar_type()).view(with_last(x.sizes(), dout))};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x16 = saved[0], &sel = saved[1], &idx = saved[2];
    Dev dev(x16);
    const auto types = ctx->saved_data["types"].toIntVector(), wshape = ctx->saved_data["wshape"].toIntVector();
    const auto M = x16.size(0), n = x16.size(1), dout = sel.size(1);
    const Tensor dy = to_bf16(dev, {g[0]})[0].view({M, dout});
    const auto x_t = at::ScalarType(types[0]);
    const Tensor dx = empty({M, n}, direct(x_t) ? x_t : F32, x16);
    mm_oi(dev, dy, sel, dx);
    const Tensor dsel = wgrad_new(dev, x16, dy, n, dout, M, F32), dwo = torch::zeros(wshape, x16.options().dtype(F32));
    check(rte_scatter_add_rows_f32(f32(dwo), i32(idx), f32(dsel), n, dout, dev.st), "rte_scatter_add_rows_f32");
    return {dx.to(x_t).view(ctx->saved_data["shape"].toIntVector()), dwo.to(at::ScalarType(types[1])), Tensor()};
  }
};
Tensor out_proj(const Tensor& x, const Tensor& wo, const Tensor& rows) { return OutProj::apply(x, wo, rows)[0]; }

// --------------------------------------------------------------------------- cross entropy
struct CrossEntropy : Function<CrossEntropy> {
  static void run(const Dev& dev, const Tensor& lg, const Tensor& tg, const Tensor& weight, const Tensor& loss, const Tensor& grad) {
    const auto rows = lg.size(0), V = lg.size(1);
    if (rows == 0) return;
    if (lg.scalar_type() == BF)
      check(rte_ce_fwd_bwd(ptr(lg), V, tg.data_ptr<int64_t>(), f32(weight), 1, f32(loss), ptr(grad), rows, V, dev.status, dev.st), "rte_ce_fwd_bwd");
    else
      check(rte_ce_fwd_bwd_f32(f32(lg), V, tg.data_ptr<int64_t>(), f32(weight), 1, f32(loss), f32(grad), rows, V, dev.status, dev.st), "rte_ce_fwd_bwd_f32");
  }
  static variable_list forward(AutogradContext* ctx, const Tensor& logits, const Tensor& targets) {
    Dev dev(logits);
    const auto V = logits.size(-1);
    Tensor lg = logits.contiguous();
    if (!direct(lg.scalar_type())) lg = lg.to(F32);
    lg = lg.view({-1, V});
    const Tensor tg = targets.to(torch::kInt64).contiguous().view({-1}), loss = empty({lg.size(0)}, F32, logits);
    Tensor lse;                                                           // long rows: kept, so that the gradient is one pass
    if (lg.size(0) > 0 && V * lg.element_size() > 16 * 1024 - 32) {
      lse = empty({lg.size(0)}, F32, logits);
      const int rc = rte_ce_loss_lse(ptr(lg), lg.scalar_type() == F32, V, tg.data_ptr<int64_t>(), f32(loss), f32(lse), lg.size(0), V, dev.status, dev.st);
      if (rc == RTE_ERR_UNSUPPORTED) lse = Tensor();
      else check(rc, "rte_ce_loss_lse");
    }
    if (!lse.defined()) run(dev, lg, tg, Tensor(), loss, Tensor());
    ctx->save_for_backward({lg, tg, lse});
    ctx->saved_data["shape"] = logits.sizes().vec();
    ctx->saved_data["type"] = int64_t(logits.scalar_type());
    return {loss.view(targets.sizes())};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &lg = saved[0], &tg = saved[1], &lse = saved[2];
    Dev dev(lg);
    const Tensor grad = at::empty_like(lg), dloss = g[0].to(F32).contiguous();         // (softmax - onehot) * dloss[row]
    int rc = RTE_ERR_UNSUPPORTED;
    if (lse.defined()) {
      rc = rte_ce_gradient(ptr(lg), lg.scalar_type() == F32, lg.size(1), tg.data_ptr<int64_t>(), f32(dloss), 1, f32(lse), ptr(grad), lg.size(0), lg.size(1),
                           dev.status, dev.st);
      if (rc != RTE_ERR_UNSUPPORTED) check(rc, "rte_ce_gradient");           // (saved-tensor hooks may bring the logits back on another boundary)
    }
    if (rc == RTE_ERR_UNSUPPORTED) run(dev, lg, tg, dloss, empty({lg.size(0)}, F32, lg), grad);
    return {grad.to(at::ScalarType(ctx->saved_data["type"].toInt())).view(ctx->saved_data["shape"].toIntVector()), Tensor()};
  }
};
Tensor cross_entropy(const Tensor& logits, const Tensor& targets) { return CrossEntropy::apply(logits, targets)[0]; }

// --------------------------------------------------------------------------- packed SwiGLU FFN
struct PackedFfn : Function<PackedFfn> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wug, const Tensor& wdown) {
    Dev dev(x);
    const auto N = x.size(0), d = x.size(1), m = wug.size(0) / 2;
    const auto conv = to_bf16(dev, {x, wug, wdown});
    const Tensor &x16 = conv[0], &wug16 = conv[1], &wd16 = conv[2];
    const Tensor ug = empty({N, 2 * m}, BF, x), z = empty({N, m}, BF, x), y = empty({N, wdown.size(1)}, direct(x.scalar_type()) ? x.scalar_type() : F32, x);
    if (N > 0) {
      if (m % 64 == 0 && N * m >= rte_swiglu_fuse_min_fwd(d)) {
        Gemm(dev, ptr(x16), d, false, ptr(wug16), d, false, ptr(z), m, N, 2 * m, d, RTE_EPI_SWIGLU_FWD).pair(ptr(ug), 2 * m, m).run();
      } else {
        mm_oi(dev, x16, wug16, ug);
        check(rte_swiglu_fwd(ptr(ug), ptr(z), N, m, dev.st), "rte_swiglu_fwd");
      }
      mm_io(dev, z, wd16, y);
    }
    ctx->save_for_backward({x16, wug16, wd16, ug, z});
    ctx->saved_data["types"] = std::vector<int64_t>{int64_t(x.scalar_type()), int64_t(wug.scalar_type()), int64_t(wdown.scalar_type())};
    return {y.to(x.scalar_type())};
  }
  static variable_list backward(AutogradContext* ctx, variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x16 = saved[0], &wug16 = saved[1], &wd16 = saved[2], &ug = saved[3], &z = saved[4];
    Dev dev(x16);
    const auto types = ctx->saved_data["types"].toIntVector();
    const auto N = x16.size(0), d = x16.size(1), m = wd16.size(0), dout = wd16.size(1);
    const Tensor dy = to_bf16(dev, {g[0]})[0], dug = empty({N, 2 * m}, BF, x16);
    const auto x_t = at::ScalarType(types[0]);
    const Tensor dx = empty({N, d}, direct(x_t) ? x_t : F32, x16);
    if (N > 0) {
      if (m % 64 == 0 && N * m >= rte_swiglu_fuse_min(1)) {
        Gemm(dev, ptr(dy), dout, false, ptr(wd16), dout, false, ptr(dug), 2 * m, N, m, dout, RTE_EPI_SWIGLU_BWD).residual(ptr(ug), 2 * m).pair(nullptr, 0, m).run();
      } else {
        const Tensor dz = empty({N, m}, BF, x16);
        mm_oi(dev, dy, wd16, dz);
        check(rte_swiglu_bwd(ptr(ug), ptr(dz), ptr(dug), N, m, dev.st), "rte_swiglu_bwd");
      }
      mm_io(dev, dug, wug16, dx);
    }
    return {dx.to(x_t), wgrad_new(dev, dug, x16, 2 * m, d, N, at::ScalarType(types[1])), wgrad_new(dev, z, dy, m, dout, N, at::ScalarType(types[2]))};
  }
};
Tensor packed_ffn(const Tensor& x, const Tensor& wug, const Tensor& wdown) { return PackedFfn::apply(x, wug, wdown)[0]; }

// --------------------------------------------------------------------------- cluster-pool FFN (buffers: cluster_pool.py)
void cast_into(const Dev& dev, const Tensor& src, const Tensor& dst) {
  if (src.scalar_type() == F32) check(rte_cast_f32_bf16(f32(src), ptr(dst), src.numel(), dev.st), "rte_cast_f32_bf16");
  else dst.copy_(src);
}

// What a caller hands a module beside x is read and written through raw pointers sized by the module: checked here, before
// any launch.
void is_dense_f32(const Tensor& t, const Tensor& like, int64_t numel, const char* what) {
  TORCH_CHECK_VALUE(t.device() == like.device() && t.scalar_type() == F32 && t.is_contiguous() && t.numel() == numel, what,
                    " must be a contiguous fp32 tensor of ", numel, " elements on ", like.device(), ", got ", t.sizes(), " ", t.scalar_type(), " on ", t.device());
}
Tensor token_rows(const Tensor& x, int64_t d) {
  TORCH_CHECK_VALUE(x.dim() > 0 && x.size(-1) == d, "the last dimension must be d_model = ", d, ", got ", x.sizes());
  const Tensor flat = x.reshape({-1, d}).contiguous();
  return direct(flat.scalar_type()) ? flat : flat.to(F32);
}

struct PoolModule {
  Tensor status, selector16, centers, idx_ug, idx_d, ug_ptr, ug_rows, d_ptr, d_rows, wdT16, wug_pool, wd_pool, q, assign, pos, perm, tile_group, counts,
      offsets, kblocks, x16, xp, ugp, zp, yp, dyp, dzp, dugp, dxp, dwug_pool, dwd_pool, dwdT;
  int64_t rank = 0, C = 0, Mc = 0, cap = 0, d = 0, F = 0, tokens = 0;

  explicit PoolModule(const std::map<std::string, Tensor>& t, const std::map<std::string, int64_t>& n) {
    const std::pair<const char*, Tensor*> fields[] = {
        {"status", &status}, {"selector16", &selector16}, {"centers", &centers}, {"idx_ug", &idx_ug}, {"idx_d", &idx_d}, {"ug_ptr", &ug_ptr},
        {"ug_rows", &ug_rows}, {"d_ptr", &d_ptr}, {"d_rows", &d_rows}, {"wdT16", &wdT16}, {"wug_pool", &wug_pool}, {"wd_pool", &wd_pool},
        {"q", &q}, {"assign", &assign}, {"pos", &pos}, {"perm", &perm}, {"tile_group", &tile_group}, {"counts", &counts}, {"offsets", &offsets},
        {"kblocks", &kblocks}, {"x16", &x16}, {"xp", &xp}, {"ugp", &ugp}, {"zp", &zp}, {"yp", &yp}, {"dyp", &dyp}, {"dzp", &dzp}, {"dugp", &dugp}, {"dxp", &dxp},
        {"dwug_pool", &dwug_pool}, {"dwd_pool", &dwd_pool}, {"dwdT", &dwdT}};
    for (const auto& [name, to] : fields) *to = t.at(name);
    rank = n.at("rank"); C = n.at("C"); Mc = n.at("Mc"); cap = n.at("cap"); d = n.at("d"); F = n.at("F");
  }

  void route(const Dev& dev, const Tensor& flat) {
    const auto N = flat.size(0);
    cast_into(dev, flat, x16.narrow(0, 0, N));
    Gemm(dev, ptr(x16), d, false, ptr(selector16), d, false, ptr(q), 2 * rank, N, 2 * rank, d, RTE_EPI_F32).run();
    check(rte_cluster_route(f32(q), 2 * rank, f32(centers), i32(assign), nullptr, N, 2 * rank, C, dev.st), "rte_cluster_route");
  }
  void pack(const Dev& dev, const Tensor& a) {
    check(rte_cluster_pack(i32(a), a.numel(), C, perm.numel(), i32(perm), i32(pos), i32(counts), i32(offsets), i32(tile_group), i32(kblocks), dev.status, dev.st),
          "rte_cluster_pack");
  }
  void prepare_pools(const Dev& dev, const Tensor& wug, const Tensor& wd) {
    gather(dev, wug, idx_ug, wug_pool);
    check(rte_transpose_f32(f32(wd), ptr(wdT16), d, F, 1, 0, dev.st), "rte_transpose_f32");
    check(rte_gather_rows(ptr(wdT16), i32(idx_d), ptr(wd_pool), idx_d.numel(), d * 2, dev.st), "rte_gather_rows");
  }
  void gather(const Dev& dev, const Tensor& src, const Tensor& idx, const Tensor& dst) {
    check(rte_gather_rows_convert(ptr(src), src.scalar_type() == BF, i32(idx), ptr(dst), dst.scalar_type() == BF, idx.numel(), d, dev.st), "rte_gather_rows_convert");
  }

  Tensor forward(const Tensor& x, const Tensor& wug, const Tensor& wd, const OptTensor& assignments) {
    Dev dev(x, status);
    const Tensor flat = token_rows(x, d);
    const auto N = flat.size(0);
    TORCH_CHECK_VALUE(N <= x16.size(0), N, " tokens exceed max_tokens=", x16.size(0));
    is_dense_f32(wug, x, 2 * F * d, "wug");
    is_dense_f32(wd, x, F * d, "wd");
    if (assignments)
      TORCH_CHECK_VALUE(assignments->device() == x.device() && assignments->numel() == N, "assignments must name the cluster of each of the ", N, " tokens on ",
                        x.device(), ", got ", assignments->sizes(), " on ", assignments->device());
    tokens = N;
    Tensor a = assign.narrow(0, 0, N);
    if (assignments) a = assignments->to(torch::kInt32).contiguous().view({-1});
    else route(dev, flat);
    pack(dev, a);
    prepare_pools(dev, wug, wd);
    gather(dev, flat, perm, xp);                                              // pack + cast, zero padding rows
    Gemm(dev, ptr(xp), d, false, ptr(wug_pool), d, false, ptr(ugp), 2 * Mc, cap, 2 * Mc, d, RTE_EPI_BF16).groups(tile_group, C, 2 * Mc).run();
    check(rte_swiglu_fwd(ptr(ugp), ptr(zp), cap, Mc, dev.st), "rte_swiglu_fwd");
    Gemm(dev, ptr(zp), Mc, false, ptr(wd_pool), d, true, ptr(yp), d, cap, d, Mc, RTE_EPI_F32).groups(tile_group, C, Mc).run();
    const Tensor out = empty({N, d}, F32, x);
    gather(dev, yp, pos.narrow(0, 0, N), out);
    return out.view(x.sizes());
  }

  Tensor backward(const Tensor& dout, const Tensor& dwug, const Tensor& dwd, bool accumulate) {
    Dev dev(dout, status);
    const Tensor flat = token_rows(dout, d);
    TORCH_CHECK_VALUE(flat.size(0) == tokens, "the gradient of ", tokens, " tokens has ", flat.size(0), " rows");
    is_dense_f32(dwug, dout, 2 * F * d, "dwug");
    is_dense_f32(dwd, dout, F * d, "dwd");
    gather(dev, flat, perm, dyp);
    Gemm(dev, ptr(dyp), d, false, ptr(wd_pool), d, false, ptr(dzp), Mc, cap, Mc, d, RTE_EPI_BF16).groups(tile_group, C, Mc).run();
    check(rte_swiglu_bwd(ptr(ugp), ptr(dzp), ptr(dugp), cap, Mc, dev.st), "rte_swiglu_bwd");
    Gemm(dev, ptr(dugp), 2 * Mc, false, ptr(wug_pool), d, true, ptr(dxp), d, cap, d, 2 * Mc, RTE_EPI_F32).groups(tile_group, C, 2 * Mc).run();
    // per-cluster weight gradients: the reduction runs over the cluster's packed rows (ragged split-K)
    Gemm(dev, ptr(zp), Mc, true, ptr(dyp), d, true, ptr(dwd_pool), d, Mc, d, cap, RTE_EPI_F32).split(C, Mc * d, i32(kblocks)).run();
    Gemm(dev, ptr(dugp), 2 * Mc, true, ptr(xp), d, true, ptr(dwug_pool), d, 2 * Mc, d, cap, RTE_EPI_F32).split(C, 2 * Mc * d, i32(kblocks)).run();
    check(rte_csr_row_reduce_f32(f32(dwug_pool), i32(ug_ptr), i32(ug_rows), f32(dwug), 2 * F, d, accumulate, dev.st), "rte_csr_row_reduce_f32");
    check(rte_csr_row_reduce_f32(f32(dwd_pool), i32(d_ptr), i32(d_rows), f32(dwdT), F, d, 0, dev.st), "rte_csr_row_reduce_f32");
    check(rte_transpose_f32(f32(dwdT), ptr(dwd), F, d, 0, accumulate, dev.st), "rte_transpose_f32");
    const Tensor dx = empty({tokens, d}, F32, dout);
    gather(dev, dxp, pos.narrow(0, 0, tokens), dx);
    return dx.view(dout.sizes());
  }
};

// --------------------------------------------------------------------------- SVD-factor sparse FFN (buffers: svd_ffn.py)
struct SvdModule {
  Tensor status, selector16, up_b16, gate_b16, wug16, wd16, wn, x16, q16, hats, ug, z, selected, cand_count, dout16, dz, dug, dwug;
  int64_t rank = 0, F = 0, d = 0, up_m = 0, gate_m = 0, product_m = 0, top_k = 0, tokens = 0;

  explicit SvdModule(const std::map<std::string, Tensor>& t, const std::map<std::string, int64_t>& n) {
    const std::pair<const char*, Tensor*> fields[] = {{"status", &status}, {"selector16", &selector16}, {"up_b16", &up_b16},
                                                      {"gate_b16", &gate_b16}, {"wug16", &wug16}, {"wd16", &wd16}, {"wn", &wn}, {"x16", &x16}, {"q16", &q16},
                                                      {"hats", &hats}, {"ug", &ug}, {"z", &z}, {"selected", &selected}, {"cand_count", &cand_count},
                                                      {"dout16", &dout16}, {"dz", &dz}, {"dug", &dug}, {"dwug", &dwug}};
    for (const auto& [name, to] : fields) *to = t.at(name);
    rank = n.at("rank"); F = n.at("F"); d = n.at("d"); up_m = n.at("up_m"); gate_m = n.at("gate_m"); product_m = n.at("product_m"); top_k = n.at("top_k");
  }

  Tensor forward(const Tensor& x, const Tensor& w_up, const Tensor& w_gate, const Tensor& w_down) {
    Dev dev(x, status);
    const Tensor flat = token_rows(x, d);
    const auto N = flat.size(0);
    TORCH_CHECK_VALUE(N <= x16.size(0), N, " tokens exceed max_tokens=", x16.size(0));
    is_dense_f32(w_up, x, F * d, "w_up");
    is_dense_f32(w_gate, x, F * d, "w_gate");
    is_dense_f32(w_down, x, F * d, "w_down");
    tokens = N;
    const auto* qb = static_cast<char*>(ptr(q16));
    auto* hb = f32(hats);
    {
      const float* src[4] = {f32(w_up), f32(w_gate), f32(w_down), f32(flat)};
      void* dst[4] = {ptr(wug16), static_cast<char*>(ptr(wug16)) + F * d * 2, ptr(wd16), ptr(x16)};
      const int64_t n[4] = {F * d, F * d, F * d, N * d};
      const bool x_too = flat.scalar_type() == F32;
      check(rte_cast_many_f32_bf16(src, dst, n, x_too ? 4 : 3, dev.st), "rte_cast_many_f32_bf16");
      if (!x_too) x16.narrow(0, 0, N).copy_(flat);
    }
    check(rte_row_norm_f32(f32(w_down), f32(wn), F, d, dev.st), "rte_row_norm_f32");
    Gemm(dev, ptr(x16), d, false, ptr(selector16), d, false, ptr(q16), 2 * rank, N, 2 * rank, d, RTE_EPI_BF16).run();
    Gemm(dev, ptr(q16), 2 * rank, false, ptr(up_b16), F, true, hb, 2 * F, N, F, rank, RTE_EPI_F32).run();
    Gemm(dev, qb + rank * 2, 2 * rank, false, ptr(gate_b16), F, true, hb + F, 2 * F, N, F, rank, RTE_EPI_F32).run();
    Gemm(dev, ptr(x16), d, false, ptr(wug16), d, false, ptr(ug), 2 * F, N, 2 * F, d, RTE_EPI_BF16).run();
    check(rte_svd_ffn_select(f32(hats), ptr(ug), f32(wn), ptr(z), static_cast<uint8_t*>(ptr(selected)), i32(cand_count), N, F, up_m, gate_m, product_m, top_k, dev.st),
          "rte_svd_ffn_select");
    const Tensor out = empty({N, d}, F32, x);
    Gemm(dev, ptr(z), F, false, ptr(wd16), d, true, ptr(out), d, N, d, F, RTE_EPI_F32).run();
    return out.view(x.sizes());
  }

  // dw_up and dw_gate may be the two halves of one [2F, d] tensor: the product then writes them itself
  Tensor backward(const Tensor& dout, const Tensor& dw_up, const Tensor& dw_gate, const Tensor& dw_down) {
    Dev dev(dout, status);
    const Tensor flat = token_rows(dout, d);
    const auto N = tokens;
    TORCH_CHECK_VALUE(flat.size(0) == N, "the gradient of ", N, " tokens has ", flat.size(0), " rows");
    is_dense_f32(dw_down, dout, F * d, "dw_down");
    cast_into(dev, flat, dout16.narrow(0, 0, N));
    // Where the product's epilogue takes the mask, d z does not go through memory: two passes over [N, F] less, and the bits of the two launches
    // (d z rounded to bf16, the same divide), so that a gradient does not depend on which of them its size takes.
    // us, two launches -> one: 16384 x 2048 x 512 101.5 -> 84.6, 8192 x 4096 x 1024 121.4 -> 95.0, 8192 x 2048 x 512 55.8 -> 50.9, 2048 x 2048 x 512 18.5 -> 17.9,
    // 5000 x 1536 x 384 26.5 -> 28.1 (d z stays in L2 there), 512 x 2048 x 512 9.7 -> 9.1.
    int rc = RTE_ERR_UNSUPPORTED;
    if (N * F >= rte_swiglu_fuse_min(1)) {
      Gemm fused(dev, ptr(dout16), d, false, ptr(wd16), d, false, ptr(dug), 2 * F, N, F, d, RTE_EPI_SWIGLU_BWD);
      fused.residual(ptr(ug), 2 * F).pair(nullptr, 0, F);
      rc = rte_svd_ffn_hidden_bwd(&fused.a, static_cast<uint8_t*>(ptr(selected)), dev.st);
      if (rc != RTE_ERR_UNSUPPORTED) check(rc, "rte_svd_ffn_hidden_bwd");
    }
    if (rc == RTE_ERR_UNSUPPORTED) {
      Gemm(dev, ptr(dout16), d, false, ptr(wd16), d, false, ptr(dz), F, N, F, d, RTE_EPI_BF16).run();
      check(rte_svd_ffn_swiglu_bwd(ptr(ug), ptr(dz), static_cast<uint8_t*>(ptr(selected)), ptr(dug), N, F, dev.st), "rte_svd_ffn_swiglu_bwd");
    }
    const Tensor dx = empty({N, d}, F32, dout);
    Gemm(dev, ptr(dug), 2 * F, false, ptr(wug16), d, true, ptr(dx), d, N, d, 2 * F, RTE_EPI_F32).run();
    const bool halves = dw_up.scalar_type() == F32 && dw_gate.scalar_type() == F32 && dw_up.is_contiguous() && dw_gate.is_contiguous() &&
                        f32(dw_gate) == f32(dw_up) + F * d;
    float* both = halves ? f32(dw_up) : f32(dwug);
    wgrad(dev, dug, x16, both, 2 * F, d, N);
    if (!halves) {
      const_cast<Tensor&>(dw_up).copy_(dwug.narrow(0, 0, F));
      const_cast<Tensor&>(dw_gate).copy_(dwug.narrow(0, F, F));
    }
    wgrad(dev, z, dout16, f32(dw_down), F, d, N);
    return dx.view(dout.sizes());
  }
};

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  m.def("bind_status", &bind_status);
  m.def("rmsnorm", &rmsnorm);
  m.def("rope", &rope);
  m.def("attention", &attention);
  m.def("matmul_io", &matmul_io);
  m.def("qkv_dense", &qkv_dense);
  m.def("matmul_oi", &matmul_oi);
  m.def("out_proj", &out_proj);
  m.def("cross_entropy", &cross_entropy);
  m.def("packed_ffn", &packed_ffn);
  pybind11::class_<PoolModule>(m, "PoolModule")
      .def(pybind11::init<const std::map<std::string, Tensor>&, const std::map<std::string, int64_t>&>())
      .def("forward", &PoolModule::forward)
      .def("backward", &PoolModule::backward)
      .def_readonly("tokens", &PoolModule::tokens);
  pybind11::class_<SvdModule>(m, "SvdModule")
      .def(pybind11::init<const std::map<std::string, Tensor>&, const std::map<std::string, int64_t>&>())
      .def("forward", &SvdModule::forward)
      .def("backward", &SvdModule::backward)
      .def_readonly("tokens", &SvdModule::tokens);
}
