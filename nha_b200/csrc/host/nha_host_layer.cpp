// Host side of the operators that a layer runs around the attention operator: slot gates, rotary, feature maps, silu + RMS
// norm, and the consumers of the two log-sum-exps.  One autograd node each.
#include <string.h>

#include <map>
#include <mutex>

#include "nha_host.h"

namespace nha_host {

using torch::autograd::AutogradContext;
using torch::autograd::Function;
using torch::autograd::variable_list;

static Tensor back_to(const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt ? t : t.to(dt); }
static int64_t type_int(at::ScalarType t) { return (int64_t)t; }
static at::ScalarType type_of(const c10::IValue& v) { return (at::ScalarType)v.toInt(); }

// ---- slot gates (nha_fla/layers/nha.py:229-231) ----------------------------------------------------------------------
struct SlotGates : Function<SlotGates> {
  static variable_list forward(AutogradContext* ctx, const Tensor& f, double normalizer) {
    ctx->set_materialize_grads(false);
    const c10::cuda::OptionalCUDAGuard guard(f.device());
    const Tensor fc = bf16c(f);
    const Tensor g = empty_same(fc), s = empty_same(fc);
    if (fc.numel())
      check(nha_slot_gates_fwd(fc.data_ptr(), g.data_ptr(), s.data_ptr(), fc.numel(), (float)normalizer, stream_of(fc)), "nha_slot_gates_fwd");
    ctx->save_for_backward({fc});
    ctx->saved_data["n"] = normalizer;
    ctx->saved_data["t"] = type_int(f.scalar_type());
    return {g, s};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const Tensor fc = ctx->get_saved_variables()[0];
    if (!grads[0].defined() && !grads[1].defined()) return {Tensor(), Tensor()};
    const c10::cuda::OptionalCUDAGuard guard(fc.device());
    const Tensor dg = grads[0].defined() ? bf16c(grads[0]) : Tensor(), ds = grads[1].defined() ? bf16c(grads[1]) : Tensor();
    const Tensor df = empty_same(fc);
    if (fc.numel())
      check(nha_slot_gates_bwd(fc.data_ptr(), ptr(dg), ptr(ds), df.data_ptr(), fc.numel(), (float)ctx->saved_data["n"].toDouble(),
                               stream_of(fc)), "nha_slot_gates_bwd");
    return {back_to(df, type_of(ctx->saved_data["t"])), Tensor()};
  }
};

// slot_gates(f, normalizer) -> (g, s)
NHA_METHOD(slot_gates) {
  NHA_BEGIN(2)
  const Tensor& f = tensor(args[0], "f");
  const double n = real(args[1]);
  require(f.is_cuda(), "slot_gates runs on the CUDA library only (there is no CPU path)");
  require(n > 0, "gate_logit_normalizer must be positive");
  variable_list out;
  {
    pybind11::gil_scoped_release no_gil;
    out = SlotGates::apply(f, n);
  }
  return tuple({wrap(out[0]), wrap(out[1])});
  NHA_END
}

// ---- rotary of q and k (nha_fla/layers/nha.py:145, 235) --------------------------------------------------------------
static variable_list rotate(const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin, const Tensor& cu, int64_t offset,
                            int64_t T, int inverse) {
  const Tensor qo = empty_same(q), ko = empty_same(k);
  const int64_t K = q.size(-1), HQ = q.size(-2), Ttot = HQ * K ? q.numel() / (HQ * K) : 0;
  if (Ttot)
    check(nha_rope_pair(q.data_ptr(), k.data_ptr(), qo.data_ptr(), ko.data_ptr(), cos.data_ptr(), sin.data_ptr(), cos.stride(0),
                        (int)cos.size(0), (const int32_t*)ptr(cu), cu.defined() ? (int)cu.numel() - 1 : 0, (int)T, Ttot, (int)HQ,
                        (int)k.size(-2), (int)K, (int)offset, inverse, stream_of(q)), "nha_rope_pair");
  return {qo, ko};
}

struct RotaryPair : Function<RotaryPair> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& cos, const Tensor& sin,
                               const std::optional<Tensor>& cu, int64_t offset, int64_t T) {
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    const Tensor c = cu.has_value() ? *cu : Tensor();
    ctx->save_for_backward({cos, sin, c});
    ctx->saved_data["o"] = offset;
    ctx->saved_data["T"] = T;
    ctx->saved_data["q"] = type_int(q.scalar_type());
    ctx->saved_data["k"] = type_int(k.scalar_type());
    return rotate(bf16c(q), bf16c(k), cos, sin, c, offset, T, 0);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list sv = ctx->get_saved_variables();
    const c10::cuda::OptionalCUDAGuard guard(grads[0].device());
    const variable_list g = rotate(bf16c(grads[0]), bf16c(grads[1]), sv[0], sv[1], sv[2], ctx->saved_data["o"].toInt(),
                                   ctx->saved_data["T"].toInt(), 1);
    return {back_to(g[0], type_of(ctx->saved_data["q"])), back_to(g[1], type_of(ctx->saved_data["k"])), Tensor(), Tensor(), Tensor(),
            Tensor(), Tensor()};
  }
};

// rotary_pair(q, k, cos, sin, seqlen_offset, cu_seqlens) -> (q_rot, k_rot)
NHA_METHOD(rotary_pair) {
  NHA_BEGIN(6)
  const Tensor& q = tensor(args[0], "q");
  const Tensor& k = tensor(args[1], "k");
  const Tensor& cos = tensor(args[2], "cos");
  const Tensor& sin = tensor(args[3], "sin");
  const long offset = integer(args[4]);
  require(q.is_cuda() && k.is_cuda(), "rotary_pair runs on the CUDA library only (there is no CPU path)");
  require(q.dim() == 4 && k.dim() == 4 && q.size(0) == k.size(0) && q.size(1) == k.size(1) && q.size(3) == k.size(3),
          "q [B,T,HQ,K] and k [B,T,H,K] must hold the same tokens");
  const int64_t B = q.size(0), T = q.size(1), K = q.size(3);
  require(K % 16 == 0, "head dim must be a multiple of 16");
  require(cos.dim() == 2 && cos.sizes() == sin.sizes() && (cos.size(1) == K / 2 || cos.size(1) == K), "cos/sin must be [P, K/2] or [P, K]");
  require(offset >= 0, "seqlen_offset must not be negative");
  std::optional<Tensor> cu;
  if (args[5] != Py_None) {
    require(B == 1, "packed input has batch size 1");
    cu = typed(tensor(args[5], "cu_seqlens"), at::kInt);
  } else {
    require(offset + T <= cos.size(0), "cos/sin tables do not cover the positions");
  }
  same_device(q, {&k, &cos, &sin}, "rotary_pair");
  if (cu) same_device(q, {&*cu}, "rotary_pair");
  variable_list out;
  {
    pybind11::gil_scoped_release no_gil;
    Tensor c, s;
    {
      at::AutoGradMode off(false);
      c = bf16c(cos);
      s = bf16c(sin);
      if (c.size(1) % 8) {                                   // rows of 16-byte pieces
        const int64_t pad = 8 - c.size(1) % 8;
        c = at::constant_pad_nd(c, {0, pad});
        s = at::constant_pad_nd(s, {0, pad});
      }
    }
    out = RotaryPair::apply(q, k, c, s, cu, (int64_t)offset, T);
  }
  return tuple({wrap(out[0]), wrap(out[1])});
  NHA_END
}

// ---- feature map of q and k, silu(v) (nha_fla/layers/nha.py:219-223) -------------------------------------------------
// up to three tensors per launch; an undefined tensor is left out
static void activate(const Tensor* x, const Tensor* dy, Tensor* y, const int* relu) {
  const void *xp[3], *dp[3];
  void* yp[3];
  int64_t n[3];
  int flag[3], count = 0;
  for (int i = 0; i < 3; ++i) {
    if (!x[i].defined()) continue;
    y[i] = empty_same(x[i]);
    xp[count] = x[i].data_ptr();
    dp[count] = dy ? dy[i].data_ptr() : nullptr;
    yp[count] = y[i].data_ptr();
    n[count] = x[i].numel();
    flag[count++] = relu[i];
  }
  void* st = stream_of(x[2]);
  if (dy) check(nha_act3_bwd(xp, dp, yp, n, flag, count, st), "nha_act3_bwd");
  else check(nha_act3_fwd(xp, yp, n, flag, count, st), "nha_act3_fwd");
}

struct FeatureMaps : Function<FeatureMaps> {
  static variable_list forward(AutogradContext* ctx, const std::optional<Tensor>& q, const std::optional<Tensor>& k, const Tensor& v,
                               bool relu) {
    const c10::cuda::OptionalCUDAGuard guard(v.device());
    Tensor x[3], y[3];
    if (q.has_value()) { x[0] = bf16c(*q); x[1] = bf16c(*k); }
    x[2] = bf16c(v);
    const int flags[3] = {relu, relu, 0};
    activate(x, nullptr, y, flags);
    ctx->save_for_backward({x[0], x[1], x[2]});
    ctx->saved_data["r"] = relu;
    ctx->saved_data["q"] = type_int(q.has_value() ? q->scalar_type() : at::kBFloat16);
    ctx->saved_data["k"] = type_int(q.has_value() ? k->scalar_type() : at::kBFloat16);
    ctx->saved_data["v"] = type_int(v.scalar_type());
    if (!q.has_value()) return {y[2]};
    return {y[0], y[1], y[2]};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list x = ctx->get_saved_variables();
    const c10::cuda::OptionalCUDAGuard guard(x[2].device());
    const int relu = ctx->saved_data["r"].toBool();
    const int flags[3] = {relu, relu, 0};
    Tensor dy[3], dx[3];
    const bool all = x[0].defined();
    for (int i = 0; i < 3; ++i)
      if (x[i].defined()) dy[i] = bf16c(grads[all ? i : 0]);
    activate(x.data(), dy, dx, flags);
    static const char* key[3] = {"q", "k", "v"};
    for (int i = 0; i < 3; ++i)
      if (dx[i].defined()) dx[i] = back_to(dx[i], type_of(ctx->saved_data[key[i]]));
    return {dx[0], dx[1], dx[2], Tensor()};
  }
};

// feature_maps(q, k, v, mode) with mode 0 = swish, 1 = relu, 2 = silu(v) alone -> (q', k', v')
NHA_METHOD(feature_maps) {
  NHA_BEGIN(4)
  const Tensor& q = tensor(args[0], "q");
  const Tensor& k = tensor(args[1], "k");
  const Tensor& v = tensor(args[2], "v");
  const long mode = integer(args[3]);
  require(q.is_cuda() && k.is_cuda() && v.is_cuda(), "feature_maps runs on the CUDA library only (there is no CPU path)");
  if (mode != 2) same_device(v, {&q, &k}, "feature_maps");
  variable_list out;
  {
    pybind11::gil_scoped_release no_gil;
    std::optional<Tensor> a, b;
    if (mode != 2) { a = q; b = k; }
    out = FeatureMaps::apply(a, b, v, mode == 1);
  }
  if (mode == 2) return tuple({wrap(q), wrap(k), wrap(out[0])});
  return tuple({wrap(out[0]), wrap(out[1]), wrap(out[2])});
  NHA_END
}

// ---- silu + RMS norm (nha_fla/layers/nha.py:277-278) -----------------------------------------------------------------
struct SiluRmsNorm : Function<SiluRmsNorm> {
  static variable_list forward(AutogradContext* ctx, const Tensor& o, const Tensor& weight, const std::optional<Tensor>& bias, double eps) {
    const c10::cuda::OptionalCUDAGuard guard(o.device());
    const int64_t cols = o.size(-1), rows = cols ? o.numel() / cols : 0;
    const Tensor oc = bf16c(o), w = typed(weight, at::kFloat), b = bias.has_value() ? typed(*bias, at::kFloat) : Tensor();
    const Tensor y = empty_same(oc), rstd = empty({rows}, at::kFloat, oc);
    check(nha_silu_rmsnorm_fwd(oc.data_ptr(), (const float*)w.data_ptr(), (const float*)ptr(b), y.data_ptr(), (float*)rstd.data_ptr(), rows,
                               (int)cols, (float)eps, stream_of(oc)), "nha_silu_rmsnorm_fwd");
    ctx->save_for_backward({oc, w, rstd});
    ctx->saved_data["o"] = type_int(o.scalar_type());
    ctx->saved_data["w"] = type_int(weight.scalar_type());
    ctx->saved_data["b"] = bias.has_value() ? type_int(bias->scalar_type()) : (int64_t)-1;
    return {y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list sv = ctx->get_saved_variables();
    const Tensor oc = sv[0], w = sv[1], rstd = sv[2];
    const c10::cuda::OptionalCUDAGuard guard(oc.device());
    const int64_t cols = oc.size(-1), rows = rstd.numel();
    const Tensor dy = bf16c(grads[0]), d_o = empty_same(oc);
    const int parts = nha_silu_rmsnorm_bwd_ctas(rows);
    const bool has_bias = ctx->saved_data["b"].toInt() >= 0;
    const Tensor pw = empty({std::max(1, parts), cols}, at::kFloat, oc), pb = has_bias ? empty({std::max(1, parts), cols}, at::kFloat, oc) : Tensor();
    const Tensor dw = empty({cols}, at::kFloat, oc), db = has_bias ? empty({cols}, at::kFloat, oc) : Tensor();
    check(nha_silu_rmsnorm_bwd(oc.data_ptr(), (const float*)w.data_ptr(), (const float*)rstd.data_ptr(), dy.data_ptr(), d_o.data_ptr(),
                               (float*)pw.data_ptr(), (float*)ptr(pb), rows, (int)cols, stream_of(oc)), "nha_silu_rmsnorm_bwd");
    check(nha_silu_rmsnorm_part_sum((const float*)pw.data_ptr(), (const float*)ptr(pb), (float*)dw.data_ptr(), (float*)ptr(db), parts,
                                    (int)cols, stream_of(oc)), "nha_silu_rmsnorm_part_sum");
    return {back_to(d_o, type_of(ctx->saved_data["o"])), back_to(dw, type_of(ctx->saved_data["w"])),
            has_bias ? back_to(db, type_of(ctx->saved_data["b"])) : Tensor(), Tensor()};
  }
};

// silu_rms_norm(o, weight, bias, eps) -> y
NHA_METHOD(silu_rms_norm) {
  NHA_BEGIN(4)
  const Tensor& o = tensor(args[0], "o");
  const Tensor& w = tensor(args[1], "weight");
  std::optional<Tensor> b;
  if (args[2] != Py_None) b = tensor(args[2], "bias");
  const double eps = real(args[3]);
  require(o.is_cuda(), "silu_rms_norm runs on the CUDA library only (there is no CPU path)");
  same_device(o, {&w}, "silu_rms_norm");
  if (b) same_device(o, {&*b}, "silu_rms_norm");
  // the kernel reads one weight (and bias) per column through their pointers
  require(o.dim() >= 1 && w.numel() >= o.size(-1) && (!b || b->numel() >= o.size(-1)), "the weight and bias must hold one value per column");
  variable_list out;
  {
    pybind11::gil_scoped_release no_gil;
    out = SiluRmsNorm::apply(o, w, b, eps);
  }
  return wrap(out[0]);
  NHA_END
}

// ---- aux loss and slot share from the two log-sum-exps (nha_fla/layers/nha.py:255-264, 288-323) ----------------------
// scratch of the statistics kernel, one per (device, stream), zeroed once: the kernel leaves it ready for the next call
static Tensor stats_scratch(const Tensor& like) {
  static std::mutex mu;
  static std::map<std::pair<int, void*>, Tensor>& pool = *new std::map<std::pair<int, void*>, Tensor>();
  std::lock_guard<std::mutex> lock(mu);
  Tensor& t = pool[{(int)like.device().index(), stream_of(like)}];
  if (!t.defined()) t = zeros({nha_lse_stats_scratch_bytes()}, at::kByte, like);
  return t;
}

struct GsaAuxLoss : Function<GsaAuxLoss> {
  static variable_list forward(AutogradContext* ctx, const Tensor& lse_swa, const Tensor& lse_gsa, double target) {
    ctx->set_materialize_grads(false);
    const c10::cuda::OptionalCUDAGuard guard(lse_swa.device());
    const Tensor ls = typed(lse_swa, at::kFloat), lg = typed(lse_gsa, at::kFloat);
    const Tensor out = empty({2}, at::kFloat, ls);
    check(nha_lse_stats((const float*)ls.data_ptr(), (const float*)lg.data_ptr(), ls.numel(), (float)target, (float*)out.data_ptr(),
                        stats_scratch(ls).data_ptr(), stream_of(ls)), "nha_lse_stats");
    ctx->save_for_backward({ls, lg});
    ctx->saved_data["r"] = target;
    ctx->saved_data["t"] = type_int(lse_gsa.scalar_type());
    const Tensor ratio = out.select(0, 1);
    ctx->mark_non_differentiable({ratio});
    return {out.select(0, 0), ratio};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor()};
    const variable_list sv = ctx->get_saved_variables();
    const c10::cuda::OptionalCUDAGuard guard(sv[0].device());
    const Tensor d = empty_same(sv[1]), dl = typed(grads[0], at::kFloat);
    check(nha_lse_aux_grad((const float*)sv[0].data_ptr(), (const float*)sv[1].data_ptr(), (const float*)dl.data_ptr(), sv[0].numel(),
                           (float)ctx->saved_data["r"].toDouble(), (float*)d.data_ptr(), stream_of(sv[0])), "nha_lse_aux_grad");
    return {Tensor(), back_to(d, type_of(ctx->saved_data["t"])), Tensor()};
  }
};

// gsa_aux_loss(lse_swa, lse_gsa, target) -> (loss, share)
NHA_METHOD(gsa_aux_loss) {
  NHA_BEGIN(3)
  const Tensor& ls = tensor(args[0], "lse_swa");
  const Tensor& lg = tensor(args[1], "lse_gsa");
  const double target = real(args[2]);
  require(ls.is_cuda() && lg.is_cuda(), "gsa_aux_loss runs on the CUDA library only (there is no CPU path)");
  same_device(ls, {&lg}, "gsa_aux_loss");
  require(ls.sizes() == lg.sizes() && ls.numel() > 0, "lse_swa and lse_gsa must have the same, non-empty shape");
  variable_list out;
  {
    pybind11::gil_scoped_release no_gil;
    out = GsaAuxLoss::apply(ls.detach(), lg, target);
  }
  return tuple({wrap(out[0]), wrap(out[1])});
  NHA_END
}

}  // namespace nha_host
