// Host side of chunk_nha (with its autograd node) and fused_chunk_nha_prefill: checks, allocation and launches of one call.
// Semantics of the reference's nha_fla/ops/nha/chunk.py:352-564, 568-690 and chunk_fused.py:291-380.
#include <string.h>

#include <vector>

#include "nha_host.h"

namespace nha_host {

using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

enum { QS, KS, QG, KG, VV, SS, GG, NIN };      // the operator's argument order: q_swa, k_swa, q_gsa, k_gsa, v, s, g

int type_code(at::ScalarType t) { return t == at::kBFloat16 ? NHA_BF16 : t == at::kHalf ? NHA_FP16 : t == at::kFloat ? NHA_FP32 : -1; }

// dst[i] = src[i] in another type, as many tensors as possible in one launch.  Undefined sources are skipped.
void cast_all(const Tensor* src, Tensor* dst, const at::ScalarType* to, int n) {
  const void* from[8];
  void* into[8];
  int64_t len[8];
  int count = 0, a = -1, b = -1;
  Tensor held[8];
  for (int i = 0; i < n; ++i) {
    if (!src[i].defined()) continue;
    const Tensor x = held[i] = src[i].contiguous();
    const int sa = type_code(x.scalar_type()), sb = type_code(to[i]);
    if (sa == sb && sa >= 0) {
      dst[i] = on_16(x);
    } else if (sa < 0 || sb < 0 || (count && (sa != a || sb != b))) {
      dst[i] = on_16(x.to(to[i]));
    } else {
      dst[i] = empty(x.sizes(), to[i], x);
      a = sa;
      b = sb;
      from[count] = x.data_ptr();
      into[count] = dst[i].data_ptr();
      len[count++] = x.numel();
    }
  }
  if (count) check(nha_cast_many(from, into, len, count, a, b, stream_of(src[0].defined() ? src[0] : src[n - 1])), "nha_cast_many");
}

// one tensor in another type, by the same kernel
Tensor in_type(const Tensor& x, at::ScalarType to) {
  Tensor y;
  cast_all(&x, &y, &to, 1);
  return y;
}

struct Call {
  nha_chunk_desc d;
  int dense_T = -1;                            // tokens per sequence of an unpacked batch
  int64_t B = 1, T = 0;
  Tensor in[NIN], cu, wl, sh, hk0, hv0;        // bf16 inputs; int32 tensors (or undefined); fp32 states (or undefined)
  at::ScalarType out_type;
  Tensor o, lse_swa, lse_gsa, hkt, hvt, arena;
};

int64_t up(int64_t x) { return (x + 255) & ~(int64_t)255; }

void check_device(const nha_chunk_desc* d, void* stream, const char* what) {
  if (!check_device_words()) return;
  const int e = nha_chunk_device_error(d, stream);
  if (e != 0)
    raise(library_error, std::string(what) + ": device error word " + std::to_string(e) +
                             " (a bounded wait on a tensor-core completion ran out; the outputs of this call are invalid)");
}

// pointers of the call's inputs, plan and chunk-start states
void point(Call& c) {
  nha_chunk_desc& d = c.d;
  d.q_swa = c.in[QS].data_ptr(); d.k_swa = c.in[KS].data_ptr(); d.q_gsa = c.in[QG].data_ptr(); d.k_gsa = c.in[KG].data_ptr();
  d.v = c.in[VV].data_ptr(); d.s = c.in[SS].data_ptr(); d.g = c.in[GG].data_ptr();
  d.window_left = (const int32_t*)ptr(c.wl);
  d.shift = (const int32_t*)ptr(c.sh);
  d.hk0 = (const float*)ptr(c.hk0);
  d.hv0 = (const float*)ptr(c.hv0);
  // what a call keeps for its backward sits in one buffer: boundaries (unpacked batch), plan, chunk-start states
  char* p = (char*)c.arena.data_ptr();
  const int64_t ncb = nha_chunk_count_bound(d.Ttot, d.N);
  d.cu_seqlens = c.dense_T >= 0 ? (const int32_t*)p : (const int32_t*)c.cu.data_ptr();
  p += up(4 * ((int64_t)d.N + 1));
  d.plan = (int32_t*)p;
  p += up(4 * nha_chunk_plan_ints(d.Ttot, d.N, d.H));
  d.hk_chunks = p;
  p += up(ncb * d.H * d.K * d.M * 2);
  d.hv_chunks = p;
  d.o = ptr(c.o);
  d.lse_swa = (float*)ptr(c.lse_swa);
  d.lse_gsa = (float*)ptr(c.lse_gsa);
  d.hkt = (float*)ptr(c.hkt);
  d.hvt = (float*)ptr(c.hvt);
}

void forward(Call& c, bool want_state) {
  nha_chunk_desc& d = c.d;
  const Tensor& like = c.in[QS];
  c.o = empty({c.B, c.T, d.HQ, d.V}, at::kBFloat16, like);
  c.lse_swa = empty({c.B, c.T, d.HQ}, at::kFloat, like);
  c.lse_gsa = empty({c.B, c.T, d.HQ}, at::kFloat, like);
  if (want_state) {
    c.hkt = empty({d.N, d.H, d.K, d.M}, at::kFloat, like);
    c.hvt = empty({d.N, d.H, d.M, d.V}, at::kFloat, like);
  }
  const int64_t ncb = nha_chunk_count_bound(d.Ttot, d.N);
  c.arena = empty({up(4 * ((int64_t)d.N + 1)) + up(4 * nha_chunk_plan_ints(d.Ttot, d.N, d.H)) + 2 * up(ncb * d.H * d.K * d.M * 2) +
                   (d.V > d.K ? 2 * ncb * d.H * (int64_t)(d.V - d.K) * d.M : 0)}, at::kByte, like);
  point(c);
  const int64_t nbytes = nha_chunk_fwd_workspace_bytes(&d);
  Tensor ws;
  if (nbytes > 0) {
    ws = empty({nbytes}, at::kByte, like);
    d.workspace = ws.data_ptr();
    d.workspace_bytes = nbytes;
  }
  void* stream = stream_of(like);
  if (c.dense_T >= 0)
    check(nha_chunk_fwd_dense(&d, c.dense_T, stream), "nha_chunk_fwd");
  else
    check(nha_chunk_fwd(&d, stream), "nha_chunk_fwd");
  check_device(&d, stream, "nha_chunk_fwd");
}

// Sizes and the bf16 / int32 / fp32 forms of a call's inputs.  `raw`: the seven tensors as given, in the order of NIN.
void set_up(Call& c, const Tensor* raw, const Tensor& cu, int64_t max_seqlen, double scale, const Tensor& hk0, const Tensor& hv0) {
  memset(&c.d, 0, sizeof(c.d));
  nha_chunk_desc& d = c.d;
  c.B = raw[QS].size(0);
  c.T = raw[QS].size(1);
  for (int i = 0; i < NIN; ++i)
    require(raw[i].dim() == 4 && raw[i].size(0) == c.B && raw[i].size(1) == c.T, "the seven inputs must be [B, T, heads, dim] with the same B and T");
  d.HQ = raw[QG].size(2);
  d.K = raw[QG].size(3);
  d.H = raw[KG].size(2);
  d.V = raw[VV].size(3);
  d.M = raw[SS].size(3);
  require(raw[QS].sizes() == raw[QG].sizes() && raw[KS].sizes() == raw[KG].sizes() && raw[KG].size(3) == d.K && raw[VV].size(2) == d.H &&
              raw[SS].size(2) == d.H && raw[GG].sizes() == raw[SS].sizes(), "head counts or dims of the inputs do not match");
  d.Ttot = c.B * c.T;
  c.out_type = raw[QS].scalar_type();
  if (cu.defined()) {
    c.cu = cu;
    d.N = (int32_t)cu.numel() - 1;
    d.max_seqlen = (int32_t)max_seqlen;
  } else {
    c.dense_T = (int)c.T;
    d.N = (int32_t)c.B;
    d.max_seqlen = (int32_t)c.T;
  }
  d.scale = (float)scale;
  if (hk0.defined()) {
    require(hk0.numel() == (int64_t)d.N * d.H * d.K * d.M && hv0.numel() == (int64_t)d.N * d.H * d.M * d.V,
            "initial_state must be ([N,H,K,M], [N,H,M,V]) at the kv-head count");
    c.hk0 = on_16(typed(hk0, at::kFloat));
    c.hv0 = on_16(typed(hv0, at::kFloat));
  }
  at::ScalarType to[NIN];
  bool all = true;
  for (int i = 0; i < NIN; ++i) {
    to[i] = at::kBFloat16;
    all = all && raw[i].scalar_type() == at::kBFloat16 && raw[i].is_contiguous() && on_16_bytes(raw[i]);
  }
  if (all) {
    for (int i = 0; i < NIN; ++i) c.in[i] = raw[i];
  } else {
    cast_all(raw, c.in, to, NIN);
  }
}

struct Meta : torch::CustomClassHolder {
  Call c;
  at::ScalarType types[NIN];
  bool state_grad = false;
};

struct Params {
  Call* c;
  bool want_state;
};

// Gradients flow to q_swa, k_swa, q_gsa, k_gsa, v, s, g and the initial states; a gradient arriving on lse_gsa is honoured,
// one arriving on lse_swa is dropped as the reference drops it (nha_fla/ops/nha/chunk.py:491-512).
struct ChunkFunction : torch::autograd::Function<ChunkFunction> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q_swa, const Tensor& k_swa, const Tensor& q_gsa, const Tensor& k_gsa,
                               const Tensor& v, const Tensor& s, const Tensor& g, const std::optional<Tensor>& hk0,
                               const std::optional<Tensor>& hv0, const Params& p) {
    ctx->set_materialize_grads(false);
    Call& c = *p.c;
    nha_host::forward(c, p.want_state);
    const bool converted = c.out_type != at::kBFloat16;
    const Tensor out = converted ? in_type(c.o, c.out_type) : c.o;
    auto meta = c10::make_intrusive<Meta>();
    const Tensor* raw[NIN] = {&q_swa, &k_swa, &q_gsa, &k_gsa, &v, &s, &g};
    for (int i = 0; i < NIN; ++i) meta->types[i] = raw[i]->scalar_type();
    meta->state_grad = hk0.has_value() && (hk0->requires_grad() || hv0->requires_grad());
    ctx->save_for_backward({c.in[0], c.in[1], c.in[2], c.in[3], c.in[4], c.in[5], c.in[6], c.cu, c.wl, c.sh, c.hk0, c.hv0, c.o, c.lse_swa,
                            c.lse_gsa, c.hkt, c.hvt, c.arena});
    meta->c.d = c.d;
    meta->c.dense_T = c.dense_T;
    meta->c.B = c.B;
    meta->c.T = c.T;
    meta->c.out_type = c.out_type;
    ctx->saved_data["meta"] = c10::IValue::make_capsule(std::move(meta));
    ctx->mark_non_differentiable({c.lse_swa});
    if (!p.want_state) return {out, c.lse_swa, c.lse_gsa};
    return {out, c.lse_swa, c.lse_gsa, c.hkt, c.hvt};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list sv = ctx->get_saved_variables();
    const auto meta = c10::static_intrusive_pointer_cast<Meta>(ctx->saved_data["meta"].toCapsule());
    Call c = meta->c;                                   // this run's own copy: a graph may be run backward more than once
    for (int i = 0; i < NIN; ++i) c.in[i] = sv[i];
    c.cu = sv[7]; c.wl = sv[8]; c.sh = sv[9]; c.hk0 = sv[10]; c.hv0 = sv[11]; c.o = sv[12]; c.lse_swa = sv[13]; c.lse_gsa = sv[14];
    c.hkt = sv[15]; c.hvt = sv[16]; c.arena = sv[17];
    const c10::cuda::OptionalCUDAGuard guard(c.in[0].device());
    point(c);
    nha_chunk_desc& d = c.d;
    const Tensor& like = c.in[0];
    variable_list out(NIN + 3);
    Tensor d_o = grads[0];
    if (!d_o.defined()) d_o = zeros({c.B, c.T, d.HQ, d.V}, at::kBFloat16, like);
    if (d_o.scalar_type() != at::kBFloat16) {
      d_o = in_type(d_o, at::kBFloat16);
    }
    d_o = on_16(d_o.contiguous());
    Tensor d_lse, d_hkt, d_hvt;
    if (grads[2].defined()) d_lse = typed(grads[2], at::kFloat);
    if (grads.size() > 3 && (grads[3].defined() || grads[4].defined())) {
      d_hkt = grads[3].defined() ? typed(grads[3], at::kFloat) : zeros(c.hkt.sizes(), at::kFloat, like);
      d_hvt = grads[4].defined() ? typed(grads[4], at::kFloat) : zeros(c.hvt.sizes(), at::kFloat, like);
    }
    Tensor gr[NIN], dhk0, dhv0;
    for (int i = 0; i < NIN; ++i) gr[i] = empty(c.in[i].sizes(), at::kBFloat16, like);
    if (meta->state_grad) {
      dhk0 = empty({d.N, d.H, d.K, d.M}, at::kFloat, like);
      dhv0 = empty({d.N, d.H, d.M, d.V}, at::kFloat, like);
    }
    d.d_o = d_o.data_ptr();
    d.d_lse_gsa = (const float*)ptr(d_lse);
    d.d_hkt = (const float*)ptr(d_hkt);
    d.d_hvt = (const float*)ptr(d_hvt);
    d.dq_swa = gr[QS].data_ptr(); d.dk_swa = gr[KS].data_ptr(); d.dq_gsa = gr[QG].data_ptr(); d.dk_gsa = gr[KG].data_ptr();
    d.dv = gr[VV].data_ptr(); d.ds = gr[SS].data_ptr(); d.dg = gr[GG].data_ptr();
    d.dhk0 = (float*)ptr(dhk0);
    d.dhv0 = (float*)ptr(dhv0);
    const int64_t nbytes = std::max<int64_t>(nha_chunk_bwd_workspace_bytes(&d), 16);
    const Tensor ws = empty({nbytes}, at::kByte, like);
    d.workspace = ws.data_ptr();
    d.workspace_bytes = nbytes;
    void* stream = stream_of(like);
    check(c.dense_T > 0 ? nha_chunk_bwd_dense(&d, c.dense_T, stream) : nha_chunk_bwd(&d, stream), "nha_chunk_bwd");
    check_device(&d, stream, "nha_chunk_bwd");
    bool same = true;
    for (int i = 0; i < NIN; ++i) same = same && meta->types[i] == at::kBFloat16;
    if (same) {
      for (int i = 0; i < NIN; ++i) out[i] = gr[i];
    } else {
      Tensor conv[NIN];
      cast_all(gr, conv, meta->types, NIN);
      for (int i = 0; i < NIN; ++i) out[i] = conv[i];
    }
    out[NIN] = dhk0;
    out[NIN + 1] = dhv0;
    return out;
  }
};

// a window or shift argument: one value for all sequences, or an int32 tensor with one per sequence
void per_sequence(PyObject* o, int64_t N, const Tensor& like, Tensor& t, int32_t& all) {
  if (!THPVariable_Check(o)) {
    all = (int32_t)integer(o);
    return;
  }
  const Tensor& x = THPVariable_Unpack(o);
  if (x.numel() == 1) {
    all = (int32_t)x.item().toLong();
    return;
  }
  if (x.numel() != N)
    raise(PyExc_AssertionError, "per-sequence tensor must have " + std::to_string(N) + " entries, got " + std::to_string(x.numel()));
  t = x.to(like.device(), at::kInt).contiguous();
}

}  // namespace

// chunk_nha(q_swa, k_swa, q_gsa, k_gsa, v, s, g, cu_seqlens, max_seqlen, scale, window_size_left, window_size_right, gsa_kv_shift,
//           initial_state, output_final_state) -> (o, lse_swa, lse_gsa[, (hkt, hvt)])
NHA_METHOD(chunk_nha) {
  NHA_BEGIN(15)
  static const char* names[NIN] = {"q_swa", "k_swa", "q_gsa", "k_gsa", "v", "s", "g"};
  Tensor raw[NIN];
  for (int i = 0; i < NIN; ++i) raw[i] = tensor(args[i], names[i]);
  require(raw[QS].dim() == 4, "Expected [B, T, H, D] for input");
  const long right = integer(args[11]);
  require(right == 0 || right == -1, "the window branch is causal: window_size_right must be 0 or -1");
  const double scale = args[9] == Py_None ? 1.0 / sqrt((double)raw[QS].size(3)) : real(args[9]);
  Tensor hk0, hv0;
  state_pair(args[13], hk0, hv0);
  same_device(raw[QS], {&raw[KS], &raw[QG], &raw[KG], &raw[VV], &raw[SS], &raw[GG], &hk0, &hv0}, "chunk_nha");
  const c10::cuda::OptionalCUDAGuard guard(raw[QS].device());
  Tensor cu;
  int64_t max_seqlen = 0;
  if (args[7] != Py_None) {
    require(raw[QS].size(0) == 1, "varlen inputs must be packed into a single batch row");
    cu = tensor(args[7], "cu_seqlens").to(raw[QS].device(), at::kInt).contiguous();
    if (args[8] != Py_None)
      max_seqlen = integer(args[8]);
    else
      max_seqlen = (cu.narrow(0, 1, cu.numel() - 1) - cu.narrow(0, 0, cu.numel() - 1)).max().item().toLong();
  }
  const bool want = truth(args[14]);
  Call c;
  const int64_t N = cu.defined() ? cu.numel() - 1 : raw[QS].size(0);
  int32_t wl_all = 0, sh_all = 0;
  per_sequence(args[10], N, raw[QS], c.wl, wl_all);
  per_sequence(args[12], N, raw[QS], c.sh, sh_all);
  variable_list out;
  {
    pybind11::gil_scoped_release no_gil;
    auto needs = [](const Tensor& t) { return t.defined() && t.requires_grad(); };
    auto tangent = [](const Tensor& t) { return t.defined() && t._fw_grad(0).defined(); };
    bool grad = needs(hk0) || needs(hv0), dual = tangent(hk0) || tangent(hv0);
    for (int i = 0; i < NIN; ++i) {
      grad = grad || needs(raw[i]);
      dual = dual || tangent(raw[i]);
    }
    // an input with a forward-mode tangent goes to the autograd node too, which refuses it: nothing may drop it silently
    grad = (grad && at::GradMode::is_enabled()) || dual;
    {
      at::AutoGradMode off(false);
      set_up(c, raw, cu, max_seqlen, scale, hk0, hv0);
    }
    c.d.window_left_all = wl_all;
    c.d.shift_all = sh_all;
    if (grad) {
      std::optional<Tensor> a, b;
      if (hk0.defined()) { a = hk0; b = hv0; }
      const Params p{&c, want};
      out = ChunkFunction::apply(raw[0], raw[1], raw[2], raw[3], raw[4], raw[5], raw[6], a, b, p);
    } else {
      at::AutoGradMode off(false);
      forward(c, want);
      out = {c.out_type != at::kBFloat16 ? in_type(c.o, c.out_type) : c.o, c.lse_swa, c.lse_gsa};
      if (want) { out.push_back(c.hkt); out.push_back(c.hvt); }
    }
  }
  if (!want) return tuple({wrap(out[0]), wrap(out[1]), wrap(out[2])});
  return tuple({wrap(out[0]), wrap(out[1]), wrap(out[2]), tuple({wrap(out[3]), wrap(out[4])})});
  NHA_END
}

// prefill(q, k, v, rotary_q, rotary_k, s, g, window_size, initial_state, output_final_state, scale) -> (o, (hkt, hvt))
NHA_METHOD(prefill) {
  NHA_BEGIN(11)
  const Tensor& q = tensor(args[0], "q");
  const Tensor& k = tensor(args[1], "k");
  const Tensor& v = tensor(args[2], "v");
  const Tensor& rq = tensor(args[3], "rotary_q");
  const Tensor& rk = tensor(args[4], "rotary_k");
  const Tensor& s = tensor(args[5], "s");
  const Tensor& g = tensor(args[6], "g");
  const long W = integer(args[7]);
  Tensor hk0, hv0;
  state_pair(args[8], hk0, hv0);
  const bool want = truth(args[9]);
  require(q.dim() == 4 && k.dim() == 4 && v.dim() == 4 && s.dim() == 4 && g.dim() == 4, "Expected [B, T, H, D] for input");
  const int64_t B = q.size(0), T = q.size(1), HQ = q.size(2), K = q.size(3), H = k.size(2), V = v.size(3), M = s.size(3);
  const double scale = args[10] == Py_None ? 1.0 / sqrt((double)K) : real(args[10]);
  require(k.size(1) == T && v.size(1) == T && s.size(1) == T && g.size(1) == T, "q, k, v, s and g must hold the same tokens");
  require(rq.sizes() == q.sizes() && rk.sizes() == k.sizes(), "rotary_q / rotary_k must have the shapes of q / k");
  require(H > 0 && HQ % H == 0, "HQ must be a multiple of H");
  require(W >= 1, "window_size must be at least 1");
  if (hk0.defined() && (hk0.sizes() != at::IntArrayRef({B, H, K, M}) || hv0.sizes() != at::IntArrayRef({B, H, M, V})))
    raise(PyExc_AssertionError, "initial_state must be at the kv-head count [B, " + std::to_string(H) + ", ...], got " + c10::str(hk0.sizes()) +
                                    " / " + c10::str(hv0.sizes()));
  same_device(q, {&k, &v, &rq, &rk, &s, &g, &hk0, &hv0}, "fused_chunk_nha_prefill");
  Call c;
  Tensor o;
  {
    pybind11::gil_scoped_release no_gil;
    at::AutoGradMode off(false);
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    const Tensor raw[NIN] = {rq, rk, q, k, v, s, g};
    set_up(c, raw, Tensor(), 0, scale, hk0, hv0);
    c.d.window_left_all = (int32_t)W - 1;
    c.d.shift_all = (int32_t)W;
    forward(c, want);
    o = q.scalar_type() != at::kBFloat16 ? in_type(c.o, q.scalar_type()) : c.o;
  }
  return tuple({wrap(o), want ? tuple({wrap(c.hkt), wrap(c.hvt)}) : tuple({none(), none()})});
  NHA_END
}

}  // namespace nha_host
