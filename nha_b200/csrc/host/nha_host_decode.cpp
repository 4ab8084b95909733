// Host side of the single-token operators (fused_recurrent_nha_decode, fused_recurrent_nha, the ring cache's step):
// argument checks, output allocation and the library call, without a trip through Python.  Semantics of the reference's
// nha_fla/ops/nha/fused_recurrent.py:431-584, :588-682.
#include <map>
#include <mutex>
#include <tuple>

#include "nha_host.h"

namespace nha_host {

Tensor decode_workspace(const Tensor& like, int B, int HQ, int H, int V, int W) {
  struct Entry {
    Tensor t;
    unsigned long long capture = 0, used = 0;                  // the capture it was made in (0: none); when it was last asked for
  };
  constexpr size_t kMost = 64;                                 // buffers kept; a server's batch sizes come and go
  static std::mutex mu;
  static std::map<std::tuple<int, void*, int64_t>, Entry>& pool = *new std::map<std::tuple<int, void*, int64_t>, Entry>();
  static unsigned long long now = 0;
  const int64_t need = nha_decode_workspace_bytes(B, HQ, H, V, W);
  void* stream = stream_of(like);
  // A graph keeps the address that it was captured with, so a capture has a buffer of its own: it lies in the graph's memory, which
  // stays with the graph when the buffer leaves this pool, and each replay zeroes it.
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo((cudaStream_t)stream, &status, &id) != cudaSuccess) (void)cudaGetLastError();
  if (status != cudaStreamCaptureStatusActive) id = 0;
  std::lock_guard<std::mutex> lock(mu);
  Entry& e = pool[std::make_tuple((int)like.device().index(), stream, (int64_t)B * H)];
  if (!e.t.defined() || e.t.numel() < need || e.capture != id) {
    e.t = zeros({need}, at::kByte, like);
    e.capture = id;
  }
  e.used = ++now;
  const Tensor ws = e.t;
  if (pool.size() > kMost) {                                   // memory goes back in the order of its stream
    auto oldest = pool.begin();
    for (auto it = pool.begin(); it != pool.end(); ++it)
      if (it->second.used < oldest->second.used) oldest = it;
    pool.erase(oldest);
  }
  return ws;
}

static void check_state(const Tensor& hk0, const Tensor& hv0, int64_t B, int64_t H, int64_t K, int64_t V, int64_t M) {
  if (hk0.defined() && (hk0.sizes() != at::IntArrayRef({B, H, K, M}) || hv0.sizes() != at::IntArrayRef({B, H, M, V})))
    raise(PyExc_AssertionError, "initial_state must be ([B,H,K,M], [B,H,M,V]) at the kv-head count " + std::to_string(H) + ", got " +
                                    c10::str(hk0.sizes()) + " / " + c10::str(hv0.sizes()));
}

// The slot memory of a step (its shapes have been checked): the caller's own buffers when they can be updated in place, else copies (or, with no initial
// state, fresh buffers that the kernel takes as zero).  A caller's buffer that does not start on 16 bytes is updated through a copy.
struct State {
  Tensor hk, hv;
  Tensor back_k, back_v;                         // where the copies go after the step
  int zero = 0;
  State(Tensor hk0, Tensor hv0, int64_t B, int64_t H, int64_t K, int64_t V, int64_t M, bool keep, at::ScalarType dt,
        const Tensor& like) {
    if (!hk0.defined()) {
      hk = empty({B, H, K, M}, dt, like);
      hv = empty({B, H, M, V}, dt, like);
      zero = 1;
      return;
    }
    if (keep && hk0.scalar_type() == dt && hv0.scalar_type() == dt && hk0.is_contiguous() && hv0.is_contiguous()) {
      hk = on_16(hk0);
      hv = on_16(hv0);
      if (C10_UNLIKELY(!hk.is_same(hk0))) back_k = hk0;
      if (C10_UNLIKELY(!hv.is_same(hv0))) back_v = hv0;
    } else {
      hk = hk0.to(dt).contiguous().clone();
      hv = hv0.to(dt).contiguous().clone();
    }
  }
  // after the launch: the updated buffers, the caller's own where it gave some
  void done(Tensor& k, Tensor& v) {
    if (C10_UNLIKELY(back_k.defined())) hk = back_k.copy_(hk);
    if (C10_UNLIKELY(back_v.defined())) hv = back_v.copy_(hv);
    k = std::move(hk);
    v = std::move(hv);
  }
};

static bool table_ok(const Tensor& t, int64_t skip) {
  return t.scalar_type() == at::kBFloat16 && t.stride(2) == 1 && t.stride(1) % 8 == 0 && t.stride(0) % 8 == 0 &&
         (reinterpret_cast<uintptr_t>(t.data_ptr()) + 2 * skip * t.stride(1)) % 16 == 0;
}

// decode(q, k, v, g, sw_k, sw_v, sq, s, cos, sin, initial_state, output_final_state, scale, bf16_state) -> (o, (hk, hv))
NHA_METHOD(decode) {
  NHA_BEGIN(14)
  const Tensor& q = tensor(args[0], "q");
  const Tensor& k = tensor(args[1], "k");
  const Tensor& v = tensor(args[2], "v");
  const Tensor& g = tensor(args[3], "g");
  const Tensor& sw_k = tensor(args[4], "sw_k");
  const Tensor& sw_v = tensor(args[5], "sw_v");
  const Tensor sq = tensor_or_none(args[6], "sq"), s = tensor_or_none(args[7], "s");
  Tensor cos = tensor_or_none(args[8], "cos"), sin = tensor_or_none(args[9], "sin");
  Tensor hk0, hv0;
  state_pair(args[10], hk0, hv0);
  const bool keep = truth(args[11]);
  const bool bf16_state = truth(args[13]);
  require(q.dim() == 4 && k.dim() == 4 && v.dim() == 4 && g.dim() == 4 && sw_k.dim() == 4 && sw_v.dim() == 4,
          "q, k, v, g and the window tensors must have four dimensions");
  const int64_t B = q.size(0), HQ = q.size(2), K = q.size(3), W = sw_k.size(1), H = sw_k.size(2), V = v.size(3), M = g.size(3);
  const double scale = args[12] == Py_None ? 1.0 / sqrt((double)K) : real(args[12]);
  require(q.size(1) == 1 && k.size(1) == 1 && g.size(1) == 1, "a decode step takes one token per sequence");
  if (k.size(2) != H || v.size(2) != H || g.size(2) != H)
    raise(PyExc_AssertionError, "popped-entry head count must match the kv-head count (" + std::to_string(H) + ") of the window tensors");
  require(sw_v.size(1) == W && sw_v.size(2) == H, "sw_k and sw_v must hold the same keys and heads");
  // the kernel takes raw pointers: what it reads must be there
  require(k.numel() == B * H * K && v.numel() == B * H * V && g.numel() == B * H * M,
          "k, v and g must hold one token per sequence, with the head dim of q in k");
  if (sw_k.size(0) != B || sw_k.size(3) != K || sw_v.size(0) != B || sw_v.size(3) != V)
    raise(PyExc_AssertionError, "sw_k and sw_v must be " + c10::str(at::IntArrayRef({B, W, H, K})) + " and " +
                                    c10::str(at::IntArrayRef({B, W, H, V})) + ", got " + c10::str(sw_k.sizes()) + " / " + c10::str(sw_v.sizes()));
  require(H > 0 && HQ % H == 0, "HQ must be a multiple of H");
  require(K >= 16 && V >= 16, "K and V must be at least 16");
  const bool rotary = cos.defined();
  int64_t cs_batch = 0, cs_row = 0, skip = 0;
  if (rotary) {
    require(!sq.defined(), "pass either sq (pre-rotated) or cos/sin (in-kernel rotary), not both");
    require(sin.defined() && cos.sizes() == sin.sizes(), "cos and sin must have the same shape");
    if (cos.dim() != 3 || (cos.size(0) != 1 && cos.size(0) != B) || cos.size(1) < W || cos.size(2) != K)
      raise(PyExc_AssertionError, "rotary cos/sin must be [1|" + std::to_string(B) + ", W2>=" + std::to_string(W) + ", K=" +
                                      std::to_string(K) + "], got " + c10::str(cos.sizes()));
    require(K % 2 == 0, "in-kernel rotate-half requires an even head dim");
    skip = cos.size(1) - W;                                   // the last W rows are the window positions
    if (!(table_ok(cos, skip) && table_ok(sin, skip) && cos.strides() == sin.strides())) {
      cos = on_16(cos.narrow(1, skip, W).to(at::kBFloat16).contiguous());
      sin = on_16(sin.narrow(1, skip, W).to(at::kBFloat16).contiguous());
      skip = 0;
    }
    cs_batch = cos.size(0) == B && B > 1 ? cos.stride(0) : 0;
    cs_row = cos.stride(1);
  } else {
    require(sq.defined() && sq.sizes() == q.sizes(), "sq must have the shape of q");
  }
  if (s.defined()) require(s.sizes() == g.sizes(), "s must have the shape of g");
  check_state(hk0, hv0, B, H, K, V, M);
  same_device(q, {&k, &v, &g, &sw_k, &sw_v, &sq, &s, &cos, &sin, &hk0, &hv0}, "fused_recurrent_nha_decode");

  Tensor o, hk, hv;
  {
    pybind11::gil_scoped_release no_gil;
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    const Tensor qf = on_16(bf16c(q)), sqf = sq.defined() ? on_16(bf16c(sq)) : sq, kf = on_16(bf16c(k)), vf = on_16(bf16c(v));
    const Tensor gf = bf16c(g), sf = s.defined() ? bf16c(s) : s, wk = on_16(bf16c(sw_k)), wv = on_16(bf16c(sw_v));
    State st(hk0, hv0, B, H, K, V, M, keep, bf16_state ? at::kBFloat16 : at::kFloat, q);
    o = empty({B, 1, HQ, V}, at::kBFloat16, q);
    Tensor ws;
    if (W > 64 || M > 64 || bf16_state) ws = decode_workspace(q, B, HQ, H, V, W);
    void* stream = stream_of(q);
    const char* cp = rotary ? (const char*)cos.data_ptr() + 2 * skip * cs_row : nullptr;
    const char* sp = rotary ? (const char*)sin.data_ptr() + 2 * skip * cs_row : nullptr;
    const int64_t wsb = ws.defined() ? ws.numel() : 0;
    if (bf16_state)
      check(nha_decode_step_bf16_state(qf.data_ptr(), ptr(sqf), kf.data_ptr(), vf.data_ptr(), gf.data_ptr(), ptr(sf), wk.data_ptr(),
                                       wv.data_ptr(), cp, sp, cs_batch, cs_row, st.hk.data_ptr(), st.hv.data_ptr(), st.zero,
                                       o.data_ptr(), ptr(ws), wsb, B, HQ, H, K, V, M, W, (float)scale, stream),
            "nha_decode_step");
    else
      check(nha_decode_step(qf.data_ptr(), ptr(sqf), kf.data_ptr(), vf.data_ptr(), gf.data_ptr(), ptr(sf), wk.data_ptr(), wv.data_ptr(),
                            cp, sp, cs_batch, cs_row, nullptr, (float*)st.hk.data_ptr(), (float*)st.hv.data_ptr(), st.zero, o.data_ptr(),
                            nullptr, ptr(ws), wsb, B, HQ, H, K, V, M, W, (float)scale, stream),
            "nha_decode_step");
    if (q.scalar_type() != at::kBFloat16) o = o.to(q.scalar_type());
    st.done(hk, hv);
  }
  // buffers that were updated in place go back as the objects they came in
  PyObject* states;
  if (!keep) {
    states = tuple({none(), none()});
  } else {
    states = tuple({wrap(hk), wrap(hv)});
  }
  return tuple({wrap(o), states});
  NHA_END
}

// decode_logits(q, k, v, sliding_window, s, g, scale, initial_state, output_final_state) -> (o, swa_score, [hk, hv])
NHA_METHOD(decode_logits) {
  NHA_BEGIN(9)
  const Tensor& q = tensor(args[0], "q");
  const Tensor& k = tensor(args[1], "k");
  const Tensor& v = tensor(args[2], "v");
  const Tensor& win = tensor(args[3], "sliding_window");
  const Tensor& s = tensor(args[4], "s");
  const Tensor& g = tensor(args[5], "g");
  Tensor hk0, hv0;
  state_pair(args[7], hk0, hv0);
  const bool keep = truth(args[8]);
  require(!q.requires_grad(), "fused_recurrent_nha is inference-only (no autograd)");
  const int64_t B = q.size(0), HQ = q.size(2), K = q.size(3), H = k.size(2), V = v.size(-1), M = s.size(-1), W = win.size(-1);
  require(H > 0 && HQ % H == 0, "HQ must be a multiple of H");
  const double scale = args[6] == Py_None ? 1.0 / sqrt((double)k.size(-1)) : real(args[6]);
  require(k.numel() == B * H * K && v.numel() == B * H * V && s.numel() == B * H * M && g.numel() == B * H * M && win.numel() == B * HQ * W,
          "q, k, v, s, g and sliding_window must hold one token per sequence");
  check_state(hk0, hv0, B, H, K, V, M);
  same_device(q, {&k, &v, &win, &s, &g, &hk0, &hv0}, "fused_recurrent_nha");
  Tensor o, prob, hk, hv;
  {
    pybind11::gil_scoped_release no_gil;
    const c10::cuda::OptionalCUDAGuard guard(q.device());
    const Tensor qf = on_16(bf16c(q)), kf = on_16(bf16c(k)), vf = on_16(bf16c(v)), sf = bf16c(s), gf = bf16c(g), wf = bf16c(win);
    State st(hk0, hv0, B, H, K, V, M, keep, at::kFloat, q);
    o = empty({B, 1, HQ, V}, at::kBFloat16, q);
    prob = empty({B, 1, HQ, W}, at::kFloat, q);
    check(nha_decode_step(qf.data_ptr(), nullptr, kf.data_ptr(), vf.data_ptr(), gf.data_ptr(), sf.data_ptr(), nullptr, nullptr, nullptr,
                          nullptr, 0, 0, wf.data_ptr(), (float*)st.hk.data_ptr(), (float*)st.hv.data_ptr(), st.zero, o.data_ptr(),
                          (float*)prob.data_ptr(), nullptr, 0, B, HQ, H, K, V, M, W, (float)scale, stream_of(q)),
          "nha_decode_step");
    if (v.scalar_type() != at::kBFloat16) o = o.to(v.scalar_type());
    st.done(hk, hv);
  }
  PyObject* states = PyList_New(2);
  PyList_SET_ITEM(states, 0, keep ? wrap(hk) : none());
  PyList_SET_ITEM(states, 1, keep ? wrap(hv) : none());
  return tuple({wrap(o), wrap(prob), states});
  NHA_END
}

// The rings of a layer: W rows per sequence, whatever way the heads and dims of a row are written; one index of the oldest entry per
// sequence, or per (sequence, kv head) when the step also appends its token.
static void check_rings(const Tensor& ring_k, const Tensor& ring_v, const Tensor& ring_g, const Tensor& head, int64_t B, int64_t W, int64_t H,
                        int64_t K, int64_t V, int64_t M, bool fused) {
  auto ring = [&](const Tensor& t, int64_t dim) {
    return t.dim() >= 2 && t.size(0) == B && t.size(1) == W && t.numel() == B * W * H * dim && t.scalar_type() == at::kBFloat16 &&
           t.is_contiguous();
  };
  require(ring(ring_k, K) && ring(ring_v, V) && ring(ring_g, M), "the rings must be contiguous bf16 [B, W, H, K|V|M] with the batch and heads of the step");
  require(head.scalar_type() == at::kInt && head.is_contiguous() && head.numel() == (fused ? B * H : B),
          "the ring index must be contiguous int32, one per sequence (with the token appended in the step: per kv head)");
}

// decode_ring(q, k, v, g, ring_k, ring_v, ring_g, head, cos, sin, hk, hv, fill, fused, scale) -> o
NHA_METHOD(decode_ring) {
  NHA_BEGIN(15)
  const Tensor& q = tensor(args[0], "q");
  const Tensor& k = tensor(args[1], "k");
  const Tensor& v = tensor(args[2], "v");
  const Tensor& g = tensor(args[3], "g");
  const Tensor& ring_k = tensor(args[4], "ring_k");
  const Tensor& ring_v = tensor(args[5], "ring_v");
  const Tensor& ring_g = tensor(args[6], "ring_g");
  const Tensor& head = tensor(args[7], "head");
  const Tensor& cos = tensor(args[8], "cos");
  const Tensor& sin = tensor(args[9], "sin");
  const Tensor& hk = tensor(args[10], "hk");
  const Tensor& hv = tensor(args[11], "hv");
  const long fill = integer(args[12]);
  const bool fused = truth(args[13]);
  require(q.dim() == 4 && k.dim() == 4 && v.dim() == 4 && g.dim() == 4 && ring_k.dim() >= 2, "q, k, v and g must have four dimensions");
  const int64_t B = q.size(0), HQ = q.size(2), K = q.size(3), H = k.size(2), V = v.size(3), M = g.size(3), W = ring_k.size(1);
  const double scale = args[14] == Py_None ? 1.0 / sqrt((double)K) : real(args[14]);
  const int64_t wlen = fill >= W ? W : fill + 1;
  require(cos.dim() >= 2 && cos.size(-2) == wlen && cos.size(-1) == K, "cos/sin must cover the window positions");
  require(sin.sizes() == cos.sizes() && (cos.dim() == 2 || (cos.dim() == 3 && (cos.size(0) == 1 || cos.size(0) == B))),
          "cos/sin must be [W, K] or [1|B, W, K]");
  // the kernel takes raw pointers: what it reads and writes must be there
  require(H > 0 && k.numel() == B * H * K && v.numel() == B * H * V && g.numel() == B * H * M,
          "k, v and g must hold one token per sequence, with the head dim of q in k");
  check_rings(ring_k, ring_v, ring_g, head, B, W, H, K, V, M, fused);
  require(hk.scalar_type() == at::kFloat && hv.scalar_type() == at::kFloat && hk.is_contiguous() && hv.is_contiguous() &&
              hk.numel() == B * H * K * M && hv.numel() == B * H * M * V,
          "the slot memory must be contiguous fp32 [B,H,K,M] and [B,H,M,V]");
  same_device(q, {&k, &v, &g, &ring_k, &ring_v, &ring_g, &head, &cos, &sin, &hk, &hv}, "fused_recurrent_nha_decode_ring");
  Tensor o;
  {
    pybind11::gil_scoped_release no_gil;
    const c10::cuda::OptionalCUDAGuard guard(q.device());        // split count and launches follow the tensors' device
    const Tensor qc = on_16(bf16c(q)), kc = on_16(bf16c(k)), vc = on_16(bf16c(v)), gc = on_16(bf16c(g));
    const Tensor cc = on_16(bf16c(cos)), sc = on_16(bf16c(sin));
    const int64_t cs_batch = cc.dim() == 3 && cc.size(0) > 1 ? cc.stride(0) : 0, cs_row = cc.stride(-2);
    o = empty({B, 1, HQ, V}, at::kBFloat16, q);
    const Tensor ws = decode_workspace(q, B, HQ, H, V, W);
    void* stream = stream_of(q);
    if (fused) {
      check(nha_decode_step_ring_fused(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), gc.data_ptr(), ring_k.data_ptr(), ring_v.data_ptr(),
                                       ring_g.data_ptr(), (int32_t*)head.data_ptr(), cc.data_ptr(), sc.data_ptr(), cs_batch, cs_row,
                                       (float*)hk.data_ptr(), (float*)hv.data_ptr(), o.data_ptr(), ws.data_ptr(), ws.numel(), B, HQ, H, K,
                                       V, M, W, fill, (float)scale, stream),
            "nha_decode_step_ring_fused");
    } else {
      check(nha_decode_step_ring(qc.data_ptr(), kc.data_ptr(), vc.data_ptr(), ring_k.data_ptr(), ring_v.data_ptr(), ring_g.data_ptr(),
                                 (const int32_t*)head.data_ptr(), cc.data_ptr(), sc.data_ptr(), cs_batch, cs_row, (float*)hk.data_ptr(),
                                 (float*)hv.data_ptr(), o.data_ptr(), ws.data_ptr(), ws.numel(), B, HQ, H, K, V, M, W, fill, (float)scale,
                                 stream),
            "nha_decode_step_ring");
      check(nha_ring_append(ring_k.data_ptr(), ring_v.data_ptr(), ring_g.data_ptr(), kc.data_ptr(), vc.data_ptr(), gc.data_ptr(),
                            (int32_t*)head.data_ptr(), B, H, K, V, M, W, fill, stream),
            "nha_ring_append");
    }
  }
  return wrap(o);
  NHA_END
}

// decode_workspace(like, B, HQ, H, V, W) -> the scratch tensor of the current stream
NHA_METHOD(decode_workspace_for) {
  NHA_BEGIN(6)
  return wrap(decode_workspace(tensor(args[0], "like"), integer(args[1]), integer(args[2]), integer(args[3]), integer(args[4]), integer(args[5])));
  NHA_END
}

}  // namespace nha_host
