// Decode step with caller-supplied window logits (no window keys or values): slot-state update, slot logits, joint softmax and
// slot readout of one (sequence, kv head) per CTA, for 64 slots and head dims 64 or 128.  The other shapes take the general
// kernel (nha_decode.cu).
//
// HBM-bound: the fp32 state is read and written once.  The whole state of a CTA is in registers - 16-byte pieces, a warp's lanes
// along the rows - so that all of it is in flight before the first value is used, and the update, the products with the queries
// and the store need no pass through shared memory; only the sums over the warps do.  Against the general kernel (copies through
// shared memory, four threads a product): 64 sequences x 16 heads of 64, 28.4 -> 11.6 us (HBM floor 10.4); 32 sequences, 32 heads of
// 128 on 8, 512 logits, 27.6 -> 7.8 us; 8 sequences, 8 heads a group, 18.9 -> 7.1 us.  Four CTAs per SM at 64 registers: 12.5 us.
//
// Replaces the kernels of fused_recurrent_nha (nha_fla/ops/nha/fused_recurrent.py:48-147).
#include "nha_decode_args.cuh"

namespace nha {

constexpr int kLogThreads = 256, kLogWarps = kLogThreads / 32;

template <int D>
__global__ void __launch_bounds__(kLogThreads, D == 64 ? 3 : 2) nha_decode_logits_kernel(const DecodeArgs a) {
  constexpr int M = 64, M4 = M / 4, D4 = D / 4, JK = D * M4 / kLogThreads, JV = M * D4 / kLogThreads;
  constexpr int RK = kLogThreads / M4, RV = kLogThreads / D4;             // rows of a pass of the CTA
  extern __shared__ __align__(16) float sm[];
  const int NG = a.NG, W = a.W, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  float* part = sm;                                                      // [8 warps][max(M, D)]
  float* eg = part + kLogWarps * (D > M ? D : M);                        // [M] decay of the step
  float* prob = eg + M;                                                  // [NG][M] slot logits, then weights
  float* win = prob + NG * M;                                            // [NG][W] window logits, then weights
  const int bh = blockIdx.x, b = bh / a.H, h = bh - b * a.H;
  const int ck = tid % M4, rk = tid / M4, cv = tid % D4, rv = tid / D4;  // this thread's 4 columns and first row of hk / hv
  float4* hkp = reinterpret_cast<float4*>(a.hk + (size_t)bh * D * M) + tid;
  float4* hvp = reinterpret_cast<float4*>(a.hv + (size_t)bh * M * D) + tid;
  float4 hk[JK], hv[JV];
#pragma unroll
  for (int j = 0; j < JK; ++j) hk[j] = a.zero_state ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcs(hkp + j * kLogThreads);
#pragma unroll
  for (int j = 0; j < JV; ++j) hv[j] = a.zero_state ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcs(hvp + j * kLogThreads);
  auto four = [](const bf16* p) {
    const uint2 u = __ldg(reinterpret_cast<const uint2*>(p));
    const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(x.x, x.y, y.x, y.y);
  };
  const float4 g4 = four(a.g + (size_t)bh * M + 4 * ck);
  const float4 e4 = make_float4(__expf(g4.x), __expf(g4.y), __expf(g4.z), __expf(g4.w));
  const float4 s4 = a.s ? four(a.s + (size_t)bh * M + 4 * ck) : make_float4(1.f - e4.x, 1.f - e4.y, 1.f - e4.z, 1.f - e4.w);
  const float4 v4 = four(a.v + (size_t)bh * D + 4 * cv);
  const size_t hq0 = (size_t)b * a.HQ + (size_t)h * NG;
  float kv[JK], sr[JV];
  bf16 qv[JK];                                                           // the next head's query
#pragma unroll
  for (int j = 0; j < JK; ++j) {
    kv[j] = bf2f(__ldg(a.k + (size_t)bh * D + rk + RK * j));
    qv[j] = __ldg(a.q + hq0 * D + rk + RK * j);
  }
#pragma unroll
  for (int j = 0; j < JV; ++j) {
    const int m = rv + RV * j;
    sr[j] = a.s ? bf2f(a.s[(size_t)bh * M + m]) : 1.f - __expf(bf2f(a.g[(size_t)bh * M + m]));
  }
  if (rk == 0) *reinterpret_cast<float4*>(eg + 4 * ck) = e4;
  for (int i = tid; i < NG * W; i += kLogThreads) win[i] = bf2f(a.win_logits[hq0 * W + i]);
  // ---- hk <- hk e^g + k s^T
#pragma unroll
  for (int j = 0; j < JK; ++j) {
    hk[j].x = hk[j].x * e4.x + kv[j] * s4.x;
    hk[j].y = hk[j].y * e4.y + kv[j] * s4.y;
    hk[j].z = hk[j].z * e4.z + kv[j] * s4.z;
    hk[j].w = hk[j].w * e4.w + kv[j] * s4.w;
    hkp[j * kLogThreads] = hk[j];
  }
  // ---- slot logits q hk, one head at a time
  for (int qh = 0; qh < NG; ++qh) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < JK; ++j) {
      const float x = bf2f(qv[j]) * a.scale;
      if (qh + 1 < NG) qv[j] = __ldg(a.q + (hq0 + qh + 1) * D + rk + RK * j);
      acc.x += x * hk[j].x; acc.y += x * hk[j].y; acc.z += x * hk[j].z; acc.w += x * hk[j].w;
    }
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
    acc.z += __shfl_xor_sync(0xffffffffu, acc.z, 16);
    acc.w += __shfl_xor_sync(0xffffffffu, acc.w, 16);
    if (qh > 0) __syncthreads();                                         // the sums of the head before have been read
    if (lane < M4) *reinterpret_cast<float4*>(part + warp * M + 4 * lane) = acc;
    __syncthreads();
    if (tid < M) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < kLogWarps; ++w) t += part[w * M + tid];
      prob[qh * M + tid] = t;
    }
  }
  __syncthreads();
  // ---- joint softmax of a head's slot and window logits, one warp per head
  for (int qh = warp; qh < NG; qh += kLogWarps) {
    float* pr = prob + qh * M;
    float* wi = win + qh * W;
    float mx = fmaxf(pr[lane], pr[lane + 32]);
    for (int w = lane; w < W; w += 32) mx = fmaxf(mx, wi[w]);
    mx = warp_max(mx);
    const float p0 = __expf(pr[lane] - mx), p1 = __expf(pr[lane + 32] - mx);
    float sum = p0 + p1;
    for (int w = lane; w < W; w += 32) {
      const float e = __expf(wi[w] - mx);
      wi[w] = e;
      sum += e;
    }
    sum = warp_sum(sum);
    pr[lane] = p0 / sum;
    pr[lane + 32] = p1 / sum;
    if (a.win_prob)
      for (int w = lane; w < W; w += 32) a.win_prob[(hq0 + qh) * W + w] = wi[w] / sum;
  }
  // ---- hv <- diag(e^g) hv + s v^T
#pragma unroll
  for (int j = 0; j < JV; ++j) {
    const float e = eg[rv + RV * j];
    hv[j].x = hv[j].x * e + sr[j] * v4.x;
    hv[j].y = hv[j].y * e + sr[j] * v4.y;
    hv[j].z = hv[j].z * e + sr[j] * v4.z;
    hv[j].w = hv[j].w * e + sr[j] * v4.w;
    hvp[j * kLogThreads] = hv[j];
  }
  // ---- readout p hv
  for (int qh = 0; qh < NG; ++qh) {
    __syncthreads();                                                     // the weights are complete; part is free
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int j = 0; j < JV; ++j) {
      const float p = prob[qh * M + rv + RV * j];
      acc.x += p * hv[j].x; acc.y += p * hv[j].y; acc.z += p * hv[j].z; acc.w += p * hv[j].w;
    }
    if (D == 64) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, 16);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, 16);
      acc.z += __shfl_xor_sync(0xffffffffu, acc.z, 16);
      acc.w += __shfl_xor_sync(0xffffffffu, acc.w, 16);
    }
    if (lane < D4) *reinterpret_cast<float4*>(part + warp * D + 4 * lane) = acc;
    __syncthreads();
    if (tid < D) {
      float t = 0.f;
#pragma unroll
      for (int w = 0; w < kLogWarps; ++w) t += part[w * D + tid];
      a.o[(hq0 + qh) * D + tid] = f2bf(t);
    }
  }
}

static int logits_smem(int D, int NG, int W) { return (kLogWarps * (D > 64 ? D : 64) + 64 + NG * (64 + W)) * 4; }

// Up to eight heads a group, whose heads each cost two block barriers here; larger groups have not been measured and stay with the
// general kernel.  A CTA per (sequence, kv head) pays from the smallest grid on, kernel time against the general kernel's, windows of
// 32 and 512 logits: one head of 64, 1 sequence 2.8 / 6.4 and 3.6 / 7.1 us; 16 heads of 64, 4 sequences 3.2 / 6.7 and 3.7 / 7.4, 64
// sequences 10.5 / 26.9 and 12.6 / 30.2; 32 heads of 128 on 4, 1 sequence 6.8 / 18.4 and 7.5 / 20.9, 64 sequences 9.6 / 29.1 and
// 10.6 / 41.1.  Vectors of eight bytes are loaded from v, s and g.
bool decode_logits_supported(const DecodeArgs& a) {
  const uintptr_t al8 = (uintptr_t)a.v | (uintptr_t)a.s | (uintptr_t)a.g, al16 = (uintptr_t)a.hk | (uintptr_t)a.hv;
  return a.win_logits && a.K == a.V && (a.K == 64 || a.K == 128) && a.M == 64 && a.NG <= 8 && logits_smem(a.K, a.NG, a.W) <= 48 * 1024 &&
         !(al8 & 7) && !(al16 & 15);
}

int decode_logits_launch(const DecodeArgs& a, cudaStream_t cs) {
  const int smem = logits_smem(a.K, a.NG, a.W);
  if (a.K == 64) nha_decode_logits_kernel<64><<<a.B * a.H, kLogThreads, smem, cs>>>(a);
  else nha_decode_logits_kernel<128><<<a.B * a.H, kLogThreads, smem, cs>>>(a);
  return check_launch();
}

}  // namespace nha
