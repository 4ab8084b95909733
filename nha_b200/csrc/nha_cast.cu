// Type conversion of several tensors in one launch.
//
// A call of the operator with fp32 or fp16 tensors converts seven inputs on the way in and seven gradients on the way out.
// One element-wise launch per tensor is 2-4 us of GPU time and as much host time each whatever the size, which is most of a
// small call; here they are one launch, bound by HBM (6 bytes per fp32 <-> bf16 element) once the tensors are large.
#include <cuda_fp16.h>

#include "nha_common.cuh"

namespace nha {

struct CastArgs {
  const void* src[8];
  void* dst[8];
  int64_t first[9];      // first 8-element piece of each tensor; first[count] is the total
  int64_t n[8];
  int count, vec;        // vec: every pointer is 16-byte aligned
};

template <typename T> __device__ __forceinline__ float to_f(T x) { return (float)x; }
template <> __device__ __forceinline__ float to_f<bf16>(bf16 x) { return __bfloat162float(x); }
template <> __device__ __forceinline__ float to_f<__half>(__half x) { return __half2float(x); }
template <typename T> __device__ __forceinline__ T from_f(float x) { return (T)x; }
template <> __device__ __forceinline__ bf16 from_f<bf16>(float x) { return __float2bfloat16_rn(x); }
template <> __device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }

template <typename S, typename D>
__global__ void __launch_bounds__(256) nha_cast_kernel(const CastArgs a) {
  const int64_t total = a.first[a.count];
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    int t = 0;
    while (i >= a.first[t + 1]) ++t;
    const int64_t e = 8 * (i - a.first[t]);
    const S* src = (const S*)a.src[t] + e;
    D* dst = (D*)a.dst[t] + e;
    if (a.vec && e + 8 <= a.n[t]) {
      __align__(16) S in[8];
      __align__(16) D out[8];
#pragma unroll
      for (int u = 0; u < (int)(8 * sizeof(S) / 16); ++u) reinterpret_cast<uint4*>(in)[u] = __ldg(reinterpret_cast<const uint4*>(src) + u);
#pragma unroll
      for (int u = 0; u < 8; ++u) out[u] = from_f<D>(to_f<S>(in[u]));
#pragma unroll
      for (int u = 0; u < (int)(8 * sizeof(D) / 16); ++u) reinterpret_cast<uint4*>(dst)[u] = reinterpret_cast<uint4*>(out)[u];
    } else {
      for (int u = 0; u < 8 && e + u < a.n[t]; ++u) dst[u] = from_f<D>(to_f<S>(src[u]));
    }
  }
}

}  // namespace nha

using namespace nha;

extern "C" int nha_cast_many(const void* const* src, void* const* dst, const int64_t* n, int count, int src_type, int dst_type, void* stream) {
  if (!src || !dst || !n || count < 1 || count > 8) return NHA_ERR_BAD_ARG;
  CastArgs a;
  a.count = count;
  a.first[0] = 0;
  a.vec = 1;
  for (int i = 0; i < count; ++i) {
    if (n[i] < 0 || (n[i] > 0 && (!src[i] || !dst[i]))) return NHA_ERR_BAD_ARG;
    a.src[i] = src[i];
    a.dst[i] = dst[i];
    a.n[i] = n[i];
    a.first[i + 1] = a.first[i] + (n[i] + 7) / 8;
    if (((uintptr_t)src[i] | (uintptr_t)dst[i]) & 15) a.vec = 0;
  }
  const int64_t total = a.first[count];
  if (total == 0) return NHA_OK;
  const int64_t want = (total + 255) / 256, most = (int64_t)sm_count() * 8;     // whole waves of eight 256-thread CTAs per SM
  const dim3 grid((unsigned)(want < most ? want : most));
  cudaStream_t cs = (cudaStream_t)stream;
#define NHA_CAST(s_, d_, S_, D_) if (src_type == s_ && dst_type == d_) { nha_cast_kernel<S_, D_><<<grid, 256, 0, cs>>>(a); return check_launch(); }
  NHA_CAST(NHA_FP32, NHA_BF16, float, bf16)
  NHA_CAST(NHA_BF16, NHA_FP32, bf16, float)
  NHA_CAST(NHA_FP16, NHA_BF16, __half, bf16)
  NHA_CAST(NHA_BF16, NHA_FP16, bf16, __half)
#undef NHA_CAST
  return NHA_ERR_UNSUPPORTED;
}
