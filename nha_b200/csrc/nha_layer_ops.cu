// Element-wise work of the calling layer on either side of the operator, one pass each (sm_100a, HBM-bound).
//
//   * Feature map and value activation (nha_fla/layers/nha.py:219-223): q_gsa = swish(q), k_gsa = swish(k),
//     v = silu(v) - the layer launches three element-wise torch kernels (SwishFeatureMap is x * sigmoid(x), the
//     same function as silu; feature_map='relu' is max(x, 0)).  nha_act3_fwd / nha_act3_bwd take up to three tensors
//     in ONE launch.
//   * Output side (nha_fla/layers/nha.py:277-278): o = rms_norm_linear(silu(o), g_norm.weight, g_norm.bias,
//     o_proj.weight, o_proj.bias).  nha_silu_rmsnorm_fwd / _bwd fuse silu, the RMS normalisation and its affine part
//     into one pass over the rows (forward: one warp per row, the row held in registers), leaving the projection itself to
//     the GEMM library.  The backward also produces the gradients of the norm's weight and bias: per-CTA column sums in
//     registers, written as partial rows that a second launch adds up.
//
// fp32 arithmetic, one rounding to bf16 per output, 16-byte accesses.
#include "nha_common.cuh"

namespace nha {

constexpr int kActThreads = 256;
constexpr int kActVecFwd = 4, kActVecBwd = 2;        // 16-byte vectors of each operand in flight per thread

struct Act3 {
  const bf16* x[3];
  const bf16* dy[3];
  bf16* y[3];
  int64_t n[3];
  int relu[3];       // 1: max(x, 0) instead of x * sigmoid(x)
  unsigned first[3]; // first CTA of a tensor
};

__device__ __forceinline__ float sigmoid_fast(float x) { return __fdividef(1.0f, 1.0f + __expf(-x)); }
__device__ __forceinline__ float act_fwd(float x, int relu) { return relu ? fmaxf(x, 0.0f) : x * sigmoid_fast(x); }
// d/dx x sigmoid(x) = sigmoid(x) (1 + x (1 - sigmoid(x)))
__device__ __forceinline__ float act_grad(float x, float dy, int relu) {
  if (relu) return x > 0.0f ? dy : 0.0f;
  const float s = sigmoid_fast(x);
  return dy * s * (1.0f + x * (1.0f - s));
}

// One CTA = one block of kActThreads x ACTV vectors of one tensor.  HBM-bound; blocks are handed out as CTAs finish, because a
// fixed number of them striding through the tensors left SMs idle at the end of each.  3 x 64 MB, forward 75 -> 58 us, backward
// 123 -> 90 us.
template <bool BWD>
__global__ void __launch_bounds__(kActThreads) nha_act3_kernel(const __grid_constant__ Act3 a) {
  constexpr int V = BWD ? kActVecBwd : kActVecFwd;
  const int t = blockIdx.x >= a.first[2] ? 2 : blockIdx.x >= a.first[1] ? 1 : 0;
  const int64_t n = a.n[t];
  const int relu = a.relu[t];
  const int64_t nvec = n >> 3, i0 = (int64_t)(blockIdx.x - a.first[t]) * (kActThreads * V) + threadIdx.x;
  const uint4* x4 = reinterpret_cast<const uint4*>(a.x[t]);
  const uint4* d4 = reinterpret_cast<const uint4*>(a.dy[t]);
  uint4* y4 = reinterpret_cast<uint4*>(a.y[t]);
  uint4 xin[V], din[V];
#pragma unroll
  for (int u = 0; u < V; ++u) {
    const int64_t i = i0 + u * kActThreads;
    if (i < nvec) {
      xin[u] = __ldcs(x4 + i);
      if (BWD) din[u] = __ldcs(d4 + i);
    }
  }
#pragma unroll
  for (int u = 0; u < V; ++u) {
    const int64_t i = i0 + u * kActThreads;
    if (i >= nvec) continue;
    float xv[8], dv[8], out[8];
    unpack8(xin[u], xv);
    if (BWD) unpack8(din[u], dv);
#pragma unroll
    for (int e = 0; e < 8; ++e) out[e] = BWD ? act_grad(xv[e], dv[e], relu) : act_fwd(xv[e], relu);
    y4[i] = pack8(out);
  }
  if (blockIdx.x == a.first[t]) {               // ragged tail (n not a multiple of 8)
    const int64_t i = (nvec << 3) + threadIdx.x;
    if (i < n) {
      const float xv = bf2f(a.x[t][i]);
      a.y[t][i] = f2bf(BWD ? act_grad(xv, bf2f(a.dy[t][i]), relu) : act_fwd(xv, relu));
    }
  }
}

static int wave_grid(int64_t work_items, int64_t per_cta, int ctas_per_sm) {
  const int64_t want = (work_items + per_cta - 1) / per_cta;
  const int64_t cap = (int64_t)sm_count() * ctas_per_sm;
  return (int)(want < 1 ? 1 : (want < cap ? want : cap));
}
static bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// ---------------------------------------------------------------------------------------------
// y = rmsnorm(silu(o)) * w + b, one warp per row.  PIECES = cols / 256: 16-byte pieces of the row per lane.
constexpr int kNormThreads = 256;
constexpr int kNormWarps = kNormThreads / 32;

template <int PIECES>
__global__ void __launch_bounds__(kNormThreads) nha_silu_rmsnorm_fwd_kernel(const bf16* __restrict__ o, const float* __restrict__ w,
                                                                            const float* __restrict__ b, bf16* __restrict__ y,
                                                                            float* __restrict__ rstd, int64_t rows, int cols,
                                                                            float eps) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t wstride = (int64_t)gridDim.x * kNormWarps;
  for (int64_t r = (int64_t)blockIdx.x * kNormWarps + warp; r < rows; r += wstride) {
    const uint4* src = reinterpret_cast<const uint4*>(o + r * cols);
    uint4 in[PIECES];
#pragma unroll
    for (int p = 0; p < PIECES; ++p) in[p] = __ldcs(src + lane + 32 * p);
    float x[PIECES][8];
    float ss = 0.f;
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      unpack8(in[p], x[p]);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        x[p][e] = x[p][e] * sigmoid_fast(x[p][e]);
        ss += x[p][e] * x[p][e];
      }
    }
    ss = warp_sum(ss);
    const float rs = rsqrtf(ss / (float)cols + eps);
    if (lane == 0 && rstd) rstd[r] = rs;
    uint4* dst = reinterpret_cast<uint4*>(y + r * cols);
#pragma unroll
    for (int p = 0; p < PIECES; ++p) {
      const int c = 8 * (lane + 32 * p);
      const float4 w0 = *reinterpret_cast<const float4*>(w + c), w1 = *reinterpret_cast<const float4*>(w + c + 4);
      float4 b0 = make_float4(0.f, 0.f, 0.f, 0.f), b1 = b0;
      if (b) {
        b0 = *reinterpret_cast<const float4*>(b + c);
        b1 = *reinterpret_cast<const float4*>(b + c + 4);
      }
      float out[8];
      out[0] = x[p][0] * rs * w0.x + b0.x; out[1] = x[p][1] * rs * w0.y + b0.y;
      out[2] = x[p][2] * rs * w0.z + b0.z; out[3] = x[p][3] * rs * w0.w + b0.w;
      out[4] = x[p][4] * rs * w1.x + b1.x; out[5] = x[p][5] * rs * w1.y + b1.y;
      out[6] = x[p][6] * rs * w1.z + b1.z; out[7] = x[p][7] * rs * w1.w + b1.w;
      dst[lane + 32 * p] = pack8(out);
    }
  }
}

// Backward of the above for dy (gradient of y).  With x = silu(o), xh = x rstd, dyh = dy w, c = mean(dyh xh):
//     dx = (dyh - xh c) rstd,  do = dx silu'(o),  dw[j] += dy xh,  db[j] += dy.
// A row belongs to PIECES warps, eight columns to a thread: dw / db are then sixteen sums in registers over all rows that the
// thread sees (one partial row per CTA: part_w, part_b [gridDim.x][cols] fp32), and the two rows in work with the two on their
// way fit 128 registers, four CTAs of four warps per SM.  With a warp per row, 32 columns to a lane, it took 250 registers and
// left one CTA of eight warps per SM with two rows each in flight: 32768 x 1024, 57 -> 46 us (HBM floor 31).
constexpr int kNormRows = 2, kNormCtas = 4;               // rows of a team in work; CTAs per SM
__host__ __device__ constexpr int norm_teams(int pieces) { return pieces >= 4 ? 1 : 4 / pieces; }

template <int PIECES>
__global__ void __launch_bounds__(32 * PIECES * norm_teams(PIECES), PIECES >= 5 ? 2 : kNormCtas)
    nha_silu_rmsnorm_bwd_kernel(const bf16* __restrict__ o, const float* __restrict__ w, const float* __restrict__ rstd,
                                const bf16* __restrict__ dy, bf16* __restrict__ d_o, float* __restrict__ part_w,
                                float* __restrict__ part_b, int64_t rows) {
  constexpr int TEAMS = norm_teams(PIECES), cols = 256 * PIECES, R = kNormRows;
  __shared__ float red[2][TEAMS][R][PIECES];
  __shared__ float comb[TEAMS > 1 ? TEAMS - 1 : 1][TEAMS > 1 ? 2 * cols : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, team = warp / PIECES, piece = warp - team * PIECES;
  const int c = 256 * piece + 8 * lane;
  const float4 w0 = *reinterpret_cast<const float4*>(w + c), w1 = *reinterpret_cast<const float4*>(w + c + 4);
  const float wv[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
  float aw[8], ab[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) aw[e] = ab[e] = 0.f;
  uint4 on[R], dn[R];
  float rn[R];
  auto request = [&](int64_t r0) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      const int64_t r = r0 + i;
      on[i] = dn[i] = make_uint4(0u, 0u, 0u, 0u);
      rn[i] = 0.f;
      if (r < rows) {
        on[i] = __ldcs(reinterpret_cast<const uint4*>(o + r * cols + c));
        dn[i] = __ldcs(reinterpret_cast<const uint4*>(dy + r * cols + c));
        rn[i] = __ldg(rstd + r);
      }
    }
  };
  const int64_t step = (int64_t)gridDim.x * TEAMS * R;
  request(((int64_t)blockIdx.x * TEAMS + team) * R);
  int buf = 0;
  for (int64_t b0 = (int64_t)blockIdx.x * TEAMS * R; b0 < rows; b0 += step, buf ^= 1) {     // the same trips for every warp
    const int64_t r0 = b0 + team * R;
    uint4 oc[R], dc[R];
    float rc[R], sg[R][8];
#pragma unroll
    for (int i = 0; i < R; ++i) { oc[i] = on[i]; dc[i] = dn[i]; rc[i] = rn[i]; }
    request(r0 + step);
#pragma unroll
    for (int i = 0; i < R; ++i) {
      float ov[8], dv[8], cs = 0.f;
      unpack8(oc[i], ov);
      unpack8(dc[i], dv);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        sg[i][e] = sigmoid_fast(ov[e]);
        const float xh = ov[e] * sg[i][e] * rc[i];
        cs += dv[e] * wv[e] * xh;
        aw[e] += dv[e] * xh;
        ab[e] += dv[e];
      }
      cs = warp_sum(cs);
      if (lane == 0) red[buf][team][i][piece] = cs;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < R; ++i) {
      if (r0 + i >= rows) continue;
      float cs = 0.f;
#pragma unroll
      for (int p = 0; p < PIECES; ++p) cs += red[buf][team][i][p];
      cs /= (float)cols;
      float ov[8], dv[8], out[8];
      unpack8(oc[i], ov);
      unpack8(dc[i], dv);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float sv = sg[i][e], xh = ov[e] * sv * rc[i], dx = (dv[e] * wv[e] - xh * cs) * rc[i];
        out[e] = dx * sv * (1.0f + ov[e] * (1.0f - sv));
      }
      *reinterpret_cast<uint4*>(d_o + (r0 + i) * cols + c) = pack8(out);
    }
  }
  if (TEAMS > 1) {
    if (team > 0) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        comb[team - 1][c + e] = aw[e];
        comb[team - 1][cols + c + e] = ab[e];
      }
    }
    __syncthreads();
    if (team > 0) return;
#pragma unroll
    for (int t = 0; t < TEAMS - 1; ++t)
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        aw[e] += comb[t][c + e];
        ab[e] += comb[t][cols + c + e];
      }
  }
  float* pw = part_w + (size_t)blockIdx.x * cols + c;
  *reinterpret_cast<float4*>(pw) = make_float4(aw[0], aw[1], aw[2], aw[3]);
  *reinterpret_cast<float4*>(pw + 4) = make_float4(aw[4], aw[5], aw[6], aw[7]);
  if (part_b) {
    float* pb = part_b + (size_t)blockIdx.x * cols + c;
    *reinterpret_cast<float4*>(pb) = make_float4(ab[0], ab[1], ab[2], ab[3]);
    *reinterpret_cast<float4*>(pb + 4) = make_float4(ab[4], ab[5], ab[6], ab[7]);
  }
}

// Column sums of the partial rows: 32 columns to a CTA, 32 groups of rows; blockIdx.y: weight or bias.  592 x 1024: 3.5 us (the
// library's sum over 296 rows: 9.8 us).
__global__ void __launch_bounds__(1024) nha_norm_part_sum_kernel(const float* __restrict__ pw, const float* __restrict__ pb,
                                                                 float* __restrict__ dw, float* __restrict__ db, int parts, int cols) {
  __shared__ float red[32][33];
  const float* p = blockIdx.y ? pb : pw;
  const int cx = threadIdx.x & 31, g = threadIdx.x >> 5, c = 32 * blockIdx.x + cx;
  float s = 0.f;
#pragma unroll 8
  for (int r = g; r < parts; r += 32) s += p[(size_t)r * cols + c];
  red[g][cx] = s;
  __syncthreads();
  const float t = warp_sum(red[cx][g]);
  if (cx == 0) (blockIdx.y ? db : dw)[32 * blockIdx.x + g] = t;
}


}  // namespace nha

using namespace nha;

static int act3_launch(bool bwd, const void* const* x, const void* const* dy, void* const* y, const int64_t* n, const int* relu,
                       int count, void* stream) {
  if (count < 1 || count > 3 || !x || !y || !n) return NHA_ERR_BAD_ARG;
  Act3 a;
  int64_t ctas = 0;
  const int64_t per = (int64_t)kActThreads * 8 * (bwd ? kActVecBwd : kActVecFwd);
  for (int t = 0; t < 3; ++t) {
    a.x[t] = nullptr; a.dy[t] = nullptr; a.y[t] = nullptr; a.n[t] = 0; a.relu[t] = 0;
    a.first[t] = (unsigned)ctas;               // a tensor without elements has no CTA: the next one starts at the same number
    if (t >= count) continue;
    if (n[t] < 0) return NHA_ERR_BAD_ARG;
    if (n[t] == 0) continue;
    if (!x[t] || !y[t] || (bwd && (!dy || !dy[t]))) return NHA_ERR_BAD_ARG;
    if (!aligned16(x[t]) || !aligned16(y[t]) || (bwd && !aligned16(dy[t]))) return NHA_ERR_BAD_ARG;
    a.x[t] = (const bf16*)x[t]; a.y[t] = (bf16*)y[t]; a.n[t] = n[t];
    if (bwd) a.dy[t] = (const bf16*)dy[t];
    a.relu[t] = relu ? relu[t] : 0;
    ctas += (n[t] + per - 1) / per;
    if (ctas > 0x7fffffff) return NHA_ERR_UNSUPPORTED;
  }
  if (ctas == 0) return NHA_OK;
  const unsigned grid = (unsigned)ctas;
  if (bwd) nha_act3_kernel<true><<<grid, kActThreads, 0, (cudaStream_t)stream>>>(a);
  else nha_act3_kernel<false><<<grid, kActThreads, 0, (cudaStream_t)stream>>>(a);
  return check_launch();
}

extern "C" int nha_act3_fwd(const void* const* x, void* const* y, const int64_t* n, const int* relu, int count, void* stream) {
  return act3_launch(false, x, nullptr, y, n, relu, count, stream);
}
extern "C" int nha_act3_bwd(const void* const* x, const void* const* dy, void* const* dx, const int64_t* n, const int* relu,
                            int count, void* stream) {
  return act3_launch(true, x, dy, dx, n, relu, count, stream);
}

extern "C" int nha_silu_rmsnorm_fwd(const void* o, const float* weight, const float* bias, void* y, float* rstd, int64_t rows,
                                    int cols, float eps, void* stream) {
  if (!o || !weight || !y || rows < 0 || cols <= 0 || !(eps >= 0.0f)) return NHA_ERR_BAD_ARG;
  if (cols % 256 || cols > 2048) return NHA_ERR_UNSUPPORTED;
  if (!aligned16(o) || !aligned16(y) || !aligned16(weight) || !aligned16(bias)) return NHA_ERR_BAD_ARG;
  if (rows == 0) return NHA_OK;
  if (rows > (int64_t)0x7fffffff * kNormWarps) return NHA_ERR_UNSUPPORTED;
  const unsigned grid = (unsigned)((rows + kNormWarps - 1) / kNormWarps);
  cudaStream_t cs = (cudaStream_t)stream;
#define NHA_NORM_FWD(P)                                                                                                  \
  case P:                                                                                                                \
    nha_silu_rmsnorm_fwd_kernel<P><<<grid, kNormThreads, 0, cs>>>((const bf16*)o, weight, bias, (bf16*)y, rstd, rows, cols, eps); \
    break;
  switch (cols / 256) {
    NHA_NORM_FWD(1) NHA_NORM_FWD(2) NHA_NORM_FWD(3) NHA_NORM_FWD(4) NHA_NORM_FWD(5) NHA_NORM_FWD(6) NHA_NORM_FWD(7) NHA_NORM_FWD(8)
    default: return NHA_ERR_UNSUPPORTED;
  }
#undef NHA_NORM_FWD
  return check_launch();
}

extern "C" int nha_silu_rmsnorm_bwd_ctas(int64_t rows) { return rows <= 0 ? 0 : wave_grid(rows, 8, kNormCtas); }

extern "C" int nha_silu_rmsnorm_bwd(const void* o, const float* weight, const float* rstd, const void* dy, void* d_o,
                                    float* part_w, float* part_b, int64_t rows, int cols, void* stream) {
  if (!o || !weight || !rstd || !dy || !d_o || !part_w || rows < 0 || cols <= 0) return NHA_ERR_BAD_ARG;
  if (cols % 256 || cols > 2048) return NHA_ERR_UNSUPPORTED;
  if (!aligned16(o) || !aligned16(dy) || !aligned16(d_o) || !aligned16(weight) || !aligned16(part_w) || !aligned16(part_b))
    return NHA_ERR_BAD_ARG;
  if (rows == 0) return NHA_OK;
  const int grid = nha_silu_rmsnorm_bwd_ctas(rows);
  cudaStream_t cs = (cudaStream_t)stream;
#define NHA_NORM_BWD(P)                                                                                                    \
  case P:                                                                                                                  \
    nha_silu_rmsnorm_bwd_kernel<P><<<grid, 32 * P * norm_teams(P), 0, cs>>>((const bf16*)o, weight, rstd, (const bf16*)dy, \
                                                                            (bf16*)d_o, part_w, part_b, rows);             \
    break;
  switch (cols / 256) {
    NHA_NORM_BWD(1) NHA_NORM_BWD(2) NHA_NORM_BWD(3) NHA_NORM_BWD(4) NHA_NORM_BWD(5) NHA_NORM_BWD(6) NHA_NORM_BWD(7) NHA_NORM_BWD(8)
    default: return NHA_ERR_UNSUPPORTED;
  }
#undef NHA_NORM_BWD
  return check_launch();
}

extern "C" int nha_silu_rmsnorm_part_sum(const float* part_w, const float* part_b, float* dw, float* db, int parts, int cols,
                                         void* stream) {
  if (!part_w || !dw || (!part_b != !db) || parts < 0 || cols <= 0) return NHA_ERR_BAD_ARG;
  if (cols % 32) return NHA_ERR_UNSUPPORTED;
  nha_norm_part_sum_kernel<<<dim3(cols / 32, part_b ? 2 : 1), 1024, 0, (cudaStream_t)stream>>>(part_w, part_b, dw, db, parts, cols);
  return check_launch();
}
