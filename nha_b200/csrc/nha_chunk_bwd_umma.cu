// Backward of the chunked NHA operator on the sm_100a tensor-core path (tcgen05.mma, accumulators in
// tensor memory) at head dim 128 (head dim 64: nha_chunk_bwd_slot64.cu).  Two chunk-parallel passes bracket the state-gradient scan of
// nha_chunk_bwd.cu: the rows pass (nha_chunk_bwd_rows128.cu) and the columns pass (here).
//
//   rows pass  (per chunk, kv head; query-row side)
//       ok, p_slot recomputed as in the forward;  dp_slot = exp(G) .* (do Hv^T) + a .* (tril(do v'^T) SB)
//       dz_slot = p (dp - delta) + d_lse_gsa softmax(ok);  dz_win = p_win (do v_win^T - delta)
//       dq_gsa = scale (dz exp G) Hk^T + tril(scale (dz a) SB^T) k',   dq_swa = scale dz_win k_swa
//       stores delta, the joint LSE, dgA = ok dz + p dp, and the bf16 copies of dz and p (decayed by
//       exp(G) for the march, by a for the columns pass)
//   columns pass (per chunk, kv head; key-row side), after the march has left DK, DV at every chunk end
//       dk' = tril(dza SB^T)^T q + sbe DK^T,   dv' = tril(pa SB^T)^T do + sbe DV
//       ds' = b .* (tril(q k'^T)^T dza + tril(do v'^T)^T pa) + be .* (k' DK + v' DV^T)
//       dg  = reverse cumulative sum of dgA - s' ds' inside the chunk + carry <DK,hk> + <DV,hv>
//       un-shifted stores of dk_gsa, dv (+ window part), ds, dg
//   (SB = s' .* b, sbe = s' .* exp(Gend - G), a = exp(G - R), b = exp(R - G), R = Gend / 2 per slot.)
// Transposed products use MN-major operand descriptors, so no tile is ever transposed in memory.
// Chunks the forward flagged (gates too steep for the single reference R) are skipped here and
// handled by the general kernels.
//
// Replaces, with nha_chunk_bwd.cu, ChunkNativeHybridAttentionFunction.backward
// (nha_fla/ops/nha/chunk.py:491-564) and chunk_gsa_bwd_with_lse (nha_fla/ops/nha/chunk_gsa.py:52-122).
#include "nha_bwd_common.cuh"
#include "nha_common.cuh"
#include "nha_umma.cuh"

namespace nha {

using namespace umma;

constexpr int kColsThreads = 256;        // columns pass: two threads per row

// ================================================================================================
// gate-gradient carry and bf16 copies of the state gradients (between the scan and the columns pass)
// ================================================================================================
// For chunk c the gate gradient of every later chunk enters as one number per slot,
//     carry[m] = <DK_end[:, m], hk_next[:, m]> + <DV_end[m, :], hv_next[m, :]>,
// with the states at the end of chunk c (the next chunk's start state; the fp32 final state for the
// last chunk of a sequence).  The same sweep over DK_end / DV_end stores the bf16 operand copies the
// columns pass multiplies with.  One CTA per (chunk, kv head); M == 64.
constexpr int kCarryThreads = 256;
__global__ void __launch_bounds__(kCarryThreads) nha_bwd_gate_carry_kernel(const nha_chunk_desc d, const BwdWs w) {
  grid_dep_wait();
  grid_dep_launch();
  constexpr int M = 64;
  const int H = d.H, N = d.N, K = d.K, V = d.V;
  const int cg = blockIdx.x, h = blockIdx.y;
  const ChunkRec rc = chunk_rec(d, cg);
  const int n = rc.n;
  if (n < 0) return;
  if (!chunk_gate(w, cg, h, H)) return;
  const int ci = rc.ci;
  const int len = rc.len;
  const int nchunks = (len + kChunk - 1) / kChunk;
  const int tid = threadIdx.x, lane = tid & 31;
  const size_t nh = (size_t)n * H + h, ch = (size_t)cg * H + h;
  // per-warp partial sums, added in a fixed order afterwards (no floating-point atomics: the result must not
  // depend on the order in which warps arrive)
  constexpr int kCW = kCarryThreads / 32;
  __shared__ float part_k[kCW][M];
  __shared__ float part_v[kCarryThreads / 32][M];
  const int warp = tid >> 5;
  for (int i = tid; i < kCW * M; i += kCarryThreads) (&part_v[0][0])[i] = 0.f;
  __syncthreads();
  const bool last = ci >= nchunks - 1;
  const bool have_next = !last || (d.d_hkt && d.hkt && d.hvt);
  const float* dkg = w.dkc + ch * K * M;
  const float* dvg = w.dvc + ch * M * V;
  bf16* dkb = w.dkb + ch * K * M;
  bf16* dvb = w.dvb + ch * M * V;
  const bf16* hkn = (const bf16*)d.hk_chunks + ((size_t)(cg + 1) * H + h) * K * M;
  const bf16* hvn = (const bf16*)d.hv_chunks + ((size_t)(cg + 1) * H + h) * M * V;
  const float* hkf = d.hkt ? d.hkt + nh * K * M : nullptr;
  const float* hvf = d.hvt ? d.hvt + nh * M * V : nullptr;
  // DK [K][64]: a thread always owns the same four slots
  float ck[4] = {0.f, 0.f, 0.f, 0.f};
  for (int i = tid; i < K * (M / 4); i += kCarryThreads) {
    const float4 f = *reinterpret_cast<const float4*>(dkg + 4 * (size_t)i);
    float4 nx = make_float4(0.f, 0.f, 0.f, 0.f);
    if (have_next) {
      if (!last) {
        const uint2 u = *reinterpret_cast<const uint2*>(hkn + 4 * (size_t)i);
        const float2 lo2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
        const float2 hi2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        nx = make_float4(lo2.x, lo2.y, hi2.x, hi2.y);
      } else {
        nx = *reinterpret_cast<const float4*>(hkf + 4 * (size_t)i);
      }
    }
    uint2 o;
    *reinterpret_cast<__nv_bfloat162*>(&o.x) = __floats2bfloat162_rn(f.x, f.y);
    *reinterpret_cast<__nv_bfloat162*>(&o.y) = __floats2bfloat162_rn(f.z, f.w);
    *reinterpret_cast<uint2*>(dkb + 4 * (size_t)i) = o;
    ck[0] += f.x * nx.x; ck[1] += f.y * nx.y; ck[2] += f.z * nx.z; ck[3] += f.w * nx.w;
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) ck[e] += __shfl_xor_sync(0xffffffffu, ck[e], 16);
  if (lane < 16) {
#pragma unroll
    for (int e = 0; e < 4; ++e) part_k[warp][4 * lane + e] = ck[e];
  }
  // DV [64][V]: a slot's row is spread over V/4 neighbouring lanes
  const int C4 = V / 4;
  for (int i = tid; i < M * C4; i += kCarryThreads) {
    const int r = i / C4, c = i - r * C4;
    const float4 f = *reinterpret_cast<const float4*>(dvg + 4 * (size_t)i);
    float4 nx = make_float4(0.f, 0.f, 0.f, 0.f);
    if (have_next) {
      if (!last) {
        const uint2 u = *reinterpret_cast<const uint2*>(hvn + 4 * (size_t)i);
        const float2 lo2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
        const float2 hi2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        nx = make_float4(lo2.x, lo2.y, hi2.x, hi2.y);
      } else {
        nx = *reinterpret_cast<const float4*>(hvf + 4 * (size_t)i);
      }
    }
    uint2 o;
    *reinterpret_cast<__nv_bfloat162*>(&o.x) = __floats2bfloat162_rn(f.x, f.y);
    *reinterpret_cast<__nv_bfloat162*>(&o.y) = __floats2bfloat162_rn(f.z, f.w);
    *reinterpret_cast<uint2*>(dvb + 4 * (size_t)i) = o;
    float acc = f.x * nx.x + f.y * nx.y + f.z * nx.z + f.w * nx.w;
    for (int o2 = 1; o2 < C4 && o2 < 32; o2 <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o2);
    if (c == 0) part_v[warp][r] = acc;                 // one writer per (warp, slot): row r belongs to one warp only
  }
  __syncthreads();
  if (tid < M) {
    float sum = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < kCW; ++w8) sum += part_k[w8][tid];
#pragma unroll
    for (int w8 = 0; w8 < kCW; ++w8) sum += part_v[w8][tid];
    w.gcarry[ch * M + tid] = sum;
  }
}

// ================================================================================================
// columns pass
// ================================================================================================
#define NHA_MMA_WAIT()                                   \
  do {                                                   \
    if (!failed && !mbar_wait(mbar, phase)) failed = true;          \
    phase ^= 1;                                          \
    tc_fence_after();                                    \
  } while (0)
#define NHA_SMEM_TO_MMA()                                \
  do {                                                   \
    fence_async_smem();                                  \
    tc_fence_before();                                   \
    __syncthreads();                                     \
    tc_fence_after();                                    \
  } while (0)
// this thread's half of tril of a [R][64] accumulator (row token tk keeps columns i <= tk) -> bf16 A-operand tile
#define NHA_TRIL_TO_SMEM(col0, dst_off)                                                          \
  do {                                                                                           \
    float tv_[32];                                                                               \
    tmem_ld32(tlane + (col0) + 32 * half, tv_);                                                  \
    if (active) {                                                                                \
      _Pragma("unroll") for (int c8 = 0; c8 < 4; ++c8) {                                         \
        float o8[8];                                                                             \
        _Pragma("unroll") for (int e = 0; e < 8; ++e) {                                          \
          const int i_ = 32 * half + 8 * c8 + e;                                                 \
          o8[e] = i_ <= tk ? tv_[8 * c8 + e] : 0.f;                                              \
        }                                                                                        \
        *reinterpret_cast<uint4*>(sm + (dst_off) + sw_off(row, 4 * half + c8)) = pack8(o8);      \
      }                                                                                          \
    }                                                                                            \
  } while (0)

template <int R>
struct ColsLayout {
  static constexpr int D = 128, KT = D / 64;
  static constexpr int kATile = R * 128;
  // per-head tiles and the tril buffers first: together they are dead once the head loop is over and
  // then hold the staged epilogue inputs (gate terms, window dv, s') and the dg scan
  static constexpr int tQ = 0;                          // q_gsa [R][D]
  static constexpr int tDO = tQ + KT * kATile;          // do [R][D]
  static constexpr int tZA = tDO + KT * kATile;         // scale dz a [R][64]
  static constexpr int tPA = tZA + kATile;              // p a [R][64]
  static constexpr int bufA = tPA + kATile;             // tril(A) -> tril(E)
  static constexpr int bufB = bufA + kATile;            // tril(Av) -> tril(Bv)
  static constexpr int tK = bufB + kATile;              // k' [64][D]
  static constexpr int tV = tK + KT * 8192;             // v' [64][D]
  static constexpr int tSB = tV + KT * 8192;            // s' b, after the head loop s' exp(Gend - G)
  static constexpr int tDK = tSB + 8192;                // DK at the chunk end [D][64]
  static constexpr int tDV = tDK + D * 128;             // DV at the chunk end [64][D]
  static constexpr int oG = tDV + KT * 8192;
  static constexpr int oR = oG + 64 * 65 * 4;           // [64] reference, [64] carry
  static constexpr int oBar = oR + 512;
  static constexpr int total = oBar + 64 + 1024;
  // staged epilogue inputs, fp32 rows padded to 16-byte multiples that spread over the banks
  static constexpr int kLdG = 68, kLdV = D + 4, kLdS = 72;
  static constexpr int eG = 0;                          // [64][68] fp32 dgA, then dgraw and its scan
  static constexpr int eV = eG + 64 * kLdG * 4;         // [64][D+4] fp32 window part of dv
  static constexpr int eS = eV + 64 * kLdV * 4;         // [64][72] bf16 s'
  static_assert(eS + 64 * kLdS * 2 <= tK, "the staged epilogue inputs must fit in the per-head tiles");
  static constexpr int kTmemCols = 512;
  static constexpr int cA = 0, cAv = 64, cDK = 128, cDV = 128 + D, cDS = 128 + 2 * D, cDS2 = cA;
};

// Two threads per row, as in the rows pass: the warps w and w + 4 share a TMEM lane quarter and take
// alternate 32-column halves of every 64-column accumulator.
template <int R>
__global__ void __launch_bounds__(kColsThreads, 1) nha_bwd_cols_umma_kernel(const nha_chunk_desc d, const BwdWs w, int* __restrict__ err) {
  grid_dep_wait();
  grid_dep_launch();
  typedef ColsLayout<R> L;
  constexpr int D = L::D, KT = L::KT, TH = R / 64, M = 64, NT = kColsThreads;
  const int H = d.H, HQ = d.HQ, NG = HQ / H, N = d.N;
  const int cg = blockIdx.x, h = blockIdx.y;
  const ChunkRec rc = chunk_rec(d, cg);
  const int n = rc.n;
  if (n < 0) return;
  if (!chunk_gate(w, cg, h, H)) return;
  const int ci = rc.ci;
  const int t0 = rc.t0;
  const int len = rc.len;
  const int c0 = ci * kChunk;
  const int shift = seq_shift(d, n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t ch = (size_t)cg * H + h;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  float* Bs = (float*)(sm + L::oG);                   // cumulative gates, then b = exp(R - G)
  float* ER = (float*)(sm + L::oR);                   // exp(R)
  float* cgv = ER + 64;
  uint64_t* mbar = (uint64_t*)(sm + L::oBar);
  uint32_t* tslot = (uint32_t*)(sm + L::oBar + 16);

  // ---- gate / write-weight loads first, then everything the first head tile needs goes in flight at once -------
  const int lo = 0, hi = len - shift;
  constexpr int kGS = 512 / NT;
  uint4 sreg[kGS], greg[kGS];
#pragma unroll
  for (int j = 0; j < kGS; ++j) {
    const int i = tid + NT * j;
    const int r = i >> 3, c8 = i & 7;
    const int src = c0 + r - shift;
    sreg[j] = make_uint4(0u, 0u, 0u, 0u);
    greg[j] = make_uint4(0u, 0u, 0u, 0u);
    if (src >= lo && src < hi) {
      greg[j] = *reinterpret_cast<const uint4*>((const bf16*)d.g + ((size_t)(t0 + src) * H + h) * M + 8 * c8);
      sreg[j] = *reinterpret_cast<const uint4*>((const bf16*)d.s + ((size_t)(t0 + src) * H + h) * M + 8 * c8);
    }
  }
  float carry_in = 0.f;
  if (tid < 64) carry_in = w.gcarry[ch * M + tid];
  load_sw<D, NT>(sm + L::tK, 8192, (const bf16*)d.k_gsa + ((size_t)t0 * H + h) * D, (int64_t)H * D, c0 - shift, lo, hi, 64, 0, tid);
  load_sw<D, NT>(sm + L::tV, 8192, (const bf16*)d.v + ((size_t)t0 * H + h) * D, (int64_t)H * D, c0 - shift, lo, hi, 64, 0, tid);
  load_sw<64, NT>(sm + L::tDK, 0, w.dkb + ch * D * M, M, 0, 0, D, D, 0, tid);
  load_sw<D, NT>(sm + L::tDV, 8192, w.dvb + ch * M * D, D, 0, 0, M, M, 0, tid);
#define NHA_LOAD_HEAD_TILE(ht_)                                                                                      \
  do {                                                                                                               \
    const int hq0_ = h * NG + (ht_) * TH;                                                                            \
    _Pragma("unroll") for (int t2 = 0; t2 < TH; ++t2) {                                                              \
      load_sw<D, NT>(sm + L::tQ, L::kATile, (const bf16*)d.q_gsa + ((size_t)t0 * HQ + hq0_ + t2) * D,                \
                     (int64_t)HQ * D, c0, 0, len, 64, 64 * t2, tid);                                                 \
      load_sw<D, NT>(sm + L::tDO, L::kATile, (const bf16*)d.d_o + ((size_t)t0 * HQ + hq0_ + t2) * D,                 \
                     (int64_t)HQ * D, c0, 0, len, 64, 64 * t2, tid);                                                 \
      load_sw<64, NT>(sm + L::tZA, 0, w.dza + ((size_t)t0 * HQ + hq0_ + t2) * M, (int64_t)HQ * M, c0, 0, len, 64,    \
                      64 * t2, tid);                                                                                 \
      load_sw<64, NT>(sm + L::tPA, 0, w.paq + ((size_t)t0 * HQ + hq0_ + t2) * M, (int64_t)HQ * M, c0, 0, len, 64,    \
                      64 * t2, tid);                                                                                 \
    }                                                                                                                \
    cp_commit();                                                                                                     \
  } while (0)
  NHA_LOAD_HEAD_TILE(0);
#pragma unroll
  for (int j = 0; j < kGS; ++j) {
    const int i = tid + NT * j;
    const int r = i >> 3, c8 = i & 7;
    float gv[8];
    unpack8(greg[j], gv);
#pragma unroll
    for (int e = 0; e < 8; ++e) Bs[r * 65 + 8 * c8 + e] = gv[e];
  }
  if (tid < 64) cgv[tid] = carry_in;
  if (tid == 0) mbar_init(mbar, 1);
  __syncthreads();
  // inclusive scan along the rows: four threads per column (16 rows each), then the earlier quarters' totals
  {
    const int m = tid & 63, seg = tid >> 6;
    float run = 0.f;
#pragma unroll
    for (int r = 16 * seg; r < 16 * seg + 16; ++r) {
      run += Bs[r * 65 + m];
      Bs[r * 65 + m] = run;
    }
    __syncthreads();
    float add = 0.f;
    for (int s2 = 0; s2 < seg; ++s2) add += Bs[(16 * s2 + 15) * 65 + m];
    __syncthreads();
    if (seg > 0) {
#pragma unroll
      for (int r = 16 * seg; r < 16 * seg + 16; ++r) Bs[r * 65 + m] += add;
    }
    __syncthreads();
  }
  // b = exp(R - G) replaces G in place; s' .* b goes into its swizzled tile (s' .* b .* exp(R) = s' exp(Gend - G)
  // follows after the head loop)
  float rref[8];
  {
    const int c8 = tid & 7;
#pragma unroll
    for (int e = 0; e < 8; ++e) rref[e] = 0.5f * Bs[63 * 65 + 8 * c8 + e];
  }
  __syncthreads();
  if (tid < 8) {
#pragma unroll
    for (int e = 0; e < 8; ++e) ER[8 * tid + e] = __expf(rref[e]);
  }
  uint4 sbe[kGS];                                      // s' exp(Gend - G), written after the head loop
#pragma unroll
  for (int j = 0; j < kGS; ++j) {
    const int i = tid + NT * j;
    const int r = i >> 3, c8 = i & 7;
    float sv[8], o1[8], o2[8];
    unpack8(sreg[j], sv);
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const float b = __expf(rref[e] - Bs[r * 65 + 8 * c8 + e]);
      Bs[r * 65 + 8 * c8 + e] = b;
      o1[e] = sv[e] * b;
      o2[e] = o1[e] * __expf(rref[e]);
    }
    *reinterpret_cast<uint4*>(sm + L::tSB + sw_off(r, c8)) = pack8(o1);
    sbe[j] = pack8(o2);
  }
  if (warp == 0) tmem_alloc(tslot, L::kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  const int quarter = warp & 3, half = warp >> 2;
  const uint32_t tlane = tbase + ((uint32_t)(quarter * 32) << 16);
  uint32_t phase = 0;
  bool failed = false;

  // rows of the R-row products (query rows) and of the 64-row products (key rows)
  const bool active = R == 128 ? true : lane < 16;
  const int row = R == 128 ? quarter * 32 + lane : quarter * 16 + (lane & 15);
  const int tk = row & 63;
  const bool kactive = lane < 16;
  const int krow = quarter * 16 + (lane & 15);
  const bool issuer = uniform(threadIdx.x >> 5) == 0;
  // one round of products by the elected lane of warp 0, committed to the barrier of NHA_MMA_WAIT: f(address of shared memory, tensor memory)
  auto round = [&](auto f) {
    if (issuer) {
      const uint32_t sb = uniform(smem_u32(sm)), tb = uniform(tbase);
      if (elect_one()) {
        f(sb, tb);
        commit(mbar);
      }
    }
  };

  for (int ht = 0; ht < NG / TH; ++ht) {
    if (ht > 0) NHA_LOAD_HEAD_TILE(ht);
    cp_wait_all();
    NHA_SMEM_TO_MMA();
    round([&](uint32_t sb, uint32_t tb) {
      mma_tile(tb + L::cA, sb + L::tQ, L::kATile, sb + L::tK, 8192, R, 64, D / 16, 0, false);         // A  = q k'^T
      mma_tile(tb + L::cAv, sb + L::tDO, L::kATile, sb + L::tV, 8192, R, 64, D / 16, 0, false);       // Av = do v'^T
    });
    NHA_MMA_WAIT();
    NHA_TRIL_TO_SMEM(L::cA, L::bufA);
    NHA_TRIL_TO_SMEM(L::cAv, L::bufB);
    NHA_SMEM_TO_MMA();
    round([&](uint32_t sb, uint32_t tb) {
      // ds' (intra) += tril(A)^T dza + tril(Av)^T pa      (both operands MN-major, k = query row)
      mma_tile_ex(tb + L::cDS, sb + L::bufA, 0, 1, sb + L::tZA, 0, 1, 64, 64, R / 16, ht > 0);
      mma_tile_ex(tb + L::cDS, sb + L::bufB, 0, 1, sb + L::tPA, 0, 1, 64, 64, R / 16, true);
      mma_tile(tb + L::cA, sb + L::tZA, L::kATile, sb + L::tSB, 0, R, 64, 4, 0, false);                // E  = dza SB^T
      mma_tile(tb + L::cAv, sb + L::tPA, L::kATile, sb + L::tSB, 0, R, 64, 4, 0, false);               // Bv = pa SB^T
    });
    NHA_MMA_WAIT();
    NHA_TRIL_TO_SMEM(L::cA, L::bufA);
    NHA_TRIL_TO_SMEM(L::cAv, L::bufB);
    NHA_SMEM_TO_MMA();
    round([&](uint32_t sb, uint32_t tb) {
#pragma unroll
      for (int nb = 0; nb < KT; ++nb) {
        // dk' += tril(E)^T q,  dv' += tril(Bv)^T do      (64 output columns at a time)
        mma_tile_ex(tb + L::cDK + 64 * nb, sb + L::bufA, 0, 1, sb + L::tQ + nb * L::kATile, 0, 1, 64, 64, R / 16, ht > 0);
        mma_tile_ex(tb + L::cDV + 64 * nb, sb + L::bufB, 0, 1, sb + L::tDO + nb * L::kATile, 0, 1, 64, 64, R / 16, ht > 0);
      }
    });
    NHA_MMA_WAIT();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  }
#undef NHA_LOAD_HEAD_TILE
  // ---- inter-chunk parts from the state gradients at the chunk end ------------------------------------------
  // The per-head tiles are dead now: the rows the epilogue needs from global memory (gate terms of the
  // rows pass, window part of dv, s') are fetched into their place while the last products run.
  const int kp = c0 + krow, kj = kp - shift;                     // this thread's key row: shifted position, source token
  const bool keep = kactive && kj >= 0 && kp < len;
  float* eG = (float*)(sm + L::eG);
  float* eV = (float*)(sm + L::eV);
  bf16* eS = (bf16*)(sm + L::eS);
  {
    const float* gsrc = w.dga + ((size_t)t0 * H + h) * M;
    for (int i = tid; i < 64 * 16; i += NT) {
      const int r = i >> 4, c = i & 15;
      const int p = c0 + r;
      const bool ok = p - shift >= 0 && p < len;
      cp16(eG + r * L::kLdG + 4 * c, gsrc + (size_t)(ok ? p : 0) * H * M + 4 * c, ok);
    }
    const float* vsrc = w.dvacc + ((size_t)t0 * H + h) * D;
    for (int i = tid; i < 64 * (D / 4); i += NT) {
      const int r = i / (D / 4), c = i % (D / 4);
      const int p = c0 + r, j = p - shift;
      const bool ok = j >= 0 && p < len;
      cp16(eV + r * L::kLdV + 4 * c, vsrc + (size_t)(ok ? j : 0) * H * D + 4 * c, ok);
    }
    const bf16* ssrc = (const bf16*)d.s + ((size_t)t0 * H + h) * M;
    for (int i = tid; i < 64 * 8; i += NT) {
      const int r = i >> 3, c = i & 7;
      const int p = c0 + r, j = p - shift;
      const bool ok = j >= 0 && p < len;
      cp16(eS + r * L::kLdS + 8 * c, ssrc + (size_t)(ok ? j : 0) * H * M + 8 * c, ok);
    }
    cp_commit();
  }
  // s' exp(Gend - G) replaces s' b (every product that read it has completed)
#pragma unroll
  for (int j = 0; j < kGS; ++j) {
    const int i = tid + NT * j;
    const int r = i >> 3, c8 = i & 7;
    *reinterpret_cast<uint4*>(sm + L::tSB + sw_off(r, c8)) = sbe[j];
  }
  NHA_SMEM_TO_MMA();
  {
    round([&](uint32_t sb, uint32_t tb) {
#pragma unroll
      for (int nb = 0; nb < KT; ++nb) {
        // dk' += sbe DK^T (DK rows kk as the N rows of a K-major operand), dv' += sbe DV (DV as MN-major, k = slot)
        mma_tile(tb + L::cDK + 64 * nb, sb + L::tSB, 0, sb + L::tDK + nb * 8192, 0, 64, 64, 4, 0, true);
        mma_tile(tb + L::cDV + 64 * nb, sb + L::tSB, 0, sb + L::tDV + nb * 8192, 0, 64, 64, 4, 1, true);
      }
      // DS2 = k' DK + v' DV^T
      mma_tile(tb + L::cDS2, sb + L::tK, 8192, sb + L::tDK, 0, 64, 64, D / 16, 1, false);
      mma_tile(tb + L::cDS2, sb + L::tV, 8192, sb + L::tDV, 8192, 64, 64, D / 16, 0, true);
    });
    NHA_MMA_WAIT();
  }
  cp_wait_all();
  __syncthreads();
  // ---- epilogue: two threads per key row, each its half of the columns ----------------------------------------------
  {
    float dsi[32], ds2[32];
    tmem_ld32(tlane + L::cDS + 32 * half, dsi);
    tmem_ld32(tlane + L::cDS2 + 32 * half, ds2);
    if (kactive) {
#pragma unroll
      for (int c8 = 0; c8 < 4; ++c8) {
        const int m0 = 32 * half + 8 * c8;
        float ds8[8], sv[8];
        unpack8(*reinterpret_cast<const uint4*>(eS + krow * L::kLdS + m0), sv);
        float* grow = eG + krow * L::kLdG + m0;
        const float4 g0 = *reinterpret_cast<const float4*>(grow), g1 = *reinterpret_cast<const float4*>(grow + 4);
        const float ga[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        float gr[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const int m = m0 + e;
          // ds' = b .* (intra-chunk part) + exp(Gend - G) .* (inter-chunk part), exp(Gend - G) = b exp(R)
          const float ds = Bs[krow * 65 + m] * (dsi[8 * c8 + e] + ER[m] * ds2[8 * c8 + e]);
          ds8[e] = ds;
          gr[e] = keep ? ga[e] - sv[e] * ds : 0.f;
        }
        *reinterpret_cast<float4*>(grow) = make_float4(gr[0], gr[1], gr[2], gr[3]);
        *reinterpret_cast<float4*>(grow + 4) = make_float4(gr[4], gr[5], gr[6], gr[7]);
        if (keep) *reinterpret_cast<uint4*>((bf16*)d.ds + ((size_t)(t0 + kj) * H + h) * M + m0) = pack8(ds8);
      }
    }
    float ov[32];
#pragma unroll
    for (int pp = 0; pp < D / 64; ++pp) {
      const int part = (D / 64) * half + pp;
      tmem_ld32(tlane + L::cDK + 32 * part, ov);
      if (keep) {
        bf16* orow = (bf16*)d.dk_gsa + ((size_t)(t0 + kj) * H + h) * D + 32 * part;
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) *reinterpret_cast<uint4*>(orow + 8 * c8) = pack8(ov + 8 * c8);
      }
      tmem_ld32(tlane + L::cDV + 32 * part, ov);
      if (keep) {
        const float* wa = eV + krow * L::kLdV + 32 * part;
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const float4 a4 = *reinterpret_cast<const float4*>(wa + e);
          ov[e] += a4.x; ov[e + 1] += a4.y; ov[e + 2] += a4.z; ov[e + 3] += a4.w;
        }
        bf16* orow = (bf16*)d.dv + ((size_t)(t0 + kj) * H + h) * D + 32 * part;
#pragma unroll
        for (int c8 = 0; c8 < 4; ++c8) *reinterpret_cast<uint4*>(orow + 8 * c8) = pack8(ov + 8 * c8);
      }
    }
  }
  // the accumulators are drained: release the tensor memory before the tail of the epilogue
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, L::kTmemCols);
  // reverse cumulative sum of dgraw along the rows (four threads per column), plus the carry
  {
    const int m = tid & 63, seg = tid >> 6;
    float run = 0.f;
#pragma unroll
    for (int r = 16 * seg + 15; r >= 16 * seg; --r) {
      run += eG[r * L::kLdG + m];
      eG[r * L::kLdG + m] = run;
    }
    __syncthreads();
    float add = cgv[m];
    for (int s2 = seg + 1; s2 < 4; ++s2) add += eG[(16 * s2) * L::kLdG + m];
    __syncthreads();                                  // every read of the later quarters' totals precedes their update
#pragma unroll
    for (int r = 16 * seg; r < 16 * seg + 16; ++r) eG[r * L::kLdG + m] += add;
    __syncthreads();
  }
  if (keep) {
#pragma unroll
    for (int c8 = 0; c8 < 4; ++c8) {
      const int m0 = 32 * half + 8 * c8;
      const float* grow = eG + krow * L::kLdG + m0;
      const float4 g0 = *reinterpret_cast<const float4*>(grow), g1 = *reinterpret_cast<const float4*>(grow + 4);
      const float g8[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
      *reinterpret_cast<uint4*>((bf16*)d.dg + ((size_t)(t0 + kj) * H + h) * M + m0) = pack8(g8);
    }
  }
  if (failed) atomicExch(err, 1);
}
#undef NHA_MMA_WAIT
#undef NHA_SMEM_TO_MMA
#undef NHA_TRIL_TO_SMEM

template <int R>
static int launch_cols(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  typedef ColsLayout<R> L;
  cudaError_t e = set_max_smem((const void*)nha_bwd_cols_umma_kernel<R>, L::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  const int NCB = (int)nha_chunk_count_bound(d->Ttot, d->N);
  launch_after(nha_bwd_gate_carry_kernel, dim3(NCB, d->H), kCarryThreads, 0, cs, *d, w);
  int st = check_launch();
  if (st != NHA_OK) return st;
  launch_after(nha_bwd_cols_umma_kernel<R>, dim3(NCB, d->H), kColsThreads, L::total, cs, *d, w, err);
  return check_launch();
}

int bwd_rows128_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs);

bool bwd_umma_supported(const nha_chunk_desc* d) {
  return d->K == 128 && d->V == 128 && d->M == 64 && d->scale > 0.f;
}

// which: 0 = rows pass, 1 = columns pass.  The caller has checked bwd_umma_supported().
int bwd_umma_launch(const nha_chunk_desc* d, const BwdWs& w, int which, int* err, cudaStream_t cs) {
  if (which == 0) return bwd_rows128_launch(d, w, err, cs);
  // two heads to a 128-row tile where the group is even, one head to a 64-row tile where it is odd (2 x 1999 tokens, seven heads
  // a group, whole training pass: 440 us, 1774 us with the general kernels)
  return (d->HQ / d->H) % 2 ? launch_cols<64>(d, w, err, cs) : launch_cols<128>(d, w, err, cs);
}

}  // namespace nha
