// Backward of the chunked NHA operator, key-row side of the slot branch, for head dim 64: 64-row products with every lane at
// work (nha_frag64.cuh).  What it computes is in nha_chunk_bwd_umma.cu, whose columns pass and gate-carry kernel it replaces
// at this head dim.
//
// One CTA = one (chunk, kv head), two CTAs per SM with one query head per kv head.  Rounds of products:
//     x = G - Gend / 2,  y = Gend - G                          (b = exp(-x) and exp(y) in registers, SB = s' b, SBE = s' exp(y))
//     per head:  A = q k'^T,  Av = do v'^T,  E = za SB^T,  Bv = pa SB^T
//                dS += tril(A)^T za + tril(Av)^T pa,  dk' += tril(E)^T q,  dv' += tril(Bv)^T do
//     with the last of them:  dk' += SBE DK^T,  dv' += SBE DV,  dS2 = k' DK + v' DV^T
// (za = scale dz a, pa = p a from the rows pass; DK, DV: gradients of the states at the chunk end, fp32 from the scan, rounded
// to bf16 here.)  ds' = b dS + exp(y) dS2.  dg is the reverse running sum of dga - s' ds' over the chunk's rows (shuffles inside
// a quarter, shared memory across the quarters) plus the carry <DK, hk_next> + <DV, hv_next>, formed in fp32 from the same loads.
//
// Replaces, with the other backward kernels, ChunkNativeHybridAttentionFunction.backward (nha_fla/ops/nha/chunk.py:491-564).
#include <string.h>

#include "nha_bwd_common.cuh"
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

namespace cl64 {
constexpr int tQ = 0, tDO = 1, tZA = 2, tPA = 3, tK = 4, tV = 5, tSB = 6, tSBE = 7, tDK = 8, tDV = 9, b1 = 10, b2 = 11, b3 = 12, kTiles = 13;
constexpr int oPart = kTiles * kTile;                         // fp32 [8 warps][64] column dots of DK, [64] row dots of DV
constexpr int oTot = oPart + 9 * 64 * 4;                      // fp32 [4 quarters][64] totals of the gate terms
constexpr int oBar = oTot + 4 * 64 * 4;
constexpr int total = oBar + 64 + 1024;
static_assert(total <= 113 * 1024, "two CTAs per SM");
}  // namespace cl64

// Tensor maps of the call's tensors (this GPU's own memory).  A tile whose 64 rows lie inside its sequence comes by TMA; the
// others (ragged ends, rows in front of a sequence) are copied piece by piece with zero fill.  use == 0: all tiles are copied
// (fewer than 64 slots, or no tensor maps).
struct ColsMaps {
  CUtensorMap qg, kg, v, g, s, dout, za, pa;
  int use;
};

// ONE: one query head per kv head.  Several heads accumulate in columns of their own (512 columns, one CTA per SM).
template <bool ONE>
__global__ void __launch_bounds__(kThreads, ONE ? 2 : 1) nha_bwd_cols64_kernel(const nha_chunk_desc d, const BwdWs w, int* __restrict__ err,
                                                                                 const __grid_constant__ ColsMaps maps, const unsigned ahead) {
  grid_dep_wait();
  grid_dep_launch();
  using namespace cl64;
  constexpr int c0_ = 0, c1_ = 64, c2_ = 128, c3_ = 192, kTmemCols = ONE ? 256 : 512;
  constexpr int cDS = ONE ? 0 : 256, cDK = ONE ? 64 : 320, cDV = ONE ? 128 : 384, cDS2 = ONE ? 192 : 448;
  const int H = d.H, HQ = d.HQ, M = d.M, NG = ONE ? 1 : HQ / H;
  const int cg = blockIdx.x / H, h = blockIdx.x - cg * H;
  const ChunkRec rc = chunk_rec(d, cg);
  if (rc.n < 0) return;
  if (!chunk_gate(w, cg, h, H)) return;
  const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
  const int shift = seq_shift(d, rc.n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;
  const size_t ch = (size_t)cg * H + h;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* part = (float*)(sm + oPart);
  float* tot = (float*)(sm + oTot);
  uint64_t* mbar = (uint64_t*)(sm + oBar);
  uint32_t* tslot = (uint32_t*)(mbar + 1);   // then the load barriers
  auto tile = [&](int i) { return sm + i * kTile; };

  // ---- loads: gates and write weights first, then the first head's tiles -------------------------------------------------
  const int lr = tid >> 3, lc = tid & 7;
  const uint32_t loff = sw_off(lr, lc);
  const int64_t rq = (int64_t)HQ * 64, rp = (int64_t)H * 64, rm = (int64_t)H * M, rz = (int64_t)HQ * M;
  // load barriers: each phase is closed by one arrival of thread 0 behind its last TMA; bits of lph: their parities
  uint64_t* bl = mbar + 2;                                     // [0] gates and write weights, [1] the rest
  uint32_t lph = 0;
  auto loads_done = [&](int bar) {
    cp_commit();
    if (tid == 0) mbar_arrive(&bl[bar]);
  };
  bool failed = false;
  auto loads_wait = [&](int bar, bool newest) {                // newest == false: a later group may stay in flight
    if (newest) cp_wait_all(); else cp_wait_but_one();
    if (!failed && !mbar_wait(&bl[bar], (lph >> bar) & 1u)) failed = true;
    lph ^= 1u << bar;
  };
  auto load_tokens = [&](int t, const CUtensorMap& map, int head, const void* base, int64_t pitch, int width, int row, int lo, int hi, int bar) {
    if (maps.use && row >= lo && row + kChunk <= hi) {
      if (tid == 0) {
        mbar_expect_more(&bl[bar], kTile);
        tma_load_3d(tile(t), &map, 0, head, t0 + row, &bl[bar]);
      }
    } else {
      const bf16* p = (const bf16*)base + (int64_t)t0 * pitch + head * width + 8 * lc;
      const bool cok = 8 * lc < width;
      const bool ok0 = cok && row + lr >= lo && row + lr < hi, ok1 = cok && row + lr + 32 >= lo && row + lr + 32 < hi;
      tile_in(tile(t), loff, p + (ok0 ? row + lr : 0) * pitch, ok0, p + (ok1 ? row + lr + 32 : 0) * pitch, ok1);
    }
  };
  const bool mcol = 8 * lc < M;
  if (tid == 0) {
    mbar_init(mbar, 1);
    mbar_init(&bl[0], 1);
    mbar_init(&bl[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  load_tokens(b2, maps.g, h, d.g, rm, M, c0 - shift, 0, len - shift, 0);
  load_tokens(tSB, maps.s, h, d.s, rm, M, c0 - shift, 0, len - shift, 0);
  loads_done(0);
  auto load_head = [&](int hq) {
    load_tokens(tQ, maps.qg, hq, d.q_gsa, rq, 64, c0, 0, len, 1);
    load_tokens(tDO, maps.dout, hq, d.d_o, rq, 64, c0, 0, len, 1);
    load_tokens(tZA, maps.za, hq, w.dza, rz, M, c0, 0, len, 1);
    load_tokens(tPA, maps.pa, hq, w.paq, rz, M, c0, 0, len, 1);
    loads_done(1);
  };
  load_tokens(tK, maps.kg, h, d.k_gsa, rp, 64, c0 - shift, 0, len - shift, 1);
  load_tokens(tV, maps.v, h, d.v, rp, 64, c0 - shift, 0, len - shift, 1);
  load_head(h * NG);
  // state gradients at the chunk end and the next chunk's start state, requested into registers beside the tiles: rows lr and
  // lr + 32, eight columns
  const int nchunks = (len + kChunk - 1) / kChunk;
  const bool last = ci >= nchunks - 1, have_next = !last || (d.d_hkt && d.hkt && d.hvt);
  const size_t nh = (size_t)rc.n * H + h;
  const float* hkf = d.hkt ? d.hkt + nh * 64 * M : nullptr;
  const float* hvf = d.hvt ? d.hvt + nh * M * 64 : nullptr;
  float4 gk[2][2], gv[2][2];
  uint4 nk[2], nv[2];
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = lr + 32 * u;
    const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
    gk[u][0] = gk[u][1] = gv[u][0] = gv[u][1] = z;
    nk[u] = nv[u] = make_uint4(0u, 0u, 0u, 0u);
    if (mcol) {
      const float4* p = reinterpret_cast<const float4*>(w.dkc + ch * 64 * M + r * M + 8 * lc);
      gk[u][0] = p[0]; gk[u][1] = p[1];
      if (!last) nk[u] = *reinterpret_cast<const uint4*>((const bf16*)d.hk_chunks + ((size_t)(cg + 1) * H + h) * 64 * M + r * M + 8 * lc);
    }
    if (r < M) {
      const float4* p = reinterpret_cast<const float4*>(w.dvc + ch * M * 64 + r * 64 + 8 * lc);
      gv[u][0] = p[0]; gv[u][1] = p[1];
      if (!last) nv[u] = *reinterpret_cast<const uint4*>((const bf16*)d.hv_chunks + ((size_t)(cg + 1) * H + h) * M * 64 + r * 64 + 8 * lc);
    }
  }
  // The pass waits for its loads: two CTAs an SM keep too few bytes in flight, so each prefetches the inputs of the CTA `ahead`
  // places on into L2, one per SM.  16 x 2048 tokens, 16 heads, W 64: 386 us without it, 325-330 so, 341 and 374 two and three
  // places per SM ahead.
  if (maps.use && tid == 64 && blockIdx.x + ahead < gridDim.x) {
    const int ncg = (blockIdx.x + ahead) / H, nhd = blockIdx.x + ahead - ncg * H;
    const ChunkRec nr = chunk_rec(d, ncg);
    if (nr.n >= 0) {
      const int row = nr.t0 + nr.ci * kChunk;
      const size_t nch = (size_t)ncg * H + nhd;
      prefetch_tile(maps.g, 0, nhd, row);
      prefetch_tile(maps.s, 0, nhd, row);
      prefetch_tile(maps.kg, 0, nhd, row);
      prefetch_tile(maps.v, 0, nhd, row);
      prefetch_tile(maps.qg, 0, nhd * NG, row);
      prefetch_tile(maps.dout, 0, nhd * NG, row);
      prefetch_tile(maps.za, 0, nhd * NG, row);
      prefetch_tile(maps.pa, 0, nhd * NG, row);
      prefetch_bytes(w.dkc + nch * 4096, 16384);
      prefetch_bytes(w.dvc + nch * 4096, 16384);
      prefetch_bytes((const bf16*)d.hk_chunks + nch * 4096, kTile);
      prefetch_bytes((const bf16*)d.hv_chunks + nch * 4096, kTile);
    }
  }
  fill_half_signs(tile(b1), tid);
  {
    // strictly upper triangular ones: row t of y sums the gates of the rows after t
    const int r = tid >> 2;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int c = 2 * (tid & 3) + u;
      uint32_t pr[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 8 * c + 2 * e;
        pr[e] = (i > r ? 0x3F80u : 0u) | (i + 1 > r ? 0x3F800000u : 0u);
      }
      *reinterpret_cast<uint4*>(tile(b3) + sw_off(r, c)) = make_uint4(pr[0], pr[1], pr[2], pr[3]);
    }
  }
  if (warp == 0) tmem_alloc(tslot, kTmemCols);
  __syncthreads();                                             // the barriers are initialised
  loads_wait(0, false);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  const uint32_t tl = tbase + ((uint32_t)(quarter * 32) << 16) + 32 * half;       // this warp's columns of an accumulator at +0
  uint32_t phase = 0;
  auto mma_wait = [&]() {
    if (tid == 0) commit(mbar);
    if (!failed && !mbar_wait(mbar, phase)) failed = true;
    phase ^= 1;
    tc_fence_after();
  };
  auto hand_over = [&]() {
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  };
  const uint32_t sbase = smem_u32(sm);
  auto at = [&](int t, uint32_t off) { return sbase + (uint32_t)(t * kTile) + off; };
  auto desc = [&](int t) { return make_desc(sbase + t * kTile); };
  const uint32_t iKK = idesc64(0, 0), iKM = idesc64(0, 1), iMM = idesc64(1, 1);

  if (tid == 0) {
    mma64<0, 1>(tbase + c0_, desc(b1), desc(b2), iKM, false);          // x
    mma64<0, 1>(tbase + c1_, desc(b3), desc(b2), iKM, false);          // y
  }
  // ---- state gradients at the chunk end: bf16 operands, and the carry's dot products with the next chunk's start state --------
  uint4 dkp[2];                                                        // rows lr, lr + 32 of DK, columns 8 lc .. + 7
  {
    auto next = [&](const uint4& n, const float* fin, int64_t at_, float (&f)[8]) {
      if (last && have_next) {                                         // the fp32 final state stands in for a next chunk's start
        const float4 x = *reinterpret_cast<const float4*>(fin + at_), y = *reinterpret_cast<const float4*>(fin + at_ + 4);
        f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w; f[4] = y.x; f[5] = y.y; f[6] = y.z; f[7] = y.w;
      } else {
        unpack8(n, f);
      }
    };
    float ck[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) ck[e] = 0.f;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = lr + 32 * u;
      dkp[u] = make_uint4(0u, 0u, 0u, 0u);
      if (mcol) {
        const float f[8] = {gk[u][0].x, gk[u][0].y, gk[u][0].z, gk[u][0].w, gk[u][1].x, gk[u][1].y, gk[u][1].z, gk[u][1].w};
        float n[8];
        next(nk[u], hkf, r * M + 8 * lc, n);
#pragma unroll
        for (int e = 0; e < 8; ++e) ck[e] += f[e] * n[e];
        dkp[u] = pack8(f);
      }
      float cv = 0.f;
      uint4 dvp = make_uint4(0u, 0u, 0u, 0u);
      if (r < M) {
        const float f[8] = {gv[u][0].x, gv[u][0].y, gv[u][0].z, gv[u][0].w, gv[u][1].x, gv[u][1].y, gv[u][1].z, gv[u][1].w};
        float n[8];
        next(nv[u], hvf, r * 64 + 8 * lc, n);
#pragma unroll
        for (int e = 0; e < 8; ++e) cv += f[e] * n[e];
        dvp = pack8(f);
      }
      *reinterpret_cast<uint4*>(tile(tDV) + loff + 4096 * u) = dvp;
      cv += __shfl_xor_sync(0xffffffffu, cv, 1);
      cv += __shfl_xor_sync(0xffffffffu, cv, 2);
      cv += __shfl_xor_sync(0xffffffffu, cv, 4);
      if (lc == 0) part[8 * 64 + r] = cv;
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      ck[e] += __shfl_xor_sync(0xffffffffu, ck[e], 8);
      ck[e] += __shfl_xor_sync(0xffffffffu, ck[e], 16);
    }
    if (lane < 8) {
#pragma unroll
      for (int e = 0; e < 8; ++e) part[warp * 64 + 8 * lane + e] = ck[e];
    }
  }
  mma_wait();
  // ---- b = exp(-x), exp(y), SB, SBE; s' stays packed in registers -----------------------------------------------------------
  const uint32_t fo0 = frag_off(quarter, half, lane, 0), fo1 = frag_off(quarter, half, lane, 1);
  const int r0 = 16 * quarter + gq;                            // this lane's key rows: r0 and r0 + 8
  float b[16], ey[16];
  uint32_t s[2][4];
  {
    frag_ld_nowait(tl + c0_, b);
    frag_ld_nowait(tl + c1_, ey);
    tmem_ld_wait();
    ldm4(at(tSB, fo0), s[0]);
    ldm4(at(tSB, fo1), s[1]);
    uint32_t sb[2][4], se[2][4];
#pragma unroll
    for (int jp = 0; jp < 2; ++jp)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = 4 * (2 * jp + (q >> 1)) + 2 * (q & 1);
        const float2 sv = pair_f32(s[jp][q]);
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          b[e + x] = exp2f(-b[e + x] * kLog2e);
          ey[e + x] = exp2f(ey[e + x] * kLog2e);
        }
        sb[jp][q] = pair_bf16(sv.x * b[e], sv.y * b[e + 1]);
        se[jp][q] = pair_bf16(sv.x * ey[e], sv.y * ey[e + 1]);
      }
    stm4(at(tSB, fo0), sb[0][0], sb[0][1], sb[0][2], sb[0][3]);
    stm4(at(tSB, fo1), sb[1][0], sb[1][1], sb[1][2], sb[1][3]);
    stm4(at(tSBE, fo0), se[0][0], se[0][1], se[0][2], se[0][3]);
    stm4(at(tSBE, fo1), se[1][0], se[1][1], se[1][2], se[1][3]);
  }
  auto tril_to = [&](int col, int t) {
    float v[16];
    frag_ld(tl + col, v);
    const int c = 32 * half + 2 * tq;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c + 8 * j + (e & 1) > r0 + 8 * (e >> 1)) v[4 * j + e] = 0.f;
    frag_to_tile(at(t, fo0), at(t, fo1), v);
  };
  // rows of this lane: shifted position p, source token j = p - shift
  bool keep[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int p = c0 + r0 + 8 * i;
    keep[i] = p >= shift && p < len;
  }
  float ga[16];                                                // gate terms of the rows pass, fetched behind the last products
  for (int ht = 0; ht < NG; ++ht) {
    const bool fin = ht + 1 == NG;
    if (!ONE && ht > 0) load_head(h * NG + ht);
    loads_wait(1, true);
    hand_over();
    if (tid == 0) {
      mma64<0, 0>(tbase + c0_, desc(tQ), desc(tK), iKK, false);
      mma64<0, 0>(tbase + c1_, desc(tDO), desc(tV), iKK, false);
      mma64<0, 0>(tbase + c2_, desc(tZA), desc(tSB), iKK, false);
      mma64<0, 0>(tbase + c3_, desc(tPA), desc(tSB), iKK, false);
    }
    if (fin) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int m = 32 * half + 8 * j + 2 * tq;
          const float2 x = keep[i] && m < M ? *reinterpret_cast<const float2*>(w.dga + ((size_t)(t0 + c0 + r0 + 8 * i) * H + h) * M + m)
                                            : make_float2(0.f, 0.f);
          ga[4 * j + 2 * i] = x.x;
          ga[4 * j + 2 * i + 1] = x.y;
        }
    }
    mma_wait();
    // the fourth operand: over s' b once its last reader is done, over DK's tile (written for the last head) before that
    const int b4 = fin ? tSB : tDK;
    tril_to(c0_, b1);
    tril_to(c1_, b2);
    tril_to(c2_, b3);
    tril_to(c3_, b4);
    if (fin) {
      *reinterpret_cast<uint4*>(tile(tDK) + loff) = dkp[0];
      *reinterpret_cast<uint4*>(tile(tDK) + loff + 4096) = dkp[1];
    }
    hand_over();
    if (tid == 0) {
      const bool acc = ht > 0;
      mma64<1, 1>(tbase + cDS, desc(b1), desc(tZA), iMM, acc);
      mma64<1, 1>(tbase + cDK, desc(b3), desc(tQ), iMM, acc);
      mma64<1, 1>(tbase + cDV, desc(b4), desc(tDO), iMM, acc);
      mma64<1, 1>(tbase + cDS, desc(b2), desc(tPA), iMM, true);
      if (fin) {
        mma64<0, 1>(tbase + cDS2, desc(tK), desc(tDK), iKM, false);
        mma64<0, 0>(tbase + cDK, desc(tSBE), desc(tDK), iKK, true);
        mma64<0, 1>(tbase + cDV, desc(tSBE), desc(tDV), iKM, true);
        mma64<0, 0>(tbase + cDS2, desc(tV), desc(tDV), iKK, true);
      }
    }
    if (!fin) mma_wait();
  }
  // window part of dv, fetched while the last products run
  float wv[16];
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 x = keep[i] ? *reinterpret_cast<const float2*>(w.dvacc + ((size_t)(t0 + c0 + r0 + 8 * i - shift) * H + h) * 64 + 32 * half + 8 * j + 2 * tq)
                               : make_float2(0.f, 0.f);
      wv[4 * j + 2 * i] = x.x;
      wv[4 * j + 2 * i + 1] = x.y;
    }
  mma_wait();
  // ---- epilogue --------------------------------------------------------------------------------------------------------
  {
    float v[16];
    frag_ld(tl + cDV, v);
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] += wv[k];
    frag_to_tile(at(b3, fo0), at(b3, fo1), v);
    frag_ld(tl + cDK, v);
    frag_to_tile(at(b2, fo0), at(b2, fo1), v);
    frag_ld_nowait(tl + cDS, v);
    frag_ld_nowait(tl + cDS2, wv);
    tmem_ld_wait();
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = b[k] * v[k] + ey[k] * wv[k];
    frag_to_tile(at(b1, fo0), at(b1, fo1), v);
#pragma unroll
    for (int jp = 0; jp < 2; ++jp)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = 4 * (2 * jp + (q >> 1)) + 2 * (q & 1), i = q & 1;
        const float2 sv = pair_f32(s[jp][q]);
        ga[e] = keep[i] ? ga[e] - sv.x * v[e] : 0.f;
        ga[e + 1] = keep[i] ? ga[e + 1] - sv.y * v[e + 1] : 0.f;
      }
  }
  // reverse running sum over the rows: inside the blocks of eight rows over the lanes, then the later block, then the later
  // quarters and the carry
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      float lo = ga[4 * j + e], hi = ga[4 * j + 2 + e];
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        const float l2 = __shfl_down_sync(0xffffffffu, lo, 4 * o), h2 = __shfl_down_sync(0xffffffffu, hi, 4 * o);
        if (gq + o < 8) { lo += l2; hi += h2; }
      }
      lo += __shfl_sync(0xffffffffu, hi, tq);
      ga[4 * j + e] = lo;
      ga[4 * j + 2 + e] = hi;
      if (gq == 0) tot[quarter * 64 + 32 * half + 8 * j + 2 * tq + e] = lo;
    }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int m = 32 * half + 8 * j + 2 * tq + e;
      float add = part[8 * 64 + m];
#pragma unroll
      for (int w8 = 0; w8 < 8; ++w8) add += part[w8 * 64 + m];
#pragma unroll
      for (int q = 1; q < 4; ++q) add += q > quarter ? tot[q * 64 + m] : 0.f;
      ga[4 * j + e] += add;
      ga[4 * j + 2 + e] += add;
    }
  frag_to_tile(at(tQ, fo0), at(tQ, fo1), ga);
  auto rows_out = [&](int t, void* base, int64_t pitch, int col, int ncol) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = lr + 32 * u, p = c0 + r;
      if (p >= shift && p < len && 8 * lc < ncol)
        *reinterpret_cast<uint4*>((bf16*)base + (int64_t)(t0 + p - shift) * pitch + col + 8 * lc) =
            *reinterpret_cast<const uint4*>(tile(t) + loff + 4096 * u);
    }
  };
  rows_out(b1, d.ds, rm, h * M, M);
  rows_out(b2, d.dk_gsa, rp, h * 64, 64);
  rows_out(b3, d.dv, rp, h * 64, 64);
  __syncthreads();
  rows_out(tQ, d.dg, rm, h * M, M);
  if (failed) atomicExch(err, 1);
}

int bwd_cols64_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  const void* fn = d->HQ == d->H ? (const void*)nha_bwd_cols64_kernel<true> : (const void*)nha_bwd_cols64_kernel<false>;
  cudaError_t e = set_max_smem(fn, cl64::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  ColsMaps maps;
  memset(&maps, 0, sizeof(maps));
  maps.use = d->M == 64 && make_map_rows_heads(&maps.qg, d->q_gsa, d->Ttot, d->HQ, 64) && make_map_rows_heads(&maps.kg, d->k_gsa, d->Ttot, d->H, 64) &&
             make_map_rows_heads(&maps.v, d->v, d->Ttot, d->H, 64) && make_map_rows_heads(&maps.g, d->g, d->Ttot, d->H, 64) &&
             make_map_rows_heads(&maps.s, d->s, d->Ttot, d->H, 64) && make_map_rows_heads(&maps.dout, d->d_o, d->Ttot, d->HQ, 64) &&
             make_map_rows_heads(&maps.za, w.dza, d->Ttot, d->HQ, 64) && make_map_rows_heads(&maps.pa, w.paq, d->Ttot, d->HQ, 64);
  const dim3 grid((unsigned)(nha_chunk_count_bound(d->Ttot, d->N) * d->H));
  const unsigned ahead = (unsigned)sm_count();
  if (d->HQ == d->H) launch_after(nha_bwd_cols64_kernel<true>, grid, kThreads, cl64::total, cs, *d, w, err, maps, ahead);
  else launch_after(nha_bwd_cols64_kernel<false>, grid, kThreads, cl64::total, cs, *d, w, err, maps, ahead);
  return check_launch();
}

}  // namespace nha
