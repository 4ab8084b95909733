// Backward of the chunked NHA operator, query-row side, for head dim 64: 64-row products with every lane at work
// (nha_frag64.cuh).  What it computes and stores is in nha_chunk_bwd_umma.cu, whose rows pass it replaces at this head dim.
//
// One CTA = one (chunk, kv head), two CTAs per SM (13 operand tiles, 256 tensor-memory columns).  It walks the query heads of
// the group; per head the rounds of products, each handed to the tensor core behind one block barrier, are
//     x  = G - Gend / 2                                              (first head only)
//     A  = q k'^T,  Av = do v'^T,  QH = q Hk,  Y = do Hv^T
//     X  = tril(A) SB,  X2 = tril(Av) SB                              -> p, dz, gate terms of the slots
//     E  = (scale dz a) SB^T,  LK = q^T (scale dz e^G),  LV = (p e^G)^T do   (the chunk's own state-gradient terms)
//     dq_gsa = (scale dz e^G) Hk^T + tril(E) k',  S, dP of the first window tile
//     then one round per 64 window keys: dq_swa += dz_win k_swa together with S, dP of the next tile.
// Gate terms are summed over the heads in registers (one writer per element: repeatable bits for any group size).
// Up to 64 slots (a multiple of 16; missing columns are zeros and masked).
//
// What bounds it: the chain of rounds of a CTA (HBM at 40 % of its rate).  Measured against the version with one row per lane,
// the gate scan in shared memory and eleven rounds instead of seven: B16 T2048 H16 W64 627 -> 421 us; 32768 packed tokens,
// windows 32-512, 740 -> 500 us; 16 query heads on 4, 4 x 2000 tokens, W 64, 164 -> 108 us (two heads to a tile before).
// One head a kv head as a variant of its own 398 -> 388 us (first shape), sums over the heads as reductions in memory 112 -> 102 us
// (last shape).
//
// Replaces, with the other backward kernels, ChunkNativeHybridAttentionFunction.backward (nha_fla/ops/nha/chunk.py:491-564).
#include "nha_bwd_common.cuh"
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

namespace rw64 {
constexpr int tQ = 0, tQS = 1, tDO = 2, tK = 3, tV = 4, tHk = 5, tHv = 6, tSB = 7, bufA = 8, bufB = 9, tW0 = 10, tWV0 = 11, tX = 12, kTiles = 13;
constexpr int tPA = tV, tPG = tHv, tE = tQ;                   // operands written over tiles that have been read
constexpr int tW1 = tV, tWV1 = tX, tOut = tHv;                // second window buffers; staging of the output rows
constexpr int oER = kTiles * kTile;                           // fp32 [64] exp(R)
constexpr int oRow = oER + 256;                               // fp32 [4][64] delta, -Lj, -lse_gsa (log2 units), d_lse_gsa
constexpr int oBar = oRow + 4 * 64 * 4;
constexpr int total = oBar + 64 + 1024;
constexpr int cA = 0, cAv = 64, cQH = 128, cY = 192, kTmemCols = 256;
constexpr int cLK = cAv, cLV = cY, cDQ = cQH, cS = cA, cDP = cAv, cDQS = cY;
static_assert(total <= 113 * 1024, "two CTAs per SM");
}  // namespace rw64

// ONE: one query head per kv head (no loop over heads, nothing added up in memory)
template <bool ONE>
__global__ void __launch_bounds__(kThreads, 2) nha_bwd_rows64_kernel(const nha_chunk_desc d, const BwdWs w, int* __restrict__ err) {
  grid_dep_wait();
  grid_dep_launch();
  using namespace rw64;
  const int H = d.H, HQ = d.HQ, M = d.M, NG = ONE ? 1 : HQ / H;
  const int cg = blockIdx.x / H, h = blockIdx.x - cg * H;
  const ChunkRec rc = chunk_rec(d, cg);
  if (rc.n < 0) return;
  if (!chunk_gate(w, cg, h, H)) return;
  const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
  const int wl = seq_window(d, rc.n), shift = seq_shift(d, rc.n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* ER = (float*)(sm + oER);
  float* rowv = (float*)(sm + oRow);
  uint64_t* mbar = (uint64_t*)(sm + oBar);
  uint32_t* tslot = (uint32_t*)(mbar + 1);
  auto tile = [&](int i) { return sm + i * kTile; };

  // ---- loads: gates and write weights first, everything the first rounds need behind them ----------------------------------
  const int lr = tid >> 3, lc = tid & 7;
  const uint32_t loff = sw_off(lr, lc);
  const int64_t rq = (int64_t)HQ * 64, rp = (int64_t)H * 64, rm = (int64_t)H * M;
  auto load_tokens = [&](int t, const void* base, int64_t pitch, int col, int row, int lo, int hi, bool col_ok) {
    const bf16* p = (const bf16*)base + (int64_t)t0 * pitch + col + 8 * lc;
    const bool ok0 = col_ok && row + lr >= lo && row + lr < hi, ok1 = col_ok && row + lr + 32 >= lo && row + lr + 32 < hi;
    tile_in(tile(t), loff, p + (ok0 ? row + lr : 0) * pitch, ok0, p + (ok1 ? row + lr + 32 : 0) * pitch, ok1);
  };
  const bool mcol = 8 * lc < M;
  load_tokens(bufB, d.g, rm, h * M, c0 - shift, 0, len - shift, mcol);
  load_tokens(tSB, d.s, rm, h * M, c0 - shift, 0, len - shift, mcol);
  cp_commit();
  const int jt_lo = wl < 0 ? 0 : max(0, c0 - wl) / kChunk;
  const int ntile = ci - jt_lo + 1;
  auto load_window = [&](int i) {                               // window tile i (oldest first) into its set of buffers
    load_tokens(i & 1 ? tW1 : tW0, d.k_swa, rp, h * 64, (jt_lo + i) * kChunk, 0, len, true);
    load_tokens(i & 1 ? tWV1 : tWV0, d.v, rp, h * 64, (jt_lo + i) * kChunk, 0, len, true);
  };
  auto load_head = [&](int hq) {                                // tiles that a head leaves overwritten
    load_tokens(tQ, d.q_gsa, rq, hq * 64, c0, 0, len, true);
    load_tokens(tDO, d.d_o, rq, hq * 64, c0, 0, len, true);
    load_tokens(tV, d.v, rp, h * 64, c0 - shift, 0, len - shift, true);
    const bf16* hv = (const bf16*)d.hv_chunks + ((size_t)cg * H + h) * M * 64;      // [M][64]
    const bool v0 = lr < M, v1 = lr + 32 < M;
    tile_in(tile(tHv), loff, hv + (v0 ? lr * 64 + 8 * lc : 0), v0, hv + (v1 ? (lr + 32) * 64 + 8 * lc : 0), v1);
    load_tokens(tQS, d.q_swa, rq, hq * 64, c0, 0, len, true);
    load_window(0);
    cp_commit();
  };
  load_tokens(tK, d.k_gsa, rp, h * 64, c0 - shift, 0, len - shift, true);
  {
    const bf16* hk = (const bf16*)d.hk_chunks + ((size_t)cg * H + h) * 64 * M;      // [64][M]
    const int o0 = lr * M + 8 * lc, o1 = o0 + 32 * M;
    tile_in(tile(tHk), loff, hk + (mcol ? o0 : 0), mcol, hk + (mcol ? o1 : 0), mcol);
  }
  // row statistics of a head: delta = <do, o> by four threads per row, the joint log-sum-exp by one (requested first, formed later)
  uint4 o0, o1, g0, g1;
  float lsw, lgs, dl;
  auto row_request = [&](int hq) {
    const int r = tid >> 2, part = tid & 3, pos = c0 + r;
    o0 = o1 = g0 = g1 = make_uint4(0u, 0u, 0u, 0u);
    lsw = lgs = dl = 0.f;
    if (pos < len) {
      const size_t at = (size_t)(t0 + pos) * HQ + hq;
      const uint4* o = reinterpret_cast<const uint4*>((const bf16*)d.o + at * 64 + 16 * part);
      const uint4* g = reinterpret_cast<const uint4*>((const bf16*)d.d_o + at * 64 + 16 * part);
      o0 = __ldg(o); o1 = __ldg(o + 1); g0 = __ldg(g); g1 = __ldg(g + 1);
      if (part == 0) {
        lsw = d.lse_swa[at];
        lgs = d.lse_gsa[at];
        dl = d.d_lse_gsa ? d.d_lse_gsa[at] : 0.f;
      }
    }
  };
  row_request(h * NG);
  load_head(h * NG);
  auto row_stats = [&](int hq) {
    const int r = tid >> 2, part = tid & 3, pos = c0 + r;
    float del = 0.f, x[8], y[8];
    unpack8(o0, x); unpack8(g0, y);
#pragma unroll
    for (int e = 0; e < 8; ++e) del += x[e] * y[e];
    unpack8(o1, x); unpack8(g1, y);
#pragma unroll
    for (int e = 0; e < 8; ++e) del += x[e] * y[e];
    del += __shfl_xor_sync(0xffffffffu, del, 1);
    del += __shfl_xor_sync(0xffffffffu, del, 2);
    if (part == 0) {
      const float mx = fmaxf(lsw, lgs), lj = mx + __logf(__expf(lsw - mx) + __expf(lgs - mx));
      rowv[r] = del;
      rowv[64 + r] = -lj * kLog2e;
      rowv[128 + r] = -lgs * kLog2e;
      rowv[192 + r] = dl;
      if (pos < len) {
        w.delta[(size_t)(t0 + pos) * HQ + hq] = del;
        w.lj[(size_t)(t0 + pos) * HQ + hq] = lj;
      }
    }
  };
  fill_half_signs(tile(bufA), tid);
  if (tid == 0) {
    mbar_init(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(tslot, kTmemCols);
  cp_wait_but_one();
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  const uint32_t tl = tbase + ((uint32_t)(quarter * 32) << 16) + 32 * half;       // this warp's columns of an accumulator at +0
  uint32_t phase = 0;
  bool failed = false;
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

  // ---- x, then a and s' .* b ------------------------------------------------------------------------------------------
  if (tid == 0) mma64<0, 1>(tbase + cA, desc(bufA), desc(bufB), iKM, false);
  row_stats(h * NG);
  mma_wait();
  const uint32_t fo0 = frag_off(quarter, half, lane, 0), fo1 = frag_off(quarter, half, lane, 1);
  const int r0 = 16 * quarter + gq;                            // this lane's rows: r0 and r0 + 8
  const int pos0 = c0 + r0;
  float a[16];
  {
    frag_ld(tl + cA, a);
    const bool last = quarter == 3 && gq == 7;                 // row 63: x = R = Gend / 2, a = exp(R)
    if (last) {
      float* ge = w.gend + ((size_t)cg * H + h) * M;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int m = 32 * half + 8 * j + 2 * tq;
        if (m < M) *reinterpret_cast<float2*>(ge + m) = make_float2(2.f * a[4 * j + 2], 2.f * a[4 * j + 3]);
      }
    }
    uint32_t s[2][4];
    ldm4(at(tSB, fo0), s[0]);
    ldm4(at(tSB, fo1), s[1]);
#pragma unroll
    for (int jp = 0; jp < 2; ++jp)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = 4 * (2 * jp + (q >> 1)) + 2 * (q & 1);
        const float2 sv = pair_f32(s[jp][q]);
        s[jp][q] = pair_bf16(sv.x * exp2f(-a[e] * kLog2e), sv.y * exp2f(-a[e + 1] * kLog2e));
        a[e] = exp2f(a[e] * kLog2e);
        a[e + 1] = exp2f(a[e + 1] * kLog2e);
      }
    stm4(at(tSB, fo0), s[0][0], s[0][1], s[0][2], s[0][3]);
    stm4(at(tSB, fo1), s[1][0], s[1][1], s[1][2], s[1][3]);
    if (last) {
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(ER + 32 * half + 8 * j + 2 * tq) = make_float2(a[4 * j + 2], a[4 * j + 3]);
    }
  }
  const float sc2 = d.scale * kLog2e;
  // visible keys of a row: klo <= key <= pos, tested as (unsigned)(key - klo) <= kspan; a row past the end sees nothing
  int klo[2];
  unsigned kspan[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int pos = pos0 + 8 * i;
    klo[i] = pos < len ? (wl < 0 ? 0 : max(0, pos - wl)) : (1 << 30);
    kspan[i] = pos < len ? (unsigned)(pos - klo[i]) : 0u;
  }
  // tril of an accumulator -> bf16 tile (columns i <= row)
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
  // whole rows of a bf16 tile to a [tokens][HQ][cols] tensor
  auto rows_out = [&](int t, bf16* base, int64_t pitch, int ncol) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = lr + 32 * u;
      if (c0 + r < len && 8 * lc < ncol)
        *reinterpret_cast<uint4*>(base + (int64_t)(t0 + c0 + r) * pitch + 8 * lc) = *reinterpret_cast<const uint4*>(tile(t) + loff + 4096 * u);
    }
  };
  float ga[16];                                                // gate terms ok dz + p dp, summed over the heads
#pragma unroll
  for (int k = 0; k < 16; ++k) ga[k] = 0.f;

  for (int ht = 0; ht < NG; ++ht) {
    const int hq = h * NG + ht;
    if (!ONE && ht > 0) {
      load_head(hq);
      row_request(hq);
      row_stats(hq);
    }
    cp_wait_all();
    hand_over();
    if (tid == 0) {
      mma64<0, 0>(tbase + cA, desc(tQ), desc(tK), iKK, false);
      mma64<0, 0>(tbase + cAv, desc(tDO), desc(tV), iKK, false);
      mma64<0, 1>(tbase + cQH, desc(tQ), desc(tHk), iKM, false);
      mma64<0, 0>(tbase + cY, desc(tDO), desc(tHv), iKK, false);
    }
    mma_wait();
    tril_to(cA, bufA);
    tril_to(cAv, bufB);
    hand_over();
    if (tid == 0) {
      mma64<0, 1>(tbase + cA, desc(bufA), desc(tSB), iKM, false);
      mma64<0, 1>(tbase + cAv, desc(bufB), desc(tSB), iKM, false);
    }
    float delta[2], nLj[2], nLg[2], dls[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      delta[i] = rowv[r0 + 8 * i];
      nLj[i] = rowv[64 + r0 + 8 * i];
      nLg[i] = rowv[128 + r0 + 8 * i];
      dls[i] = rowv[192 + r0 + 8 * i];
    }
    mma_wait();
    // ---- slot part of dz (16 columns at a time), decayed bf16 operands, gate terms ---------------------------------------
#pragma unroll
    for (int jp = 0; jp < 2; ++jp) {
      float qh[8], xv[8], y0[8], x2[8];
      frag_ld8_nowait(tl + cQH + 16 * jp, qh);
      frag_ld8_nowait(tl + cA + 16 * jp, xv);
      frag_ld8_nowait(tl + cY + 16 * jp, y0);
      frag_ld8_nowait(tl + cAv + 16 * jp, x2);
      tmem_ld_wait();
      float pg[8];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const int m = 32 * half + 16 * jp + 8 * j;
        const float2 er2 = *reinterpret_cast<const float2*>(ER + m + 2 * tq);
        const bool mlive = m < M;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int k = 4 * j + e, i = e >> 1;
          const float er = (e & 1) ? er2.y : er2.x, aI = a[8 * jp + k];
          const float ok = sc2 * aI * (er * qh[k] + xv[k]);     // log2 units
          const float dps = aI * (er * y0[k] + x2[k]);
          float ps = 0.f, dz = 0.f;
          if (mlive && pos0 + 8 * i < len) {
            ps = exp2f(ok + nLj[i]);
            dz = ps * (dps - delta[i]) + dls[i] * exp2f(ok + nLg[i]);
          }
          ga[8 * jp + k] += ok * kLn2 * dz + ps * dps;
          xv[k] = d.scale * dz * aI;                            // scale dz a
          qh[k] = xv[k] * er;                                   // scale dz e^G
          y0[k] = ps * aI;                                      // p a
          pg[k] = y0[k] * er;                                   // p e^G
        }
      }
      const uint32_t fo = jp ? fo1 : fo0;
      frag8_to_tile(at(bufB, fo), qh);
      frag8_to_tile(at(bufA, fo), xv);
      frag8_to_tile(at(tPA, fo), y0);
      frag8_to_tile(at(tPG, fo), pg);
    }
    hand_over();
    if (tid == 0) {
      mma64<0, 0>(tbase + cA, desc(bufA), desc(tSB), iKK, false);       // E
      mma64<1, 1>(tbase + cLK, desc(tQ), desc(bufB), iMM, false);
      mma64<1, 1>(tbase + cLV, desc(tPG), desc(tDO), iMM, false);
    }
    // the two copies that the columns pass reads
    rows_out(bufA, w.dza + (size_t)hq * M, (int64_t)HQ * M, M);
    rows_out(tPA, w.paq + (size_t)hq * M, (int64_t)HQ * M, M);
    mma_wait();
    tril_to(cA, tE);
    {
      float v[16];
      frag_ld(tl + cLK, v);
      float* dk = w.dkc + ((size_t)cg * H + h) * 64 * M;        // [64][M]
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int m = 32 * half + 8 * j + 2 * tq;
          if (m < M) {
            float2* p = reinterpret_cast<float2*>(dk + (size_t)(r0 + 8 * i) * M + m);
            if (!ONE && ht > 0) red_add2(reinterpret_cast<float*>(p), v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
            else *p = make_float2(v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
          }
        }
      frag_ld(tl + cLV, v);
      float* dv = w.dvc + ((size_t)cg * H + h) * M * 64;        // [M][64]
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (r0 + 8 * i < M) {
            float2* p = reinterpret_cast<float2*>(dv + (r0 + 8 * i) * 64 + 32 * half + 8 * j + 2 * tq);
            if (!ONE && ht > 0) red_add2(reinterpret_cast<float*>(p), v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
            else *p = make_float2(v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
          }
    }
    hand_over();
    if (tid == 0) {
      mma64<0, 0>(tbase + cDQ, desc(bufB), desc(tHk), iKK, false);
      mma64<0, 1>(tbase + cDQ, desc(tE), desc(tK), iKM, true);
      mma64<0, 0>(tbase + cS, desc(tQS), desc(tW0), iKK, false);
      mma64<0, 0>(tbase + cDP, desc(tDO), desc(tWV0), iKK, false);
    }
    if (ntile > 1) load_window(1);                              // (p a, in its place until now, has been stored)
    cp_commit();
    mma_wait();
    {
      float v[16];
      frag_ld(tl + cDQ, v);
      frag_to_tile(at(tOut, fo0), at(tOut, fo1), v);            // p e^G has been read
    }
    // ---- window tiles: dz_win, dq_swa ----------------------------------------------------------------------------------
    for (int i = 0; i < ntile; ++i) {
      {
        float s[16], dp[16];
        frag_ld_nowait(tl + cS, s);
        frag_ld_nowait(tl + cDP, dp);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int key = (jt_lo + i) * kChunk + 32 * half + 8 * j + 2 * tq + (e & 1), x = e >> 1, k = 4 * j + e;
            s[k] = (unsigned)(key - klo[x]) <= kspan[x] ? exp2f(fmaf(s[k], sc2, nLj[x])) * (dp[k] - delta[x]) * d.scale : 0.f;
          }
        frag_to_tile(at(bufA, fo0), at(bufA, fo1), s);
      }
      cp_wait_all();
      hand_over();
      if (i == 0) rows_out(tOut, (bf16*)d.dq_gsa + hq * 64, rq, 64);
      if (tid == 0) {
        mma64<0, 1>(tbase + cDQS, desc(bufA), desc(i & 1 ? tW1 : tW0), iKM, i > 0);
        if (i + 1 < ntile) {
          mma64<0, 0>(tbase + cS, desc(tQS), desc(i & 1 ? tW0 : tW1), iKK, false);
          mma64<0, 0>(tbase + cDP, desc(tDO), desc(i & 1 ? tWV0 : tWV1), iKK, false);
        }
      }
      mma_wait();
      if (i + 2 < ntile) load_window(i + 2);                    // this tile's buffers are free again
      cp_commit();
    }
    {
      float v[16];
      frag_ld(tl + cDQS, v);
      frag_to_tile(at(bufA, fo0), at(bufA, fo1), v);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    rows_out(bufA, (bf16*)d.dq_swa + hq * 64, rq, 64);
    if (ht + 1 < NG) __syncthreads();                           // the next head writes the tiles
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (pos0 + 8 * i < len) {
      float* g = w.dga + ((size_t)(t0 + pos0 + 8 * i) * H + h) * M;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int m = 32 * half + 8 * j + 2 * tq;
        if (m < M) *reinterpret_cast<float2*>(g + m) = make_float2(ga[4 * j + 2 * i], ga[4 * j + 2 * i + 1]);
      }
    }
  if (failed) atomicExch(err, 1);
  cp_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
}

bool bwd64_supported(const nha_chunk_desc* d) { return d->K == 64 && d->V == 64 && d->M <= 64 && d->scale > 0.f; }

int bwd_rows64_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  const bool one = d->HQ == d->H;
  const auto kernel = one ? nha_bwd_rows64_kernel<true> : nha_bwd_rows64_kernel<false>;
  cudaError_t e = set_max_smem((const void*)kernel, rw64::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  launch_after(kernel, dim3((unsigned)(nha_chunk_count_bound(d->Ttot, d->N) * d->H)), kThreads, rw64::total, cs, *d, w, err);
  return check_launch();
}

}  // namespace nha
