// Backward of the chunked NHA operator, query-row side, for head dim 128 and 64 slots: 64-row products with every lane at work
// (nha_frag64.cuh), two CTAs per SM.  What it computes and stores is in nha_chunk_bwd_umma.cu.
//
// One CTA = one (chunk, kv head).  It walks the query heads of the group; the rounds of products per head are
//     x  = G - Gend / 2                                              (first head only)
//     A  = q k'^T,  Av = do v'^T,  Y = do Hv^T
//     X  = tril(A) SB,  X2 = tril(Av) SB,  QH = q Hk                   -> p, dz, gate terms of the slots
//     E  = (scale dz a) SB^T,  LK (rows 0-63) = q^T (scale dz e^G),  LV = (p e^G)^T do
//     dq_gsa = (scale dz e^G) Hk^T + tril(E) k',  LK (rows 64-127)
//     S, dP of the first window tile, then one round per 64 window keys: dq_swa += dz_win k_swa with S, dP of the next tile.
// Operands take 13 tiles of 8 KB and 256 tensor-memory columns, so that two CTAs share an SM: k' / v' / Hv / Hk / window tiles
// follow one another in three places, each requested as soon as the last product that reads its place is done and hidden behind
// the element-wise work of a round:
//     place    round 1   rounds 2-4     window
//     S0       k'        k'             keys of odd tiles
//     S1       v'        p a, p e^G     keys of even tiles
//     S2       Hv        Hk             values
//     Q        q         q              q_swa
// Gate terms are summed over the heads in registers, the local state-gradient terms in memory by the thread that wrote them: one
// writer per element, repeatable bits for any group size.
//
// What bounds it: the chain of rounds of a CTA (HBM at 22 % of its rate, issue slots at 27 %).  Measured, 2 x 1999 tokens, 32 heads
// on 8, window 127: 270 us with two heads to a 128-row tile and one CTA per SM, 204 us so, 187 us once the sums over the heads
// are reductions in memory instead of loads, additions and stores, 158 us with products issued by an elected lane, addresses formed where they are
// used (no spills: 128 registers a thread are all that two CTAs leave) and the weights of the slots two at a time.
//
// Replaces, with the other backward kernels, ChunkNativeHybridAttentionFunction.backward (nha_fla/ops/nha/chunk.py:491-564).
#include "nha_bwd_common.cuh"
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

namespace rw128 {
constexpr int D = 128, M = 64;
constexpr int tQ = 0, tDO = 2, tS0 = 4, tS1 = 6, tS2 = 8, tSB = 10, bufA = 11, bufB = 12, kTiles = 13;
constexpr int tPA = tS1, tPG = tS1 + 1;
constexpr int oER = kTiles * kTile;                           // fp32 [64] exp(R)
constexpr int oRow = oER + 256;                               // fp32 [4][64] delta, -Lj, -lse_gsa (log2 units), d_lse_gsa
constexpr int oBar = oRow + 4 * 64 * 4;
constexpr int total = oBar + 64 + 1024;
constexpr int cA = 0, cAv = 64, cQH = 128, cY = 192, kTmemCols = 256;
constexpr int cLK0 = cAv, cLV = 128, cDQ = 128, cLK1 = cA, cS = cA, cDP = cAv, cDQS = 128;      // cLV, cDQ, cDQS: 128 columns
static_assert(total <= 113 * 1024, "two CTAs per SM");
}  // namespace rw128

__global__ void __launch_bounds__(kThreads, 2) nha_bwd_rows128_kernel(const nha_chunk_desc d, const BwdWs w, int* __restrict__ err) {
  grid_dep_wait();
  grid_dep_launch();
  using namespace rw128;
  const int H = d.H, HQ = d.HQ, NG = HQ / H;
  const int cg = blockIdx.x / H, h = blockIdx.x - cg * H;
  const ChunkRec rc = chunk_rec(d, cg);
  if (rc.n < 0) return;
  if (!chunk_gate(w, cg, h, H)) return;
  const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
  const int wl = seq_window(d, rc.n), shift = seq_shift(d, rc.n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;
  const bool issuer = uniform(threadIdx.x >> 5) == 0;          // the warp whose elected lane issues the products

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  float* ER = (float*)(sm + oER);
  float* rowv = (float*)(sm + oRow);
  uint64_t* mbar = (uint64_t*)(sm + oBar);
  uint32_t* tslot = (uint32_t*)(mbar + 1);
  auto tile = [&](int i) { return sm + i * kTile; };

  // ---- loads: gates and write weights first, everything the first round needs behind them ----------------------------------
  const int lr = tid >> 3, lc = tid & 7;
  const uint32_t loff = sw_off(lr, lc);
  const int64_t rq = (int64_t)HQ * D, rp = (int64_t)H * D, rm = (int64_t)H * M;
  // nt tiles of 64 columns each: rows row .. row + 63 of a [tokens][pitch] tensor from column col on, zeros outside [0, hi)
  auto load_tokens = [&](int t, int nt, const void* base, int64_t pitch, int col, int row, int hi) {
    const int lr = from_here(tid >> 3);
    const bf16* p = (const bf16*)base + (int64_t)t0 * pitch + col + 8 * lc;
    const bool ok0 = row + lr >= 0 && row + lr < hi, ok1 = row + lr + 32 >= 0 && row + lr + 32 < hi;
    const bf16 *p0 = p + (ok0 ? row + lr : 0) * pitch, *p1 = p + (ok1 ? row + lr + 32 : 0) * pitch;
    for (int k = 0; k < nt; ++k) tile_in(tile(t + k), loff, p0 + 64 * k, ok0, p1 + 64 * k, ok1);
  };
  load_tokens(bufB, 1, d.g, rm, h * M, c0 - shift, len - shift);
  load_tokens(tSB, 1, d.s, rm, h * M, c0 - shift, len - shift);
  cp_commit();
  const int jt_lo = wl < 0 ? 0 : max(0, c0 - wl) / kChunk;
  const int ntile = ci - jt_lo + 1;
  auto load_wk = [&](int i) {                                   // window tile i (oldest first)
    load_tokens(i & 1 ? tS0 : tS1, 2, d.k_swa, rp, h * D, (jt_lo + i) * kChunk, len);
  };
  auto load_wv = [&](int i) { load_tokens(tS2, 2, d.v, rp, h * D, (jt_lo + i) * kChunk, len); };
  auto load_q = [&](const void* base, int t, int hq) { load_tokens(t, 2, base, rq, hq * D, c0, len); };
  auto load_kp = [&]() { load_tokens(tS0, 2, d.k_gsa, rp, h * D, c0 - shift, len - shift); };
  auto load_vp = [&]() { load_tokens(tS1, 2, d.v, rp, h * D, c0 - shift, len - shift); };
  auto load_hk = [&]() {
    const int lr = from_here(tid >> 3);
    const bf16* hk = (const bf16*)d.hk_chunks + ((size_t)cg * H + h) * D * M;     // [D][M]
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const bf16* p = hk + (64 * k + lr) * M + 8 * lc;
      tile_in(tile(tS2 + k), loff, p, true, p + 32 * M, true);
    }
  };
  auto load_hv = [&]() {
    const int lr = from_here(tid >> 3);
    const bf16* hv = (const bf16*)d.hv_chunks + ((size_t)cg * H + h) * M * D;     // [M][D]
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const bf16* p = hv + lr * D + 64 * k + 8 * lc;
      tile_in(tile(tS2 + k), loff, p, true, p + 32 * D, true);
    }
  };
  // row statistics of a head: delta = <do, o> by four threads per row (o from memory, do from its tile), the joint log-sum-exp
  // by one of them
  uint4 oreg[4];
  float lsw, lgs, dl;
  auto row_request = [&](int hq) {
    const int r = from_here(tid >> 2), part = tid & 3, pos = c0 + r;
#pragma unroll
    for (int e = 0; e < 4; ++e) oreg[e] = make_uint4(0u, 0u, 0u, 0u);
    lsw = lgs = dl = 0.f;
    if (pos < len) {
      const size_t at = (size_t)(t0 + pos) * HQ + hq;
      const uint4* o = reinterpret_cast<const uint4*>((const bf16*)d.o + at * D + 32 * part);
#pragma unroll
      for (int e = 0; e < 4; ++e) oreg[e] = __ldg(o + e);
      if (part == 0) {
        lsw = d.lse_swa[at];
        lgs = d.lse_gsa[at];
        dl = d.d_lse_gsa ? d.d_lse_gsa[at] : 0.f;
      }
    }
  };
  auto row_stats = [&](int hq) {
    const int r = from_here(tid >> 2), part = tid & 3, pos = c0 + r;
    float del = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float x[8], y[8];
      unpack8(oreg[e], x);
      unpack8(*reinterpret_cast<const uint4*>(tile(tDO + (part >> 1)) + sw_off(r, 4 * (part & 1) + e)), y);
#pragma unroll
      for (int k = 0; k < 8; ++k) del += x[k] * y[k];
    }
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
  load_q(d.q_gsa, tQ, h * NG);
  load_kp();
  load_q(d.d_o, tDO, h * NG);
  load_vp();
  load_hv();
  cp_commit();
  row_request(h * NG);
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
  // one round of products by the elected lane of warp 0, committed to the barrier of mma_wait(): f(descriptor of a tile, of an MN-major
  // operand of two 64-column tiles, tensor memory)
  auto round = [&](auto f) {
    if (issuer) {
      const uint32_t sb = uniform(sbase), tb = uniform(tbase);
      if (elect_one()) {
        f([&](int t) { return make_desc(sb + t * kTile); }, [&](int t) { return make_desc_lbo(sb + t * kTile, kTile); }, tb);
        commit(mbar);
      }
    }
  };
  const uint32_t iKK = idesc64(0, 0), iKM = idesc64(0, 1), iMM = idesc64(1, 1);
  const uint32_t iKK2 = idesc64(0, 0, 128), iKM2 = idesc64(0, 1, 128), iMM2 = idesc64(1, 1, 128);
  // a product over the head dim, both operands K-major
  auto mma_dd = [&](auto desc, uint32_t d, int x, int y) {
    mma64<0, 0>(d, desc(x), desc(y), iKK, false);
    mma64<0, 0>(d, desc(x + 1), desc(y + 1), iKK, true);
  };

  // ---- x, then a and s' .* b ------------------------------------------------------------------------------------------
  round([&](auto desc, auto desc2, uint32_t tb) { mma64<0, 1>(tb + cA, desc(bufA), desc(bufB), iKM, false); });
  mma_wait();
  const uint32_t fo0 = frag_off(quarter, half, lane, 0), fo1 = frag_off(quarter, half, lane, 1);
  const int r0 = 16 * quarter + gq;                            // this lane's rows: r0 and r0 + 8
  const int pos0 = c0 + r0;
  float a[16];
  {
    frag_ld(tl + cA, a);
    const bool last = quarter == 3 && gq == 7;                 // row 63: x = R = Gend / 2, a = exp(R)
    if (last) {
      float* ge = w.gend + ((size_t)cg * H + h) * M + 32 * half + 2 * tq;
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(ge + 8 * j) = make_float2(2.f * a[4 * j + 2], 2.f * a[4 * j + 3]);
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
  // the warp's own 16 rows x 32 columns of a tile to a [tokens][pitch] tensor (64 bytes of a row to a group of four lanes)
  auto block_out = [&](int t, bf16* base, int64_t pitch) {
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = from_here(r0) + 8 * u;
      if (c0 + r < len)
        *reinterpret_cast<uint4*>(base + (int64_t)(t0 + c0 + r) * pitch + 32 * half + 8 * tq) =
            *reinterpret_cast<const uint4*>(tile(t) + sw_off(r, 4 * half + tq));
    }
    __syncwarp();
  };
  // 64 x 128 accumulator to two column blocks of a tensor, staged in tile bufB
  auto acc_out = [&](int col, bf16* base, int64_t pitch) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      float v[16];
      frag_ld(tl + col + 64 * k, v);
      frag_to_tile(at(bufB, fo0), at(bufB, fo1), v);
      block_out(bufB, base + 64 * k, pitch);
    }
  };
  // fp32 accumulator rows r0, r0 + 8 (pitch ld) added to what the heads before left there
  auto acc_add = [&](int col, float* base, int ld, bool add) {
    float v[16];
    frag_ld(tl + col, v);
    const int r = from_here(r0);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2* p = reinterpret_cast<float2*>(base + (size_t)(r + 8 * i) * ld + 32 * half + 8 * j + 2 * tq);
        if (add) red_add2(reinterpret_cast<float*>(p), v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
        else *p = make_float2(v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
      }
  };
  auto dkc = [&]() { return w.dkc + ((size_t)from_here(cg) * H + h) * D * M; };     // [D][M]
  auto dvc = [&]() { return w.dvc + ((size_t)from_here(cg) * H + h) * M * D; };     // [M][D]
  float ga[16];                                                // gate terms ok dz + p dp, summed over the heads
#pragma unroll
  for (int k = 0; k < 16; ++k) ga[k] = 0.f;

  for (int ht = 0; ht < NG; ++ht) {
    const int hq = h * NG + ht;
    cp_wait_all();
    hand_over();
    round([&](auto desc, auto desc2, uint32_t tb) {
      mma_dd(desc, tb + cA, tQ, tS0);
      mma_dd(desc, tb + cAv, tDO, tS1);
      mma_dd(desc, tb + cY, tDO, tS2);
    });
    row_stats(hq);
    mma_wait();
    load_hk();
    cp_commit();
    tril_to(cA, bufA);
    tril_to(cAv, bufB);
    cp_wait_all();
    hand_over();
    round([&](auto desc, auto desc2, uint32_t tb) {
      mma64<0, 1>(tb + cA, desc(bufA), desc(tSB), iKM, false);
      mma64<0, 1>(tb + cAv, desc(bufB), desc(tSB), iKM, false);
      mma64<0, 1>(tb + cQH, desc(tQ), desc(tS2), iKM, false);
      mma64<0, 1>(tb + cQH, desc(tQ + 1), desc(tS2 + 1), iKM, true);
    });
    float delta[2], nLj[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      delta[i] = rowv[r0 + 8 * i];
      nLj[i] = pos0 + 8 * i < len ? rowv[64 + r0 + 8 * i] : -INFINITY;   // a row past the end has no weights
    }
    const uint64_t sc22 = pack2(sc2, sc2), scale2 = pack2(d.scale, d.scale);
    mma_wait();
    // ---- slot part of dz, decayed bf16 operands, gate terms: eight columns at a time (more do not fit the registers), two by two -----
#pragma unroll
    for (int jp = 0; jp < 2; ++jp) {
      uint32_t za[4], zg[4], pa[4], pg[4];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float qh[4], xv[4], y0[4], x2[4];
        frag_ld4_nowait(tl + cQH + 16 * jp + 8 * j, qh);
        frag_ld4_nowait(tl + cA + 16 * jp + 8 * j, xv);
        frag_ld4_nowait(tl + cY + 16 * jp + 8 * j, y0);
        frag_ld4_nowait(tl + cAv + 16 * jp + 8 * j, x2);
        tmem_ld_wait();
        const float2 erf = *reinterpret_cast<const float2*>(ER + 32 * half + 16 * jp + 8 * j + 2 * tq);
        const uint64_t er = pack2(erf.x, erf.y);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int k = 2 * i, K = 8 * jp + 4 * j + k, q = 2 * j + i;
          const uint64_t aI = pack2(a[K], a[K + 1]);
          const uint64_t ok = fmul2(aI, ffma2(er, pack2(qh[k], qh[k + 1]), pack2(xv[k], xv[k + 1])));
          const uint64_t dps = fmul2(aI, ffma2(er, pack2(y0[k], y0[k + 1]), pack2(x2[k], x2[k + 1])));
          float e0, e1;
          unpack2(ffma2(ok, sc22, pack2(nLj[i], nLj[i])), e0, e1);
          const uint64_t ps = pack2(exp2f(e0), exp2f(e1));
          uint64_t dz = fmul2(ps, fadd2(dps, pack2(-delta[i], -delta[i])));
          if (d.d_lse_gsa) {
            const float g = nLj[i] > -INFINITY ? rowv[128 + r0 + 8 * i] : -INFINITY, dl = rowv[192 + r0 + 8 * i];
            unpack2(ffma2(ok, sc22, pack2(g, g)), e0, e1);
            dz = ffma2(pack2(dl, dl), pack2(exp2f(e0), exp2f(e1)), dz);
          }
          const uint64_t zs = fmul2(dz, scale2);
          unpack2(ffma2(ps, dps, ffma2(ok, zs, pack2(ga[K], ga[K + 1]))), ga[K], ga[K + 1]);
          const uint64_t z2 = fmul2(zs, aI), p2 = fmul2(ps, aI);
          unpack2(z2, e0, e1);
          za[q] = pair_bf16(e0, e1);                            // scale dz a
          unpack2(fmul2(z2, er), e0, e1);
          zg[q] = pair_bf16(e0, e1);                            // scale dz e^G
          unpack2(p2, e0, e1);
          pa[q] = pair_bf16(e0, e1);                            // p a
          unpack2(fmul2(p2, er), e0, e1);
          pg[q] = pair_bf16(e0, e1);                            // p e^G
        }
      }
      const uint32_t fo = jp ? fo1 : fo0;
      stm4(at(bufB, fo), zg[0], zg[1], zg[2], zg[3]);
      stm4(at(bufA, fo), za[0], za[1], za[2], za[3]);
      stm4(at(tPA, fo), pa[0], pa[1], pa[2], pa[3]);
      stm4(at(tPG, fo), pg[0], pg[1], pg[2], pg[3]);
    }
    hand_over();
    round([&](auto desc, auto desc2, uint32_t tb) {
      mma64<0, 0>(tb + cA, desc(bufA), desc(tSB), iKK, false);       // E
      mma64<1, 1>(tb + cLK0, desc(tQ), desc(bufB), iMM, false);
      mma64<1, 1>(tb + cLV, desc(tPG), desc2(tDO), iMM2, false);
    });
    // the two copies that the columns pass reads
    block_out(bufA, w.dza + (size_t)hq * M, (int64_t)HQ * M);
    block_out(tPA, w.paq + (size_t)hq * M, (int64_t)HQ * M);
    mma_wait();
    tril_to(cA, bufA);                                          // (a warp writes the blocks that it has copied out itself)
    acc_add(cLK0, dkc(), M, ht > 0);
    acc_add(cLV, dvc(), D, ht > 0);
    acc_add(cLV + 64, dvc() + 64, D, ht > 0);
    hand_over();
    round([&](auto desc, auto desc2, uint32_t tb) {
      mma64<0, 0>(tb + cDQ, desc(bufB), desc(tS2), iKK2, false);
      mma64<0, 1>(tb + cDQ, desc(bufA), desc2(tS0), iKM2, true);
      mma64<1, 1>(tb + cLK1, desc(tQ + 1), desc(bufB), iMM, false);
    });
    load_wk(0);                                                 // p a and p e^G have been read
    mma_wait();
    load_q(d.q_swa, tQ, hq);
    load_wv(0);
    cp_commit();
    if (ntile > 1) load_wk(1);
    cp_commit();
    acc_out(cDQ, (bf16*)d.dq_gsa + hq * D, rq);
    acc_add(cLK1, dkc() + 64 * M, M, ht > 0);
    cp_wait_but_one();
    hand_over();
    round([&](auto desc, auto desc2, uint32_t tb) {
      mma_dd(desc, tb + cS, tQ, tS1);
      mma_dd(desc, tb + cDP, tDO, tS2);
    });
    mma_wait();
    // ---- window tiles: dz_win, dq_swa ----------------------------------------------------------------------------------
    const bool more = ht + 1 < NG;
    for (int i = 0; i < ntile; ++i) {
      const bool fin = i + 1 == ntile;
      if (!fin) {
        load_wv(i + 1);                                         // the values, q_swa and do of the last tile have been read
        cp_commit();
      } else if (more) {
        load_q(d.q_gsa, tQ, hq + 1);
        load_q(d.d_o, tDO, hq + 1);
        load_hv();
        if (i & 1) load_vp(); else load_kp();                   // the place that does not hold this tile's keys
      }
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
      if (!fin) cp_wait_all();
      hand_over();
      round([&](auto desc, auto desc2, uint32_t tb) {
        mma64<0, 1>(tb + cDQS, desc(bufA), desc2(i & 1 ? tS0 : tS1), iKM2, i > 0);
        if (!fin) {
          mma_dd(desc, tb + cS, tQ, i & 1 ? tS1 : tS0);
          mma_dd(desc, tb + cDP, tDO, tS2);
        }
      });
      mma_wait();
      if (i + 2 < ntile) load_wk(i + 2);                        // this tile's keys have been read
      if (fin && more) {
        if (i & 1) load_kp(); else load_vp();
        row_request(hq + 1);
      }
      cp_commit();
    }
    acc_out(cDQS, (bf16*)d.dq_swa + hq * D, rq);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (pos0 + 8 * i < len) {
      float* g = w.dga + ((size_t)(t0 + pos0 + 8 * i) * H + h) * M + 32 * half + 2 * tq;
#pragma unroll
      for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(g + 8 * j) = make_float2(ga[4 * j + 2 * i], ga[4 * j + 2 * i + 1]);
    }
  if (failed) atomicExch(err, 1);
  cp_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
}

int bwd_rows128_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  cudaError_t e = set_max_smem((const void*)nha_bwd_rows128_kernel, rw128::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  launch_after(nha_bwd_rows128_kernel, dim3((unsigned)(nha_chunk_count_bound(d->Ttot, d->N) * d->H)), kThreads, rw128::total, cs, *d, w, err);
  return check_launch();
}

}  // namespace nha
