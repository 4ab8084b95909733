// Output pass of the chunked NHA forward for head dim 64: 64-row products with every lane at work (nha_frag64.cuh).
//
// One CTA = one (chunk, query head), two CTAs per SM (13 operand tiles, 256 tensor-memory columns).  Rounds of products, each handed
// to the tensor core behind one block barrier:
//     x  = G - Gend / 2                                       (a = exp(x) in registers, s' .* b = s' exp(-x) into its tile)
//     A  = q k'^T,  QH = q Hk,  S = q_swa k_swa^T             (the newest 128 window keys)
//     X  = tril(A) (s' .* b)
//     O  = (p~ a e^R) Hv + P~ v_win,  Bv = (p~ a)(s' .* b)^T    with ok = scale a .* (e^R .* QH + X) and ONE softmax over slots and keys
//     O += tril(Bv) v'
//     then, for a window of more than 128 keys, one round per 128 older keys: O += P~ v_win of a step together with S of the
//     next one; the reference of the probabilities follows the running maximum (and O is rescaled when it moves), so that the
//     largest of them, rounded to bf16 for the product, is exactly 1: error of o against 64 bits at 16 heads, W 512, 2.17e-3, and
//     2.25e-3 with a reference that may lag by 2^8; no difference in time (32768 packed tokens, windows 32-512: 1.685 ms a step).
// What bounds it: the chain of rounds (two CTAs of eight warps per SM; about 13 k cycles per CTA, HBM at half its rate).
// It waits for the scan as its first instruction, although it needs only Hk and Hv from it: the early start of nha_fwd_pipe_kernel has not
// been tried here.
// Measured against the version with one row per lane and the gate scan in shared memory: B16 T2048 H16 W64 373 -> 230 us, with products issued
// by an elected lane (see elect_one()) 221-229 us;
// 32768 packed tokens, windows 32-512, 555 -> 328 us; 8 query heads on 2, 4 x 3000 tokens, W 512, 136 -> 90 us; 32 slots
// (general kernel before), 4 x 2000 tokens, 194 -> 33 us.
// Decay factorisation, flags for chunks that decay too fast for one reference per chunk, and the general kernel that takes
// those: as in nha_chunk_fwd_umma.cu.  Up to 64 slots (a multiple of 16; missing columns are zeros and masked).
//
// Replaces chunk_nha_fused_o_kernel (nha_fla/ops/nha/chunk_fused.py:117-283) and, for chunk_nha, the flash-attn varlen
// forward + fla chunk_gsa forward + log-sum-exp merge (nha_fla/ops/nha/chunk.py:423-470).
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

namespace fw64 {
constexpr int tQ = 0, tQS = 1, tK = 2, tV = 3, tHk = 4, tHv = 5, tSB = 6, tBuf = 7, tP1 = 8, tWK = 9, tWV = 11, kTiles = 13;
constexpr int tPA = tQ, tPG = tK, tP0 = tHk;                  // operands written over tiles that have been read
constexpr int tWK1 = tK, tWV1 = tHv;                          // second window buffers, once k', v', Hv and s' b are dead
constexpr int oER = kTiles * kTile;                           // fp32 [64] exp(R)
constexpr int oX = oER + 256;                                 // fp32 [4][2 halves][64 rows] row statistics swapped between the halves
constexpr int oBar = oX + 4 * 2 * 64 * 4;
constexpr int total = oBar + 64 + 1024;
constexpr int cA = 0, cO = 64, cS = 128, kTmemCols = 256;     // O takes QH's columns
constexpr float kDecayLimit = 140.0f;
static_assert(total <= 113 * 1024, "two CTAs per SM");
}  // namespace fw64

__global__ void __launch_bounds__(kThreads, 2) nha_fwd64_kernel(const nha_chunk_desc d, int* __restrict__ flags, int* __restrict__ err) {
  grid_dep_wait();
  grid_dep_launch();
  using namespace fw64;
  const int H = d.H, HQ = d.HQ, M = d.M, NG = HQ / H;
  const int cg = blockIdx.x / HQ, hq = blockIdx.x - cg * HQ, h = hq / NG;
  const ChunkRec rc = chunk_rec(d, cg);
  if (rc.n < 0) return;
  const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
  const int wl = seq_window(d, rc.n), shift = seq_shift(d, rc.n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;
  const bool issuer = uniform(threadIdx.x >> 5) == 0;          // the warp whose elected lane issues the products

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  float* ER = (float*)(sm + oER);
  float* xch = (float*)(sm + oX);
  uint64_t* mbar = (uint64_t*)(sm + oBar);
  uint32_t* tslot = (uint32_t*)(mbar + 1);
  auto tile = [&](int i) { return sm + i * kTile; };

  // ---- loads: gates and write weights first, everything else behind them ------------------------------------------------
  const int lr = tid >> 3, lc = tid & 7;
  const uint32_t loff = sw_off(lr, lc);
  const int64_t rq = (int64_t)HQ * 64, rp = (int64_t)H * 64, rm = (int64_t)H * M;
  auto load_tokens = [&](int t, const void* base, int64_t pitch, int col, int row, int lo, int hi, bool col_ok) {
    const bf16* p = (const bf16*)base + (int64_t)t0 * pitch + col + 8 * lc;
    const bool ok0 = col_ok && row + lr >= lo && row + lr < hi, ok1 = col_ok && row + lr + 32 >= lo && row + lr + 32 < hi;
    tile_in(tile(t), loff, p + (ok0 ? row + lr : 0) * pitch, ok0, p + (ok1 ? row + lr + 32 : 0) * pitch, ok1);
  };
  const bool mcol = 8 * lc < M;
  load_tokens(tBuf, d.g, rm, h * M, c0 - shift, 0, len - shift, mcol);
  load_tokens(tSB, d.s, rm, h * M, c0 - shift, 0, len - shift, mcol);
  cp_commit();
  load_tokens(tQ, d.q_gsa, rq, hq * 64, c0, 0, len, true);
  load_tokens(tK, d.k_gsa, rp, h * 64, c0 - shift, 0, len - shift, true);
  {
    const bf16* hk = (const bf16*)d.hk_chunks + ((size_t)cg * H + h) * 64 * M;      // [64][M]
    const bf16* hv = (const bf16*)d.hv_chunks + ((size_t)cg * H + h) * M * 64;      // [M][64]
    const int o0 = lr * M + 8 * lc, o1 = o0 + 32 * M;
    tile_in(tile(tHk), loff, hk + (mcol ? o0 : 0), mcol, hk + (mcol ? o1 : 0), mcol);
    const bool v0 = lr < M, v1 = lr + 32 < M;
    tile_in(tile(tHv), loff, hv + (v0 ? lr * 64 + 8 * lc : 0), v0, hv + (v1 ? (lr + 32) * 64 + 8 * lc : 0), v1);
  }
  load_tokens(tQS, d.q_swa, rq, hq * 64, c0, 0, len, true);
  // window steps of 128 keys, newest first: step p covers [kbase(p), kbase(p) + 128)
  const int jt_lo = wl < 0 ? 0 : max(0, c0 - wl) / kChunk;
  const int nsteps = (ci - jt_lo + 2) / 2;
  auto kbase = [&](int p) { return (ci + 1 - 2 * (p + 1)) * kChunk; };
  auto load_step = [&](int p, int set) {
    const int kb = kbase(p), tk = set ? tWK1 : tWK, tv = set ? tWV1 : tWV;
    load_tokens(tk, d.k_swa, rp, h * 64, kb, 0, len, true);
    load_tokens(tk + 1, d.k_swa, rp, h * 64, kb + 64, 0, len, true);
    load_tokens(tv, d.v, rp, h * 64, kb, 0, len, true);
    load_tokens(tv + 1, d.v, rp, h * 64, kb + 64, 0, len, true);
  };
  load_step(0, 0);
  load_tokens(tV, d.v, rp, h * 64, c0 - shift, 0, len - shift, true);
  cp_commit();
  fill_half_signs(tile(tP1), tid);
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
  const uint32_t iKK = idesc64(0, 0), iKM = idesc64(0, 1);
  const uint32_t sbase = smem_u32(sm);
  // one round of products: f(descriptor of a tile, tensor memory), committed to the barrier of mma_wait()
  auto round = [&](auto f) {
    if (issuer) {
      const uint32_t sb = uniform(sbase), tb = uniform(tbase);
      if (elect_one()) {
        f([&](int t) { return make_desc(sb + t * kTile); }, tb);
        commit(mbar);
      }
    }
  };

  // ---- x, then a and s' .* b ------------------------------------------------------------------------------------------
  round([&](auto desc, uint32_t tb) { mma64<0, 1>(tb + cA, desc(tP1), desc(tBuf), iKM, false); });
  mma_wait();
  const uint32_t fo0 = frag_off(quarter, half, lane, 0), fo1 = frag_off(quarter, half, lane, 1);
  auto at = [&](int t, uint32_t off) { return sbase + (uint32_t)(t * kTile) + off; };
  const int r0 = 16 * quarter + gq;                            // this lane's rows: r0 and r0 + 8
  float a[16];
  bool steep = false;
  {
    frag_ld(tl + cA, a);
    const bool last = quarter == 3 && gq == 7;                 // row 63: x = R, a = exp(R)
    if (last) {
#pragma unroll
      for (int j = 0; j < 4; ++j) steep = steep || fabsf(a[4 * j + 2]) > 0.5f * kDecayLimit || fabsf(a[4 * j + 3]) > 0.5f * kDecayLimit;
    }
    uint32_t s[2][4];
    ldm4(at(tSB, fo0), s[0]);
    ldm4(at(tSB, fo1), s[1]);
#pragma unroll
    for (int jp = 0; jp < 2; ++jp)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        // matrix q of the pair: rows gq (+ 8 for odd q), columns of block 2 jp + q / 2
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
  cp_wait_all();
  fence_async_smem();
  tc_fence_before();
  const int unsafe = __syncthreads_or(steep ? 1 : 0);
  tc_fence_after();
  if (tid == 0 && hq == h * NG) flags[(size_t)cg * H + h] = unsafe;
  if (unsafe) {                                                // the general kernel computes this chunk
    if (failed) atomicExch(err, 1);
    if (warp == 0) tmem_dealloc(tbase, kTmemCols);
    return;
  }
  // ---- A, QH, S of the newest step -------------------------------------------------------------------------------------
  auto issue_s = [&](auto desc, uint32_t tb, int set) { mma64<0, 0>(tb + cS, desc(tQS), desc(set ? tWK1 : tWK), idesc64(0, 0, 128), false); };
  auto issue_pv = [&](auto desc, uint32_t tb, int set) {
    const uint64_t v = desc(set ? tWV1 : tWV);
    mma64<0, 1>(tb + cO, desc(tP0), v, iKM, true);
    mma64<0, 1>(tb + cO, desc(tP1), v + 512, iKM, true);         // the second 64 keys: 8192 bytes on
  };
  round([&](auto desc, uint32_t tb) {
    mma64<0, 0>(tb + cA, desc(tQ), desc(tK), iKK, false);
    mma64<0, 1>(tb + cO, desc(tQ), desc(tHk), iKM, false);
    issue_s(desc, tb, 0);
  });
  mma_wait();
  // tril of the accumulator at cA -> bf16 tile (columns i <= row)
  auto tril_to = [&](int t) {
    float v[16];
    frag_ld(tl + cA, v);
    const int c = 32 * half + 2 * tq;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (c + 8 * j + (e & 1) > r0 + 8 * (e >> 1)) v[4 * j + e] = 0.f;
    frag_to_tile(at(t, fo0), at(t, fo1), v);
  };
  tril_to(tBuf);
  hand_over();
  round([&](auto desc, uint32_t tb) { mma64<0, 1>(tb + cA, desc(tBuf), desc(tSB), iKM, false); });
  // ---- the newest step's logits and maxima while X is formed: this warp's 64 keys, two blocks of 32 ----------------------------
  const float sc2 = d.scale * kLog2e;
  const int pos0 = c0 + r0;
  int klo[2];
  unsigned kspan[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    // visible keys of a row: klo <= key <= pos, tested as (unsigned)(key - klo) <= kspan; a row past the end sees nothing
    const int pos = pos0 + 8 * i;
    klo[i] = pos < len ? (wl < 0 ? 0 : max(0, pos - wl)) : (1 << 30);
    kspan[i] = pos < len ? (unsigned)(pos - klo[i]) : 0u;
  }
  float s[2][16];
  // window products of a step (unscaled; invisible keys -inf) and the maxima of this thread's part of its two rows.  They stay
  // unscaled up to the exponent, (x - max) times the scale, so that no logit is rounded before its maximum is taken off: error of
  // lse_swa against 64 bits at logits of up to 50, with the sum below, 8.1e-8 -> 6.9e-8
  auto step_logits = [&](int kb, float (&mx)[2]) {
    frag_ld_nowait(tl + cS + 32 * half, s[0]);                 // columns 64 half .. + 31
    frag_ld_nowait(tl + cS + 32 * half + 32, s[1]);
    tmem_ld_wait();
    mx[0] = mx[1] = -INFINITY;
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int key = kb + 64 * half + 32 * b + 8 * j + 2 * tq + (e & 1), i = e >> 1;
          float& v = s[b][4 * j + e];
          v = (unsigned)(key - klo[i]) <= kspan[i] ? v : -INFINITY;
          mx[i] = fmaxf(mx[i], v);
        }
  };
  // a statistic of the rows over the four lanes of a row and the two halves of its columns; slot: exchange buffer
  auto over_row = [&](float (&v)[2], int slot, auto op) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      v[i] = op(v[i], __shfl_xor_sync(0xffffffffu, v[i], 1));
      v[i] = op(v[i], __shfl_xor_sync(0xffffffffu, v[i], 2));
      if (tq == 0) xch[(slot * 2 + half) * 64 + r0 + 8 * i] = v[i];
    }
  };
  auto join = [&](float (&v)[2], int slot, auto op) {
#pragma unroll
    for (int i = 0; i < 2; ++i) v[i] = op(v[i], xch[(slot * 2 + (half ^ 1)) * 64 + r0 + 8 * i]);
  };
  auto maxf = [](float x, float y) { return fmaxf(x, y); };
  auto addf = [](float x, float y) { return x + y; };
  float mw[2], mg[2];
  step_logits(kbase(0), mw);
  over_row(mw, 0, maxf);
  mma_wait();
  // ---- slot logits ok (log2 units) -----------------------------------------------------------------------------------
  float ok[16];
  {
    float qh[16];
    frag_ld_nowait(tl + cO, qh);
    frag_ld_nowait(tl + cA, ok);
    tmem_ld_wait();
    mg[0] = mg[1] = -INFINITY;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 er = *reinterpret_cast<const float2*>(ER + 32 * half + 8 * j + 2 * tq);
      const bool live = 32 * half + 8 * j < M;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = 4 * j + e;
        ok[k] = live ? sc2 * a[k] * (((e & 1) ? er.y : er.x) * qh[k] + ok[k]) : -INFINITY;
        mg[e >> 1] = fmaxf(mg[e >> 1], ok[k]);
      }
    }
  }
  over_row(mg, 1, maxf);
  quarter_sync(quarter);
  join(mw, 0, maxf);
  join(mg, 1, maxf);
  float mref[2], cw[2], cgs[2], lg[2] = {0.f, 0.f}, ls[2] = {0.f, 0.f};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    mref[i] = fmaxf(mg[i], mw[i] * sc2);
    cgs[i] = exp2f(mg[i] - mref[i]);                           // slot entries:   p~ = 2^(ok - mg) cgs
    cw[i] = exp2f(mw[i] * sc2 - mref[i]);                      // window entries: p~ = 2^(sc2 (s - mw)) cw
  }
  // ---- operands p~ a e^R, p~ a and P~ of the newest step ---------------------------------------------------------------------
  {
    float pg[16];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 er = *reinterpret_cast<const float2*>(ER + 32 * half + 8 * j + 2 * tq);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = 4 * j + e, i = e >> 1;
        const float p = exp2f(ok[k] - mg[i]);
        lg[i] += p;
        ok[k] = p * cgs[i] * a[k];
        pg[k] = ok[k] * ((e & 1) ? er.y : er.x);
      }
    }
    frag_to_tile(at(tPG, fo0), at(tPG, fo1), pg);
    frag_to_tile(at(tPA, fo0), at(tPA, fo1), ok);
  }
  const uint32_t po[4] = {frag_off(quarter, 0, lane, 0), frag_off(quarter, 0, lane, 1), frag_off(quarter, 1, lane, 0),
                          frag_off(quarter, 1, lane, 1)};
  auto step_probs = [&]() {
#pragma unroll
    for (int b = 0; b < 2; ++b) {
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        const int i = (k >> 1) & 1;
        const float p = s[b][k] == -INFINITY ? 0.f : exp2f((s[b][k] - mw[i]) * sc2);     // a NaN stays one
        ls[i] += p;
        s[b][k] = p * cw[i];
      }
      const int t = half ? tP1 : tP0;
      frag_to_tile(at(t, po[2 * b]), at(t, po[2 * b + 1]), s[b]);
    }
  };
  step_probs();
  hand_over();
  round([&](auto desc, uint32_t tb) {
    mma64<0, 1>(tb + cO, desc(tPG), desc(tHv), iKM, false);
    mma64<0, 0>(tb + cA, desc(tPA), desc(tSB), iKK, false);
    issue_pv(desc, tb, 0);
  });
  mma_wait();
  tril_to(tBuf);
  hand_over();
  round([&](auto desc, uint32_t tb) { mma64<0, 1>(tb + cO, desc(tBuf), desc(tV), iKM, true); });
  mma_wait();
  // ---- older window steps ----------------------------------------------------------------------------------------------
  if (nsteps > 1) {
    load_step(1, 1);
    cp_commit();
    if (nsteps > 2) load_step(2, 0);
    cp_commit();
    cp_wait_but_one();
    hand_over();
    round([&](auto desc, uint32_t tb) { issue_s(desc, tb, 1); });
    mma_wait();
    for (int p = 1; p < nsteps; ++p) {
      float mx[2];
      step_logits(kbase(p), mx);
      over_row(mx, p & 1, maxf);
      quarter_sync(quarter);
      join(mx, p & 1, maxf);
      bool rescale = false;
      float f[2] = {1.f, 1.f};
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        if (mx[i] > mw[i]) {
          ls[i] *= exp2f((mw[i] - mx[i]) * sc2);
          mw[i] = mx[i];
          const float m2 = mw[i] * sc2;
          if (m2 > mref[i]) {
            f[i] = exp2f(mref[i] - m2);
            mref[i] = m2;
            rescale = true;
          }
          cw[i] = exp2f(m2 - mref[i]);
        }
      }
      if (__any_sync(0xffffffffu, rescale)) {                  // (every product issued on O has completed)
        float o[16];
        frag_ld(tl + cO, o);
#pragma unroll
        for (int k = 0; k < 16; ++k) o[k] *= f[(k >> 1) & 1];
        frag_st(tl + cO, o);
      }
      step_probs();
      cp_wait_all();
      hand_over();
      round([&](auto desc, uint32_t tb) {
        issue_pv(desc, tb, p & 1);
        if (p + 1 < nsteps) issue_s(desc, tb, (p + 1) & 1);
      });
      mma_wait();
      if (p + 2 < nsteps) load_step(p + 2, p & 1);             // this step's buffers are free again
      cp_commit();
    }
  }
  // ---- row sums, normalise, store ---------------------------------------------------------------------------------------
  over_row(lg, 2, addf);
  over_row(ls, 3, addf);
  quarter_sync(quarter);
  join(lg, 2, addf);
  join(ls, 3, addf);
  {
    float o[16], inv[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float l = lg[i] * exp2f(mg[i] - mref[i]) + ls[i] * exp2f(mw[i] * sc2 - mref[i]);
      inv[i] = l > 0.f ? 1.f / l : 0.f;
      const int pos = pos0 + 8 * i;
      if (tq == 0 && half == 0 && pos < len) {
        const size_t at_ = (size_t)(t0 + pos) * HQ + hq;
        // (the small product is rounded, the one inside the logarithm is fused into the sum)
        d.lse_gsa[at_] = __fmul_rn(mg[i], kLn2) + __logf(lg[i]);
        d.lse_swa[at_] = __fmul_rn(mw[i], d.scale) + __logf(ls[i]);
      }
    }
    frag_ld(tl + cO, o);
#pragma unroll
    for (int k = 0; k < 16; ++k) o[k] *= inv[(k >> 1) & 1];
    frag_to_tile(at(tBuf, fo0), at(tBuf, fo1), o);
  }
  quarter_sync(quarter);
  {
    // whole rows of 128 bytes: this warp takes eight of the quarter's sixteen
    const int c = lane & 7;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = 16 * quarter + 8 * half + 4 * u + (lane >> 3);
      if (c0 + r < len)
        *reinterpret_cast<uint4*>((bf16*)d.o + ((size_t)(t0 + c0 + r) * HQ + hq) * 64 + 8 * c) =
            *reinterpret_cast<const uint4*>(tile(tBuf) + sw_off(r, c));
    }
  }
  if (failed) atomicExch(err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
}

bool fwd64_supported(const nha_chunk_desc* d) {
  return d->K == 64 && d->V == 64 && d->M <= 64 && d->scale > 0.f && d->q_offset == 0;
}
int fwd64_launch(const nha_chunk_desc* d, int* flags, int* err, cudaStream_t cs) {
  cudaError_t e = set_max_smem((const void*)nha_fwd64_kernel, fw64::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  launch_after(nha_fwd64_kernel, dim3((unsigned)(nha_chunk_count_bound(d->Ttot, d->N) * d->HQ)), kThreads, fw64::total, cs, *d, flags, err);
  return check_launch();
}

}  // namespace nha
