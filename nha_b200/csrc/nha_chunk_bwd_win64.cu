// Backward of the window branch for head dim 64, both sides: dq_swa, dk_swa and dv, 64-row products with every lane at work
// (nha_frag64.cuh).  For every visible pair of a query row (joint log-sum-exp L, delta = <do, o>) and a key:
//     p = exp(scale q_swa k - L),  dz = scale p (do v - delta),  dq_swa += dz k,  dk_swa += dz q_swa,  dv += p do.
//
// One CTA = one (chunk, kv head): first its query rows, head by head, against the key tiles that they see (oldest first), then its
// keys against the query blocks that see them.  With one query head per kv head the pair of the chunk with itself, the last of the
// first part, serves both.  One round of products per pair, the next pair's S = q_swa k^T and dP = do v^T among them, its rows on
// their way.  dv is completed here: the slot part comes from memory (fp32, left by nha_bwd_slot64_kernel), and tokens that never
// enter the slot memory get their zeros in dk_gsa, ds and dg.
// FULL = false: the key side alone, the window part of dv to memory in fp32 (shapes whose slot branch the general kernels compute).
//
// Three CTAs per SM: four accumulators in the lane halves of 128 tensor-memory columns and eight operand tiles (67 KB).
// What bounds it: the chain of a round (product, weights, barrier) and the loads of the next pair; issue slots are 47 % busy, HBM at 30 %.
// B16 T2048 H16 W64: 205 us.  Before, the key side alone was a pass of its own, 153 us, and the query side a part of the slot branch's query-row
// pass.  Tiles by TMA with S and dP on a barrier of their own and packed arithmetic: the same time (905 -> 903 us of a whole training pass, 32768 packed
// tokens 1326 -> 1336): not kept.
//
// Replaces the third-party flash-attn varlen backward (call site nha_fla/ops/nha/chunk.py:333-344).
#include "nha_bwd_common.cuh"
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

namespace wn64 {
constexpr int tP = 6, tZ = 7, kTiles = 8;                      // three pairs of tiles in front: (q, do) or (k, v)
constexpr int oBar = kTiles * kTile;
constexpr int total = oBar + 64 + 1024;
// query side: S, dP, dq in s0, s1, s2; key side: S, dP in s1, s2, dv and dk in s0, s3
constexpr uint32_t s0 = 0, s1 = kOtherLanes, s2 = 64, s3 = 64 + kOtherLanes;
constexpr int kTmemCols = 128;
}  // namespace wn64

template <bool FULL>
__global__ void __launch_bounds__(kThreads, 3) nha_bwd_win64_kernel(const nha_chunk_desc d, const BwdWs w, int* __restrict__ err) {
  grid_dep_wait();
  grid_dep_launch();
  using namespace wn64;
  const int H = d.H, HQ = d.HQ, NG = HQ / H;
  const int cg = blockIdx.x / H, h = blockIdx.x - cg * H;
  const ChunkRec rc = chunk_rec(d, cg);
  if (rc.n < 0) return;
  const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
  const int wl = seq_window(d, rc.n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;
  const bool issuer = uniform(threadIdx.x >> 5) == 0;          // the warp whose elected lane issues the products

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  uint64_t* mbar = (uint64_t*)(sm + oBar);
  uint32_t* tslot = (uint32_t*)(mbar + 1);
  auto tile = [&](int i) { return sm + i * kTile; };
  const int lr = tid >> 3, lc = tid & 7;
  const uint32_t loff = sw_off(lr, lc);
  const int64_t rq = (int64_t)HQ * 64, rp = (int64_t)H * 64;
  auto load_tokens = [&](int t, const void* base, int64_t pitch, int col, int row) {
    const bf16* p = (const bf16*)base + (int64_t)t0 * pitch + col + 8 * lc;
    const bool ok0 = row + lr < len, ok1 = row + lr + 32 < len;
    tile_in(tile(t), loff, p + (ok0 ? row + lr : 0) * pitch, ok0, p + (ok1 ? row + lr + 32 : 0) * pitch, ok1);
  };
  auto load_queries = [&](int pair, int qi, int hq) {
    load_tokens(2 * pair, d.q_swa, rq, hq * 64, qi * kChunk);
    load_tokens(2 * pair + 1, d.d_o, rq, hq * 64, qi * kChunk);
  };
  auto load_keys = [&](int pair, int jt) {
    load_tokens(2 * pair, d.k_swa, rp, h * 64, jt * kChunk);
    load_tokens(2 * pair + 1, d.v, rp, h * 64, jt * kChunk);
  };
  const int r0 = 16 * quarter + gq, cbase = 32 * half + 2 * tq;  // this lane's rows r0, r0 + 8; columns cbase + 8 j, + 1
  float nL[2], nD[2];                                          // -log-sum-exp (log2 units) and delta of a query block's two rows
  auto load_rows = [&](int qi, int hq) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int pq = qi * kChunk + r0 + 8 * x;
      const size_t at = (size_t)(t0 + pq) * HQ + hq;
      nL[x] = pq < len ? -w.lj[at] * kLog2e : 0.f;
      nD[x] = pq < len ? w.delta[at] : 0.f;
    }
  };
  const bool shared_pair = FULL && NG == 1;
  // key tiles that a row of this chunk sees, query blocks that see a key of it
  const int jt_lo = wl < 0 ? 0 : max(0, c0 - wl) / kChunk, nt = ci - jt_lo + 1;
  const int nchunks = (len + kChunk - 1) / kChunk;
  const int qi_hi = wl < 0 ? nchunks - 1 : min(nchunks - 1, (int)(((int64_t)c0 + kChunk - 1 + wl) / kChunk));
  const int nblk = (qi_hi - ci + 1) * NG;
  // query side: q, do in pair 0, key tile i in pair 1 + i % 2.  Key side: k, v of this chunk where the first part left them (or in
  // pair 1), query block i in pair 0 (even) or the third one (odd).
  const int own = FULL ? 1 + ((nt - 1) & 1) : 1;
  auto block_pair = [&](int i) { return (i & 1) ? 3 - own : 0; };
  auto load_block = [&](int i) { load_queries(block_pair(i), ci + i / NG, h * NG + i % NG); };
  if (FULL) {
    load_queries(0, ci, h * NG);
    load_keys(1, jt_lo);
    cp_commit();
    if (nt > 1) load_keys(2, jt_lo + 1);
    else if (shared_pair && nblk > 1) load_block(1);
    cp_commit();
    load_rows(ci, h * NG);
  } else {
    load_keys(own, ci);
    load_block(0);
    cp_commit();
    if (nblk > 1) load_block(1);
    cp_commit();
    load_rows(ci, h * NG);
  }
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
  const uint32_t tl = tbase + ((uint32_t)(quarter * 32) << 16) + 32 * half;
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
  const uint32_t iKK = idesc64(0, 0), iKM = idesc64(0, 1), iMM = idesc64(1, 1);
  // one round of products by the elected lane of warp 0: `more(sb, tb)` and the two of a pair, S and dP, where s != dp
  auto round = [&](int qpair, int kpair, uint32_t s, uint32_t dp, auto more) {
    if (issuer) {
      const uint32_t sb = uniform(sbase), tb = uniform(tbase);
      if (elect_one()) {
        if (s != dp) {
          const uint64_t q = make_desc(sb + 2 * qpair * kTile), k = make_desc(sb + 2 * kpair * kTile);
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            mma_f16(tb + s, q + 2 * ks, k + 2 * ks, iKK, ks > 0);
            mma_f16(tb + dp, q + kTile / 16 + 2 * ks, k + kTile / 16 + 2 * ks, iKK, ks > 0);
          }
        }
        more(sb, tb);
        commit(mbar);
      }
    }
  };
  auto nothing = [](uint32_t, uint32_t) {};
  const uint32_t fo0 = frag_off(quarter, half, lane, 0), fo1 = frag_off(quarter, half, lane, 1);
  const float sc2 = d.scale * kLog2e;
  // p (where `want_p`) and dz of a pair into their tiles: query rows from position q0, keys from position k0
  auto weights = [&](uint32_t cs, uint32_t cd, int q0, int k0, bool want_p) {
    float s[16], dp[16];
    frag_ld_nowait(tl + cs, s);
    frag_ld_nowait(tl + cd, dp);
    tmem_ld_wait();
    // visible keys of a query row: klo <= key <= pq, tested as (unsigned)(key - klo) <= kspan; a row past the end sees nothing
    int off[2];
    unsigned kspan[2];
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int pq = q0 + r0 + 8 * x, klo = pq < len ? (wl < 0 ? 0 : max(0, pq - wl)) : (1 << 30);
      kspan[x] = pq < len ? (unsigned)(pq - klo) : 0u;
      off[x] = k0 + cbase - klo;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int k = 4 * j + e, x = e >> 1;
        const float p = (unsigned)(off[x] + 8 * j + (e & 1)) <= kspan[x] ? exp2f(fmaf(s[k], sc2, nL[x])) : 0.f;
        s[k] = p;
        dp[k] = p * (dp[k] - nD[x]) * d.scale;
      }
    if (want_p) frag_to_tile(at(tP, fo0), at(tP, fo1), s);
    frag_to_tile(at(tZ, fo0), at(tZ, fo1), dp);
  };
  // this warp's 16 x 32 block through its own part of a tile (no other warp writes or reads it): half rows of 64 bytes out
  const int wr = 16 * quarter + (lane >> 2), wc = 4 * half + (lane & 3);
  auto block_out = [&](int t, const float (&v)[16], bf16* base, int64_t pitch) {
    frag_to_tile(at(t, fo0), at(t, fo1), v);
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = wr + 8 * u;
      if (c0 + r < len) *reinterpret_cast<uint4*>(base + (int64_t)(t0 + c0 + r) * pitch + 8 * wc) = *reinterpret_cast<const uint4*>(tile(t) + sw_off(r, wc));
    }
    __syncwarp();
  };

  int first = 0;                                               // first query block of the key side that is still to do
  if (FULL) {
    for (int ht = 0; ht < NG; ++ht) {
      const int hq = h * NG + ht;
      if (ht > 0) {                                            // (every product that read these tiles has completed)
        load_queries(0, ci, hq);
        load_keys(1, jt_lo);
        cp_commit();
        if (nt > 1) load_keys(2, jt_lo + 1);
        cp_commit();
        load_rows(ci, hq);
        cp_wait_but_one();
        hand_over();
      }
      round(0, 1, s0, s1, nothing);
      mma_wait();
      for (int i = 0; i < nt; ++i) {
        const bool diag = shared_pair && i + 1 == nt;
        weights(s0, s1, c0, (jt_lo + i) * kChunk, diag);
        cp_wait_all();
        hand_over();
        const int kp = 1 + (i & 1);
        round(0, 3 - kp, s0, i + 1 < nt ? s1 : s0, [&](uint32_t sb, uint32_t tb) {
          const uint64_t z = make_desc(sb + tZ * kTile), k = make_desc(sb + 2 * kp * kTile);
          mma64<0, 1>(tb + s2, z, k, iKM, i > 0);
          if (diag) {
            mma64<1, 1>(tb + s0, make_desc(sb + tP * kTile), make_desc(sb + kTile), iMM, false);
            mma64<1, 1>(tb + s3, z, make_desc(sb), iMM, false);
          }
        });
        mma_wait();
        // this pair's rows are free again: the key tile after the next one, or the first query block of the key side
        if (i + 2 < nt) load_keys(kp, jt_lo + i + 2);
        else if (shared_pair && i + 2 == nt && nblk > 1) load_block(1);
        cp_commit();
      }
      float v[16];
      frag_ld(tl + s2, v);
      block_out(tZ, v, (bf16*)d.dq_swa + hq * 64, rq);
    }
    if (shared_pair) {
      first = 1;
      if (nblk > 2) load_block(2);                             // (q, do of this chunk have been read)
      cp_commit();
    } else {
      load_block(0);
      cp_commit();
      if (nblk > 1) load_block(1);
      cp_commit();
    }
  }
  if (first < nblk) {
    if (FULL) load_rows(ci + first / NG, h * NG + first % NG);
    cp_wait_but_one();
    hand_over();
    round(block_pair(first), own, s1, s2, nothing);
    mma_wait();
    for (int i = first; i < nblk; ++i) {
      weights(s1, s2, (ci + i / NG) * kChunk, c0, true);
      if (i + 1 < nblk) load_rows(ci + (i + 1) / NG, h * NG + (i + 1) % NG);
      cp_wait_all();
      hand_over();
      round(block_pair(i + 1), own, s1, i + 1 < nblk ? s2 : s1, [&](uint32_t sb, uint32_t tb) {
        const uint64_t q = make_desc(sb + 2 * block_pair(i) * kTile);
        mma64<1, 1>(tb + s0, make_desc(sb + tP * kTile), q + kTile / 16, iMM, i > 0);
        mma64<1, 1>(tb + s3, make_desc(sb + tZ * kTile), q, iMM, i > 0);
      });
      mma_wait();
      if (i + 2 < nblk) load_block(i + 2);                     // this block's buffers are free again
      cp_commit();
    }
  }
  // ---- dk_swa; dv with the slot part (or the window part alone, in fp32) ---------------------------------------------------------
  const int shift = seq_shift(d, rc.n);
  {
    float v[16];
    frag_ld(tl + s0, v);
#pragma unroll
    for (int x = 0; x < 2; ++x)
      if (c0 + r0 + 8 * x < len) {
        float* dst = w.dvacc + ((size_t)(t0 + c0 + r0 + 8 * x) * H + h) * 64 + cbase;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (!FULL) {
            *reinterpret_cast<float2*>(dst + 8 * j) = make_float2(v[4 * j + 2 * x], v[4 * j + 2 * x + 1]);
          } else if (c0 + r0 + 8 * x < len - shift) {
            const float2 f = *reinterpret_cast<const float2*>(dst + 8 * j);
            v[4 * j + 2 * x] += f.x;
            v[4 * j + 2 * x + 1] += f.y;
          }
        }
      }
    if (FULL) block_out(tP, v, (bf16*)d.dv + h * 64, rp);
    frag_ld(tl + s3, v);
    block_out(tZ, v, (bf16*)d.dk_swa + h * 64, rp);
  }
  if (FULL && c0 + kChunk > len - shift) {                     // tokens that never enter the slot memory
    const int M = d.M;
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = lr + 32 * u;
      if (c0 + r >= len - shift && c0 + r < len) {
        const int64_t row = (int64_t)(t0 + c0 + r) * H + h;
        *reinterpret_cast<uint4*>((bf16*)d.dk_gsa + row * 64 + 8 * lc) = z;
        if (8 * lc < M) {
          *reinterpret_cast<uint4*>((bf16*)d.ds + row * M + 8 * lc) = z;
          *reinterpret_cast<uint4*>((bf16*)d.dg + row * M + 8 * lc) = z;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
  if (failed) atomicExch(err, 1);
}

template <bool FULL>
static int win64_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  cudaError_t e = set_max_smem((const void*)nha_bwd_win64_kernel<FULL>, wn64::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  launch_after(nha_bwd_win64_kernel<FULL>, dim3((unsigned)(nha_chunk_count_bound(d->Ttot, d->N) * d->H)), kThreads, wn64::total, cs, *d, w, err);
  return check_launch();
}

// Both sides, behind bwd_slot64_launch().
int bwd_win64_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) { return win64_launch<true>(d, w, err, cs); }

bool bwd_wcols_umma_supported(const nha_chunk_desc* d) { return d->K == d->V && (d->K == 64 || d->K == 128); }

int bwd_wcols128_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs);

// The key side alone.  The caller has checked bwd_wcols_umma_supported().
int bwd_wcols_umma_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  return d->K == 64 ? win64_launch<false>(d, w, err, cs) : bwd_wcols128_launch(d, w, err, cs);
}

}  // namespace nha
