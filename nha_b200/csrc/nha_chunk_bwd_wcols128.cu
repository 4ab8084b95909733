// Backward of the window branch, key side, for head dim 128: dk_swa and the window part of dv, every lane at work (nha_frag64.cuh),
// two CTAs per SM.  With the joint log-sum-exp L and delta = <do, o> of the query-row pass, for every visible pair of a key and a query row
//     p = exp(scale q_swa k - L),  dz = scale p (do v - delta),  dv += p do,  dk_swa += dz q_swa,
// one round of products per block of 64 query rows:
//     dv^T += do^T P,  dk^T += q_swa^T dZ  of block i   together with   S = q_swa k^T,  dP = do v^T  of block i + 1.
// The sums are kept transposed, head dim along the 128 lanes and keys along 64 columns: as [64 keys][128] accumulators they would
// take 384 tensor-memory columns with the scores, and only one CTA would fit an SM.
//
// What bounds it: the chain of rounds of a CTA.  Measured against two blocks of 64 rows to a product with two rounds per pair and
// one CTA per SM: 2 x 1999 tokens, 32 heads on 8, window 127, 122 -> 75 us; issued by an elected lane 73 us.
//
// Replaces the third-party flash-attn varlen backward's dk / dv (call site nha_fla/ops/nha/chunk.py:333-344).
#include "nha_bwd_common.cuh"
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

namespace wc128 {
constexpr int D = 128;
constexpr int tK = 0, tV = 2, tQ = 4, tDO = 6, kSet = 4, tP = 12, tZ = 13, kTiles = 14;     // tQ, tDO: two sets
constexpr int oBar = kTiles * kTile;
constexpr int total = oBar + 64;                          // (the array itself is 1024-byte aligned: no slack)
constexpr int cS = 0, cDP = 64, cDV = 128, cDK = 192, kTmemCols = 256;
static_assert(total <= 113 * 1024, "two CTAs per SM");
}  // namespace wc128

__global__ void __launch_bounds__(kThreads, 2) nha_bwd_wcols128_kernel(const nha_chunk_desc d, const BwdWs w, int* __restrict__ err) {
  grid_dep_wait();
  grid_dep_launch();
  using namespace wc128;
  const int H = d.H, HQ = d.HQ, NG = HQ / H;
  const int cg = blockIdx.x / H, h = blockIdx.x - cg * H;
  const ChunkRec rc = chunk_rec(d, cg);
  if (rc.n < 0) return;
  const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
  const int wl = seq_window(d, rc.n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;
  const bool issuer = uniform(threadIdx.x >> 5) == 0;          // the warp whose elected lane issues the products

  extern __shared__ __align__(1024) unsigned char sm[];
  uint64_t* mbar = (uint64_t*)(sm + oBar);
  uint32_t* tslot = (uint32_t*)(mbar + 1);
  auto tile = [&](int i) { return sm + i * kTile; };
  const int lr = tid >> 3, lc = tid & 7;
  const uint32_t loff = sw_off(lr, lc);
  const int64_t rq = (int64_t)HQ * D, rp = (int64_t)H * D;
  auto load_tokens = [&](int t, const void* base, int64_t pitch, int col, int row) {
    const bf16* p = (const bf16*)base + (int64_t)t0 * pitch + col + 8 * lc;
    const bool ok0 = row + lr < len, ok1 = row + lr + 32 < len;
    const bf16 *p0 = p + (ok0 ? row + lr : 0) * pitch, *p1 = p + (ok1 ? row + lr + 32 : 0) * pitch;
#pragma unroll
    for (int k = 0; k < 2; ++k) tile_in(tile(t + k), loff, p0 + 64 * k, ok0, p1 + 64 * k, ok1);
  };
  // query blocks that can see a key of this chunk
  const int nchunks = (len + kChunk - 1) / kChunk;
  const int qi_hi = wl < 0 ? nchunks - 1 : min(nchunks - 1, (c0 + kChunk - 1 + wl) / kChunk);
  const int nblk = (qi_hi - ci + 1) * NG;
  const int r0 = 16 * quarter + gq;                            // this lane's rows: r0 and r0 + 8
  auto load_block = [&](int i) {
    const int qrow = (ci + i / NG) * kChunk, hq = h * NG + i % NG, set = (i & 1) * kSet;
    load_tokens(tQ + set, d.q_swa, rq, hq * D, qrow);
    load_tokens(tDO + set, d.d_o, rq, hq * D, qrow);
    cp_commit();
  };
  float nL[2], nD[2];                                          // -log-sum-exp (log2 units) and delta of a block's two rows
  auto load_rows = [&](int i) {
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int pq = (ci + i / NG) * kChunk + r0 + 8 * x;
      const size_t at = (size_t)(t0 + pq) * HQ + h * NG + i % NG;
      nL[x] = pq < len ? -w.lj[at] * kLog2e : 0.f;
      nD[x] = pq < len ? w.delta[at] : 0.f;
    }
  };
  load_tokens(tK, d.k_swa, rp, h * D, c0);
  load_tokens(tV, d.v, rp, h * D, c0);
  load_block(0);
  if (nblk > 1) load_block(1);
  load_rows(0);
  if (tid == 0) {
    mbar_init(mbar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc(tslot, kTmemCols);
  if (nblk > 1) cp_wait_but_one(); else cp_wait_all();
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
  const uint32_t iKK = idesc64(0, 0), iMM = make_idesc(128, 64, 1) | (1u << 15);
  auto issue_s = [&](auto desc, uint32_t tb, int set) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      mma64<0, 0>(tb + cS, desc(tQ + set + k), desc(tK + k), iKK, k > 0);
      mma64<0, 0>(tb + cDP, desc(tDO + set + k), desc(tV + k), iKK, k > 0);
    }
  };
  const uint32_t fo0 = frag_off(quarter, half, lane, 0), fo1 = frag_off(quarter, half, lane, 1);
  const float sc2 = d.scale * kLog2e;
  round([&](auto desc, auto desc2, uint32_t tb) { issue_s(desc, tb, 0); });
  mma_wait();
  for (int i = 0; i < nblk; ++i) {
    const int pq0 = (ci + i / NG) * kChunk + r0, set = (i & 1) * kSet;
    const float Lj[2] = {nL[0], nL[1]}, delta[2] = {nD[0], nD[1]};
    if (i + 1 < nblk) load_rows(i + 1);
    {
      float s[16], dp[16];
      frag_ld_nowait(tl + cS, s);
      frag_ld_nowait(tl + cDP, dp);
      tmem_ld_wait();
      // visible keys of a query row: klo <= key <= pq, tested as (unsigned)(key - klo) <= kspan; a row past the end sees nothing
      int off[2];
      unsigned kspan[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        const int pq = pq0 + 8 * x, klo = pq < len ? (wl < 0 ? 0 : max(0, pq - wl)) : (1 << 30);
        kspan[x] = pq < len ? (unsigned)(pq - klo) : 0u;
        off[x] = c0 + 32 * half + 2 * tq - klo;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int k = 4 * j + e, x = e >> 1;
          const float p = (unsigned)(off[x] + 8 * j + (e & 1)) <= kspan[x] ? exp2f(fmaf(s[k], sc2, Lj[x])) : 0.f;
          s[k] = p;
          dp[k] = p * (dp[k] - delta[x]) * d.scale;
        }
      frag_to_tile(at(tP, fo0), at(tP, fo1), s);
      frag_to_tile(at(tZ, fo0), at(tZ, fo1), dp);
    }
    cp_wait_all();
    hand_over();
    round([&](auto desc, auto desc2, uint32_t tb) {
      mma64<1, 1>(tb + cDV, desc2(tDO + set), desc(tP), iMM, i > 0);
      mma64<1, 1>(tb + cDK, desc2(tQ + set), desc(tZ), iMM, i > 0);
      if (i + 1 < nblk) issue_s(desc, tb, kSet - set);
    });
    mma_wait();
    if (i + 2 < nblk) load_block(i + 2);                       // this block's buffers are free again
  }
  // ---- dk_swa and the window part of dv (fp32): a thread holds 32 keys of one column, a warp 32 neighbouring columns of a key ----
  {
    const int dim = 32 * quarter + lane;
    float v[32];
    tmem_ld32(tl + cDV, v);
    if (!failed) {
      float* dst = w.dvacc + ((size_t)(t0 + c0 + 32 * half) * H + h) * D + dim;
#pragma unroll
      for (int e = 0; e < 32; ++e)
        if (c0 + 32 * half + e < len) dst[e * rp] = v[e];
    }
    tmem_ld32(tl + cDK, v);
    if (!failed) {
      bf16* dst = (bf16*)d.dk_swa + ((size_t)(t0 + c0 + 32 * half) * H + h) * D + dim;
#pragma unroll
      for (int e = 0; e < 32; ++e)
        if (c0 + 32 * half + e < len) dst[e * rp] = f2bf(v[e]);
    }
  }
  if (failed) atomicExch(err, 1);
  cp_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
}

int bwd_wcols128_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  cudaError_t e = set_max_smem((const void*)nha_bwd_wcols128_kernel, wc128::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  launch_after(nha_bwd_wcols128_kernel, dim3((unsigned)(nha_chunk_count_bound(d->Ttot, d->N) * d->H)), kThreads, wc128::total, cs, *d, w, err);
  return check_launch();
}

}  // namespace nha
