// Backward of the window branch, key side, for head dim 64: dk_swa and the window part of dv, 64-row products with every lane at
// work (nha_frag64.cuh).  For every query row that can see a key, with the row's joint log-sum-exp L and delta = <do, o>:
//     p = exp(scale q_swa k - L),  dz = scale p (do v - delta),  dv += p do,  dk_swa += dz q_swa.
//
// One CTA = the 64 keys of one (chunk, kv head), three CTAs per SM: the four accumulators lie two and two in the lane halves of
// 128 tensor-memory columns, and eight operand tiles are 67 KB.  It walks the blocks of 64 query rows that can see a key (query
// chunk x head of the group), one round of products per block:
//     dv += P^T do,  dk += dZ^T q_swa  of block i   together with   S = q_swa k^T,  dP = do v^T  of block i + 1
// with the rows of block i + 2 on their way.  The window part does not depend on the gates, so flagged chunks are done here too.
//
// What bounds it: the chain of rounds of a CTA, so that a third CTA of an SM is nearly as good as the first two: against two CTAs
// with 256 columns each B16 T2048 H16 W64 181 -> 153 us (48 % of the copy rate); 32768 packed tokens, windows 32-512, 288 -> 233 us.
// Fetching the rows of later CTAs into L2 does not help (with two CTAs: 181 us without, 186 with it).
//
// Replaces the third-party flash-attn varlen backward's dk / dv (call site nha_fla/ops/nha/chunk.py:333-344).
#include "nha_bwd_common.cuh"
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

namespace wc64 {
constexpr int tK = 0, tV = 1, tQ = 2, tDO = 3, kSet = 2, tP = 6, tZ = 7, kTiles = 8;       // tQ, tDO: two sets
constexpr int oBar = kTiles * kTile;
constexpr int total = oBar + 64 + 1024;
// an accumulator of 64 rows takes half of the lanes of its columns, and the next one the other half
constexpr uint32_t cS = 0, cDP = kOtherLanes, cDV = 64, cDK = 64 + kOtherLanes;
constexpr int kTmemCols = 128;
}  // namespace wc64

__global__ void __launch_bounds__(kThreads, 3) nha_bwd_wcols64_kernel(const nha_chunk_desc d, const BwdWs w, int* __restrict__ err) {
  grid_dep_wait();
  grid_dep_launch();
  using namespace wc64;
  const int H = d.H, HQ = d.HQ, NG = HQ / H;
  const int cg = blockIdx.x / H, h = blockIdx.x - cg * H;
  const ChunkRec rc = chunk_rec(d, cg);
  if (rc.n < 0) return;
  const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
  const int wl = seq_window(d, rc.n);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
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
  // query blocks that can see a key of this chunk
  const int nchunks = (len + kChunk - 1) / kChunk;
  const int qi_hi = wl < 0 ? nchunks - 1 : min(nchunks - 1, (c0 + kChunk - 1 + wl) / kChunk);
  const int nblk = (qi_hi - ci + 1) * NG;
  const int r0 = 16 * quarter + gq;                            // this lane's rows: r0 and r0 + 8
  auto load_block = [&](int i) {
    const int qrow = (ci + i / NG) * kChunk, hq = h * NG + i % NG, set = (i & 1) * kSet;
    load_tokens(tQ + set, d.q_swa, rq, hq * 64, qrow);
    load_tokens(tDO + set, d.d_o, rq, hq * 64, qrow);
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
  load_tokens(tK, d.k_swa, rp, h * 64, c0);
  load_tokens(tV, d.v, rp, h * 64, c0);
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
  const uint32_t iKK = idesc64(0, 0), iMM = idesc64(1, 1);
  auto issue_s = [&](int set) {
    mma64<0, 0>(tbase + cS, desc(tQ + set), desc(tK), iKK, false);
    mma64<0, 0>(tbase + cDP, desc(tDO + set), desc(tV), iKK, false);
  };
  const uint32_t fo0 = frag_off(quarter, half, lane, 0), fo1 = frag_off(quarter, half, lane, 1);
  const float sc2 = d.scale * kLog2e;
  if (tid == 0) issue_s(0);
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
    if (tid == 0) {
      mma64<1, 1>(tbase + cDV, desc(tP), desc(tDO + set), iMM, i > 0);
      mma64<1, 1>(tbase + cDK, desc(tZ), desc(tQ + set), iMM, i > 0);
      if (i + 1 < nblk) issue_s(kSet - set);
    }
    mma_wait();
    if (i + 2 < nblk) load_block(i + 2);                       // this block's buffers are free again
  }
  // ---- dk_swa as whole rows, the window part of dv in fp32 ------------------------------------------------------------------
  {
    float v[16];
    frag_ld(tl + cDK, v);
    frag_to_tile(at(tP, fo0), at(tP, fo1), v);
    frag_ld(tl + cDV, v);
#pragma unroll
    for (int x = 0; x < 2; ++x)
      if (c0 + r0 + 8 * x < len) {
        float* dst = w.dvacc + ((size_t)(t0 + c0 + r0 + 8 * x) * H + h) * 64 + 32 * half + 2 * tq;
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(dst + 8 * j) = make_float2(v[4 * j + 2 * x], v[4 * j + 2 * x + 1]);
      }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int r = lr + 32 * u;
    if (c0 + r < len && !failed)
      *reinterpret_cast<uint4*>((bf16*)d.dk_swa + (int64_t)(t0 + c0 + r) * rp + h * 64 + 8 * lc) =
          *reinterpret_cast<const uint4*>(tile(tP) + loff + 4096 * u);
  }
  if (failed) atomicExch(err, 1);
}

static int bwd_wcols64_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  cudaError_t e = set_max_smem((const void*)nha_bwd_wcols64_kernel, wc64::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  launch_after(nha_bwd_wcols64_kernel, dim3((unsigned)(nha_chunk_count_bound(d->Ttot, d->N) * d->H)), kThreads, wc64::total, cs, *d, w, err);
  return check_launch();
}

bool bwd_wcols_umma_supported(const nha_chunk_desc* d) { return d->K == d->V && (d->K == 64 || d->K == 128); }

int bwd_wcols128_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs);

// The caller has checked bwd_wcols_umma_supported().
int bwd_wcols_umma_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, cudaStream_t cs) {
  return d->K == 64 ? bwd_wcols64_launch(d, w, err, cs) : bwd_wcols128_launch(d, w, err, cs);
}

}  // namespace nha
