// State pass, per-chunk terms on the tensor cores (sm_100a): TMA loads, tcgen05 products, accumulators in tensor memory.
//
// One CTA per (chunk, kv head) forms, for K == V in {64, 128} and M == 64,
//     E[r,m]  = sum_{i > r} g'[i,m]                    (log decay from row r to the end of the chunk)
//     sb[r,m] = s'[r,m] exp(E[r,m])
//     L_k = k'^T sb  [K x M],   L_v = sb^T v'  [M x V],   Gend[m] = E[0,m] + g'[0,m]
// (primes: rows shifted right by gsa_kv_shift inside their sequence).  The running sum over rows is itself a matrix
// product, E = U g' with U the strictly upper triangular matrix of ones, so no thread scans anything: the gate tile
// goes from global memory to the tensor core without passing through registers, and bf16 gates times 1.0 summed in
// fp32 are exact up to the order of the additions.  All four inputs arrive by TMA into 128-byte-swizzled tiles that
// the products read in place (k', v', g', sb as MN-major operands: the token index is the contraction dimension of
// every product).  The wmma version of this kernel (nha_state_local_kernel) was bound by shared-memory bandwidth
// (fragment loads); this one touches shared memory from threads for the 8 KB weight tile and for the terms on their way out: stored
// straight from the accumulators' lanes, 16 bytes to a line, they took 94 us instead of 73 (16 x 2048 tokens, 16 heads of 64; 85 % of
// the copy rate) and 306 instead of 244 (131072 tokens, 8 heads of 128).  What bounds it: memory, then the chain of two rounds.
//
// Chunks whose rows are not all inside their sequence (the first chunks of a shifted sequence, a ragged last chunk,
// a sequence start inside a packed buffer) are filled by the threads with zero fill instead of TMA, so that no row of
// a neighbouring sequence enters a product.
//
// Same outputs as nha_state_local_kernel: L [NCB*H][K*M + M*V] bf16 and Gend [NCB*H][M] fp32 in the state scratch,
// consumed by nha_state_scan_kernel.  Replaces the per-chunk part of chunk_nha_fused_state_kernel
// (nha_fla/ops/nha/chunk_fused.py:31-114).
#include <cstdlib>
#include <cstring>

#include "nha_frag64.cuh"

namespace nha {

using namespace umma;

namespace stu {
constexpr int kThreads = 128;
constexpr int kTile = 8192;        // one [64][64] bf16 operand tile
// E, then L_k in columns 0-63; 64 columns of L_v are an accumulator of 64 rows, which takes half of the lanes: D = 64 in the lanes
// that L_k leaves of columns 0-63, D = 128 both halves side by side in columns 64-127
template <int D> constexpr int kCols = D == 64 ? 64 : 128;
constexpr int kPoll = 1 << 12;     // polls of at most kWaitHintNs each before a wait gives up
constexpr int kSmem = 228 * 1024;  // shared memory of an SM, of which every CTA takes 1 KB more than it asks for
}  // namespace stu

struct StateMaps {
  CUtensorMap k, v, g, s;
};

template <int D>
__global__ void __launch_bounds__(stu::kThreads) nha_state_local_umma_kernel(const nha_chunk_desc d, const StateWs w,
                                                                             int* __restrict__ err, const int chunk_lo,
                                                                             const __grid_constant__ StateMaps maps, const int dense_T,
                                                                             const int first_wave) {
  // Behind the plan of a batch of equal lengths (dense_T tokens each; that kernel lets this one start when it has itself waited for all
  // that came before) a CTA forms its chunk's record itself, reads the inputs from L2 and waits when its products are done.  Whole
  // prefill without and with it, nothing else changed: 777 tokens, 32 heads on 4, W 512: 38.0 -> 36.9 us; 4 x 500, 28 heads on 4, W 64:
  // 51.3 -> 50.4; 777 tokens, 16 heads of 64: 27.3 -> 26.5; training steps: no difference.
  // So does the first wave alone, which may run beside the plan and cannot tell whether the error word is set already or still what the
  // memory held before.  A later CTA finds the plan done: its wait costs nothing, and it does not start where one before it gave up.
  const bool beside = dense_T != 0 && (int)(blockIdx.y * gridDim.x + blockIdx.x) < first_wave;
  if (!beside) grid_dep_wait();
  grid_dep_launch();
  using namespace stu;
  constexpr int DT = D / 64;                      // 64-column tiles of k' and v'
  constexpr int kTmemCols = kCols<D>;
  constexpr int M = 64;
  const int cg = chunk_lo + blockIdx.x, h = blockIdx.y;
  ChunkRec rc;
  if (dense_T == 0) {
    rc = chunk_rec(d, cg);
  } else {
    const int per = (dense_T + kChunk - 1) / kChunk;
    rc.n = cg / per;
    rc.ci = cg - rc.n * per;
    rc.t0 = rc.n * dense_T;
    rc.len = dense_T;
    if (rc.n >= d.N) rc.n = -1;
  }
  if (rc.n < 0) {
    grid_dep_wait();
    return;
  }
  const int H = d.H;
  const int t0 = rc.t0, len = rc.len, p0 = rc.ci * kChunk;
  const int shift = seq_shift(d, rc.n, beside);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  unsigned char* sU = sm;                         // strictly upper triangular ones [64][64], K-major
  unsigned char* sG = sm + kTile;                 // g' [64 rows][64 slots]
  unsigned char* sS = sm + 2 * kTile;             // s', overwritten by sb
  unsigned char* sK = sm + 3 * kTile;             // k' [64 rows][D] as DT tiles
  unsigned char* sV = sK + DT * kTile;
  uint64_t* bar = (uint64_t*)(sV + DT * kTile);   // [0] loads, [1] products
  uint32_t* tslot = (uint32_t*)(bar + 2);
  __shared__ int s_abort;

  // rows of the chunk hold shifted positions p = p0 + r, token p - shift; valid while shift <= p < len
  const bool full = p0 >= shift && p0 + kChunk <= len;
  const int64_t row0 = (int64_t)t0 + p0 - shift;  // packed row of the chunk's first row
  if (warp == 0) tmem_alloc(tslot, kTmemCols);
  if (tid == 32) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = beside ? 0 : *(volatile int*)err;         // an earlier CTA of this launch gave up on a wait: do not start
    if (full && !s_abort) {                             // (the tiles are on their way while the others reach the barrier)
      fence_async_smem();
      mbar_expect_tx(&bar[0], (2 + 2 * DT) * kTile);
      tma_load_3d(sG, &maps.g, 0, h, (int)row0, &bar[0]);
      tma_load_3d(sS, &maps.s, 0, h, (int)row0, &bar[0]);
#pragma unroll
      for (int kt = 0; kt < DT; ++kt) {
        tma_load_3d(sK + kt * kTile, &maps.k, 64 * kt, h, (int)row0, &bar[0]);
        tma_load_3d(sV + kt * kTile, &maps.v, 64 * kt, h, (int)row0, &bar[0]);
      }
    }
  }
  if (tid < 64) {
    // row r of U: ones right of the diagonal
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      uint32_t pr[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 8 * c + 2 * e;
        pr[e] = (i > tid ? 0x3F80u : 0u) | (i + 1 > tid ? 0x3F800000u : 0u);
      }
      *reinterpret_cast<uint4*>(sU + sw_off(tid, c)) = make_uint4(pr[0], pr[1], pr[2], pr[3]);
    }
  }
  if (!full) {
    // zero-filling copies by the threads: 16-byte pieces into the swizzled tiles
    auto fill = [&](unsigned char* dst, const bf16* base, int width, int col0) {
      for (int i = tid; i < kChunk * 8; i += kThreads) {
        const int r = i >> 3, c = i & 7;
        const int p = p0 + r;
        const bool ok = p >= shift && p < len;
        cp16(dst + sw_off(r, c), ok ? base + ((row0 + r) * H + h) * width + col0 + 8 * c : base, ok);
      }
    };
    fill(sG, (const bf16*)d.g, M, 0);
    fill(sS, (const bf16*)d.s, M, 0);
#pragma unroll
    for (int kt = 0; kt < DT; ++kt) {
      fill(sK + kt * kTile, (const bf16*)d.k_gsa, D, 64 * kt);
      fill(sV + kt * kTile, (const bf16*)d.v, D, 64 * kt);
    }
    cp_commit();
    cp_wait_all();
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  if (s_abort) {
    if (warp == 0) tmem_dealloc(tbase, kTmemCols);
    grid_dep_wait();
    return;
  }
  bool failed = false;
  // every thread observes the arrival of the tiles itself (it reads the weight tile with ordinary loads later)
  if (full && !mbar_wait_limit(&bar[0], 0, kPoll)) failed = true;
  const bool issuer = uniform(threadIdx.x >> 5) == 0;          // the warp whose elected lane issues the products
  if (issuer) {
    tc_fence_after();
    const uint32_t u = uniform(smem_u32(sU)), g = uniform(smem_u32(sG)), tb = uniform(tbase);
    if (elect_one()) {
      f64::mma64<0, 1>(tb, make_desc(u), make_desc(g), f64::idesc64(0, 1), false);
      commit(&bar[1]);
    }
  }
  if (!failed && !mbar_wait_limit(&bar[1], 0, kPoll)) failed = true;
  tc_fence_after();
  // E is an M = 64 accumulator, read in fragments (nha_frag64.cuh): this warp has the rows 16 warp + gq (+ 8), 32 columns at a time
  const int gq = lane >> 2, tq = lane & 3;
  const uint32_t tl = tbase + ((uint32_t)(warp * 32) << 16);
  float e0[16], e1[16];
  f64::frag_ld_nowait(tl, e0);
  f64::frag_ld_nowait(tl + 32, e1);
  tmem_ld_wait();
  if (warp == 0 && gq == 0 && !failed) {          // row 0: Gend = E + g'
    float* ge = w.gend + ((size_t)cg * H + h) * M + 2 * tq;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const float2 g0 = f64::pair_f32(*reinterpret_cast<const uint32_t*>(sG + sw_off(0, c) + 4 * tq));
      const float *e = c < 4 ? e0 + 4 * c : e1 + 4 * (c - 4);
      *reinterpret_cast<float2*>(ge + 8 * c) = make_float2(e[0] + g0.x, e[1] + g0.y);
    }
  }
  uint32_t fo[2][2];                              // this lane's rows of the blocks that one stmatrix / ldmatrix moves
#pragma unroll
  for (int x = 0; x < 4; ++x) fo[x >> 1][x & 1] = f64::frag_off(warp, x >> 1, lane, x & 1);
#pragma unroll
  for (int half = 0; half < 2; ++half)
#pragma unroll
    for (int jp = 0; jp < 2; ++jp) {
      uint32_t sv[4];
      const uint32_t at = smem_u32(sS) + fo[half][jp];
      f64::ldm4(at, sv);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        // matrix q of the pair: rows gq (+ 8 for odd q), columns of block 2 jp + q / 2
        const float* e = (half ? e1 : e0) + 4 * (2 * jp + (q >> 1)) + 2 * (q & 1);
        const float2 x = f64::pair_f32(sv[q]);
        sv[q] = f64::pair_bf16(x.x * __expf(e[0]), x.y * __expf(e[1]));
      }
      f64::stm4(at, sv[0], sv[1], sv[2], sv[3]);
    }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  const uint32_t cV = D == 64 ? f64::kOtherLanes : 64u;
  if (issuer) {
    tc_fence_after();
    // L_k [D x 64] = k'^T sb: both operands MN-major, 16 tokens per k step; with D = 128 the A operand spans two
    // 64-column tiles, kTile bytes apart (LBO).  L_v [64 x D] = sb^T v', 64 columns to an accumulator.
    const uint32_t idk = make_idesc(D, 64, 1) | (1u << 15);
    const uint32_t idv = make_idesc(64, 64, 1) | (1u << 15);
    const uint32_t ak = uniform(smem_u32(sK)), as = uniform(smem_u32(sS)), av = uniform(smem_u32(sV)), tb = uniform(tbase);
    if (elect_one()) {
#pragma unroll
      for (int ks = 0; ks < 4; ++ks) {
        mma_f16(tb, make_desc_lbo(ak + ks * 2048, kTile), make_desc(as + ks * 2048), idk, ks > 0);
#pragma unroll
        for (int t = 0; t < DT; ++t)
          mma_f16(tb + cV + t * f64::kOtherLanes, make_desc(as + ks * 2048), make_desc(av + t * kTile + ks * 2048), idv, ks > 0);
      }
      commit(&bar[1]);
    }
  }
  if (!failed && !mbar_wait_limit(&bar[1], 1, kPoll)) failed = true;
  tc_fence_after();
  grid_dep_wait();                                // (the plan sets the error word to zero, and every CTA outlasts it)
  // The terms leave through the tiles that the products have read, in whole rows of 128 bytes: stored straight from the accumulators'
  // lanes every 16 bytes would be a line of their own.
  bf16* Lk = w.local + ((size_t)cg * H + h) * ((size_t)D * M + (size_t)M * D);
  bf16* Lv = Lk + (size_t)D * M;
  const int sr = lane >> 3, sc = lane & 7;
  auto stage = [&](unsigned char* tile, uint32_t taddr) {       // an accumulator of 64 rows: this warp's sixteen
    float x[16];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      f64::frag_ld(taddr + 32 * half, x);
      f64::frag_to_tile(smem_u32(tile) + fo[half][0], smem_u32(tile) + fo[half][1], x);
    }
  };
  auto store = [&](bf16* dst, int pitch, const unsigned char* tile, int r0, auto rows) {
#pragma unroll
    for (int u = 0; u < decltype(rows)::value / 4; ++u) {
      const int r = r0 + 4 * u + sr;
      *reinterpret_cast<uint4*>(dst + (size_t)r * pitch + 8 * sc) = *reinterpret_cast<const uint4*>(tile + sw_off(r, sc));
    }
  };
  if (D == 128) {                                               // M = 128 accumulator: row = lane
    float x[64];
    tmem_ld64(tl, x);
#pragma unroll
    for (int c = 0; c < 8; ++c) *reinterpret_cast<uint4*>(sK + sw_off(tid, c)) = pack8(x + 8 * c);
  } else {
    stage(sK, tl);
  }
#pragma unroll
  for (int t = 0; t < DT; ++t) stage(sV + t * kTile, tl + cV + t * f64::kOtherLanes);
  __syncwarp();
  if (!failed) {
    if (D == 128) store(Lk, M, sK, 32 * warp, std::integral_constant<int, 32>{});
    else store(Lk, M, sK, 16 * warp, std::integral_constant<int, 16>{});
#pragma unroll
    for (int t = 0; t < DT; ++t) store(Lv + 64 * t, D, sV + t * kTile, 16 * warp, std::integral_constant<int, 16>{});
  }
  if (failed) atomicExch(err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
}

bool state_local_umma_supported(const nha_chunk_desc* d) {
  if (d->K != d->V || (d->K != 64 && d->K != 128) || d->M != 64) return false;
  const char* off = getenv("NHA_B200_NO_UMMA");
  if (off && off[0] == '1') return false;
  off = getenv("NHA_B200_NO_STATE_UMMA");
  return !(off && off[0] == '1');
}

// Launches the tensor-core version of the per-chunk terms; NHA_ERR_UNSUPPORTED when the tensor maps cannot be made (the
// caller then runs nha_state_local_kernel).
int state_local_umma_launch(const nha_chunk_desc* d, const StateWs& w, int* err, int chunk_lo, int chunk_n, cudaStream_t cs, int dense_T) {
  using namespace stu;
  StateMaps maps;
  memset(&maps, 0, sizeof(maps));
  const bool ok = make_map_rows_heads(&maps.k, d->k_gsa, d->Ttot, d->H, d->K) &&
                  make_map_rows_heads(&maps.v, d->v, d->Ttot, d->H, d->V) &&
                  make_map_rows_heads(&maps.g, d->g, d->Ttot, d->H, d->M) &&
                  make_map_rows_heads(&maps.s, d->s, d->Ttot, d->H, d->M);
  if (!ok) return NHA_ERR_UNSUPPORTED;
  const int DT = d->K / 64;
  const int total = 1024 + (3 + 2 * DT) * kTile + 64;
  const void* fn = DT == 2 ? (const void*)nha_state_local_umma_kernel<128> : (const void*)nha_state_local_umma_kernel<64>;
  cudaError_t e = set_max_smem(fn, total);
  if (e != cudaSuccess) return record_cuda_error(e);
  // shared memory is what limits the CTAs of an SM: five at head dim 64, three at 128
  const int first_wave = sm_count() * (kSmem / (total + 1024));
  if (DT == 2) launch_after(nha_state_local_umma_kernel<128>, dim3(chunk_n, d->H), kThreads, total, cs, *d, w, err, chunk_lo, maps, dense_T, first_wave);
  else launch_after(nha_state_local_umma_kernel<64>, dim3(chunk_n, d->H), kThreads, total, cs, *d, w, err, chunk_lo, maps, dense_T, first_wave);
  return check_launch();
}

}  // namespace nha
