// Output pass of the chunked NHA forward for head dim 128, as a
// warp-specialised pipeline on the sm_100a tensor-core path.
//
// One CTA = one 128-row tile: a 64-token chunk of TWO query heads of one kv head.  320 threads and about 107 KB of
// shared memory, so that TWO CTAs share an SM: while one of them runs its prologue, its slot phase (a chain of four
// short product groups with element-wise work in between) or its epilogue, the other keeps the tensor pipe and the
// exponential unit busy with window steps.  Roles:
//   warps 0-7   softmax group: TWO threads per row (warps w and w + 4, alternate 32-column halves of every 64-column
//               accumulator; tcgen05.ld gives a thread its row); element-wise work only.  Everything it hands to the
//               tensor pipe is written back into TENSOR MEMORY as bf16 pairs (tcgen05.st), each thread over columns that
//               it has read itself, and read from there as the A operand of the next product, so it never stores an
//               operand to shared memory;
//   warp 8      loads: every operand tile by TMA (cp.async.bulk.tensor on maps of this GPU's own tensors, no
//               multicast) into 128-byte-swizzled tiles, bytes counted on mbarriers; q_gsa, the slot operands and the
//               window tiles stream through a ring of 16 KB slots (three, and the storage of the sign matrix as a fourth
//               once its product is done); window keys and values are polled independently, a slot is refilled as soon as
//               the product that read it has completed; a tile that sticks out of its sequence is written by the
//               warp itself with zero fill, so that no row of a neighbouring sequence ever enters a product;
//   warp 9      one thread issues every tcgen05.mma and commits completions to mbarriers.
// Products of a tile (S0, S1: two 64-column accumulators; O: the 128-column output accumulator):
//     G0  x = G - Gend / 2 -> O's last columns       group: a = exp(x) in its place, s' .* b = s' exp(-x), e^R = a of row 63
//         (the running sum of the gates as a product with +-1/2, exact in bf16: every thread gets its own row's exponents)
//     G1  A = q k'^T -> S0, QH = q Hk -> S1          group: tril(A) -> bf16 in O's first columns
//     G2  X = tril(A) (s' .* b) -> S0                group: slot logits ok = scale a .* (e^R .* QH + X), p~ = exp(ok - max),
//                                                            p~ a e^R and p~ a -> bf16 in S0
//     G3  O = (p~ a e^R) Hv, Bv = (p~ a)(s' .* b)^T -> S1      group: tril(Bv) -> bf16 in S1
//     G4  O += tril(Bv) v'
//     window steps, newest key tile first (64 keys each):   S_j = q_swa K_j^T into S(j & 1) (S_{j+2} is issued as soon
//         as the group has read S_j);   group: P~_j = exp(scale S_j - m) -> bf16 over half of the columns of S_j;
//         O += P~_j V_j
// Shared-memory bandwidth is what bounds the tensor pipe here (a 128 x 64 x 16 product reads 6 KB of operands in its
// 32 cycles): the value products therefore take all 128 columns of V at once (an MN-major operand spanning two
// swizzle atoms) and every A operand but q comes from tensor memory.
// ONE softmax over the slot logits and all window logits, in a single sweep: the running reference m of a row starts
// as its slot maximum and is only raised when a window logit exceeds it by more than 8 ln 2 (probabilities then stay
// below 256, exact in the fp32 accumulator); raising it rescales the row of O in tensor memory (tcgen05.ld / st by the
// row's thread, after the products in flight on O have completed).  With one head per kv head the reference follows the
// maximum itself: those calls came from a kernel with exact maxima, whose largest probability, rounded to bf16 for the value
// product, is exactly 1 (error of o against 64 bits, W 512: 2.14e-3, with the lagging reference 2.34e-3; the rescaling that it
// costs would be 7 % of the document prefill of a grouped model, which never had it).  Decay factorisation, flags for chunks that decay
// too fast for one reference per chunk, and the general kernel that takes those: as in nha_chunk_fwd_umma.cu.
//
// What bounds it: latencies that two CTAs an SM cover in part (issue slots 48 % busy, DRAM 28 %).  Clocks of a tile at W 512, two CTAs
// an SM: 8 k to the decay factors, 10 k for the slot rounds, 2.0 k for each of nine window steps (400 waiting for the scores, 650 maxima,
// 850 exponentials), 3 k to the end: nearly half lies in front of the window steps, and all of that but the products
// with q is the same for every pair of heads of a kv head.  Against one thread a
// row, the gates scanned in shared memory, and the tiles of a chunk far apart in the grid: 131072 tokens, 32 heads on 8, W 512,
// 2714 -> 2600-2640 us, and 2578 with products issued by an elected lane and shared memory
// addressed as such (on a GPU where it was 2909 before); 2 x 1999 tokens, 32 heads on 8, W 127, 76 -> 71 us.  An L2 prefetch of a later CTA's tiles: 1 % better in
// the first, 4 % worse in the second.
//
// Replaces chunk_nha_fused_o_kernel (nha_fla/ops/nha/chunk_fused.py:117-283) at the long-context shape.
#include <cuda.h>
#include <string.h>

#include "nha_common.cuh"
#include "nha_tma.cuh"
#include "nha_umma.cuh"

namespace nha {

using namespace umma;

namespace pipe {
constexpr int D = 128, M = 64;
constexpr int kGroup = 256;                       // threads of the softmax group
constexpr int kThreads = kGroup + 64;
constexpr int kQTile = 128 * 128;                 // one 64-wide k tile of a 128-row A operand
constexpr int kSlot = 16384;
constexpr int oQS = 0;                            // q_swa [2 k tiles][128][64]; at the end the staging of the output rows
constexpr int oRing = oQS + 2 * kQTile;           // ring slots 0-2
constexpr int oSign = oRing + 3 * kSlot;          // coefficients of x, [128][64] (both heads' rows alike); then ring slot 3
constexpr int oSB = oSign + kSlot;                // s', then s' .* b [64][64]
constexpr int oG = oQS + kQTile;                  // gates [64][64], in the second q_swa tile until G0 has read them
constexpr int oER = oSB + 8192;                   // fp32 [64] exp(R)
constexpr int oX = oER + 256;                     // fp32 [2][128] exchanges between the two threads of a row
constexpr int oBar = oX + 1024;
constexpr int total = oBar + 256 + 1024;          // + slack for the 1024-byte alignment of the base
static_assert(total <= 113 * 1024, "two CTAs of the pipelined output pass per SM");
// mbarriers
constexpr int bQ = 0, bFull = 1, bEmpty = 5, bGS = 9, bG = 10, bW = 11, bS = 12, bP = 14, bPV = 16, bKq = 18, bX = 19, nBar = 20;
constexpr int kPoll = 1 << 15;                    // polls of a bounded wait (each sleeps up to 20 us in hardware)
constexpr float kDecayLimit = 140.0f;
constexpr float kRaise = 5.545177f;               // 8 ln 2
constexpr int kTmemCols = 256;
}  // namespace pipe

struct PipeMaps {
  CUtensorMap qg, qs, kg, ks, v, g, s, hk, hv;
};

__device__ __forceinline__ void tmem_st32(uint32_t taddr, const uint32_t* in) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,"
      "%31,%32};" ::"r"(taddr),
      "r"(in[0]), "r"(in[1]), "r"(in[2]), "r"(in[3]), "r"(in[4]), "r"(in[5]), "r"(in[6]), "r"(in[7]), "r"(in[8]), "r"(in[9]),
      "r"(in[10]), "r"(in[11]), "r"(in[12]), "r"(in[13]), "r"(in[14]), "r"(in[15]), "r"(in[16]), "r"(in[17]), "r"(in[18]),
      "r"(in[19]), "r"(in[20]), "r"(in[21]), "r"(in[22]), "r"(in[23]), "r"(in[24]), "r"(in[25]), "r"(in[26]), "r"(in[27]),
      "r"(in[28]), "r"(in[29]), "r"(in[30]), "r"(in[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* in) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
      "r"(in[0]), "r"(in[1]), "r"(in[2]), "r"(in[3]), "r"(in[4]), "r"(in[5]), "r"(in[6]), "r"(in[7]), "r"(in[8]), "r"(in[9]),
      "r"(in[10]), "r"(in[11]), "r"(in[12]), "r"(in[13]), "r"(in[14]), "r"(in[15])
      : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* in) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(in[0]), "r"(in[1]), "r"(in[2]),
               "r"(in[3]), "r"(in[4]), "r"(in[5]), "r"(in[6]), "r"(in[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t bf16_pair(float lo, float hi) {
  const __nv_bfloat162 h2 = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h2);
}

__global__ void __launch_bounds__(pipe::kThreads, 2)
    nha_fwd_pipe_kernel(const nha_chunk_desc d, int* __restrict__ flags, int* __restrict__ err,
                        const __grid_constant__ PipeMaps maps, const int early) {
  // Only Hk and Hv come from the kernel in front.  Behind the scan of the state pass (`early`), whose CTAs let this grid start when they
  // have themselves waited for all that came before, everything else is in memory: the loads, the decay factors and A = q k'^T go
  // ahead, and the load warp alone waits, in front of Hk.  (What threads read before that they read from L2.)  Whole prefill without
  // and with it, nothing else changed: 777 tokens, 32 heads on 4, W 512: 42.1 -> 36.9 us; where the grid is several waves, the first of
  // them gains: 4 x 500 tokens, 28 heads on 4, W 64: 50.9 -> 50.4; 1500 tokens, 32 heads on 8, W 64: 47.1 -> 46.5; 8000 tokens, W 512:
  // 211.6 -> 210.3; 32768 tokens: no difference.
  if (!early) grid_dep_wait();
  grid_dep_launch();
  using namespace pipe;
  const int H = d.H, HQ = d.HQ, NG = HQ / H;
  // tiles of a chunk are neighbours in the grid: two heads a tile fastest, then the kv heads
  const int NZ = (NG + 1) / 2;
  const int u = blockIdx.x / NZ, z = blockIdx.x - u * NZ, cg = u / H, h = u - cg * H;
  const ChunkRec rc = chunk_rec(d, cg, early);
  if (rc.n < 0) {
    grid_dep_wait();
    return;
  }
  const int n = rc.n, ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
  if (c0 < d.q_offset) {
    grid_dep_wait();
    return;
  }
  // chunks below q_offset have no queries (q_offset is a multiple of 64)
  const int tq0 = t0 - d.q_offset;                 // row of q / o / lse that holds position 0 of the sequence
  const int wl = seq_window(d, n, early), shift = seq_shift(d, n, early);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int hq0 = h * NG + 2 * z;
  // an odd group's last tile holds one head: its other 64 rows are computed (on the next group's queries, or on the zeros
  // that TMA reads past the last head) and never stored
  const bool two = 2 * z + 1 < NG;

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  float* ER = (float*)(sm + oER);
  float* xch = (float*)(sm + oX);
  uint64_t* bar = (uint64_t*)(sm + oBar);
  uint32_t* tslot = (uint32_t*)(bar + nBar);
  __shared__ int s_abort;

  // window key tiles, newest first: step j covers the keys [64 (ci - j), 64 (ci - j) + 64)
  const int jt_lo = wl < 0 ? 0 : max(0, c0 - wl) / kChunk;
  const int nst = ci - jt_lo + 1;

  if (warp == 9) {
    if (lane < nBar) {
      const bool many = lane == bW || lane == bP || lane == bP + 1;
      mbar_init(&bar[lane], many ? kGroup : 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (lane == 31) s_abort = *(volatile int*)err;    // an earlier CTA of this launch gave up on a wait: do not start
  }
  if (warp == 0) tmem_alloc(tslot, kTmemCols);
  if (tid < kGroup) {
    // coefficients of x: row t has 1/2 up to column t (mod 64) and -1/2 after it
    const int r = tid >> 1, t = r & 63;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int c = 4 * (tid & 1) + u;
      uint32_t pr[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int i = 8 * c + 2 * e;
        pr[e] = (i <= t ? 0x3F00u : 0xBF00u) | (i + 1 <= t ? 0x3F000000u : 0xBF000000u);
      }
      *reinterpret_cast<uint4*>(sm + oSign + sw_off(r, c)) = make_uint4(pr[0], pr[1], pr[2], pr[3]);
    }
    fence_async_smem();
  }
  const int hi = len - shift;
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
#define NHA_WAIT(idx_, par_)                                                       \
  do {                                                                             \
    if (!failed && !mbar_wait_limit(&bar[idx_], (uint32_t)(par_), kPoll)) failed = true; \
  } while (0)

  // ---- loads (warp 8) ---------------------------------------------------------------------------------------------
  // Ring slots and what passes through them, in fill order:
  //   slot 0: q_gsa k tile 0, Hv, window values of the even steps      slot 1: q_gsa k tile 1, v', window keys of the odd steps
  //   slot 2: Hk, window keys of the even steps (k' passes through the q_swa tiles)                    slot 3 (the sign matrix's storage): values of the odd steps
  // Fill number f of a slot waits for release number f - 1 of that slot (a commit of the MMA thread behind the last
  // product that read it); the first fill of slot 3 waits for the product with the sign matrix.
  auto slot_ptr = [&](int slot) { return sm + (slot < 3 ? oRing + slot * kSlot : oSign); };
  auto ragged_fill = [&](unsigned char* dst, const bf16* base, int r0, int rlo, int rhi) {
    // [64 rows][128 columns] as two swizzled 64-column tiles; rows outside [rlo, rhi) become zeros
#pragma unroll 1
    for (int it = 0; it < 32; it += 8) {
      uint4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = lane + 32 * (it + u);
        const int r = i >> 4, c = i & 15;
        const int gr = r0 + r;
        v[u] = make_uint4(0u, 0u, 0u, 0u);
        if (gr >= rlo && gr < rhi) v[u] = ld_l2(reinterpret_cast<const uint4*>(base + (size_t)gr * H * D + 8 * c));
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int i = lane + 32 * (it + u);
        const int r = i >> 4, c = i & 15;
        *reinterpret_cast<uint4*>(dst + (c >> 3) * 8192 + sw_off(r, c & 7)) = v[u];
      }
    }
    fence_async_smem();
    __syncwarp();
  };
  // rows [r0, r0 + 64) of one kv head of a [tokens][H][128] tensor into a slot: by TMA when they lie inside [rlo, rhi)
  auto load_rows_to = [&](unsigned char* dst, uint64_t* fb, const CUtensorMap* mp, const bf16* base, int r0, int rlo, int rhi) {
    if (r0 >= rlo && r0 + kChunk <= rhi) {
      if (lane == 0) {
        mbar_expect_tx(fb, 16384);
        tma_load_3d(dst, mp, 0, h, t0 + r0, fb);
        tma_load_3d(dst + 8192, mp, 64, h, t0 + r0, fb);
      }
    } else {
      ragged_fill(dst, base + ((size_t)t0 * H + h) * D, r0, rlo, rhi);
      if (lane == 0) mbar_arrive(fb);
    }
  };
  auto load_rows = [&](int slot, const CUtensorMap* mp, const bf16* base, int r0, int rlo, int rhi) {
    load_rows_to(slot_ptr(slot), &bar[bFull + slot], mp, base, r0, rlo, rhi);
  };
  // rows of the chunk's gates or write weights ([tokens][H][64]) into one 64-column tile
  auto load_slots_to = [&](unsigned char* dst, const CUtensorMap* mp, const bf16* base, int r0) {
    if (r0 >= 0 && r0 + kChunk <= hi) {
      if (lane == 0) {
        mbar_expect_more(&bar[bGS], 8192);
        tma_load_3d(dst, mp, 0, h, t0 + r0, &bar[bGS]);
      }
    } else {
#pragma unroll 1
      for (int it = 0; it < 16; it += 8) {
        uint4 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = lane + 32 * (it + u), r = i >> 3, c = i & 7, gr = r0 + r;
          v[u] = make_uint4(0u, 0u, 0u, 0u);
          if (gr >= 0 && gr < hi) v[u] = ld_l2(reinterpret_cast<const uint4*>(base + ((size_t)(t0 + gr) * H + h) * M + 8 * c));
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int i = lane + 32 * (it + u);
          *reinterpret_cast<uint4*>(dst + sw_off(i >> 3, i & 7)) = v[u];
        }
      }
      fence_async_smem();
      __syncwarp();
    }
  };
  if (warp == 8) {
    load_slots_to(sm + oG, &maps.g, (const bf16*)d.g, c0 - shift);
    load_slots_to(sm + oSB, &maps.s, (const bf16*)d.s, c0 - shift);
    if (lane == 0) mbar_arrive(&bar[bGS]);
    // Everything the first product group needs goes in flight at once: q_gsa (k tile kt into slot kt; rows 0-63 head hq0,
    // rows 64-127 head hq0 + 1), Hk into slot 2, and k' into the first half of the q_swa tiles, which the window steps
    // need only much later (q_swa is fetched once A = q k'^T has read k').
    if (lane == 0) {
      mbar_expect_tx(&bar[bFull + 0], 16384);
      mbar_expect_tx(&bar[bFull + 1], 16384);
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int kt = 0; kt < 2; ++kt)
          tma_load_3d(slot_ptr(kt) + hh * 8192, &maps.qg, 64 * kt, hq0 + hh, tq0 + c0, &bar[bFull + kt]);
    }
    load_rows_to(sm + oQS, &bar[bQ], &maps.kg, (const bf16*)d.k_gsa, c0 - shift, 0, hi);     // k'
    grid_dep_wait();
    if (lane == 0) {
      mbar_expect_tx(&bar[bFull + 2], 16384);
      tma_load_2d(slot_ptr(2), &maps.hk, 0, (cg * H + h) * D, &bar[bFull + 2]);              // Hk [128][64]
    }
  }

  // ---- G0, G1 (MMA thread); decay factors (group) ------------------------------------------------------------------
  constexpr uint32_t kT16 = kQTile >> 4;               // k-tile pitch of a 128-row A operand, in descriptor units
  const uint32_t iK = make_idesc(128, 64, 0), iMN = make_idesc(128, 64, 1), iMN128 = make_idesc(128, 128, 1);
  const int half = warp >> 2;                          // softmax group: which 32 columns of 64
  const int row = (warp & 3) * 32 + lane;              // softmax group: row of the tile
  const uint32_t tl = tbase + ((uint32_t)((warp & 3) * 32) << 16);     // S0 at +0, S1 at +64, O at +128
  constexpr float kLog2e = 1.4426950408889634f;
  int mine_unsafe = 0;
  // The MMA warp waits as a whole and issues from one elected lane, with addresses that the compiler can see to be the same in all
  // lanes (see elect_one()), formed close to their use.  Against a branch on lane 0: 131072 tokens, 32 heads on 8, W 512, 2909 -> 2675 us;
  // 777 tokens, 32 heads on 4, 29.3 -> 27.1; 4 x 500, 28 on 4, W 64, 37.7 -> 35.8.
  const int uwarp = (int)uniform(threadIdx.x >> 5);
  auto slot_off = [](int slot) { return (uint32_t)(slot < 3 ? oRing + slot * kSlot : oSign); };
  if (uwarp == 9) {
    const uint32_t su = uniform(smem_u32(sm)), tu = uniform(tbase);
    {
      NHA_WAIT(bGS, 0);
      tc_fence_after();
      if (elect_one()) {
        mma_run<4, 1>(tu + 192, make_desc(su + oSign), 0, make_desc(su + oG), 0, iMN, false);
        commit(&bar[bX]);
      }
      // G1: A = q k'^T (q_gsa k tiles in slots 0 and 1, 16384 bytes apart; k' in the q_swa tiles), QH = q Hk (Hk in slot 2)
      NHA_WAIT(bFull + 0, 0);
      NHA_WAIT(bFull + 1, 0);
      NHA_WAIT(bQ, 0);                                   // k' in the first half of the q_swa tiles
      tc_fence_after();
      const uint64_t dQG = make_desc(su + slot_off(0));
      if (elect_one()) {
        mma_run<8, 0>(tu, dQG, kSlot >> 4, make_desc(su + oQS), 8192 >> 4, iK, false);
        commit(&bar[bKq]);
      }
      NHA_WAIT(bFull + 2, 0);
      tc_fence_after();
      if (elect_one()) {
        mma_run<8, 1>(tu + 64, dQG, kSlot >> 4, make_desc(su + slot_off(2)), 0, iMN, false);
        commit(&bar[bG]);
        commit(&bar[bEmpty + 0]);
        commit(&bar[bEmpty + 1]);
        commit(&bar[bEmpty + 2]);
      }
    }
  } else if (warp < 8) {
    NHA_WAIT(bGS, 0);
    NHA_WAIT(bX, 0);
    tc_fence_after();
    float x[32];
    tmem_ld32(tl + 192 + 32 * half, x);
    if (row == 63) {                                   // x = R = Gend / 2
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        mine_unsafe |= fabsf(x[e]) > 0.5f * kDecayLimit;
        ER[32 * half + e] = exp2f(x[e] * kLog2e);
      }
    }
    if (row < 64) {                                    // s' .* b, in place
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        uint4* at = reinterpret_cast<uint4*>(sm + oSB + sw_off(row, 4 * half + c));
        float sv[8];
        unpack8(*at, sv);
#pragma unroll
        for (int e = 0; e < 8; ++e) sv[e] *= exp2f(-x[8 * c + e] * kLog2e);
        *at = pack8(sv);
      }
    }
#pragma unroll
    for (int e = 0; e < 32; ++e) x[e] = exp2f(x[e] * kLog2e);
    tmem_st32(tl + 192 + 32 * half, reinterpret_cast<const uint32_t*>(x));
    tmem_st_wait();
    fence_async_smem();
  }
  const int unsafe = __syncthreads_or(mine_unsafe);
  if (tid == 0 && z == 0) flags[(size_t)cg * H + h] = unsafe;
  if (unsafe) {
    // the general kernel computes this chunk; the loads and products in flight must be done before the CTA may leave
    if (warp == 8 && lane == 0) {
      NHA_WAIT(bQ, 0);
      for (int i = 0; i < 3; ++i) NHA_WAIT(bFull + i, 0);
      NHA_WAIT(bEmpty + 2, 0);                         // the last commit of the products issued so far
    }
    if (failed) atomicExch(err, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tbase, kTmemCols);
    return;
  }

  if (warp == 8) {
    // ================= load warp: the rest of the slot operands, then the window tiles ===============================
    NHA_WAIT(bKq, 0);                                                          // k' has been read (A = q k'^T)
    if (lane == 0) {
      mbar_expect_tx(&bar[bQ], 32768);
#pragma unroll
      for (int hh = 0; hh < 2; ++hh)
#pragma unroll
        for (int kt = 0; kt < 2; ++kt)
          tma_load_3d(sm + oQS + kt * kQTile + hh * 8192, &maps.qs, 64 * kt, hq0 + hh, tq0 + c0, &bar[bQ]);
    }
    NHA_WAIT(bEmpty + 0, 0);                                                   // q_gsa has been read (QH = q Hk)
    if (lane == 0) {
      mbar_expect_tx(&bar[bFull + 0], 16384);
      tma_load_2d(slot_ptr(0), &maps.hv, 0, (cg * H + h) * M, &bar[bFull + 0]);            // Hv [64][128] as two tiles
      tma_load_2d(slot_ptr(0) + 8192, &maps.hv, 64, (cg * H + h) * M, &bar[bFull + 0]);
    }
    NHA_WAIT(bEmpty + 1, 0);
    load_rows(1, &maps.v, (const bf16*)d.v, c0 - shift, 0, hi);               // v'
    // Window keys: step j into slot 2 (j even) or 1 (j odd) as that slot's fill 2 + j / 2; values: slot 0 (j even, fill
    // 2 + j / 2) or 3 (j odd, fill j / 2).  The two sequences are polled side by side: whichever next load finds its
    // slot free is issued.
    int kn = 0, vn = 0, spins = 0;
    while (kn < nst || vn < nst) {
      bool did = false;
      if (kn < nst) {
        const int slot = (kn & 1) ? 1 : 2;
        // fill f of a slot waits for its release f - 1; keys are fills 1, 2, .. of slot 2 (after Hk) and 2, 3, .. of slot 1
        const int free_ = lane == 0 ? (int)mbar_test(&bar[bEmpty + slot], ((kn & 1) + (kn >> 1)) & 1) : 0;
        if (__shfl_sync(0xffffffffu, free_, 0)) {
          load_rows(slot, &maps.ks, (const bf16*)d.k_swa, (ci - kn) * kChunk, 0, len);
          ++kn;
          did = true;
        }
      }
      if (vn < nst) {
        const int slot = (vn & 1) ? 3 : 0;
        const int f = vn >> 1;                           // fill number on slot 3; on slot 0 it is 2 + f
        int free_ = 0;
        if (lane == 0) {
          if (slot == 0) free_ = mbar_test(&bar[bEmpty + 0], (1 + f) & 1);
          else free_ = f == 0 ? mbar_test(&bar[bX], 0) : mbar_test(&bar[bEmpty + 3], (f - 1) & 1);
        }
        if (__shfl_sync(0xffffffffu, free_, 0)) {
          load_rows(slot, &maps.v, (const bf16*)d.v, (ci - vn) * kChunk, 0, len);
          ++vn;
          did = true;
        }
      }
      if (did) spins = 0;
      else __nanosleep(256);
      if (!did && ++spins > 64 * kPoll) {                     // nothing was released for a very long time: give up
        failed = true;
        break;
      }
    }
  } else if (uwarp == 9) {
    // ================= MMA warp: one elected lane issues everything ==================================================
    {
      auto place = [&](int slot) { return make_desc_lbo(uniform(smem_u32(sm)) + slot_off(slot), 8192); };
      auto wait_full = [&](int slot, int fill) {
        NHA_WAIT(bFull + slot, fill & 1);
        tc_fence_after();
      };
      // D (+)= A B with A from tensor memory: 4 k steps of 16 (8 columns of bf16 pairs each; the second two steps 32 columns
      // on, where the other thread of a row has written its half), B MN-major or K-major
      auto mma_ta = [&](uint32_t dcol, uint32_t acol, uint64_t db, bool b_mn, uint32_t idesc, bool acc) {
#pragma unroll
        for (int ks = 0; ks < 4; ++ks)
          mma_f16_ta(dcol, acol + 8 * (ks & 1) + 32 * (ks >> 1), db + (uint64_t)(b_mn ? ks * 128 : ks * 2), idesc, acc || ks > 0);
      };
      auto s_mma = [&](int j) {          // S_j into accumulator j & 1, then release the keys
        const int slot = (j & 1) ? 1 : 2;
        wait_full(slot, (j & 1) + 1 + (j >> 1));
        const uint32_t su = uniform(smem_u32(sm)), tu = uniform(tbase) + 64 * (j & 1);
        const uint64_t keys = make_desc(su + oRing + (2 - (j & 1)) * kSlot);
        if (elect_one()) {
          mma_run<8, 0>(tu, make_desc(su + oQS), kT16, keys, 8192 >> 4, iK, false);
          commit(&bar[bS + (j & 1)]);
          commit(&bar[bEmpty + slot]);
        }
      };
      uint32_t wph = 0u;
      // G2: X = tril(A) (s' .* b), tril(A) in the first columns of O
      NHA_WAIT(bW, wph); wph ^= 1u;
      tc_fence_after();
      const uint32_t tu = uniform(tbase), uS0 = tu, uS1 = tu + 64, uO = tu + 128;
      const uint64_t dSB = make_desc(uniform(smem_u32(sm)) + oSB);
      if (elect_one()) {
        mma_ta(uS0, uO, dSB, true, iMN, false);
        commit(&bar[bG]);
      }
      // G3: O = (p~ a e^R) Hv over all 128 columns (the two 64-column tiles of Hv are 8192 bytes apart), Bv = (p~ a) SB^T;
      //     p~ a e^R in columns 0-15 and 32-47 of S0, p~ a in columns 16-31 and 48-63
      NHA_WAIT(bW, wph); wph ^= 1u;
      wait_full(0, 1);
      const uint64_t dHv = place(0), dV = place(1);
      if (elect_one()) {
        mma_ta(uO, uS0, dHv, true, iMN128, false);
        mma_ta(uS1, uS0 + 16, dSB, false, iK, false);
        commit(&bar[bG]);
        commit(&bar[bEmpty + 0]);
      }
      NHA_WAIT(bQ, 1);                                   // q_swa
      s_mma(0);                                          // S0 is free once G3 has read the operands in it (in order)
      // G4: O += tril(Bv) v', tril(Bv) in S1
      NHA_WAIT(bW, wph); wph ^= 1u;
      wait_full(1, 1);
      if (elect_one()) {
        mma_ta(uO, uS1, dV, true, iMN128, true);
        commit(&bar[bG]);
        commit(&bar[bEmpty + 1]);
      }
      if (nst > 1) s_mma(1);
      // window steps: O += P~_j V_j with P~_j in S_j, then S_{j+2} into that accumulator
      for (int j = 0; j < nst; ++j) {
        const int b = j & 1;
        NHA_WAIT(bP + b, (j >> 1) & 1);
        const int vslot = b ? 3 : 0;
        wait_full(vslot, b ? (j >> 1) : 2 + (j >> 1));
        const uint32_t to = uniform(tbase) + 128;
        const uint64_t values = place(vslot);
        if (elect_one()) {
          mma_ta(to, to - 128 + 64 * b, values, true, iMN128, true);
          commit(&bar[bPV + b]);
          commit(&bar[bEmpty + vslot]);
        }
        if (j + 2 < nst) s_mma(j + 2);
      }
    }
  } else {
    // ================= softmax group: two threads per row ===========================================================
    const int tk = row & 63, th = row >> 6;
    const int pos = c0 + tk;
    const bool in_seq = pos < len && (th == 0 || two);
    const int hq = hq0 + th;
    const uint32_t th32 = tl + 32 * half;                          // this thread's half of S0; of S1 at +64
    const int klo = in_seq ? (wl < 0 ? 0 : max(0, pos - wl)) : (1 << 30);
    const unsigned kspan = in_seq ? (unsigned)(pos - klo) : 0u;
    const float sc2 = d.scale * kLog2e;
    const float lag = NG == 1 ? 0.f : kRaise;                      // how far a window logit may exceed the reference of its row
    uint32_t gph = 0u;
    // one lane of a warp polls a barrier, the others wait at the warp barrier: far fewer shared-memory polls
#define NHA_WAIT_WARP(idx_, par_)                        \
  do {                                                   \
    if (lane == 0) NHA_WAIT(idx_, par_);                 \
    __syncwarp();                                        \
  } while (0)
    // the two warps that share 32 rows; the second form also tells whether a thread of either has `p`
    const int pairbar = 1 + (warp & 3);
    auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(pairbar) : "memory"); };
    auto pair_any = [&](bool p) {
      uint32_t any;
      asm volatile(
          "{\n.reg .pred p, q;\nsetp.ne.u32 p, %1, 0;\nbarrier.cta.red.or.aligned.pred q, %2, 64, p;\nselp.u32 %0, 1, 0, q;\n}\n"
          : "=r"(any)
          : "r"((uint32_t)p), "r"(pairbar)
          : "memory");
      return any != 0;
    };
    // the partner's value of x (every thread of both warps calls it; a pair barrier lies between two calls)
    auto partner = [&](float x) {
      xch[128 * half + row] = x;
      pair_sync();
      return xch[128 * (half ^ 1) + row];
    };
    // this thread's half of its row of tril of a [128][64] accumulator (token tk keeps columns i <= tk) as bf16 pairs
    auto tril_to = [&](uint32_t src_col, uint32_t dst_col) {
      float v[32];
      tmem_ld32(th32 + src_col, v);
      uint32_t pk[16];
      const int c = 32 * half;
#pragma unroll
      for (int e = 0; e < 16; ++e) pk[e] = bf16_pair(c + 2 * e <= tk ? v[2 * e] : 0.f, c + 2 * e + 1 <= tk ? v[2 * e + 1] : 0.f);
      tmem_st16(th32 + dst_col, pk);
      tmem_st_wait();
    };
    auto hand_over = [&](int b_) {
      tc_fence_before();
      mbar_arrive(&bar[b_]);
    };
    // G1 -> tril(A) into the first columns of O (not used before G3)
    NHA_WAIT_WARP(bG, gph); gph ^= 1u;
    tc_fence_after();
    tril_to(0, 128);
    hand_over(bW);
    // G2 -> slot logits, p~, operands
    NHA_WAIT_WARP(bG, gph); gph ^= 1u;
    tc_fence_after();
    float mg, lg0;
    {
      float ok[32];
      tmem_ld32(th32 + 64, ok);
      float m4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int q2 = 0; q2 < 2; ++q2) {
        float x[16], a[16];
        tmem_ld16(th32 + 16 * q2, x);
        tmem_ld16(th32 + 192 + 16 * q2, a);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 e4 = *reinterpret_cast<const float4*>(ER + 32 * half + 16 * q2 + 4 * q);
          const float er[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int k = 16 * q2 + 4 * q + e;
            ok[k] = d.scale * a[4 * q + e] * (er[e] * ok[k] + x[4 * q + e]);
            m4[e] = fmaxf(m4[e], ok[k]);
          }
        }
      }
      mg = fmaxf(fmaxf(m4[0], m4[1]), fmaxf(m4[2], m4[3]));
      mg = fmaxf(mg, partner(mg));
      const float nmg = -mg * kLog2e;
      float l4[4] = {0.f, 0.f, 0.f, 0.f};
      // p~ a e^R -> the first 16 columns of this thread's half of S0, p~ a -> the other 16 (X and QH are in registers by now)
#pragma unroll
      for (int q2 = 0; q2 < 2; ++q2) {
        float a[16];
        tmem_ld16(th32 + 192 + 16 * q2, a);
        uint32_t pg[8], pa[8];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float4 e4 = *reinterpret_cast<const float4*>(ER + 32 * half + 16 * q2 + 4 * q);
          const int k = 16 * q2 + 4 * q;
          const float p0 = exp2f(fmaf(ok[k], kLog2e, nmg)), p1 = exp2f(fmaf(ok[k + 1], kLog2e, nmg));
          const float p2 = exp2f(fmaf(ok[k + 2], kLog2e, nmg)), p3 = exp2f(fmaf(ok[k + 3], kLog2e, nmg));
          l4[0] += p0; l4[1] += p1; l4[2] += p2; l4[3] += p3;
          const float a0 = in_seq ? p0 * a[4 * q] : 0.f, a1 = in_seq ? p1 * a[4 * q + 1] : 0.f;
          const float a2 = in_seq ? p2 * a[4 * q + 2] : 0.f, a3 = in_seq ? p3 * a[4 * q + 3] : 0.f;
          pa[2 * q] = bf16_pair(a0, a1);
          pa[2 * q + 1] = bf16_pair(a2, a3);
          pg[2 * q] = bf16_pair(a0 * e4.x, a1 * e4.y);
          pg[2 * q + 1] = bf16_pair(a2 * e4.z, a3 * e4.w);
        }
        tmem_st8(th32 + 8 * q2, pg);
        tmem_st8(th32 + 16 + 8 * q2, pa);
      }
      tmem_st_wait();
      lg0 = (l4[0] + l4[1]) + (l4[2] + l4[3]);
    }
    hand_over(bW);
    // G3 -> tril(Bv) over the columns of S1 it is read from
    NHA_WAIT_WARP(bG, gph); gph ^= 1u;
    tc_fence_after();
    tril_to(64, 64);
    hand_over(bW);
    // G4
    NHA_WAIT_WARP(bG, gph); gph ^= 1u;
    tc_fence_after();

    float mref = mg;            // reference of the unnormalised probabilities of this row (both threads hold the same)
    float lgs = lg0;            // slot sum of this thread's half, in units of exp(-mref)
    float ls = 0.f;             // window sum, likewise
    // P~ V of step j has completed (steps alternate between two barriers; a wait names a phase whose predecessor was seen)
    auto wait_pv = [&](int j) { NHA_WAIT_WARP(bPV + (j & 1), (j >> 1) & 1); };
    for (int j = 0; j < nst; ++j) {
      const int b = j & 1;
      NHA_WAIT_WARP(bS + b, (j >> 1) & 1);
      tc_fence_after();
      float s[32];
      tmem_ld32(th32 + 64 * b, s);
      const int kb = (ci - j) * kChunk;
      const int off = kb - klo + 32 * half;
      // the diagonal tile (causal edge) and tiles that reach below the oldest visible key of the chunk's last row need
      // the per-element test; every row of the chunk sees all keys of the tiles in between
      const bool masked = j == 0 || (wl >= 0 && kb < c0 + kChunk - 1 - wl) || c0 + kChunk > len;
      {
        if (masked) {
#pragma unroll
          for (int e = 0; e < 32; ++e) s[e] = (unsigned)(off + e) <= kspan ? s[e] : -INFINITY;
        }
        float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          m0 = max3(m0, s[e], s[e + 1]);
          m1 = max3(m1, s[e + 2], s[e + 3]);
        }
        float mc = d.scale * fmaxf(m0, m1);
        if (pair_any(mc > mref + lag)) {
          mc = fmaxf(mc, partner(mc));
          float f = 1.f;
          if (mc > mref + lag) {
            f = __expf(mref - mc);
            mref = mc;
          }
          // rescale this thread's half of its row of O: everything issued on O so far must have completed
          if (j > 0) wait_pv(j - 1);
          tc_fence_after();
#pragma unroll 1
          for (int q4 = 0; q4 < 4; ++q4) {
            float ov[16];
            tmem_ld16(tl + 128 + 64 * half + 16 * q4, ov);
#pragma unroll
            for (int e = 0; e < 16; ++e) ov[e] *= f;
            tmem_st16(tl + 128 + 64 * half + 16 * q4, reinterpret_cast<const uint32_t*>(ov));
          }
          tmem_st_wait();
          lgs *= f;
          ls *= f;
        }
      }
      const float nm = -mref * kLog2e;
      const uint64_t sc2p = pack2(sc2, sc2), nmp = pack2(nm, nm);
      uint64_t l0 = pack2(0.f, 0.f), l1 = l0;
      uint32_t pk[16];                                  // P~_j as bf16 pairs: the A operand of the value product
#pragma unroll
      for (int e = 0; e < 32; e += 4) {
        float a0, a1, a2, a3;
        unpack2(ffma2(pack2(s[e], s[e + 1]), sc2p, nmp), a0, a1);
        unpack2(ffma2(pack2(s[e + 2], s[e + 3]), sc2p, nmp), a2, a3);
        a0 = exp2f(a0); a1 = exp2f(a1); a2 = exp2f(a2); a3 = exp2f(a3);
        l0 = fadd2(l0, pack2(a0, a1));
        l1 = fadd2(l1, pack2(a2, a3));
        pk[e / 2] = bf16_pair(a0, a1);
        pk[e / 2 + 1] = bf16_pair(a2, a3);
      }
      tmem_st16(th32 + 64 * b, pk);
      tmem_st_wait();
      {
        float a0, a1;
        unpack2(fadd2(l0, l1), a0, a1);
        ls += a0 + a1;
      }
      // Step j - 2 on this step's barrier: complete already, since S_j was issued behind it.  The value product of step j - 1
      // may still run: nothing here waits for it.
      if (j > 1) wait_pv(j - 2);
      tc_fence_before();
      mbar_arrive(&bar[bP + b]);
    }
    wait_pv(nst - 1);
    tc_fence_after();
    ls += partner(ls);
    pair_sync();
    lgs += partner(lgs);
    pair_sync();
    lg0 += partner(lg0);
    const float lsum = lgs + ls;
    const float inv = lsum > 0.f ? 1.f / lsum : 0.f;
    if (in_seq && half == 0) {
      d.lse_gsa[(size_t)(tq0 + pos) * HQ + hq] = mg + __logf(lg0);
      d.lse_swa[(size_t)(tq0 + pos) * HQ + hq] = mref + __logf(ls);
    }
    // Output rows leave through shared memory: a thread holds half of a row (128 bytes), and stores of 32 lanes to 32
    // rows 8 KB apart would cost one memory transaction per lane.  The rows are staged in the q_swa tiles (dead: every
    // S product has completed) with the 16-byte pieces of a row rotated by the row index (no bank conflicts), and each
    // of the two warps then writes 16 of their 32 rows, two whole rows per instruction.
    unsigned char* stage = sm + oQS + (size_t)((warp & 3) * 32) * 256;     // the 32 rows of this pair of warps
#pragma unroll 1
    for (int q2 = 0; q2 < 2; ++q2) {
      float ov[32];
      tmem_ld32(tl + 128 + 64 * half + 32 * q2, ov);
#pragma unroll
      for (int e = 0; e < 32; ++e) ov[e] *= inv;
#pragma unroll
      for (int c8 = 0; c8 < 4; ++c8)
        *reinterpret_cast<uint4*>(stage + lane * 256 + (((8 * half + 4 * q2 + c8) ^ (lane & 15)) << 4)) = pack8(ov + 8 * c8);
    }
    pair_sync();
    {
      const int hl = lane >> 4, c = lane & 15;            // two rows per instruction, 16 pieces of 16 bytes per row
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int r = 16 * half + 2 * i + hl;             // row of this pair of warps
        const int rr = (warp & 3) * 32 + r;               // row of the tile
        const int p2 = c0 + (rr & 63);
        if (p2 < len && (rr < 64 || two)) {
          const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 256 + ((c ^ (r & 15)) << 4));
          bf16* dst = (bf16*)d.o + ((size_t)(tq0 + p2) * HQ + hq0 + (rr >> 6)) * D + 8 * c;
          *reinterpret_cast<uint4*>(dst) = v;
        }
      }
    }
#undef NHA_WAIT_WARP
  }
#undef NHA_WAIT
  if (failed) atomicExch(err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tbase, kTmemCols);
}

// Any number of query heads per kv head: an odd group's last tile is half empty, and so is every tile of a group of one,
// where two 64-row CTAs of nha_fwd_umma_kernel would do the same work - slower all the same (B4 T2048 H16 W64, whole
// prefill: 195 us here, 301 us there; seven heads a group, B2 T2048 W512: 110 us here, 1570 us with the general kernel).
bool fwd_pipe_supported(const nha_chunk_desc* d) {
  if (d->K != 128 || d->V != 128 || d->M != 64 || !(d->scale > 0.f)) return false;
  const char* off = getenv("NHA_B200_NO_PIPE");
  return !(off && off[0] == '1');
}

// Launches the pipelined output pass; NHA_ERR_UNSUPPORTED when the tensor maps cannot be made (the caller then takes
// the non-pipelined tensor-memory kernel).
int fwd_pipe_launch(const nha_chunk_desc* d, int* flags, int* err, cudaStream_t cs, bool early) {
  using namespace pipe;
  const int NCB = (int)nha_chunk_count_bound(d->Ttot, d->N);
  PipeMaps maps;
  memset(&maps, 0, sizeof(maps));
  const bool ok = make_map_rows_heads(&maps.qg, d->q_gsa, d->Ttot - d->q_offset, d->HQ, D) &&
                  make_map_rows_heads(&maps.qs, d->q_swa, d->Ttot - d->q_offset, d->HQ, D) &&
                  make_map_rows_heads(&maps.kg, d->k_gsa, d->Ttot, d->H, D) &&
                  make_map_rows_heads(&maps.ks, d->k_swa, d->Ttot, d->H, D) &&
                  make_map_rows_heads(&maps.v, d->v, d->Ttot, d->H, D) && make_map_rows_heads(&maps.g, d->g, d->Ttot, d->H, M) &&
                  make_map_rows_heads(&maps.s, d->s, d->Ttot, d->H, M) &&
                  make_map_matrix(&maps.hk, d->hk_chunks, (int64_t)NCB * d->H * D, M, 128) &&
                  make_map_matrix(&maps.hv, d->hv_chunks, (int64_t)NCB * d->H * M, D, 64);
  if (!ok) return NHA_ERR_UNSUPPORTED;
  cudaError_t e = set_max_smem((const void*)nha_fwd_pipe_kernel, total);
  if (e != cudaSuccess) return record_cuda_error(e);
  launch_after(nha_fwd_pipe_kernel, dim3((unsigned)(NCB * d->H * ((d->HQ / d->H + 1) / 2))), kThreads, total, cs, *d, flags, err, maps, early ? 1 : 0);
  return check_launch();
}

}  // namespace nha
