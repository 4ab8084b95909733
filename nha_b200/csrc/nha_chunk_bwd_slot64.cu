// Backward of the chunked NHA operator, slot branch, head dim 64: dq_gsa, dk_gsa, the slot part of dv, ds, dg, and the row
// statistics that the window branch needs, in one kernel.
//
// One CTA = a run of consecutive chunks of one kv head, walked from the last chunk to the first with the state gradient on chip
// (tensor memory in fp32; with several query heads per kv head in a scratch row of L2).  Per chunk and query head:
//     x = G - Gend / 2,  A = q k'^T,  Av = do v'^T
//     Z = tril(A) SB + q Hk',   Y = tril(Av) SB + do Hv'                 -> p, dz, gate terms (ok = scale a Z, dp = a Y)
//     E = za SB^T,  Bv = pa SB^T,  dS = tril(A)^T za + tril(Av)^T pa
//     dq = za Hk'^T,  LK = q^T za,  LV = pa^T do,  dS += k' DK' + v' DV'^T
//     dq += tril(E) k',  dk' = tril(E)^T q + SB DK'^T,  dv' = tril(Bv)^T do + SB DV'
// with SB = s' exp(R - G), a = exp(G - R), za = scale dz a, pa = p a.  The reference R of a slot is the power of two next to
// exp(Gend / 2), so that the factors exp(R) are exact in bf16: Hk' = Hk exp(R) and Hv' are the stored states themselves with
// other exponents, and nothing else has to be scaled in front of a product.  DK' = DK exp(Gend - R) is rounded once, from fp32.
//     ds' = dS / a,   DK(start) = exp(Gend) DK(end) + exp(R) LK,   dg = reverse running sum of the gate terms - s' ds' plus the
//     carry <DK, hk> + <DV, hv> at the chunk's end (rebuilt at every chunk: a running sum loses dg to cancellation).
//
// A run has to know the state gradient at its end.  Where it ends with a sequence that is the caller's (or zero); otherwise it
// comes from the scan over the terms LK, LV of every chunk (TERMS: the same kernel, one chunk a CTA, the first two rounds).  Both
// ways give the same bits: the walk updates the state gradient by the scan's arithmetic, element by element in fp32.  (All but the carry of dg where a
// chunk comes within about a nat of the limit below: products with its start state, which the walk has scaled by exp(R), may then underflow.)
//
// A chunk that decays by more than 140 nats (the forward's flag) cannot have one reference.  It takes R = 0 and forms the sums
// over pairs of rows directly in fp32 (steep_*), exact for any gate, inside the same walk.  What bounds that is the sums' arithmetic: 64 x 64 / 2 pairs of
// rows by 64 slots, five times.  Backward, us, B x 2048 tokens, 16 heads, chunks with one steep slot or all of them: general kernels beside
// the former three passes | sums of each element by itself, its gates read for each | blocks of four rows with running products:
// B 16: 0.2 % 1262 | 2622 | 933, 1 % 1260 | 3600 | 1025, 10 % 2303 | 11371 | 1422, all 9208 | 51862 | 3346 (none: 982 | 540 | 541);
// B 2: 1 % 434 | 1769 | 256, all 2222 | 10774 | 592;  4 x 1999 tokens, 16 heads on 4: 1 % 948 | 5717 | 551, all 5091 | 20365 | 1043;
// 256 tokens, 4 heads, 32 slots: all 342 | 3171 | 338.
//
// What bounds it: the chain of a chunk, five rounds of products with the element-wise work between them, about 2000 instructions a warp.  With two
// CTAs of eight warps on an SM the issue slots are 38 % busy, the tensor cores 26 %, HBM a quarter to a third; a warp waits, per instruction
// issued, 1.6 for tensor memory or a global load, 1.6 for shared memory and shuffles, 1.2 at barriers.  A body beyond 64 KB of
// code waits for its instructions (2.4 cycles for each at 96-128 KB, 6 at 192), which is why rare cases are bodies or functions of their own.  16 warps to a CTA, half as much
// work for each, were slower (490 us against 384 of that build): the same chain, and more code fetches.
// Measured, B16 T2048 H16 M64: query-row pass, state-gradient scan and key-row pass of this branch, three kernels that hand dz, p, the terms and
// the state gradients to each other through memory, 810 us with the rows' window part (about 50); this kernel 335 us, and nothing in between but delta, L
// and the slot part of dv.  Runs that cut sequences pay the terms and the scan: 32768 packed tokens, longest sequence 8192: 340 us behind 160 + 75.
// One reference that is a power of two, the states as they are stored, and products issued by an elected lane (see elect_one()) took
// the walk from 384 to 335 us; dz, p and SB rounded the same way on both sides of the gate terms took dg's error against 64 bits from
// 2.07e-2 to 4.3e-3 at no cost.
//
// Replaces, with nha_chunk_bwd_win64.cu, ChunkNativeHybridAttentionFunction.backward (nha_fla/ops/nha/chunk.py:491-564).
#include <string.h>

#include <algorithm>

#include "nha_bwd_common.cuh"
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

// Tensor maps of the call's tensors (this GPU's own memory).  A chunk whose 64 rows lie inside its sequence, shifted or not, is moved by
// TMA: warp i asks for tile i of `in` and for `out` i - 1.  Others (ragged ends, rows in front of a sequence) are copied piece by piece with
// zero fill.  use == 0: all chunks are (fewer than 64 slots, or no tensor maps).
enum { kInQ, kInDO, kInK, kInS, kInG, kInV, kInHk, kInHv, kIns };
struct SlotMaps {
  CUtensorMap in[kIns], out[4], o;
  int use;
};

// Tiles.  g comes into A's place and the signs of the running sum into B's (both are read by the first products alone); tril(E),
// tril(Bv) take A and B over; results are staged in ZA, PA, DK, DV.  TERMS with one head: ZA, PA over k', v'.
template <bool ONE, bool TERMS>
struct SlotSm {
  static constexpr int tQ = 0, tDO = 1, tK = 2, tV = 3, tHk = 4, tHv = 5, tSB = 6, tA = 7, tB = 8;
  static constexpr int tZA = TERMS && ONE ? tK : 9, tPA = TERMS && ONE ? tV : 10, tDK = 11, tDV = 12;
  static constexpr int kTiles = TERMS ? (ONE ? 9 : 11) : 13;
  static constexpr int oTab = kTiles * kTile;                   // fp32 [5][64]: see kTab*
  static constexpr int oRow = oTab + (TERMS ? 2 : 5) * 256;     // fp32 [4][64] delta, -Lj, -lse_gsa (log2 units), d_lse_gsa
  static constexpr int oTot = oRow + 4 * 256;                   // fp32 [64][4 quarters] totals of the gate terms
  static constexpr int oPart = oTot + (TERMS ? 0 : 4 * 256);                  // fp32 [2][64][4 quarters, 2 halves, -] dot products of the carry
  static constexpr int oBar = oPart + (TERMS ? 0 : 16 * 256);
  static constexpr int oRec = oBar + 64;
  static constexpr int total = oRec + 128 + 1024;
  static constexpr int kCtas = TERMS && ONE ? 3 : 2;
  // accumulators: four of a head, the chunk's terms, and the state gradient (one head) or dk', dv' (summed over the heads)
  static constexpr uint32_t cA = 0, cB = kOtherLanes, cC = 64, cD = 64 + kOtherLanes;
  static constexpr uint32_t cLK = TERMS && ONE ? cA : 128, cLV = TERMS && ONE ? cB : 128 + kOtherLanes;
  static constexpr uint32_t cSK = 192, cSV = 192 + kOtherLanes;
  static constexpr uint32_t cOK = ONE ? cA : cSK, cOV = ONE ? cB : cSV;
  static constexpr int kTmemCols = TERMS && ONE ? 128 : 256;
  static_assert(total <= (kCtas == 3 ? 75 : 113) * 1024, "CTAs per SM");
};
enum { kTabP = 0, kTabC = 64, kTabIP = 128, kTabF = 192, kTabD = 256 };   // 2^n, R log2e - n; 2^-n, F, exp(Gend)  (R = Gend / 2)

// ---- steep chunks ---------------------------------------------------------------------------------------------------------
// The chunk's rows of g: row r at g + r * pitch if lo <= r < hi, or nothing (g = 0).  Handed on by value: the kernel's stack does not fit the L1 cache
// that two CTAs' shared memory leaves, and a field read from there takes as long as the rows themselves.
struct SteepCtx {
  const bf16* g;      // row 0, this head
  int pitch, lo, hi, M;
};
__device__ __forceinline__ const bf16* steep_row(const SteepCtx& c, int r) { return r >= c.lo && r < c.hi ? c.g + (int64_t)r * c.pitch : nullptr; }
// In these functions a warp has two blocks of four rows, one as far from the chunk's start as the other from its end (so that all have the
// same number of blocks in front of theirs, and behind), and a lane two slots.  Decays are products of exp(g), never differences of sums (a gate
// of minus infinity leaves no difference of infinities): from a row outside the block the factors up to the block's edge, one run of products
// for all four rows, times those inside it.
__device__ __forceinline__ float2 steep_mul(float2 x, float2 y) { return make_float2(x.x * y.x, x.y * y.y); }
__device__ __forceinline__ float2 steep_fma(float a, float2 x, float2 y) { return make_float2(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y)); }
// g of rows i .. i + 3, slots m and m + 1 (rows outside the chunk as well: those of the next block are asked for while a block is worked on), and exp of it
__device__ __forceinline__ void steep_gates(const SteepCtx& c, int i, int m, uint32_t (&g)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bf16* gr = m < c.M ? steep_row(c, i + k) : nullptr;
    g[k] = gr ? *reinterpret_cast<const uint32_t*>(gr + m) : 0u;
  }
}
__device__ __forceinline__ void steep_factors(const uint32_t (&g)[4], float2 (&f)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float2 x = pair_f32(g[k]);
    f[k] = make_float2(__expf(x.x), __expf(x.y));
  }
}
// two neighbouring elements, and four, of a row of a tile
__device__ __forceinline__ float2 steep_pair(const unsigned char* t, int r, int m) { return pair_f32(*reinterpret_cast<const uint32_t*>(t + sw_off(r, m >> 3) + 2 * (m & 7))); }
__device__ __forceinline__ void steep_quad(const unsigned char* t, int r, int i, float (&v)[4]) {
  const uint2 x = *reinterpret_cast<const uint2*>(t + sw_off(r, i >> 3) + 2 * (i & 7));
  const float2 a = pair_f32(x.x), b = pair_f32(x.y);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void steep_put(unsigned char* t, int r, int m, float2 v) { *reinterpret_cast<uint32_t*>(t + sw_off(r, m >> 3) + 2 * (m & 7)) = pair_bf16(v.x, v.y); }
// element pair of an fp32 [64][64] array in two tiles, turned so that a warp's accumulator fragments and its rows both are free of conflicts
__device__ __forceinline__ float2* steep_at(unsigned char* stage, int r, int m) { return reinterpret_cast<float2*>(stage) + r * 32 + ((m >> 1) ^ ((r & 7) << 2)); }
__device__ __forceinline__ void steep_stage_in(unsigned char* stage, uint32_t acc, int r0, int cbase) {
  float v[16];
  frag_ld(acc, v);
#pragma unroll
  for (int k = 0; k < 16; k += 2) *steep_at(stage, r0 + 4 * (k & 2), cbase + 2 * (k & 12)) = make_float2(v[k], v[k + 1]);
  __syncthreads();
}
__device__ __forceinline__ void steep_stage_out(unsigned char* stage, uint32_t acc, int r0, int cbase) {
  float v[16];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 16; k += 2) {
    const float2 x = *steep_at(stage, r0 + 4 * (k & 2), cbase + 2 * (k & 12));
    v[k] = x.x;
    v[k + 1] = x.y;
  }
  frag_st(acc, v);
  __syncthreads();
}
// The rows' products with a start state, in the accumulator, become what the whole chunk gives: times exp(G), plus sum_{i<=t} A[t,i] s_i[m]
// exp(G_t - G_i) from the tiles of tril(q k'^T) (or tril(do v'^T)) and s'.  Through the two tiles at `stage`.
__device__ __noinline__ void steep_rows(const SteepCtx c, int A, int S, int stage_tile, uint32_t acc, int r0, int cbase) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  const unsigned char *tA = sm + A * kTile, *tS = sm + S * kTile;
  unsigned char* stage = sm + stage_tile * kTile;
  steep_stage_in(stage, acc, r0, cbase);
  const int warp = threadIdx.x >> 5, m = 2 * (threadIdx.x & 31);
#pragma unroll 1
  for (int x = 0; x < 2; ++x) {
    const int b = x ? 15 - warp : warp;
    float2 v[4], u = make_float2(1.f, 1.f), f[4];
    uint32_t g[4], own[4];
    steep_gates(c, 4 * b - 4, m, g);
    steep_gates(c, 4 * b, m, own);
#pragma unroll
    for (int t = 0; t < 4; ++t) v[t] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int ib = b - 1; ib >= 0; --ib) {
      steep_factors(g, f);
      steep_gates(c, 4 * ib - 4, m, g);
      float w[4][4];
#pragma unroll
      for (int t = 0; t < 4; ++t) steep_quad(tA, 4 * b + t, 4 * ib, w[t]);
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        const float2 sv = steep_mul(steep_pair(tS, 4 * ib + i, m), u);
#pragma unroll
        for (int t = 0; t < 4; ++t) v[t] = steep_fma(w[t][i], sv, v[t]);
        u = steep_mul(u, f[i]);
      }
    }
    steep_factors(own, f);
    float2 sv[4], pr = make_float2(1.f, 1.f);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      float w[4];
      steep_quad(tA, 4 * b + t, 4 * b, w);
      pr = steep_mul(pr, f[t]);
#pragma unroll
      for (int i = 0; i < t; ++i) sv[i] = steep_mul(sv[i], f[t]);
      sv[t] = steep_pair(tS, 4 * b + t, m);
      float2* at = steep_at(stage, 4 * b + t, m);
      const float2 h = steep_mul(*at, u);
      float2 y = steep_mul(make_float2(v[t].x + h.x, v[t].y + h.y), pr);
#pragma unroll
      for (int i = 0; i <= t; ++i) y = steep_fma(w[i], sv[i], y);
      *at = y;
    }
  }
  steep_stage_out(stage, acc, r0, cbase);
}
// dS[i,m] (+)= sum_{t>=i} (A[t,i] dz_t[m] + Av[t,i] p_t[m]) exp(G_t - G_i) into scratch
__device__ __noinline__ void steep_keys(const SteepCtx c, int A, int Av, int dz, int p, float* ds, int64_t dpitch, bool add) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  const unsigned char *tA = sm + A * kTile, *tAv = sm + Av * kTile, *tz = sm + dz * kTile, *tp = sm + p * kTile;
  const int warp = threadIdx.x >> 5, m = 2 * (threadIdx.x & 31);
#pragma unroll 1
  for (int x = 0; x < 2; ++x) {
    const int b = x ? 15 - warp : warp;
    float2 v[4], u = make_float2(1.f, 1.f), f[4];
    uint32_t g[4], own[4];
    steep_gates(c, 4 * b + 4, m, g);
    steep_gates(c, 4 * b, m, own);
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = make_float2(0.f, 0.f);
#pragma unroll 1
    for (int tb = b + 1; tb < 16; ++tb) {
      steep_factors(g, f);
      steep_gates(c, 4 * tb + 4, m, g);
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        float wa[4], wv[4];
        steep_quad(tA, 4 * tb + t, 4 * b, wa);
        steep_quad(tAv, 4 * tb + t, 4 * b, wv);
        u = steep_mul(u, f[t]);
        const float2 zv = steep_mul(steep_pair(tz, 4 * tb + t, m), u), pv = steep_mul(steep_pair(tp, 4 * tb + t, m), u);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = steep_fma(wv[i], pv, steep_fma(wa[i], zv, v[i]));
      }
    }
    steep_factors(own, f);
    // from the block's last row to its first: what the rows behind have left for row t is carried on to the rows in front of it
#pragma unroll
    for (int t = 3; t >= 0; --t) {
      float wa[4], wv[4];
      steep_quad(tA, 4 * b + t, 4 * b, wa);
      steep_quad(tAv, 4 * b + t, 4 * b, wv);
      const float2 zv = steep_pair(tz, 4 * b + t, m), pv = steep_pair(tp, 4 * b + t, m);
#pragma unroll
      for (int i = 0; i <= t; ++i) v[i] = steep_fma(wv[i], pv, steep_fma(wa[i], zv, v[i]));
#pragma unroll
      for (int i = 0; i < t; ++i) v[i] = steep_mul(v[i], f[t]);
      if (m < c.M && 4 * b + t < c.hi) {
        float2* o = reinterpret_cast<float2*>(ds + (int64_t)(4 * b + t) * dpitch + m);
        const float2 old = add ? *o : make_float2(0.f, 0.f);
        *o = make_float2(old.x + v[t].x, old.y + v[t].y);
      }
    }
  }
}
// The tiles of dz and p become dz exp(G) and p exp(G).  PAIRS: before that E[t,i] = sum_m dz_t[m] s_i[m] exp(G_t - G_i) and Bv likewise from p,
// into the tiles E and Bv (zeros above the diagonal).
template <bool PAIRS>
__device__ __noinline__ void steep_pairs(const SteepCtx c, int E, int Bv, int dz, int p, int S) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  const unsigned char* tS = sm + S * kTile;
  unsigned char *tz = sm + dz * kTile, *tp = sm + p * kTile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, m = 2 * lane;
  // this lane's element of the 32 sums of a block: E or Bv, row, column
  unsigned char* const te = sm + (lane & 16 ? Bv : E) * kTile;
  const int lt = (lane >> 2) & 3, li = lane & 3;
  auto sums_out = [&](float (&v)[32], int r, int i) {
#pragma unroll
    for (int n = 16; n > 0; n >>= 1) {
      const bool up = lane & n;
#pragma unroll
      for (int k = 0; k < n; ++k) {
        const float keep = up ? v[k + n] : v[k], give = up ? v[k] : v[k + n];
        v[k] = keep + __shfl_xor_sync(0xffffffffu, give, n);
      }
    }
    *reinterpret_cast<bf16*>(te + sw_off(r + lt, i >> 3) + 2 * ((i & 7) + li)) = f2bf(v[0]);
  };
#pragma unroll 1
  for (int x = 0; x < 2; ++x) {
    const int b = x ? 15 - warp : warp;
    float2 zv[4], pv[4], f[4], u = make_float2(1.f, 1.f);
    uint32_t g[4];
    steep_gates(c, 4 * b, m, g);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      zv[t] = steep_pair(tz, 4 * b + t, m);
      pv[t] = steep_pair(tp, 4 * b + t, m);
    }
    steep_factors(g, f);
    steep_gates(c, 4 * b - 4, m, g);
    if (PAIRS) {
      float v[32];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float2 sv = steep_pair(tS, 4 * b + i, m);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (t > i) sv = steep_mul(sv, f[t]);
          v[4 * t + i] = t >= i ? fmaf(zv[t].x, sv.x, zv[t].y * sv.y) : 0.f;
          v[16 + 4 * t + i] = t >= i ? fmaf(pv[t].x, sv.x, pv[t].y * sv.y) : 0.f;
        }
      }
      sums_out(v, 4 * b, 4 * b);
      for (int k = lane; k < 8 * (15 - b); k += 32) {          // the blocks above the diagonal
        const int i = 4 * (b + 1 + (k >> 3)), r = 4 * b + (k & 3);
        *reinterpret_cast<uint2*>(sm + (k & 4 ? Bv : E) * kTile + sw_off(r, i >> 3) + 2 * (i & 7)) = make_uint2(0u, 0u);
      }
    }
    float2 pr = make_float2(1.f, 1.f);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      pr = steep_mul(pr, f[t]);
      zv[t] = steep_mul(zv[t], pr);
      pv[t] = steep_mul(pv[t], pr);
    }
#pragma unroll 1
    for (int ib = b - 1; ib >= 0; --ib) {
      steep_factors(g, f);
      steep_gates(c, 4 * ib - 4, m, g);
      float v[32];
#pragma unroll
      for (int i = 3; i >= 0; --i) {
        if (PAIRS) {
          const float2 sv = steep_mul(steep_pair(tS, 4 * ib + i, m), u);
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            v[4 * t + i] = fmaf(zv[t].x, sv.x, zv[t].y * sv.y);
            v[16 + 4 * t + i] = fmaf(pv[t].x, sv.x, pv[t].y * sv.y);
          }
        }
        u = steep_mul(u, f[i]);
      }
      if (PAIRS) sums_out(v, 4 * b, 4 * ib);
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      steep_put(tz, 4 * b + t, m, steep_mul(zv[t], u));
      steep_put(tp, 4 * b + t, m, steep_mul(pv[t], u));
    }
  }
}
// With the factors exp(Gend - G): the tile of s' times them (stage_tile < 0), or the products with the state gradient at the chunk's end, in the
// accumulator, times them plus dS from scratch: ds', through the two tiles at `stage`.
__device__ __noinline__ void steep_ends(const SteepCtx c, int S, int stage_tile, uint32_t acc, const float* ds, int64_t dpitch, int r0, int cbase) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  unsigned char *tS = sm + S * kTile, *stage = sm + stage_tile * kTile;
  const bool tile = stage_tile < 0;
  if (!tile) steep_stage_in(stage, acc, r0, cbase);
  const int warp = threadIdx.x >> 5, m = 2 * (threadIdx.x & 31);
#pragma unroll 1
  for (int x = 0; x < 2; ++x) {
    const int b = x ? 15 - warp : warp;
    float2 u = make_float2(1.f, 1.f), f[4];
    uint32_t g[4];
    steep_gates(c, 60, m, g);
#pragma unroll 1
    for (int tb = 15; tb >= b; --tb) {
      steep_factors(g, f);
      steep_gates(c, 4 * tb - 4, m, g);
#pragma unroll
      for (int t = 3; t >= 0; --t) {
        if (tb == b) {
          const int r = 4 * b + t;
          if (tile) {
            steep_put(tS, r, m, steep_mul(steep_pair(tS, r, m), u));
          } else {
            float2* at = steep_at(stage, r, m);
            const float2 d = m < c.M && r < c.hi ? *reinterpret_cast<const float2*>(ds + (int64_t)r * dpitch + m) : make_float2(0.f, 0.f);
            const float2 h = steep_mul(*at, u);
            *at = make_float2(h.x + d.x, h.y + d.y);
          }
        }
        u = steep_mul(u, f[t]);
      }
    }
  }
  if (!tile) steep_stage_out(stage, acc, r0, cbase);
}

// ---- rows that are not whole tiles ------------------------------------------------------------------------------------------
// [64][64] tile <- rows row .. row + 63 of a sequence's tensor (p: the sequence's first row), zeros outside [0, hi) and behind `width` columns
__device__ void rows_in(unsigned char* t, const bf16* p, int64_t pitch, int width, int row, int hi, int tid, int nt) {
  const int c = tid & 7;
  const bool cok = 8 * c < width;
  for (int r = tid >> 3; r < kChunk; r += nt >> 3) {
    const bool ok = cok && row + r >= 0 && row + r < hi;
    cp16(t + sw_off(r, c), p + (ok ? (int64_t)(row + r) * pitch + 8 * c : 0), ok);
  }
}
// rows [lo, hi) of a tile to `width` columns of a tensor
__device__ void rows_out(const unsigned char* t, bf16* base, int64_t pitch, int width, int lo, int hi, int tid, int nt) {
  const int c = tid & 7;
  for (int r = tid >> 3; r < kChunk; r += nt >> 3)
    if (8 * c < width && r >= lo && r < hi) *reinterpret_cast<uint4*>(base + (int64_t)r * pitch + 8 * c) = *reinterpret_cast<const uint4*>(t + sw_off(r, c));
}
// the tiles of a ragged chunk: which & 1: v', Hk, Hv; & 2: q, do of head hq; & 4: g', k', s'
template <typename S>
__device__ __noinline__ void ragged_in(const nha_chunk_desc& d, unsigned char* sm, const ChunkRec& r, int shift, int c, int h, int hq, int which, int tid) {
  const int c0 = r.ci * kChunk, H = d.H, HQ = d.HQ, M = d.M, hi = r.len - shift;
  const size_t ch = (size_t)c * H + h;
  const int64_t rq = (int64_t)HQ * 64, rp = (int64_t)H * 64, rm = (int64_t)H * M, t0 = r.t0;
  auto t = [&](int i) { return sm + i * kTile; };
  if (which & 1) {
    rows_in(t(S::tV), (const bf16*)d.v + t0 * rp + h * 64, rp, 64, c0 - shift, hi, tid, kThreads);
    rows_in(t(S::tHk), (const bf16*)d.hk_chunks + ch * 64 * M, M, M, 0, kChunk, tid, kThreads);       // [64][M]
    rows_in(t(S::tHv), (const bf16*)d.hv_chunks + ch * M * 64, 64, 64, 0, M, tid, kThreads);          // [M][64]
  }
  if (which & 2) {
    rows_in(t(S::tQ), (const bf16*)d.q_gsa + t0 * rq + hq * 64, rq, 64, c0, r.len, tid, kThreads);
    rows_in(t(S::tDO), (const bf16*)d.d_o + t0 * rq + hq * 64, rq, 64, c0, r.len, tid, kThreads);
  }
  if (which & 4) {
    rows_in(t(S::tA), (const bf16*)d.g + t0 * rm + h * M, rm, M, c0 - shift, hi, tid, kThreads);
    rows_in(t(S::tK), (const bf16*)d.k_gsa + t0 * rp + h * 64, rp, 64, c0 - shift, hi, tid, kThreads);
    rows_in(t(S::tSB), (const bf16*)d.s + t0 * rm + h * M, rm, M, c0 - shift, hi, tid, kThreads);
  }
}
// the results of a ragged chunk: dq of a head, and with the last one dk', ds', dg
template <typename S>
__device__ __noinline__ void ragged_out(const nha_chunk_desc& d, const unsigned char* sm, const ChunkRec& r, int shift, int h, int hq, bool keys, int tid) {
  const int c0 = r.ci * kChunk, H = d.H, HQ = d.HQ, M = d.M, n = r.len - c0, lo = max(0, shift - c0);
  auto t = [&](int i) { return sm + i * kTile; };
  rows_out(t(S::tZA), (bf16*)d.dq_gsa + ((int64_t)(r.t0 + c0) * HQ + hq) * 64, (int64_t)HQ * 64, 64, 0, n, tid, kThreads);
  if (keys) {
    const int64_t row = ((int64_t)r.t0 + c0 - shift) * H + h;
    rows_out(t(S::tPA), (bf16*)d.dk_gsa + row * 64, (int64_t)H * 64, 64, lo, n, tid, kThreads);
    rows_out(t(S::tDK), (bf16*)d.ds + row * M, (int64_t)H * M, M, lo, n, tid, kThreads);
    rows_out(t(S::tDV), (bf16*)d.dg + row * M, (int64_t)H * M, M, lo, n, tid, kThreads);
  }
}

// Sums over the eight lanes of equal lane % 4 of eight values each, by halving: the lane returns the sum of value gq.
__device__ __forceinline__ float lanes_sum(const float (&v)[8], int lane) {
  float u[4], t[2];
  const bool h2 = lane & 16, h1 = lane & 8, h0 = lane & 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) u[k] = (h2 ? v[k + 4] : v[k]) + __shfl_xor_sync(0xffffffffu, h2 ? v[k] : v[k + 4], 16);
#pragma unroll
  for (int k = 0; k < 2; ++k) t[k] = (h1 ? u[k + 2] : u[k]) + __shfl_xor_sync(0xffffffffu, h1 ? u[k] : u[k + 2], 8);
  return (h0 ? t[1] : t[0]) + __shfl_xor_sync(0xffffffffu, h0 ? t[0] : t[1], 4);
}

// k step ks of a product of 64-deep operands (mma64).  The steps of one product wait for one another; those of several products,
// dealt in turn, do not.
template <int AMN, int BMN>
__device__ __forceinline__ void mma_step(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int ks, bool acc) {
  mma_f16(d, a + (uint64_t)(ks * (AMN ? 128 : 2)), b + (uint64_t)(ks * (BMN ? 128 : 2)), idesc, acc || ks > 0);
}

// scanned: the terms kernel ran.  It has left delta and the joint log-sum-exp of the chunks that it took: those whose sequence starts in an
// earlier run (nothing starts from the others' terms).
// STEEP: some chunk of the run may be steep; DL: a gradient arrives on lse_gsa.  (Bodies of their own, so that the usual one is small.)
template <bool ONE, bool TERMS, bool STEEP, bool DL, bool M64>
__device__ __forceinline__ void slot64_run(const nha_chunk_desc& d, const BwdWs& w, int* __restrict__ err, const SlotMaps& maps, const int scanned,
                                           const int h, const int lo, const int top) {
  typedef SlotSm<ONE, TERMS> S;
  const int H = d.H, HQ = d.HQ, M = M64 ? 64 : d.M, NG = ONE ? 1 : HQ / H;
  int cg = top;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;
  const int uwarp = (int)uniform(threadIdx.x >> 5);
  const bool issuer = uwarp == 0;                              // the warp whose elected lane issues the products

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = align_1024(smem_raw);
  float* tab = (float*)(sm + S::oTab);
  float* rowv = (float*)(sm + S::oRow);
  float* tot = (float*)(sm + S::oTot);
  uint64_t* mb = (uint64_t*)(sm + S::oBar);                    // [0..4] products, [5] loads
  uint32_t* tslot = (uint32_t*)(mb + 6);
  // records of the chunk behind, this one and the next (chunk % 4): {sequence, chunk, first token, length, shift, flag}
  int4* recs = (int4*)(sm + S::oRec);
  auto rec_put = [&](int c, const ChunkRec& r) {
    recs[2 * (c & 3)] = make_int4(r.n, r.ci, r.t0, r.len);
    recs[2 * (c & 3) + 1] = make_int4(seq_shift(d, r.n), w.flags[(size_t)c * H + h], 0, 0);
  };
  auto rec_get = [&](int c) {
    const int4 r = recs[2 * (c & 3)];
    return ChunkRec{r.x, r.y, r.z, r.w};
  };
  auto rec_shift = [&](int c) { return recs[2 * (c & 3) + 1].x; };
  auto tile = [&](int i) { return sm + i * kTile; };
  const uint32_t sbase = smem_u32(sm);
  auto at = [&](int t, uint32_t off) { return sbase + (uint32_t)(t * kTile) + off; };

  bool failed = false;
  uint32_t lph = 0, ph = 0;
  const int64_t rm = (int64_t)H * M;

  // ---- loads: warp i's elected lane asks for tile i of SlotMaps::in, so that no warp is held up by all of them ---------------------
  // The load barrier's phase takes one arrival of each of these warps, with the bytes of its tile where that comes by TMA.
  auto ask = [&](const ChunkRec& r, int shift, int c, int hq, int from, int to) {
    const int c0 = r.ci * kChunk;
    if (maps.use && c0 >= shift && c0 + kChunk <= r.len) {
      if (uwarp >= from && uwarp <= to && elect_one()) {
        constexpr uint32_t kIn = S::tQ | S::tDO << 4 | S::tK << 8 | S::tSB << 12 | S::tA << 16 | S::tV << 20 | S::tHk << 24 | S::tHv << 28;
        const int y = uwarp < kInK ? hq : uwarp < kInHk ? h : 0, z = uwarp < kInK ? r.t0 + c0 : uwarp < kInHk ? r.t0 + c0 - shift : (c * H + h) * 64;
        mbar_expect_tx(&mb[5], kTile);
        tma_load_3d(tile((kIn >> (4 * uwarp)) & 15), &maps.in[uwarp], 0, y, z, &mb[5]);
      }
    } else {
      ragged_in<S>(d, sm, r, shift, c, h, hq, from >= kInV ? 1 : to <= kInDO ? 2 : 6, tid);
      if (uwarp >= from && uwarp <= to && elect_one()) mbar_arrive(&mb[5]);
    }
  };
  auto loads_wait = [&]() {
    cp_wait_all();
    if (!failed && !mbar_wait(&mb[5], lph)) failed = true;
    lph ^= 1;
  };
  // row statistics of a head: delta = <do, o> by the threads of a row (do from its tile) and the joint log-sum-exp.  Rows past the end
  // read the last one's.
  struct RowIn { uint4 o[2]; float lsw, lgs, dl; };
  auto row_request = [&](const ChunkRec& r, int hq, bool have_stats) {
    const int row = from_here(tid >> 2), part = tid & 3, pos = min(r.ci * kChunk + row, r.len - 1);
    const size_t i = (size_t)(r.t0 + pos) * HQ + hq;
    RowIn x;
    x.lgs = d.lse_gsa[i];
    x.dl = DL && d.d_lse_gsa ? d.d_lse_gsa[i] : 0.f;
    x.lsw = have_stats ? w.lj[i] : d.lse_swa[i];
    if (have_stats) {
      x.o[0].x = __float_as_uint(w.delta[i]);
    } else {
      const uint4* o = reinterpret_cast<const uint4*>((const bf16*)d.o + i * 64 + 16 * part);
#pragma unroll
      for (int u = 0; u < 2; ++u) x.o[u] = __ldg(o + u);
    }
    return x;
  };
  auto row_stats = [&](const RowIn& in, const ChunkRec& r, int hq, bool have_stats) {
    const int row = from_here(tid >> 2), part = tid & 3, pos = r.ci * kChunk + row;
    float del = __uint_as_float(in.o[0].x), lj = in.lsw;
    if (!have_stats) {
      del = 0.f;
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float x[8], y[8];
        unpack8(in.o[u], x);
        unpack8(*reinterpret_cast<const uint4*>(tile(S::tDO) + sw_off(row, 2 * part + u)), y);
#pragma unroll
        for (int e = 0; e < 8; ++e) del += x[e] * y[e];
      }
#pragma unroll
      for (int o = 1; o < 4; o <<= 1) del += __shfl_xor_sync(0xffffffffu, del, o);
      const float mx = fmaxf(in.lsw, in.lgs);
      lj = mx + __logf(__expf(in.lsw - mx) + __expf(in.lgs - mx));
    }
    if (part == 0) {
      rowv[row] = -del;
      rowv[64 + row] = pos < r.len ? -lj * kLog2e : -INFINITY;  // a row past the end has no weights
      if (DL) {
        rowv[128 + row] = pos < r.len ? -in.lgs * kLog2e : -INFINITY;
        rowv[192 + row] = in.dl;
      }
      if (pos < r.len && !have_stats) {
        w.delta[(size_t)(r.t0 + pos) * HQ + hq] = del;
        w.lj[(size_t)(r.t0 + pos) * HQ + hq] = lj;
      }
    }
  };

  if (tid == 0) {
    rec_put(cg, chunk_rec(d, cg));
#pragma unroll
    for (int i = 0; i < 6; ++i) mbar_init(&mb[i], i == 5 ? kIns : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 0) tmem_alloc(tslot, S::kTmemCols);
  fill_half_signs(tile(S::tB), tid);
  tc_fence_before();
  __syncthreads();                                             // the barriers are initialised
  tc_fence_after();
  ask(rec_get(cg), rec_shift(cg), cg, h * NG, kInV, kInHv);
  ask(rec_get(cg), rec_shift(cg), cg, h * NG, kInQ, kInG);
  cp_commit();
  const uint32_t tbase = *tslot;
  const uint32_t tl = tbase + ((uint32_t)(quarter * 32) << 16) + 32 * half;  // this warp's columns of an accumulator at +0
  auto mma_wait = [&](int i) {
    if (!failed && !mbar_wait(&mb[i], ph)) failed = true;
    tc_fence_after();
  };
  auto hand_over = [&]() {
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  };
  const uint32_t iKK = idesc64(0, 0), iKM = idesc64(0, 1), iMM = idesc64(1, 1);
  uint32_t fo[2];
#pragma unroll
  for (int jp = 0; jp < 2; ++jp) fo[jp] = frag_off(quarter, half, lane, jp);
  const int r0 = 16 * quarter + gq, cbase = 32 * half + 2 * tq;  // this lane's rows r0, r0 + 8; columns cbase + 8 j, + 1
  auto to_tile = [&](int t, const float (&v)[16]) {
#pragma unroll
    for (int jp = 0; jp < 2; ++jp)
      stm4(at(t, fo[jp]), pair_bf16(v[8 * jp], v[8 * jp + 1]), pair_bf16(v[8 * jp + 2], v[8 * jp + 3]), pair_bf16(v[8 * jp + 4], v[8 * jp + 5]),
           pair_bf16(v[8 * jp + 6], v[8 * jp + 7]));
  };
  // tril of an accumulator -> bf16 tile (columns i <= row)
  auto tril_to = [&](uint32_t col, int t) {
    float v[16];
    frag_ld(tl + col, v);
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (cbase + 8 * (k >> 2) + (k & 1) > r0 + 4 * (k & 2)) v[k] = 0.f;
    to_tile(t, v);
  };
  // fp32 rows of a [64][M] or [M][64] state: this thread's part of block jp of 16 columns
  auto state_k8 = [&](const float* p, int jp, float (&v)[8]) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const int m = cbase + 16 * jp + 2 * (k & 4);
      const float2 x = p && m < M ? *reinterpret_cast<const float2*>(p + (r0 + 4 * (k & 2)) * M + m) : make_float2(0.f, 0.f);
      v[k] = x.x;
      v[k + 1] = x.y;
    }
  };
  auto state_v8 = [&](const float* p, int jp, float (&v)[8]) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const int m = r0 + 4 * (k & 2);
      const float2 x = p && m < M ? *reinterpret_cast<const float2*>(p + m * 64 + cbase + 16 * jp + 2 * (k & 4)) : make_float2(0.f, 0.f);
      v[k] = x.x;
      v[k + 1] = x.y;
    }
  };
  auto put_k8 = [&](float* p, int jp, const float (&v)[8]) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const int m = cbase + 16 * jp + 2 * (k & 4);
      if (m < M) *reinterpret_cast<float2*>(p + (r0 + 4 * (k & 2)) * M + m) = make_float2(v[k], v[k + 1]);
    }
  };
  auto put_v8 = [&](float* p, int jp, const float (&v)[8]) {
#pragma unroll
    for (int k = 0; k < 8; k += 2) {
      const int m = r0 + 4 * (k & 2);
      if (m < M) *reinterpret_cast<float2*>(p + m * 64 + cbase + 16 * jp + 2 * (k & 4)) = make_float2(v[k], v[k + 1]);
    }
  };
  // dot products of the carry from a thread's products: columns m of DK . hk over the rows (one part per quarter), rows m of DV . hv
  // (one part per block of columns)
  auto part_k = [&](const float (&c)[8], float* part, bool unscale) {
    const float sum = lanes_sum(c, lane);
    const int m = cbase + 8 * (gq >> 1) + (gq & 1);             // value gq = 2 j + e
    part[8 * m + quarter] = unscale ? sum * tab[kTabIP + m] : sum;
  };
  auto part_v = [&](float (&c)[2], float* part, bool unscale) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      c[i] += __shfl_xor_sync(0xffffffffu, c[i], 1);
      c[i] += __shfl_xor_sync(0xffffffffu, c[i], 2);
      const int m = r0 + 8 * i;
      if (tq == 0) part[8 * m + 4 + half] = unscale ? c[i] * tab[kTabIP + m] : c[i];
    }
  };
  // Results wait in their tiles until the products of the next round have been issued: whole tiles leave by TMA (one elected lane
  // for each, which sees to it that the tile has been read before anything is written there again), others as rows.
  int out_c = -1, out_h = 0;                                    // chunk and head of the waiting rows of dq; the chunk's last head: keys too
  auto flush = [&]() {
    if (out_c < 0) return;
    const ChunkRec r = rec_get(out_c);
    const int sh = rec_shift(out_c), c0 = r.ci * kChunk;
    const bool keys = ONE || out_h + 1 == (h + 1) * NG;
    if (maps.use && c0 >= sh && c0 + kChunk <= r.len) {
      if (uwarp >= 1 && uwarp <= (keys ? 4 : 1) && elect_one()) {
        static_assert(TERMS || (S::tZA == 9 && S::tPA == 10 && S::tDK == 11 && S::tDV == 12), "order of SlotMaps::out");
        tma_store_3d(&maps.out[uwarp - 1], tile(8 + uwarp), 0, uwarp == 1 ? out_h : h, r.t0 + c0 - (uwarp == 1 ? 0 : sh));
        bulk_commit();
      }
    } else {
      ragged_out<S>(d, sm, r, sh, h, out_h, keys, tid);
    }
    out_c = -1;
  };
  auto flushed = [&]() {                                        // in front of the barrier behind which the tiles are written again
    if (uwarp >= 1 && uwarp <= 4 && elect_one()) bulk_wait_read();
  };

  int par = 0;
  for (;; --cg) {
    const ChunkRec rc = rec_get(cg);
    const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk, shift = rec_shift(cg);
    const size_t ch = (size_t)cg * H + h, nh = (size_t)rc.n * H + h;
    const bool steep = STEEP && recs[2 * (cg & 3) + 1].y != 0;
    const bool more = cg > lo, last = c0 + kChunk >= len, have_stats = !TERMS && scanned && cg - ci < lo;
    float* part = (float*)(sm + S::oPart) + par * 512;
    float* part_next = (float*)(sm + S::oPart) + (par ^ 1) * 512;
    // the state gradient at this chunk's end where it does not come from the chunk behind
    const float* endk = last ? (d.d_hkt ? d.d_hkt + nh * 64 * M : nullptr) : w.dkc + ch * 64 * M;
    const float* endv = last ? (d.d_hvt ? d.d_hvt + nh * M * 64 : nullptr) : w.dvc + ch * M * 64;
    if (!TERMS && (last || cg == top)) {
      float v[8], x[8], c[8], cv[2] = {0.f, 0.f};
      auto next = [&](const bf16* p, bool ok) { return ok ? pair_f32(*reinterpret_cast<const uint32_t*>(p)) : make_float2(0.f, 0.f); };
#pragma unroll
      for (int jp = 0; jp < 2; ++jp) {
        state_k8(endk, jp, v);
        if (ONE) frag_st8(tl + S::cSK + 16 * jp, v);
        if (last) state_k8(d.d_hkt ? d.hkt + nh * 64 * M : nullptr, jp, x);
#pragma unroll
        for (int k = 0; k < 8 && !last; k += 2) {
          const int m = cbase + 16 * jp + 2 * (k & 4);
          const float2 f = next((const bf16*)d.hk_chunks + (ch + H) * 64 * M + (r0 + 4 * (k & 2)) * M + m, m < M);
          x[k] = f.x;
          x[k + 1] = f.y;
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) c[4 * jp + 2 * j + e] = fmaf(v[4 * j + e], x[4 * j + e], v[4 * j + 2 + e] * x[4 * j + 2 + e]);
      }
      part_k(c, part, false);
#pragma unroll
      for (int jp = 0; jp < 2; ++jp) {
        state_v8(endv, jp, v);
        if (ONE) frag_st8(tl + S::cSV + 16 * jp, v);
        if (last) state_v8(d.d_hkt ? d.hvt + nh * M * 64 : nullptr, jp, x);
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const int m = r0 + 4 * (k & 2);
          if (!last) {
            const float2 f = next((const bf16*)d.hv_chunks + (ch + H) * M * 64 + m * 64 + cbase + 16 * jp + 2 * (k & 4), m < M);
            x[k] = f.x;
            x[k + 1] = f.y;
          }
          cv[(k >> 1) & 1] = fmaf(v[k + 1], x[k + 1], fmaf(v[k], x[k], cv[(k >> 1) & 1]));
        }
      }
      part_v(cv, part, false);
      if (ONE) tmem_st_wait();
    }
    SteepCtx sx;
    if (steep) sx = SteepCtx{(const bf16*)d.g + (int64_t)(t0 + c0 - shift) * rm + h * M, (int)rm, shift - c0, len - c0, M};
    float a[16], ga[16], dsum[16];
    uint32_t s[8];                                              // SB, as its tile has it
#pragma unroll
    for (int k = 0; k < 16; ++k) ga[k] = dsum[k] = 0.f;
    for (int ht = 0; ht < NG; ++ht) {
      const int hq = h * NG + ht;
      const bool first = ONE || ht == 0, fin = ONE || ht + 1 == NG;
      const RowIn rows = row_request(rc, hq, have_stats);
      if (!first) {
        ask(rc, shift, cg, hq, kInQ, kInDO);
        cp_commit();
        if (uwarp > kInDO && uwarp < kIns && elect_one()) mbar_arrive(&mb[5]);
      }
      loads_wait();
      hand_over();
      if (issuer) {
        const uint32_t sb = uniform(sbase), tb = uniform(tbase);
        auto desc = [&](int t) { return make_desc(sb + t * kTile); };
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            if (first) mma_step<0, 1>(tb + S::cC, desc(S::tB), desc(S::tA), iKM, ks, false);
            mma_step<0, 0>(tb + S::cA, desc(S::tQ), desc(S::tK), iKK, ks, false);
            mma_step<0, 0>(tb + S::cB, desc(S::tDO), desc(S::tV), iKK, ks, false);
          }
          commit(&mb[0]);
        }
      }
      if (!TERMS) flush();
      row_stats(rows, rc, hq, have_stats);
      mma_wait(0);
      if (first) {
        frag_ld(tl + S::cC, a);
        if (quarter == 3 && gq == 7) {                         // row 63: x = R = Gend / 2
#pragma unroll
          for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float R = a[4 * j + 2 + e], n = steep ? 0.f : rintf(__fmul_rn(R, kLog2e));   // (explicit roundings: the two kernels agree)
              const int m = cbase + 8 * j + e;
              tab[kTabP + m] = __int_as_float((127 + (int)n) << 23);
              tab[kTabC + m] = fmaf(R, kLog2e, -n);
              if (!TERMS) {
                tab[kTabIP + m] = __int_as_float((127 - (int)n) << 23);
                tab[kTabF + m] = steep ? 1.f : exp2f(fmaf(2.f * R, kLog2e, -n));
                tab[kTabD + m] = __expf(2.f * R);
              }
            }
            if (TERMS) {
              const int m = cbase + 8 * j;
              if (m < M) *reinterpret_cast<float2*>(w.gend + ch * M + m) = make_float2(2.f * a[4 * j + 2], 2.f * a[4 * j + 3]);
            }
          }
        }
      }
      tril_to(S::cA, S::tA);
      tril_to(S::cB, S::tB);
      if (first) {
        __syncthreads();
        // a = exp(G - R), SB = s' exp(R - G), and the states times exp(R)
        const uint32_t pv0 = pair_bf16(tab[kTabP + r0], tab[kTabP + r0]), pv1 = pair_bf16(tab[kTabP + r0 + 8], tab[kTabP + r0 + 8]);
        auto times = [](uint32_t x, uint32_t y) {
          const __nv_bfloat162 z = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
          return *reinterpret_cast<const uint32_t*>(&z);
        };
#pragma unroll
        for (int jp = 0; jp < 2; ++jp) {
          uint32_t hk[4], hv[4], sv[4], sb[4];
          ldm4(at(S::tSB, fo[jp]), sv);
          ldm4(at(S::tHk, fo[jp]), hk);
          ldm4(at(S::tHv, fo[jp]), hv);
#pragma unroll
          for (int q = 0; q < 4; ++q) {                        // rows gq (+ 8 for odd q), columns of block 2 jp + q / 2
            const int e = 8 * jp + 2 * q, m = cbase + 16 * jp + 8 * (q >> 1);
            const float2 c2 = *reinterpret_cast<const float2*>(tab + kTabC + m), p2 = *reinterpret_cast<const float2*>(tab + kTabP + m);
            const float x0 = fmaf(a[e], kLog2e, c2.x), x1 = fmaf(a[e + 1], kLog2e, c2.y);
            const float2 f = pair_f32(sv[q]);
            sb[q] = steep ? sv[q] : pair_bf16(f.x * exp2f(-x0), f.y * exp2f(-x1));
            a[e] = exp2f(x0);
            a[e + 1] = exp2f(x1);
            hk[q] = times(hk[q], pair_bf16(p2.x, p2.y));
            hv[q] = times(hv[q], (q & 1) ? pv1 : pv0);
          }
#pragma unroll
          for (int q = 0; q < 4; ++q) s[4 * jp + q] = sb[q];
          stm4(at(S::tSB, fo[jp]), sb[0], sb[1], sb[2], sb[3]);
          stm4(at(S::tHk, fo[jp]), hk[0], hk[1], hk[2], hk[3]);
          stm4(at(S::tHv, fo[jp]), hv[0], hv[1], hv[2], hv[3]);
        }
        if (steep) {                                           // no factors on the rows: the steep_ functions put them in
#pragma unroll
          for (int k = 0; k < 16; ++k) a[k] = 1.f;
        }
      }
      if (!TERMS) flushed();
      hand_over();
      if (issuer) {
        const uint32_t sb = uniform(sbase), tb = uniform(tbase);
        auto desc = [&](int t) { return make_desc(sb + t * kTile); };
        if (elect_one()) {
          if (!steep) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              mma_step<0, 1>(tb + S::cC, desc(S::tA), desc(S::tSB), iKM, ks, false);
              mma_step<0, 1>(tb + S::cD, desc(S::tB), desc(S::tSB), iKM, ks, false);
            }
          }
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            mma_step<0, 1>(tb + S::cC, desc(S::tQ), desc(S::tHk), iKM, ks, !steep);
            mma_step<0, 0>(tb + S::cD, desc(S::tDO), desc(S::tHv), iKK, ks, !steep);
          }
          commit(&mb[1]);
        }
      }
      if (!TERMS && fin) {                                     // DK' and DV'
        const float f0 = tab[kTabF + r0], f1 = tab[kTabF + r0 + 8];
#pragma unroll
        for (int jp = 0; jp < 2; ++jp) {
          float g[8], v[8];
          if (ONE) {
            frag_ld8_nowait(tl + S::cSK + 16 * jp, g);
            frag_ld8_nowait(tl + S::cSV + 16 * jp, v);
            tmem_ld_wait();
          } else {
            state_k8(endk, jp, g);
            state_v8(endv, jp, v);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j) {
            const float2 f = *reinterpret_cast<const float2*>(tab + kTabF + cbase + 16 * jp + 8 * j);
#pragma unroll
            for (int k = 4 * j; k < 4 * j + 4; ++k) {
              g[k] *= (k & 1) ? f.y : f.x;
              v[k] *= (k & 2) ? f1 : f0;
            }
          }
          frag8_to_tile(at(S::tDK, fo[jp]), g);
          frag8_to_tile(at(S::tDV, fo[jp]), v);
        }
      }
      const float nd[2] = {rowv[r0], rowv[r0 + 8]}, nLj[2] = {rowv[64 + r0], rowv[64 + r0 + 8]};   // -delta, -Lj
      const float sc2 = d.scale * kLog2e;
      const uint64_t sc22 = pack2(sc2, sc2), scale2 = pack2(d.scale, d.scale);
      mma_wait(1);
      if (steep) {                                             // (the results that waited in ZA and PA have left)
        steep_rows(sx, S::tA, S::tSB, S::tZA, tl + S::cC, r0, cbase);
        steep_rows(sx, S::tB, S::tSB, S::tZA, tl + S::cD, r0, cbase);
      }
      // ---- slot part of dz, decayed bf16 operands, gate terms --------------------------------------------------------------
#pragma unroll
      for (int jp = 0; jp < 2; ++jp) {
        float z[8], y[8];
        uint32_t pa[4];
        frag_ld8_nowait(tl + S::cC + 16 * jp, z);
        frag_ld8_nowait(tl + S::cD + 16 * jp, y);
        tmem_ld_wait();
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const int i = (k >> 1) & 1, K = 8 * jp + k;
          const bool mlive = M == 64 || cbase + 16 * jp + 2 * (k & 4) < M;
          const float L = mlive ? nLj[i] : -INFINITY;
          const uint64_t a2 = pack2(a[K], a[K + 1]), ok = fmul2(a2, pack2(z[k], z[k + 1])), y2 = pack2(y[k], y[k + 1]);
          float e0, e1;
          unpack2(ffma2(ok, sc22, pack2(L, L)), e0, e1);
          const uint64_t ps = pack2(exp2f(e0), exp2f(e1));
          uint64_t dz = fmul2(ps, ffma2(a2, y2, pack2(nd[i], nd[i])));   // (one operation: the two kernels of a call agree to the bit)
          if (DL && d.d_lse_gsa) {
            const float g = mlive ? rowv[128 + r0 + 8 * i] : -INFINITY, dl = rowv[192 + r0 + 8 * i];
            unpack2(ffma2(ok, sc22, pack2(g, g)), e0, e1);
            dz = ffma2(pack2(dl, dl), pack2(exp2f(e0), exp2f(e1)), dz);
          }
          const uint64_t zs = fmul2(dz, scale2);
          unpack2(fmul2(ps, a2), e0, e1);                      // p a
          pa[k >> 1] = pair_bf16(e0, e1);
          if (!TERMS) {
            const float2 r = pair_f32(pa[k >> 1]);             // gate terms ok dz + p dp, the latter as (p a) Y: see below
            unpack2(ffma2(pack2(r.x, r.y), y2, ffma2(ok, zs, pack2(ga[K], ga[K + 1]))), ga[K], ga[K + 1]);
          }
          unpack2(fmul2(zs, a2), z[k], z[k + 1]);              // scale dz a
        }
        frag8_to_tile(at(S::tZA, fo[jp]), z);
        stm4(at(S::tPA, fo[jp]), pa[0], pa[1], pa[2], pa[3]);
      }
      if (steep) {
        __syncthreads();
        if (!TERMS) {
          steep_keys(sx, S::tA, S::tB, S::tZA, S::tPA, w.dsp + ((size_t)(t0 + c0) * H + h) * M, rm, !first);
          __syncthreads();
        }
        steep_pairs<!TERMS>(sx, S::tA, S::tB, S::tZA, S::tPA, S::tSB);
        if (!TERMS && fin) {
          __syncthreads();
          steep_ends(sx, S::tSB, -1, 0, nullptr, 0, r0, cbase);
        }
      }
      hand_over();
      if (issuer) {
        const uint32_t sb = uniform(sbase), tb = uniform(tbase);
        auto desc = [&](int t) { return make_desc(sb + t * kTile); };
        if (elect_one()) {
          if (!TERMS) {
            if (!steep) {
#pragma unroll
              for (int ks = 0; ks < 4; ++ks) {
                mma_step<0, 0>(tb + S::cA, desc(S::tZA), desc(S::tSB), iKK, ks, false);
                mma_step<0, 0>(tb + S::cB, desc(S::tPA), desc(S::tSB), iKK, ks, false);
                mma_step<1, 1>(tb + S::cD, desc(S::tA), desc(S::tZA), iMM, ks, false);
              }
              mma64<1, 1>(tb + S::cD, desc(S::tB), desc(S::tPA), iMM, true);
            }
            commit(&mb[2]);
          }
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            mma_step<1, 1>(tb + S::cLK, desc(S::tQ), desc(S::tZA), iMM, ks, !first);
            mma_step<1, 1>(tb + S::cLV, desc(S::tPA), desc(S::tDO), iMM, ks, !first);
            if (!TERMS && fin) mma_step<0, 1>(tb + S::cD, desc(S::tK), desc(S::tDK), iKM, ks, !steep);
            if (!TERMS) mma_step<0, 0>(tb + S::cC, desc(S::tZA), desc(S::tHk), iKK, ks, false);
          }
          if (!TERMS && fin) mma64<0, 0>(tb + S::cD, desc(S::tV), desc(S::tDV), iKK, true);
          commit(&mb[3]);
        }
      }
      if (TERMS) {
        mma_wait(3);
        ph ^= 1;
        continue;
      }
      if (first && more) {                                     // the next chunk's record, and its rows into L2
        const ChunkRec rn = chunk_rec(d, cg - 1);
        const int i = uwarp, row = rn.t0 + rn.ci * kChunk;
        // (where the keys are shifted theirs are other rows: asked for here they gain nothing, 16 x 2048 tokens, 16 heads, shift 64: 539.7 us of a
        // backward with and 539.1 without)
        const bool shifted = i >= kInK && i < kInHk && seq_shift(d, rn.n) > 0;
        if (i == kInHv && lane == 0) rec_put(cg - 1, rn);
        if (maps.use && !shifted && elect_one()) {
          prefetch_tile(maps.in[i], 0, i < kInK ? h * NG : i < kInHk ? h : 0, i < kInHk ? row : (int)((ch - H) * 64));
          if (i == 1 && !(scanned && cg - 1 - rn.ci < lo)) prefetch_tile(maps.o, 0, h * NG, row);
        }
      }
      mma_wait(2);
      if (!steep) {
        tril_to(S::cA, S::tA);
        tril_to(S::cB, S::tB);
      }
      hand_over();
      if (issuer) {
        const uint32_t sb = uniform(sbase), tb = uniform(tbase);
        auto desc = [&](int t) { return make_desc(sb + t * kTile); };
        if (elect_one()) {
#pragma unroll
          for (int ks = 0; ks < 4; ++ks) {
            mma_step<0, 1>(tb + S::cC, desc(S::tA), desc(S::tK), iKM, ks, true);
            mma_step<1, 1>(tb + S::cOK, desc(S::tA), desc(S::tQ), iMM, ks, !first);
            mma_step<1, 1>(tb + S::cOV, desc(S::tB), desc(S::tDO), iMM, ks, !first);
          }
          if (fin) {
#pragma unroll
            for (int ks = 0; ks < 4; ++ks) {
              mma_step<0, 0>(tb + S::cOK, desc(S::tSB), desc(S::tDK), iKK, ks, true);
              mma_step<0, 1>(tb + S::cOV, desc(S::tSB), desc(S::tDV), iKM, ks, true);
            }
          }
          commit(&mb[4]);
        }
      }
      mma_wait(3);
      bool keep[2];
      uint32_t dsp[8];
      if (!fin) {
        if (!steep) {
          float v[16];
          frag_ld(tl + S::cD, v);
#pragma unroll
          for (int k = 0; k < 16; ++k) dsum[k] += v[k];
        }
      } else {
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int p = c0 + r0 + 8 * i;
          keep[i] = p >= shift && p < len;                     // rows of this lane that are a token's
        }
        if (steep) steep_ends(sx, 0, S::tZA, tl + S::cD, w.dsp + ((size_t)(t0 + c0) * H + h) * M, rm, r0, cbase);
        float v[16];
        frag_ld(tl + S::cD, v);
        // The gate terms less s' ds', as SB times what is divided by a for ds'.  A pair of rows adds (p a)[t] Av[t,i] SB[i] to the terms of
        // row t and takes it off those of row i; with the operands as the products had them, rounded, on both sides the pairs cancel to the
        // last bit in the sums over the rows behind (error of dg against 64 bits 2.07e-2 with p dp and s' ds' formed in fp32, 4.3e-3 so).
#pragma unroll
        for (int jp = 0; jp < 2; ++jp) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int k = 8 * jp + 2 * q, i = q & 1;
            if (!ONE) { v[k] += dsum[k]; v[k + 1] += dsum[k + 1]; }
            const float2 sv = pair_f32(s[4 * jp + q]);         // (a steep chunk's is s' itself, and a is 1)
            ga[k] = keep[i] ? ga[k] - sv.x * v[k] : 0.f;
            ga[k + 1] = keep[i] ? ga[k + 1] - sv.y * v[k + 1] : 0.f;
            dsp[k >> 1] = pair_bf16(__fdividef(v[k], a[k]), __fdividef(v[k + 1], a[k + 1]));
          }
        }
        // the state gradient at the chunk's start, and its dot products with the chunk's start state: the next chunk's carry
        {
          // (16 columns at a time: with whole fragments the registers do not suffice)
          float c[8], cv[2] = {0.f, 0.f};
#pragma unroll
          for (int jp = 0; jp < 2; ++jp) {
            float g[8], l[8];
            uint32_t x[4];
            if (ONE) frag_ld8_nowait(tl + S::cSK + 16 * jp, g); else state_k8(endk, jp, g);
            frag_ld8_nowait(tl + S::cLK + 16 * jp, l);
            ldm4(at(S::tHk, fo[jp]), x);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 2; ++j) {
              const int m = cbase + 16 * jp + 8 * j;
              const float2 dec = *reinterpret_cast<const float2*>(tab + kTabD + m), p2 = *reinterpret_cast<const float2*>(tab + kTabP + m);
              const float2 h0 = pair_f32(x[2 * j]), h1 = pair_f32(x[2 * j + 1]);
#pragma unroll
              for (int k = 4 * j; k < 4 * j + 4; ++k) g[k] = fmaf(g[k], (k & 1) ? dec.y : dec.x, __fmul_rn(l[k], (k & 1) ? p2.y : p2.x));
              c[4 * jp + 2 * j] = fmaf(g[4 * j], h0.x, g[4 * j + 2] * h1.x);
              c[4 * jp + 2 * j + 1] = fmaf(g[4 * j + 1], h0.y, g[4 * j + 3] * h1.y);
            }
            if (ONE) frag_st8(tl + S::cSK + 16 * jp, g);
            else if (more && ci > 0) put_k8(w.dkc + (ch - H) * 64 * M, jp, g);
            if (ci == 0 && d.dhk0) put_k8(d.dhk0 + nh * 64 * M, jp, g);
          }
          part_k(c, part_next, true);
          const float d0 = tab[kTabD + r0], d1 = tab[kTabD + r0 + 8], p0 = tab[kTabP + r0], p1 = tab[kTabP + r0 + 8];
#pragma unroll
          for (int jp = 0; jp < 2; ++jp) {
            float g[8], l[8];
            uint32_t x[4];
            if (ONE) frag_ld8_nowait(tl + S::cSV + 16 * jp, g); else state_v8(endv, jp, g);
            frag_ld8_nowait(tl + S::cLV + 16 * jp, l);
            ldm4(at(S::tHv, fo[jp]), x);
            tmem_ld_wait();
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int k = 2 * q, i = q & 1;
              const float2 hv = pair_f32(x[q]);
              g[k] = fmaf(g[k], i ? d1 : d0, __fmul_rn(l[k], i ? p1 : p0));
              g[k + 1] = fmaf(g[k + 1], i ? d1 : d0, __fmul_rn(l[k + 1], i ? p1 : p0));
              cv[i] = fmaf(g[k + 1], hv.y, fmaf(g[k], hv.x, cv[i]));
            }
            if (ONE) frag_st8(tl + S::cSV + 16 * jp, g);
            else if (more && ci > 0) put_v8(w.dvc + (ch - H) * M * 64, jp, g);
            if (ci == 0 && d.dhv0) put_v8(d.dhv0 + nh * M * 64, jp, g);
          }
          part_v(cv, part_next, true);
          if (ONE) tmem_st_wait();
        }
        // reverse running sum over the rows: inside the blocks of eight rows over the lanes, then the later block, then the later
        // quarters and the carry
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            float x = ga[4 * j + e], y = ga[4 * j + 2 + e];
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) {
              const float x2 = __shfl_down_sync(0xffffffffu, x, 4 * o), y2 = __shfl_down_sync(0xffffffffu, y, 4 * o);
              if (gq + o < 8) { x += x2; y += y2; }
            }
            x += __shfl_sync(0xffffffffu, y, tq);
            ga[4 * j + e] = x;
            ga[4 * j + 2 + e] = y;
            if (gq == 0) tot[4 * (cbase + 8 * j + e) + quarter] = x;
          }
        hand_over();
        if (more) ask(rec_get(cg - 1), rec_shift(cg - 1), cg - 1, h * NG, kInV, kInHv);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int m = cbase + 8 * j + e;
            const float4 p4 = *reinterpret_cast<const float4*>(part + 8 * m), t4 = *reinterpret_cast<const float4*>(tot + 4 * m);
            const float2 v2 = *reinterpret_cast<const float2*>(part + 8 * m + 4);
            float add = ((p4.x + p4.y) + (p4.z + p4.w)) + (v2.x + v2.y);
            add += (quarter < 1 ? t4.y : 0.f) + ((quarter < 2 ? t4.z : 0.f) + (quarter < 3 ? t4.w : 0.f));
            ga[4 * j + e] += add;
            ga[4 * j + 2 + e] += add;
          }
      }
      mma_wait(4);
      ph ^= 1;
      if (fin && more) {
        ask(rec_get(cg - 1), rec_shift(cg - 1), cg - 1, h * NG, kInQ, kInG);
        cp_commit();
      }
      float v[16];
      frag_ld(tl + S::cC, v);
      to_tile(S::tZA, v);
      out_c = cg;
      out_h = hq;
      if (fin) {
        frag_ld(tl + S::cOK, v);
        to_tile(S::tPA, v);
#pragma unroll
        for (int jp = 0; jp < 2; ++jp) stm4(at(S::tDK, fo[jp]), dsp[4 * jp], dsp[4 * jp + 1], dsp[4 * jp + 2], dsp[4 * jp + 3]);
        to_tile(S::tDV, ga);
        frag_ld(tl + S::cOV, v);
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (keep[i]) {
            float* p = w.dvacc + ((size_t)(t0 + c0 + r0 + 8 * i - shift) * H + h) * 64 + cbase;
#pragma unroll
            for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(p + 8 * j) = make_float2(v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
          }
        if (more) fill_half_signs(tile(S::tB), tid);
      }
    }
    if (TERMS) {
      const float p0 = tab[kTabP + r0], p1 = tab[kTabP + r0 + 8];
#pragma unroll
      for (int jp = 0; jp < 2; ++jp) {
        float g[8], v[8];
        frag_ld8_nowait(tl + S::cLK + 16 * jp, g);
        frag_ld8_nowait(tl + S::cLV + 16 * jp, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 p2 = *reinterpret_cast<const float2*>(tab + kTabP + cbase + 16 * jp + 8 * j);
#pragma unroll
          for (int k = 4 * j; k < 4 * j + 4; ++k) {
            g[k] *= (k & 1) ? p2.y : p2.x;
            v[k] *= (k & 2) ? p1 : p0;
          }
        }
        put_k8(w.dkc + ch * 64 * M, jp, g);
        put_v8(w.dvc + ch * M * 64, jp, v);
      }
      break;
    }
    if (!more) break;
    par ^= 1;
  }
  if (failed) atomicExch(err, 1);
  cp_wait_all();
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  if (!TERMS) {
    flush();
    if (uwarp >= 1 && uwarp <= 4 && elect_one()) bulk_wait_all();
  }
  if (warp == 0) tmem_dealloc(tbase, S::kTmemCols);
}

// The body for runs with steep chunks, as a function of its own: the registers of the other are then not shared out together with its.
template <bool ONE, bool TERMS>
__device__ __noinline__ void slot64_steep(const nha_chunk_desc& d, const BwdWs& w, int* __restrict__ err, const SlotMaps& maps, const int scanned,
                                          const int h, const int lo, const int top) {
  slot64_run<ONE, TERMS, true, true, false>(d, w, err, maps, scanned, h, lo, top);
}

template <bool ONE, bool TERMS, bool DL, bool M64>
__global__ void __launch_bounds__(kThreads, SlotSm<ONE, TERMS>::kCtas)
nha_bwd_slot64_kernel(const __grid_constant__ nha_chunk_desc d, const __grid_constant__ BwdWs w, int* __restrict__ err,
                      const __grid_constant__ SlotMaps maps, const int win, const int scanned) {
  grid_dep_wait();
  grid_dep_launch();
  const int ncb = (int)((d.Ttot + kChunk - 1) / kChunk + d.N);
  const int wi = blockIdx.x / d.H, h = blockIdx.x - wi * d.H;
  const bool whole = !TERMS && win == 0;                       // a run is a sequence
  const int lo = TERMS ? wi : whole ? d.plan[wi] : wi * win;
  int top = TERMS ? wi : whole ? d.plan[wi + 1] - 1 : min(ncb, lo + win) - 1, steep = 0;
  if (whole && top < lo) {                                     // no tokens: the initial state's gradient is the final state's
    for (int i = threadIdx.x; i < 64 * d.M; i += kThreads) {
      const size_t at = (size_t)blockIdx.x * 64 * d.M + i;
      if (d.dhk0) d.dhk0[at] = d.d_hkt ? d.d_hkt[at] : 0.f;
      if (d.dhv0) d.dhv0[at] = d.d_hvt ? d.d_hvt[at] : 0.f;
    }
    return;
  }
  if (TERMS) {
    const ChunkRec rc = chunk_rec(d, top);
    steep = w.flags[(size_t)top * d.H + h];
    if (rc.n < 0 || top - rc.ci >= top / win * win) return;     // an unused chunk, or its sequence starts in the chunk's own run
  } else {
    while (top >= lo && d.plan[d.N + 1 + top] < 0) --top;       // chunks that the plan does not use are the last ones
    if (top < lo) return;
    for (int c = lo + threadIdx.x; c <= top; c += kThreads) steep |= w.flags[(size_t)c * d.H + h];
    steep = __syncthreads_or(steep);
  }
  if (steep) slot64_steep<ONE, TERMS>(d, w, err, maps, scanned, h, lo, top);
  else slot64_run<ONE, TERMS, false, DL, M64>(d, w, err, maps, scanned, h, lo, top);
}

bool bwd64_supported(const nha_chunk_desc* d) { return d->K == 64 && d->V == 64 && d->M <= 64 && d->scale > 0.f; }

template <bool ONE, bool TERMS, bool DL, bool M64>
static int slot64_launch_as(const nha_chunk_desc* d, const BwdWs& w, int* err, const SlotMaps& maps, int win, bool scanned, cudaStream_t cs) {
  typedef SlotSm<ONE, TERMS> S;
  const auto kernel = nha_bwd_slot64_kernel<ONE, TERMS, DL, M64>;
  cudaError_t e = set_max_smem((const void*)kernel, S::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  const int64_t ncb = nha_chunk_count_bound(d->Ttot, d->N);
  launch_after(kernel, dim3((unsigned)((TERMS ? ncb : win ? (ncb + win - 1) / win : d->N) * d->H)), kThreads, S::total, cs, *d, w, err, maps, win, (int)scanned);
  return check_launch();
}
template <bool ONE, bool TERMS>
static int slot64_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, const SlotMaps& maps, int win, bool scanned, cudaStream_t cs) {
  const auto as = d->M == 64 ? (d->d_lse_gsa ? slot64_launch_as<ONE, TERMS, true, true> : slot64_launch_as<ONE, TERMS, false, true>)
                             : (d->d_lse_gsa ? slot64_launch_as<ONE, TERMS, true, false> : slot64_launch_as<ONE, TERMS, false, false>);
  return as(d, w, err, maps, win, scanned, cs);
}

void bwd_state_scan_launch(const nha_chunk_desc* d, const BwdWs& w, int win, cudaStream_t cs);

// Chunks per CTA of the walk; 0: a CTA takes a whole sequence, whatever its length, and nothing runs in front of it.  dense_T: tokens of every
// sequence of the call, or 0 (the caller's max_seqlen is then taken at its word, for this choice alone).  With whole sequences the longest chain has
// `steps` chunks: as many waves of CTAs as there are, or the even share and one sequence more.  Equal runs have `even`, and cost the terms and the
// scan besides, about half as much again, and two launches.  A chunk takes a CTA that has its SM to itself two thirds of the time that it takes one of
// two with one head a kv head (8.5 us | 12.8), four fifths with several, whose chain fills an SM better (four heads 37 | 45, seven 60 | 71).  Where
// the line lies, us, whole | cut, 148 SMs; backward of B x T tokens, or with * forward and backward in a graph; the tenths below stand for these:
//   one head, a CTA an SM:  16 heads, 4 x 2048 285 | 216, 6 x 311 | 308, 7 x 322 | 350, 9 x 347 | 427; 8 x 8192 1285 | 1407; 4 x 1024 150 | 120, 6 x 165 | 172;
//                           * 1 x 192 49 | 47, 1 x 256 56 | 47, 1 x 384 70 | 49, 3 x 512 103 | 90, 6 x 512 136 | 144
//                           (four chunks go whole all the same: such calls wait for the host, whom two launches cost more)
//   one head, two:          16 heads, 10 x 2048 459 | 459, 11 x 476 | 496, 16 x 535 | 677; 10 x 8192 1779 | 1748; 10 x 1024 237 | 254
//   several, a CTA an SM:   2, 4, 7 heads on each of 4, 36 x 512 217 | 243, 361 | 379, 582 | 583; 36 x 1024 417 | 437, 698 | 689, 1145 | 1069;
//                           * 1 x 128 65 | 62, 92 | 84, 133 | 119; 1 x 256 99 | 66, 147 | 88, 219 | 127; 30 x 128 92 | 103, 139 | 149, 225 | 222
//   several, two:           40 x 512 262 | 253, 421 | 391, 662 | 599; 44 x 512 270 | 280, 439 | 440, 697 | 685; 60 x 1024 579 | 655, 949 | 1037, 1499 | 1604
// Packed sequences of unequal length leave the whole ones ahead for longer than the bound on their chain says: 20 of 64-1024 tokens, 16 heads, 240 | 287.
static int slot64_plan(const nha_chunk_desc* d, int dense_T) {
  const int64_t ncb = nha_chunk_count_bound(d->Ttot, d->N), sms = sm_count(), places = 2 * sms, ctas = (int64_t)d->N * d->H;
  const int64_t even = (ncb * d->H + places - 1) / places;       // one wave of equal runs
  const int64_t T = dense_T > 0 ? dense_T : d->max_seqlen;
  if (T > 0) {
    const int64_t per = (T + kChunk - 1) / kChunk, waves = (ctas + places - 1) / places, steps = std::min(waves * per, even + per);
    const int64_t most = d->HQ == d->H ? (ctas <= sms ? 24 * even + 16 : 15 * even + 25) : (ctas <= sms ? 17 * even : 15 * even + 2);
    if (10 * steps <= most) return 0;
  }
  return (int)std::max<int64_t>(even, 1);
}

// The caller has checked bwd64_supported().
int bwd_slot64_launch(const nha_chunk_desc* d, const BwdWs& w, int dense_T, int* err, cudaStream_t cs) {
  SlotMaps maps;
  memset(&maps, 0, sizeof(maps));
  const int64_t rows = nha_chunk_count_bound(d->Ttot, d->N) * d->H * 64;
  CUtensorMap* in = maps.in;
  maps.use = d->M == 64 && rows < (int64_t)1 << 31 && make_map_rows_heads(&in[kInQ], d->q_gsa, d->Ttot, d->HQ, 64) &&
             make_map_rows_heads(&in[kInDO], d->d_o, d->Ttot, d->HQ, 64) && make_map_rows_heads(&in[kInK], d->k_gsa, d->Ttot, d->H, 64) &&
             make_map_rows_heads(&in[kInS], d->s, d->Ttot, d->H, 64) && make_map_rows_heads(&in[kInG], d->g, d->Ttot, d->H, 64) &&
             make_map_rows_heads(&in[kInV], d->v, d->Ttot, d->H, 64) && make_map_rows_heads(&in[kInHk], d->hk_chunks, rows, 1, 64) &&
             make_map_rows_heads(&in[kInHv], d->hv_chunks, rows, 1, 64) && make_map_rows_heads(&maps.out[0], d->dq_gsa, d->Ttot, d->HQ, 64) &&
             make_map_rows_heads(&maps.out[1], d->dk_gsa, d->Ttot, d->H, 64) && make_map_rows_heads(&maps.out[2], d->ds, d->Ttot, d->H, 64) &&
             make_map_rows_heads(&maps.out[3], d->dg, d->Ttot, d->H, 64) && make_map_rows_heads(&maps.o, d->o, d->Ttot, d->HQ, 64);
  const int win = slot64_plan(d, dense_T);
  const bool one = d->HQ == d->H;
  if (win) {
    const int st = one ? slot64_launch<true, true>(d, w, err, maps, win, false, cs) : slot64_launch<false, true>(d, w, err, maps, win, false, cs);
    if (st != NHA_OK) return st;
    bwd_state_scan_launch(d, w, win, cs);
    const int sc = check_launch();
    if (sc != NHA_OK) return sc;
  }
  return one ? slot64_launch<true, false>(d, w, err, maps, win, win > 0, cs) : slot64_launch<false, false>(d, w, err, maps, win, win > 0, cs);
}

}  // namespace nha
