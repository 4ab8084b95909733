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
// ways give the same bits: the walk updates the state gradient by the scan's arithmetic, element by element in fp32.
//
// A chunk that decays by more than 140 nats (the forward's flag) cannot have one reference.  It takes R = 0 and forms the sums
// over pairs of rows directly in fp32 (steep_*): slow, exact for any gate, and inside the same walk.
//
// What bounds it: SLOT64_BOUND
//
// Replaces, with nha_chunk_bwd_win64.cu, ChunkNativeHybridAttentionFunction.backward (nha_fla/ops/nha/chunk.py:491-564).
#include <string.h>

#include "nha_bwd_common.cuh"
#include "nha_frag64.cuh"

namespace nha {

using namespace f64;

// Tensor maps of the call's tensors (this GPU's own memory).  A tile whose 64 rows lie inside its sequence comes by TMA; the
// others (ragged ends, rows in front of a sequence) are copied piece by piece with zero fill.  use == 0: all tiles are copied
// (fewer than 64 slots, or no tensor maps).
struct SlotMaps {
  CUtensorMap qg, kg, v, g, s, dout, hk, hv, o, dq, dk, ds, dg;
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
  static constexpr int total = oBar + 64 + 1024;
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
// Rows of g, s of position r of the chunk: token c0 + r - shift, or nothing (g = s = 0).
struct SteepCtx {
  const bf16* g;      // d.g + head offset, row pitch H M
  const bf16* s;
  int64_t pitch;
  int t0, c0, len, shift, M;
};
__device__ __forceinline__ const bf16* steep_row(const SteepCtx& c, const bf16* base, int r) {
  const int p = c.c0 + r;
  return p >= c.shift && p < c.len ? base + (int64_t)(c.t0 + p - c.shift) * c.pitch : nullptr;
}
__device__ __forceinline__ float tile_at(const unsigned char* t, int r, int c) {
  return bf2f(*reinterpret_cast<const bf16*>(t + sw_off(r, c >> 3) + 2 * (c & 7)));
}
// log decays up to row r and behind it, columns m and m + 1: {G, G, Gend - G, Gend - G} (sums of their own, so that a gate of minus
// infinity leaves no difference of infinities)
__device__ __noinline__ float4 steep_sums(const SteepCtx& c, int r, int m) {
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int i = 0; i < kChunk && m < c.M; ++i) {
    const bf16* gr = steep_row(c, c.g, i);
    const float2 gv = gr ? __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gr + m)) : make_float2(0.f, 0.f);
    if (i <= r) { x.x += gv.x; x.y += gv.y; } else { x.z += gv.x; x.w += gv.y; }
  }
  return x;
}
// X[t,m] = sum_{i<=t} A[t,i] s_i[m] exp(G_t - G_i), the same for Av: fp32 rows of 64 in scratch (row = position)
__device__ __noinline__ void steep_x(const SteepCtx& c, const unsigned char* A, const unsigned char* Av, float* x, float* x2, int64_t xpitch, int tid) {
  const int r = tid >> 2, m0 = 16 * (tid & 3);
  if (m0 >= c.M || c.c0 + r >= c.len) return;
  for (int mm = m0; mm < m0 + 16; mm += 2) {
    float w0 = 1.f, w1 = 1.f, a0 = 0.f, a1 = 0.f, b0 = 0.f, b1 = 0.f;
    for (int i = r; i >= 0; --i) {
      const bf16* sr = steep_row(c, c.s, i);
      if (!sr) break;                                          // rows in front of the sequence's first token
      const float2 sv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sr + mm));
      const float2 gv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(steep_row(c, c.g, i) + mm));
      const float ai = tile_at(A, r, i), vi = tile_at(Av, r, i);
      a0 += ai * (sv.x * w0); a1 += ai * (sv.y * w1);
      b0 += vi * (sv.x * w0); b1 += vi * (sv.y * w1);
      w0 *= __expf(gv.x); w1 *= __expf(gv.y);
    }
    *reinterpret_cast<float2*>(x + (int64_t)r * xpitch + mm) = make_float2(a0, a1);
    *reinterpret_cast<float2*>(x2 + (int64_t)r * xpitch + mm) = make_float2(b0, b1);
  }
}
// dS[i,m] (+)= sum_{t>=i} (A[t,i] dz_t[m] + Av[t,i] p_t[m]) exp(G_t - G_i) into scratch; then E[t,i] = sum_m dz_t[m] s_i[m]
// exp(G_t - G_i) and Bv likewise, into A's and Av's tiles (zeros above the diagonal).  dz (times scale) and p: bf16 rows of positions.
__device__ __noinline__ void steep_grads(const SteepCtx& c, unsigned char* A, unsigned char* Av, const bf16* dz, const bf16* p, int64_t zpitch,
                                         float* ds, int64_t dpitch, bool add, int tid) {
  {
    const int r = tid >> 2, m0 = 16 * (tid & 3);
    if (m0 < c.M && c.c0 + r < c.len) {
      for (int mm = m0; mm < m0 + 16; mm += 2) {
        float w0 = 1.f, w1 = 1.f, a0 = 0.f, a1 = 0.f;
        for (int t = r; t < kChunk && c.c0 + t < c.len; ++t) {
          if (t > r) {
            const bf16* gr = steep_row(c, c.g, t);
            const float2 gv = gr ? __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gr + mm)) : make_float2(0.f, 0.f);
            w0 *= __expf(gv.x); w1 *= __expf(gv.y);
          }
          const float2 zv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dz + (int64_t)t * zpitch + mm));
          const float2 pv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + (int64_t)t * zpitch + mm));
          const float ai = tile_at(A, t, r), vi = tile_at(Av, t, r);
          a0 += (ai * zv.x + vi * pv.x) * w0;
          a1 += (ai * zv.y + vi * pv.y) * w1;
        }
        float2* o = reinterpret_cast<float2*>(ds + (int64_t)r * dpitch + mm);
        const float2 old = add ? *o : make_float2(0.f, 0.f);
        *o = make_float2(old.x + a0, old.y + a1);
      }
    }
  }
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31, m = 2 * lane;
  for (int t = warp; t < kChunk; t += kThreads / 32) {
    float2 zv = make_float2(0.f, 0.f), pv = zv;
    if (m < c.M && c.c0 + t < c.len) {
      zv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(dz + (int64_t)t * zpitch + m));
      pv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p + (int64_t)t * zpitch + m));
    }
    float w0 = 1.f, w1 = 1.f;
    for (int i = kChunk - 1; i >= 0; --i) {
      float e = 0.f, b = 0.f;
      if (i <= t) {                                            // (the same for all lanes)
        const bf16* sr = steep_row(c, c.s, i);
        if (sr && m < c.M) {
          const float2 sv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(sr + m));
          const float2 gv = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(steep_row(c, c.g, i) + m));
          e = zv.x * (sv.x * w0) + zv.y * (sv.y * w1);
          b = pv.x * (sv.x * w0) + pv.y * (sv.y * w1);
          w0 *= __expf(gv.x); w1 *= __expf(gv.y);
        }
        e = warp_sum(e);
        b = warp_sum(b);
      }
      if (lane == 0) {
        const int at = sw_off(t, i >> 3) + 2 * (i & 7);
        *reinterpret_cast<bf16*>(A + at) = f2bf(e);
        *reinterpret_cast<bf16*>(Av + at) = f2bf(b);
      }
    }
  }
}

// Sum of v[c] over the eight lanes of equal lane % 4, for eight values c: lane (gq, tq) returns the sum of value gq (bits reversed in
// the order of the halvings: 4 (gq >> 2) + ..., see the indexing below).  Seven exchanges instead of 24.
__device__ __forceinline__ float lanes_sum8(const float (&v)[8], int lane) {
  float u[4], t[2];
  const bool h2 = lane & 16, h1 = lane & 8, h0 = lane & 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float mine = h2 ? v[k + 4] : v[k], other = h2 ? v[k] : v[k + 4];
    u[k] = mine + __shfl_xor_sync(0xffffffffu, other, 16);
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const float mine = h1 ? u[k + 2] : u[k], other = h1 ? u[k] : u[k + 2];
    t[k] = mine + __shfl_xor_sync(0xffffffffu, other, 8);
  }
  const float mine = h0 ? t[1] : t[0], other = h0 ? t[0] : t[1];
  return mine + __shfl_xor_sync(0xffffffffu, other, 4);          // value 4 h2 + 2 h1 + h0 = gq
}

// k step ks of a product of 64-deep operands (mma64).  The steps of one product wait for one another; those of several products,
// dealt in turn, do not.
template <int AMN, int BMN>
__device__ __forceinline__ void mma_step(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int ks, bool acc) {
  mma_f16(d, a + (uint64_t)(ks * (AMN ? 128 : 2)), b + (uint64_t)(ks * (BMN ? 128 : 2)), idesc, acc || ks > 0);
}

// win: chunks per CTA (TERMS: one).  have_stats: delta and the joint log-sum-exp are in memory already (the terms kernel ran).
template <bool ONE, bool TERMS>
__global__ void __launch_bounds__(kThreads, SlotSm<ONE, TERMS>::kCtas)
nha_bwd_slot64_kernel(const nha_chunk_desc d, const BwdWs w, int* __restrict__ err, const __grid_constant__ SlotMaps maps, const int win,
                      const int have_stats) {
  grid_dep_wait();
  grid_dep_launch();
  typedef SlotSm<ONE, TERMS> S;
  const int H = d.H, HQ = d.HQ, M = d.M, NG = ONE ? 1 : HQ / H;
  const int ncb = (int)((d.Ttot + kChunk - 1) / kChunk + d.N);
  const int wi = blockIdx.x / H, h = blockIdx.x - wi * H, lo = wi * win;
  int cg = min(ncb, lo + win) - 1;
  ChunkRec rc = chunk_rec(d, cg);
  while (rc.n < 0 && --cg >= lo) rc = chunk_rec(d, cg);         // chunks that the plan does not use are the last ones
  if (rc.n < 0) return;
  const int top = cg;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int quarter = warp & 3, half = warp >> 2, gq = lane >> 2, tq = lane & 3;
  const int uwarp = (int)uniform(threadIdx.x >> 5);
  const bool issuer = uwarp == 0;                              // the warp whose elected lane issues the products

  extern __shared__ unsigned char smem_raw[];
  unsigned char* sm = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* tab = (float*)(sm + S::oTab);
  float* rowv = (float*)(sm + S::oRow);
  float* tot = (float*)(sm + S::oTot);
  uint64_t* mb = (uint64_t*)(sm + S::oBar);                    // [0..4] products, [5] loads
  uint32_t* tslot = (uint32_t*)(mb + 6);
  auto tile = [&](int i) { return sm + i * kTile; };
  const uint32_t sbase = smem_u32(sm);
  auto at = [&](int t, uint32_t off) { return sbase + (uint32_t)(t * kTile) + off; };

  bool failed = false;
  uint32_t lph = 0, ph = 0;
  const int lr = tid >> 3, lc = tid & 7;
  const uint32_t loff = sw_off(lr, lc);
  const bool mcol = 8 * lc < M;
  const int64_t rq = (int64_t)HQ * 64, rp = (int64_t)H * 64, rm = (int64_t)H * M;

  // ---- loads: each warp's elected lane asks for one tile, so that no warp is held up by all of them -----------------------------
  // the load barrier's phase takes one arrival of each warp, with the bytes of its tile where that comes by TMA
  auto whole = [&](int row, int hi) { return maps.use && row >= 0 && row + kChunk <= hi; };
  auto load_tokens = [&](int by, int t, const CUtensorMap& map, int head, const void* base, int64_t pitch, int width, int t0, int row, int hi) {
    if (whole(row, hi)) {
      if (uwarp == by && elect_one()) {
        mbar_expect_tx(&mb[5], kTile);
        tma_load_3d(tile(t), &map, 0, head, t0 + row, &mb[5]);
      }
    } else {
      const bf16* p = (const bf16*)base + (int64_t)t0 * pitch + head * width + 8 * lc;
      const bool cok = 8 * lc < width;
      const bool ok0 = cok && row + lr >= 0 && row + lr < hi, ok1 = cok && row + lr + 32 >= 0 && row + lr + 32 < hi;
      tile_in(tile(t), loff, p + (ok0 ? row + lr : 0) * pitch, ok0, p + (ok1 ? row + lr + 32 : 0) * pitch, ok1);
      if (uwarp == by && elect_one()) mbar_arrive(&mb[5]);
    }
  };
  auto load_states = [&](const ChunkRec& r, int c, int shift) {  // v', Hk, Hv
    const int c0 = r.ci * kChunk;
    const size_t ch = (size_t)c * H + h;
    load_tokens(5, S::tV, maps.v, h, d.v, rp, 64, r.t0, c0 - shift, r.len - shift);
    if (maps.use) {
      if (uwarp >= 6 && elect_one()) {
        mbar_expect_tx(&mb[5], kTile);
        tma_load_2d(tile(uwarp == 6 ? S::tHk : S::tHv), uwarp == 6 ? &maps.hk : &maps.hv, 0, (int)(ch * 64), &mb[5]);
      }
    } else {
      const bf16* hk = (const bf16*)d.hk_chunks + ch * 64 * M;      // [64][M]
      const bf16* hv = (const bf16*)d.hv_chunks + ch * M * 64;      // [M][64]
      const int o0 = lr * M + 8 * lc, o1 = o0 + 32 * M;
      tile_in(tile(S::tHk), loff, hk + (mcol ? o0 : 0), mcol, hk + (mcol ? o1 : 0), mcol);
      const bool v0 = lr < M, v1 = lr + 32 < M;
      tile_in(tile(S::tHv), loff, hv + (v0 ? lr * 64 + 8 * lc : 0), v0, hv + (v1 ? (lr + 32) * 64 + 8 * lc : 0), v1);
      if (uwarp >= 6 && elect_one()) mbar_arrive(&mb[5]);
    }
  };
  auto load_head = [&](const ChunkRec& r, int hq) {
    load_tokens(0, S::tQ, maps.qg, hq, d.q_gsa, rq, 64, r.t0, r.ci * kChunk, r.len);
    load_tokens(1, S::tDO, maps.dout, hq, d.d_o, rq, 64, r.t0, r.ci * kChunk, r.len);
  };
  auto load_rows = [&](const ChunkRec& r, int shift) {           // the first head's rows, k', s', g'
    const int c0 = r.ci * kChunk;
    load_tokens(4, S::tA, maps.g, h, d.g, rm, M, r.t0, c0 - shift, r.len - shift);
    load_head(r, h * NG);
    load_tokens(2, S::tK, maps.kg, h, d.k_gsa, rp, 64, r.t0, c0 - shift, r.len - shift);
    load_tokens(3, S::tSB, maps.s, h, d.s, rm, M, r.t0, c0 - shift, r.len - shift);
    cp_commit();
  };
  auto loads_wait = [&]() {
    cp_wait_all();
    if (!failed && !mbar_wait(&mb[5], lph)) failed = true;
    lph ^= 1;
  };
  // row statistics of a head: delta = <do, o> by four threads per row (do from its tile), the joint log-sum-exp by one
  uint4 o0, o1;
  float lsw, lgs, dl;
  auto row_request = [&](const ChunkRec& r, int hq) {
    const int row = tid >> 2, part = tid & 3, pos = r.ci * kChunk + row;
    o0 = o1 = make_uint4(0u, 0u, 0u, 0u);
    lsw = lgs = dl = 0.f;
    if (pos < r.len) {
      const size_t i = (size_t)(r.t0 + pos) * HQ + hq;
      if (!have_stats) {
        const uint4* o = reinterpret_cast<const uint4*>((const bf16*)d.o + i * 64 + 16 * part);
        o0 = __ldg(o); o1 = __ldg(o + 1);
      }
      if (part == 0) {
        lgs = d.lse_gsa[i];
        dl = d.d_lse_gsa ? d.d_lse_gsa[i] : 0.f;
        if (have_stats) {
          lsw = w.lj[i];
          o0.x = __float_as_uint(w.delta[i]);
        } else {
          lsw = d.lse_swa[i];
        }
      }
    }
  };
  auto row_stats = [&](const ChunkRec& r, int hq) {
    const int row = tid >> 2, part = tid & 3, pos = r.ci * kChunk + row;
    float del, lj;
    if (have_stats) {
      del = __uint_as_float(o0.x);
      lj = lsw;
    } else {
      float x[8], y[8];
      const unsigned char* t = tile(S::tDO);
      unpack8(o0, x);
      unpack8(*reinterpret_cast<const uint4*>(t + sw_off(row, 2 * part)), y);
      del = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) del += x[e] * y[e];
      unpack8(o1, x);
      unpack8(*reinterpret_cast<const uint4*>(t + sw_off(row, 2 * part + 1)), y);
#pragma unroll
      for (int e = 0; e < 8; ++e) del += x[e] * y[e];
      del += __shfl_xor_sync(0xffffffffu, del, 1);
      del += __shfl_xor_sync(0xffffffffu, del, 2);
      const float mx = fmaxf(lsw, lgs);
      lj = mx + __logf(__expf(lsw - mx) + __expf(lgs - mx));
    }
    if (part == 0) {
      rowv[row] = del;
      rowv[64 + row] = -lj * kLog2e;
      rowv[128 + row] = -lgs * kLog2e;
      rowv[192 + row] = dl;
      if (pos < r.len && !have_stats) {
        w.delta[(size_t)(r.t0 + pos) * HQ + hq] = del;
        w.lj[(size_t)(r.t0 + pos) * HQ + hq] = lj;
      }
    }
  };

  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < 6; ++i) mbar_init(&mb[i], i == 5 ? kThreads / 32 : 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_smem();
  }
  if (warp == 0) tmem_alloc(tslot, S::kTmemCols);
  fill_half_signs(tile(S::tB), tid);
  tc_fence_before();
  __syncthreads();                                             // the barriers are initialised
  tc_fence_after();
  {
    const int sh = seq_shift(d, rc.n);
    load_states(rc, cg, sh);
    load_rows(rc, sh);
  }
  const uint32_t tbase = *tslot;
  const uint32_t tl = tbase + ((uint32_t)(quarter * 32) << 16) + 32 * half;       // this warp's columns of an accumulator at +0
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
  const uint32_t fo0 = frag_off(quarter, half, lane, 0), fo1 = frag_off(quarter, half, lane, 1);
  const int r0 = 16 * quarter + gq, cbase = 32 * half + 2 * tq;  // this lane's rows r0, r0 + 8; columns cbase + 8 j, + 1
  const float sc2 = d.scale * kLog2e;
  // tril of an accumulator -> bf16 tile (columns i <= row)
  auto tril_to = [&](uint32_t col, int t) {
    float v[16];
    frag_ld(tl + col, v);
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e)
        if (cbase + 8 * j + (e & 1) > r0 + 8 * (e >> 1)) v[4 * j + e] = 0.f;
    frag_to_tile(at(t, fo0), at(t, fo1), v);
  };
  // fp32 rows of a [64][M] or [M][64] state, this thread's fragment
  auto state_k = [&](const float* p, float (&v)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = cbase + 8 * j;
        const float2 x = p && m < M ? *reinterpret_cast<const float2*>(p + (r0 + 8 * i) * M + m) : make_float2(0.f, 0.f);
        v[4 * j + 2 * i] = x.x;
        v[4 * j + 2 * i + 1] = x.y;
      }
  };
  auto state_v = [&](const float* p, float (&v)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float2 x = p && r0 + 8 * i < M ? *reinterpret_cast<const float2*>(p + (r0 + 8 * i) * 64 + cbase + 8 * j) : make_float2(0.f, 0.f);
        v[4 * j + 2 * i] = x.x;
        v[4 * j + 2 * i + 1] = x.y;
      }
  };
  auto put_k = [&](float* p, const float (&v)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int m = cbase + 8 * j;
        if (m < M) *reinterpret_cast<float2*>(p + (r0 + 8 * i) * M + m) = make_float2(v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
      }
  };
  auto put_v = [&](float* p, const float (&v)[16]) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 2; ++i)
        if (r0 + 8 * i < M) *reinterpret_cast<float2*>(p + (r0 + 8 * i) * 64 + cbase + 8 * j) = make_float2(v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
  };
  // dot products of the carry: columns m of DK . hk over the rows (one part per quarter), rows m of DV . hv (one part per half)
  auto dots_k = [&](const float (&v)[16], const float (&x)[16], float* part, bool unscale) {
    float c[8];
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) c[2 * j + e] = fmaf(v[4 * j + e], x[4 * j + e], v[4 * j + 2 + e] * x[4 * j + 2 + e]);
    const float sum = lanes_sum8(c, lane);
    const int m = cbase + 8 * (gq >> 1) + (gq & 1);             // value gq = 2 j + e
    part[8 * m + quarter] = unscale ? sum * tab[kTabIP + m] : sum;
  };
  auto dots_v = [&](const float (&v)[16], const float (&x)[16], float* part, bool unscale) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float c = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) c = fmaf(v[4 * j + 2 * i + e], x[4 * j + 2 * i + e], c);
      c += __shfl_xor_sync(0xffffffffu, c, 1);
      c += __shfl_xor_sync(0xffffffffu, c, 2);
      const int m = r0 + 8 * i;
      if (tq == 0) part[8 * m + 4 + half] = unscale ? c * tab[kTabIP + m] : c;
    }
  };
  auto tile_frag = [&](int t, float (&x)[16]) {
#pragma unroll
    for (int jp = 0; jp < 2; ++jp) {
      uint32_t u[4];
      ldm4(at(t, jp ? fo1 : fo0), u);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float2 f = pair_f32(u[q]);
        const int e = 4 * (2 * jp + (q >> 1)) + 2 * (q & 1);
        x[e] = f.x;
        x[e + 1] = f.y;
      }
    }
  };
  // Results wait in their tiles until the products of the next round have been issued: whole tiles leave by TMA (one elected lane
  // for each, which sees to it that the tile has been read before anything is written there again), others as rows.
  struct { int tok, hq, n, lo, key; bool q, k; } out;           // first token, head, valid rows; first valid key row, first key token
  out.q = out.k = false;
  auto rows_out = [&](int t, bf16* base, int64_t pitch, int lo_, int hi_, bool cok) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = lr + 32 * u;
      if (cok && r >= lo_ && r < hi_) *reinterpret_cast<uint4*>(base + (int64_t)r * pitch + 8 * lc) = *reinterpret_cast<const uint4*>(tile(t) + loff + 4096 * u);
    }
  };
  auto flush = [&]() {
    if (out.q) {
      if (maps.use && out.n >= kChunk) {
        if (uwarp == 1 && elect_one()) tma_store_3d(&maps.dq, tile(S::tZA), 0, out.hq, out.tok);
      } else {
        rows_out(S::tZA, (bf16*)d.dq_gsa + ((int64_t)out.tok * HQ + out.hq) * 64, rq, 0, out.n, true);
      }
    }
    if (out.k) {
      if (maps.use && out.n >= kChunk && out.lo == 0) {
        if (uwarp == 2 && elect_one()) tma_store_3d(&maps.dk, tile(S::tPA), 0, h, out.key);
        if (uwarp == 3 && elect_one()) tma_store_3d(&maps.ds, tile(S::tDK), 0, h, out.key);
        if (uwarp == 4 && elect_one()) tma_store_3d(&maps.dg, tile(S::tDV), 0, h, out.key);
      } else {
        const int64_t row = (int64_t)out.key * H + h;
        rows_out(S::tPA, (bf16*)d.dk_gsa + row * 64, rp, out.lo, out.n, true);
        rows_out(S::tDK, (bf16*)d.ds + row * M, rm, out.lo, out.n, mcol);
        rows_out(S::tDV, (bf16*)d.dg + row * M, rm, out.lo, out.n, mcol);
      }
    }
    out.q = out.k = false;
    if (uwarp >= 1 && uwarp <= 4 && elect_one()) bulk_commit();
  };
  auto flushed = [&]() {                                        // in front of the barrier behind which the tiles are written again
    if (uwarp >= 1 && uwarp <= 4 && elect_one()) bulk_wait_read();
  };

  int par = 0, shift = seq_shift(d, rc.n), flag = w.flags[(size_t)cg * H + h];
  row_request(rc, h * NG);
  for (;; --cg) {
    const int ci = rc.ci, t0 = rc.t0, len = rc.len, c0 = ci * kChunk;
    const size_t ch = (size_t)cg * H + h, nh = (size_t)rc.n * H + h;
    const bool steep = flag != 0;
    const bool more = cg > lo;
    ChunkRec rn = rc;                                          // the next chunk's record, shift and flag
    int shift_next = 0;
    const int nchunks = (len + kChunk - 1) / kChunk;
    const bool last = ci == nchunks - 1;
    float* part = (float*)(sm + S::oPart) + par * 512;
    float* part_next = (float*)(sm + S::oPart) + (par ^ 1) * 512;
    // the state gradient at this chunk's end where it does not come from the chunk behind
    const float* endk = last ? (d.d_hkt ? d.d_hkt + nh * 64 * M : nullptr) : w.dkc + ch * 64 * M;
    const float* endv = last ? (d.d_hvt ? d.d_hvt + nh * M * 64 : nullptr) : w.dvc + ch * M * 64;
    if (!TERMS && (last || cg == top)) {
      float v[16], x[16];
      state_k(endk, v);
      if (ONE) frag_st(tl + S::cSK, v);
      if (last) {
        state_k(d.d_hkt ? d.hkt + nh * 64 * M : nullptr, x);
      } else {
        const bf16* p = (const bf16*)d.hk_chunks + (ch + H) * 64 * M;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int m = cbase + 8 * j;
            const float2 f = m < M ? pair_f32(*reinterpret_cast<const uint32_t*>(p + (r0 + 8 * i) * M + m)) : make_float2(0.f, 0.f);
            x[4 * j + 2 * i] = f.x;
            x[4 * j + 2 * i + 1] = f.y;
          }
      }
      dots_k(v, x, part, false);
      state_v(endv, v);
      if (ONE) frag_st(tl + S::cSV, v);
      if (last) {
        state_v(d.d_hkt ? d.hvt + nh * M * 64 : nullptr, x);
      } else {
        const bf16* p = (const bf16*)d.hv_chunks + (ch + H) * M * 64;
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const float2 f = r0 + 8 * i < M ? pair_f32(*reinterpret_cast<const uint32_t*>(p + (r0 + 8 * i) * 64 + cbase + 8 * j)) : make_float2(0.f, 0.f);
            x[4 * j + 2 * i] = f.x;
            x[4 * j + 2 * i + 1] = f.y;
          }
      }
      dots_v(v, x, part, false);
    }
    SteepCtx sx;
    if (steep) sx = SteepCtx{(const bf16*)d.g + (size_t)h * M, (const bf16*)d.s + (size_t)h * M, rm, t0, c0, len, shift, M};
    float a[16], ga[16], dsum[16];
    uint32_t s[2][4];
#pragma unroll
    for (int k = 0; k < 16; ++k) ga[k] = dsum[k] = 0.f;
    for (int ht = 0; ht < NG; ++ht) {
      const int hq = h * NG + ht;
      const bool first = ONE || ht == 0, fin = ONE || ht + 1 == NG;
      if (!first) {
        load_head(rc, hq);
        cp_commit();
        if (uwarp >= 2 && elect_one()) mbar_arrive(&mb[5]);
        row_request(rc, hq);
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
      row_stats(rc, hq);
      mma_wait(0);
      if (first) {
        frag_ld(tl + S::cC, a);
        if (quarter == 3 && gq == 7) {                         // row 63: x = R = Gend / 2
#pragma unroll
          for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float R = a[4 * j + 2 + e], n = steep ? 0.f : rintf(R * kLog2e);
              const int m = cbase + 8 * j + e;
              tab[kTabP + m] = __int_as_float((127 + (int)n) << 23);
              tab[kTabC + m] = R * kLog2e - n;
              if (!TERMS) {
                tab[kTabIP + m] = __int_as_float((127 - (int)n) << 23);
                tab[kTabF + m] = steep ? 1.f : exp2f(2.f * R * kLog2e - n);
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
        // a = exp(G - R), SB = s' exp(R - G) (steep: R = 0, and s' exp(Gend - G)), and the states times exp(R)
        ldm4(at(S::tSB, fo0), s[0]);
        ldm4(at(S::tSB, fo1), s[1]);
        uint32_t hk[2][4], hv[2][4], sb[2][4];
        ldm4(at(S::tHk, fo0), hk[0]);
        ldm4(at(S::tHk, fo1), hk[1]);
        ldm4(at(S::tHv, fo0), hv[0]);
        ldm4(at(S::tHv, fo1), hv[1]);
        const uint32_t pv0 = pair_bf16(tab[kTabP + r0], tab[kTabP + r0]), pv1 = pair_bf16(tab[kTabP + r0 + 8], tab[kTabP + r0 + 8]);
        auto times = [](uint32_t x, uint32_t y) {
          const __nv_bfloat162 z = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&x), *reinterpret_cast<const __nv_bfloat162*>(&y));
          return *reinterpret_cast<const uint32_t*>(&z);
        };
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 c2 = *reinterpret_cast<const float2*>(tab + kTabC + cbase + 8 * j);
          const float2 p2 = *reinterpret_cast<const float2*>(tab + kTabP + cbase + 8 * j);
          const uint32_t pk = pair_bf16(p2.x, p2.y);
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int e = 4 * j + 2 * i, q = 2 * (j & 1) + i, jp = j >> 1;
            const float x0 = fmaf(a[e], kLog2e, c2.x), x1 = fmaf(a[e + 1], kLog2e, c2.y);
            const float2 sv = pair_f32(s[jp][q]);
            sb[jp][q] = pair_bf16(sv.x * exp2f(-x0), sv.y * exp2f(-x1));
            a[e] = exp2f(x0);
            a[e + 1] = exp2f(x1);
            hk[jp][q] = times(hk[jp][q], pk);
            hv[jp][q] = times(hv[jp][q], i ? pv1 : pv0);
          }
        }
        if (steep) {
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int e = 4 * j + 2 * i, q = 2 * (j & 1) + i, jp = j >> 1, m = cbase + 8 * j, p = c0 + r0 + 8 * i;
              const float4 g4 = steep_sums(sx, r0 + 8 * i, m);
              const float b0 = __expf(g4.z), b1 = __expf(g4.w);
              const float2 sv = pair_f32(s[jp][q]);
              sb[jp][q] = pair_bf16(sv.x * b0, sv.y * b1);
              a[e] = __expf(g4.x);
              a[e + 1] = __expf(g4.y);
              // the factor of ds, which is not 1 / a here
              if (!TERMS && m < M && p < len) *reinterpret_cast<float2*>(w.dga + ((size_t)(t0 + p) * H + h) * M + m) = make_float2(b0, b1);
            }
        }
#pragma unroll
        for (int jp = 0; jp < 2; ++jp) {
          const uint32_t fo = jp ? fo1 : fo0;
          stm4(at(S::tSB, fo), sb[jp][0], sb[jp][1], sb[jp][2], sb[jp][3]);
          stm4(at(S::tHk, fo), hk[jp][0], hk[jp][1], hk[jp][2], hk[jp][3]);
          stm4(at(S::tHv, fo), hv[jp][0], hv[jp][1], hv[jp][2], hv[jp][3]);
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
      if (steep) {
        steep_x(sx, tile(S::tA), tile(S::tB), w.dkp + ((size_t)(t0 + c0) * H + h) * 64, w.dvp + ((size_t)(t0 + c0) * H + h) * 64, rp, tid);
        __syncthreads();
      }
      if (!TERMS && fin) {                                     // DK' and DV'
        float v[16];
        if (ONE) frag_ld(tl + S::cSK, v); else state_k(endk, v);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = *reinterpret_cast<const float2*>(tab + kTabF + cbase + 8 * j);
          v[4 * j] *= f.x; v[4 * j + 1] *= f.y; v[4 * j + 2] *= f.x; v[4 * j + 3] *= f.y;
        }
        frag_to_tile(at(S::tDK, fo0), at(S::tDK, fo1), v);
        if (ONE) frag_ld(tl + S::cSV, v); else state_v(endv, v);
        const float f0 = tab[kTabF + r0], f1 = tab[kTabF + r0 + 8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          v[4 * j] *= f0; v[4 * j + 1] *= f0; v[4 * j + 2] *= f1; v[4 * j + 3] *= f1;
        }
        frag_to_tile(at(S::tDV, fo0), at(S::tDV, fo1), v);
      }
      if (!TERMS && first && more) {
        rn = chunk_rec(d, cg - 1);
        flag = w.flags[ch - H];
      }
      float delta[2], nLj[2], nLg[2], dls[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        delta[i] = rowv[r0 + 8 * i];
        nLj[i] = rowv[64 + r0 + 8 * i];
        nLg[i] = rowv[128 + r0 + 8 * i];
        dls[i] = rowv[192 + r0 + 8 * i];
      }
      mma_wait(1);
      // ---- slot part of dz (16 columns at a time), decayed bf16 operands, gate terms ---------------------------------------
#pragma unroll
      for (int jp = 0; jp < 2; ++jp) {
        float z[8], y[8];
        frag_ld8_nowait(tl + S::cC + 16 * jp, z);
        frag_ld8_nowait(tl + S::cD + 16 * jp, y);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const int m = cbase + 16 * jp + 8 * j;
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const bool live = m < M && c0 + r0 + 8 * i < len;
            float2 x = make_float2(0.f, 0.f), x2 = x, pr, zr;
            if (steep && live) {
              const size_t row = ((size_t)(t0 + c0 + r0 + 8 * i) * H + h) * 64 + m;
              x = *reinterpret_cast<const float2*>(w.dkp + row);
              x2 = *reinterpret_cast<const float2*>(w.dvp + row);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int k = 4 * j + 2 * i + e;
              const float aI = a[8 * jp + k];
              float ok = aI * z[k], dps = aI * y[k];
              if (steep) {
                ok += e ? x.y : x.x;
                dps += e ? x2.y : x2.x;
              }
              ok *= sc2;                                       // log2 units
              float ps = 0.f, dz = 0.f;
              if (live) {
                ps = exp2f(ok + nLj[i]);
                dz = ps * (dps - delta[i]);
                if (d.d_lse_gsa) dz += dls[i] * exp2f(ok + nLg[i]);
              }
              if (!TERMS) ga[8 * jp + k] += ok * kLn2 * dz + ps * dps;
              const float zs = d.scale * dz;
              (e ? pr.y : pr.x) = ps;
              (e ? zr.y : zr.x) = zs;
              z[k] = zs * aI;                                  // scale dz a
              y[k] = ps * aI;                                  // p a
            }
            if (!TERMS && steep && live) {
              const size_t row = ((size_t)(t0 + c0 + r0 + 8 * i) * HQ + hq) * M + m;
              *reinterpret_cast<uint32_t*>(w.dza + row) = pair_bf16(zr.x, zr.y);
              *reinterpret_cast<uint32_t*>(w.paq + row) = pair_bf16(pr.x, pr.y);
            }
          }
        }
        const uint32_t fo = jp ? fo1 : fo0;
        frag8_to_tile(at(S::tZA, fo), z);
        frag8_to_tile(at(S::tPA, fo), y);
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
      if (!TERMS && first && more) {                           // the next chunk's rows into L2
        shift_next = seq_shift(d, rn.n);
        if (maps.use && elect_one()) {
          const int row = rn.t0 + rn.ci * kChunk;
          if (uwarp == 0) prefetch_tile(maps.qg, 0, h * NG, row);
          if (uwarp == 1) prefetch_tile(maps.dout, 0, h * NG, row);
          if (uwarp == 2) prefetch_tile(maps.kg, 0, h, row);
          if (uwarp == 3) prefetch_tile(maps.s, 0, h, row);
          if (uwarp == 4) prefetch_tile(maps.g, 0, h, row);
          if (uwarp == 5) prefetch_tile(maps.v, 0, h, row);
          if (uwarp == 6) prefetch_bytes((const bf16*)d.hk_chunks + (ch - H) * 4096, kTile);
          if (uwarp == 7) prefetch_bytes((const bf16*)d.hv_chunks + (ch - H) * 4096, kTile);
          if (uwarp == 6 && !have_stats) prefetch_tile(maps.o, 0, h * NG, row);
        }
      }
      if (steep) {
        steep_grads(sx, tile(S::tA), tile(S::tB), w.dza + ((size_t)(t0 + c0) * HQ + hq) * M, w.paq + ((size_t)(t0 + c0) * HQ + hq) * M,
                    (int64_t)HQ * M, w.dsp + ((size_t)(t0 + c0) * H + h) * M, rm, !first, tid);
        mma_wait(2);
      } else {
        mma_wait(2);
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
        float v[16];
        if (!steep) {
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
        float v[16];
        frag_ld(tl + S::cD, v);
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const int e = 4 * j + 2 * i, q = 2 * (j & 1) + i, jp = j >> 1, m = cbase + 8 * j;
            float d0, d1;
            if (steep) {
              float2 f = make_float2(0.f, 0.f), add = f;
              if (keep[i] && m < M) {
                const size_t row = ((size_t)(t0 + c0 + r0 + 8 * i) * H + h) * M + m;
                f = *reinterpret_cast<const float2*>(w.dga + row);
                add = *reinterpret_cast<const float2*>(w.dsp + row);
              }
              d0 = fmaf(v[e], f.x, add.x);
              d1 = fmaf(v[e + 1], f.y, add.y);
            } else {
              if (!ONE) { v[e] += dsum[e]; v[e + 1] += dsum[e + 1]; }
              d0 = __fdividef(v[e], a[e]);
              d1 = __fdividef(v[e + 1], a[e + 1]);
            }
            const float2 sv = pair_f32(s[jp][q]);
            ga[e] = keep[i] ? ga[e] - sv.x * d0 : 0.f;
            ga[e + 1] = keep[i] ? ga[e + 1] - sv.y * d1 : 0.f;
            dsp[2 * j + i] = pair_bf16(d0, d1);
          }
        // the state gradient at the chunk's start, and its dot products with the chunk's start state: the next chunk's carry
        {
          float g[16], x[16];
          if (ONE) frag_ld_nowait(tl + S::cSK, g); else state_k(endk, g);
          frag_ld(tl + S::cLK, v);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 dec = *reinterpret_cast<const float2*>(tab + kTabD + cbase + 8 * j);
            const float2 p2 = *reinterpret_cast<const float2*>(tab + kTabP + cbase + 8 * j);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int e = 4 * j + 2 * i;
              g[e] = fmaf(g[e], dec.x, v[e] * p2.x);
              g[e + 1] = fmaf(g[e + 1], dec.y, v[e + 1] * p2.y);
            }
          }
          if (ONE) frag_st(tl + S::cSK, g);
          else if (more && ci > 0) put_k(w.dkc + (ch - H) * 64 * M, g);
          if (ci == 0 && d.dhk0) put_k(d.dhk0 + nh * 64 * M, g);
          tile_frag(S::tHk, x);
          dots_k(g, x, part_next, true);
          if (ONE) frag_ld_nowait(tl + S::cSV, g); else state_v(endv, g);
          frag_ld(tl + S::cLV, v);
          const float d0 = tab[kTabD + r0], d1 = tab[kTabD + r0 + 8], p0 = tab[kTabP + r0], p1 = tab[kTabP + r0 + 8];
#pragma unroll
          for (int k = 0; k < 16; ++k) g[k] = fmaf(g[k], (k & 2) ? d1 : d0, v[k] * ((k & 2) ? p1 : p0));
          if (ONE) frag_st(tl + S::cSV, g);
          else if (more && ci > 0) put_v(w.dvc + (ch - H) * M * 64, g);
          if (ci == 0 && d.dhv0) put_v(d.dhv0 + nh * M * 64, g);
          tile_frag(S::tHv, x);
          dots_v(g, x, part_next, true);
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
        if (more) load_states(rn, cg - 1, shift_next);
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
        load_rows(rn, shift_next);
        row_request(rn, h * NG);
      }
      float v[16];
      frag_ld(tl + S::cC, v);
      frag_to_tile(at(S::tZA, fo0), at(S::tZA, fo1), v);
      out.q = true;
      out.tok = t0 + c0;
      out.hq = hq;
      out.n = len - c0;
      if (fin) {
        frag_ld(tl + S::cOK, v);
        frag_to_tile(at(S::tPA, fo0), at(S::tPA, fo1), v);
        stm4(at(S::tDK, fo0), dsp[0], dsp[1], dsp[2], dsp[3]);
        stm4(at(S::tDK, fo1), dsp[4], dsp[5], dsp[6], dsp[7]);
        frag_to_tile(at(S::tDV, fo0), at(S::tDV, fo1), ga);
        frag_ld(tl + S::cOV, v);
#pragma unroll
        for (int i = 0; i < 2; ++i)
          if (keep[i]) {
            float* p = w.dvacc + ((size_t)(t0 + c0 + r0 + 8 * i - shift) * H + h) * 64 + cbase;
#pragma unroll
            for (int j = 0; j < 4; ++j) *reinterpret_cast<float2*>(p + 8 * j) = make_float2(v[4 * j + 2 * i], v[4 * j + 2 * i + 1]);
          }
        out.k = true;
        out.lo = max(0, shift - c0);
        out.key = t0 + c0 - shift;
        if (more) fill_half_signs(tile(S::tB), tid);
      }
    }
    if (TERMS) {
      float v[16];
      frag_ld(tl + S::cLK, v);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 p2 = *reinterpret_cast<const float2*>(tab + kTabP + cbase + 8 * j);
        v[4 * j] *= p2.x; v[4 * j + 1] *= p2.y; v[4 * j + 2] *= p2.x; v[4 * j + 3] *= p2.y;
      }
      put_k(w.dkc + ch * 64 * M, v);
      frag_ld(tl + S::cLV, v);
      const float p0 = tab[kTabP + r0], p1 = tab[kTabP + r0 + 8];
#pragma unroll
      for (int k = 0; k < 16; ++k) v[k] *= (k & 2) ? p1 : p0;
      put_v(w.dvc + ch * M * 64, v);
      break;
    }
    if (!more) break;
    rc = rn;
    shift = shift_next;
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

bool bwd64_supported(const nha_chunk_desc* d) { return d->K == 64 && d->V == 64 && d->M <= 64 && d->scale > 0.f; }

template <bool ONE, bool TERMS>
static int slot64_launch(const nha_chunk_desc* d, const BwdWs& w, int* err, const SlotMaps& maps, int win, bool stats, cudaStream_t cs) {
  typedef SlotSm<ONE, TERMS> S;
  cudaError_t e = set_max_smem((const void*)nha_bwd_slot64_kernel<ONE, TERMS>, S::total);
  if (e != cudaSuccess) return record_cuda_error(e);
  const int64_t ncb = nha_chunk_count_bound(d->Ttot, d->N);
  launch_after(nha_bwd_slot64_kernel<ONE, TERMS>, dim3((unsigned)((ncb + win - 1) / win * d->H)), kThreads, S::total, cs, *d, w, err, maps, win, (int)stats);
  return check_launch();
}

void bwd_state_scan_launch(const nha_chunk_desc* d, const BwdWs& w, int win, cudaStream_t cs);

// Chunks per CTA of the walk, and whether the terms and the scan are needed in front of it.  dense_T: tokens of every sequence of the
// call, or 0.
struct SlotPlan { int win; bool scan; };
static SlotPlan slot64_plan(const nha_chunk_desc* d, int dense_T) {
  const int64_t ncb = nha_chunk_count_bound(d->Ttot, d->N), places = 2 * (int64_t)sm_count();
  const int64_t even = (ncb * d->H + places - 1) / places;       // one wave of equal runs
  if (dense_T > 0) {
    const int64_t per = (dense_T + kChunk - 1) / kChunk, seqs = (int64_t)d->N * d->H;
    // whole sequences
    const int64_t waves = (seqs + places - 1) / places;
    if (2 * waves * per <= 3 * even + 6) return {(int)per, false};
  }
  return {(int)(even > 0 ? even : 1), true};
}

// The caller has checked bwd64_supported().
int bwd_slot64_launch(const nha_chunk_desc* d, const BwdWs& w, int dense_T, int* err, cudaStream_t cs) {
  SlotMaps maps;
  memset(&maps, 0, sizeof(maps));
  const int64_t rows = nha_chunk_count_bound(d->Ttot, d->N) * d->H * 64;
  maps.use = d->M == 64 && rows < (int64_t)1 << 31 && make_map_rows_heads(&maps.qg, d->q_gsa, d->Ttot, d->HQ, 64) &&
             make_map_rows_heads(&maps.kg, d->k_gsa, d->Ttot, d->H, 64) && make_map_rows_heads(&maps.v, d->v, d->Ttot, d->H, 64) &&
             make_map_rows_heads(&maps.g, d->g, d->Ttot, d->H, 64) && make_map_rows_heads(&maps.s, d->s, d->Ttot, d->H, 64) &&
             make_map_rows_heads(&maps.dout, d->d_o, d->Ttot, d->HQ, 64) && make_map_rows_heads(&maps.o, d->o, d->Ttot, d->HQ, 64) &&
             make_map_matrix(&maps.hk, d->hk_chunks, rows, 64, 64) && make_map_matrix(&maps.hv, d->hv_chunks, rows, 64, 64) &&
             make_map_rows_heads(&maps.dq, d->dq_gsa, d->Ttot, d->HQ, 64) && make_map_rows_heads(&maps.dk, d->dk_gsa, d->Ttot, d->H, 64) &&
             make_map_rows_heads(&maps.ds, d->ds, d->Ttot, d->H, 64) && make_map_rows_heads(&maps.dg, d->dg, d->Ttot, d->H, 64);
  const SlotPlan p = slot64_plan(d, dense_T);
  const bool one = d->HQ == d->H;
  if (p.scan) {
    const int st = one ? slot64_launch<true, true>(d, w, err, maps, 1, false, cs) : slot64_launch<false, true>(d, w, err, maps, 1, false, cs);
    if (st != NHA_OK) return st;
    bwd_state_scan_launch(d, w, p.win, cs);
    const int sc = check_launch();
    if (sc != NHA_OK) return sc;
  }
  return one ? slot64_launch<true, false>(d, w, err, maps, p.win, p.scan, cs) : slot64_launch<false, false>(d, w, err, maps, p.win, p.scan, cs);
}

}  // namespace nha
