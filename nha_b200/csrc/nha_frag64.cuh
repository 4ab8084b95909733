// Building blocks of the chunk kernels with 64-row products: those at head dim 64, the query-row and window-key passes of the
// backward at head dim 128.
//
// The accumulator of a product with M = 64 fills only the first 16 lanes of each tensor-memory quarter, so a warp that reads
// it with one row per lane leaves half of its lanes without work.  These kernels read it with tcgen05.ld.16x256b, which spreads
// the 16 rows over all 32 lanes in the layout of an mma.sync accumulator: lane (gq, tq) = (lane / 4, lane % 4) holds rows gq
// and gq + 8 and the columns 8 j + 2 tq, + 1.  The same fragment is what stmatrix and ldmatrix move between registers and the
// 128-byte-swizzled operand tiles, 16 bytes per lane.  Eight warps: warp w has the 16 rows of quarter w & 3 and the 32
// columns of half w >> 2.
//
// The running sum of the gates is a product, too: x[t,m] = G_t - Gend/2 = sum_i (i <= t ? 1/2 : -1/2) g'_i with the coefficients
// exact in bf16, which leaves every thread with exactly the decay exponents of its own rows and slots (no table in shared
// memory, no scan along the rows; the scan was 40 % of these kernels' time).
#pragma once

#include "nha_common.cuh"
#include "nha_tma.cuh"
#include "nha_umma.cuh"

namespace nha {
namespace f64 {

using namespace umma;

constexpr int kThreads = 256;
constexpr int kTile = 8192;                        // [64][64] bf16 operand tile
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr uint32_t kOtherLanes = 16u << 16;        // tensor-memory address of lanes 16-31 of each quarter, where a second such accumulator fits

// 32 columns of the warp's 16 rows: v[4 j + e] = (row gq + 8 (e >> 1), column 8 j + 2 tq + (e & 1))
__device__ __forceinline__ void frag_ld_nowait(uint32_t taddr, float (&v)[16]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void frag_ld(uint32_t taddr, float (&v)[16]) {
  frag_ld_nowait(taddr, v);
  tmem_ld_wait();
}
// 16 columns: v[4 j + e], j = 0, 1
__device__ __forceinline__ void frag_ld8_nowait(uint32_t taddr, float (&v)[8]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}
// 8 columns: v[e]
__device__ __forceinline__ void frag_ld4_nowait(uint32_t taddr, float (&v)[4]) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x1.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void frag_st8(uint32_t taddr, const float (&v)[8]) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]),
               "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// the reverse (rescaling an accumulator in place)
__device__ __forceinline__ void frag_st(uint32_t taddr, const float (&v)[16]) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]),
      "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
      "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ uint32_t pair_bf16(float lo, float hi) {
  const __nv_bfloat162 h2 = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h2);
}
__device__ __forceinline__ float2 pair_f32(uint32_t u) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u)); }

// This lane's row address of the four 8x8 blocks (rows 0-7 / 8-15 of the quarter x two blocks of 8 columns) that one
// stmatrix / ldmatrix moves, as an offset into a swizzled tile; block column pair jp (0, 1) of the warp's 32 columns.
__device__ __forceinline__ uint32_t frag_off(int quarter, int half, int lane, int jp) {
  const int mtx = lane >> 3, r = lane & 7, c = 4 * half + 2 * jp + (mtx >> 1);
  return (uint32_t)(quarter * 2048 + (mtx & 1) * 1024 + r * 128 + ((c ^ r) << 4));
}
__device__ __forceinline__ void stm4(uint32_t saddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(saddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void ldm4(uint32_t saddr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(saddr) : "memory");
}
// 16 x 16: one column pair
__device__ __forceinline__ void frag8_to_tile(uint32_t o, const float (&v)[8]) {
  stm4(o, pair_bf16(v[0], v[1]), pair_bf16(v[2], v[3]), pair_bf16(v[4], v[5]), pair_bf16(v[6], v[7]));
}
// the warp's 16 x 32 block of a tile from fp32 fragments (o0, o1: frag_off of the two column pairs + the tile's address)
__device__ __forceinline__ void frag_to_tile(uint32_t o0, uint32_t o1, const float (&v)[16]) {
  stm4(o0, pair_bf16(v[0], v[1]), pair_bf16(v[2], v[3]), pair_bf16(v[4], v[5]), pair_bf16(v[6], v[7]));
  stm4(o1, pair_bf16(v[8], v[9]), pair_bf16(v[10], v[11]), pair_bf16(v[12], v[13]), pair_bf16(v[14], v[15]));
}

// one product of 64-deep operands, descriptors formed by the caller: K-major operands advance by 32 bytes a k step, MN-major
// ones (AMN / BMN) by 16 rows
template <int AMN, int BMN>
__device__ __forceinline__ void mma64(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool acc) {
#pragma unroll
  for (int ks = 0; ks < 4; ++ks) mma_f16(d, a + (uint64_t)(ks * (AMN ? 128 : 2)), b + (uint64_t)(ks * (BMN ? 128 : 2)), idesc, acc || ks > 0);
}
__device__ __forceinline__ uint32_t idesc64(int amn, int bmn, int n = 64) { return make_idesc(64, n, bmn) | ((uint32_t)amn << 15); }

// adds to two fp32 words of memory without reading them into the thread (their only writer is this thread, which wrote them before)
__device__ __forceinline__ void red_add2(float* p, float x, float y) {
  asm volatile("red.relaxed.gpu.global.add.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(x), "f"(y) : "memory");
}

// rows r and r + 32 of a [64][64] tile, piece c (r = tid / 8, c = tid % 8); off = sw_off(r, c)
__device__ __forceinline__ void tile_in(unsigned char* tile, uint32_t off, const bf16* p0, bool ok0, const bf16* p1, bool ok1) {
  cp16(tile + off, p0, ok0);
  cp16(tile + off + 4096, p1, ok1);
}

// coefficients of x = G - Gend / 2: row t has 1/2 up to column t and -1/2 after it
__device__ __forceinline__ void fill_half_signs(unsigned char* tile, int tid) {
  const int r = tid >> 2;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int c = 2 * (tid & 3) + u;
    uint32_t pr[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 8 * c + 2 * e;
      pr[e] = (i <= r ? 0x3F00u : 0xBF00u) | (i + 1 <= r ? 0x3F000000u : 0xBF000000u);
    }
    *reinterpret_cast<uint4*>(tile + sw_off(r, c)) = make_uint4(pr[0], pr[1], pr[2], pr[3]);
  }
}

// barrier of the two warps that share the rows of a quarter
__device__ __forceinline__ void quarter_sync(int quarter) { asm volatile("bar.sync %0, 64;" ::"r"(quarter + 1) : "memory"); }

}  // namespace f64
}  // namespace nha
