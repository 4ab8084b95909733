// Streaming variant of the fused NHA decode step (sm_100a) for the common shapes: K == V in {64, 128},
// window keys in the cache (not caller-supplied logits).
//
// A (sequence, kv head) is cut into SPLITS CTAs so that the GPU is filled (two CTAs per SM); split s owns a contiguous
// range of window keys and of slots.  Inside a CTA every WARP works on its own, with a softmax of its own (running maximum,
// unnormalised weights); the only block barriers are the one behind the small inputs and those of the final merge.
//   * Slot memory: a warp takes eight slots.  Its hk columns and hv rows are updated in registers and stored; the slot
//     logits of all query heads are summed over the lanes by a halving exchange, and the readout of the warp's slots joins
//     the warp's window output.
//   * Window: the warps share the split's keys, those with slots taking fewer (a task of eight slots counts as kSlotCost
//     groups of eight keys).  A warp walks its keys eight at a time, keys and values side by side, each fetched by 16-byte
//     asynchronous copies into rings of two key and two value slots that only this warp touches.  S = q K^T by mma.sync
//     m16n8k16 with the keys as the n dimension: the order of the features inside a product is free as long as q and K
//     agree, so a lane takes 16 consecutive bytes of its key row (two k steps), no ldmatrix is needed, and the two halves
//     that rotate-half pairs up lie in the same lane, where they are rotated on their way from shared memory to the product.
//     At D = 128 a lane's two pieces of a half are neighbours: a row of the tables is then read 32 bytes a lane, four lanes to a
//     whole line, in half the requests.
//     O^T = V^T P^T by m16n8k8: the accumulator layout of S is the B fragment of P^T as it stands, the heads are the n
//     dimension (a group of up to eight heads wastes nothing), V^T is packed from two value rows by byte permutes.
//   * Under dependent launch a CTA asks for its share of the window and of the slot memory (contiguous pieces, bulk prefetch
//     into L2) before it waits for the kernel in front: a prefetch has no value to get wrong.  The slot memory is therefore
//     read last, from L2, while the first window loads go out at once.  The small inputs are asked for first: behind the
//     window they would arrive last and hold up everything.
//   * The warps' outputs are merged in shared memory, the splits through the cluster's shared memory (2, 4 or 8 splits)
//     or by the last CTA of a (sequence, kv head) to arrive (a ticket in global memory).
//
// What bounds it: the chain of a CTA, about 4 us whatever it holds, and the requests to the first-level cache (table rows, window,
// state), not the instructions: a version with half of them, sixteen keys a step, was slower.  32 sequences, HQ 32, H 4, D 128, W 512:
// 17.3 -> 16.3 us a layer with 32-byte table loads and the small inputs fetched ahead (48 % of the copy rate).  Without the table loads
// 2.2 us less, without the slot memory 3.8, without the window 5.2.  Measured per layer in a stack, against
// a version that formed all logits of a CTA first and requested the values only when the keys had been used: 32 sequences,
// HQ 32, H 4, D 128, W 512: 18.8 -> 17.3 us; H 8: 41.8 -> 25.9 us (3.9 TB/s); the same on rings 47.1 -> 28.7 us; 64 sequences,
// H 8, W 64: 41.4 -> 26.1 us; one sequence, H 16, D 64, W 64: 7.3 -> 5.0 us.
//
// Replaces the two Triton launches of fused_recurrent_nha_decode
// (nha_fla/ops/nha/fused_recurrent.py:229-353 k-kernel, :356-428 v-kernel).
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <type_traits>
#include <atomic>

#include "nha_common.cuh"
#include "nha_umma.cuh"

namespace nha {

constexpr int kStrThreads = 256;
constexpr int kStrWarps = kStrThreads / 32;
constexpr int kGroup = 8;                // keys of one step of a warp, slots of one task of a warp
constexpr int kAhead = 4;                // loads a warp keeps in flight: keys and values of two steps
template <int D> constexpr int kLdq = D == 128 ? D + 8 : D + 32;   // row pitch of the rotated query
constexpr int kMinKeys = 128;            // a split holds at least this many window keys: a CTA costs about 4 us whatever it holds
constexpr int kSlotCost = 4;             // eight slots cost a warp about as much as this many groups of eight keys

struct DecodeStreamArgs {
  const bf16* q; const bf16* sq; const bf16* k; const bf16* v; const bf16* g; const bf16* s;
  const bf16* sw_k; const bf16* sw_v; const bf16* cosp; const bf16* sinp;
  float* hk; float* hv; bf16* o;
  float* part_o;      // [B*H, SPLITS, NG, V] unnormalised partial outputs
  float* part_ml;     // [B*H, SPLITS, NG, 2] maximum and sum of each split
  int* tickets;       // [B*H] arrival counters, zero between calls
  // ring mode (head != NULL): sw_k / sw_v are rings of W physical rows per sequence whose oldest entry sits at
  // row head[b]; that entry is the token that leaves the window and enters the slot memory in this step (its
  // gate row comes from ring_g, the popped k / v from the rings), the token of this step (k, v: not yet in the
  // ring) is the newest window entry
  const int* head; const bf16* ring_g;
  // ring_kraw != NULL (ring mode only): sw_k is a ring of keys that were rotated when they entered it (rotary by
  // absolute position does not change while the window slides), so only the token of this step is rotated here;
  // the raw key that enters the slot memory comes from ring_kraw
  const bf16* ring_kraw;
  // fused append (ring mode, raw keys): g_new != NULL makes the CTA that merges the splits of a (sequence, kv head)
  // also store the step's token (k, v, g_new) over the entry that left the window (or into the next free row of a
  // filling ring) and advance that kv head's index.  `head` then holds one index per (sequence, kv head), [B*H]: every
  // (sequence, kv head) is finished by exactly one CTA, after all its splits have read the rings, so no other CTA
  // reads the index or the row that is overwritten.
  const bf16* g_new;
  int64_t cs_batch, cs_row;
  int WR;             // rows of a ring (W outside ring mode)
  // the rings are still filling - they hold the W - 1 oldest window entries in rows 0 .. W - 2, nothing leaves the window and the
  // slot memory keeps its value
  int nopop;
  int state_bf16;     // hk and hv point to bf16 tensors (half the state bytes; arithmetic stays fp32 in registers)
  int zero_state;
  bool ahead;         // the window goes into L2 ahead of its use
  bool tab32;         // rows of the rotary tables start on 32 bytes
  int cluster;        // the SPLITS CTAs of a (sequence, kv head) form a thread-block cluster and merge through shared memory
  // programmatic dependent launch: 0 = plain launch; 1 = the grid may be scheduled before the kernel in front of it on
  // the stream has finished and waits for it before its first global read (it only prefetches into L2 before that); 2 = as 1,
  // but the first window loads of this call go out BEFORE that wait (the caller asserts that the kernel in front writes
  // neither the window nor the slot memory)
  int pdl;
  int B, HQ, H, M, W, NG, SPLITS, KSPL, MQ;
  float scale;
  int off_ring, off_q, off_sqA, off_p, off_eg, off_sv, off_kpop, off_vpop, off_wml, off_ml, off_out;
};
// The host's part of a dependent launch depends on the size of the argument block.  Us a launch of an empty kernel, median of 41 rounds
// with the sizes in random order, spread 0.06: 240 to 272 bytes 1.95-2.00, 280 to 288 1.64, 292 to 336 1.94-2.02 (driver 580.159).  A step
// of 24 layers for one sequence, which the host bounds: 132.7 us with 288 bytes, 137.3 with 296.  Hence `bool` twice.
static_assert(sizeof(DecodeStreamArgs) >= 280 && sizeof(DecodeStreamArgs) <= 288, "another size costs 0.3 us a launch: measure it");

// four elements of the slot memory, fp32 or bf16 storage
template <bool SB16>
__device__ __forceinline__ float4 ld_state4(const float* base, size_t idx) {
  if (!SB16) return *reinterpret_cast<const float4*>(base + idx);
  const uint2 raw = *reinterpret_cast<const uint2*>(reinterpret_cast<const bf16*>(base) + idx);
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}
template <bool SB16>
__device__ __forceinline__ void st_state4(float* base, size_t idx, float4& v) {
  if (!SB16) {
    *reinterpret_cast<float4*>(base + idx) = v;
    return;
  }
  uint2 pk;
  *reinterpret_cast<__nv_bfloat162*>(&pk.x) = __floats2bfloat162_rn(v.x, v.y);
  *reinterpret_cast<__nv_bfloat162*>(&pk.y) = __floats2bfloat162_rn(v.z, v.w);
  *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(base) + idx) = pk;
  const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pk.x));
  const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pk.y));
  v = make_float4(lo.x, lo.y, hi.x, hi.y);       // the rounded value is the state from here on
}
// thread-block cluster: barrier over all threads of all CTAs, and loads from another CTA's shared memory
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_map(const void* p, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(umma::smem_u32(p)), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ float2 ld_cluster_f2(uint32_t addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr) : "memory");
  return v;
}

// 32 bytes of constant memory at a 32-byte boundary, in one load
__device__ __forceinline__ void ld32(const void* p, uint4& x, uint4& y) {
  asm volatile("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w), "=r"(y.x), "=r"(y.y), "=r"(y.z), "=r"(y.w) : "l"(p));
}
// the line of an address into L2
__device__ __forceinline__ void prefetch_line(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// start of a 16-byte aligned range into L2
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// c[16x8] += a[16x16] b[16x8]
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// c[16x8] += a[16x8] b[8x8]
__device__ __forceinline__ void mma_1688(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(b0));
}

// shared-memory row pitches of a warp's ring slots, in bytes: 16-byte pieces of eight lanes (rows gq, pieces of lane tq for keys
// and the rotated query, see key_piece; rows 2 tq, pieces gq for values) fall into eight different bank groups
template <int D> struct DecodeRing {
  static constexpr int kKRow = D == 128 ? D * 2 + 16 : D * 2 + 64, kVRow = D * 2 + 16;
  static constexpr int kKSlot = kGroup * kKRow, kVSlot = kGroup * kVRow;
  static constexpr int kWarp = 2 * (kKSlot + kVSlot);              // two key slots, two value slots
};

// first feature of piece i of lane tq (i < D / 32; pieces i and i + D / 64 are rotated with each other): at D = 128 the two pieces of
// a half are neighbours, so that a table row is read 32 bytes a lane in whole lines
template <int D> __device__ __forceinline__ constexpr int key_piece(int tq, int i) {
  return D == 128 ? 16 * tq + 8 * (i & 1) + 64 * (i >> 1) : 8 * tq + 32 * i;
}

__device__ __forceinline__ void store_row4(bf16* o, const float4& x) {
  uint2 pk;
  *reinterpret_cast<__nv_bfloat162*>(&pk.x) = __floats2bfloat162_rn(x.x, x.y);
  *reinterpret_cast<__nv_bfloat162*>(&pk.y) = __floats2bfloat162_rn(x.z, x.w);
  *reinterpret_cast<uint2*>(o) = pk;
}

// The merges of a (sequence, kv head) that several CTAs share.  They are the last link of the call's chain: their loads are asked for together.  Us a
// layer in a graph of 16, one load waited for at a time | so: one sequence, 16 heads of 64, W 256 (two CTAs) 5.26 | 5.1, W 512 (four) 5.5 | 4.7,
// W 1200 (eight) 7.4 | 5.5; 28 heads of 128 on 4, W 512 7.43 | 6.7, W 1200 8.60 | 6.9; through the workspace, W 1200, 12.6-14.6 | 7.8-9.4.
// INLINE where the rest of the kernel is small (one head a kv head): as functions they cost 0.2-0.3 us there (5.3, 5.0, 5.8 us of the first three
// above; 4 sequences, 16 heads of 128, W 64, not shared, 7.05 us beside the functions, 6.75 without).  Elsewhere functions, so that the registers and
// the code in front of them are the same whether they run or not: 8 layers of 32 sequences on rings, HQ 32, H 8, W 512, not shared either, 26.3 us
// a layer with the merges inline, 25.6 so.

// From the shared memory of the cluster's CTAs: ml [NG][2] maxima and sums, outp [NG][V] partial outputs; at most eight of them.
template <int V, int NT>
__device__ __forceinline__ void merge_cluster_inline(const float* ml, const float* outp, bf16* o, int NG, int SPL) {
  constexpr int V4 = V / 4;
#pragma unroll 1
  for (int u = 0; u < NT; ++u) {
    const int i = threadIdx.x + u * kStrThreads;
    if (i >= NG * V4) return;
    const int qh = i / V4, c = i - qh * V4;
    float mx = -INFINITY, den = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float2 t2[8];
#pragma unroll
    for (int s2 = 0; s2 < 8; ++s2) t2[s2] = s2 < SPL ? ld_cluster_f2(cluster_map(ml + 2 * qh, s2)) : make_float2(-INFINITY, 0.f);
#pragma unroll
    for (int s2 = 0; s2 < 8; ++s2) mx = fmaxf(mx, t2[s2].x);
#pragma unroll
    for (int s4 = 0; s4 < 8; s4 += 4) {
      if (s4 >= SPL) break;
      float4 pv[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) pv[k] = s4 + k < SPL ? ld_cluster_f4(cluster_map(outp + qh * V + 4 * c, s4 + k)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float w2 = t2[s4 + k].x > -INFINITY ? __expf(t2[s4 + k].x - mx) : 0.f;
        den += t2[s4 + k].y * w2;
        acc.x += w2 * pv[k].x; acc.y += w2 * pv[k].y; acc.z += w2 * pv[k].z; acc.w += w2 * pv[k].w;
      }
    }
    const float inv = 1.0f / den;
    store_row4(o + qh * V + 4 * c, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
  }
}

// From the workspace: all_ml [SPL][NG][2], all_o [SPL][NG][V]; wgt: [SPL][NG] floats of shared memory.
template <int V, int NT>
__device__ __forceinline__ void merge_workspace_inline(const float* all_ml, const float* all_o, float* wgt, bf16* o, int NG, int SPL) {
  constexpr int V4 = V / 4;
  const int tid = threadIdx.x;
  if (SPL <= 4) {
    // few splits: a thread fetches the maxima, sums and partial outputs of its element in one go (one trip to L2)
    // and forms the merge weights itself
#pragma unroll
    for (int u = 0; u < NT; ++u) {
      const int i = tid + u * kStrThreads;
      if (i < NG * V4) {
        const int qh = i / V4, c = i - qh * V4;
        float4 pv[4];
        float m2[4], l2[4];
#pragma unroll
        for (int s2 = 0; s2 < 4; ++s2) {
          if (s2 < SPL) {
            pv[s2] = __ldcg(reinterpret_cast<const float4*>(all_o + ((size_t)s2 * NG + qh) * V + 4 * c));
            const float2 t2 = __ldcg(reinterpret_cast<const float2*>(all_ml + ((size_t)s2 * NG + qh) * 2));
            m2[s2] = t2.x; l2[s2] = t2.y;
          } else {
            pv[s2] = make_float4(0.f, 0.f, 0.f, 0.f);
            m2[s2] = -INFINITY; l2[s2] = 0.f;
          }
        }
        const float mx = fmaxf(fmaxf(m2[0], m2[1]), fmaxf(m2[2], m2[3]));
        float wq[4], den = 0.f;
#pragma unroll
        for (int s2 = 0; s2 < 4; ++s2) {
          wq[s2] = m2[s2] > -INFINITY ? __expf(m2[s2] - mx) : 0.f;
          den += l2[s2] * wq[s2];
        }
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int s2 = 0; s2 < 4; ++s2) {
          const float w2 = wq[s2] / den;
          acc.x += w2 * pv[s2].x; acc.y += w2 * pv[s2].y; acc.z += w2 * pv[s2].z; acc.w += w2 * pv[s2].w;
        }
        store_row4(o + qh * V + 4 * c, acc);
      }
    }
    return;
  }
  // merge weights exp(m_s - m) / denominator
  for (int qh = tid; qh < NG; qh += kStrThreads) {
    float mx = -INFINITY;
    for (int s2 = 0; s2 < SPL; ++s2) mx = fmaxf(mx, __ldcg(all_ml + ((size_t)s2 * NG + qh) * 2));
    float den = 0.f;
    for (int s2 = 0; s2 < SPL; ++s2) {
      const float m2 = __ldcg(all_ml + ((size_t)s2 * NG + qh) * 2);
      const float l2 = __ldcg(all_ml + ((size_t)s2 * NG + qh) * 2 + 1);
      den += m2 > -INFINITY ? l2 * __expf(m2 - mx) : 0.f;
    }
    for (int s2 = 0; s2 < SPL; ++s2) {
      const float m2 = __ldcg(all_ml + ((size_t)s2 * NG + qh) * 2);
      wgt[s2 * NG + qh] = m2 > -INFINITY ? __expf(m2 - mx) / den : 0.f;
    }
  }
  __syncthreads();
  for (int i = tid; i < NG * V4; i += kStrThreads) {
    const int qh = i / V4, c = i - qh * V4;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int s2 = 0; s2 < SPL; ++s2) {
      const float wq = wgt[s2 * NG + qh];
      const float4 pv = __ldcg(reinterpret_cast<const float4*>(all_o + ((size_t)s2 * NG + qh) * V + 4 * c));
      acc.x += wq * pv.x; acc.y += wq * pv.y; acc.z += wq * pv.z; acc.w += wq * pv.w;
    }
    store_row4(o + qh * V + 4 * c, acc);
  }
}

template <int V, int NT>
__device__ __noinline__ void merge_cluster_call(const float* ml, const float* outp, bf16* o, int NG, int SPL) { merge_cluster_inline<V, NT>(ml, outp, o, NG, SPL); }
template <int V, int NT>
__device__ __noinline__ void merge_workspace_call(const float* all_ml, const float* all_o, float* wgt, bf16* o, int NG, int SPL) {
  merge_workspace_inline<V, NT>(all_ml, all_o, wgt, o, NG, SPL);
}
template <int V, int NT, bool INLINE>
__device__ __forceinline__ void merge_cluster(const float* ml, const float* outp, bf16* o, int NG, int SPL) {
  if constexpr (INLINE) merge_cluster_inline<V, NT>(ml, outp, o, NG, SPL);
  else merge_cluster_call<V, NT>(ml, outp, o, NG, SPL);
}
template <int V, int NT, bool INLINE>
__device__ __forceinline__ void merge_workspace(const float* all_ml, const float* all_o, float* wgt, bf16* o, int NG, int SPL) {
  if constexpr (INLINE) merge_workspace_inline<V, NT>(all_ml, all_o, wgt, o, NG, SPL);
  else merge_workspace_call<V, NT>(all_ml, all_o, wgt, o, NG, SPL);
}

// HB: heads that the slot part of a tile of eight is compiled for (1, 4 or 8).  The kernel is straight-line code that a CTA runs once, and
// code that an SM has not run before comes at 2 cycles an instruction up to 64 KB and at 4.7 and more from 96; with the padding heads out of it and the
// loops whose length the compiler does not know kept as loops it is 49-68 KB instead of 97-105 at four heads (8 layers of 32 sequences on
// rings, HQ 32, H 8, W 512: 211.3 -> 204.3 us), 66 at eight (calls that are not split: no difference there).
template <int D, int NT, int HB, bool SB16, bool RING>
__global__ void __launch_bounds__(kStrThreads, NT == 1 ? 2 : 1) nha_decode_stream_kernel(const DecodeStreamArgs a) {
  extern __shared__ __align__(128) unsigned char smem[];
  typedef DecodeRing<D> RG;
  constexpr int K = D, V = D, ldq = kLdq<D>, NH = 8 * NT;           // NH: heads, padded to the products' n tiles
  constexpr int V4 = V / 4, kRowsI = 32 / V4;                      // lanes of an hv row; hv rows a warp touches at once
  constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
  float* qT = reinterpret_cast<float*>(smem + a.off_q);            // [K][NH] raw query, fp32 (columns >= NG zero)
  bf16* sqA = reinterpret_cast<bf16*>(smem + a.off_sqA);           // [16][ldq] rotated query (rows >= NG zero)
  float* eg = reinterpret_cast<float*>(smem + a.off_eg);
  float* sv = reinterpret_cast<float*>(smem + a.off_sv);
  float* kpop = reinterpret_cast<float*>(smem + a.off_kpop);
  float* vpop = reinterpret_cast<float*>(smem + a.off_vpop);
  float* wml = reinterpret_cast<float*>(smem + a.off_wml);         // [warps][NH][4] max and sum of the slots, of the window
  float* ml = reinterpret_cast<float*>(smem + a.off_ml);           // [NG][2] of the split (natural units)
  float* outp = reinterpret_cast<float*>(smem + a.off_out);        // [NG][V] partial output of the split

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int SPL = a.SPLITS, NG = a.NG, M = a.M, W = a.W, MQ = a.MQ;
  const int bh = blockIdx.x / SPL, sp = blockIdx.x % SPL;
  const int b = bh / a.H, h = bh % a.H;
  const bool rotary = a.cosp != nullptr;
  const int m0 = sp * MQ;
  const int nslots = max(0, min(MQ, M - m0));
  const int ntask = (nslots + kGroup - 1) / kGroup;                // tasks of eight slots, at most one a warp
  // this warp's keys: logical window positions [wk0, wk0 + nk), eight at a time
  int wk0, nk;
  {
    const int skeys = max(0, min(a.KSPL, W - sp * a.KSPL)), sgrp = (skeys + kGroup - 1) / kGroup;
    const int busy = min(ntask, kStrWarps), free_ = kStrWarps - busy;
    // groups of a warp without slots and of one with: the difference is kSlotCost as far as there are groups for it
    int gf = (sgrp + busy * kSlotCost + kStrWarps - 1) / kStrWarps;
    int gb = max(0, gf - kSlotCost);
    if (free_ * gf + busy * gb < sgrp) gb = (sgrp - free_ * gf + busy - 1) / max(busy, 1);
    const int first = warp < busy ? warp * gb : busy * gb + (warp - busy) * gf;
    const int last = min(sgrp, first + (warp < busy ? gb : gf));
    wk0 = sp * a.KSPL + min(first, sgrp) * kGroup;
    nk = max(0, min(last * kGroup, skeys) - first * kGroup);
  }
  const int ngrp = (nk + kGroup - 1) / kGroup;
  const int WR = a.WR;
  if (a.pdl) {
    // The window and the slot memory of this call go into L2 while the kernel in front is still draining.  A prefetch has
    // no value to get wrong, L2 is where the kernel in front writes, and it also brings the address translations in.
    // The CTAs of a sequence share its window, which is contiguous over the heads, and those of a (sequence, kv head) its state.
    const int64_t wbytes = (int64_t)WR * a.H * D * 2, part = (wbytes / (a.H * SPL)) & ~(int64_t)15;
    const int64_t sbytes = (int64_t)K * M * (SB16 ? 2 : 4), spart = (sbytes / SPL) & ~(int64_t)15;
    const int idx = h * SPL + sp;
    // The small inputs too, in front of all that: behind the rest of the window a miss in L2 takes longer than the rest of the prologue
    // (32 sequences, HQ 32, H 4, D 128, W 512, inputs in memory: 4.9 k cycles to the first barrier).
    if (warp == 4) {
      auto lines = [&](const void* p, int bytes) {
#pragma unroll 1
        for (int at = lane * 128; at < bytes; at += 32 * 128) prefetch_line((const char*)p + at);
      };
      lines(a.q + ((size_t)b * a.HQ + h * NG) * K, NG * K * 2);
      if (rotary) {
        lines(a.cosp + b * a.cs_batch + (int64_t)(W - 1) * a.cs_row, K * 2);
        lines(a.sinp + b * a.cs_batch + (int64_t)(W - 1) * a.cs_row, K * 2);
      } else {
        lines(a.sq + ((size_t)b * a.HQ + h * NG) * K, NG * K * 2);
      }
      if (!RING) lines(a.g + (size_t)bh * M, M * 2);
      lines(a.k + (size_t)bh * K, K * 2);
      lines(a.v + (size_t)bh * V, V * 2);
    }
    if (warp < 4) {
      const bool win = warp < 2;
      const char* base = win ? (const char*)(warp == 0 ? a.sw_k : a.sw_v) + b * wbytes + idx * part
                             : (const char*)(warp == 2 ? a.hk : a.hv) + bh * sbytes + sp * spart;
      const int64_t n = win ? (a.ahead ? part : 0) : (a.zero_state ? 0 : spart);
#pragma unroll 1
      for (int64_t at = lane * 4096; at < n; at += 32 * 4096) prefetch_l2(base + at, (uint32_t)min((int64_t)4096, n - at));
    }
  }
  if (a.pdl == 1) {                                                // before the first global read
    grid_dep_wait();
    grid_dep_launch();
  }
  const int hd = RING ? (a.nopop ? -1 : a.head[a.g_new ? bh : b]) : 0;   // physical row of the oldest ring entry
  // the token that enters the slot memory: separate small tensors, or the oldest ring entry
  const bool prerot = RING && a.ring_kraw != nullptr;
  const bf16* kpop_g = RING ? (prerot ? a.ring_kraw : a.sw_k) + (((size_t)b * WR + max(hd, 0)) * a.H + h) * D
                              : a.k + (size_t)bh * D;
  const bf16* vpop_g = RING ? a.sw_v + (((size_t)b * WR + max(hd, 0)) * a.H + h) * D : a.v + (size_t)bh * D;
  const bf16* gpop_g = RING ? a.ring_g + (((size_t)b * WR + max(hd, 0)) * a.H + h) * M : a.g + (size_t)bh * M;
  // the step's token into the rings (called by the one CTA that finishes this (sequence, kv head))
  auto append_token = [&]() {
    if (!RING || !a.g_new) return;
    const int row = a.nopop ? W - 1 : hd;                          // a filling ring holds W - 1 entries: next free row
    const size_t at = ((size_t)b * WR + row) * a.H + h;
    uint4* rk = reinterpret_cast<uint4*>(const_cast<bf16*>(a.sw_k) + at * D);
    uint4* rv = reinterpret_cast<uint4*>(const_cast<bf16*>(a.sw_v) + at * D);
    uint4* rg = reinterpret_cast<uint4*>(const_cast<bf16*>(a.ring_g) + at * M);
    const uint4* kn = reinterpret_cast<const uint4*>(a.k + (size_t)bh * D);
    const uint4* vn = reinterpret_cast<const uint4*>(a.v + (size_t)bh * D);
    const uint4* gn = reinterpret_cast<const uint4*>(a.g_new + (size_t)bh * M);
    const int nd = D / 8, ng = M / 8;
#pragma unroll 1
    for (int i = tid; i < 2 * nd + ng; i += kStrThreads) {
      if (i < nd) rk[i] = kn[i];
      else if (i < 2 * nd) rv[i - nd] = vn[i - nd];
      else rg[i - 2 * nd] = gn[i - 2 * nd];
    }
    if (tid == 0 && !a.nopop) const_cast<int*>(a.head)[bh] = hd + 1 == WR ? 0 : hd + 1;
  };

  // Load j of this warp: keys (j even) or values (j odd) of its group j / 2, into slot (j / 2) & 1 of that kind.  A lane
  // always copies the same 16-byte column; rows past the warp's keys are zero-filled.  One commit group per load: groups
  // complete in order, which is the order they are used in.
  unsigned char* ring = smem + a.off_ring + warp * RG::kWarp;
  constexpr int kC8 = D / 8;                                       // 16-byte columns of a row
  constexpr int kRStep = 32 / kC8;                                 // rows between two copies of a lane
  const int lc = lane % kC8, lr = lane / kC8;
  const uint32_t rpitch = a.H * D;
  const bf16* kbase = a.sw_k + ((size_t)b * WR * a.H + h) * D + 8 * lc;
  const bf16* vbase = a.sw_v + ((size_t)b * WR * a.H + h) * D + 8 * lc;
  // (rows past the warp's keys repeat its last one: their logits are masked and their weights are zero.  Every call commits
  // a group, empty past the last load: a warp always has kAhead groups behind the one it waits for.)
  const int rlast = wk0 + nk - 1;
  auto issue = [&](int g, auto kind) {
    constexpr int kv = decltype(kind)::value, pitch = kv ? RG::kVRow : RG::kKRow;
    if (g < ngrp) {
      const bf16* base = kv ? vbase : kbase;
      unsigned char* dst = ring + (kv ? 2 * RG::kKSlot : 0) + (g & 1) * (kv ? RG::kVSlot : RG::kKSlot) + 16 * lc + lr * pitch;
      const int r0 = wk0 + g * kGroup + lr;
#pragma unroll
      for (int i = 0; i < kGroup / kRStep; ++i) {
        int row = min(r0 + i * kRStep, rlast);                     // logical window index, then physical row
        const bf16* src;
        if (RING) {
          const bool fresh = row == W - 1;                         // the token of this step
          row += hd + 1;
          row -= row >= WR ? WR : 0;
          src = fresh ? (kv ? a.v : a.k) + (size_t)bh * D + 8 * lc : base + (uint64_t)((uint32_t)row) * rpitch;
        } else {
          src = base + (uint64_t)((uint32_t)row) * rpitch;
        }
        umma::cp16(dst + i * kRStep * pitch, src, true);
      }
    }
    umma::cp_commit();
  };
  constexpr std::integral_constant<int, 0> kKeys{};
  constexpr std::integral_constant<int, 1> kValues{};
  // wait until the oldest load in flight has landed: the kAhead - 1 issued after it may stay
  auto wait_load = [&]() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(kAhead - 1) : "memory");
    __syncwarp();                                                  // every lane's copies have landed
  };

  // ---- requests: the small inputs and the first window loads (the slot memory comes last, behind the window) -------------
  // hk of a task: lane -> slots 4 (lane & 1) .. + 3 of the eight, rows 16 i + lane / 2; hv: rows (slots) kRowsI u + lane / V4
  constexpr int kHk = K / 16, kHv = kGroup / kRowsI;
  const int hs = 4 * (lane & 1), hr = lane >> 1;
  const int vsub = lane / V4, vcol = 4 * (lane % V4);
  float4 hreg[kHk], vreg[kHv];
  auto load_state = [&]() {
    const int ms = kGroup * warp;
#pragma unroll
    for (int i = 0; i < kHk; ++i)
      hreg[i] = !a.zero_state && ms + hs < nslots ? ld_state4<SB16>(a.hk, ((size_t)bh * K + 16 * i + hr) * M + m0 + ms + hs)
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int u = 0; u < kHv; ++u)
      vreg[u] = !a.zero_state && ms + kRowsI * u + vsub < nslots
                    ? ld_state4<SB16>(a.hv, ((size_t)bh * M + m0 + ms + kRowsI * u + vsub) * V + vcol) : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  // Dependent launch with early requests (pdl == 2): the window of this call does not depend on the kernel in front, so its
  // first loads go out before the wait.  In ring mode the newest window entry is the token of
  // this step (a.k / a.v, written by the caller's projections): the loads from the first one that holds it on
  // are issued after the wait, in the same order as always.
  int npre = 0;                                                    // groups requested before the wait
  if (a.pdl == 2) {
    npre = kAhead / 2;
    if (RING && nk > 0 && wk0 + nk == W) npre = min(npre, ngrp - 1);
#pragma unroll 1
    for (int g = 0; g < npre; ++g) { issue(g, kKeys); issue(g, kValues); }
    grid_dep_wait();
    grid_dep_launch();
  }
  constexpr int c8h = K >> 4;
  const int qi = tid - 128, q_r = qi / c8h, q_c = qi - q_r * c8h;
  const bool qthread = tid >= 128 && qi < 16 * c8h, qlive = qthread && q_r < NG;
  uint4 rq_x = make_uint4(0u, 0u, 0u, 0u), rq_y = rq_x, rq_c1 = rq_x, rq_s1 = rq_x, rq_c2 = rq_x, rq_s2 = rq_x;
  if (qlive) {
    const bf16* qrow = a.q + ((size_t)b * a.HQ + h * NG + q_r) * K;
    rq_x = __ldg(reinterpret_cast<const uint4*>(qrow + 8 * q_c));
    rq_y = __ldg(reinterpret_cast<const uint4*>(qrow + 8 * (q_c + c8h)));
    if (rotary) {
      // the query position is the last row of the window tables
      const bf16* cq = a.cosp + b * a.cs_batch + (int64_t)(W - 1) * a.cs_row;
      const bf16* sn = a.sinp + b * a.cs_batch + (int64_t)(W - 1) * a.cs_row;
      rq_c1 = __ldg(reinterpret_cast<const uint4*>(cq + 8 * q_c));
      rq_s1 = __ldg(reinterpret_cast<const uint4*>(sn + 8 * q_c));
      rq_c2 = __ldg(reinterpret_cast<const uint4*>(cq + 8 * (q_c + c8h)));
      rq_s2 = __ldg(reinterpret_cast<const uint4*>(sn + 8 * (q_c + c8h)));
    } else {
      const bf16* srow = a.sq + ((size_t)b * a.HQ + h * NG + q_r) * K;
      rq_c1 = __ldg(reinterpret_cast<const uint4*>(srow + 8 * q_c));
      rq_c2 = __ldg(reinterpret_cast<const uint4*>(srow + 8 * (q_c + c8h)));
    }
  }
  // the gates (threads 0..63) and the popped token (one warp each for k and v)
  bf16 gb[2], sb[2];
  gb[0] = gb[1] = sb[0] = sb[1] = f2bf(0.f);
  uint4 rpop = make_uint4(0u, 0u, 0u, 0u);
  if (tid < 64) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int m = tid + 64 * u;
      if (m < nslots && !a.nopop) {
        gb[u] = gpop_g[m0 + m];
        if (a.s) sb[u] = a.s[(size_t)bh * M + m0 + m];
      }
    }
  } else if (tid < 96) {
    if (tid - 64 < (K >> 3) && !a.nopop) rpop = __ldg(reinterpret_cast<const uint4*>(kpop_g + 8 * (tid - 64)));
  } else if (tid < 128) {
    if (tid - 96 < (V >> 3) && !a.nopop) rpop = __ldg(reinterpret_cast<const uint4*>(vpop_g + 8 * (tid - 96)));
  }
#pragma unroll 1
  for (int g = npre; g < kAhead / 2; ++g) { issue(g, kKeys); issue(g, kValues); }
  // registers -> shared memory
  if (tid < 64) {
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int m = tid + 64 * u;
      if (m < MQ) {
        float e = 1.f, sm = 0.f;
        if (m < nslots) {
          e = __expf(bf2f(gb[u]));
          sm = a.s ? bf2f(sb[u]) : 1.0f - e;
        }
        eg[m] = e;
        sv[m] = sm;
      }
    }
  } else if (tid < 128) {
    const int i = (tid - 64) & 31;
    if (i < (K >> 3)) {
      float f[8];
      unpack8(rpop, f);
      float* dstp = tid < 96 ? kpop : vpop;
#pragma unroll
      for (int e = 0; e < 8; ++e) dstp[8 * i + e] = f[e];
    }
  } else if (qthread) {
    uint4 o1 = make_uint4(0u, 0u, 0u, 0u), o2 = o1;
    float x[8], y[8];
    unpack8(rq_x, x); unpack8(rq_y, y);
    if (qlive) {
      if (rotary) {
        float c1[8], s1[8], c2[8], s2[8], p1[8], p2[8];
        unpack8(rq_c1, c1); unpack8(rq_s1, s1); unpack8(rq_c2, c2); unpack8(rq_s2, s2);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          p1[e] = x[e] * c1[e] - y[e] * s1[e];
          p2[e] = y[e] * c2[e] + x[e] * s2[e];
        }
        o1 = pack8(p1); o2 = pack8(p2);
      } else {
        o1 = rq_c1; o2 = rq_c2;
      }
    }
    if (q_r < NH) {
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        qT[(8 * q_c + e) * NH + q_r] = x[e];
        qT[(8 * (q_c + c8h) + e) * NH + q_r] = y[e];
      }
    }
    *reinterpret_cast<uint4*>(sqA + q_r * ldq + 8 * q_c) = o1;
    *reinterpret_cast<uint4*>(sqA + q_r * ldq + 8 * (q_c + c8h)) = o2;
  }
  __syncthreads();
  const float sc2 = a.scale * kLog2e;
  // A warp raises its reference (and rescales its output) when a key exceeds it by this much (log2): the weights are rounded to bf16
  // for the product with the values, and the key a reference was taken from has the weight 1, which is exact.  Error of the output
  // against 64 bits, 32 heads on 4, D 128, W 512: 3.42e-3 with 8, 3.31e-3 with 1, 3.27e-3 with 0; 48 layers of 32 sequences 817, 823 and 828 us.
  constexpr float kRaise = 1.f;

  // ---- the window, eight keys at a time --------------------------------------------------------------------------------
  const int gq = lane >> 2, tq = lane & 3;                         // fragment coordinates of the lane
  float oacc[NT][D / 64][4][4];                                    // [heads 2 tq, 2 tq + 1 of tile t][columns 64 j + 8 gq + 2 u, + 1]
  float m_run[NT], l_run[NT];                                      // of head gq + 8 t
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    m_run[t] = -INFINITY;
    l_run[t] = 0.f;
#pragma unroll
    for (int j = 0; j < D / 64; ++j)
#pragma unroll
      for (int u = 0; u < 4; ++u) oacc[t][j][u][0] = oacc[t][j][u][1] = oacc[t][j][u][2] = oacc[t][j][u][3] = 0.f;
  }
  constexpr int kHalf = D / 64;                                    // 16-byte pieces of a lane in each half of a key row
  uint4 cs[kHalf][4];                                              // rotate-half table entries of the group's key gq
  const bf16* ctab = rotary ? a.cosp + b * a.cs_batch + key_piece<D>(tq, 0) : nullptr;
  const bf16* stab = rotary ? a.sinp + b * a.cs_batch + key_piece<D>(tq, 0) : nullptr;
  auto load_table = [&](int g) {
    const int lw = wk0 + min(g * kGroup + gq, nk - 1);
    if (prerot && lw != W - 1) return;                             // rotated ring: only the token of this step is rotated
    const uint64_t at = (uint64_t)(uint32_t)lw * (uint32_t)a.cs_row;
    if (D == 128 && a.tab32) {
      ld32(ctab + at, cs[0][0], cs[kHalf - 1][0]);
      ld32(stab + at, cs[0][1], cs[kHalf - 1][1]);
      ld32(ctab + at + D / 2, cs[0][2], cs[kHalf - 1][2]);
      ld32(stab + at + D / 2, cs[0][3], cs[kHalf - 1][3]);
      return;
    }
#pragma unroll
    for (int i = 0; i < kHalf; ++i) {
      cs[i][0] = __ldg(reinterpret_cast<const uint4*>(ctab + at + 8 * i));
      cs[i][1] = __ldg(reinterpret_cast<const uint4*>(stab + at + 8 * i));
      cs[i][2] = __ldg(reinterpret_cast<const uint4*>(ctab + at + 8 * i + D / 2));
      cs[i][3] = __ldg(reinterpret_cast<const uint4*>(stab + at + 8 * i + D / 2));
    }
  };
  if (rotary && ngrp > 0) load_table(0);
#pragma unroll 1
  for (int g = 0; g < ngrp; ++g) {
    const unsigned char* kst = ring + (g & 1) * RG::kKSlot + gq * RG::kKRow;
    wait_load();
    uint4 kf[2 * kHalf];
#pragma unroll
    for (int i = 0; i < 2 * kHalf; ++i) kf[i] = *reinterpret_cast<const uint4*>(kst + 2 * key_piece<D>(tq, i));
    if (rotary) {
      if (!prerot || wk0 + g * kGroup + gq == W - 1) {
#pragma unroll
        for (int i = 0; i < kHalf; ++i) {
          // packed bf16 arithmetic: x c1 - y s1 and y c2 + x s2 on pairs, the first product rounded to bf16
          const __nv_bfloat162* c1v = reinterpret_cast<const __nv_bfloat162*>(&cs[i][0]);
          const __nv_bfloat162* s1v = reinterpret_cast<const __nv_bfloat162*>(&cs[i][1]);
          const __nv_bfloat162* c2v = reinterpret_cast<const __nv_bfloat162*>(&cs[i][2]);
          const __nv_bfloat162* s2v = reinterpret_cast<const __nv_bfloat162*>(&cs[i][3]);
          __nv_bfloat162* xv = reinterpret_cast<__nv_bfloat162*>(&kf[i]);
          __nv_bfloat162* yv = reinterpret_cast<__nv_bfloat162*>(&kf[i + kHalf]);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const __nv_bfloat162 x = xv[e], y = yv[e];
            xv[e] = __hfma2(x, c1v[e], __hneg2(__hmul2(y, s1v[e])));
            yv[e] = __hfma2(y, c2v[e], __hmul2(x, s2v[e]));
          }
        }
      }
      if (g + 1 < ngrp) load_table(g + 1);                         // travels while this group is worked on
    }
    float c0[4] = {0.f, 0.f, 0.f, 0.f}, c1[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int jj = 0; jj < D / 32; ++jj) {
      // the query fragments are read anew for every group: they would not fit the registers beside the table entries
      const uint4 qh0 = *reinterpret_cast<const uint4*>(sqA + gq * ldq + key_piece<D>(tq, jj));
      const uint4 qh1 = NT > 1 ? *reinterpret_cast<const uint4*>(sqA + (gq + 8) * ldq + key_piece<D>(tq, jj)) : make_uint4(0u, 0u, 0u, 0u);
      mma_16816(c0, qh0.x, qh1.x, qh0.y, qh1.y, kf[jj].x, kf[jj].y);
      mma_16816(c1, qh0.z, qh1.z, qh0.w, qh1.w, kf[jj].z, kf[jj].w);
    }
    // softmax step of head gq (+ 8): this lane has keys 2 tq, 2 tq + 1 of the group
    const int left = nk - g * kGroup - 2 * tq;
    uint32_t pb[NT];
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const float x0 = left > 0 ? (c0[2 * t] + c1[2 * t]) * sc2 : -INFINITY;
      const float x1 = left > 1 ? (c0[2 * t + 1] + c1[2 * t + 1]) * sc2 : -INFINITY;
      float mx = fmaxf(x0, x1);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const bool raise = mx > m_run[t] + kRaise;
      if (__any_sync(0xffffffffu, raise)) {
        const float f = raise ? exp2f(m_run[t] - mx) : 1.f;        // 0 when nothing came before
        if (raise) m_run[t] = mx;
        l_run[t] *= f;
        const float f0 = __shfl_sync(0xffffffffu, f, 8 * tq), f1 = __shfl_sync(0xffffffffu, f, 8 * tq + 4);
#pragma unroll
        for (int j = 0; j < D / 64; ++j)
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            oacc[t][j][u][0] *= f0; oacc[t][j][u][1] *= f1;
            oacc[t][j][u][2] *= f0; oacc[t][j][u][3] *= f1;
          }
      }
      const float ref = m_run[t] > -INFINITY ? m_run[t] : 0.f;     // every logit so far minus infinity: weights zero (a NaN stays one)
      const float p0 = exp2f(x0 - ref), p1 = exp2f(x1 - ref);
      l_run[t] += p0 + p1;
      const __nv_bfloat162 pk = __floats2bfloat162_rn(p0, p1);
      pb[t] = *reinterpret_cast<const uint32_t*>(&pk);
    }
    __syncwarp();                                                  // every lane is done with the key slot
    issue(g + kAhead / 2, kKeys);
    wait_load();
    const unsigned char* vst = ring + 2 * RG::kKSlot + (g & 1) * RG::kVSlot + 2 * tq * RG::kVRow + 16 * gq;
#pragma unroll
    for (int j = 0; j < D / 64; ++j) {
      const uint4 va = *reinterpret_cast<const uint4*>(vst + 128 * j), vb = *reinterpret_cast<const uint4*>(vst + RG::kVRow + 128 * j);
      const uint32_t ea[4] = {va.x, va.y, va.z, va.w}, eb[4] = {vb.x, vb.y, vb.z, vb.w};
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t a0 = __byte_perm(ea[u], eb[u], 0x5410), a1 = __byte_perm(ea[u], eb[u], 0x7632);
#pragma unroll
        for (int t = 0; t < NT; ++t) mma_1688(oacc[t][j][u], a0, a1, pb[t]);
      }
    }
    __syncwarp();                                                  // every lane is done with the value slot
    issue(g + kAhead / 2, kValues);
  }

  // ---- the window output into the warp's own (now dead) ring memory: [NG][ldo] ----------------------------------------
  constexpr int ldo = V + 4, kOut = RG::kWarp / 4;
  static_assert(16 * ldo * 4 <= RG::kWarp || NT == 1, "a warp's output fits its ring");
  static_assert(8 * ldo * 4 <= RG::kWarp, "a warp's output fits its ring");
  float* osm = reinterpret_cast<float*>(smem + a.off_ring);        // warp w: at w kOut
  float* myml = wml + warp * NH * 4;
  __syncwarp();
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    float l = l_run[t];
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    if (tq == 0) *reinterpret_cast<float4*>(myml + 4 * (8 * t + gq)) = make_float4(-INFINITY, 0.f, m_run[t], l);
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
      const int qh = 8 * t + 2 * tq + hf;
      if (qh < NG) {
        float* orow = osm + warp * kOut + qh * ldo + 8 * gq;
#pragma unroll
        for (int j = 0; j < D / 64; ++j) {
          *reinterpret_cast<float4*>(orow + 64 * j) = make_float4(oacc[t][j][0][hf], oacc[t][j][0][2 + hf], oacc[t][j][1][hf], oacc[t][j][1][2 + hf]);
          *reinterpret_cast<float4*>(orow + 64 * j + 4) = make_float4(oacc[t][j][2][hf], oacc[t][j][2][2 + hf], oacc[t][j][3][hf], oacc[t][j][3][2 + hf]);
        }
      }
    }
  }
  __syncwarp();

  // ---- slot memory: the warp's eight slots (their lines were brought into L2 by the prefetch at the start) -------------
  float* pS = reinterpret_cast<float*>(smem + a.off_p) + warp * kGroup * NH;     // [8 slots][NH] weights of the task
  if (warp < ntask) {
    const int ms = kGroup * warp;
    load_state();
    {
      // h <- h e^g + k s with the small product rounded: the large one is the fused one, as the error of the state is made of it
      // (against 64 bits 8.3e-8 a step; 8.7e-8 with the other one fused)
      const float4 e4 = *reinterpret_cast<const float4*>(eg + ms + hs), s4 = *reinterpret_cast<const float4*>(sv + ms + hs);
#pragma unroll
      for (int i = 0; i < kHk; ++i) {
        const float kk = kpop[16 * i + hr];
        hreg[i].x = fmaf(hreg[i].x, e4.x, __fmul_rn(kk, s4.x));
        hreg[i].y = fmaf(hreg[i].y, e4.y, __fmul_rn(kk, s4.y));
        hreg[i].z = fmaf(hreg[i].z, e4.z, __fmul_rn(kk, s4.z));
        hreg[i].w = fmaf(hreg[i].w, e4.w, __fmul_rn(kk, s4.w));
      }
      // (stores behind the updates: between them, 4 sequences, 32 heads on 8, W 128 take 9.2 us a layer and not 8.6)
#pragma unroll
      for (int i = 0; i < kHk; ++i)
        if (ms + hs < nslots) st_state4<SB16>(a.hk, ((size_t)bh * K + 16 * i + hr) * M + m0 + ms + hs, hreg[i]);
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      // logits: acc[4 head + slot], summed over the sixteen lanes that share a slot quad by exchanging halves, after which
      // a lane holds two neighbouring slots of one head
      float acc[4 * HB];
#pragma unroll
      for (int i = 0; i < 4 * HB; ++i) acc[i] = 0.f;
#pragma unroll
      for (int i = 0; i < kHk; ++i) {
        float qv[HB];
        if constexpr (HB == 1) {
          qv[0] = qT[(16 * i + hr) * NH];
        } else {
#pragma unroll
          for (int c = 0; c < HB; c += 4) {
            const float4 q4 = *reinterpret_cast<const float4*>(qT + (16 * i + hr) * NH + 8 * t + c);
            qv[c] = q4.x; qv[c + 1] = q4.y; qv[c + 2] = q4.z; qv[c + 3] = q4.w;
          }
        }
#pragma unroll
        for (int qh = 0; qh < HB; ++qh) {
          acc[4 * qh] += qv[qh] * hreg[i].x;
          acc[4 * qh + 1] += qv[qh] * hreg[i].y;
          acc[4 * qh + 2] += qv[qh] * hreg[i].z;
          acc[4 * qh + 3] += qv[qh] * hreg[i].w;
        }
      }
      // the sixteen lanes that share a slot quad, by lane bits 4, 3, 2, 1: halving while there are values to halve (head first, then
      // the slot pair, then the slot), whole sums after that
#pragma unroll
      for (int st = 0; st < 4; ++st) {
        const int n = (2 * HB) >> st, bit = 16 >> st;
        const bool up = lane & bit;
        if (n > 0) {
#pragma unroll
          for (int i = 0; i < n; ++i) {
            const float keep = up ? acc[i + n] : acc[i], give = up ? acc[i] : acc[i + n];
            acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
          }
        } else {
          acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], bit);
        }
      }
      // this lane's head and its slot (HB == 8: two neighbouring ones); the lanes of a head's other slots: `mask`
      constexpr int kOwn = HB == 8 ? 2 : 1, kM1 = 1, kM2 = HB == 8 ? 2 : HB == 4 ? 2 : 16, kM3 = HB == 8 ? 0 : HB == 4 ? 4 : 8;
      const int qh = 8 * t + (HB == 8 ? lane >> 2 : HB == 4 ? lane >> 3 : 0);
      const int sl = hs + (HB == 8 ? lane & 2 : HB == 4 ? ((lane >> 1) & 2) + ((lane >> 1) & 1) : ((lane >> 3) & 2) + ((lane >> 3) & 1));
      const float x0 = ms + sl < nslots ? acc[0] * sc2 : -INFINITY, x1 = kOwn == 2 && ms + sl + 1 < nslots ? acc[kOwn - 1] * sc2 : -INFINITY;
      float mx = fmaxf(x0, x1);
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, kM1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, kM2));
      if (kM3) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, kM3));
      const float ref = mx > -INFINITY ? mx : 0.f;                 // eight logits of minus infinity: weights zero (a NaN stays one)
      const float p0 = exp2f(x0 - ref), p1 = kOwn == 2 ? exp2f(x1 - ref) : 0.f;
      pS[sl * NH + qh] = p0;
      if (kOwn == 2) pS[(sl + 1) * NH + qh] = p1;
      float sum = p0 + p1;
      sum += __shfl_xor_sync(0xffffffffu, sum, kOwn == 2 ? kM1 : kM3 == 8 ? 8 : 2);
      sum += __shfl_xor_sync(0xffffffffu, sum, kOwn == 2 ? kM2 : kM3 == 8 ? 1 : 1);
      if (kM3) sum += __shfl_xor_sync(0xffffffffu, sum, kM3 == 8 ? 16 : 4);
      if (HB == 8 ? (lane & 3) == 0 : HB == 4 ? (lane & 7) == 0 : lane == 0) {
        myml[4 * qh] = mx;
        myml[4 * qh + 1] = sum;
      }
    }
    __syncwarp();
    float sacc[NT][HB][4];                                         // readout of the warp's slots: heads 8 t + i, columns vcol ..
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < HB; ++i) sacc[t][i][0] = sacc[t][i][1] = sacc[t][i][2] = sacc[t][i][3] = 0.f;
    const float4 vp = *reinterpret_cast<const float4*>(vpop + vcol);
#pragma unroll
    for (int u = 0; u < kHv; ++u) {
      const int m = ms + kRowsI * u + vsub;
      if (m < nslots) {
        const float e = eg[m], sm = sv[m];
        vreg[u].x = fmaf(vreg[u].x, e, __fmul_rn(sm, vp.x));
        vreg[u].y = fmaf(vreg[u].y, e, __fmul_rn(sm, vp.y));
        vreg[u].z = fmaf(vreg[u].z, e, __fmul_rn(sm, vp.z));
        vreg[u].w = fmaf(vreg[u].w, e, __fmul_rn(sm, vp.w));
        st_state4<SB16>(a.hv, ((size_t)bh * M + m0 + m) * V + vcol, vreg[u]);
      }
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        float p[HB];
        if constexpr (HB == 1) {
          p[0] = pS[(kRowsI * u + vsub) * NH];
        } else {
#pragma unroll
          for (int c = 0; c < HB; c += 4) {
            const float4 p4 = *reinterpret_cast<const float4*>(pS + (kRowsI * u + vsub) * NH + 8 * t + c);
            p[c] = p4.x; p[c + 1] = p4.y; p[c + 2] = p4.z; p[c + 3] = p4.w;
          }
        }
#pragma unroll
        for (int i = 0; i < HB; ++i) {
          sacc[t][i][0] += p[i] * vreg[u].x; sacc[t][i][1] += p[i] * vreg[u].y;
          sacc[t][i][2] += p[i] * vreg[u].z; sacc[t][i][3] += p[i] * vreg[u].w;
        }
      }
    }
    // slots and window of the warp together
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int i = 0; i < HB; ++i) {
        const int qh = 8 * t + i;
        float4 x = make_float4(sacc[t][i][0], sacc[t][i][1], sacc[t][i][2], sacc[t][i][3]);
        if (kRowsI == 2) {                                         // D = 64: the two halves of the warp hold different slots
          x.x += __shfl_xor_sync(0xffffffffu, x.x, 16); x.y += __shfl_xor_sync(0xffffffffu, x.y, 16);
          x.z += __shfl_xor_sync(0xffffffffu, x.z, 16); x.w += __shfl_xor_sync(0xffffffffu, x.w, 16);
        }
        if (qh < NG && (kRowsI == 1 || lane < 16)) {
          const float m1 = myml[4 * qh], m2 = myml[4 * qh + 2], mx = fmaxf(m1, m2);
          const float f1 = m1 > -INFINITY ? exp2f(m1 - mx) : 0.f, f2 = m2 > -INFINITY ? exp2f(m2 - mx) : 0.f;
          float4* o4 = reinterpret_cast<float4*>(osm + warp * kOut + qh * ldo + vcol);
          const float4 w4 = *o4;
          *o4 = make_float4(f1 * x.x + f2 * w4.x, f1 * x.y + f2 * w4.y, f1 * x.z + f2 * w4.z, f1 * x.w + f2 * w4.w);
        }
      }
  }
  __syncthreads();
  float* po = a.part_o + ((size_t)bh * SPL + sp) * NG * V;
  auto store_row = [&](int qh, int c, const float4& x) { store_row4(a.o + ((size_t)b * a.HQ + h * NG + qh) * V + 4 * c, x); };
#pragma unroll 1
  for (int i = tid; i < NG * V4; i += kStrThreads) {
    const int qh = i / V4, c = i - qh * V4;
    float mw[kStrWarps], lw[kStrWarps], mx = -INFINITY;
#pragma unroll
    for (int w8 = 0; w8 < kStrWarps; ++w8) {
      const float4 s4 = *reinterpret_cast<const float4*>(wml + (w8 * NH + qh) * 4);
      mw[w8] = fmaxf(s4.x, s4.z);
      lw[w8] = (s4.x > -INFINITY ? s4.y * exp2f(s4.x - mw[w8]) : 0.f) + (s4.z > -INFINITY ? s4.w * exp2f(s4.z - mw[w8]) : 0.f);
      mx = fmaxf(mx, mw[w8]);
    }
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float den = 0.f;
#pragma unroll
    for (int w8 = 0; w8 < kStrWarps; ++w8) {
      const float wgt = mw[w8] > -INFINITY ? exp2f(mw[w8] - mx) : 0.f;
      const float4 wv = *reinterpret_cast<const float4*>(osm + w8 * kOut + qh * ldo + 4 * c);
      den += wgt * lw[w8];
      acc.x += wgt * wv.x; acc.y += wgt * wv.y; acc.z += wgt * wv.z; acc.w += wgt * wv.w;
    }
    if (SPL == 1) {
      const float inv = 1.0f / den;
      store_row(qh, c, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
    } else {
      if (a.cluster) *reinterpret_cast<float4*>(outp + qh * V + 4 * c) = acc;
      else *reinterpret_cast<float4*>(po + qh * V + 4 * c) = acc;
      if (c == 0) {
        ml[2 * qh] = mx * kLn2;
        ml[2 * qh + 1] = den;
      }
    }
  }
  if (SPL == 1) {
    append_token();
    return;
  }

  if (a.cluster) {
    // ---- merge inside the cluster: CTA 0 reads the partial outputs, maxima and sums of its peers from their shared
    //      memory; the second barrier keeps the peers' memory alive until it has ----------------------------------
    cluster_sync_all();
    if (sp == 0) {
      append_token();
      merge_cluster<V, NT, HB == 1>(ml, outp, a.o + ((size_t)b * a.HQ + h * NG) * V, NG, SPL);
    }
    cluster_sync_all();
    return;
  }

  // ---- merge: the last split of this (sequence, kv head) to arrive combines all partials ------------
  float* pml = a.part_ml + ((size_t)bh * SPL + sp) * NG * 2;
  __syncthreads();                      // ml is complete
#pragma unroll 1
  for (int i = tid; i < NG * 2; i += kStrThreads) pml[i] = ml[i];
  __syncthreads();
  __shared__ int s_last;
  if (tid == 0) {
    __threadfence();                    // the partials of this CTA are visible before its ticket
    const int t = atomicAdd(a.tickets + bh, 1);
    s_last = (t == SPL - 1);
    if (s_last) a.tickets[bh] = 0;      // leave the counter at zero for the next call
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  append_token();
  const float* all_ml = a.part_ml + (size_t)bh * SPL * NG * 2;
  const float* all_o = a.part_o + (size_t)bh * SPL * NG * V;
  merge_workspace<V, NT, HB == 1>(all_ml, all_o, outp, a.o + ((size_t)b * a.HQ + h * NG) * V, NG, SPL);
}

static int stream_layout(DecodeStreamArgs& a, int D) {
  const int NG = a.NG, MQ = a.MQ, NH = NG > 8 ? 16 : 8;
  int off = 0;
  auto take = [&](int bytes) { int o = off; off = (off + bytes + 127) / 128 * 128; return o; };
  a.off_ring = take(kStrWarps * (D == 128 ? DecodeRing<128>::kWarp : DecodeRing<64>::kWarp));
  a.off_out = take(std::max(NG * D, a.SPLITS * NG) * 4);
  a.off_q = take(D * NH * 4);
  a.off_sqA = take(16 * (D == 128 ? kLdq<128> : kLdq<64>) * 2);
  a.off_p = take(kStrWarps * kGroup * NH * 4);
  a.off_eg = take(MQ * 4);
  a.off_sv = take(MQ * 4);
  a.off_kpop = take(D * 4);
  a.off_vpop = take(D * 4);
  a.off_wml = take(kStrWarps * NH * 4 * 4);
  a.off_ml = take(NG * 2 * 4);
  return off;
}

// Splits of a (sequence, kv head) for the streaming kernel: as many as keep the whole grid in one wave of two
// CTAs per SM, each split keeping at least kMinKeys keys and 4 slots.
int decode_stream_splits(int B, int H, int W, int M) {
  const int sms = sm_count();
  int spl = M > 64 && M <= 128 ? 2 : 1;            // a split has at most 64 slots: eight a warp
  while (spl < 16 && (int64_t)B * H * spl * 2 <= 2 * (int64_t)sms && W / (spl * 2) >= kMinKeys && M / (spl * 2) >= 4 &&
         M % (spl * 2 * 4) == 0)
    spl *= 2;
  return spl;
}

// Whether a call's window goes into L2 ahead of its use, as its state always does.  The resident CTAs of this call prefetch while those of
// the call in front still use what they have prefetched; L2 serves both as long as one wave takes up to a third of it.  Us a layer in a
// stack, HQ 32, D 128 (132.6 MB of L2), without and with the prefetch of the window, by what a wave holds:
//   W 512, decode: 31 MB 16.20 | 15.03, 42 MB 16.62 | 16.61, 47 MB 16.90 | 17.57, 52 MB 22.6 | 24.5, 63 MB 23.7 | 24.8, 84 MB 25.2 | 25.2;
//   on rings: 42 MB 18.28 | 18.67, 52 MB 25.8 | 27.2, 84 MB 26.5 | 28.2;  W 1200: 33 MB 15.57 | 14.67, 44 MB 16.01 | 16.51;
// grids of several waves, H 4, HQ 16, W 128: 39 of 59 MB 29.26 | 27.75; 16 heads of 64, W 128: 19 of 84 MB 42.9 | 41.3.
// The line lies behind 42 MB, where the window tensors of a 48-layer stack gain 0.5 % and rings lose 2 %, and in front of 44.
// state_bytes: of an element of the slot memory, 0 where none is read.
bool decode_window_ahead(int B, int H, int D, int M, int rows, int splits, int state_bytes, int ctas_per_sm, int sms, int64_t l2) {
  const int64_t each = ((int64_t)D * (4 * (int64_t)rows + 2 * (int64_t)state_bytes * M)) / splits;
  const int64_t ctas = std::min((int64_t)B * H * splits, (int64_t)ctas_per_sm * sms);
  return ctas * each <= l2 / 100 * 32;
}

// Mode of the programmatic dependent launch of the streaming kernel (see DecodeStreamArgs::pdl): set by
// nha_decode_set_pdl(), else taken once from the environment variable NHA_PDL (the reference's switch of the same
// name, nha_fla/ops/nha/fused_recurrent.py:32-34: "0" turns it off), default 1.
static std::atomic<int> g_pdl_mode{-1};
int decode_pdl_mode() {
  int m = g_pdl_mode.load(std::memory_order_relaxed);
  if (m < 0) {
    const char* e = getenv("NHA_PDL");
    m = 1;
    if (e && e[0] >= '0' && e[0] <= '2' && e[1] == 0) m = e[0] - '0';
    g_pdl_mode.store(m, std::memory_order_relaxed);
  }
  return m;
}
void decode_set_pdl_mode(int m) { g_pdl_mode.store(m, std::memory_order_relaxed); }

bool decode_stream_supported(int K, int V, int M, int W, int NG, bool logits_mode) {
  return !logits_mode && K == V && (K == 64 || K == 128) && M % 4 == 0 && M <= 128 && NG <= 16 && W >= 1;
}

// The caller has checked decode_stream_supported() and sized the workspace for `splits`.
int decode_stream_launch(const DecodeStreamArgs& in, int D, cudaStream_t st) {
  DecodeStreamArgs a = in;
  a.KSPL = ((a.W + a.SPLITS - 1) / a.SPLITS + kGroup - 1) / kGroup * kGroup;
  a.MQ = ((a.M + a.SPLITS - 1) / a.SPLITS + kGroup - 1) / kGroup * kGroup;
  const int smem = stream_layout(a, D);
  if (smem > kMaxSmem) return NHA_ERR_SMEM;
  dim3 grid(a.B * a.H * a.SPLITS), block(kStrThreads);
  // 2, 4 or 8 splits merge through the cluster's shared memory
  a.cluster = a.SPLITS == 2 || a.SPLITS == 4 || a.SPLITS == 8;
  if (const char* nc = getenv("NHA_B200_DECODE_NO_CLUSTER")) {
    if (nc[0] == '1') a.cluster = 0;                 // merge through the workspace instead
  }
  const void* fn;
#define NHA_PICK(D_, T_, H_)                                                                                   \
  (a.state_bf16 ? (const void*)nha_decode_stream_kernel<D_, T_, H_, true, false>                               \
                : a.head ? (const void*)nha_decode_stream_kernel<D_, T_, H_, false, true>                      \
                         : (const void*)nha_decode_stream_kernel<D_, T_, H_, false, false>)
#define NHA_PICK_H(D_) (a.NG > 8 ? NHA_PICK(D_, 2, 8) : a.NG > 4 ? NHA_PICK(D_, 1, 8) : a.NG > 1 ? NHA_PICK(D_, 1, 4) : NHA_PICK(D_, 1, 1))
  fn = D == 128 ? NHA_PICK_H(128) : NHA_PICK_H(64);
#undef NHA_PICK_H
#undef NHA_PICK
  cudaError_t e = set_max_smem(fn, smem);
  if (e != cudaSuccess) return record_cuda_error(e);
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  a.pdl = decode_pdl_mode();
  cudaLaunchAttribute attr[2];
  auto attributes = [&]() {
    cfg.attrs = attr;
    cfg.numAttrs = 0;
    if (a.pdl) {
      attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr[cfg.numAttrs++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (a.cluster) {
      attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
      attr[cfg.numAttrs].val.clusterDim.x = a.SPLITS;
      attr[cfg.numAttrs].val.clusterDim.y = 1;
      attr[cfg.numAttrs++].val.clusterDim.z = 1;
    }
  };
  attributes();
  a.ahead = decode_window_ahead(a.B, a.H, D, a.M, a.WR, a.SPLITS, a.zero_state ? 0 : a.state_bf16 ? 2 : 4, a.NG > 8 ? 1 : 2, sm_count(), l2_bytes());
  a.tab32 = ((uintptr_t)a.cosp | (uintptr_t)a.sinp | (uintptr_t)(2 * a.cs_row) | (uintptr_t)(2 * a.cs_batch)) % 32 == 0;
  void* args[1] = {(void*)&a};
  e = cudaLaunchKernelExC(&cfg, fn, args);
  if (e != cudaSuccess && a.cluster) {
    // the device could not place the cluster (partitioned GPU, ...): the same kernel merges through the workspace
    (void)cudaGetLastError();
    a.cluster = 0;
    attributes();
    e = cudaLaunchKernelExC(&cfg, fn, args);
  }
  if (e != cudaSuccess) return record_cuda_error(e);
  return check_launch();
}

// Runs the streaming kernel when the shape has one; *used tells the caller whether it did.
int decode_stream_try(const void* q, const void* sq, const void* k, const void* v, const void* g, const void* s,
                      const void* sw_k, const void* sw_v, const void* cosp, const void* sinp, int64_t cs_batch,
                      int64_t cs_row, float* hk, float* hv, int zero_state, void* o, int* tickets,
                      float* part_ml, float* part_o, int splits, int B, int HQ, int H, int D, int M, int W, float scale,
                      cudaStream_t st, const int* head, const void* ring_g, int ring_rows, int nopop,
                      const void* ring_kraw, const void* g_new, int state_bf16) {
  DecodeStreamArgs a;
  a.q = (const bf16*)q; a.sq = (const bf16*)sq; a.k = (const bf16*)k; a.v = (const bf16*)v; a.g = (const bf16*)g;
  a.s = (const bf16*)s; a.sw_k = (const bf16*)sw_k; a.sw_v = (const bf16*)sw_v; a.cosp = (const bf16*)cosp;
  a.sinp = (const bf16*)sinp;
  a.hk = hk; a.hv = hv; a.o = (bf16*)o;
  a.part_o = part_o; a.part_ml = part_ml; a.tickets = tickets;
  a.head = head; a.ring_g = (const bf16*)ring_g;
  a.WR = head ? ring_rows : W; a.nopop = head ? nopop : 0;
  a.ring_kraw = head ? (const bf16*)ring_kraw : nullptr;
  a.g_new = (head && !ring_kraw) ? (const bf16*)g_new : nullptr;
  a.state_bf16 = state_bf16;
  a.cs_batch = cs_batch; a.cs_row = cs_row;
  a.B = B; a.HQ = HQ; a.H = H; a.M = M; a.W = W; a.NG = HQ / H; a.SPLITS = splits;
  a.zero_state = zero_state; a.scale = scale;
  return decode_stream_launch(a, D, st);
}

}  // namespace nha
