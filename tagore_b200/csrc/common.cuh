// common.cuh -- device helpers shared by the graph-build kernels (sm_100a).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace tagore {

constexpr uint32_t kInv = 0xFFFFFFFFu;
constexpr float kInfDis = 10000000.0f;   // INF_DIS of the reference (include/common.cuh:29)
constexpr uint32_t kReserve = 128;       // RESERVENUM: row stride of reverse_distance
constexpr uint32_t kSelectCand = 480;    // SELECT_CAND: ring capacity of the path collect
constexpr uint32_t kSample = 32;         // SAMPLE: hybrid_list rows are 4*SAMPLE wide
constexpr unsigned kFull = 0xFFFFFFFFu;

__device__ __forceinline__ float2 h2lo(uint32_t v) {
  return __half22float2(*reinterpret_cast<const __half2*>(&v));
}

// Packed FP32 pair arithmetic of sm_100 (PTX .f32x2): each half is its own
// IEEE operation rounded to nearest, so a pair op equals the two scalar ops.
// (x, y) += (a, b), and (x, y) = (d0*d0 + x, d1*d1 + y).
__device__ __forceinline__ void add2(float& x, float& y, float a, float b) {
  asm("{.reg .b64 p, q;\n\t"
      "mov.b64 p, {%0, %1};\n\t"
      "mov.b64 q, {%2, %3};\n\t"
      "add.rn.f32x2 p, p, q;\n\t"
      "mov.b64 {%0, %1}, p;}"
      : "+f"(x), "+f"(y)
      : "f"(a), "f"(b));
}
__device__ __forceinline__ void fma2_sq(float& x, float& y, float d0, float d1) {
  asm("{.reg .b64 p, q;\n\t"
      "mov.b64 p, {%0, %1};\n\t"
      "mov.b64 q, {%2, %3};\n\t"
      "fma.rn.f32x2 p, q, q, p;\n\t"
      "mov.b64 {%0, %1}, p;}"
      : "+f"(x), "+f"(y)
      : "f"(d0), "f"(d1));
}
// (d0, d1) = (float(a.lo) - b0, float(a.hi) - b1), one rounding each: the
// mixed f16/f32 subtract widens a exactly, as __half2float would.
__device__ __forceinline__ void sub_h2(uint32_t a, float b0, float b1, float& d0, float& d1) {
  asm("{.reg .b16 lo, hi;\n\t"
      "mov.b32 {lo, hi}, %2;\n\t"
      "sub.rn.f32.f16 %0, lo, %3;\n\t"
      "sub.rn.f32.f16 %1, hi, %4;}"
      : "=f"(d0), "=f"(d1)
      : "r"(a), "f"(b0), "f"(b1));
}

// Accumulates one 4-dim chunk into the lane's (x, y) pair exactly as the
// reference's two __hfma2 steps do (src/Tagore_src.cu:1431-1435), in FP32:
// x takes dims 0 and 2, y takes dims 1 and 3, each a fused multiply-add of the
// rounded difference.
__device__ __forceinline__ void chunk_acc(uint2 a, uint2 b, float& x, float& y) {
  const float2 b01 = h2lo(b.x), b23 = h2lo(b.y);
  float d0, d1, d2, d3;
  sub_h2(a.x, b01.x, b01.y, d0, d1);
  sub_h2(a.y, b23.x, b23.y, d2, d3);
  fma2_sq(x, y, d0, d1);
  fma2_sq(x, y, d2, d3);
}

// Reduces the per-lane pairs with the reference's shuffle-down tree (offsets
// 16..1) and returns x + y in every lane.
__device__ __forceinline__ float warp_tree(float x, float y) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1)
    add2(x, y, __shfl_down_sync(kFull, x, off), __shfl_down_sync(kFull, y, off));
  return __shfl_sync(kFull, __fadd_rn(x, y), 0);
}

// Exact FP32 squared L2 between two FP16 rows, in the reference's lane order.
// Executed by a full warp; `dim` is a multiple of 4.
__device__ __forceinline__ float warp_dist(const __half* __restrict__ a, const __half* __restrict__ b,
                                           uint32_t dim, int lane) {
  float x = 0.0f, y = 0.0f;
  const uint32_t chunks = dim >> 2;
  for (uint32_t j = lane; j < chunks; j += 32) {
    const uint2 va = __ldg(reinterpret_cast<const uint2*>(a) + j);
    const uint2 vb = __ldg(reinterpret_cast<const uint2*>(b) + j);
    chunk_acc(va, vb, x, y);
  }
  return warp_tree(x, y);
}

// Four independent distances against one query, interleaving their shuffle
// trees. Rows with id kInv yield 0 and must be ignored by the caller. DIM,
// when given, fixes the width at compile time (`dim` is then DIM).
template <uint32_t DIM = 0>
__device__ __forceinline__ void warp_dist4(const __half* __restrict__ q, const __half* __restrict__ base,
                                           uint32_t dim, const uint32_t ids[4], float out[4],
                                           int lane) {
  float x[4] = {0.f, 0.f, 0.f, 0.f}, y[4] = {0.f, 0.f, 0.f, 0.f};
  if constexpr (DIM != 0) dim = DIM;
  auto chunk = [&](uint32_t j) {
    const uint2 vq = *(reinterpret_cast<const uint2*>(q) + j);
#pragma unroll
    for (int t = 0; t < 4; ++t) {
      if (ids[t] != kInv) {
        const uint2 vb = __ldg(reinterpret_cast<const uint2*>(base + (size_t)ids[t] * dim) + j);
        chunk_acc(vq, vb, x[t], y[t]);
      }
    }
  };
  if constexpr (DIM != 0) {
#pragma unroll
    for (uint32_t i = 0; i < (DIM / 4 + 31) / 32; ++i)
      if (lane + 32 * i < DIM / 4) chunk(lane + 32 * i);
  } else {
    const uint32_t chunks = dim >> 2;
    for (uint32_t j = lane; j < chunks; j += 32) chunk(j);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int t = 0; t < 4; ++t)
      add2(x[t], y[t], __shfl_down_sync(kFull, x[t], off), __shfl_down_sync(kFull, y[t], off));
  }
#pragma unroll
  for (int t = 0; t < 4; ++t) out[t] = __shfl_sync(kFull, __fadd_rn(x[t], y[t]), 0);
}

// The reference's shuffle-down tree evaluated by one thread over the 32 lane
// slots: v_L[l] = v_{L-1}[l] + v_{L-1}[l + (32 >> L)], root v_5[0]. Walking
// the tree depth-first visits the slots in bit-reversed order and keeps at
// most five partial pairs alive. `leaf(slot, x, y)` accumulates that slot's
// chunks (slot, slot + 32, ...) into (x, y) exactly as the lane would.
template <int Level, int Slot, class Leaf>
__device__ __forceinline__ void lane_tree(Leaf& leaf, float& x, float& y) {
  if constexpr (Level == 0) {
    x = 0.0f;
    y = 0.0f;
    leaf(Slot, x, y);
  } else {
    float ax, ay, bx, by;
    lane_tree<Level - 1, Slot>(leaf, ax, ay);
    lane_tree<Level - 1, Slot + (32 >> Level)>(leaf, bx, by);
    add2(ax, ay, bx, by);
    x = ax;
    y = ay;
  }
}

// Exact FP32 squared L2 in the reference's lane order by a single thread;
// chunk(j) returns the two 4-half chunks j of the operands.
template <int D, class Chunk>
__device__ __forceinline__ float serial_dist(Chunk chunk) {
  auto leaf = [&](int slot, float& x, float& y) {
#pragma unroll
    for (int j = slot; j < D / 4; j += 32) {
      const uint2 a = chunk(j, 0), b = chunk(j, 1);
      chunk_acc(a, b, x, y);
    }
  };
  float x, y;
  lane_tree<5, 0>(leaf, x, y);
  return __fadd_rn(x, y);
}

// The 128-dim tree with 16-byte loads. At 128 dims each lane slot holds one
// chunk, so level-1 node l is leaf l + leaf l+16 and level-2 node m is
// level-1 m + level-1 m+8; chunks 2p and 2p+1 share a 16-byte load. Level-2
// nodes are built in pairs (2p, 2p+1) from four loads per row and combined
// exactly as the tree combines them.
__device__ __forceinline__ void pair_acc(uint4 a, uint4 b, float& x0, float& y0, float& x1,
                                         float& y1) {
  chunk_acc(make_uint2(a.x, a.y), make_uint2(b.x, b.y), x0, y0);
  chunk_acc(make_uint2(a.z, a.w), make_uint2(b.z, b.w), x1, y1);
}

// load(p, w) returns chunks 2p and 2p+1 of operand w as one 16-byte value.
template <class Load16>
__device__ __forceinline__ void level2_pair(Load16& load, int p, float (&x)[2], float (&y)[2]) {
  // leaves 2p, 2p+1 (pair p), 2p+8.. (pair p+4), 2p+16.. (p+8), 2p+24.. (p+12)
  float lx[4][2], ly[4][2];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    lx[q][0] = ly[q][0] = lx[q][1] = ly[q][1] = 0.0f;
    pair_acc(load(p + 4 * q, 0), load(p + 4 * q, 1), lx[q][0], ly[q][0], lx[q][1], ly[q][1]);
  }
  // q indexes leaf offsets 0, 8, 16, 24: level 1 pairs (0,16) and (8,24),
  // level 2 pairs the two results.
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float ax = lx[0][h], ay = ly[0][h], bx = lx[1][h], by = ly[1][h];
    add2(ax, ay, lx[2][h], ly[2][h]);
    add2(bx, by, lx[3][h], ly[3][h]);
    add2(ax, ay, bx, by);
    x[h] = ax;
    y[h] = ay;
  }
}

template <class Load16>
__device__ __forceinline__ float dist128_pairs(Load16 load) {
  float x0[2], y0[2], x1[2], y1[2], x2[2], y2[2], x3[2], y3[2];
  level2_pair(load, 0, x0, y0);  // level-2 nodes 0, 1
  level2_pair(load, 2, x2, y2);  // 4, 5
  level2_pair(load, 1, x1, y1);  // 2, 3
  level2_pair(load, 3, x3, y3);  // 6, 7
  // level 3: m + m+4; level 4: m + m+2; level 5: 0 + 1
  add2(x0[0], y0[0], x2[0], y2[0]);
  add2(x0[1], y0[1], x2[1], y2[1]);
  add2(x1[0], y1[0], x3[0], y3[0]);
  add2(x1[1], y1[1], x3[1], y3[1]);
  add2(x0[0], y0[0], x1[0], y1[0]);
  add2(x0[1], y0[1], x1[1], y1[1]);
  add2(x0[0], y0[0], x0[1], y0[1]);
  return __fadd_rn(x0[0], y0[0]);
}

// The same tree for any width that is a multiple of 8 halves (`units`
// 16-byte units): lane slot s accumulates chunks s, s + 32, ... in order, so
// the leaves of pair p + 4q are summed over the units p + 4q, p + 4q + 16, ...
// before the level-1 and level-2 combining above. At 128 dims there is one
// round and this is dist128_pairs.
template <class Load16>
__device__ __forceinline__ void level2_pair_rounds(Load16& load, int p, uint32_t units,
                                                   float (&x)[2], float (&y)[2]) {
  float lx[4][2], ly[4][2];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    lx[q][0] = ly[q][0] = lx[q][1] = ly[q][1] = 0.0f;
    for (uint32_t u = p + 4 * q; u < units; u += 16)
      pair_acc(load(u, 0), load(u, 1), lx[q][0], ly[q][0], lx[q][1], ly[q][1]);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float ax = lx[0][h], ay = ly[0][h], bx = lx[1][h], by = ly[1][h];
    add2(ax, ay, lx[2][h], ly[2][h]);
    add2(bx, by, lx[3][h], ly[3][h]);
    add2(ax, ay, bx, by);
    x[h] = ax;
    y[h] = ay;
  }
}

template <class Load16>
__device__ __forceinline__ float dist_pairs_rounds(Load16 load, uint32_t units) {
  float x0[2], y0[2], x1[2], y1[2], x2[2], y2[2], x3[2], y3[2];
  level2_pair_rounds(load, 0, units, x0, y0);
  level2_pair_rounds(load, 2, units, x2, y2);
  level2_pair_rounds(load, 1, units, x1, y1);
  level2_pair_rounds(load, 3, units, x3, y3);
  add2(x0[0], y0[0], x2[0], y2[0]);
  add2(x0[1], y0[1], x2[1], y2[1]);
  add2(x1[0], y1[0], x3[0], y3[0]);
  add2(x1[1], y1[1], x3[1], y3[1]);
  add2(x0[0], y0[0], x1[0], y1[0]);
  add2(x0[1], y0[1], x1[1], y1[1]);
  add2(x0[0], y0[0], x0[1], y0[1]);
  return __fadd_rn(x0[0], y0[0]);
}

// dist_pairs_rounds with the width fixed at compile time (U 16-byte units),
// so that every load of the tree is issued up front; the same operations in
// the same order.
template <uint32_t U, class Load16>
__device__ __forceinline__ void level2_pair_fixed(Load16& load, int p, float (&x)[2],
                                                  float (&y)[2]) {
  float lx[4][2], ly[4][2];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    lx[q][0] = ly[q][0] = lx[q][1] = ly[q][1] = 0.0f;
#pragma unroll
    for (uint32_t u = p + 4 * q; u < U; u += 16)
      pair_acc(load(u, 0), load(u, 1), lx[q][0], ly[q][0], lx[q][1], ly[q][1]);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float ax = lx[0][h], ay = ly[0][h], bx = lx[1][h], by = ly[1][h];
    add2(ax, ay, lx[2][h], ly[2][h]);
    add2(bx, by, lx[3][h], ly[3][h]);
    add2(ax, ay, bx, by);
    x[h] = ax;
    y[h] = ay;
  }
}

template <uint32_t U, class Load16>
__device__ __forceinline__ float dist_pairs_fixed(Load16 load) {
  float x0[2], y0[2], x1[2], y1[2], x2[2], y2[2], x3[2], y3[2];
  level2_pair_fixed<U>(load, 0, x0, y0);
  level2_pair_fixed<U>(load, 2, x2, y2);
  level2_pair_fixed<U>(load, 1, x1, y1);
  level2_pair_fixed<U>(load, 3, x3, y3);
  add2(x0[0], y0[0], x2[0], y2[0]);
  add2(x0[1], y0[1], x2[1], y2[1]);
  add2(x1[0], y1[0], x3[0], y3[0]);
  add2(x1[1], y1[1], x3[1], y3[1]);
  add2(x0[0], y0[0], x1[0], y1[0]);
  add2(x0[1], y0[1], x1[1], y1[1]);
  add2(x0[0], y0[0], x0[1], y0[1]);
  return __fadd_rn(x0[0], y0[0]);
}

__device__ __forceinline__ float row_dist128(const __half* __restrict__ a,
                                             const __half* __restrict__ b) {
  const uint4* A = reinterpret_cast<const uint4*>(a);
  const uint4* B = reinterpret_cast<const uint4*>(b);
  return dist128_pairs([&](int p, int w) { return __ldg((w ? B : A) + p); });
}

// Whether rows of `dim` halves (a multiple of 4) from `p` on may be read 16 bytes at
// a time. A caller's buffers may start on any 8 bytes.
__device__ __forceinline__ bool rows_of_16(const __half* p, uint32_t dim) {
  return (dim & 7u) == 0 && ((uintptr_t)p & 15u) == 0;
}

// The same distance between two FP16 rows of `dim` halves (a multiple of 4)
// by a single thread, so that the 32 lanes of a warp score 32 rows at once.
// Kept out of line: one copy of the unrolled tree serves every call site and
// stays in the instruction cache.
static __device__ __noinline__ float row_dist(const __half* __restrict__ a,
                                              const __half* __restrict__ b, uint32_t dim) {
  const uint2* A = reinterpret_cast<const uint2*>(a);
  const uint2* B = reinterpret_cast<const uint2*>(b);
  if (rows_of_16(a, dim) && rows_of_16(b, dim)) {
    if (dim == 128) return row_dist128(a, b);
    const uint4* A4 = reinterpret_cast<const uint4*>(a);
    const uint4* B4 = reinterpret_cast<const uint4*>(b);
    auto load = [&](uint32_t u, int w) { return __ldg((w ? B4 : A4) + u); };
    return dim == 96 ? dist_pairs_fixed<12>(load) : dist_pairs_rounds(load, dim >> 3);
  }
  const uint32_t chunks = dim >> 2;
  auto leaf = [&](int slot, float& x, float& y) {
    for (uint32_t j = slot; j < chunks; j += 32) chunk_acc(__ldg(A + j), __ldg(B + j), x, y);
  };
  float x, y;
  lane_tree<5, 0>(leaf, x, y);
  return __fadd_rn(x, y);
}

// Distances of up to 32 rows ids[0, m) (shared memory, m >= 1) to one query by a
// warp, in the reference's lane order; lane l returns the one of row rows32_of(l).
//
// Four lanes share a row: lane j holds the 16-byte units j, j + 4, j + 8 and j + 12 of
// every 16, so levels 1 and 2 of the tree (slots 16 and 8 apart) are its own sums and
// level 5 (neighbouring slots) too. Levels 3 and 4 exchange with lanes j ^ 2 and j ^ 1;
// a lane keeps the half of its rows that its bit names and passes the other on, so
// that 12 exchanges serve 32 rows and each lane ends with one.
//
// A lane per row, as before, touches 32 lines with each load: at 200K x 128 the L1 pipe
// was 78 % busy and bounded the collect, and its unrolled tree left the instruction
// cache. Eight lanes per row read whole lines, but their third exchange and half empty
// loads at 96 dims took 1.8 times the instructions.
// Collect with these, chained membership and rolled sorts: 1M x 128, K = 96, 98.4 ->
// 79.6 ms; 500K x 96, K = 64, 32.1 -> 29.4 ms.
//
// warp_rows32_fixed holds a lane's units in registers, at the two widths up to 128
// that the configurations have: the collect takes 18.4 ms with it and 25.4 ms without
// at 300K x 128, 29.0 and 39.2 ms at 500K x 96. Each width is one more copy in code
// that waits for instructions (5.2 of 13.8 stall cycles per issue), so the others
// share warp_rows32_any (300K x 64: 21.4 ms, 300K x 112: 25.5 ms).
__device__ __forceinline__ uint32_t rows32_of(int lane) {
  return 8 * ((uint32_t)lane & 3u) + ((uint32_t)lane >> 2);
}

__device__ __forceinline__ void unit_acc(uint4 v, const float2 (&q)[4], float (&x)[2],
                                         float (&y)[2]) {
  float d0, d1, d2, d3;
  sub_h2(v.x, q[0].x, q[0].y, d0, d1);
  sub_h2(v.y, q[1].x, q[1].y, d2, d3);
  fma2_sq(x[0], y[0], d0, d1);
  fma2_sq(x[0], y[0], d2, d3);
  sub_h2(v.z, q[2].x, q[2].y, d0, d1);
  sub_h2(v.w, q[3].x, q[3].y, d2, d3);
  fma2_sq(x[1], y[1], d0, d1);
  fma2_sq(x[1], y[1], d2, d3);
}
__device__ __forceinline__ void widen(uint4 v, float2 (&q)[4]) {
  q[0] = h2lo(v.x);
  q[1] = h2lo(v.y);
  q[2] = h2lo(v.z);
  q[3] = h2lo(v.w);
}
// Keeps row a's sums (b's where `up`) and adds the partner's of the same row.
__device__ __forceinline__ void pass_half(float (&xa)[2], float (&ya)[2], const float (&xb)[2],
                                          const float (&yb)[2], bool up, int off) {
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const float kx = up ? xb[s] : xa[s], sx = up ? xa[s] : xb[s];
    const float ky = up ? yb[s] : ya[s], sy = up ? ya[s] : yb[s];
    xa[s] = kx;
    ya[s] = ky;
    add2(xa[s], ya[s], __shfl_xor_sync(kFull, sx, off), __shfl_xor_sync(kFull, sy, off));
  }
}

// Rows of D = 96 or 128 halves (one chunk per slot).
template <int D>
__device__ __forceinline__ float warp_rows32_fixed(const __half* q, const __half* __restrict__ base,
                                                   const uint32_t* ids, uint32_t m) {
  static_assert(D == 96 || D == 128, "whole units of four lanes");
  constexpr int U = D / 32;  // units per lane
  const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, j = lane & 3u;
  const uint4* Q = reinterpret_cast<const uint4*>(q) + j;
  const uint4* R[4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
    R[i] = reinterpret_cast<const uint4*>(base + (size_t)ids[min(8u * i + g, m - 1)] * D) + j;
  float x[4][2], y[4][2];
  // units k and k + 2 are level 1, the two sums level 2; slots without a chunk add
  // an exact zero
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    float2 q0[4], q1[4];
    widen(__ldg(Q + 4 * h), q0);
    if (h + 2 < U) widen(__ldg(Q + 4 * (h + 2)), q1);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (8u * i >= m) break;
      const uint4 v0 = __ldg(R[i] + 4 * h);
      uint4 v1 = v0;
      if (h + 2 < U) v1 = __ldg(R[i] + 4 * (h + 2));
      float x0[2] = {0.0f, 0.0f}, y0[2] = {0.0f, 0.0f};
      unit_acc(v0, q0, x0, y0);
      if (h + 2 < U) {
        float x1[2] = {0.0f, 0.0f}, y1[2] = {0.0f, 0.0f};
        unit_acc(v1, q1, x1, y1);
#pragma unroll
        for (int s = 0; s < 2; ++s) add2(x0[s], y0[s], x1[s], y1[s]);
      }
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        if (h == 0) {
          x[i][s] = x0[s];
          y[i][s] = y0[s];
        } else {
          add2(x[i][s], y[i][s], x0[s], y0[s]);
        }
      }
    }
  }
  pass_half(x[0], y[0], x[2], y[2], j & 2u, 2);
  pass_half(x[1], y[1], x[3], y[3], j & 2u, 2);
  pass_half(x[0], y[0], x[1], y[1], j & 1u, 1);
  add2(x[0][0], y[0][0], x[0][1], y[0][1]);
  return __fadd_rn(x[0][0], y[0][0]);
}

// Any width that is a multiple of four, 16 rows at a time.
template <bool kWide>
static __device__ __noinline__ float warp_rows32_any(const __half* q,
                                                     const __half* __restrict__ base, uint32_t dim,
                                                     const uint32_t* ids, uint32_t m) {
  const uint32_t lane = threadIdx.x & 31u, g = lane >> 2, j = lane & 3u;
  const uint32_t chunks = dim >> 2, units = (dim + 7) >> 3;
  const bool aligned = kWide && (dim & 7u) == 0;
  auto unit = [&](const __half* row, uint32_t u) {
    if (aligned) return __ldg(reinterpret_cast<const uint4*>(row) + u);
    const uint2* r = reinterpret_cast<const uint2*>(row);
    const uint2 a = __ldg(r + 2 * u);
    const uint2 b = 2 * u + 1 < chunks ? __ldg(r + 2 * u + 1) : make_uint2(0u, 0u);
    return make_uint4(a.x, a.y, b.x, b.y);
  };
  float half[2] = {0.0f, 0.0f};
#pragma unroll 1
  for (uint32_t b = 0; b < 2 && 16 * b < m; ++b) {
    const __half* R0 = base + (size_t)ids[min(16 * b + g, m - 1)] * dim;
    const __half* R1 = base + (size_t)ids[min(16 * b + 8 + g, m - 1)] * dim;
    float x[2][4][2], y[2][4][2];  // row, unit of the lane, slot of the unit
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int s = 0; s < 2; ++s) x[0][k][s] = y[0][k][s] = x[1][k][s] = y[1][k][s] = 0.0f;
#pragma unroll 1
    for (uint32_t u0 = 0; u0 < units; u0 += 16) {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t u = u0 + 4 * k + j;
        if (u < units) {
          float2 qf[4];
          widen(unit(q, u), qf);
          unit_acc(unit(R0, u), qf, x[0][k], y[0][k]);
          unit_acc(unit(R1, u), qf, x[1][k], y[1][k]);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        add2(x[i][0][s], y[i][0][s], x[i][2][s], y[i][2][s]);
        add2(x[i][1][s], y[i][1][s], x[i][3][s], y[i][3][s]);
        add2(x[i][0][s], y[i][0][s], x[i][1][s], y[i][1][s]);
      }
    pass_half(x[0][0], y[0][0], x[1][0], y[1][0], j & 2u, 2);
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const float ox = __shfl_xor_sync(kFull, x[0][0][s], 1),
                  oy = __shfl_xor_sync(kFull, y[0][0][s], 1);
      add2(x[0][0][s], y[0][0][s], ox, oy);
    }
    add2(x[0][0][0], y[0][0][0], x[0][0][1], y[0][0][1]);
    half[b] = __fadd_rn(x[0][0][0], y[0][0][0]);  // row 16 b + 8 (j / 2) + g
  }
  const float lo = __shfl_sync(kFull, half[0], (int)((lane & ~3u) + 2 * (j & 1u)));
  const float hi = __shfl_sync(kFull, half[1], (int)((lane & ~3u) + 2 * (j & 1u)));
  return j < 2 ? lo : hi;
}

// kWide: rows and query may be read 16 bytes at a time where the width allows it. At
// compile time: a flag carried through the collect costs it 2.6 ms of spills (79.7 ->
// 82.3 ms at 1M x 128).
template <bool kWide>
__device__ __forceinline__ float warp_rows32(const __half* q, const __half* __restrict__ base,
                                             uint32_t dim, const uint32_t* ids, uint32_t m) {
  if constexpr (kWide) {
    if (dim == 128) return warp_rows32_fixed<128>(q, base, ids, m);
    if (dim == 96) return warp_rows32_fixed<96>(q, base, ids, m);
  }
  return warp_rows32_any<kWide>(q, base, dim, ids, m);
}

// distance_filter (src/Tagore_src.cu:1488-1490) as nvcc compiles it, one fused
// multiply-add, and angle_filter (:1493-1495) with IEEE-rounded operations.
__device__ __forceinline__ bool pruned_by(int metric, float res, float dis, float cur, float thre) {
  if (metric == 0) return __fmaf_rn(thre, res, -dis) < 0.0f;
  float v = __fsub_rn(__fadd_rn(dis, cur), res);
  v = __fdiv_rn(v, 2.0f);
  v = __fdiv_rn(v, __fsqrt_rn(__fmul_rn(dis, cur)));
  return __fsub_rn(thre, v) < 0.0f;
}

// The reference's block-wide bitonic network (src/Tagore_src.cu:29-44),
// executed by one warp over shared arrays: strides 1,2,4,.., steps stride..1,
// the first step of each merge mirrored, pairs past `len` skipped. Each pass
// touches disjoint pairs, so lane order inside a pass does not matter; the
// swap sequence, and therefore tie placement, equals the reference's.
template <class Gt, class Sw>
__device__ __forceinline__ void warp_network(uint32_t len, int lane, Gt gt, Sw sw) {
  for (uint32_t stride = 1; stride < len; stride <<= 1) {
    for (uint32_t step = stride; step > 0; step >>= 1) {
      const uint32_t sh = __ffs(step) - 1;
      for (uint32_t k = lane; k < (len >> 1); k += 32) {
        const uint32_t a = (k >> sh) << (sh + 1), b = k & (step - 1);
        const uint32_t u = (step == stride) ? (a + step - 1 - b) : (a + b);
        const uint32_t d = a + b + step;
        if (d < len && gt(u, d)) sw(u, d);
      }
      __syncwarp();
    }
  }
}

template <class T>
__device__ __forceinline__ void swap_(T& a, T& b) {
  T t = a;
  a = b;
  b = t;
}

}  // namespace tagore
