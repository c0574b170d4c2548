// screen.cuh -- distance tests decided on tensor cores, for the prune kernels.
//
// A prune asks many times whether the distance of two rows is on one side of a
// value. screen_tile answers that for 32 rows against up to 16 by one warp: a Gram tile by mma.sync (FP16 operands, which are the base itself, so
// every product is exact in FP32), the screened distance n_r + n_q - 2 g, and a
// bound e on how far it can lie from the exact reference-order distance. A test
// whose sides differ by more than e is decided; the few others come back as
// ambiguous, and the caller takes the exact distance for them. So the answers
// are those of exact distances, and each row is gathered once per tile instead
// of once per test.
//
// mma.sync and not tcgen05: a node's tile is 32 x 16 and what it holds depends on
// the outcome of the tile before it, so a 128-row TMEM tile would be mostly
// empty and its shared-memory staging would cost the warps in flight that hide
// the gathers.
#pragma once
#include "common.cuh"

namespace tagore {

// e = kScreenEps * (n_r + n_q), times d / 1024 above 1,024 dims. The Gram sum is
// taken in groups of 64 dims: within a group each of the 64 exact products is
// added with an error of at most one ulp (2^-23, also if the tensor core
// truncates) of the group's largest partial sum, which Cauchy-Schwarz bounds by
// the group norms' product; over the groups that is 64 * 2^-23 * (n_r + n_q) / 2,
// so 2 g is within 2^-17 (n_r + n_q). The FP32 sum of the groups adds
// (d / 64) 2^-24, the two norms 2^-18.7 and the reference-order distance itself
// (at most 2 (n_r + n_q)) 2^-18.5: in all 1.37e-5, below 2^-16 = 1.53e-5.
constexpr float kScreenEps = 1.52587890625e-05f;

__host__ __device__ inline float screen_eps(uint32_t dim) {
  return dim <= 1024 ? kScreenEps : kScreenEps * (float)dim / 1024.0f;
}

__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                         uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The rule a test is taken by: metric 0, thre * res < dis (distance_filter);
// metric 1, the angle rule of pruned_by, in the form
// dis + cur - res > 2 thre sqrt(dis cur).
struct ScreenRule {
  int metric;
  float thre, eps;
};

// Decides one test from its screened distance: bit 0 the rule fires, bit 1
// ambiguous. The margins hold the rounding of these few operations too; a NaN
// compares false both ways and is ambiguous.
__device__ __forceinline__ uint32_t screen_test(const ScreenRule& r, float g, float nr, float nq,
                                                float dis, float cur) {
  const float n = nr + nq, res = fmaf(-2.0f, g, n), e = r.eps * n;
  float x, m;
  if (r.metric == 0) {
    x = fmaf(-r.thre, res, dis);
    m = fabsf(r.thre) * e;
  } else {
    const float s = 2.0f * r.thre * sqrt_approx(dis * cur), t = dis + cur;
    x = t - res - s;
    m = fmaf(9.5367431640625e-07f, t + fabsf(res) + fabsf(s), e);  // 2^-20
  }
  m += 1e-18f;
  return x > m ? 1u : (x < -m ? 0u : 2u);
}

// Columns of one screen, and the floats of shared memory a warp's tile takes.
constexpr uint32_t kScreenCols = 16;
constexpr uint32_t kScreenFloats = 32 * (kScreenCols + 1);

// One warp: lane r's row `id` (kInv: none; norm `nr`, distance to the node `dis`)
// against the rows bid[0, nb), nb <= kScreenCols, with norms bn and distances bd
// in shared memory. Lane r's result: bit q of x when the rule surely fires
// against row q, bit q of y when the screen cannot tell. With kAny the caller
// asks only whether some rule fires: a repeat of a column's id counts as firing,
// and the columns end once every row has one. Rows are multiples of 4 halves.
//
// Lane (g, t) = (lane / 4, lane % 4) loads 16-byte unit 4 j + t of rows g, g + 8,
// g + 16, g + 24 and of rows g and g + 8 of B: the same permutation of the
// dimensions for both operands, so the Gram sums are unchanged, and each load
// feeds two k = 16 steps. The tile goes through shared memory so that each lane
// tests its own row in a rolled loop: with the tests unrolled over the
// accumulators in 8, 16 and 32 column versions, two thirds of the filter's time
// went to instruction-cache misses (200K x 128 filter: 24.9 ms, now 6.1 ms).
template <bool kAligned, bool kAny>
static __device__ __noinline__ uint2 screen_tile(const __half* __restrict__ data, uint32_t dim,
                                                 ScreenRule rule, uint32_t id, float nr, float dis,
                                                 const uint32_t* bid, const float* bn,
                                                 const float* bd, uint32_t nb, float* tile) {
  constexpr int NT = kScreenCols / 8;
  const int lane = threadIdx.x & 31;
  const uint32_t g = (uint32_t)lane >> 2, t = (uint32_t)lane & 3u;
  const uint32_t chunks = dim >> 2, units = (chunks + 1) >> 1;  // the last unit may be half a unit
  const uint2* row[4 + NT];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t r = __shfl_sync(kFull, id, (int)(g + 8 * i));
    row[i] = reinterpret_cast<const uint2*>(data + (size_t)(r == kInv ? 0u : r) * dim);
  }
#pragma unroll
  for (int j = 0; j < NT; ++j) {
    const uint32_t q = 8 * j + g;
    row[4 + j] = reinterpret_cast<const uint2*>(data + (size_t)(q < nb ? bid[q] : 0u) * dim);
  }
  float acc[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[i][j][k] = 0.0f;
#pragma unroll 1
  for (uint32_t u0 = 0; u0 < units; u0 += 8) {  // 64 dims
    float part[2][NT][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) part[i][j][k] = 0.0f;
#pragma unroll
    for (uint32_t h = 0; h < 8; h += 4) {
      const uint32_t u = u0 + h + t;
      uint4 v[4 + NT];
#pragma unroll
      for (int i = 0; i < 4 + NT; ++i) {
        v[i] = make_uint4(0u, 0u, 0u, 0u);
        if (u < units) {
          if constexpr (kAligned) {
            v[i] = __ldg(reinterpret_cast<const uint4*>(row[i]) + u);
          } else {
            const uint2 lo = __ldg(row[i] + 2 * u);
            uint2 hi = make_uint2(0u, 0u);
            if (2 * u + 1 < chunks) hi = __ldg(row[i] + 2 * u + 1);
            v[i] = make_uint4(lo.x, lo.y, hi.x, hi.y);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const uint4 a = v[2 * i], c = v[2 * i + 1], b = v[4 + j];
          mma16816(part[i][j], a.x, c.x, a.y, c.y, b.x, b.y);
          mma16816(part[i][j], a.z, c.z, a.w, c.w, b.z, b.w);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[i][j][k] += part[i][j][k];
  }
  // lane (g, t) holds rows g + 8 i against columns 8 j + 2 t and 8 j + 2 t + 1
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int k = 0; k < 2; ++k)
        tile[(g + 8 * i) * (kScreenCols + 1) + 8 * j + 2 * t + k] =
            acc[i >> 1][j][2 * (i & 1) + k];
  __syncwarp();
  uint32_t fire = 0, amb = 0;
  const float* mine = tile + lane * (kScreenCols + 1);
#pragma unroll 1
  for (uint32_t q = 0; q < nb; ++q) {
    uint32_t v = screen_test(rule, mine[q], nr, bn[q], dis, bd[q]);
    if constexpr (kAny) v = bid[q] == id ? 1u : v;
    fire |= (v & 1u) << q;
    amb |= (v >> 1) << q;
    if constexpr (kAny)
      if (__all_sync(kFull, fire != 0 || id == kInv)) break;
  }
  return id == kInv ? make_uint2(0u, 0u) : make_uint2(fire, amb);
}

template <bool kAny>
__device__ __forceinline__ uint2 screen_rows(const __half* __restrict__ data, uint32_t dim,
                                             const ScreenRule& rule, uint32_t id, float nr,
                                             float dis, const uint32_t* bid, const float* bn,
                                             const float* bd, uint32_t nb, float* tile) {
  if (rows_of_16(data, dim))
    return screen_tile<true, kAny>(data, dim, rule, id, nr, dis, bid, bn, bd, nb, tile);
  return screen_tile<false, kAny>(data, dim, rule, id, nr, dis, bid, bn, bd, nb, tile);
}

}  // namespace tagore
