// search.cu -- batched greedy graph search: the recall evaluator for built
// indexes. It is NSG's search (src/common.cu:65-127): a sorted pool of L
// candidates, each expanded once in pool order, its unseen neighbours scored
// and merged; the pool starts from the entry point's neighbours, topped up to
// L with seeded random nodes (seed != 0) or preceded by the entry point itself
// (seed == 0).
//
// Layout: one warp per query, queries taken from a counter by a resident grid.
// The query, the pool and its merge buffer sit in shared memory. The visited set
// is an open-addressing table in shared memory; ids past its share go to a
// table in global memory whose keys carry the query number in their high half
// and which a warp clears when it first needs it.
//
// The visiting order is the sequential one, done 32 ids at a time: a batch of
// neighbours (in adjacency order) is deduplicated with __match_any_sync, the
// unseen ones are scored, and the batch is merged into the pool as if the ids
// had been inserted one by one -- a pool entry goes before a new one at equal
// distance, earlier new ones before later ones. Distances are summed in
// dimension order with round-to-nearest adds and multiplies (no contraction),
// the same arithmetic as a plain C loop, so the result equals the sequential
// search id for id.
//
// What bounds it: the sum's order makes each distance one chain of `dim`
// dependent adds, so that chain is all a lane does alone. The squared
// differences are made by the whole warp, which reads the rows coalesced
// (several rows per load, next chunk ahead of the chain) and leaves the squares
// in a shared tile, row per chain. The next expansion's list is loaded during
// the current one, and a batch that lies beyond a full pool is not merged.
// 10,000 queries, L = 128, 100K x 128: 7.43 ms with a lane per row and all visited
// ids in a global table (310 MB of tables over the chip, cleared by each call), 3.28
// ms now; with 1,024 probed slots of shared memory in place of the buckets, 8.2 ms,
// since a query visits more than that.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "internal.h"

namespace tagore {
namespace {

constexpr uint32_t kOpen = 0x80000000u;  // pool entry not yet expanded
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint64_t kGold = 0x9E3779B97F4A7C15ull;
constexpr uint32_t kBlockWarps = 2, kSmWarps = 16;  // per block, and at most per SM
constexpr uint32_t kMul0 = 0x9E3779B1u, kMul1 = 0x85EBCA6Bu;  // odd: bijections mod 2^b
constexpr uint32_t kMinNear = 7, kMaxNear = 10;  // log2 of the shared table's buckets

struct Entry {
  float d;
  uint32_t id;  // | kOpen while unexpanded
};

struct SearchArgs {
  const float* base;
  uint32_t n, dim;
  const uint64_t* offs;
  const uint32_t* adj;
  uint64_t edges;
  uint32_t ep;
  const float* queries;
  uint32_t nq;
  uint32_t L, k;
  uint64_t seed;
  uint32_t cap_log2, near_log2, id_bits;  // of the visited tables (Visited)
  uint32_t lanes_log2;           // lanes that share a row's load
  unsigned long long* table;
  uint32_t* out;
  uint32_t *next, *err;
};

// splitmix64's output function (Steele, Lea and Flood, OOPSLA 2014).
__device__ __forceinline__ uint64_t mix64(uint64_t x) {
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

// Visited set of one query. Its first part is a table in shared memory: buckets of
// eight 16-bit remainders, an id in the emptier of two buckets. The hashes are
// bijections of [0, 2^id_bits) (odd multipliers), so bucket, remainder and the hash
// it comes from (the lowest of the 16 bits) name the id exactly. An id whose two
// buckets are full goes to `tab`, 2^cap_log2 slots in global memory probed linearly
// and filled to half at most, whose keys carry the query number in their high half
// and which a warp clears when it first needs it. Only the owning warp touches
// either; reads of `tab` go to L2 (ld.cg) so a slot claimed by another lane's
// atomicCAS is never read stale from L1.
struct Visited {
  unsigned long long* tab;
  uint4* bucket;
  uint32_t* count;  // a byte per bucket
  uint32_t cap_log2, near_log2, id_bits;  // near_log2: log2 of the buckets, 0 for none
  uint32_t tag;  // query number + 1
  bool spilled, cleared;  // this query uses `tab`; this warp has cleared it

  __device__ __forceinline__ void start(uint32_t q, uint32_t lane) {
    tag = q + 1;
    spilled = false;
    if (near_log2) {
      for (uint32_t i = lane; i < (1u << near_log2); i += 32)
        bucket[i] = make_uint4(kNone, kNone, kNone, kNone);
      for (uint32_t i = lane; i < (1u << near_log2) / 16; i += 32)
        reinterpret_cast<uint4*>(count)[i] = make_uint4(0, 0, 0, 0);
    }
    __syncwarp();
  }
  __device__ __forceinline__ uint32_t hash(uint32_t id, uint32_t mul) const {
    return (id * mul) & ((1u << id_bits) - 1u);
  }
  __device__ __forceinline__ uint32_t held(uint32_t b) const {
    return (count[b >> 2] >> (8 * (b & 3u))) & 255u;
  }
  // Whether bucket b holds remainder r: whether one of its halves equals it. The
  // borrow of the test starts in a half that is equal, so it adds no false hit.
  __device__ __forceinline__ bool in_bucket(uint32_t b, uint32_t r) const {
    const uint4 v = bucket[b];
    const uint32_t rr = r * 0x10001u;
    auto equal = [rr](uint32_t w) { return ((w ^ rr) - 0x00010001u) & ~(w ^ rr); };
    return ((equal(v.x) | equal(v.y) | equal(v.z) | equal(v.w)) & 0x80008000u) != 0;
  }
  __device__ __forceinline__ bool contains(uint32_t id) const {
    if (near_log2) {
      const uint32_t rbits = id_bits - near_log2, rmask = (1u << rbits) - 1u;
      const uint32_t x = hash(id, kMul0), y = hash(id, kMul1);
      const uint32_t bx = x >> rbits, by = y >> rbits;
      if (in_bucket(bx, (x & rmask) << 1) || in_bucket(by, (y & rmask) << 1 | 1u)) return true;
      if (!spilled || held(bx) < 8 || held(by) < 8) return false;
    } else if (!spilled) {
      return false;
    }
    const uint32_t mask = (1u << cap_log2) - 1u;
    for (uint32_t h = (id * kMul0) >> (32u - cap_log2);; h = (h + 1) & mask) {
      const unsigned long long v = __ldcg(tab + h);
      if ((uint32_t)(v >> 32) != tag) return false;
      if ((uint32_t)v == id) return true;
    }
  }
  __device__ __forceinline__ bool put(uint32_t b, uint32_t r) {
    const uint32_t s = 8 * (b & 3u);
    const uint32_t at = (atomicAdd(count + (b >> 2), 1u << s) >> s) & 255u;
    if (at >= 8) return false;  // at most 32 lanes add past a full bucket
    reinterpret_cast<uint16_t*>(bucket + b)[at] = (uint16_t)r;
    return true;
  }
  // Inserts the ids of the lanes with `take`, none of which is in the set. By the
  // whole warp.
  __device__ __forceinline__ void insert(uint32_t id, bool take, uint32_t lane) {
    bool left = take;
    if (near_log2 && take) {
      const uint32_t rbits = id_bits - near_log2, rmask = (1u << rbits) - 1u;
      const uint32_t x = hash(id, kMul0), y = hash(id, kMul1);
      const uint32_t bx = x >> rbits, by = y >> rbits;
      const uint32_t nx = held(bx), ny = held(by);
      const uint32_t rx = (x & rmask) << 1, ry = (y & rmask) << 1 | 1u;
      const bool second = ny < nx;
      if ((second ? ny : nx) < 8) left = !put(second ? by : bx, second ? ry : rx);
      if (left && held(second ? bx : by) < 8) left = !put(second ? bx : by, second ? rx : ry);
    }
    if (!__any_sync(~0u, left)) return;
    spilled = true;
    if (!cleared) {
      const uint32_t slots = 1u << cap_log2;
      for (uint32_t i = lane; i < slots / 2; i += 32)
        __stcg(reinterpret_cast<ulonglong2*>(tab) + i, make_ulonglong2(0, 0));
      cleared = true;
      __threadfence();
      __syncwarp();
    }
    if (!left) return;
    const uint32_t mask = (1u << cap_log2) - 1u;
    const unsigned long long key = ((unsigned long long)tag << 32) | id;
    for (uint32_t h = (id * kMul0) >> (32u - cap_log2);;) {
      const unsigned long long v = __ldcg(tab + h);
      if ((uint32_t)(v >> 32) != tag) {
        if (atomicCAS(tab + h, v, key) == v) return;
        continue;  // another lane took the slot: read it again
      }
      h = (h + 1) & mask;
    }
  }
};

// (a - q)^2 of two dimension pairs; nq = -q, and the square has the bits of
// (q - a)^2.
__device__ __forceinline__ float4 sq_diff(float4 v, float4 nq) {
  float4 r;
  asm("{.reg .b64 a, b, p, q;\n\t"
      "mov.b64 a, {%4, %5};\n\t"
      "mov.b64 b, {%6, %7};\n\t"
      "mov.b64 p, {%8, %9};\n\t"
      "mov.b64 q, {%10, %11};\n\t"
      "add.rn.f32x2 a, a, p;\n\t"
      "add.rn.f32x2 b, b, q;\n\t"
      "mul.rn.f32x2 a, a, a;\n\t"
      "mul.rn.f32x2 b, b, b;\n\t"
      "mov.b64 {%0, %1}, a;\n\t"
      "mov.b64 {%2, %3}, b;}"
      : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w)
      : "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "f"(nq.x), "f"(nq.y), "f"(nq.z), "f"(nq.w));
  return r;
}

// Unit j (four dims) of a row; dims past `dim` are zero.
template <bool kVec>
__device__ __forceinline__ float4 row_unit(const float* __restrict__ y, uint32_t j, uint32_t dim) {
  if (kVec) return __ldg(reinterpret_cast<const float4*>(y) + j);
  const uint32_t at = 4 * j;
  float4 v;
  v.x = __ldg(y + at);
  v.y = at + 1 < dim ? __ldg(y + at + 1) : 0.0f;
  v.z = at + 2 < dim ? __ldg(y + at + 2) : 0.0f;
  v.w = at + 3 < dim ? __ldg(y + at + 3) : 0.0f;
  return v;
}

__device__ __forceinline__ void chain4(float& acc, float4 s) {
  acc = __fadd_rn(acc, s.x);
  acc = __fadd_rn(acc, s.y);
  acc = __fadd_rn(acc, s.z);
  acc = __fadd_rn(acc, s.w);
}

// Tile of squares (64 dims per row: 4.66 ms, 32: 4.09 ms, by the warps that fit):
// 32 rows of kUnits 16-byte units, one unit of padding per row so that eight lanes
// reading a unit each of eight rows meet no bank twice.
constexpr uint32_t kUnits = 8, kRowFloats = 4 * kUnits + 4;
constexpr uint32_t kAhead = 4;  // loads in flight per lane

// Shared bytes per warp in front of the tile and the near table.
__host__ __device__ inline size_t pool_bytes(uint32_t dim, uint32_t L) {
  return (size_t)((dim + 3) & ~3u) * 4 + 2ull * L * sizeof(Entry) + 32 * 4;
}
__host__ __device__ inline size_t tile_bytes() { return 32 * kRowFloats * 4; }

// The shared visited table: 2^near_log2 buckets of 16 bytes and their counts.
__host__ __device__ inline size_t near_bytes(uint32_t near_log2) {
  return near_log2 ? (size_t)17 << near_log2 : 0;
}

template <bool kVec, bool kTile>
struct WarpSearch {
  const SearchArgs& a;
  uint32_t lane;
  float* qv;       // query, negated, padded with zeros to whole units
  Entry* P;        // pool, `size` entries sorted by (d, arrival)
  Entry* Q;        // merge target
  float* fresh_d;  // the batch's new distances in sorted order
  float* tile;     // squares
  uint32_t* row_id;  // the batch's rows
  Visited vis;
  uint32_t size, touched, limit;
  uint32_t low;  // pool entries before this one are expanded
  bool over;
  // the list expected next: its node, its range and its first 32 ids
  uint32_t ahead_u, ahead_id;
  uint64_t ahead_lo, ahead_hi;
  // the current list: what is left of it, and its first 32 ids
  uint64_t at, end;
  uint32_t first_id;
  bool first;

  // Loads the first ids of the expected list; its range has been asked for long
  // enough ago.
  __device__ __forceinline__ void load_ahead() {
    if (ahead_u == kNone) return;
    ahead_hi = min(ahead_hi, a.edges);
    ahead_id = ahead_lo + lane < ahead_hi ? __ldg(a.adj + ahead_lo + lane) : kNone;
  }

  // Distance of row row_id[lane] for lane < m.
  __device__ __forceinline__ float score(uint32_t m) {
    const uint32_t units = (a.dim + 3) / 4;
    float acc = 0.0f;
    if (!kTile) {
      load_ahead();
      if (lane < m) {
        const float* y = a.base + (size_t)row_id[lane] * a.dim;
        const float4* q4 = reinterpret_cast<const float4*>(qv);
#pragma unroll 4
        for (uint32_t j = 0; j < units; ++j)
          chain4(acc, sq_diff(row_unit<kVec>(y, j, a.dim), q4[j]));
      }
      __syncwarp();
      return acc;
    }
    const uint32_t sub = lane & ((1u << a.lanes_log2) - 1u), grp = lane >> a.lanes_log2;
    const uint32_t step = 32u >> a.lanes_log2;  // rows per load
    float4 v[kAhead];
    auto load = [&](uint32_t r0, uint32_t u) {
#pragma unroll
      for (uint32_t i = 0; i < kAhead; ++i) {
        const uint32_t r = r0 + i * step + grp;
        if (r0 + i * step < m && r < m && u < units)
          v[i] = row_unit<kVec>(a.base + (size_t)row_id[r] * a.dim, u, a.dim);
      }
    };
    load(0, sub);
    load_ahead();
    for (uint32_t c = 0; c < units; c += kUnits) {
      const uint32_t u = c + sub, left = min(units - c, kUnits);
      const float4 nq = u < units ? reinterpret_cast<const float4*>(qv)[u] : make_float4(0, 0, 0, 0);
      for (uint32_t r0 = 0; r0 < m; r0 += kAhead * step) {
        if (r0) load(r0, u);
#pragma unroll
        for (uint32_t i = 0; i < kAhead; ++i) {
          const uint32_t r = r0 + i * step + grp;
          if (r0 + i * step < m && r < m && u < units)
            *reinterpret_cast<float4*>(tile + r * kRowFloats + 4 * sub) = sq_diff(v[i], nq);
        }
      }
      __syncwarp();
      if (c + kUnits < units) load(0, u + kUnits);
      if (lane < m) {
        const float4* s = reinterpret_cast<const float4*>(tile + lane * kRowFloats);
        if (left == kUnits) {
#pragma unroll
          for (uint32_t j = 0; j < kUnits; ++j) chain4(acc, s[j]);
        } else {
          for (uint32_t j = 0; j < left; ++j) chain4(acc, s[j]);
        }
      }
      __syncwarp();
    }
    return acc;
  }

  // Visits the ids of the active lanes in lane order; at most `need` unseen
  // ones are taken (the rest stay unvisited).
  __device__ __forceinline__ void batch(uint32_t id, bool active, uint32_t need) {
    const bool valid = active && id < a.n;
    const uint32_t same = __match_any_sync(~0u, valid ? id : kNone);
    const bool first = valid && (uint32_t)(__ffs(same) - 1) == lane;
    const bool unseen = first && !vis.contains(id);
    const uint32_t ub = __ballot_sync(~0u, unseen);
    const bool take = unseen && (uint32_t)__popc(ub & ((1u << lane) - 1u)) < need;
    const uint32_t tb = __ballot_sync(~0u, take);
    uint32_t m = __popc(tb);
    if (m == 0 || touched + m > limit) {
      over = m != 0;
      load_ahead();
      return;
    }
    touched += m;
    vis.insert(id, take, lane);
    if (take) row_id[__popc(tb & ((1u << lane) - 1u))] = id;
    __syncwarp();
    // lane i < m holds the batch's i-th new entry from here on
    const uint32_t mine = lane < m ? row_id[lane] : kNone;
    // A NaN ranks as infinite: the places below need an order of all distances, or
    // two entries take one place and another keeps a stale id.
    const float d = fminf(score(m), INFINITY);
    // with a full pool, one no closer than its last entry changes nothing
    const uint32_t L = a.L;
    const bool enter = lane < m && !(size == L && P[L - 1].d <= d);
    const uint32_t eb = __ballot_sync(~0u, enter);
    m = __popc(eb);
    if (m == 0) return;
    // Rank among the batch's new entries: earlier lanes first on ties.
    uint32_t within = 0;
    for (uint32_t b = eb; b; b &= b - 1) {
      const uint32_t j = __ffs(b) - 1;
      const float dj = __shfl_sync(~0u, d, j);
      within += (dj < d) || (dj == d && j < lane);
    }
    if (enter) fresh_d[within] = d;
    __syncwarp();
    for (uint32_t p = lane; p < size; p += 32) {
      const Entry e = P[p];
      uint32_t lo = 0, hi = m;  // new entries strictly closer than e
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (fresh_d[mid] < e.d) lo = mid + 1;
        else hi = mid;
      }
      if (p + lo < L) Q[p + lo] = e;
    }
    uint32_t place = kNone;
    if (enter) {
      uint32_t lo = 0, hi = size;  // pool entries at most as far as d
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (P[mid].d <= d) lo = mid + 1;
        else hi = mid;
      }
      place = lo + within;
      if (place < L) Q[place] = Entry{d, mine | kOpen};
    }
    low = min(low, __reduce_min_sync(~0u, place));
    __syncwarp();
    size = min(L, size + m);
    Entry* t = P;
    P = Q;
    Q = t;
  }

  // Makes u's list the current one; `next` is the node whose list is expected
  // after it.
  __device__ __forceinline__ void open_list(uint32_t u, uint32_t next) {
    if (u == ahead_u) {
      at = ahead_lo;
      end = ahead_hi;
      first_id = ahead_id;
    } else {
      at = a.offs[u];
      end = min(a.offs[u + 1], a.edges);
      first_id = at + lane < end ? __ldg(a.adj + at + lane) : kNone;
    }
    first = true;
    ahead_u = next;
    if (next != kNone) {
      ahead_lo = a.offs[next];
      ahead_hi = a.offs[next + 1];
      if (at >= end) load_ahead();
    }
  }

  __device__ __forceinline__ void run(uint32_t q) {
    size = 0;
    touched = 0;
    low = 0;
    over = false;
    ahead_u = kNone;
    at = end = 0;
    vis.start(q, lane);
    for (uint32_t j = lane; j < ((a.dim + 3) & ~3u); j += 32)
      qv[j] = j < a.dim ? -a.queries[(size_t)q * a.dim + j] : 0.0f;
    __syncwarp();
    // The batches in order: the entry point alone (seed 0), its list, random
    // nodes (seed != 0), then the lists of the pool's open entries; one call of
    // batch() serves all, so its code is there once.
    enum { kEntry, kEntryList, kRandom, kExpand };
    int phase = a.seed == 0 ? kEntry : kEntryList;
    // splitmix64's stream: z advances by the golden gamma per draw, lane i
    // takes draw i of the batch, and a batch that fills the pool ends it.
    uint64_t z = a.seed ^ (kGold * (uint64_t)(q + 1));
    const uint32_t want = min(a.L, a.n);
    while (!over) {
      uint32_t id = kNone, need = kNone;
      bool act = true;
      if (at < end) {
        act = at + lane < end;
        id = first ? first_id : act ? __ldg(a.adj + at + lane) : kNone;
        first = false;
        at += 32;
      } else if (phase == kExpand) {
        // The first open entry, and the one after it in the same 32. Every
        // expansion closes an entry that was opened by a first visit, so the
        // loop ends.
        int idx = -1, then = -1;
        for (uint32_t c = low & ~31u; c < size; c += 32) {
          const bool open = c + lane < size && (P[c + lane].id & kOpen);
          const uint32_t b = __ballot_sync(~0u, open);
          if (b) {
            idx = (int)(c + __ffs(b) - 1);
            const uint32_t b2 = b & (b - 1);
            if (b2) then = (int)(c + __ffs(b2) - 1);
            break;
          }
        }
        if (idx < 0) break;
        const uint32_t u = P[idx].id & ~kOpen;
        const uint32_t next = then < 0 ? kNone : P[then].id & ~kOpen;
        __syncwarp();
        if (lane == 0) P[idx].id = u;
        low = idx;
        __syncwarp();
        open_list(u, next);
        continue;
      } else if (phase == kEntry) {
        id = a.ep;
        act = lane == 0;
        phase = kEntryList;
      } else if (phase == kEntryList) {
        phase = a.seed == 0 ? kExpand : kRandom;
        open_list(a.ep, kNone);
        continue;
      } else {
        if (touched >= want) {
          phase = kExpand;
          continue;
        }
        id = (uint32_t)(mix64(z + kGold * (uint64_t)(lane + 1)) % (uint64_t)a.n);
        need = want - touched;
        z += kGold * 32ull;
      }
      batch(id, act, need);
    }
    for (uint32_t j = lane; j < a.k; j += 32)
      a.out[(size_t)q * a.k + j] = (over || j >= size) ? kNone : (P[j].id & ~kOpen);
    if (over && lane == 0) atomicOr(a.err, 1u);
    __syncwarp();
  }
};

template <bool kVec, bool kTile>
__global__ void __launch_bounds__(kBlockWarps * 32, kSmWarps / kBlockWarps) k_search(const __grid_constant__ SearchArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t nw = blockDim.x >> 5;
  const size_t pool = pool_bytes(a.dim, a.L), tile = kTile ? tile_bytes() : 0;
  const size_t near = near_bytes(a.near_log2);
  unsigned char* mine = smem + wib * (pool + tile + near);
  WarpSearch<kVec, kTile> w{a, lane};
  w.qv = reinterpret_cast<float*>(mine);
  w.P = reinterpret_cast<Entry*>(mine + (size_t)((a.dim + 3) & ~3u) * 4);
  w.Q = w.P + a.L;
  w.fresh_d = reinterpret_cast<float*>(w.Q + a.L);
  w.row_id = reinterpret_cast<uint32_t*>(w.fresh_d);  // read before fresh_d is written
  w.tile = reinterpret_cast<float*>(mine + pool);
  const uint32_t gwarp = blockIdx.x * nw + wib;
  w.vis.tab = a.table + ((size_t)gwarp << a.cap_log2);
  w.vis.bucket = reinterpret_cast<uint4*>(mine + pool + tile);
  w.vis.count = reinterpret_cast<uint32_t*>(w.vis.bucket + (1u << a.near_log2));
  w.vis.id_bits = a.id_bits;
  w.vis.cap_log2 = a.cap_log2;
  w.vis.near_log2 = a.near_log2;
  w.vis.cleared = false;
  w.limit = 1u << (a.cap_log2 - 1);
  for (;;) {
    uint32_t q = 0;
    if (lane == 0) q = atomicAdd(a.next, 1u);
    q = __shfl_sync(~0u, q, 0);
    if (q >= a.nq) break;
    w.run(q);
  }
}

uint32_t ceil_log2(uint64_t v) {
  uint32_t r = 0;
  while ((1ull << r) < v) ++r;
  return r;
}

}  // namespace

int search_check(const TagoreSearchParams& p, const float* base, uint64_t n, uint32_t dim,
                 const uint64_t* offs, const uint32_t* adj, uint64_t edges, uint32_t ep,
                 const float* queries, uint32_t nq, const uint32_t* out) {
  if (n == 0 || n >= kOpen || dim == 0 || p.L == 0 || p.k == 0)
    return fail(TAGORE_EINVAL, "search: need 0 < n < 2^31 and dim, L, k > 0");
  if (ep >= n) return fail(TAGORE_EINVAL, "search: entry point %u outside %llu nodes", ep,
                           (unsigned long long)n);
  if (p.visit_cap > (1u << 28)) return fail(TAGORE_EINVAL, "search: visit_cap above 2^28");
  if (nq == 0) return TAGORE_OK;
  if (!base || !offs || (!adj && edges) || !queries || !out)
    return fail(TAGORE_EINVAL, "search: null pointer");
  return TAGORE_OK;
}

int greedy_search(const TagoreSearchParams& p, const float* base, uint64_t n, uint32_t dim,
                  const uint64_t* offs, const uint32_t* adj, uint64_t edges, uint32_t ep,
                  const float* queries, uint32_t nq, uint32_t* out, cudaStream_t s) {
  TG_TRY(search_check(p, base, n, dim, offs, adj, edges, ep, queries, nq, out));
  if (nq == 0) return TAGORE_OK;
  uint32_t cap_log2 = p.visit_cap ? ceil_log2(p.visit_cap) : ceil_log2(64ull * p.L);
  if (cap_log2 < 14) cap_log2 = 14;

  int dev = 0, sms = 0, smem_max = 0;
  TG_CUDA(cudaGetDevice(&dev));
  TG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  TG_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  const size_t pool = pool_bytes(dim, p.L);
  if (pool > (size_t)smem_max)
    return fail(TAGORE_EINVAL, "search: dim %u with L %u needs %zu B of shared memory per warp",
                dim, p.L, pool);
  // A pool that leaves no room for the tile is searched without it, each lane
  // reading its own rows; one that leaves none for the near table keeps all
  // its visited ids in global memory.
  const bool tile = pool + tile_bytes() <= (size_t)smem_max;
  size_t per_warp = pool + (tile ? tile_bytes() : 0);
  // A query visits a few times L lists; at four ids a bucket almost none spills.
  // Remainders have 14 bits (with the hash's bit never all ones, an empty place),
  // so more than 2^14 ids per bucket take more buckets.
  const uint32_t id_bits = std::max(kMinNear, ceil_log2(n));
  const uint64_t ids = (uint64_t)p.L * (1 + edges / n);
  uint32_t near_log2 = std::min({kMaxNear, std::max(kMinNear, ceil_log2((ids + 3) / 4)), id_bits});
  if (id_bits > near_log2 + 14) near_log2 = id_bits - 14;
  if (near_log2 > kMaxNear + 1 || per_warp + near_bytes(near_log2) > (size_t)smem_max) near_log2 = 0;
  per_warp += near_bytes(near_log2);
  // Few queries: a warp on each SM before a second one on any. Two warps per block
  // leave less of an SM's shared memory unused than four (3.28 ms against 3.57).
  const uint32_t nw = (uint32_t)std::min<size_t>({kBlockWarps, (size_t)smem_max / per_warp,
                                                  std::max<size_t>(1, (nq + sms - 1) / sms)});
  const bool vec = dim % 4 == 0 && ((uintptr_t)base & 15) == 0;
  using Kernel = void (*)(const SearchArgs);
  const Kernel fn = tile ? (vec ? k_search<true, true> : k_search<false, true>)
                         : (vec ? k_search<true, false> : k_search<false, false>);
  const size_t smem = per_warp * nw;
  TG_CUDA(cudaFuncSetAttribute((const void*)fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem));
  int per_sm = 0;
  TG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, (const void*)fn, nw * 32, smem));
  per_sm = std::max(1, std::min(per_sm, (int)(kSmWarps / nw)));
  const uint64_t want = (nq + nw - 1) / nw;
  const uint32_t grid = (uint32_t)std::min<uint64_t>(want, (uint64_t)sms * per_sm);
  const uint32_t units = (dim + 3) / 4;
  uint32_t lanes_log2 = 0;
  while ((1u << lanes_log2) < std::min(units, kUnits)) ++lanes_log2;

  Scratch tab(s);
  const size_t tab_bytes = ((size_t)grid * nw << cap_log2) * sizeof(unsigned long long);
  TG_TRY(tab.alloc(tab_bytes + 16));
  uint32_t* ctl = reinterpret_cast<uint32_t*>(tab.as<unsigned char>() + tab_bytes);
  TG_CUDA(cudaMemsetAsync(ctl, 0, 16, s));
  SearchArgs a{base, (uint32_t)n, dim, offs, adj, edges, ep, queries, nq, p.L, p.k, p.seed, cap_log2,
               near_log2, id_bits, lanes_log2, tab.as<unsigned long long>(), out, ctl,
               ctl + 1};
  stage_begin("search", s);
  fn<<<grid, nw * 32, smem, s>>>(a);
  TG_CUDA(cudaGetLastError());
  count_launch();
  stage_end("search", s, 0, nq);
  uint32_t err = 0;
  TG_CUDA(cudaMemcpyAsync(&err, a.err, 4, cudaMemcpyDeviceToHost, s));
  TG_CUDA(cudaStreamSynchronize(s));
  if (err) return fail(TAGORE_EINVAL, "search: a query visited more than %u nodes; raise visit_cap",
                       1u << (cap_log2 - 1));
  return TAGORE_OK;
}

}  // namespace tagore
