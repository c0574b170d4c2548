// prune.cu -- Collect / Filter / Store prune of a kNN graph on sm_100a.
//
// Restates the CFS framework of ZJU-DAILY/Tagore (src/Tagore_src.cu:1209-2058,
// pybind.cu:145-295) with one warp per node and results that are a function of
// the input graph only:
//  * every distance is FP32 arithmetic on the FP16 base in the reference's
//    lane order (common.cuh), every sort is the reference's bitonic network on
//    the same positions, so ties fall where the reference puts them;
//  * the Collect stage reads the kNN graph as a snapshot: pruned rows go to
//    scratch and reach `graph` only in the Store stage;
//  * reverse edges are inserted in ascending source order (a stable radix sort
//    by target), so the reference's replacement rule for full lists
//    (:1465-1475, :1697-1707) gives one defined answer;
//  * the Filter stage is evaluated lazily: a candidate is tested against the
//    kept neighbours before it and dropped when any rule fires, which keeps
//    exactly the set the reference's round-by-round sweep (:1416-1460) keeps;
//    the tests are decided on tensor cores where the screened distance is clear
//    of the rule's value by its error bound (screen.cuh), and by the exact
//    distance where it is not.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <string>

#include "common.cuh"
#include "internal.h"
#include "knn_shared.cuh"
#include "screen.cuh"

namespace tagore {
namespace {

constexpr int kWarps = 4;  // warps (= nodes in flight) per block


// ---------------------------------------------------------------------------
// Beam search shared by cal_ep_gpu (:1905-2047) and collect_path (:1211-1335).
// The helpers below are __noinline__ and their sorts rolled: the warps sit in
// different phases, so one small copy of each sort and merge keeps the code they
// run within the instruction cache. Inlined copies at every call site cost 8 % of
// the select at 1M points; the sorts with their passes unrolled, 10.6 of the
// collect's 89.8 ms.
struct Beam {
  uint32_t* id;
  float* dis;
  uint8_t* ex;
  // membership set of the W beam ids, as chains: heads, the ids as they were when
  // the set was made, and links
  uint32_t *head, *nid;
  uint16_t* next;
  float* sb;       // scratch (K): the fresh positions, then sorted entering distances
  float* sm;       // staging: merged distances of positions 0..TOPM, or K entering ones
  uint32_t* sid;   // staging: their ids
  uint8_t* sex;    // staging: their explored flags
};

constexpr uint32_t kBeamHeads = 256;

__host__ __device__ inline size_t beam_bytes(uint32_t topm, uint32_t K) {
  const uint32_t W = topm + K, S = topm + 1 > K ? topm + 1 : K;
  return kBeamHeads * 4 + (size_t)W * 12 + K * 4 + (size_t)S * 8 + ((W * 2 + 3u) & ~3u) + W +
         topm + 1;
}

__device__ inline Beam beam_carve(unsigned char* p, uint32_t topm, uint32_t K) {
  const uint32_t W = topm + K, S = topm + 1 > K ? topm + 1 : K;
  Beam b;
  b.head = reinterpret_cast<uint32_t*>(p);
  b.id = b.head + kBeamHeads;
  b.dis = reinterpret_cast<float*>(b.id + W);
  b.nid = reinterpret_cast<uint32_t*>(b.dis + W);
  b.sb = reinterpret_cast<float*>(b.nid + W);
  b.sm = b.sb + K;
  b.sid = reinterpret_cast<uint32_t*>(b.sm + S);
  b.next = reinterpret_cast<uint16_t*>(b.sid + S);
  b.ex = reinterpret_cast<uint8_t*>(b.next) + ((W * 2 + 3u) & ~3u);
  b.sex = b.ex + W;
  return b;
}

__device__ __forceinline__ uint32_t beam_head(uint32_t key) { return (key * 0x9E3779B1u) >> 24; }

// The reference keeps the beam ids sorted (top_M_Cand2, :1253-1259) only to
// test membership (:1282-1290); a set of the same ids answers the same question
// without a sort. Chains take one exchange per id, where a probed table's 32
// lanes wait for the longest run of tries among them.
__device__ __noinline__ void beam_rehash(Beam bm, uint32_t W, int lane) {
#pragma unroll
  for (uint32_t t = lane; t < kBeamHeads / 4; t += 32)
    reinterpret_cast<uint4*>(bm.head)[t] = make_uint4(kInv, kInv, kInv, kInv);
  __syncwarp();
  for (uint32_t t = lane; t < W; t += 32) {
    const uint32_t key = bm.id[t];
    if (key == kInv) continue;
    bm.nid[t] = key;
    bm.next[t] = (uint16_t)atomicExch(&bm.head[beam_head(key)], t);
  }
  __syncwarp();
}

__device__ __forceinline__ bool beam_has(const Beam& bm, uint32_t key) {
  uint32_t t = bm.head[beam_head(key)];
  while ((t & 0xFFFFu) != 0xFFFFu) {
    if (bm.nid[t] == key) return true;
    t = bm.next[t];
  }
  return false;
}

__device__ __noinline__ void beam_network(Beam bm, uint32_t off, uint32_t len, int lane) {
  float* D = bm.dis + off;
  uint32_t* I = bm.id + off;
  uint8_t* E = bm.ex + off;
  warp_network(len, lane, [&](uint32_t u, uint32_t d) { return D[u] > D[d]; },
               [&](uint32_t u, uint32_t d) {
                 swap_(D[u], D[d]);
                 swap_(I[u], I[d]);
                 swap_(E[u], E[d]);
               });
}

// kSolo: the entry point's beam, one warp on an idle chip, which waits for latency
// alone: its sorts are unrolled and its rows read by a lane each, all their loads at
// once (at 1M x 128, K = 96, TOPM 64: 0.33 ms, with the collect's forms 0.45 ms).
template <bool kSolo, int E>
__device__ __forceinline__ void sort_keys(uint64_t (&key)[E], int lane) {
  if constexpr (kSolo) knn::warp_sort_keys<E>(key, lane);
  else knn::warp_sort_keys_rolled<E>(key, lane);
}

// Sorted (distance, position) keys of the n <= 128 entries at [off, off+n),
// element-major in four registers per lane.
template <bool kSolo>
__device__ __forceinline__ void sorted_keys(const Beam& bm, uint32_t off, uint32_t n, uint64_t (&key)[4],
                                            int lane) {
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    const uint32_t j = lane + 32 * t;
    key[t] = j < n ? (((uint64_t)__float_as_uint(bm.dis[off + j]) << 32) | j) : ~0ull;
  }
  sort_keys<kSolo, 4>(key, lane);
}

__device__ __forceinline__ float key_dis(uint64_t k) { return __uint_as_float((uint32_t)(k >> 32)); }

// Merges the m entering entries, whose (distance, slot) keys sit in sm/sid
// [0, m), into the sorted prefix [0, topm) by rank, through the staging
// arrays. Returns false (nothing moved) when two merged positions 0..topm tie, or when
// the prefix is out of order, as the network leaves it where distances are NaN: two
// entries would take one place, and another keep whatever the staging held.
template <bool kSolo, int E>
__device__ __noinline__ bool beam_merge(Beam bm, uint32_t topm, uint32_t m, int lane) {
  uint64_t key[E];
#pragma unroll
  for (int t = 0; t < E; ++t) {
    const uint32_t q = lane + 32 * t;
    key[t] = q < m ? (((uint64_t)__float_as_uint(bm.sm[q]) << 32) | bm.sid[q]) : ~0ull;
  }
  sort_keys<kSolo, E>(key, lane);
#pragma unroll
  for (int t = 0; t < E; ++t) {
    const uint32_t q = lane + 32 * t;
    if (q < m) bm.sb[q] = key_dis(key[t]);
  }
  __syncwarp();
  // merged rank: prefix i -> i + #(entering < A_i); entering q -> q + #(prefix <= B_q)
  bool bad = false;
  for (uint32_t i = lane; i < topm; i += 32) {
    const float a = bm.dis[i];
    bad |= i > 0 && !(bm.dis[i - 1] <= a);
    uint32_t lo = 0, hi = m;
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (bm.sb[mid] < a) lo = mid + 1;
      else hi = mid;
    }
    const uint32_t r = i + lo;
    if (r <= topm) {
      bm.sm[r] = a;
      bm.sid[r] = bm.id[i];
      bm.sex[r] = bm.ex[i];
    }
  }
#pragma unroll
  for (int t = 0; t < E; ++t) {
    const uint32_t q = lane + 32 * t;
    if (q < m) {
      const float v = key_dis(key[t]);
      uint32_t lo = 0, hi = topm;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (bm.dis[mid] <= v) lo = mid + 1;
        else hi = mid;
      }
      const uint32_t r = q + lo;
      if (r <= topm) {
        const uint32_t j = (uint32_t)(key[t] & 0xFFFFFFFFu);
        bm.sm[r] = v;
        bm.sid[r] = bm.id[topm + j];
        bm.sex[r] = bm.ex[topm + j];
      }
    }
  }
  __syncwarp();
  for (uint32_t p = lane + 1; p <= topm; p += 32) bad |= bm.sm[p] == bm.sm[p - 1];
  if (__any_sync(kFull, bad)) return false;
  for (uint32_t i = lane; i < topm; i += 32) {
    bm.dis[i] = bm.sm[i];
    bm.id[i] = bm.sid[i];
    bm.ex[i] = bm.sex[i];
  }
  __syncwarp();
  return true;
}

// After an expansion: [0, topm) holds the previous sorted prefix, [topm, W)
// the K new entries, of which the `nfresh` at slots fresh[0, nfresh) were
// scored and the rest are beam members at INF_DIS. The reference sorts all W
// with its network; only [0, topm) and the set of the W ids survive into the
// next expansion (the rest is overwritten), and with strictly increasing
// distances over merged positions 0..topm that part is the same for every
// correct sort. With a full prefix only scored entries no farther than its
// last one can reach positions 0..topm, so just those are sorted and merged
// by rank; a tie there, or a prefix that is not full, runs the network.
template <bool kSolo>
__device__ __noinline__ void beam_update(Beam bm, uint32_t topm, uint32_t K, const uint32_t* fresh,
                            uint32_t nfresh, int lane) {
  const uint32_t W = topm + K;
  beam_rehash(bm, W, lane);  // the set of all W ids, before anything moves
  const float worst = bm.dis[topm - 1];
  if (topm > 128 || !(worst < kInfDis)) {
    beam_network(bm, 0, W, lane);
    return;
  }
  const unsigned below = (1u << lane) - 1u;
  uint32_t m = 0;
  for (uint32_t base = 0; base < nfresh; base += 32) {
    const uint32_t r = base + lane;
    bool enter = false;
    float d = 0.0f;
    uint32_t j = 0;
    if (r < nfresh) {
      j = fresh[r];
      d = bm.dis[topm + j];
      enter = d <= worst;
    }
    const unsigned mk = __ballot_sync(kFull, enter);
    if (enter) {
      const uint32_t q = m + __popc(mk & below);
      bm.sm[q] = d;
      bm.sid[q] = j;
    }
    m += __popc(mk);
  }
  if (m == 0) return;  // every scored entry lies beyond the prefix: nothing moves
  __syncwarp();
  bool ok;
  if (m <= 32) ok = beam_merge<kSolo, 1>(bm, topm, m, lane);
  else if (m <= 64) ok = beam_merge<kSolo, 2>(bm, topm, m, lane);
  else ok = beam_merge<kSolo, 4>(bm, topm, m, lane);
  if (!ok) beam_network(bm, 0, W, lane);
}

// kSolo: as sort_keys'; kWide: as warp_rows32's, without a meaning for kSolo.
template <bool kSolo, bool kWide>
__device__ uint32_t warp_beam(const uint32_t* __restrict__ G, const __half* __restrict__ data,
                              uint32_t dim, uint32_t K, const __half* query, uint32_t start,
                              uint32_t topm, uint32_t iters, Beam bm, uint32_t* ring_id,
                              float* ring_dis, uint32_t* ring_count, int lane) {
  const uint32_t W = topm + K;
  for (uint32_t t = lane; t < W; t += 32) {
    bm.id[t] = kInv;
    bm.dis[t] = kInfDis;
    bm.ex[t] = 1;
  }
  __syncwarp();
  const uint32_t own = kSolo ? lane : rows32_of(lane);
  uint32_t* fresh_at = reinterpret_cast<uint32_t*>(bm.sb);  // K <= 128 slots
  uint32_t curr = 0, to_explore = start;
  // Round 0 scores the start node's whole row (the seeds), the later ones the
  // neighbours of an explored node that are not in the beam.
  for (uint32_t it = 0; it <= iters; ++it) {
    if (it > 0) {
      // First unexplored of the top TOPM; when none is left the reference keeps
      // the previous node (its `j == TOPM` test never fires, :1270).
      for (uint32_t base = 0; base < topm; base += 32) {
        const uint32_t j = base + lane;
        const unsigned m = __ballot_sync(kFull, j < topm && !bm.ex[j]);
        if (m) {
          const uint32_t f = base + __ffs(m) - 1;
          to_explore = bm.id[f];
          __syncwarp();
          if (lane == 0) bm.ex[f] = 1;
          break;
        }
      }
      __syncwarp();
      if (to_explore == kInv) break;
    }
    // Members of the beam keep INF_DIS; the others are listed in ascending
    // neighbour order (which fixes their ring slots) and scored 32 at a time.
    uint32_t nfresh = 0;
    for (uint32_t base = 0; base < K; base += 32) {
      const uint32_t j = base + lane;
      bool fresh = false;
      uint32_t a = kInv;
      if (j < K) {
        a = __ldg(G + (size_t)to_explore * K + j);
        fresh = it == 0 || !beam_has(bm, a);
        bm.id[topm + j] = a;
        bm.ex[topm + j] = 0;
        bm.dis[topm + j] = kInfDis;
      }
      const unsigned m = __ballot_sync(kFull, fresh);
      if (fresh) {
        const uint32_t r = nfresh + __popc(m & ((1u << lane) - 1u));
        fresh_at[r] = j;
        bm.sid[r] = a;
      }
      nfresh += __popc(m);
    }
    __syncwarp();
    for (uint32_t base = 0; base < nfresh; base += 32) {
      const uint32_t r = base + own;
      float d = 0.0f;
      if constexpr (!kSolo)
        d = warp_rows32<kWide>(query, data, dim, bm.sid + base, min(32u, nfresh - base));
      else if (r < nfresh)
        d = row_dist(query, data + (size_t)bm.sid[r] * dim, dim);
      if (r < nfresh) {
        bm.dis[topm + fresh_at[r]] = d;
        if (ring_id) {
          uint32_t p = curr + r;
          while (p >= kSelectCand) p -= kSelectCand;
          ring_id[p] = bm.sid[r];
          ring_dis[p] = d;
        }
      }
    }
    curr += nfresh;
    __syncwarp();
    if (it > 0) {
      beam_update<kSolo>(bm, topm, K, fresh_at, nfresh, lane);
      continue;
    }
    // Seeds: the network's order is observable on the first min(TOPM, K)
    // positions, copied into the prefix; a tie there runs the network.
    const uint32_t keep = min(topm, K);
    bool seeded = false;
    if (K <= 128) {
      uint64_t key[4];
      sorted_keys<kSolo>(bm, topm, K, key, lane);
      bool tie = false;
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const uint32_t p = lane + 32 * t;
        uint32_t prev = __shfl_up_sync(kFull, (uint32_t)(key[t] >> 32), 1);
        if (t > 0) {
          const uint32_t tail = __shfl_sync(kFull, (uint32_t)(key[t - 1] >> 32), 31);
          if (lane == 0) prev = tail;
        }
        if (p >= 1 && p <= keep && p < K && (uint32_t)(key[t] >> 32) == prev) tie = true;
      }
      if (!__any_sync(kFull, tie)) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const uint32_t p = lane + 32 * t;
          if (p < keep) {
            const uint32_t j = (uint32_t)(key[t] & 0xFFFFFFFFu);
            bm.id[p] = bm.id[topm + j];
            bm.dis[p] = key_dis(key[t]);
            bm.ex[p] = 0;
          }
        }
        for (uint32_t i = K + lane; i < topm; i += 32) {  // TOPM > K: empty slots
          bm.id[i] = kInv;
          bm.dis[i] = kInfDis;
          bm.ex[i] = 1;
        }
        seeded = true;
      }
    }
    if (!seeded) {
      beam_network(bm, topm, K, lane);
      for (uint32_t i = lane; i < topm; i += 32) {
        if (topm + i < W) {
          bm.id[i] = bm.id[topm + i];
          bm.dis[i] = bm.dis[topm + i];
          bm.ex[i] = bm.ex[topm + i];
        } else {  // slots past the K seeds start empty (TOPM > K)
          bm.id[i] = kInv;
          bm.dis[i] = kInfDis;
          bm.ex[i] = 1;
        }
      }
    }
    __syncwarp();
    beam_rehash(bm, W, lane);
    to_explore = kInv;
  }
  if (ring_count) *ring_count = curr;
  if constexpr (kSolo) {
    // The beam's first node. With TOPM > K the prefix has empty places, and they come
    // first where every distance lies beyond their kInfDis.
    for (uint32_t base = 0; base < topm; base += 32) {
      const uint32_t j = base + lane;
      const unsigned m = __ballot_sync(kFull, j < topm && bm.id[j] != kInv);
      if (m) return bm.id[base + __ffs(m) - 1];
    }
  }
  return start;
}

// Sort by distance with the reference network, then mark adjacent repeats
// using the ids as they were before marking (:1345-1348).
__device__ __noinline__ void warp_sort_mark(uint32_t* cand, float* dis, uint32_t len, int lane) {
  warp_network(len, lane, [&](uint32_t u, uint32_t d) { return dis[u] > dis[d]; },
               [&](uint32_t u, uint32_t d) {
                 swap_(dis[u], dis[d]);
                 swap_(cand[u], cand[d]);
               });
  // Marks decided from the unmarked ids: chunks from the last to the first,
  // so a chunk's comparisons read only its own entries and the last entry of
  // the chunk before it, none of them marked yet.
  const uint32_t chunks = (len + 31) / 32;
  for (uint32_t c = chunks; c-- > 0;) {
    const uint32_t i = c * 32 + lane;
    const bool rep = i >= 1 && i < len && cand[i] == cand[i - 1];
    __syncwarp();
    if (rep) cand[i] = kInv;
  }
  __syncwarp();
}

// The entries of 32 (one per lane, kInv: none) that the filter takes, of a list whose
// first m were taken before: all but the node itself, which is skipped only until
// another entry has been taken (:1399-1460). Behind rows equal to its own it is a
// candidate like any other.
__device__ __forceinline__ unsigned taken(uint32_t c, uint32_t bid, uint32_t m) {
  const unsigned any = __ballot_sync(kFull, c != kInv);
  const unsigned other = __ballot_sync(kFull, c != kInv && c != bid);
  return m ? any : any & ~((other & (0u - other)) - 1u);
}

// The length of a compacted list, with this bit where the list's last entry is left.
constexpr uint32_t kTailBit = 0x80000000u;

// Removes the marked entries and the node itself where it is skipped (taken) from a
// sorted, marked list, in place. Returns the entries left and the tail bit.
__device__ __noinline__ uint32_t warp_compact(uint32_t* cand, float* dis, uint32_t len,
                                              uint32_t bid, int lane) {
  const unsigned below = (1u << lane) - 1u;
  uint32_t m = 0;
  unsigned ok = 0;
  for (uint32_t base = 0; base < len; base += 32) {
    const uint32_t i = base + lane;
    const uint32_t c = i < len ? cand[i] : kInv;
    const float d = i < len ? dis[i] : 0.0f;
    ok = taken(c, bid, m);
    __syncwarp();  // the chunk is read before an earlier or equal place is written
    if ((ok >> lane) & 1u) {
      const uint32_t p = m + __popc(ok & below);
      cand[p] = c;
      dis[p] = d;
    }
    m += __popc(ok);
  }
  __syncwarp();
  return len > 0 && ((ok >> ((len - 1) & 31u)) & 1u) ? m | kTailBit : m;
}

// Words that mark the places of the kNN row's entries in the merged list.
constexpr uint32_t kMarkWords = (kSelectCand + 128 + 31) / 32;

// warp_sort_mark and warp_compact of a candidate list (K kNN entries, then
// kSelectCand collected ones, in shared memory) where the order of equal
// distances cannot be observed, written to out_ids / out_dis: the collected
// entries are sorted in registers and merged with the row, which is sorted
// already. Returns as warp_compact does, or kInv where the network has to decide: a
// row out of order, a distance that is negative or NaN, or equal distances of
// different ids (entries with the same id and distance are the same in any
// order). The collected part of the list is overwritten.
//
// Bound by instruction issue: about 3.5K instructions per warp against 7.6K of
// the network, its marks and the compaction. The keys lie 16 to a lane, so that 30
// of the 45 passes exchange within a lane; every merge starts mirrored, which
// leaves one direction of comparison.
// Collect at 500K x 96, K = 64: 29.1 ms with the network, 28.0 ms with this.
__device__ __noinline__ uint32_t warp_list(uint32_t* cand, float* cdis, uint32_t* mark,
                                           uint32_t K, uint32_t bid,
                                           uint32_t* __restrict__ out_ids,
                                           float* __restrict__ out_dis, int lane) {
  constexpr uint32_t kLast = 0x7F800000u;  // bits of +inf
  constexpr int E = 16;
  static_assert(kSelectCand == 30 * E, "the pads fill the last two lanes");
  uint32_t key[E], id[E];
  bool bad = false;
#pragma unroll
  for (int t = 0; t < E - 1; ++t) {
    const uint32_t e = K + 32 * t + lane;
    key[t] = __float_as_uint(cdis[e]);
    id[t] = cand[e];
    bad |= key[t] > kLast;
  }
  key[E - 1] = kInv;
  id[E - 1] = kInv;
  for (uint32_t i = lane; i < K; i += 32) {
    const uint32_t k = __float_as_uint(cdis[i]);
    bad |= k > kLast;
    if (i > 0) {
      const uint32_t p = __float_as_uint(cdis[i - 1]);
      bad |= k < p || (k == p && cand[i] != cand[i - 1]);
    }
  }
  if (__any_sync(kFull, bad)) return kInv;
  // ascending, position 16 * lane + t
  auto in_lane = [&](int a, int b) {
    const bool s = key[a] > key[b];
    const uint32_t ka = key[a], kb = key[b], ia = id[a], ib = id[b];
    key[a] = s ? kb : ka;
    key[b] = s ? ka : kb;
    id[a] = s ? ib : ia;
    id[b] = s ? ia : ib;
  };
  auto take = [&](int a, uint32_t ok, uint32_t oi, bool upper) {
    const bool s = upper ? ok > key[a] : ok < key[a];
    key[a] = s ? ok : key[a];
    id[a] = s ? oi : id[a];
  };
#pragma unroll
  for (int size = 2; size <= E; size <<= 1) {
#pragma unroll
    for (int t = 0; t < E; ++t)
      if (t < (t ^ (size - 1))) in_lane(t, t ^ (size - 1));
#pragma unroll
    for (int st = size / 4; st > 0; st >>= 1)
#pragma unroll
      for (int t = 0; t < E; ++t)
        if (!(t & st)) in_lane(t, t | st);
  }
#pragma unroll 1
  for (int lanes = 2; lanes <= 32; lanes <<= 1) {
    const bool up = lane & (lanes >> 1);
#pragma unroll
    for (int t = 0; t < E / 2; ++t) {
      const int q = E - 1 - t;
      const uint32_t k0 = __shfl_xor_sync(kFull, key[q], lanes - 1);
      const uint32_t i0 = __shfl_xor_sync(kFull, id[q], lanes - 1);
      const uint32_t k1 = __shfl_xor_sync(kFull, key[t], lanes - 1);
      const uint32_t i1 = __shfl_xor_sync(kFull, id[t], lanes - 1);
      take(t, k0, i0, up);
      take(q, k1, i1, up);
    }
#pragma unroll 1
    for (int st = lanes >> 2; st > 0; st >>= 1) {
      const bool upper = lane & st;
#pragma unroll
      for (int t = 0; t < E; ++t) {
        const uint32_t ok = __shfl_xor_sync(kFull, key[t], st);
        const uint32_t oi = __shfl_xor_sync(kFull, id[t], st);
        take(t, ok, oi, upper);
      }
    }
#pragma unroll
    for (int st = E / 2; st > 0; st >>= 1)
#pragma unroll
      for (int t = 0; t < E; ++t)
        if (!(t & st)) in_lane(t, t | st);
  }
#pragma unroll
  for (int t = 0; t + 1 < E; ++t) bad |= key[t] == key[t + 1] && id[t] != id[t + 1];
  {
    const uint32_t nk = __shfl_down_sync(kFull, key[0], 1), ni = __shfl_down_sync(kFull, id[0], 1);
    bad |= lane < 31 && key[E - 1] == nk && id[E - 1] != ni;
  }
  if (__any_sync(kFull, bad)) return kInv;
  // back to the list, the 16 places of a lane permuted against bank conflicts
  auto place = [](uint32_t p) { return (p & ~15u) | ((p ^ (p >> 4)) & 15u); };
  if (lane < 30) {
#pragma unroll
    for (int t = 0; t < E; ++t) {
      const uint32_t e = K + place(lane * E + t);
      cdis[e] = __uint_as_float(key[t]);
      cand[e] = id[t];
    }
  }
  if (lane < (int)kMarkWords) mark[lane] = 0;
  __syncwarp();
  for (uint32_t i = lane; i < K; i += 32) {
    const uint32_t k = __float_as_uint(cdis[i]);
    uint32_t lo = 0, hi = kSelectCand;  // collected entries before row entry i
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__float_as_uint(cdis[K + place(mid)]) < k) lo = mid + 1;
      else hi = mid;
    }
    if (lo < kSelectCand) {
      const uint32_t e = K + place(lo);
      bad |= __float_as_uint(cdis[e]) == k && cand[e] != cand[i];
    }
    const uint32_t f = i + lo;
    atomicOr(&mark[f >> 5], 1u << (f & 31u));
  }
  if (__any_sync(kFull, bad)) return kInv;
  __syncwarp();
  const unsigned below = (1u << lane) - 1u;
  const uint32_t total = K + kSelectCand;
  uint32_t rows = 0, m = 0, carry = kInv;
  unsigned ok = 0;
  for (uint32_t base = 0; base < total; base += 32) {
    const uint32_t f = base + lane, w = mark[base >> 5], r = rows + __popc(w & below);
    const uint32_t e = (w >> lane) & 1u ? r : K + place(f - r);
    uint32_t c = kInv;
    float d = 0.0f;
    if (f < total) {
      c = cand[e];
      d = cdis[e];
    }
    uint32_t prev = __shfl_up_sync(kFull, c, 1);
    if (lane == 0) prev = carry;
    carry = __shfl_sync(kFull, c, 31);
    if (f >= 1 && c == prev) c = kInv;
    ok = taken(c, bid, m);
    if ((ok >> lane) & 1u) {
      const uint32_t p = m + __popc(ok & below);
      out_ids[p] = c;
      out_dis[p] = d;
    }
    m += __popc(ok);
    rows += __popc(w);
  }
  return (ok >> ((total - 1) & 31u)) & 1u ? m | kTailBit : m;
}

// Kept neighbours of one node, and the rows of a tile that outlived the kept
// ones before it: shared memory of one warp.
struct Kept {
  uint32_t* id;
  float *dis, *norm;        // fd each
  uint32_t* tid;
  float *tdis, *tnorm;      // 32 each
  float* tile;              // screen_tile's
};
__host__ __device__ inline size_t kept_bytes(uint32_t fd) {
  return (size_t)fd * 12 + 32 * 12 + kScreenFloats * 4;
}
__device__ inline Kept kept_carve(unsigned char* p, uint32_t fd) {
  Kept k;
  k.id = reinterpret_cast<uint32_t*>(p);
  k.dis = reinterpret_cast<float*>(k.id + fd);
  k.norm = k.dis + fd;
  k.tid = reinterpret_cast<uint32_t*>(k.norm + fd);
  k.tdis = reinterpret_cast<float*>(k.tid + 32);
  k.tnorm = k.tdis + 32;
  k.tile = k.tnorm + 32;
  return k;
}

// The exact test of candidate row c (distance dc) against kept row q (distance
// dq), by the whole warp. Out of line: it is rarely taken.
static __device__ __noinline__ bool exact_test(const __half* __restrict__ data, uint32_t dim,
                                               ScreenRule rule, uint32_t c, float dc, uint32_t q,
                                               float dq) {
  const float res = warp_dist(data + (size_t)q * dim, data + (size_t)c * dim, dim,
                              (int)(threadIdx.x & 31u));
  return pruned_by(rule.metric, res, dc, dq, rule.thre);
}

// Filter stage over a compacted list (warp_compact) by one warp. Returns the
// number of ids the reference stores: one less than its selection steps (:1462,
// :1623). *tested: the candidates taken before the degree was full.
//
// The list is taken 32 candidates at a time. A tile is first tested against the
// kept neighbours (16 per screen, stopping when no candidate is left), then its
// survivors against one another, in list order: each candidate is dropped by a
// rule that fires against a neighbour kept before it, as in the sequential
// filter. A repeat of a kept neighbour is dropped too (:1423-1427).
//
// Bound by the gathers of the candidates' rows and by instruction issue. Each row
// is read once per screen; a test costs a fraction of an mma instead of a
// 2d-byte row and its sum.
__device__ __forceinline__ uint32_t warp_filter(const uint32_t* cand, const float* cdis,
                                                uint32_t len, bool tail, uint32_t fd, int metric,
                                                float thre, const __half* __restrict__ data,
                                                const float* __restrict__ norms, uint32_t dim,
                                                const Kept& k, int lane,
                                                uint32_t* tested = nullptr) {
  const ScreenRule rule{metric, thre, screen_eps(dim)};
  const unsigned below = (1u << lane) - 1u;
  uint32_t nsel = 0, last = 0, base = 0;
  for (; base < len && nsel < fd; base += 32) {
    const uint32_t i = base + lane;
    uint32_t c = kInv;
    float dc = 0.0f, nc = 0.0f;
    if (i < len) {
      c = cand[i];
      dc = cdis[i];
      nc = __ldg(norms + c);
    }
    // against the neighbours kept in earlier tiles
    for (uint32_t k0 = 0; k0 < nsel; k0 += kScreenCols) {
      const uint2 scr = screen_rows<true>(data, dim, rule, c, nc, dc, k.id + k0, k.norm + k0,
                                          k.dis + k0, min(kScreenCols, nsel - k0), k.tile);
      uint32_t amb = scr.x ? 0u : scr.y;
      bool drop = scr.x != 0;
      for (unsigned left = __ballot_sync(kFull, amb != 0); left;
           left = __ballot_sync(kFull, amb != 0)) {
        const int o = __ffs(left) - 1;
        const uint32_t q = k0 + __ffs(__shfl_sync(kFull, amb, o)) - 1;
        const bool f = exact_test(data, dim, rule, __shfl_sync(kFull, c, o),
                                  __shfl_sync(kFull, dc, o), k.id[q], k.dis[q]);
        if (lane == o) {
          drop = f;
          amb = f ? 0u : amb & (amb - 1u);
        }
      }
      if (drop) c = kInv;
      if (!__any_sync(kFull, c != kInv)) break;
    }
    const unsigned alive = __ballot_sync(kFull, c != kInv);
    const uint32_t ns = __popc(alive);
    if (ns == 0) continue;
    __syncwarp();
    if (c != kInv) {
      const uint32_t p = __popc(alive & below);
      k.tid[p] = c;
      k.tdis[p] = dc;
      k.tnorm[p] = nc;
    }
    __syncwarp();
    // against the survivors before it in this tile
    uint32_t fire = 0, amb = 0;
    for (uint32_t q0 = 0; q0 + 1 < ns; q0 += kScreenCols) {
      const bool in = (uint32_t)lane < ns;
      const uint32_t nb = min(kScreenCols, ns - q0);
      const uint2 scr = screen_rows<false>(data, dim, rule, in ? k.tid[lane] : kInv,
                                           in ? k.tnorm[lane] : 0.0f, in ? k.tdis[lane] : 0.0f,
                                           k.tid + q0, k.tnorm + q0, k.tdis + q0, nb, k.tile);
      fire |= scr.x << q0;
      amb |= scr.y << q0;
      if (in)
        for (uint32_t q = q0; q < min(q0 + nb, (uint32_t)lane); ++q)
          if (k.tid[q] == k.tid[lane]) fire |= 1u << q;
    }
    uint32_t kept = 0;  // survivors kept so far
    for (uint32_t r = 0; r < ns && nsel < fd; ++r) {
      if (__shfl_sync(kFull, fire, (int)r) & kept) continue;
      bool out = false;
      for (uint32_t m = __shfl_sync(kFull, amb, (int)r) & kept; m && !out; m &= m - 1u) {
        const uint32_t q = __ffs(m) - 1;
        out = exact_test(data, dim, rule, k.tid[r], k.tdis[r], k.tid[q], k.tdis[q]);
      }
      if (out) continue;
      kept |= 1u << r;
      if (lane == 0) {
        k.id[nsel] = k.tid[r];
        k.dis[nsel] = k.tdis[r];
        k.norm[nsel] = k.tnorm[r];
      }
      ++nsel;
      // the r-th survivor's place in the list
      uint32_t a = alive;
      for (uint32_t x = 0; x < r; ++x) a &= a - 1u;
      last = base + __ffs(a) - 1;
    }
    __syncwarp();
  }
  __syncwarp();
  if (tested) *tested = min(base, len);
  if (nsel == fd) return fd - 1;
  if (nsel >= 2 && last == len - 1 && tail) return nsel - 1;
  return nsel;
}

// Per-warp shared layout of the select kernels: the beam (path collect) and
// the candidate list share one region, since the list is filled only after
// the beam has finished (its ring of scored nodes lives in global memory).
struct SelLayout {
  uint32_t topm, K;  // topm 0: no beam
  size_t tail;  // bytes behind the list (kept_bytes where the kernel also filters)
  __host__ __device__ uint32_t L() const { return kSelectCand + K; }
  __host__ __device__ size_t bytes() const {
    const size_t list = (size_t)L() * 8 + kMarkWords * 4 + tail;
    const size_t beam = topm ? beam_bytes(topm, K) : 0;
    return ((beam > list ? beam : list) + 15) & ~(size_t)15;
  }
};

// ---------------------------------------------------------------------------
// Processing order of the select kernels. A node's select reads only the kNN
// snapshot and writes only its own rows, so the order in which nodes are
// taken changes no result. Taking together nodes that share kNN
// neighbourhoods keeps the rows the warps in flight gather resident in L2
// (at d = 960 the base is 15x larger than L2). Labels: each node takes the
// smallest label among itself and its first kLabelHops neighbours, in place
// (labels only decrease, so concurrent updates are harmless), for
// kLabelRounds rounds; nodes of one cluster converge to a common label. The
// order is the nodes sorted by label.
constexpr uint32_t kLabelHops = 4, kLabelRounds = 16;

__global__ void k_label_init(uint32_t* __restrict__ lab, uint32_t* __restrict__ ids, uint32_t n) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    lab[u] = u;
    ids[u] = u;
  }
}

__global__ void k_label_min(const uint32_t* __restrict__ G, uint32_t K, uint32_t hops,
                            uint32_t* lab, uint32_t n) {
  for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
    uint32_t m = lab[u];
    for (uint32_t j = 0; j < hops; ++j) m = min(m, lab[__ldg(G + (size_t)u * K + j)]);
    if (m < lab[u]) lab[u] = m;
  }
}

__global__ void k_validate(const uint32_t* __restrict__ g, size_t cnt, uint32_t n,
                           uint32_t* bad) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < cnt;
       i += (size_t)gridDim.x * blockDim.x)
    if (g[i] >= n) atomicExch(bad, 1u);
}

// cal_ep_gpu (:1889-2058): one warp, 30 expansions from node 0 toward the centre.
__global__ void k_cal_ep(const uint32_t* __restrict__ G, const __half* __restrict__ data,
                         const __half* __restrict__ center, uint32_t dim, uint32_t K,
                         uint32_t topm, uint32_t* ep) {
  extern __shared__ __align__(16) unsigned char smem[];
  Beam bm = beam_carve(smem, topm, K);
  const int lane = threadIdx.x & 31;
  if (threadIdx.x >= 32) return;
  const uint32_t best = warp_beam<true, true>(G, data, dim, K, center, 0, topm, 30, bm, nullptr,
                                              nullptr, nullptr, lane);
  if (lane == 0) *ep = best;
}

// Node handed to this warp: one shared counter, taken a node at a time, keeps
// the SMs busy to the end whatever the per-node search length.
__device__ __forceinline__ uint32_t next_node(uint32_t* ctr, int lane) {
  uint32_t b = 0;
  if (lane == 0) b = atomicAdd(ctr, 1u);
  return __shfl_sync(kFull, b, 0);
}
// The node at position i of the processing order (identity without one).
__device__ __forceinline__ uint32_t node_at(const uint32_t* __restrict__ order, uint32_t i) {
  return order ? __ldg(order + i) : i;
}

// The collect half of select_path (:1498-1517) and select_2hop (:1520-1534):
// node b's candidates (its kNN row and the collected nodes), unsorted, in
// cand / cdis. Returns the rows scored. rid / rds: this warp's ring of kSelectCand
// scored nodes (path).
template <bool kPath, bool kWide>
__device__ __forceinline__ uint32_t collect_node(
    const uint32_t* __restrict__ G, const float* __restrict__ nd, const __half* __restrict__ data,
    uint32_t dim, uint32_t K, uint32_t ep, uint32_t topm, uint32_t b, Beam bm, uint32_t* rid,
    float* rds, uint32_t* cand, float* cdis, int lane) {
  const __half* q = data + (size_t)b * dim;
  uint32_t scored = kSelectCand;  // 2-hop: the 480 collected
  if (kPath) {
    uint32_t curr = 0;
    warp_beam<false, kWide>(G, data, dim, K, q, ep, topm, 10, bm, rid, rds, &curr, lane);
    scored = curr;
    __syncwarp();  // the ring (global) and the beam's region are done
    for (uint32_t i = lane; i < kSelectCand; i += 32) {
      const bool in = i < curr;
      cand[K + i] = in ? rid[i] : kInv;
      cdis[K + i] = in ? rds[i] : kInfDis;
    }
  } else {
    for (uint32_t i = lane; i < kSelectCand; i += 32)
      cand[K + i] = __ldg(G + (size_t)__ldg(G + (size_t)b * K + i / K) * K + i % K);
    __syncwarp();
    // The two-hop rows are scored four at a time by the whole warp: each
    // lane reads its 8-byte chunks of four rows at once (coalesced across
    // the warp) and the four shuffle trees interleave. Same lane order as
    // the thread-serial distance, so the same values.
    auto score = [&](auto&& dist4) {
      for (uint32_t i = 0; i < kSelectCand; i += 4) {
        const uint32_t ids[4] = {cand[K + i], cand[K + i + 1], cand[K + i + 2], cand[K + i + 3]};
        float o[4];
        dist4(ids, o);
        if (lane < 4)
          cdis[K + i + lane] = lane == 0 ? o[0] : lane == 1 ? o[1] : lane == 2 ? o[2] : o[3];
      }
    };
    if (dim == 960) {
      score([&](const uint32_t* ids, float* o) { warp_dist4<960>(q, data, dim, ids, o, lane); });
    } else {
      score([&](const uint32_t* ids, float* o) { warp_dist4(q, data, dim, ids, o, lane); });
    }
  }
  for (uint32_t i = lane; i < K; i += 32) {
    cand[i] = __ldg(G + (size_t)b * K + i);
    cdis[i] = nd[(size_t)b * K + i];
  }
  __syncwarp();
  return scored;
}

// The filter half: select_path and select_2hop always use distance_filter and
// angle_filter respectively. Results go to scratch rows, and the selected
// distances to the node's own nd row, which no other node reads. Returns the
// candidates tested.
__device__ __forceinline__ uint32_t filter_node(const uint32_t* cand, const float* cdis, uint32_t len,
                                            bool tail, uint32_t fd, int metric, float thre,
                                            const __half* __restrict__ data,
                                            const float* __restrict__ norms, uint32_t dim,
                                            const Kept& k, uint32_t b, uint32_t K,
                                            float* __restrict__ nd, uint32_t* __restrict__ P_ids,
                                            float* __restrict__ P_dis,
                                            uint32_t* __restrict__ P_cnt, int lane) {
  uint32_t tested = 0;
  const uint32_t stored =
      warp_filter(cand, cdis, len, tail, fd, metric, thre, data, norms, dim, k, lane, &tested);
  for (uint32_t i = lane; i < stored; i += 32) {
    P_ids[(size_t)b * fd + i] = k.id[i];
    P_dis[(size_t)b * fd + i] = k.dis[i];
    nd[(size_t)b * K + i] = k.dis[i];
  }
  if (lane == 0) P_cnt[b] = stored;
  __syncwarp();
  return tested;
}

// The list as it was collected, sorted by the network: where warp_list cannot decide.
// Out of line, so that it takes no registers of the collect, which spills at its
// seven blocks per SM (1M x 128: 82.3 ms inlined, 79.5 ms; six blocks 81.0 ms).
template <bool kPath>
static __device__ __noinline__ uint32_t network_list(const uint32_t* __restrict__ G, uint32_t K,
                                                     uint32_t scored, const uint32_t* rid,
                                                     const float* rds, uint32_t* cand, float* cdis,
                                                     uint32_t b, uint32_t* __restrict__ out_ids,
                                                     float* out_dis, int lane) {
  for (uint32_t j = lane; j < kSelectCand; j += 32) {
    if (kPath) {
      cand[K + j] = j < scored ? rid[j] : kInv;
      cdis[K + j] = j < scored ? rds[j] : kInfDis;
    } else {
      cand[K + j] = __ldg(G + (size_t)cand[j / K] * K + j % K);
      cdis[K + j] = out_dis[j];
    }
  }
  __syncwarp();
  warp_sort_mark(cand, cdis, kSelectCand + K, lane);
  const uint32_t got = warp_compact(cand, cdis, kSelectCand + K, b, lane);
  for (uint32_t j = lane; j < (got & ~kTailBit); j += 32) {
    out_ids[j] = cand[j];
    out_dis[j] = cdis[j];
  }
  return got;
}

// Candidate lists of the nodes at positions [first, first + cnt) of the order,
// L entries apart; L_cnt holds a list's length and its tail bit.
// ring_ids / ring_dis: per-warp rings of kSelectCand scored nodes (path), by the
// warp's global number.
//
// Collect and filter are two kernels with the list between them in memory (about
// 4.6 KB of it per node at K = 96, 1.4 ms of a 1M prune): the beam waits on
// gathers and wants warps, the filter's tiles want registers, and each half's
// code fits the instruction cache.
template <bool kPath, bool kWide>
__global__ void __launch_bounds__(kWarps * 32, 7)
    k_collect(const uint32_t* __restrict__ G, const float* __restrict__ nd,
              const __half* __restrict__ data, uint32_t first, uint32_t cnt, uint32_t dim,
              uint32_t K, const uint32_t* __restrict__ ep_dev, uint32_t* __restrict__ ctr,
              uint32_t topm, uint32_t* __restrict__ L_ids, float* __restrict__ L_dis,
              uint32_t* __restrict__ L_cnt, unsigned long long* __restrict__ work,
              uint32_t* __restrict__ ring_ids, float* __restrict__ ring_dis,
              const uint32_t* __restrict__ order) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SelLayout lay{kPath ? topm : 0u, K, 0};
  unsigned char* mine = smem + (size_t)warp * lay.bytes();
  uint32_t* cand = reinterpret_cast<uint32_t*>(mine);
  float* cdis = reinterpret_cast<float*>(cand + lay.L());
  uint32_t* mark = reinterpret_cast<uint32_t*>(cdis + lay.L());
  Beam bm = beam_carve(mine, lay.topm, K);  // same region as the list, used before it
  const size_t gw = (size_t)blockIdx.x * kWarps + warp;
  uint32_t* rid = kPath ? ring_ids + gw * kSelectCand : nullptr;
  float* rds = kPath ? ring_dis + gw * kSelectCand : nullptr;
  const uint32_t ep = kPath ? *ep_dev : 0u;
  unsigned long long rows = 0;
  for (uint32_t i = next_node(ctr, lane); i < cnt; i = next_node(ctr, lane)) {
    const uint32_t b = node_at(order, first + i);
    const uint32_t scored =
        collect_node<kPath, kWide>(G, nd, data, dim, K, ep, topm, b, bm, rid, rds, cand, cdis, lane);
    uint32_t* out_ids = L_ids + (size_t)i * lay.L();
    float* out_dis = L_dis + (size_t)i * lay.L();
    if (!kPath) {
      // the collected entries' distances, should the network need them back
      for (uint32_t j = lane; j < kSelectCand; j += 32) out_dis[j] = cdis[K + j];
      __syncwarp();
    }
    uint32_t got = warp_list(cand, cdis, mark, K, b, out_ids, out_dis, lane);
    if (got == kInv)
      got = network_list<kPath>(G, K, scored, rid, rds, cand, cdis, b, out_ids, out_dis, lane);
    rows += scored;
    if (lane == 0) L_cnt[i] = got;
    __syncwarp();
  }
  if (work && lane == 0) atomicAdd(work, rows);
}

__global__ void __launch_bounds__(kWarps * 32, 4)
    k_filter(const uint32_t* __restrict__ L_ids, const float* __restrict__ L_dis,
             const uint32_t* __restrict__ L_cnt, uint32_t L, float* __restrict__ nd,
             const __half* __restrict__ data, const float* __restrict__ norms, uint32_t first,
             uint32_t cnt, uint32_t dim, uint32_t K, uint32_t* __restrict__ ctr, uint32_t fd,
             int metric, float thre, uint32_t* __restrict__ P_ids, float* __restrict__ P_dis,
             uint32_t* __restrict__ P_cnt, unsigned long long* __restrict__ work,
             const uint32_t* __restrict__ order) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const Kept k = kept_carve(smem + (size_t)warp * kept_bytes(fd), fd);
  uint32_t listed = 0, tested = 0;  // below 2^28 each, a batch's lists
  for (uint32_t i = next_node(ctr, lane); i < cnt; i = next_node(ctr, lane)) {
    const uint32_t b = node_at(order, first + i), lc = L_cnt[i];
    listed += lc & ~kTailBit;
    tested += filter_node(L_ids + (size_t)i * L, L_dis + (size_t)i * L, lc & ~kTailBit,
                          (lc & kTailBit) != 0, fd, metric, thre, data, norms, dim, k, b, K, nd,
                          P_ids, P_dis, P_cnt, lane);
  }
  if (lane == 0) {
    atomicAdd(work, (unsigned long long)listed);
    atomicAdd(work + 1, (unsigned long long)tested);
  }
}

// Both halves by the same warp, the list in shared memory: for the prune that
// may not allocate the lists.
template <bool kPath, bool kWide>
__global__ void __launch_bounds__(kWarps * 32, 4)
    k_select(const uint32_t* __restrict__ G, float* __restrict__ nd, const __half* __restrict__ data,
             const float* __restrict__ norms, uint32_t n, uint32_t dim, uint32_t K,
             const uint32_t* __restrict__ ep_dev, uint32_t* __restrict__ ctr, uint32_t topm,
             uint32_t fd, float thre, uint32_t* __restrict__ P_ids, float* __restrict__ P_dis,
             uint32_t* __restrict__ P_cnt, uint32_t* __restrict__ ring_ids,
             float* __restrict__ ring_dis) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const SelLayout lay{kPath ? topm : 0u, K, kept_bytes(fd)};
  unsigned char* mine = smem + (size_t)warp * lay.bytes();
  uint32_t* cand = reinterpret_cast<uint32_t*>(mine);
  float* cdis = reinterpret_cast<float*>(cand + lay.L());
  const Kept k = kept_carve(reinterpret_cast<unsigned char*>(cdis + lay.L()) + kMarkWords * 4, fd);
  Beam bm = beam_carve(mine, lay.topm, K);  // same region as the list, used before it
  const size_t gw = (size_t)blockIdx.x * kWarps + warp;
  uint32_t* rid = kPath ? ring_ids + gw * kSelectCand : nullptr;
  float* rds = kPath ? ring_dis + gw * kSelectCand : nullptr;
  const uint32_t ep = kPath ? *ep_dev : 0u;
  for (uint32_t b = next_node(ctr, lane); b < n; b = next_node(ctr, lane)) {
    collect_node<kPath, kWide>(G, nd, data, dim, K, ep, topm, b, bm, rid, rds, cand, cdis, lane);
    warp_sort_mark(cand, cdis, lay.L(), lane);
    const uint32_t len = warp_compact(cand, cdis, lay.L(), b, lane);
    filter_node(cand, cdis, len & ~kTailBit, (len & kTailBit) != 0, fd, kPath ? 0 : 1, thre, data,
                norms, dim, k, b, K, nd, P_ids, P_dis, P_cnt, lane);
  }
}

// Squared norms of the FP16 base for the screens, one warp per row.
__global__ void k_row_norms(const __half* __restrict__ data, uint32_t n, uint32_t dim,
                            float* __restrict__ norms) {
  const int lane = threadIdx.x & 31;
  for (uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n;
       r += (gridDim.x * blockDim.x) >> 5) {
    const uint2* row = reinterpret_cast<const uint2*>(data + (size_t)r * dim);
    float x = 0.0f, y = 0.0f;
    for (uint32_t j = lane; j < dim / 4; j += 32)
      chunk_acc(__ldg(row + j), make_uint2(0u, 0u), x, y);
    const float v = warp_tree(x, y);
    if (lane == 0) norms[r] = v;
  }
}

// Shared bytes per warp of k_filter_reverse.
__host__ __device__ inline size_t reverse_bytes(uint32_t fd, uint32_t K) {
  return ((size_t)(fd + K) * 8 + kept_bytes(fd) + 15) & ~(size_t)15;
}

// filter_reverse (:1537-1657) plus the in-place row writes of the select
// kernels (:1462-1464, :1477): the stored row is the kNN row overwritten by
// the select result, then by this stage's result.
__global__ void __launch_bounds__(kWarps * 32, 4)
    k_filter_reverse(uint32_t* __restrict__ graph, const float* __restrict__ nd,
                     const uint32_t* __restrict__ rg, const float* __restrict__ rd,
                     const uint32_t* __restrict__ rnum, const __half* __restrict__ data,
                     const float* __restrict__ norms, uint32_t n, uint32_t dim, uint32_t K,
                     uint32_t fd, int metric, float thre,
                     const uint32_t* __restrict__ P_ids, const uint32_t* __restrict__ P_cnt,
                     const uint32_t* __restrict__ order) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t cap = fd + K;  // cur_num <= fd - 1, rever_num <= K
  unsigned char* mine = smem + (size_t)warp * reverse_bytes(fd, K);
  uint32_t* cand = reinterpret_cast<uint32_t*>(mine);
  float* cdis = reinterpret_cast<float*>(cand + cap);
  const Kept k = kept_carve(reinterpret_cast<unsigned char*>(cdis + cap), fd);
  uint32_t* sel = k.id;
  for (uint32_t pos = blockIdx.x * kWarps + warp; pos < n; pos += gridDim.x * kWarps) {
    const uint32_t b = node_at(order, pos);
    const uint32_t cur_num = P_cnt[b];
    const uint32_t rn = min(K, rnum[b]);
    const uint32_t len = cur_num + rn;
    for (uint32_t i = lane; i < cur_num; i += 32) {
      cand[i] = P_ids[(size_t)b * fd + i];
      cdis[i] = nd[(size_t)b * K + i];
    }
    for (uint32_t i = lane; i < rn; i += 32) {
      cand[cur_num + i] = rg[(size_t)b * K + i];
      cdis[cur_num + i] = rd[(size_t)b * kReserve + i];
    }
    __syncwarp();
    uint32_t* row = graph + (size_t)b * K;
    uint32_t out_cnt;
    if (len > fd) {
      warp_sort_mark(cand, cdis, len, lane);
      const uint32_t left = warp_compact(cand, cdis, len, b, lane);
      out_cnt = warp_filter(cand, cdis, left & ~kTailBit, (left & kTailBit) != 0, fd, metric, thre,
                            data, norms, dim, k, lane);
    } else {
      // Union in ascending reverse-slot order (:1632-1647).
      for (uint32_t i = lane; i < cur_num; i += 32) sel[i] = cand[i];
      uint32_t dup = 0;
      for (uint32_t i = 0; i < rn; ++i) {
        const uint32_t r = cand[cur_num + i];
        bool found = false;
        for (uint32_t j0 = 0; j0 < cur_num; j0 += 32) {
          const uint32_t j = j0 + lane;
          if (__any_sync(kFull, j < cur_num && cand[j] == r)) {
            found = true;
            break;
          }
        }
        // A stride-K row holds at most K-1 ids; with FINAL_DEGREE == K the
        // reference would spill its last union id into the next row.
        if (!found && cur_num + dup + 1 < K) {
          if (lane == 0) sel[cur_num + dup] = r;
          ++dup;
        }
      }
      out_cnt = cur_num + dup;
    }
    __syncwarp();
    const uint32_t top = max(out_cnt, cur_num);
    for (uint32_t i = lane; i < top; i += 32)
      row[i + 1] = (i < out_cnt) ? sel[i] : P_ids[(size_t)b * fd + i];
    if (lane == 0) row[0] = out_cnt;
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Orders a node's ids by (detours << 8 | position) ranks with the reference's
// network and stores the first d.
__device__ __forceinline__ void rank_store(uint32_t* rank, const uint32_t* nei0, uint32_t K,
                                           uint32_t d, uint32_t b, uint32_t* __restrict__ hybrid,
                                           uint32_t* __restrict__ E_tgt,
                                           uint32_t* __restrict__ E_val, int lane) {
  warp_network(K, lane, [&](uint32_t u, uint32_t v) { return (rank[u] >> 8) > (rank[v] >> 8); },
               [&](uint32_t u, uint32_t v) { swap_(rank[u], rank[v]); });
  for (uint32_t i = lane; i < d; i += 32) {
    const uint32_t id = nei0[rank[i] & 0xFFu];
    E_tgt[(size_t)b * d + i] = id;
    E_val[(size_t)b * d + i] = rank[i] >> 8;
    hybrid[(size_t)b * K + i] = id;
  }
}

// Rank-based prunes. collect_1hop + filter_cagra (:1660-1710): detour[m]
// counts the kept-earlier neighbours a whose own list holds n_m, over the
// pairs the reference visits (a in {i, K-1-i : i < K/2}, m > a).
//
// Bound by instruction issue: one lookup per list entry. The node's own K ids go
// into one table and the ids of the K lists are looked up in it, with no barrier
// between lists, so several lists' loads are in flight (kCagraRows). The table is
// sparse (K <= 128 ids in 1,024 chains) so that an id which is not the node's
// ends at its empty head, and a warp rarely waits for a lane that walks on. A
// (list, position) pair counts once however often the list repeats the id, so a
// hit sets bit a of position m's mask and the counts are the masks' populations.
// Select at 1M x 128, K = 96: 19.6 ms, against 45.8 ms with a table of each list
// in turn looked up by the K positions, and 42.2 ms with the node's ids in a
// 256-slot probed table, where the longest of 32 probe runs set the pace.
constexpr uint32_t kCagraHeads = 1024;
constexpr uint32_t kCagraRows = 4;  // lists loaded ahead of their lookups

// Shared words per warp: chain heads, masks, next links, ids, ranks.
__host__ __device__ inline uint32_t cagra_words(uint32_t K) {
  return (kCagraHeads + 7 * K + 3) & ~3u;
}

__global__ void __launch_bounds__(kWarps * 32)
    k_select_cagra(const uint32_t* __restrict__ G, uint32_t n, uint32_t K, uint32_t d,
                   uint32_t* __restrict__ hybrid, uint32_t* __restrict__ E_tgt,
                   uint32_t* __restrict__ E_val, const uint32_t* __restrict__ order) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* head = reinterpret_cast<uint32_t*>(smem) + (size_t)warp * cagra_words(K);
  uint32_t* mask = head + kCagraHeads;  // bit a of position m: mask[(a / 32) * K + m]
  uint32_t* next = mask + 4 * K;
  uint32_t* nei0 = next + K;
  uint32_t* rank = nei0 + K;  // (detours << 8) | position
  auto head_of = [](uint32_t id) { return (id * 0x9E3779B1u) >> 22; };  // 10 bits
  for (uint32_t pos = blockIdx.x * kWarps + warp; pos < n; pos += gridDim.x * kWarps) {
    const uint32_t b = node_at(order, pos);
#pragma unroll
    for (uint32_t t = lane; t < kCagraHeads / 4; t += 32)
      reinterpret_cast<uint4*>(head)[t] = make_uint4(kInv, kInv, kInv, kInv);
    for (uint32_t t = lane; t < 4 * K; t += 32) mask[t] = 0;
    __syncwarp();
    for (uint32_t j = lane; j < K; j += 32) {
      const uint32_t id = __ldg(G + (size_t)b * K + j);
      nei0[j] = id;
      next[j] = atomicExch(&head[head_of(id)], j);
    }
    __syncwarp();
    for (uint32_t a0 = 0; a0 + 1 < K; a0 += kCagraRows) {
      uint32_t ids[kCagraRows][4];
#pragma unroll
      for (uint32_t r = 0; r < kCagraRows; ++r) {
        const uint32_t a = a0 + r;
        // the last list has no later position; an odd K's middle one is not visited
        const bool visit = a + 1 < K && !((K & 1u) && a == K / 2);
        const uint32_t* row = G + (size_t)(visit ? nei0[a] : 0u) * K;
#pragma unroll
        for (uint32_t t = 0; t < 4; ++t) {
          const uint32_t j = lane + 32 * t;
          ids[r][t] = visit && j < K ? __ldg(row + j) : kInv;
        }
      }
#pragma unroll
      for (uint32_t r = 0; r < kCagraRows; ++r) {
        const uint32_t a = a0 + r;
#pragma unroll
        for (uint32_t t = 0; t < 4; ++t) {
          if (32 * t >= K) break;
          const uint32_t id = ids[r][t];
          if (id == kInv) continue;
          for (uint32_t m = head[head_of(id)]; m != kInv; m = next[m])
            if (nei0[m] == id && m > a) atomicOr(&mask[(a >> 5) * K + m], 1u << (a & 31u));
        }
      }
    }
    __syncwarp();
    for (uint32_t m = lane; m < K; m += 32) {
      uint32_t det = 0;
#pragma unroll
      for (uint32_t w = 0; w < 4; ++w) det += (uint32_t)__popc(mask[w * K + m]);
      rank[m] = (det << 8) | m;
    }
    __syncwarp();
    rank_store(rank, nei0, K, d, b, hybrid, E_tgt, E_val, lane);
    __syncwarp();
  }
}

// collect_1hop + filter_dpg (:1713-1785): detour[m] counts earlier a with
// d(n_a, n_m) < d(u, n_m), over the reference's pair set (all a < m but the
// middle row of an odd K, :1715-1717), each warp with vectors of its own (the
// reference's warps race on one in shared memory). The pairs are screened 32 positions
// against 16 earlier ones at a time; the few ambiguous ones take the exact distance.
//
// Bound by the row gathers, mostly from L1.
__host__ __device__ inline uint32_t dpg_words(uint32_t K) { return 4 * K + kScreenFloats; }

__global__ void __launch_bounds__(kWarps * 32, 4)
    k_select_dpg(const uint32_t* __restrict__ G, const float* __restrict__ nd,
                 const __half* __restrict__ data, const float* __restrict__ norms, uint32_t n,
                 uint32_t dim, uint32_t K, uint32_t d, uint32_t* __restrict__ hybrid,
                 uint32_t* __restrict__ E_tgt, uint32_t* __restrict__ E_val,
                 const uint32_t* __restrict__ order) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t* nei0 = reinterpret_cast<uint32_t*>(smem) + (size_t)warp * dpg_words(K);
  float* nrow = reinterpret_cast<float*>(nei0 + K);
  float* nn = nrow + K;
  uint32_t* rank = reinterpret_cast<uint32_t*>(nn + K);
  float* tile = reinterpret_cast<float*>(rank + K);
  const ScreenRule rule{0, 1.0f, screen_eps(dim)};  // res < d(u, n_m)
  for (uint32_t pos = blockIdx.x * kWarps + warp; pos < n; pos += gridDim.x * kWarps) {
    const uint32_t b = node_at(order, pos);
    for (uint32_t j = lane; j < K; j += 32) {
      const uint32_t id = __ldg(G + (size_t)b * K + j);
      nei0[j] = id;
      nrow[j] = nd[(size_t)b * K + j];
      nn[j] = __ldg(norms + id);
    }
    __syncwarp();
    for (uint32_t m0 = 0; m0 < K; m0 += 32) {
      const uint32_t m = m0 + lane;
      const uint32_t id = m < K ? nei0[m] : kInv;
      const float dm = m < K ? nrow[m] : 0.0f, nm = m < K ? nn[m] : 0.0f;
      uint32_t det = 0;
      for (uint32_t a0 = 0; a0 < min(m0 + 32, K); a0 += kScreenCols) {
        const uint2 scr = screen_rows<false>(data, dim, rule, id, nm, dm, nei0 + a0, nn + a0,
                                             nrow + a0, min(kScreenCols, K - a0), tile);
        // a < m, and not the middle row of an odd K
        uint32_t pairs = m > a0 ? (m - a0 >= 32 ? kFull : (1u << (m - a0)) - 1u) : 0u;
        if ((K & 1u) && K / 2 >= a0 && K / 2 < a0 + kScreenCols) pairs &= ~(1u << (K / 2 - a0));
        det += (uint32_t)__popc(scr.x & pairs);
        uint32_t amb = scr.y & pairs;
        for (unsigned left = __ballot_sync(kFull, amb != 0); left;
             left = __ballot_sync(kFull, amb != 0)) {
          const int o = __ffs(left) - 1;
          const uint32_t a = a0 + __ffs(__shfl_sync(kFull, amb, o)) - 1;
          const float res = warp_dist(data + (size_t)nei0[a] * dim,
                                      data + (size_t)__shfl_sync(kFull, id, o) * dim, dim, lane);
          if (lane == o) {
            det += res < dm ? 1u : 0u;
            amb &= amb - 1u;
          }
        }
      }
      if (m < K) rank[m] = (det << 8) | m;
    }
    __syncwarp();
    rank_store(rank, nei0, K, d, b, hybrid, E_tgt, E_val, lane);
    __syncwarp();
  }
}

// filter_reverse_1hop (:1812-1886): dense stride-d rows written over the
// graph buffer (no kernel of this stage reads it), first d/2 forward,
// then reverse ids by ascending detour that are not already forward, then the
// remaining forward ids.
__global__ void __launch_bounds__(kWarps * 32)
    k_filter_reverse_1hop(uint32_t* __restrict__ out, const uint32_t* __restrict__ rg,
                          const uint32_t* __restrict__ rnum, const uint32_t* __restrict__ hybrid,
                          uint32_t n, uint32_t K, uint32_t d) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned char* mine = smem + (size_t)warp * ((size_t)d * 16);
  uint32_t* rev = reinterpret_cast<uint32_t*>(mine);
  uint32_t* rdet = rev + d;
  uint32_t* nid = rdet + d;
  uint32_t* row = nid + d;
  for (uint32_t b = blockIdx.x * kWarps + warp; b < n; b += gridDim.x * kWarps) {
    const uint32_t rn = min(d, rnum[b]);
    for (uint32_t i = lane; i < rn; i += 32) {
      rev[i] = rg[(size_t)b * d * 2 + i * 2];
      rdet[i] = rg[(size_t)b * d * 2 + i * 2 + 1];
    }
    for (uint32_t i = lane; i < d; i += 32) nid[i] = hybrid[(size_t)b * K + i];
    __syncwarp();
    warp_network(rn, lane, [&](uint32_t u, uint32_t v) { return rev[u] > rev[v]; },
                 [&](uint32_t u, uint32_t v) {
                   swap_(rev[u], rev[v]);
                   swap_(rdet[u], rdet[v]);
                 });
    {
      unsigned marks[4];
      for (uint32_t c = 0; c * 32 < rn; ++c) {
        const uint32_t i = c * 32 + lane;
        marks[c] = __ballot_sync(kFull, i >= 1 && i < rn && rev[i] == rev[i - 1]);
      }
      __syncwarp();
      for (uint32_t c = 0; c * 32 < rn; ++c)
        if ((marks[c] >> lane) & 1u) rdet[c * 32 + lane] = kInv;
      __syncwarp();
    }
    for (uint32_t i = lane; i < d / 2; i += 32) row[i] = nid[i];
    warp_network(rn, lane, [&](uint32_t u, uint32_t v) { return rdet[u] > rdet[v]; },
                 [&](uint32_t u, uint32_t v) {
                   swap_(rdet[u], rdet[v]);
                   swap_(rev[u], rev[v]);
                 });
    uint32_t cnt = 0;
    const uint32_t span = (rn < d / 2) ? (d - rn) : (d / 2);
    for (uint32_t i = 0; i < rn; ++i) {
      if (rn >= d / 2 && cnt >= d / 2) break;
      const uint32_t r = rev[i];
      bool flag = false;
      for (uint32_t j0 = 0; j0 < span; j0 += 32) {
        const uint32_t j = j0 + lane;
        if (__any_sync(kFull, j < span && nid[j] == r)) {
          flag = true;
          break;
        }
      }
      if (!flag) {
        if (lane == 0) row[d / 2 + cnt] = r;
        ++cnt;
      }
    }
    __syncwarp();
    const uint32_t m = min(cnt, d / 2);
    for (uint32_t i = lane; i < d / 2 - m; i += 32) row[d / 2 + m + i] = nid[i + d / 2];
    __syncwarp();
    const uint32_t written = 2 * (d / 2);
    for (uint32_t i = lane; i < written; i += 32) out[(size_t)b * d + i] = row[i];
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// Deterministic reverse-edge store. Edges e = src * stride + i are sorted by
// target with a stable radix sort, so each target's edges come in ascending
// (source, i). Slot s of a target then receives, in that order, the inserts
// whose running count c satisfies c == s (direct, c < cap) or c % mod == s
// (replacement, c >= cap), as in the sequential reading of :1465-1475 and
// :1697-1707.
__global__ void k_edge_keys(const uint32_t* __restrict__ E_tgt, const uint32_t* __restrict__ cnt,
                            uint32_t n, uint32_t stride, uint32_t* __restrict__ keys,
                            uint32_t* __restrict__ vals, uint32_t* __restrict__ deg) {
  const size_t total = (size_t)n * stride;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total;
       e += (size_t)gridDim.x * blockDim.x) {
    const uint32_t src = (uint32_t)(e / stride), i = (uint32_t)(e % stride);
    const bool valid = cnt ? (i < cnt[src]) : true;
    const uint32_t t = valid ? E_tgt[e] : n;
    keys[e] = t;
    vals[e] = (uint32_t)e;
    if (valid) atomicAdd(&deg[t], 1u);
  }
}

// mode 0: (id, f32 dist) into rg[t*K+s], rd[t*128+s], replace when closer.
// mode 1: (id, u32 detour) pairs into rg[t*2d + 2s], replace when fewer detours.
template <int kMode>
__global__ void k_reverse_fill(const uint32_t* __restrict__ sorted_e,
                               const uint32_t* __restrict__ deg, const uint32_t* __restrict__ off,
                               const uint32_t* __restrict__ E_val, uint32_t n, uint32_t stride,
                               uint32_t cap, uint32_t mod, uint32_t K, uint32_t* __restrict__ rg,
                               float* __restrict__ rd, uint32_t* __restrict__ rnum) {
  const int lane = threadIdx.x & 31;
  for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < n;
       t += (gridDim.x * blockDim.x) >> 5) {
    const uint32_t c0 = rnum[t], dg = deg[t], o = off[t];
    for (uint32_t s = lane; s < mod; s += 32) {
      uint32_t cur_id, cur_v;
      if (kMode == 0) {
        cur_id = rg[(size_t)t * K + s];
        cur_v = __float_as_uint(rd[(size_t)t * kReserve + s]);
      } else {
        cur_id = rg[(size_t)t * mod * 2 + 2 * s];
        cur_v = rg[(size_t)t * mod * 2 + 2 * s + 1];
      }
      bool touched = false;
      // smallest c >= c0 with c % mod == s
      uint32_t c = (c0 <= s) ? s : (s + ((c0 - s + mod - 1) / mod) * mod);
      for (; c < c0 + dg; c += mod) {
        const uint32_t e = sorted_e[o + (c - c0)];
        const uint32_t src = e / stride, v = E_val[e];
        bool take;
        if (c < cap) take = true;
        else if (kMode == 0) take = __uint_as_float(v) < __uint_as_float(cur_v);
        else take = cur_v > v;
        if (take) {
          cur_id = src;
          cur_v = v;
          touched = true;
        }
      }
      if (touched) {
        if (kMode == 0) {
          rg[(size_t)t * K + s] = cur_id;
          rd[(size_t)t * kReserve + s] = __uint_as_float(cur_v);
        } else {
          rg[(size_t)t * mod * 2 + 2 * s] = cur_id;
          rg[(size_t)t * mod * 2 + 2 * s + 1] = cur_v;
        }
      }
    }
    __syncwarp();
    if (lane == 0) rnum[t] = c0 + dg;
  }
}

int grid_for(uint32_t items_per_block, uint64_t items) {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const uint64_t need = (items + items_per_block - 1) / items_per_block;
  const uint64_t cap = (uint64_t)sms * 16;
  return (int)std::max<uint64_t>(1, std::min<uint64_t>(need, cap));
}

int reverse_store(const Dev& d, const uint32_t* E_tgt, const uint32_t* E_val, const uint32_t* cnt,
                  uint32_t stride, int mode, uint32_t cap, uint32_t mod, cudaStream_t s) {
  const size_t E = (size_t)d.n * stride;
  if (E >= 0xFFFFFFFFull) return fail(TAGORE_EINVAL, "too many reverse edges (%zu)", E);
  int end_bit = 1;
  while (end_bit < 32 && ((uint64_t)1 << end_bit) <= d.n) ++end_bit;
  size_t sort_tmp = 0, scan_tmp = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, sort_tmp, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                  (uint32_t*)nullptr, (uint32_t*)nullptr, (int)E, 0, end_bit, s);
  cub::DeviceScan::ExclusiveSum(nullptr, scan_tmp, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                (int)d.n, s);
  const size_t tmp = std::max(sort_tmp, scan_tmp);
  Scratch sc(s);
  const size_t bytes = E * 16 + (size_t)d.n * 8 + tmp + 256;
  TG_TRY(sc.alloc(bytes));
  uint32_t* keys = sc.as<uint32_t>();
  uint32_t* vals = keys + E;
  uint32_t* keys2 = vals + E;
  uint32_t* vals2 = keys2 + E;
  uint32_t* deg = vals2 + E;
  uint32_t* off = deg + d.n;
  void* tmp_p = reinterpret_cast<void*>(((uintptr_t)(off + d.n) + 255) & ~(uintptr_t)255);
  TG_CUDA(cudaMemsetAsync(deg, 0, (size_t)d.n * 4, s));
  k_edge_keys<<<grid_for(256, E), 256, 0, s>>>(E_tgt, cnt, d.n, stride, keys, vals, deg);
  TG_CUDA(cudaGetLastError());
  size_t t1 = tmp;
  TG_CUDA(cub::DeviceScan::ExclusiveSum(tmp_p, t1, deg, off, (int)d.n, s));
  t1 = tmp;
  TG_CUDA(cub::DeviceRadixSort::SortPairs(tmp_p, t1, keys, keys2, vals, vals2, (int)E, 0, end_bit,
                                          s));
  const int grid = grid_for(8, d.n);
  if (mode == 0)
    k_reverse_fill<0><<<grid, 256, 0, s>>>(vals2, deg, off, E_val, d.n, stride, cap, mod, d.k,
                                           d.rgraph, d.rd, d.rnum);
  else
    k_reverse_fill<1><<<grid, 256, 0, s>>>(vals2, deg, off, E_val, d.n, stride, cap, mod, d.k,
                                           d.rgraph, d.rd, d.rnum);
  TG_CUDA(cudaGetLastError());
  return TAGORE_OK;
}

int validate(const Dev& d, cudaStream_t s) {
  Scratch sc(s);
  TG_TRY(sc.alloc(4));
  TG_CUDA(cudaMemsetAsync(sc.p, 0, 4, s));
  const size_t cnt = (size_t)d.n * d.k;
  k_validate<<<grid_for(256, cnt), 256, 0, s>>>(d.graph, cnt, d.n, sc.as<uint32_t>());
  TG_CUDA(cudaGetLastError());
  uint32_t bad = 0;
  TG_CUDA(cudaMemcpyAsync(&bad, sc.p, 4, cudaMemcpyDeviceToHost, s));
  TG_CUDA(cudaStreamSynchronize(s));
  if (bad) return fail(TAGORE_EINVAL, "graph holds an id >= POINTS (%u)", d.n);
  return TAGORE_OK;
}

int check_shape(const Dev& d, uint32_t fd) {
  if (d.n == 0 || d.k == 0 || d.dim == 0) return fail(TAGORE_EINVAL, "empty graph");
  if (d.dim % 4) return fail(TAGORE_EINVAL, "DIM must be a multiple of 4 (got %u)", d.dim);
  if (d.k > 128) return fail(TAGORE_EINVAL, "K must be <= 128 (got %u)", d.k);
  if (fd == 0 || fd > d.k) return fail(TAGORE_EINVAL, "FINAL_DEGREE must be in [1, K]");
  return TAGORE_OK;
}

// One wave of resident blocks (SMs x blocks per SM at this shared-memory
// size), fewer when the items do not fill it.
int resident_grid(const void* fn, int threads, size_t smem, uint32_t items_per_block,
                  uint64_t items, int* grid) {
  int dev = 0, sms = 0, per_sm = 0;
  TG_CUDA(cudaGetDevice(&dev));
  TG_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  TG_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
  if (per_sm < 1) return fail(TAGORE_EINVAL, "kernel does not fit on an SM (%zu B shared)", smem);
  const uint64_t need = (items + items_per_block - 1) / items_per_block;
  *grid = (int)std::max<uint64_t>(1, std::min<uint64_t>(need, (uint64_t)sms * per_sm));
  return TAGORE_OK;
}

int set_smem(const void* fn, size_t bytes) {
  if (bytes > 227 * 1024) return fail(TAGORE_EINVAL, "shared memory request too large (%zu)", bytes);
  TG_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return TAGORE_OK;
}

// The select's processing order (see k_label_min), in scratch `sc`.
int locality_order(const Dev& d, Scratch& sc, const uint32_t** order, cudaStream_t s) {
  const uint32_t n = d.n, hops = std::min(kLabelHops, d.k);
  int end_bit = 1;
  while (end_bit < 32 && ((uint64_t)1 << end_bit) <= n) ++end_bit;
  size_t tmp = 0;
  TG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                          (uint32_t*)nullptr, (uint32_t*)nullptr, (int)n, 0,
                                          end_bit, s));
  TG_TRY(sc.alloc((size_t)n * 16 + tmp + 256));
  uint32_t* lab = sc.as<uint32_t>();
  uint32_t* ids = lab + n;
  uint32_t* lab2 = ids + n;
  uint32_t* out = lab2 + n;
  void* tmp_p = reinterpret_cast<char*>(out + n) + (256 - ((uintptr_t)(out + n) & 255)) % 256;
  const int g = grid_for(256, n);
  k_label_init<<<g, 256, 0, s>>>(lab, ids, n);
  count_launch();
  for (uint32_t r = 0; r < kLabelRounds; ++r) {
    k_label_min<<<g, 256, 0, s>>>(d.graph, d.k, hops, lab, n);
    count_launch();
  }
  TG_CUDA(cudaGetLastError());
  TG_CUDA(cub::DeviceRadixSort::SortPairs(tmp_p, tmp, lab, lab2, ids, out, (int)n, 0, end_bit, s));
  *order = out;
  return TAGORE_OK;
}

int reverse_grid(uint32_t fd, uint32_t K, uint32_t n, int* grid) {
  const size_t sm = reverse_bytes(fd, K) * kWarps;
  TG_TRY(set_smem((const void*)k_filter_reverse, sm));
  return resident_grid((const void*)k_filter_reverse, kWarps * 32, sm, kWarps, n, grid);
}

// Nodes per collect / filter pair: bounds the candidate lists in memory (about
// 1.2 GB at K = 96) and still fills the chip dozens of times over. Where the device
// has no room for them the batch is halved, down to kMinBatch (under 3 MB).
constexpr uint32_t kSelectBatch = 1u << 18, kMinBatch = 1u << 9;

bool on_16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

int launch_cal_ep(const Dev& d, uint32_t topm, uint32_t* ep_dev, cudaStream_t s) {
  const size_t sm = beam_bytes(topm, d.k);
  TG_TRY(set_smem((const void*)k_cal_ep, sm));
  k_cal_ep<<<1, 32, sm, s>>>(d.graph, d.data, d.center, d.dim, d.k, topm, ep_dev);
  count_launch();
  TG_CUDA(cudaGetLastError());
  return TAGORE_OK;
}

void launch_row_norms(const Dev& d, float* norms, cudaStream_t s) {
  k_row_norms<<<grid_for(8, d.n), 256, 0, s>>>(d.data, d.n, d.dim, norms);
  count_launch();
}

int launch_filter_reverse(const Dev& d, int grid, const float* norms, uint32_t fd, int metric,
                          float thre, const uint32_t* P_ids, const uint32_t* P_cnt,
                          const uint32_t* order, cudaStream_t s) {
  const size_t sm = reverse_bytes(fd, d.k) * kWarps;
  TG_TRY(set_smem((const void*)k_filter_reverse, sm));
  k_filter_reverse<<<grid, kWarps * 32, sm, s>>>(d.graph, d.nd, d.rgraph, d.rd, d.rnum, d.data,
                                                 norms, d.n, d.dim, d.k, fd, metric, thre, P_ids,
                                                 P_cnt, order);
  count_launch();
  TG_CUDA(cudaGetLastError());
  return TAGORE_OK;
}

// Collect (path or 2-hop) and filter, then reverse store and filter_reverse.
int run_dist_prune(const Dev& d, const PruneArgs& a, bool path, int metric, uint32_t* ep_host,
                   cudaStream_t s) {
  const uint32_t fd = a.final_degree, K = d.k;
  if (!path && K * K < kSelectCand) return fail(TAGORE_EINVAL, "2-hop collect needs K*K >= 480");
  if (path && (a.topm == 0 || a.topm > 256)) return fail(TAGORE_EINVAL, "TOPM must be in [1, 256]");
  const SelLayout lay{path ? a.topm : 0u, K, 0};
  Scratch sc(s);
  // [u64 rows scored, candidates listed, candidates tested][u32 entry point][u32 unused]
  // | select rows | norms
  const size_t head = 32;
  TG_TRY(sc.alloc(head + (size_t)d.n * fd * 8 + (size_t)d.n * 8));
  unsigned long long* work = sc.as<unsigned long long>();
  uint32_t* ep_dev = reinterpret_cast<uint32_t*>(work + 3);
  uint32_t* P_ids = reinterpret_cast<uint32_t*>(sc.as<unsigned char>() + head);
  float* P_dis = reinterpret_cast<float*>(P_ids + (size_t)d.n * fd);
  uint32_t* P_cnt = reinterpret_cast<uint32_t*>(P_dis + (size_t)d.n * fd);
  float* norms = reinterpret_cast<float*>(P_cnt + d.n);
  TG_CUDA(cudaMemsetAsync(work, 0, head, s));
  if (path) {
    stage_begin("prune_cal_ep", s);
    TG_TRY(launch_cal_ep(d, a.topm, ep_dev, s));
    stage_end("prune_cal_ep", s);
  }
  const size_t sm = lay.bytes() * kWarps, smf = kept_bytes(fd) * kWarps;
  auto* fn = !path           ? k_collect<false, true>
             : on_16(d.data) ? k_collect<true, true>
                             : k_collect<true, false>;
  TG_TRY(set_smem((const void*)fn, sm));
  TG_TRY(set_smem((const void*)k_filter, smf));
  int grid = 0, gridf = 0;
  TG_TRY(resident_grid((const void*)fn, kWarps * 32, sm, kWarps, d.n, &grid));
  TG_TRY(resident_grid((const void*)k_filter, kWarps * 32, smf, kWarps, d.n, &gridf));
  Scratch rings(s), lists(s);
  if (path) TG_TRY(rings.alloc((size_t)grid * kWarps * kSelectCand * 8));
  uint32_t* ring_ids = path ? rings.as<uint32_t>() : nullptr;
  float* ring_dis =
      path ? reinterpret_cast<float*>(ring_ids + (size_t)grid * kWarps * kSelectCand) : nullptr;
  Scratch ord(s);
  const uint32_t* order = nullptr;
  stage_begin("prune_order", s);
  TG_TRY(locality_order(d, ord, &order, s));
  launch_row_norms(d, norms, s);
  stage_end("prune_order", s);
  // candidate lists | two counters per batch; taken last and given back before the
  // reverse edges, so that they ask for no memory the prune does not find
  uint32_t batch = std::min(d.n, kSelectBatch), batches = 0;
  for (;; batch /= 2) {
    batches = (d.n + batch - 1) / batch;
    const int rc = lists.alloc((size_t)batch * (lay.L() * 8 + 4) + (size_t)batches * 8);
    if (rc == TAGORE_OK) break;
    if (rc != TAGORE_ENOMEM || batch <= kMinBatch) return rc;
  }
  uint32_t* L_ids = lists.as<uint32_t>();
  float* L_dis = reinterpret_cast<float*>(L_ids + (size_t)batch * lay.L());
  uint32_t* L_cnt = reinterpret_cast<uint32_t*>(L_dis + (size_t)batch * lay.L());
  uint32_t* ctr = L_cnt + batch;
  TG_CUDA(cudaMemsetAsync(ctr, 0, (size_t)batches * 8, s));
  const char* sel_name = path ? "prune_select_path" : "prune_select_2hop";
  for (uint32_t i = 0; i < batches; ++i) {
    const uint32_t first = i * batch, cnt = std::min(batch, d.n - first);
    stage_begin(sel_name, s);
    fn<<<grid, kWarps * 32, sm, s>>>(d.graph, d.nd, d.data, first, cnt, d.dim, K, ep_dev,
                                     ctr + 2 * i, a.topm, L_ids, L_dis, L_cnt, work, ring_ids,
                                     ring_dis, order);
    count_launch();
    stage_end(sel_name, s);
    TG_CUDA(cudaGetLastError());
    stage_begin("prune_filter", s);
    k_filter<<<gridf, kWarps * 32, smf, s>>>(L_ids, L_dis, L_cnt, lay.L(), d.nd, d.data, norms, first,
                                             cnt, d.dim, K, ctr + 2 * i + 1, fd, path ? 0 : 1,
                                             a.thre, P_ids, P_dis, P_cnt, work + 1, order);
    count_launch();
    stage_end("prune_filter", s);
    TG_CUDA(cudaGetLastError());
  }
  rings.release();
  lists.release();
  stage_begin("prune_reverse_store", s);
  TG_TRY(reverse_store(d, P_ids, reinterpret_cast<const uint32_t*>(P_dis), P_cnt, fd, 0, K, K, s));
  stage_end("prune_reverse_store", s);
  int gridr = 0;
  TG_TRY(reverse_grid(fd, K, d.n, &gridr));
  stage_begin("prune_filter_reverse", s);
  TG_TRY(launch_filter_reverse(d, gridr, norms, fd, metric, a.thre, P_ids, P_cnt, order, s));
  stage_end("prune_filter_reverse", s);
  if (path && ep_host) {
    TG_CUDA(cudaMemcpyAsync(ep_host, ep_dev, 4, cudaMemcpyDeviceToHost, s));
  }
  unsigned long long w[3] = {0, 0, 0};
  if (profiling()) TG_CUDA(cudaMemcpyAsync(w, work, sizeof(w), cudaMemcpyDeviceToHost, s));
  TG_CUDA(cudaStreamSynchronize(s));
  if (profiling()) {
    // collect: every scored row (2d bytes), the kNN row and its distances in, the
    // list out; filter: the tested candidates' entries and rows in, the selected ids
    // and distances out (8 bytes an entry throughout)
    const uint64_t row = 2ull * d.dim, n = d.n;
    stage_add(sel_name, w[0] * row + n * 8 * K + w[1] * 8, n);
    stage_add("prune_filter", w[2] * (row + 8) + n * (8ull * fd + 4), n);
  }
  return TAGORE_OK;
}

int run_rank_prune(const Dev& d, const PruneArgs& a, bool dpg, cudaStream_t s) {
  const uint32_t K = d.k, dd = a.final_degree;
  if (2 * dd > kReserve) return fail(TAGORE_EINVAL, "degree must be <= 64 for rank prunes");
  uint32_t cap = dd;
  if (dpg) {
    if (K < dd + 1 || K - dd - 1 > dd)
      return fail(TAGORE_EINVAL,
                  "DPG needs degree+1 <= K <= 2*degree+1 (the reference's reverse rows overflow)");
    cap = K - dd - 1;
  }
  Scratch sc(s);
  TG_TRY(sc.alloc((size_t)d.n * dd * 8 + (dpg ? (size_t)d.n * 4 : 0) + 16));
  uint32_t* E_tgt = sc.as<uint32_t>();
  uint32_t* E_val = E_tgt + (size_t)d.n * dd;
  float* norms = reinterpret_cast<float*>(E_val + (size_t)d.n * dd);  // DPG only
  const int grid = grid_for(kWarps, d.n);
  Scratch ord(s);
  const uint32_t* order = nullptr;
  stage_begin("prune_order", s);
  TG_TRY(locality_order(d, ord, &order, s));
  stage_end("prune_order", s);
  const char* sel_name = dpg ? "prune_select_dpg" : "prune_select_cagra";
  stage_begin(sel_name, s);
  if (!dpg) {
    const size_t sm = (size_t)cagra_words(K) * 4 * kWarps;
    TG_TRY(set_smem((const void*)k_select_cagra, sm));
    k_select_cagra<<<grid, kWarps * 32, sm, s>>>(d.graph, d.n, K, dd, d.hybrid, E_tgt, E_val,
                                                 order);
  } else {
    launch_row_norms(d, norms, s);
    const size_t sm = (size_t)dpg_words(K) * 4 * kWarps;
    TG_TRY(set_smem((const void*)k_select_dpg, sm));
    k_select_dpg<<<grid, kWarps * 32, sm, s>>>(d.graph, d.nd, d.data, norms, d.n, d.dim, K, dd,
                                               d.hybrid, E_tgt, E_val, order);
  }
  count_launch();
  TG_CUDA(cudaGetLastError());
  stage_end(sel_name, s);
  stage_begin("prune_reverse_store", s);
  TG_TRY(reverse_store(d, E_tgt, E_val, nullptr, dd, 1, cap, dd, s));
  stage_end("prune_reverse_store", s);
  stage_begin("prune_filter_reverse_1hop", s);
  const size_t sm2 = ((size_t)dd * 16) * kWarps;
  TG_TRY(set_smem((const void*)k_filter_reverse_1hop, sm2));
  k_filter_reverse_1hop<<<grid, kWarps * 32, sm2, s>>>(d.graph, d.rgraph, d.rnum, d.hybrid, d.n,
                                                       K, dd);
  count_launch();
  TG_CUDA(cudaGetLastError());
  stage_end("prune_filter_reverse_1hop", s);
  TG_CUDA(cudaStreamSynchronize(s));
  return TAGORE_OK;
}

}  // namespace

int stage_cal_ep(const Dev& d, uint32_t topm, uint32_t* ep_host, cudaStream_t s) {
  TG_TRY(check_shape(d, 1));
  TG_TRY(validate(d, s));
  Scratch sc(s);
  TG_TRY(sc.alloc(4));
  TG_TRY(launch_cal_ep(d, topm, sc.as<uint32_t>(), s));
  TG_CUDA(cudaMemcpyAsync(ep_host, sc.p, 4, cudaMemcpyDeviceToHost, s));
  TG_CUDA(cudaStreamSynchronize(s));
  return TAGORE_OK;
}

int prune_index(const Dev& d, const PruneArgs& a, const std::string& type, uint32_t* ep_host,
                cudaStream_t s) {
  TG_TRY(check_shape(d, a.final_degree));
  TG_TRY(validate(d, s));
  if (type == "NSG" || type == "Vamana") {
    PruneArgs b = a;
    if (type == "NSG") b.thre = 1.0f;  // pybind.cu:181,183 pass 1.0
    return run_dist_prune(d, b, true, 0, ep_host, s);
  }
  if (type == "NSSG") return run_dist_prune(d, a, false, 1, ep_host, s);
  if (type == "CAGRA") return run_rank_prune(d, a, false, s);
  if (type == "DPG") return run_rank_prune(d, a, true, s);
  return fail(TAGORE_EINVAL, "unknown index_type '%s' (NSG, Vamana, NSSG, CAGRA, DPG)",
              type.c_str());
}

// ---------------------------------------------------------------------------
// Pruning_with_CFS for path|2-hop with dist|angle without allocating: every
// temporary of run_dist_prune and reverse_store (the validation flag, the
// select rows, the reverse-edge keys, CUB's temporary storage) is carved
// from one file-scope device array. The array is per device and shared by all
// calls on it, so calls whose GPU work overlaps would race on it; the C entry
// point serialises its calls under a lock and returns only after the work has
// finished.
namespace {
__device__ __align__(256) unsigned char g_static_scratch[kStaticScratchBytes];

struct Carve {
  unsigned char* base;
  size_t used = 0;
  void* take(size_t bytes) {
    void* p = base ? base + used : nullptr;
    used += (bytes + 255) & ~(size_t)255;
    return p;
  }
};
}  // namespace

int prune_cfs_static(const Dev& d, const PruneArgs& a, const std::string& mode,
                     const std::string& metric, uint32_t* ep_host, cudaStream_t s) {
  TG_TRY(check_shape(d, a.final_degree));
  const bool path = mode == "path";
  if ((!path && mode != "2-hop") || (metric != "dist" && metric != "angle"))
    return fail(TAGORE_EINVAL,
                "without allocation only path|2-hop with dist|angle are offered (mode='%s' "
                "metric='%s')",
                mode.c_str(), metric.c_str());
  const int m = metric == "angle" ? 1 : 0;
  const uint32_t fd = a.final_degree, K = d.k;
  if (!path && K * K < kSelectCand) return fail(TAGORE_EINVAL, "2-hop collect needs K*K >= 480");
  if (path && (a.topm == 0 || a.topm > 256)) return fail(TAGORE_EINVAL, "TOPM must be in [1, 256]");
  const size_t E = (size_t)d.n * fd;
  if (E >= 0xFFFFFFFFull) return fail(TAGORE_EINVAL, "too many reverse edges (%zu)", E);
  int end_bit = 1;
  while (end_bit < 32 && ((uint64_t)1 << end_bit) <= d.n) ++end_bit;
  size_t sort_tmp = 0, scan_tmp = 0;
  TG_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, sort_tmp, (uint32_t*)nullptr,
                                          (uint32_t*)nullptr, (uint32_t*)nullptr,
                                          (uint32_t*)nullptr, (int)E, 0, end_bit, s));
  TG_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, scan_tmp, (uint32_t*)nullptr, (uint32_t*)nullptr,
                                        (int)d.n, s));
  const size_t tmp = std::max(sort_tmp, scan_tmp);
  // The select kernel's grid is capped here so that its per-warp rings of
  // scored nodes (path collect) stay small: 64 blocks, under 1 MB.
  SelLayout lay{path ? a.topm : 0u, K, kept_bytes(fd)};
  const size_t sm = lay.bytes() * kWarps;
  auto* fn = !path           ? k_select<false, true>
             : on_16(d.data) ? k_select<true, true>
                             : k_select<true, false>;
  TG_TRY(set_smem((const void*)fn, sm));
  int grid = 0;
  TG_TRY(resident_grid((const void*)fn, kWarps * 32, sm, kWarps, d.n, &grid));
  grid = std::min(grid, 64);
  const size_t ring_n = path ? (size_t)grid * kWarps * kSelectCand : 0;
  // Layout: flags | select rows | reverse-edge keys | CUB temporary | rings.
  uint32_t* ring_ids = nullptr;
  float* ring_dis = nullptr;
  auto layout = [&](Carve& c, uint32_t** flags, uint32_t** P_ids, float** P_dis, uint32_t** P_cnt,
                    uint32_t** keys, uint32_t** vals, uint32_t** keys2, uint32_t** vals2,
                    uint32_t** deg, uint32_t** off, void** tmp_p) {
    *flags = (uint32_t*)c.take(16);  // [0] bad id, [1] entry point, [2] node counter
    *P_ids = (uint32_t*)c.take(E * 4);
    *P_dis = (float*)c.take(E * 4);
    *P_cnt = (uint32_t*)c.take((size_t)d.n * 4);
    *keys = (uint32_t*)c.take(E * 4);
    *vals = (uint32_t*)c.take(E * 4);
    *keys2 = (uint32_t*)c.take(E * 4);
    *vals2 = (uint32_t*)c.take(E * 4);
    *deg = (uint32_t*)c.take((size_t)d.n * 4);
    *off = (uint32_t*)c.take((size_t)d.n * 4);
    *tmp_p = c.take(tmp);
    ring_ids = (uint32_t*)c.take(ring_n * 4);
    ring_dis = (float*)c.take(ring_n * 4);
  };
  uint32_t *flags, *P_ids, *P_cnt, *keys, *vals, *keys2, *vals2, *deg, *off;
  float* P_dis;
  void* tmp_p;
  Carve sizing{nullptr};
  layout(sizing, &flags, &P_ids, &P_dis, &P_cnt, &keys, &vals, &keys2, &vals2, &deg, &off, &tmp_p);
  if (sizing.used > kStaticScratchBytes)
    return fail(TAGORE_EINVAL,
                "POINTS=%u FINAL_DEGREE=%u needs %zu bytes of scratch; the static scratch holds "
                "%zu",
                d.n, fd, sizing.used, kStaticScratchBytes);
  void* base = nullptr;
  TG_CUDA(cudaGetSymbolAddress(&base, g_static_scratch));
  Carve c{static_cast<unsigned char*>(base)};
  layout(c, &flags, &P_ids, &P_dis, &P_cnt, &keys, &vals, &keys2, &vals2, &deg, &off, &tmp_p);

  // From the first queued operation on, every return waits for the stream,
  // so the caller's lock is released only when no work on the shared array
  // is still in flight, error paths included.
  struct DrainOnExit {
    cudaStream_t s;
    ~DrainOnExit() { cudaStreamSynchronize(s); }
  } drain{s};

  // validate (as validate())
  TG_CUDA(cudaMemsetAsync(flags, 0, 16, s));
  const size_t cnt = (size_t)d.n * d.k;
  k_validate<<<grid_for(256, cnt), 256, 0, s>>>(d.graph, cnt, d.n, flags);
  count_launch();
  TG_CUDA(cudaGetLastError());
  uint32_t bad = 0;
  TG_CUDA(cudaMemcpyAsync(&bad, flags, 4, cudaMemcpyDeviceToHost, s));
  TG_CUDA(cudaStreamSynchronize(s));
  if (bad) return fail(TAGORE_EINVAL, "graph holds an id >= POINTS (%u)", d.n);

  // select (as run_dist_prune)
  uint32_t* ep_dev = flags + 1;
  uint32_t* ctr = flags + 2;
  if (path) TG_TRY(launch_cal_ep(d, a.topm, ep_dev, s));
  // The screens' norms take the place of the reverse-edge keys (E >= n words),
  // which are written after the select and read before filter_reverse.
  float* norms = reinterpret_cast<float*>(keys);
  launch_row_norms(d, norms, s);
  TG_CUDA(cudaGetLastError());
  fn<<<grid, kWarps * 32, sm, s>>>(d.graph, d.nd, d.data, norms, d.n, d.dim, K, ep_dev, ctr, a.topm,
                                   fd, a.thre, P_ids, P_dis, P_cnt, ring_ids, ring_dis);
  count_launch();
  TG_CUDA(cudaGetLastError());

  // reverse store (as reverse_store with mode 0, cap = mod = K)
  TG_CUDA(cudaMemsetAsync(deg, 0, (size_t)d.n * 4, s));
  k_edge_keys<<<grid_for(256, E), 256, 0, s>>>(P_ids, P_cnt, d.n, fd, keys, vals, deg);
  count_launch();
  TG_CUDA(cudaGetLastError());
  size_t t1 = tmp;
  TG_CUDA(cub::DeviceScan::ExclusiveSum(tmp_p, t1, deg, off, (int)d.n, s));
  t1 = tmp;
  TG_CUDA(cub::DeviceRadixSort::SortPairs(tmp_p, t1, keys, keys2, vals, vals2, (int)E, 0, end_bit,
                                          s));
  k_reverse_fill<0><<<grid_for(8, d.n), 256, 0, s>>>(vals2, deg, off,
                                                     reinterpret_cast<const uint32_t*>(P_dis),
                                                     d.n, fd, K, K, d.k, d.rgraph, d.rd, d.rnum);
  count_launch();
  TG_CUDA(cudaGetLastError());

  // filter_reverse
  launch_row_norms(d, norms, s);
  TG_TRY(launch_filter_reverse(d, grid, norms, fd, m, a.thre, P_ids, P_cnt, nullptr, s));
  if (path && ep_host) TG_CUDA(cudaMemcpyAsync(ep_host, ep_dev, 4, cudaMemcpyDeviceToHost, s));
  TG_CUDA(cudaStreamSynchronize(s));
  return TAGORE_OK;
}

int prune_cfs(const Dev& d, const PruneArgs& a, const std::string& mode, const std::string& metric,
              uint32_t* ep_host, cudaStream_t s) {
  TG_TRY(check_shape(d, a.final_degree));
  TG_TRY(validate(d, s));
  const bool dist_like = metric == "dist" || metric == "angle";
  const int m = metric == "angle" ? 1 : 0;
  if (mode == "path" && dist_like) return run_dist_prune(d, a, true, m, ep_host, s);
  if (mode == "2-hop" && dist_like) return run_dist_prune(d, a, false, m, ep_host, s);
  if (mode == "1-hop" && metric == "rank") return run_rank_prune(d, a, false, s);
  return fail(TAGORE_EINVAL,
              "unsupported CFS combination mode='%s' metric='%s' (path|2-hop with dist|angle, "
              "1-hop with rank)",
              mode.c_str(), metric.c_str());
}

}  // namespace tagore
