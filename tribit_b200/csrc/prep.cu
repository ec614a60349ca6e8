// GPU preprocessing pipeline; see prep.cuh.
#include <algorithm>
#include <vector>

#include "prep.cuh"
#include "scan.cuh"

namespace tb {
namespace {

constexpr int kThreads = 256;
constexpr uint32_t kFull = 0xffffffffu;

inline unsigned grid_for(uint64_t n, int per_thread = 1) {
  uint64_t g = ceil_div<uint64_t>(n, (uint64_t)kThreads * per_thread);
  return (unsigned)(g == 0 ? 1 : g);
}

// Graph of entry i in batch mode: largest g with eoff[g] <= i.
__device__ __forceinline__ uint32_t graph_of_entry(const uint64_t* eoff, uint32_t G, uint64_t i) {
  uint32_t lo = 0, hi = G;  // answer in [0, G)
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (eoff[mid] <= i)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

constexpr uint32_t kNoId = 0xFFFFFFFFu;  // no vertex has this id (n < 2^32)

// Decodes a thread's entries, in increasing order, into global vertex ids. In
// batch mode the entry's graph is searched for once and then followed (a
// search an entry: 1,732 us of degrees and 902 of row counts in the 512-graph
// batch, now 802 and 733).
struct EntryReader {
  const PrepInput& in;
  unsigned int* err;
  uint64_t base = 0, lim, end = 0;  // the graph's first vertex, its vertices, the end of its entries
  uint32_t g = 0;
  __device__ __forceinline__ EntryReader(const PrepInput& in_, unsigned int* err_) : in(in_), err(err_), lim(in_.n) {}
  // False (ids kNoId) for an entry naming a vertex outside its graph (flagged)
  // and for a self-loop (silently dropped, as read_mtx does at tribit.cu:261-267).
  __device__ __forceinline__ bool ids(uint64_t e, uint64_t i, uint32_t& a, uint32_t& b) {
    if (in.G && i >= end) {
      for (int t = 0; t < 4 && end && in.eoff[g + 1] <= i; ++t) ++g;
      if (end == 0 || in.eoff[g + 1] <= i) g = graph_of_entry(in.eoff, in.G, i);
      end = in.eoff[g + 1];
      base = in.voff[g];
      lim = in.voff[g + 1] - base;
    }
    const uint64_t x = e >> 32, y = e & 0xffffffffull;
    a = b = kNoId;
    if (x >= lim || y >= lim) {
      atomicOr(err, kErrIdRange);
      return false;
    }
    if (x == y) return false;
    a = (uint32_t)(x + base);
    b = (uint32_t)(y + base);
    return true;
  }
};

// Lanes holding the same key in a row, as a sorted edge list gives them: the
// run's first lane, its length and whether this lane is the first. One atomic
// a run takes the place of one a lane (a warp's 32 on one address are served
// one after another: sorted cliques, degrees 906 us, now 203, row counts 1,006,
// now 127, row fill 1,226, now 97).
struct KeyRun {
  uint32_t first, len;
  bool head;
};
__device__ __forceinline__ KeyRun key_run(uint32_t key) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t prev = __shfl_up_sync(kFull, key, 1);
  const uint32_t heads = __ballot_sync(kFull, lane == 0 || key != prev);
  KeyRun r;
  r.first = 31 - __clz(heads & (kFull >> (31 - lane)));
  const uint32_t after = lane == 31 ? 0u : heads >> (lane + 1);
  r.len = (after ? lane + (uint32_t)__ffs(after) : 32u) - r.first;
  r.head = r.first == lane;
  return r;
}

// Degrees (with duplicates) over entries [i0, i1), a contiguous share a CTA. A
// power-law graph's hubs put millions of updates on a few lines of counters,
// each line served one update at a time (Chung-Lu, 7,115 vertices: 38 us, now 12), so each CTA counts the ids that win a
// slot of a table in shared memory there: its share is sampled, every sampled
// id claims its slot and the last one stays, which an id does about as often
// as it occurs. Ids without a slot are counted in global memory.
constexpr uint32_t kDegSlots = 8192;
constexpr uint32_t kDegThreads = 512;
constexpr uint32_t kDegSample = 4096;  // entries, and the fewest a CTA takes
constexpr int kDegAhead = 4;           // entries in flight a thread
static_assert((kDegSlots & (kDegSlots - 1)) == 0, "the slot hash takes the top bits");
// Hashed where there are more ids than slots, by a multiplier: hubs' ids often
// differ in few bits, and an exclusive-or of id bits put them on one another's
// slots (RMAT-20: 92% of the updates without a slot and 1.4% of all on the
// hottest line, 612 us; hashed 77% and 0.3%, the whole count 3,343 us, now 3,029).
__device__ __forceinline__ uint32_t deg_slot(uint32_t id, uint64_t n) {
  return n <= kDegSlots ? id : (id * 0x9E3779B1u) / (uint32_t)((1ull << 32) / kDegSlots);
}

__global__ void __launch_bounds__(kDegThreads) k_degree(PrepInput in, uint64_t i0, uint64_t i1,
                                                        uint32_t* __restrict__ deg, unsigned int* err) {
  extern __shared__ uint32_t deg_sm[];
  uint32_t* tag = deg_sm;
  uint32_t* cnt = deg_sm + kDegSlots;
  const uint64_t share = ceil_div<uint64_t>(i1 - i0, gridDim.x);
  const uint64_t c0 = min(i1, i0 + share * blockIdx.x), c1 = min(i1, c0 + share);
  for (uint32_t s = threadIdx.x; s < kDegSlots; s += kDegThreads) {
    tag[s] = kNoId;
    cnt[s] = 0;
  }
  __syncthreads();
  {
    EntryReader rd(in, err);
    const uint64_t step = max((c1 - c0) / kDegSample, (uint64_t)1);
    for (uint64_t j = threadIdx.x, i = c0 + j * step; j < kDegSample && i < c1; j += kDegThreads, i = c0 + j * step) {
      uint32_t a, b;
      if (rd.ids(in.entries[i], i, a, b)) {
        tag[deg_slot(a, in.n)] = a;
        tag[deg_slot(b, in.n)] = b;
      }
    }
  }
  __syncthreads();
  EntryReader rd(in, err);
  auto count = [&](uint32_t id) {
    const KeyRun r = key_run(id);
    if (!r.head || id == kNoId) return;
    const uint32_t s = deg_slot(id, in.n);
    if (tag[s] == id)
      atomicAdd(&cnt[s], r.len);
    else
      atomicAdd(&deg[id], r.len);
  };
  for (uint64_t c = c0; c < c1; c += kDegThreads * kDegAhead) {
    uint64_t e[kDegAhead];
#pragma unroll
    for (int k = 0; k < kDegAhead; ++k) {
      const uint64_t i = c + k * kDegThreads + threadIdx.x;
      e[k] = i < c1 ? in.entries[i] : 0ull;  // 0: a self-loop
    }
#pragma unroll
    for (int k = 0; k < kDegAhead; ++k) {
      const uint64_t i = c + k * kDegThreads + threadIdx.x;
      uint32_t a = kNoId, b = kNoId;
      if (i < c1) rd.ids(e[k], i, a, b);
      __syncwarp();
      count(a);
      count(b);
    }
  }
  __syncthreads();
  for (uint32_t s = threadIdx.x; s < kDegSlots; s += kDegThreads)
    if (cnt[s]) atomicAdd(&deg[tag[s]], cnt[s]);
}

void degree_pass(const PrepInput& in, uint64_t i0, uint64_t i1, uint32_t* deg, unsigned int* err, cudaStream_t st) {
  if (i0 >= i1) return;
  constexpr int kSmem = 2 * kDegSlots * sizeof(uint32_t);
  once_per_device<2>([] { TB_CUDA(cudaFuncSetAttribute(k_degree, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem)); });
  const uint64_t ctas = std::min<uint64_t>(148 * 3, ceil_div<uint64_t>(i1 - i0, kDegSample));
  k_degree<<<(unsigned)ctas, kDegThreads, kSmem, st>>>(in, i0, i1, deg, err);
  TB_LAUNCH_CHECK();
}

__device__ __forceinline__ uint32_t graph_of_vertex(const uint64_t* voff, uint32_t G, uint64_t v) {
  uint32_t lo = 0, hi = G;
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (voff[mid] <= v)
      lo = mid;
    else
      hi = mid;
  }
  return lo;
}

// Vertices are ranked by (graph, degree, id) through a degree key of `bits`
// bits, two radix passes at 16: degrees below 2^(bits - 1) are exact, larger
// ones (hubs, at most 2E >> (bits - 1) of them) keep their leading bit and the
// next `mant` ones. Hubs that share a key lie side by side after the sort and
// are then placed by their degrees (hub_place), so the order is the full
// degrees' in half the passes. That compares hubs of one key pairwise: from
// kDegreeBits on there are few, with kLeastDegreeBits where 2E >> (bits - 1) is at
// most kHubGroup. mant < 0, when many graphs leave fewer bits: degrees are capped at 2^bits - 1.
struct DegreeKey {
  int bits, mant;
};
constexpr int kDegreeBits = 16, kLeastDegreeBits = 12;
constexpr uint64_t kHubGroup = 8192;
inline bool told_apart(int bits, uint64_t E) {
  return bits >= kDegreeBits || (bits >= kLeastDegreeBits && (2 * E) >> (bits - 1) <= kHubGroup);
}
inline DegreeKey degree_key_of(int bits, uint64_t E) {
  if (bits >= 32) return {32, -1};              // exact
  if (!told_apart(bits, E)) return {bits, -1};  // at 0, degrees are not told apart
  int m = bits - 1;                          // (33 - bits) leading bits times 2^m must fit above 2^(bits - 1)
  while (((33ll - bits) << m) > (1ll << (bits - 1))) --m;
  return {bits, m};
}
__device__ __forceinline__ uint32_t degree_key(uint32_t d, DegreeKey k) {
  if (k.bits >= 32) return d;
  if (k.bits == 0) return 0;
  const uint32_t half = 1u << (k.bits - 1);
  if (d < half) return d;
  if (k.mant < 0) return min(d, 2 * half - 1);
  const int e = 31 - __clz(d);  // >= bits - 1 > mant
  return half + ((uint32_t)(e - (k.bits - 1)) << k.mant) + ((d >> (e - k.mant)) & ((1u << k.mant) - 1u));
}
// Whether vertices of other degrees may share the key (graph bits above it, if any).
__device__ __forceinline__ bool hub_key(uint32_t key, DegreeKey k) {
  return k.mant >= 0 && ((key >> (k.bits - 1)) & 1u);
}
// Place in (key, degree, id) order of the vertex at place r of the stable (key,
// id) order of n vertices, its key a hub key. key_at(p), degree_at(p): of the vertex at place p.
template <class KeyAt, class DegreeAt>
__device__ __forceinline__ uint64_t hub_place(uint64_t r, uint64_t n, const KeyAt& key_at, const DegreeAt& degree_at) {
  const uint32_t key = key_at(r), d = degree_at(r);
  uint64_t at = r;
  for (uint64_t p = r; p > 0 && key_at(p - 1) == key; --p) at -= degree_at(p - 1) > d;
  for (uint64_t p = r + 1; p < n && key_at(p) == key; ++p) at += degree_at(p) < d;
  return at;
}

// keys[v] = (graph << bits) | degree key. A stable sort of these keys over ids
// 0..n-1 gives the (graph, degree, id) order.
// Of vertices v0 .. v0 + n - 1, the graphs from g0 on; keys and vals at the first's place.
__global__ void k_vertex_keys(const uint32_t* __restrict__ deg, uint64_t v0, uint64_t n, const uint64_t* voff,
                              uint32_t G, uint32_t g0, DegreeKey dk, uint32_t* __restrict__ keys,
                              uint32_t* __restrict__ vals) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, v = v0 + i;
  if (i >= n) return;
  const uint32_t g = G ? graph_of_vertex(voff, G, v) - g0 : 0u;
  const uint32_t d = degree_key(deg[v], dk);
  keys[i] = dk.bits >= 32 ? d : ((g << dk.bits) | d);
  vals[i] = (uint32_t)v;
}

// The words the row build starts from, set while vertices are ranked: w[r] for
// rank r (slots: the vertex's degree, its row's slot; else 0), then zeros up to
// `count` words.
struct RowWords {
  uint32_t* w;
  uint64_t count;
  bool slots;
  uint32_t* off;  // slots, up to kRankOneMax vertices: the slots' starts, also to w (else null)
};

// rank[id] = v0 + position, and the row words (from the first rank's on).
__global__ void k_rank_scatter(const uint32_t* __restrict__ sorted_keys, const uint32_t* __restrict__ sorted_ids,
                               uint64_t v0, uint64_t n, DegreeKey dk, uint32_t* __restrict__ rank,
                               const uint64_t* voff, uint32_t G, uint32_t* __restrict__ graph_of_rank,
                               const uint32_t* __restrict__ deg, RowWords rw) {
  const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (uint64_t i = n + r; i < rw.count; i += (uint64_t)gridDim.x * blockDim.x) rw.w[i] = 0;
  if (r >= n) return;
  const uint32_t v = sorted_ids[r];
  uint64_t at = r;
  if (hub_key(sorted_keys[r], dk))
    at = hub_place(r, n, [&](uint64_t p) { return sorted_keys[p]; }, [&](uint64_t p) { return deg[sorted_ids[p]]; });
  rank[v] = (uint32_t)(v0 + at);
  if (at < rw.count) rw.w[at] = rw.slots ? deg[v] : 0u;
  if (graph_of_rank) graph_of_rank[v0 + at] = graph_of_vertex(voff, G, v);
}

// The same ranks for one graph of at most kRankOneMax vertices, by one CTA:
// (key << 16) | id words in shared memory, two stable 8-bit passes (a warp a
// contiguous share, digits ranked by match): one launch in the place of eight.
constexpr uint32_t kRankOneMax = 16384;
constexpr uint32_t kRankThreads = 1024;
constexpr int kRankRounds = kRankOneMax / kRankThreads;
constexpr size_t kRankSmem = (2 * kRankOneMax + (kRankThreads / 32) * 256) * sizeof(uint32_t);
__global__ void __launch_bounds__(kRankThreads) k_rank_one(const uint32_t* __restrict__ deg, uint32_t n, DegreeKey dk,
                                                           uint32_t* __restrict__ rank, RowWords rw) {
  extern __shared__ uint32_t rank_sm[];
  __shared__ uint32_t s_sum[8];
  uint32_t* src = rank_sm;
  uint32_t* dst = rank_sm + kRankOneMax;
  const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  uint32_t* wcnt = rank_sm + 2 * kRankOneMax;  // [warp][digit]
  for (uint64_t i = n + (rw.off ? 1 : 0) + tid; i < rw.count; i += kRankThreads) rw.w[i] = 0;
  bool hubs = false;  // whether a key of this thread's, then any thread's, is a hub's
  for (uint32_t i = tid; i < n; i += kRankThreads) {
    const uint32_t key = degree_key(deg[i], dk);
    hubs |= hub_key(key, dk);
    src[i] = (key << 16) | i;
  }
  const uint32_t rounds = (n + kRankThreads - 1) / kRankThreads;  // of 32 a warp
  for (int shift = 16; shift < 32; shift += 8) {
    for (uint32_t i = tid; i < (kRankThreads / 32) * 256; i += kRankThreads) wcnt[i] = 0;
    __syncthreads();
    uint32_t v[kRankRounds], pos[kRankRounds];
#pragma unroll
    for (int r = 0; r < kRankRounds; ++r) {
      if (r >= (int)rounds) break;
      const uint32_t i = (w * rounds + r) * 32 + lane;
      v[r] = i < n ? src[i] : 0u;
      const uint32_t d = i < n ? (v[r] >> shift) & 255u : 256u;
      const uint32_t peers = __match_any_sync(kFull, d);
      const int leader = __ffs(peers) - 1;
      uint32_t b = 0;
      if (d < 256 && (int)lane == leader) {
        b = wcnt[w * 256 + d];
        wcnt[w * 256 + d] = b + __popc(peers);
      }
      pos[r] = __shfl_sync(kFull, b, leader) + __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
    }
    __syncthreads();
    // Digit d's keys of warp w go after all smaller digits and the digit's of
    // the warps before.
    uint32_t tot = 0;
    if (tid < 256)
      for (uint32_t q = 0; q < kRankThreads / 32; ++q) {
        const uint32_t c = wcnt[q * 256 + tid];
        wcnt[q * 256 + tid] = tot;
        tot += c;
      }
    const uint32_t incl = warp_inclusive_sum(tot);
    if (tid < 256 && lane == 31) s_sum[w] = incl;
    __syncthreads();
    if (tid < 256) {
      uint32_t before = incl - tot;
      for (uint32_t q = 0; q < w; ++q) before += s_sum[q];
      for (uint32_t q = 0; q < kRankThreads / 32; ++q) wcnt[q * 256 + tid] += before;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRankRounds; ++r) {
      if (r >= (int)rounds) break;
      const uint32_t i = (w * rounds + r) * 32 + lane;
      if (i < n) dst[wcnt[w * 256 + ((v[r] >> shift) & 255u)] + pos[r]] = v[r];
    }
    hubs = __syncthreads_or(hubs ? 1 : 0) != 0;
    uint32_t* t = src;
    src = dst;
    dst = t;
  }
  if (hubs) {
    for (uint32_t i = tid; i < n; i += kRankThreads) {
      uint32_t at = i;
      if (hub_key(src[i] >> 16, dk))
        at = (uint32_t)hub_place(i, n, [&](uint64_t p) { return src[p] >> 16; },
                                 [&](uint64_t p) { return deg[src[p] & 0xFFFFu]; });
      dst[at] = src[i];
    }
    __syncthreads();
    uint32_t* t = src;
    src = dst;
    dst = t;
  }
  if (!rw.off) {
    for (uint32_t i = tid; i < n; i += kRankThreads) {
      const uint32_t v = src[i] & 0xFFFFu;
      rank[v] = i;
      if (i < rw.count) rw.w[i] = rw.slots ? deg[v] : 0u;
    }
    return;
  }
  // Ranks, and the scan of the degrees in rank order.
  uint32_t d[kRankRounds], sum = 0;
#pragma unroll
  for (int r = 0; r < kRankRounds; ++r) {
    const uint32_t i = (w * rounds + r) * 32 + lane;
    d[r] = 0;
    if (r < (int)rounds && i < n) {
      const uint32_t v = src[i] & 0xFFFFu;
      rank[v] = i;
      d[r] = deg[v];
    }
    sum += d[r];
  }
  sum = __reduce_add_sync(kFull, sum);
  if (lane == 0) wcnt[w] = sum;
  __syncthreads();
  const uint32_t tot = wcnt[lane], incl = warp_inclusive_sum(tot);
  uint32_t at = __shfl_sync(kFull, incl, w) - sum;
#pragma unroll
  for (int r = 0; r < kRankRounds; ++r) {
    if (r >= (int)rounds) break;
    const uint32_t i = (w * rounds + r) * 32 + lane;
    const uint32_t id = warp_inclusive_sum(d[r]);
    if (i < n) rw.off[i] = rw.w[i] = at + id - d[r];
    at += __shfl_sync(kFull, id, 31);
  }
  const uint32_t all = __shfl_sync(kFull, incl, 31);
  if (tid == 0) rw.off[n] = rw.w[n] = all;
}

__global__ void k_identity_graph_of(uint64_t n, const uint64_t* voff, uint32_t G, uint32_t* __restrict__ graph_of_rank) {
  uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r < n) graph_of_rank[r] = graph_of_vertex(voff, G, r);
}

// ---- phase 2: rows in rank space --------------------------------------------
// Every entry is oriented from its lower-ranked endpoint lo to the higher hi.
// A counting sort by lo (the histogram is the oriented out-degree) places the
// hi's of each row together; each row is then sorted and deduplicated on its
// own (rows are short: with degree order none has more than sqrt(2E) neighbours), and
// one scan of the per-row (distinct neighbours, distinct 32-column blocks)
// pairs gives the CSR and bit-row offsets. The 48-bit global radix sort of
// (lo, hi) keys that this replaces took six passes over all entries.

// Oriented key (lo << 32) | hi, in rank space, of an entry's ids.
constexpr uint64_t kDropped = ~0ull;
__device__ __forceinline__ uint64_t orient(const uint32_t* __restrict__ rank, uint32_t a, uint32_t b) {
  const uint32_t ra = rank ? rank[a] : a, rb = rank ? rank[b] : b;
  return ((uint64_t)min(ra, rb) << 32) | max(ra, rb);
}

// keys[i] = (lo << 32) | hi of entry i (kDropped for a dropped entry), and
// cnt[lo] += 1. A CTA takes tiles of kTile entries, four a thread in flight.
constexpr int kAhead = 4;
constexpr uint32_t kTile = kThreads * kAhead;
__global__ void __launch_bounds__(kThreads) k_row_count(PrepInput in, const uint32_t* __restrict__ rank,
                                                        uint32_t* __restrict__ cnt, uint64_t* __restrict__ keys,
                                                        uint32_t tiles, unsigned int* err) {
  EntryReader rd(in, err);
  uint64_t c = (uint64_t)blockIdx.x * tiles * kTile;
  for (uint32_t t = 0; t < tiles && c < in.E; ++t, c += kTile) {
    uint64_t e[kAhead], key[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint64_t i = c + k * kThreads + threadIdx.x;
      e[k] = i < in.E ? in.entries[i] : 0ull;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint64_t i = c + k * kThreads + threadIdx.x;
      uint32_t a, b;
      key[k] = i < in.E && rd.ids(e[k], i, a, b) ? orient(rank, a, b) : kDropped;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint64_t i = c + k * kThreads + threadIdx.x;
      const uint32_t lo = (uint32_t)(key[k] >> 32);  // kNoId: dropped
      const KeyRun r = key_run(lo);
      if (r.head && lo != kNoId) atomicAdd(&cnt[lo], r.len);
      if (i < in.E) keys[i] = key[k];
    }
  }
}

// nbr[cur[lo]++] = hi (cur starts as the row offsets): the only random
// accesses are the cursors, which stay in L2, one update a run of equal lo. A
// CTA takes `tiles` tiles in a row, then on by the grid (fill_keys).
__global__ void __launch_bounds__(kThreads) k_row_fill(const uint64_t* __restrict__ keys, uint64_t E, uint32_t tiles,
                                                       uint32_t* __restrict__ cur, uint32_t* __restrict__ nbr) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t ahead = ((uint64_t)(gridDim.x - 1) * tiles + 1) * kTile;  // from the last of its tiles to the next first
  uint32_t t = 1;
  for (uint64_t c = (uint64_t)blockIdx.x * tiles * kTile; c < E; c += t == 1 ? ahead : kTile) {
    t = t == tiles ? 1 : t + 1;
    uint64_t key[kAhead];
    uint32_t at[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint64_t i = c + k * kThreads + threadIdx.x;
      key[k] = i < E ? keys[i] : kDropped;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint32_t lo = (uint32_t)(key[k] >> 32);
      const KeyRun r = key_run(lo);
      uint32_t base = 0;
      if (r.head && lo != kNoId) base = atomicAdd(&cur[lo], r.len);
      at[k] = __shfl_sync(kFull, base, r.first) + lane - r.first;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (key[k] != kDropped) nbr[at[k]] = (uint32_t)key[k];
  }
}

// Slot path (degree order): row r has a slot of deg(v) entries, v the vertex of
// rank r (every entry oriented from v is one of the deg(v) entries that touch
// v), so no pass counts the rows. Without a presort the entries go straight to
// their rows: no keys are written or read either, one pass in the place of
// k_row_count and k_row_fill (RMAT-20: 194 + 235 us, now 294).
// Entries [i0, i1).
__global__ void __launch_bounds__(kThreads) k_row_fill_entries(PrepInput in, uint64_t i0, uint64_t i1,
                                                               const uint32_t* __restrict__ rank,
                                                               uint32_t* __restrict__ cur, uint32_t* __restrict__ nbr,
                                                               uint32_t tiles, unsigned int* err) {
  EntryReader rd(in, err);
  const uint32_t lane = threadIdx.x & 31;
  uint64_t c = i0 + (uint64_t)blockIdx.x * tiles * kTile;
  for (uint32_t t = 0; t < tiles && c < i1; ++t, c += kTile) {
    uint64_t e[kAhead], key[kAhead];
    uint32_t at[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint64_t i = c + k * kThreads + threadIdx.x;
      e[k] = i < i1 ? in.entries[i] : 0ull;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint64_t i = c + k * kThreads + threadIdx.x;
      uint32_t a, b;
      key[k] = i < i1 && rd.ids(e[k], i, a, b) ? orient(rank, a, b) : kDropped;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
      const uint32_t lo = (uint32_t)(key[k] >> 32);
      const KeyRun r = key_run(lo);
      uint32_t base = 0;
      if (r.head && lo != kNoId) base = atomicAdd(&cur[lo], r.len);
      at[k] = __shfl_sync(kFull, base, r.first) + lane - r.first;
    }
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
      if (key[k] != kDropped) nbr[at[k]] = (uint32_t)key[k];
  }
}

// Slot path: keys[i - i0] = (lo - r0) << 32 | hi of entry i of [i0, i1) (kDropped for a
// dropped entry; r0: at most every lo), over the presort's radix tiles, each tile also counting its keys'
// presort digits (key >> shift) & 255 into hist (digit-major, as k_radix_hist
// leaves them): the keys and the presort's histogram in one pass.
__global__ void __launch_bounds__(kSortThreads) k_row_keys_hist(PrepInput in, uint64_t i0, uint64_t i1,
                                                                 const uint32_t* __restrict__ rank, uint32_t r0,
                                                                 uint64_t* __restrict__ keys, int shift,
                                                                 uint32_t tiles, uint32_t* __restrict__ hist,
                                                                 unsigned int* err) {
  __shared__ uint32_t h[256];
  h[threadIdx.x] = 0;
  __syncthreads();
  const uint64_t base = i0 + (uint64_t)blockIdx.x * kSortTile;
  EntryReader rd(in, err);
#pragma unroll 4
  for (int j = 0; j < kSortKeysPerThread; ++j) {
    const uint64_t i = base + (uint64_t)j * kSortThreads + threadIdx.x;
    uint32_t d = 256u;
    if (i < i1) {
      uint32_t a, b;
      const uint64_t key = rd.ids(in.entries[i], i, a, b) ? orient(rank, a, b) - ((uint64_t)r0 << 32) : kDropped;
      keys[i - i0] = key;
      d = (uint32_t)((key >> shift) & 255);
    }
    const uint32_t peers = __match_any_sync(kFull, d);
    if (d < 256 && (threadIdx.x & 31) == (uint32_t)(__ffs(peers) - 1)) atomicAdd(&h[d], (uint32_t)__popc(peers));
  }
  __syncthreads();
  hist[(uint64_t)threadIdx.x * tiles + blockIdx.x] = h[threadIdx.x];
}

constexpr uint32_t kPad = 0xFFFFFFFFu;  // sorts last; no vertex has this rank (n < 2^32)
constexpr uint32_t kShortRow = 32;       // longer rows go to the lists of k_sort_long
constexpr uint32_t kWarpSortMax = 1024;  // longer rows are sorted by a CTA
constexpr uint32_t kLongThreads = 256;
static_assert(kLongThreads == kScanThreads, "window_sort scans its CTA's threads");
constexpr uint32_t kBitWords = 11520;    // 45 KiB: a bitmap of 368,640 columns (four CTAs an SM)
constexpr uint32_t kCtaSortSmem = 8192;  // bitonic rows longer than this are sorted in global scratch

// Rows of more than kShortRow entries, listed by k_sort_rows: CTA rows (over
// kWarpSortMax) from the front of rows[], warp rows from its end (index n - i).
// The lists spread the long rows over the whole grid: under degree order the
// top row blocks hold 32 rows of hundreds of entries each, and one warp a
// block left them to a few warps (RMAT-20: the row sort 607 us, the emit 487).
struct LongRows {
  uint32_t* rows;   // n + 1
  uint32_t* count;  // kLongWords words, 8-byte aligned: CTA rows, warp rows, a SortSpace of scratch words taken by CTA rows
  __device__ __forceinline__ SortSpace* taken() const { return reinterpret_cast<SortSpace*>(count + 2); }
};
constexpr uint64_t kLongWords = 2 + sizeof(SortSpace) / sizeof(uint32_t);

// Bitonic sort of the warp's 32 K values, value r * 32 + lane in x[r] of
// lane lane, ascending.
template <int K>
__device__ __forceinline__ void warp_bitonic(uint32_t (&x)[K]) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (uint32_t k = 2; k <= 32u * K; k <<= 1) {
#pragma unroll
    for (uint32_t j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
        const uint32_t jr = j >> 5;
#pragma unroll
        for (int r = 0; r < K; ++r) {
          if ((r & jr) == 0) {
            const int p = r | (int)jr;
            const bool up = ((r * 32u + lane) & k) == 0;
            const uint32_t a = x[r], b = x[p];
            const bool sw = up ? a > b : a < b;
            x[r] = sw ? b : a;
            x[p] = sw ? a : b;
          }
        }
      } else {
#pragma unroll
        for (int r = 0; r < K; ++r) {
          const uint32_t y = __shfl_xor_sync(kFull, x[r], j);
          const bool up = ((r * 32u + lane) & k) == 0;
          const bool take_min = ((lane & j) == 0) == up;
          x[r] = take_min ? min(x[r], y) : max(x[r], y);
        }
      }
    }
  }
}

// Block spans up to which a warp sorts a row of at most 32 K entries through a
// bitmap of its columns instead of the network: the network's instructions (8 K
// to 220 K a warp) against about 55 a 32 words. Cliques' and top ranks' rows are
// dense in their span (k_sort_long on cliques 506 us; a count 1,986, now 1,792).
template <int K>
constexpr uint32_t kWarpBitWords = K == 2 ? 64 : K == 4 ? 224 : K == 8 ? 608 : 1440;

// Sorts row a[0, L) (L <= 32 K) with the warp, writes its distinct values
// back to a[0, u) and returns (u << 32) | distinct 32-column blocks. bm:
// kWarpBitWords<32> words of the warp.
template <int K>
__device__ __forceinline__ uint64_t warp_sort_row(uint32_t* __restrict__ a, uint32_t L, uint32_t* __restrict__ bm) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t x[K];
  uint32_t lo = kPad, hi = 0;
#pragma unroll
  for (int r = 0; r < K; ++r) {
    const uint32_t i = r * 32u + lane;
    x[r] = i < L ? a[i] : kPad;
    lo = min(lo, x[r] >> 5);
    if (i < L) hi = max(hi, x[r] >> 5);
  }
  lo = __reduce_min_sync(kFull, lo);
  hi = __reduce_max_sync(kFull, hi);
  const uint32_t words = hi - lo + 1;
  if (words <= kWarpBitWords<K>) {
    __syncwarp();
    for (uint32_t i = lane; i < words; i += 32) bm[i] = 0;
    __syncwarp();
#pragma unroll
    for (int r = 0; r < K; ++r)
      if (r * 32u + lane < L) atomicOr(&bm[(x[r] >> 5) - lo], 1u << (x[r] & 31));
    __syncwarp();
    uint32_t nu = 0, nbk = 0;
    for (uint32_t c = 0; c < words; c += 32) {
      uint32_t m = c + lane < words ? bm[c + lane] : 0u;
      const uint32_t n = __popc(m), incl = warp_inclusive_sum(n);
      uint32_t at = nu + incl - n;
      for (; m; m &= m - 1) a[at++] = ((lo + c + lane) << 5) + (uint32_t)__ffs(m) - 1u;
      nu += __shfl_sync(kFull, incl, 31);
      nbk += __popc(__ballot_sync(kFull, n > 0));
    }
    return ((uint64_t)nu << 32) | nbk;
  }
  warp_bitonic<K>(x);
  uint32_t nu = 0, nbk = 0;
  uint32_t last = kPad;  // value 32 r - 1, from the previous register row
#pragma unroll
  for (int r = 0; r < K; ++r) {
    uint32_t prev = __shfl_up_sync(kFull, x[r], 1);
    if (lane == 0) prev = last;
    last = __shfl_sync(kFull, x[r], 31);
    const bool first = r == 0 && lane == 0;
    const bool is_new = x[r] != kPad && (first || x[r] != prev);
    const bool new_blk = is_new && (first || (x[r] >> 5) != (prev >> 5));
    const uint32_t nb = __ballot_sync(kFull, is_new);
    if (is_new) a[nu + __popc(nb & ((1u << lane) - 1u))] = x[r];
    nu += __popc(nb);
    nbk += __popc(__ballot_sync(kFull, new_blk));
  }
  return ((uint64_t)nu << 32) | nbk;
}

// Rows of at most G entries (G = 8, 16 or 32), 32 / G at a time: lane group
// g (lanes [g G, g G + G)) sorts the g-th row of the pass with a bitonic
// network inside the group, then writes the row's distinct values and
// rows[u] = (distinct << 32) | blocks. pending: the warp lanes whose rows
// belong here; lane l's row starts at s_l with L_l entries; u = ubase + l.
template <uint32_t G>
__device__ __forceinline__ void sort_short_rows(uint32_t pending, uint32_t s_l, uint32_t L_l, uint32_t ubase,
                                                uint32_t* __restrict__ nbr, uint64_t* __restrict__ rows) {
  constexpr uint32_t R = 32 / G;
  const uint32_t lane = threadIdx.x & 31, grp = lane / G, gl = lane % G;
  const uint32_t gmask = G == 32 ? kFull : ((1u << G) - 1u) << (grp * G);
  while (pending) {
    int mine = -1;  // the warp lane whose row this group sorts in this pass
#pragma unroll
    for (uint32_t r = 0; r < R; ++r) {
      const int lr = pending ? __ffs(pending) - 1 : -1;
      if (r == grp) mine = lr;
      pending &= pending - 1;
    }
    const uint32_t src = mine >= 0 ? (uint32_t)mine : 0u;
    const uint32_t s = __shfl_sync(kFull, s_l, src), L = __shfl_sync(kFull, L_l, src);
    uint32_t x = mine >= 0 && gl < L ? nbr[s + gl] : kPad;
#pragma unroll
    for (uint32_t k = 2; k <= G; k <<= 1) {
#pragma unroll
      for (uint32_t j = k >> 1; j > 0; j >>= 1) {
        const uint32_t y = __shfl_xor_sync(kFull, x, j);
        const bool up = (gl & k) == 0;
        x = (((lane & j) == 0) == up) ? min(x, y) : max(x, y);
      }
    }
    const uint32_t prev = __shfl_up_sync(kFull, x, 1);
    const bool first = gl == 0;
    const bool is_new = x != kPad && (first || x != prev);
    const bool new_blk = is_new && (first || (x >> 5) != (prev >> 5));
    const uint32_t nb = __ballot_sync(kFull, is_new) & gmask;
    const uint32_t nbk = __popc(__ballot_sync(kFull, new_blk) & gmask);
    if (is_new) nbr[s + __popc(nb & ((1u << lane) - 1u))] = x;
    if (first && mine >= 0) rows[ubase + mine] = ((uint64_t)__popc(nb) << 32) | nbk;
  }
}

// One warp per `per` rows (at most 32): rows of up to 8 and 16 entries are
// sorted four and two at a time in lane groups, up to kShortRow one at a time;
// longer rows are listed for k_sort_long. Row u holds nbr[start[u], end[u]).
// rows[u] = (distinct << 32) | blocks, rows[n] = 0.
__global__ void __launch_bounds__(256)
    k_sort_rows(const uint32_t* __restrict__ start, const uint32_t* __restrict__ end, uint32_t n, uint32_t per,
                uint32_t* __restrict__ nbr, uint64_t* __restrict__ rows, LongRows lng) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nwarps = (gridDim.x * blockDim.x) >> 5;
  if (warp == 0 && lane == 0) rows[n] = 0;
  for (uint64_t ub = (uint64_t)warp * per; ub < n; ub += (uint64_t)nwarps * per) {
    const uint32_t ubase = (uint32_t)ub, u = ubase + lane;
    const bool here = lane < per && ub + lane < n;
    const uint32_t s_l = here ? start[u] : 0u, L_l = here ? end[u] - s_l : 0u;
    if (here && L_l == 0) rows[u] = 0;
    const uint32_t cta = __ballot_sync(kFull, L_l > kWarpSortMax);
    const uint32_t mid = __ballot_sync(kFull, L_l > kShortRow && L_l <= kWarpSortMax);
    if (cta | mid) {
      const uint32_t lt = (1u << lane) - 1u;
      uint32_t at = 0;
      if (lane == 0 && cta) at = atomicAdd(&lng.count[0], (uint32_t)__popc(cta));
      if (lane == 1 && mid) at = atomicAdd(&lng.count[1], (uint32_t)__popc(mid));
      const uint32_t c0 = __shfl_sync(kFull, at, 0), m0 = __shfl_sync(kFull, at, 1);
      if ((cta >> lane) & 1u) lng.rows[c0 + __popc(cta & lt)] = u;
      if ((mid >> lane) & 1u) lng.rows[n - (m0 + __popc(mid & lt))] = u;
    }
    sort_short_rows<8>(__ballot_sync(kFull, L_l >= 1 && L_l <= 8), s_l, L_l, ubase, nbr, rows);
    sort_short_rows<16>(__ballot_sync(kFull, L_l > 8 && L_l <= 16), s_l, L_l, ubase, nbr, rows);
    sort_short_rows<32>(__ballot_sync(kFull, L_l > 16 && L_l <= kShortRow), s_l, L_l, ubase, nbr, rows);
  }
}

// Sorts and deduplicates a CTA row through bitmaps of its columns: the window
// of kBitWords words from block w0 on gets a bit per entry in it, and its set
// bits, in order, are the row's distinct values (to out[nu...)). Returns
// (values << 32) | blocks of the window. A bit set costs one shared atomic an
// entry and a window kBitWords / 256 words a thread, where a bitonic sort of P
// values takes log2(P) (log2(P) + 1) / 2 barriers.
__device__ __forceinline__ uint64_t window_sort(const uint32_t* a, uint32_t L, uint32_t w0, uint32_t words, uint32_t* sm,
                                                uint32_t* out, uint32_t nu) {
  const uint32_t tid = threadIdx.x;
  for (uint32_t i = tid; i < words; i += kLongThreads) sm[i] = 0u;
  __syncthreads();
  for (uint32_t i = tid; i < L; i += kLongThreads) {
    const uint32_t x = a[i], d = (x >> 5) - w0;
    if (d < words) atomicOr(&sm[d], 1u << (x & 31));
  }
  __syncthreads();
  // Each thread takes an odd number of words in a row (odd: its neighbours'
  // words lie in other banks).
  const uint32_t per = ((words + kLongThreads - 1) / kLongThreads) | 1u;
  const uint32_t i0 = min(tid * per, words), i1 = min(i0 + per, words);
  uint32_t c = 0, nb = 0;
  for (uint32_t i = i0; i < i1; ++i) {
    const uint32_t m = sm[i];
    c += __popc(m);
    nb += m != 0u;
  }
  uint64_t tot;
  const uint64_t ex = block_exclusive_scan<uint64_t>(((uint64_t)c << 32) | nb, OpSum{}, 0ull, &tot);
  uint32_t at = nu + (uint32_t)(ex >> 32);
  for (uint32_t i = i0; i < i1; ++i)
    for (uint32_t m = sm[i]; m; m &= m - 1) out[at++] = ((w0 + i) << 5) + (uint32_t)__ffs(m) - 1u;
  __syncthreads();  // sm is cleared for the next window or row
  return tot;
}

// The listed long rows: a CTA per row of more than kWarpSortMax entries, then
// a warp per row in registers (bitonic). A CTA row is sorted through column
// bitmaps when its block span takes at most L / 1024 windows (one window for
// rows under 2,048), else bitonically, padded to a power of two P, in shared
// memory (P <= kCtaSortSmem) or in a slice of scratch (P < 2 L; scratch holds two
// words an entry), as rows of several windows are put together. Rows are
// taken in strides over the grid (the lists run roughly by rank, so every warp
// gets the same mix), the longest first.
__global__ void __launch_bounds__(kLongThreads, 4)
    k_sort_long(const uint32_t* __restrict__ start, const uint32_t* __restrict__ end, uint32_t n,
                uint32_t* __restrict__ nbr, uint32_t* __restrict__ scratch, uint64_t* __restrict__ rows, LongRows lng) {
  __shared__ uint32_t sm[kBitWords];
  __shared__ uint32_t wsum[2][kLongThreads / 32];
  const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  __shared__ SortSpace s_at;
  auto take = [&](uint32_t words) {  // the CTA's next slice of scratch
    if (tid == 0) s_at = atomicAdd(lng.taken(), (SortSpace)words);
    __syncthreads();
    const SortSpace at = s_at;
    __syncthreads();
    return at;
  };
  const uint32_t ncta = lng.count[0], nmid = lng.count[1];
  for (uint32_t bi = blockIdx.x; bi < ncta; bi += gridDim.x) {
    const uint32_t u = lng.rows[ncta - 1 - bi];
    const uint32_t s = start[u], L = end[u] - s;
    uint32_t lo = kFull, hi = 0;
    for (uint32_t i = tid; i < L; i += kLongThreads) {
      const uint32_t b = nbr[s + i] >> 5;
      lo = min(lo, b);
      hi = max(hi, b);
    }
    lo = __reduce_min_sync(kFull, lo);
    hi = __reduce_max_sync(kFull, hi);
    if (lane == 0) {
      wsum[0][w] = lo;
      wsum[1][w] = hi;
    }
    __syncthreads();
#pragma unroll
    for (uint32_t q = 0; q < kLongThreads / 32; ++q) {
      lo = min(lo, wsum[0][q]);
      hi = max(hi, wsum[1][q]);
    }
    __syncthreads();
    const uint32_t span = hi - lo + 1, windows = (span + kBitWords - 1) / kBitWords;
    uint64_t res = 0;
    if (windows == 1) {  // every entry is read before the first is overwritten
      res = window_sort(nbr + s, L, lo, span, sm, nbr + s, 0);
    } else if ((uint64_t)windows * 1024 <= L) {
      uint32_t* out = scratch + take(L);
      for (uint32_t k = 0; k < windows; ++k) {
        const uint32_t w0 = k * kBitWords;
        res += window_sort(nbr + s, L, lo + w0, min(kBitWords, span - w0), sm, out, (uint32_t)(res >> 32));
      }
      for (uint32_t i = tid; i < (uint32_t)(res >> 32); i += kLongThreads) nbr[s + i] = out[i];
    } else {
      uint32_t P = 1;
      while (P < L) P <<= 1;
      uint32_t* a = P <= kCtaSortSmem ? sm : scratch + take(P);
      for (uint32_t i = tid; i < P; i += kLongThreads) a[i] = i < L ? nbr[s + i] : kPad;
      __syncthreads();
      for (uint32_t k = 2; k <= P; k <<= 1) {
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
          for (uint32_t t = tid; t < P / 2; t += kLongThreads) {
            const uint32_t i = ((t & ~(j - 1)) << 1) | (t & (j - 1));  // pairs (i, i + j); j is a power of 2
            const bool up = (i & k) == 0;
            const uint32_t x = a[i], y = a[i + j];
            if (up ? x > y : x < y) {
              a[i] = y;
              a[i + j] = x;
            }
          }
          __syncthreads();
        }
      }
      // Distinct values in order: per tile of kLongThreads values, a
      // block-wide count of the new ones places them.
      uint32_t nu = 0, nbk = 0;
      for (uint32_t base = 0; base < L; base += kLongThreads) {
        const uint32_t i = base + tid;
        const uint32_t x = i < L ? a[i] : kPad;
        const uint32_t p = i > 0 && i < L ? a[i - 1] : kPad;
        const bool is_new = x != kPad && (i == 0 || x != p);
        const bool new_blk = is_new && (i == 0 || (x >> 5) != (p >> 5));
        const uint32_t bn = __ballot_sync(kFull, is_new), bb = __ballot_sync(kFull, new_blk);
        if (lane == 0) {
          wsum[0][w] = __popc(bn);
          wsum[1][w] = __popc(bb);
        }
        __syncthreads();
        uint32_t before = 0, tile_u = 0, tile_b = 0;
        for (uint32_t q = 0; q < kLongThreads / 32; ++q) {
          if (q < w) before += wsum[0][q];
          tile_u += wsum[0][q];
          tile_b += wsum[1][q];
        }
        if (is_new) nbr[s + nu + before + __popc(bn & ((1u << lane) - 1u))] = x;
        nu += tile_u;
        nbk += tile_b;
        __syncthreads();  // a[] reads of this tile and wsum before the next tile
      }
      res = ((uint64_t)nu << 32) | nbk;
    }
    if (tid == 0) rows[u] = res;
  }
  __syncthreads();  // the warps' slices of sm follow the CTA rows' use of it
  uint32_t* bm = sm + w * (kBitWords / (kLongThreads / 32));
  static_assert(kBitWords / (kLongThreads / 32) >= kWarpBitWords<32>, "a warp's slice holds its bitmap");
  const uint32_t warp = blockIdx.x * (kLongThreads / 32) + w, nwarps = gridDim.x * (kLongThreads / 32);
  for (uint32_t i = warp; i < nmid; i += nwarps) {
    const uint32_t u = lng.rows[n - (nmid - 1 - i)];
    const uint32_t s = start[u], L = end[u] - s;
    uint32_t* a = nbr + s;
    uint64_t res;
    if (L <= 64)
      res = warp_sort_row<2>(a, L, bm);
    else if (L <= 128)
      res = warp_sort_row<4>(a, L, bm);
    else if (L <= 256)
      res = warp_sort_row<8>(a, L, bm);
    else if (L <= 512)
      res = warp_sort_row<16>(a, L, bm);
    else
      res = warp_sort_row<32>(a, L, bm);
    if (lane == 0) rows[u] = res;
  }
}

// The first u in [0, n] with rp_row(rp[u]) - begin + u >= t: rows and positions
// counted together, so that a run of empty rows is work like any other. The
// whole warp searches, 32 probes a step.
__device__ __forceinline__ uint64_t first_row_at(const uint64_t* __restrict__ rp, uint32_t n, uint32_t begin,
                                                 uint64_t t) {
  const uint32_t lane = threadIdx.x & 31;
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    const uint64_t step = (hi - lo + 31) / 32, u = lo + (lane + 1) * step - 1;
    const uint32_t below = __popc(__ballot_sync(kFull, u < hi && rp_row(rp[u]) - begin + u < t));
    const uint64_t next = lo + (below + 1) * step - 1;
    lo = min(hi, lo + below * step);
    if (below < 32) hi = min(hi, next);
  }
  return lo;
}

// Emits CSR positions [ps, pe): col[p] and the positions' bit-row entries from
// bent[b] on, one warp, 32 positions a step with the values of the next
// kEmitAhead steps loaded before they are used. starts(c): bit l set iff a row
// starts at position c + l (one does at ps); source(p, i): the index in nbr of
// position p, in the i-th row that starts in the range. A bit-row entry is
// written by the lane of its block's last value: the mask is a segmented OR,
// and a block cut by a step carries its partial mask over.
constexpr int kEmitAhead = 3;
template <class Starts, class Source>
__device__ __forceinline__ void emit_span(uint32_t ps, uint32_t pe, uint32_t b, const Starts& starts,
                                          const Source& source, const uint32_t* __restrict__ nbr,
                                          uint32_t* __restrict__ col, uint64_t* __restrict__ bent) {
  const uint32_t lane = threadIdx.x & 31, le = kFull >> (31 - lane);
  uint32_t m[kEmitAhead + 1], x[kEmitAhead + 1];  // row starts and values of this step and the next ones
  uint32_t at = 0, row = kFull;                   // positions loaded; rows started in them, less one
  const uint32_t len = pe - ps;
  auto load = [&](int k) {
    m[k] = 0;
    x[k] = kPad;
    if (at < len) {
      m[k] = starts(ps + at);
      const uint32_t i = row + __popc(m[k] & le);
      if (lane < len - at) x[k] = nbr[source(ps + at + lane, i)];
      row += __popc(m[k]);
      at += min(32u, len - at);
    }
  };
#pragma unroll
  for (int k = 0; k <= kEmitAhead; ++k) load(k);
  uint32_t last = kPad >> 5, carry = 0;
  for (uint32_t left = len, c = ps;; left -= 32, c += 32) {
    const bool in = lane < left, more = left > 32;
    const uint32_t blk = x[0] >> 5;
    uint32_t prev = __shfl_up_sync(kFull, blk, 1);
    if (lane == 0) prev = last;
    const uint32_t heads = __ballot_sync(kFull, in && (((m[0] >> lane) & 1u) || blk != prev));
    last = __shfl_sync(kFull, blk, 31);
    const bool next_head = !more || (m[1] & 1u) || (__shfl_sync(kFull, x[1], 0) >> 5) != last;
    const uint32_t own = heads & le, first = own ? 31 - __clz(own) : 0u;  // first lane of the block here
    uint32_t bits = in ? 1u << (x[0] & 31) : 0u;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(kFull, bits, o);
      if (lane >= first + o) bits |= y;
    }
    if (!own) bits |= carry;
    const bool end = in && (lane == 31 ? next_head : (lane + 1 >= left || ((heads >> (lane + 1)) & 1u)));
    if (in) col[c + lane] = x[0];
    if (end) bent[b + __popc(own) - 1] = ((uint64_t)blk << 32) | bits;
    if (!more) break;
    carry = __shfl_sync(kFull, bits, 31);
    b += __popc(heads);
#pragma unroll
    for (int k = 0; k < kEmitAhead; ++k) {
      m[k] = m[k + 1];
      x[k] = x[k + 1];
    }
    load(kEmitAhead);
  }
}

// The rows' distinct sorted values (the front of each row's nbr slice, from
// off[u]) to col, and their bit-row entries (block << 32 | mask) to bent, each
// written once; their totals to stats (may be null). Listed CTA rows of more than kWarpSortMax values are emitted
// by a CTA, each warp an eighth of the row from the first block that starts in
// it. All others are shared out by rows and CSR positions together (`chunk` of
// them a warp): a warp takes the rows that start in its share, 32 at a time, and
// walks their positions flat, so its work is the values it writes, whatever the
// rows' lengths. One warp per 32
// rows, a row at a time, left the top ranks to a few warps (RMAT-20: 487 us, now
// 139; RMAT-17 by id: 1,881, now 157; planted partition, even rows: 257, now 280).
__global__ void __launch_bounds__(256) k_emit_rows(const uint32_t* __restrict__ off, const uint32_t* __restrict__ nbr,
                                                   const uint64_t* __restrict__ rp, uint32_t n, uint32_t chunk,
                                                   LongRows lng, uint32_t* __restrict__ col,
                                                   uint64_t* __restrict__ bent, DeviceStats* stats) {
  __shared__ uint32_t s_delta[8][32];
  __shared__ uint32_t s_head[9], s_cnt[8];
  const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (stats && blockIdx.x == 0 && threadIdx.x == 0) {
    stats->edges = rp_row(rp[n]);
    stats->blocks = rp_blk(rp[n]);
  }
  for (uint32_t bi = blockIdx.x, ncta = lng.count[0]; bi < ncta; bi += gridDim.x) {
    const uint32_t u = lng.rows[ncta - 1 - bi];
    const uint64_t r0 = rp[u], r1 = rp[u + 1];
    const uint32_t p0 = rp_row(r0), nu = rp_row(r1) - p0;
    if (nu <= kWarpSortMax) continue;  // duplicates: walked flat below
    const uint32_t* a = nbr + off[u];
    auto new_block = [&](uint32_t i) { return i < nu && (i == 0 || (a[i] >> 5) != (a[i - 1] >> 5)); };
    // The warp's first block head at or after its share (a block has at most 32 values).
    const uint32_t s0 = (uint32_t)((uint64_t)nu * w / 8);
    const uint32_t hm = __ballot_sync(kFull, new_block(s0 + lane));
    if (lane == 0) {
      s_head[w] = hm ? s0 + (uint32_t)__ffs(hm) - 1u : nu;
      if (w == 0) s_head[8] = nu;
    }
    __syncthreads();
    const uint32_t i0 = s_head[w], i1 = s_head[w + 1];
    uint32_t c = 0;
    for (uint32_t i = i0; i < i1; i += 32) c += __popc(__ballot_sync(kFull, i + lane < i1 && new_block(i + lane)));
    if (lane == 0) s_cnt[w] = c;
    __syncthreads();
    uint32_t b = rp_blk(r0);
    for (uint32_t q = 0; q < w; ++q) b += s_cnt[q];
    if (i0 < i1)
      emit_span(p0 + i0, p0 + i1, b, [&](uint32_t p) { return p == p0 + i0 ? 1u : 0u; },
                [&](uint32_t p, uint32_t) { return off[u] + (p - p0); }, nbr, col, bent);
    __syncthreads();  // s_head and s_cnt are rewritten for the next row
  }
  const uint32_t begin = rp_row(rp[0]);
  const uint64_t total = (uint64_t)(rp_row(rp[n]) - begin) + n;
  const uint32_t warp = blockIdx.x * 8 + w, nwarps = gridDim.x * 8;
  for (uint64_t t = (uint64_t)warp * chunk; t < total; t += (uint64_t)nwarps * chunk) {
    for (uint64_t ub = first_row_at(rp, n, begin, t);; ub += 32) {
      const uint64_t ul = ub + lane;
      const uint32_t u = (uint32_t)ul;
      uint64_t r0 = 0, r1 = 0;
      bool here = ul < n;
      if (here) {
        r0 = rp[u];
        r1 = rp[u + 1];
        here = rp_row(r0) - begin + ul < t + chunk;
      }
      const uint32_t hm = __ballot_sync(kFull, here);
      if (!hm) break;
      const uint32_t p = rp_row(r0), nu = here ? rp_row(r1) - p : 0u;
      const uint32_t bigs = __ballot_sync(kFull, nu > kWarpSortMax);
      // Runs of rows between CTA rows.
      for (uint32_t todo = hm; todo;) {
        const uint32_t first = (uint32_t)__ffs(todo) - 1u;
        const uint32_t stop = bigs & todo;
        const uint32_t run = stop ? todo & ((stop & (0u - stop)) - 1u) : todo;
        todo = stop ? todo & ~((stop & (0u - stop)) | run) : 0u;
        if (!run) continue;
        const bool mine = ((run >> lane) & 1u) && nu > 0;
        const uint32_t rows = __ballot_sync(kFull, mine);
        if (!rows) continue;
        __syncwarp();
        if (mine) s_delta[w][__popc(rows & ((1u << lane) - 1u))] = off[u] - p;
        __syncwarp();
        const uint32_t ps = __shfl_sync(kFull, p, first), tail = 31u - (uint32_t)__clz(run);
        const uint32_t pe = __shfl_sync(kFull, rp_row(r1), tail), b = __shfl_sync(kFull, rp_blk(r0), first);
        emit_span(ps, pe, b,
                  [&](uint32_t c) { return __reduce_or_sync(kFull, mine && p - c < 32u ? 1u << (p - c) : 0u); },
                  [&](uint32_t q, uint32_t i) { return q + s_delta[w][i]; }, nbr, col, bent);
      }
      if (hm != kFull) break;
    }
  }
}

// Rows and CSR positions a warp of k_emit_rows takes, for at most E of them:
// enough warps to fill the chip several times over, up to 1,024 a search.
uint32_t emit_chunk(uint64_t E) {
  const uint64_t c = ceil_div<uint64_t>(E, 148ull * 64);
  return (uint32_t)std::min<uint64_t>(1024, std::max<uint64_t>(64, (c + 31) & ~31ull));
}

unsigned emit_grid(uint64_t E) {
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(ceil_div<uint64_t>(E, 8ull * emit_chunk(E)), 148ull * 32));
}

// Rows a warp of k_sort_rows takes: 32 once that fills the chip, fewer below.
uint32_t sort_rows_per_warp(uint64_t n) {
  return (uint32_t)std::min<uint64_t>(32, std::max<uint64_t>(4, ceil_div<uint64_t>(n, 148ull * 64)));
}

unsigned sort_grid(uint64_t n) {
  return (unsigned)std::max<uint64_t>(
      1, std::min<uint64_t>(ceil_div<uint64_t>(n, 8ull * sort_rows_per_warp(n)), 148ull * 32));
}

// Row u = nbr[start[u], end[u]) sorted and deduplicated in place for u < n,
// rows[u] = (distinct << 32) | blocks; E bounds the entries of all rows. The
// list lengths in lng start at 0.
void sort_rows(const uint32_t* start, const uint32_t* end, uint32_t n, uint64_t E, uint32_t* nbr, uint32_t* scratch,
               uint64_t* rows, const LongRows& lng, cudaStream_t st) {
  k_sort_rows<<<sort_grid(n), kThreads, 0, st>>>(start, end, n, sort_rows_per_warp(n), nbr, rows, lng);
  TB_LAUNCH_CHECK();
  if (E > kShortRow) {
    k_sort_long<<<(unsigned)std::min<uint64_t>(148 * 4, ceil_div<uint64_t>(E, kShortRow)), kLongThreads, 0, st>>>(
        start, end, n, nbr, scratch, rows, lng);
    TB_LAUNCH_CHECK();
  }
}

__global__ void k_finalize(const uint64_t* __restrict__ rp, uint64_t n, DeviceStats* stats) {
  const uint64_t tot = rp[n];
  stats->edges = tot >> 32;
  stats->blocks = tot & 0xffffffffull;
}

// Range-relative row starts of rows [s, s + z]: off[k] = cursor[k] =
// row_start[s + k] - row_start[s].
__global__ void k_range_starts(const uint64_t* __restrict__ row_start, uint32_t s, uint32_t z,
                               uint32_t* __restrict__ off, uint32_t* __restrict__ cursor) {
  const uint64_t base = row_start[s];
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k <= z; k += gridDim.x * blockDim.x) {
    const uint32_t v = (uint32_t)(row_start[s + k] - base);
    off[k] = v;
    cursor[k] = v;
  }
}

// The range's keys into their rows' slots (any order within a row).
__global__ void k_range_fill(const uint64_t* __restrict__ keys, uint64_t cnt, uint32_t s, uint32_t z,
                             const uint32_t* __restrict__ off, uint32_t* __restrict__ cursor,
                             uint32_t* __restrict__ nbr, unsigned int* err) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < cnt; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t key = keys[i];
    const uint32_t r = (uint32_t)(key >> 32) - s;
    if (r >= z) {
      atomicOr(err, kErrInput);
      continue;
    }
    const uint32_t pos = atomicAdd(&cursor[r], 1u);
    if (pos >= off[r + 1]) {
      atomicOr(err, kErrInput);
      continue;
    }
    nbr[pos] = (uint32_t)key;
  }
}

// Every row of the range got exactly its counted entries (a row short of them
// would hold stale slots: the entries changed between passes).
__global__ void k_range_check(const uint32_t* __restrict__ off, const uint32_t* __restrict__ cursor, uint32_t z,
                              unsigned int* err) {
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < z; k += gridDim.x * blockDim.x)
    if (cursor[k] != off[k + 1]) atomicOr(err, kErrInput);
}

// rp[k] += *carry, k < count: the range's prefix continues the ranges before.
__global__ void k_range_carry(uint64_t* __restrict__ rp, uint32_t count, const uint64_t* __restrict__ carry) {
  const uint64_t c = *carry;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) rp[k] += c;
}

bool degree_slots(const PrepInput& in);

// Batches under degree order are built in chunks of whole graphs (build_batch).
bool batch_chunks(const PrepInput& in) { return in.G && in.n > 0 && degree_slots(in); }

bool takes_presort(const PrepInput& in) {
  return in.E >= kPresortMinEntries && in.n > 256 && !batch_chunks(in);
}

uint64_t entry_tiles(uint64_t E) { return std::max<uint64_t>(1, E / (148ull * 64 * kTile)); }  // a CTA's

// Pieces a host input of E entries is copied in, of at least `least` entries each.
uint64_t upload_pieces(uint64_t E, uint64_t least) {
  return std::max<uint64_t>(1, std::min<uint64_t>(kUploadChunks, E / least));
}

// Queues the copy of host entries [i0, i1).
void upload_entries(const PrepInput& in, uint64_t i0, uint64_t i1, cudaStream_t st) {
  const HostUpload& up = in.upload;
  uint64_t* to = const_cast<uint64_t*>(in.entries) + i0;
  const uint64_t* from = up.host + i0;
  const size_t bytes = (i1 - i0) * sizeof(uint64_t);
  if (up.stage)
    up.stage(up.stage_ctx, to, from, bytes, st);
  else
    TB_CUDA(cudaMemcpyAsync(to, from, bytes, cudaMemcpyHostToDevice, st));
}

// Inputs that presort group their keys by one radix pass on the top 8 bits of
// lo into 256 ranges of rows, so the fill's cursors and stores at any time stay
// in one range's few MB of L2 instead of scattering over all rows.
int presort_digit(uint64_t rows) { return 32 + bits_for(rows) - 8; }

// Presorted keys of sparse rows are taken in launch order, four tiles a CTA, so
// that the CTAs at work stay together in the keys and their stores in a few ranges
// of rows (RMAT-24, 16 entries a vertex, 4.9 ms striding, now 3.8; RMAT-23
// preprocessing 13.7 and 13.8, Erdos-Renyi of 2^27 entries on 2^23 vertices 10.0 and
// 9.8). With more entries a row the CTAs would meet on its cursor and stride through
// all keys instead (preprocessing striding and together: RMAT-22 of 32 entries a vertex
// 12.0 and 12.2, RMAT-20 of 128 10.8 and 12.0, RMAT-16 of 2,048 8.1 and 16.3).
void fill_keys(const uint64_t* keys, uint64_t E, uint64_t rows, bool presorted, uint32_t* cur, uint32_t* nbr,
               cudaStream_t st) {
  const bool together = presorted && E < 32 * rows;
  const uint64_t tiles = together ? 4 : 1, most = together ? ~0ull : 148ull * 64;
  k_row_fill<<<(unsigned)std::min<uint64_t>(ceil_div<uint64_t>(E, tiles * kTile), most), kThreads, 0, st>>>(
      keys, E, (uint32_t)tiles, cur, nbr);
  TB_LAUNCH_CHECK();
}

void fill_entries(const PrepInput& in, uint64_t i0, uint64_t i1, const uint32_t* rank, uint32_t* cur, uint32_t* nbr,
                  unsigned int* err, cudaStream_t st) {
  if (i0 >= i1) return;
  const uint64_t per = entry_tiles(i1 - i0);
  k_row_fill_entries<<<(unsigned)ceil_div<uint64_t>(i1 - i0, per * kTile), kThreads, 0, st>>>(in, i0, i1, rank, cur, nbr,
                                                                                             (uint32_t)per, err);
  TB_LAUNCH_CHECK();
}

// The keys of entries [i0, i1), presorted, into the rows from rank r0 on, z of them, in slots. The buffers hold i1 - i0
// keys.
void fill_presorted(const PrepInput& in, uint64_t i0, uint64_t i1, const uint32_t* rank, uint64_t r0, uint64_t z,
                    uint64_t* keys, uint64_t* keys_alt, const RadixTemp& tmp, uint32_t* cur, uint32_t* nbr,
                    unsigned int* err, cudaStream_t st) {
  const uint64_t E = i1 - i0, tiles = ceil_div<uint64_t>(E, kSortTile);
  const int top = presort_digit(z);
  k_row_keys_hist<<<(unsigned)tiles, kSortThreads, 0, st>>>(in, i0, i1, rank, (uint32_t)r0, keys, top, (uint32_t)tiles,
                                                             tmp.hist, err);
  TB_LAUNCH_CHECK();
  const uint64_t* sorted =
      radix_sort<uint64_t, NoVal, false>(keys, keys_alt, nullptr, nullptr, E, top + 8, tmp, st, nullptr, top, true);
  fill_keys(sorted, E, z, true, cur + r0, nbr, st);
}

// Rows in degree-sized slots (2E entries in all, u32 offsets): no per-row
// atomics to count them, and, with the presort, its histogram counted while the
// keys are written (RMAT-24: row counts 2.9 ms and the histogram 1.0 ms, for 4
// bytes an entry more). Not where the layout has to stay small.
bool degree_slots(const PrepInput& in) {
  return in.order == TRIBIT_ORDER_DEGREE && !in.compact && 2 * in.E < 0xFFFFFFFFull;
}

// The one-CTA ranking scans the slot sizes too.
bool rank_scans(const PrepInput& in) { return degree_slots(in) && !in.G && in.n > 0 && in.n <= kRankOneMax; }

// cnt: n + 1 words, row counters at 0 or, on the slot path, slot sizes (then the
// fill cursors, which end at the rows' ends); nbig: kLongWords words at 0.
// off: n + 1 words, the row starts (set already where rank_scans(in)).
void run_rows(Arena& ar, const PrepInput& in, const uint32_t* rank, uint32_t* cnt, uint32_t* off, uint32_t* nbig,
              cudaStream_t st, Prepared* out, DeviceStats* stats, uint64_t* rp) {
  const uint64_t E = in.E, n = in.n;
  const bool presort = takes_presort(in), slots = degree_slots(in);
  const uint64_t cap = slots ? 2 * E : E;  // nbr entries
  uint32_t* otmp = take_scan_temp<uint32_t>(ar, n + 1);
  uint64_t* rtmp = take_scan_temp<uint64_t>(ar, n + 1);
  uint32_t* big = ar.take<uint32_t>(n + 1);
  uint32_t* nbr = ar.take<uint32_t>(cap ? cap : 1);
  // The oriented keys, then long rows' sort space.
  uint32_t* scratch = ar.take<uint32_t>(2 * E + 2);
  uint64_t* keys_alt = presort ? ar.take<uint64_t>(E) : nullptr;
  RadixTemp ktmp;
  if (presort) ktmp = take_radix_temp(ar, E);
  uint32_t* col = ar.take<uint32_t>(E + 4);   // + 4: 16-byte quad loads may read three ids past the end
  uint64_t* bent = ar.take<uint64_t>(E + 2);  // + 2: 16-byte pair loads may read one entry past the end
  out->view.col = col;
  out->view.bent = bent;
  if (ar.measuring()) return;

  const LongRows lng{big, nbig};
  uint64_t* keys = reinterpret_cast<uint64_t*>(scratch);
  const uint64_t per = entry_tiles(E);
  const unsigned entry_grid = (unsigned)ceil_div<uint64_t>(E, per * kTile);
  if (!slots && E > 0) {
    k_row_count<<<entry_grid, kThreads, 0, st>>>(in, rank, cnt, keys, (uint32_t)per, &stats->err);
    TB_LAUNCH_CHECK();
  }
  if (!rank_scans(in)) device_scan<uint32_t, OpSum>(cnt, off, n + 1, true, OpSum{}, 0u, otmp, st, cnt);
  if (slots && presort) {
    fill_presorted(in, 0, E, rank, 0, n, keys, keys_alt, ktmp, cnt, nbr, &stats->err, st);
  } else if (slots) {
    fill_entries(in, 0, E, rank, cnt, nbr, &stats->err, st);
  } else if (E > 0) {
    const int top = presort_digit(n);
    const uint64_t* sorted = keys;
    if (presort)
      sorted = radix_sort<uint64_t, NoVal, false>(keys, keys_alt, nullptr, nullptr, E, top + 8, ktmp, st, nullptr, top);
    fill_keys(sorted, E, n, presort && slots, cnt, nbr, st);
  }
  // Row u: nbr[off[u], cnt[u]) (with no entries every row is empty: 0, 0).
  sort_rows(off, cnt, (uint32_t)n, E, nbr, scratch, rp, lng, st);
  device_scan<uint64_t, OpSum>(rp, rp, n + 1, true, OpSum{}, 0ull, rtmp, st);
  k_emit_rows<<<emit_grid(E + n), kThreads, 0, st>>>(off, nbr, rp, (uint32_t)n, emit_chunk(E + n), lng, col, bent, stats);
  TB_LAUNCH_CHECK();
}

}  // namespace

RowRangeBuffers take_row_range_buffers(Arena& ar, uint64_t n, uint64_t cap) {
  RowRangeBuffers b;
  b.keys = ar.take<uint64_t>(cap + 1);
  b.scratch = reinterpret_cast<uint32_t*>(b.keys);
  b.nbr = ar.take<uint32_t>(cap ? cap : 1);
  b.off = ar.take<uint32_t>(n + 1);
  b.cursor = ar.take<uint32_t>(n + 1);
  b.big = ar.take<uint32_t>(n + 1);
  b.nbig = ar.take<uint32_t>(kLongWords);
  b.carry = ar.take<uint64_t>(1);
  b.scan_tmp = take_scan_temp<uint64_t>(ar, n + 1);
  return b;
}

void begin_row_range(const RowRangeBuffers& b, const uint64_t* row_start, uint32_t s, uint32_t z, uint64_t* rp,
                     cudaStream_t st) {
  if (z == 0) return;
  // The ranges before this one left rp[s] = the prefix at row s, which the
  // row sort overwrites.
  if (s == 0)
    TB_CUDA(cudaMemsetAsync(b.carry, 0, sizeof(uint64_t), st));
  else
    TB_CUDA(cudaMemcpyAsync(b.carry, rp + s, sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
  k_range_starts<<<grid_for((uint64_t)z + 1), kThreads, 0, st>>>(row_start, s, z, b.off, b.cursor);
  TB_LAUNCH_CHECK();
}

void finish_row_range(const RowRangeBuffers& b, uint32_t s, uint32_t z, uint64_t cnt, uint64_t* rp, uint32_t* col,
                      uint64_t* bent, unsigned int* err, cudaStream_t st) {
  if (z == 0) return;
  k_range_check<<<grid_for(z), kThreads, 0, st>>>(b.off, b.cursor, z, err);
  TB_LAUNCH_CHECK();
  const LongRows lng{b.big, b.nbig};
  TB_CUDA(cudaMemsetAsync(b.nbig, 0, kLongWords * sizeof(uint32_t), st));
  sort_rows(b.off, b.off + 1, z, cnt, b.nbr, b.scratch, rp + s, lng, st);
  device_scan<uint64_t, OpSum>(rp + s, rp + s, (uint64_t)z + 1, true, OpSum{}, 0ull, b.scan_tmp, st);
  k_range_carry<<<grid_for((uint64_t)z + 1), kThreads, 0, st>>>(rp + s, z + 1, b.carry);
  TB_LAUNCH_CHECK();
  k_emit_rows<<<emit_grid(cnt + z), kThreads, 0, st>>>(b.off, b.nbr, rp + s, z, emit_chunk(cnt + z), lng, col, bent, nullptr);
  TB_LAUNCH_CHECK();
}

void build_row_range(const RowRangeBuffers& b, const uint64_t* row_start, uint32_t s, uint32_t z, uint64_t cnt,
                     uint64_t* rp, uint32_t* col, uint64_t* bent, unsigned int* err, cudaStream_t st) {
  if (z == 0) return;
  begin_row_range(b, row_start, s, z, rp, st);
  if (cnt > 0) {
    k_range_fill<<<grid_for(cnt, 8), kThreads, 0, st>>>(b.keys, cnt, s, z, b.off, b.cursor, b.nbr, err);
    TB_LAUNCH_CHECK();
  }
  finish_row_range(b, s, z, cnt, rp, col, bent, err, st);
}

void finalize_rows(const uint64_t* rp, uint64_t n, DeviceStats* stats, cudaStream_t st) {
  k_finalize<<<1, 1, 0, st>>>(rp, n, stats);
  TB_LAUNCH_CHECK();
}

RankBuffers take_rank_buffers(Arena& ar, uint64_t n) {
  RankBuffers b;
  b.vk = ar.take<uint32_t>(n ? n : 1);
  b.vk2 = ar.take<uint32_t>(n ? n : 1);
  b.vv = ar.take<uint32_t>(n ? n : 1);
  b.vv2 = ar.take<uint32_t>(n ? n : 1);
  b.tmp = take_radix_temp(ar, n);
  return b;
}

namespace {

// Ranks of n vertices from v0 on, graphs [g0, g1) of a batch (a single graph: G
// = 0), from their degrees over E entries, and the row words. The buffers as take_rank_buffers
// takes them.
void rank_by_degree(const uint32_t* deg, uint64_t E, uint64_t v0, uint64_t n, const uint64_t* voff, uint32_t G,
                    uint32_t g0, uint32_t g1, const RankBuffers& b, uint32_t* rank, uint32_t* graph_of_rank, const RowWords& rw,
                    cudaStream_t st) {
  if (!G && n <= kRankOneMax) {
    once_per_device<3>(
        [] { TB_CUDA(cudaFuncSetAttribute(k_rank_one, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kRankSmem)); });
    k_rank_one<<<1, kRankThreads, kRankSmem, st>>>(deg, (uint32_t)n, degree_key_of(kDegreeBits, E), rank, rw);
    TB_LAUNCH_CHECK();
    return;
  }
  // Whole radix passes over the graph bits and as many degree bits as tell all degrees apart (or as there are).
  const int gbits = G ? bits_for((uint64_t)(g1 - g0)) : 0;
  int total = 16;
  while (total < 32 && !told_apart(total - gbits, E)) total += 8;
  const DegreeKey dk = degree_key_of(total - gbits, E);
  k_vertex_keys<<<grid_for(n), kThreads, 0, st>>>(deg, v0, n, voff, G, g0, dk, b.vk, b.vv);
  TB_LAUNCH_CHECK();
  uint32_t* sorted_ids = nullptr;
  const uint32_t* sorted_keys =
      radix_sort<uint32_t, uint32_t, true>(b.vk, b.vk2, b.vv, b.vv2, n, total, b.tmp, st, &sorted_ids);
  k_rank_scatter<<<grid_for(n), kThreads, 0, st>>>(sorted_keys, sorted_ids, v0, n, dk, rank, voff, G, graph_of_rank, deg,
                                                   rw);
  TB_LAUNCH_CHECK();
}

}  // namespace

namespace {

// ---- batches -----------------------------------------------------------------
// The graphs of a batch share no vertex, and ranks are grouped by graph, so the
// entries, vertices, ranks, rows and row offsets of consecutive graphs are
// consecutive: a chunk of graphs is ranked and its rows built as soon as its
// entries have landed, while the next chunk is copied. (All graphs built after
// the last entry had landed: 512 graphs, 87.5 million entries, 21.4 ms, now 19.1.)
// A chunk that one graph dominates is copied, and its degrees counted, in pieces
// as a single graph's are, and a graph of kPresortMinEntries or more has its
// chunk's keys presorted. (Chunks of smaller graphs need no presort: a graph's
// entries, and so its cursors, are together.)
constexpr uint64_t kBatchChunk = 1ull << 22;  // entries, at least; at most kUploadChunks chunks
// A piece's least entries: a batch's degree pass searches for its graphs, so a
// piece gains less than a single graph's (100 graphs, 2^20 entries: 620 us in
// pieces of 2^17, 594 in one; one graph of 2^22: 1,512 and 1,503 in pieces of 2^17 and 2^20, 1,538 in one).
constexpr uint64_t kBatchPiece = 1ull << 20;

struct BatchChunk {
  uint64_t g0, g1;  // its graphs
  bool presort;
};
std::vector<BatchChunk> batch_plan(const PrepInput& in) {
  const uint64_t chunks = std::max<uint64_t>(1, std::min<uint64_t>(kUploadChunks, in.E / kBatchChunk));
  std::vector<BatchChunk> plan;
  for (uint64_t k = 0, g0 = 0; k < chunks; ++k) {
    // The graphs whose entries end in the k-th share, or all that are left.
    const uint64_t g1 = k + 1 == chunks ? in.G
                                        : (uint64_t)(std::upper_bound(in.host_eoff + g0 + 1, in.host_eoff + in.G + 1,
                                                                      in.E * (k + 1) / chunks) -
                                                     in.host_eoff - 1);
    BatchChunk c{g0, g1, false};
    for (uint64_t g = g0; g < g1; ++g)
      c.presort |= in.host_eoff[g + 1] - in.host_eoff[g] >= kPresortMinEntries &&
                   in.host_voff[g + 1] - in.host_voff[g] > 256;
    if (g1 > g0) plan.push_back(c);
    g0 = g1;
  }
  return plan;
}

struct BatchBuffers {
  uint32_t *otmp = nullptr, *big = nullptr, *nbr = nullptr, *scratch = nullptr, *col = nullptr;
  uint64_t *rtmp = nullptr, *bent = nullptr, *carry = nullptr, *keys_alt = nullptr;
  RadixTemp ktmp;
};
BatchBuffers take_batch_buffers(Arena& ar, const PrepInput& in, const std::vector<BatchChunk>& plan) {
  const uint64_t n = in.n, E = in.E;
  BatchBuffers b;
  uint64_t keys = 0;  // the most that a chunk presorts; they lie in scratch
  for (const BatchChunk& c : plan)
    if (c.presort) keys = std::max(keys, in.host_eoff[c.g1] - in.host_eoff[c.g0]);
  if (keys) {
    b.keys_alt = ar.take<uint64_t>(keys);
    b.ktmp = take_radix_temp(ar, keys);
  }
  b.otmp = take_scan_temp<uint32_t>(ar, n + 1);
  b.rtmp = take_scan_temp<uint64_t>(ar, n + 1);
  b.carry = ar.take<uint64_t>(1);
  b.big = ar.take<uint32_t>(n + 1);
  b.nbr = ar.take<uint32_t>(2 * E + 1);
  b.scratch = ar.take<uint32_t>(2 * E + 2);
  b.col = ar.take<uint32_t>(E + 4);
  b.bent = ar.take<uint64_t>(E + 2);
  return b;
}

void build_batch(const PrepInput& in, const std::vector<BatchChunk>& plan, const BatchBuffers& b, uint32_t* deg,
                 const RankBuffers& rb, uint32_t* rank, uint32_t* graph_of_rank, uint32_t* cnt, uint32_t* off,
                 uint32_t* nbig, cudaStream_t st, DeviceStats* stats, uint64_t* rp) {
  const uint64_t n = in.n, E = in.E;
  const HostUpload& up = in.upload;
  const uint64_t pieces = upload_pieces(E, kBatchPiece), piece = ceil_div<uint64_t>(E, pieces);
  const bool upload = up.host && E > 0, overlap = upload && pieces > 1;
  TB_CUDA(cudaMemsetAsync(stats, 0, (size_t)((char*)(deg + n) - (char*)stats), st));
  TB_CUDA(cudaMemsetAsync(rp, 0, sizeof(uint64_t), st));
  if (overlap) {  // the copies wait for the stream's earlier work, which may still read the staging buffer
    TB_CUDA(cudaEventRecord(up.events[0], st));
    TB_CUDA(cudaStreamWaitEvent(up.copy_stream, up.events[0], 0));
  }
  for (const BatchChunk& c : plan) {
    const uint64_t e0 = in.host_eoff[c.g0], e1 = in.host_eoff[c.g1], v0 = in.host_voff[c.g0], v1 = in.host_voff[c.g1];
    const uint64_t z = v1 - v0;
    // The chunk in the pieces nearest in size to a single graph's.
    const uint64_t parts = std::max<uint64_t>(1, (e1 - e0 + piece / 2) / std::max<uint64_t>(1, piece));
    for (uint64_t k = 0; k < parts; ++k) {
      const uint64_t i0 = e0 + (e1 - e0) * k / parts, i1 = e0 + (e1 - e0) * (k + 1) / parts;
      if (upload && i1 > i0) {
        upload_entries(in, i0, i1, overlap ? up.copy_stream : st);
        if (overlap) {  // a wait keeps the record it was queued after, so one event serves all pieces
          TB_CUDA(cudaEventRecord(up.events[1], up.copy_stream));
          TB_CUDA(cudaStreamWaitEvent(st, up.events[1], 0));
        }
      }
      if (upload && i1 > i0 && i1 == E && up.uploaded) TB_CUDA(cudaEventRecord(up.uploaded, st));
      degree_pass(in, i0, i1, deg, &stats->err, st);
    }
    if (z > 0) {
      // Everything of the chunk from its first rank on; slots from 2 e0 on, offsets within the chunk.
      rank_by_degree(deg, e1 - e0, v0, z, in.voff, in.G, (uint32_t)c.g0, (uint32_t)c.g1, rb, rank, graph_of_rank,
                     RowWords{cnt + v0, z + 1, true, nullptr}, st);
      device_scan<uint32_t, OpSum>(cnt + v0, off + v0, z + 1, true, OpSum{}, 0u, b.otmp, st, cnt + v0);
      if (c.presort)
        fill_presorted(in, e0, e1, rank, v0, z, reinterpret_cast<uint64_t*>(b.scratch), b.keys_alt, b.ktmp, cnt,
                       b.nbr + 2 * e0, &stats->err, st);
      else
        fill_entries(in, e0, e1, rank, cnt, b.nbr + 2 * e0, &stats->err, st);
      TB_CUDA(cudaMemsetAsync(nbig, 0, kLongWords * sizeof(uint32_t), st));
      TB_CUDA(cudaMemcpyAsync(b.carry, rp + v0, sizeof(uint64_t), cudaMemcpyDeviceToDevice, st));
      const LongRows lng{b.big, nbig};
      sort_rows(off + v0, cnt + v0, (uint32_t)z, e1 - e0, b.nbr + 2 * e0, b.scratch, rp + v0, lng, st);
      device_scan<uint64_t, OpSum>(rp + v0, rp + v0, z + 1, true, OpSum{}, 0ull, b.rtmp, st);
      k_range_carry<<<grid_for(z + 1), kThreads, 0, st>>>(rp + v0, (uint32_t)(z + 1), b.carry);
      TB_LAUNCH_CHECK();
      k_emit_rows<<<emit_grid(e1 - e0 + z), kThreads, 0, st>>>(off + v0, b.nbr + 2 * e0, rp + v0, (uint32_t)z,
                                                               emit_chunk(e1 - e0 + z), lng, b.col, b.bent, nullptr);
      TB_LAUNCH_CHECK();
    }
  }
  k_finalize<<<1, 1, 0, st>>>(rp, n, stats);
  TB_LAUNCH_CHECK();
}

}  // namespace

void rank_vertices(const uint32_t* deg, uint64_t n, uint64_t E, const RankBuffers& b, uint32_t* rank, cudaStream_t st) {
  if (n > 0) rank_by_degree(deg, E, 0, n, nullptr, 0, 0, 0, b, rank, nullptr, RowWords{}, st);
}

void prepare_graph(Arena& ar, const PrepInput& in, cudaStream_t st, Prepared* out) {
  const uint64_t n = in.n, E = in.E;
  if (n > 0xffffffffull || E > kMaxEntries)
    throw StatusError(TRIBIT_ERR_TOO_LARGE, "graphs are limited to 2^32-1 vertices and 2^32-2 entries");
  const bool by_degree = in.order == TRIBIT_ORDER_DEGREE;
  DeviceStats* stats = ar.take<DeviceStats>(1);
  uint32_t* deg = by_degree ? ar.take<uint32_t>(n ? n : 1) : nullptr;  // right after stats: cleared together
  uint64_t* rp = ar.take<uint64_t>(n + 1);
  uint32_t* rank = nullptr;
  uint32_t* graph_of_rank = in.G ? ar.take<uint32_t>(n ? n : 1) : nullptr;
  // The row counters and, after them, the long rows' list lengths: set together.
  uint32_t* cnt = ar.take<uint32_t>(n + 1);
  uint32_t* nbig = ar.take<uint32_t>(kLongWords);
  uint32_t* off = ar.take<uint32_t>(n + 1);
  RankBuffers rb;
  if (by_degree) {
    rank = ar.take<uint32_t>(n ? n : 1);
    rb = take_rank_buffers(ar, n);
  }
  out->n = n;
  out->E = E;
  out->stats = stats;
  out->rank = rank;
  out->view.n = (uint32_t)n;
  out->view.rp = rp;
  out->view.graph_of_rank = graph_of_rank;
  out->view.eflag = nullptr;
  out->view.by_id = !by_degree;

  if (batch_chunks(in)) {
    const std::vector<BatchChunk> plan = batch_plan(in);
    const BatchBuffers b = take_batch_buffers(ar, in, plan);
    out->view.col = b.col;
    out->view.bent = b.bent;
    if (!ar.measuring()) build_batch(in, plan, b, deg, rb, rank, graph_of_rank, cnt, off, nbig, st, stats, rp);
    return;
  }
  // Phase 1 (launch only when not measuring): the upload of host entries,
  // degrees and the rank order.
  if (!ar.measuring()) {
    const RowWords rw{cnt, (uint64_t)(nbig + kLongWords - cnt), degree_slots(in), rank_scans(in) ? off : nullptr};
    TB_CUDA(cudaMemsetAsync(stats, 0, deg ? (size_t)((char*)(deg + n) - (char*)stats) : sizeof(DeviceStats), st));
    if (!by_degree || n == 0) TB_CUDA(cudaMemsetAsync(cnt, 0, rw.count * sizeof(uint32_t), st));
    const HostUpload& up = in.upload;
    const bool upload = up.host && E > 0;
    const uint64_t pieces = upload_pieces(E, kUploadMinPiece);
    const bool overlap = upload && by_degree && n > 0 && pieces > 1;
    if (upload && !overlap) upload_entries(in, 0, E, st);
    if (upload && !overlap && up.uploaded) TB_CUDA(cudaEventRecord(up.uploaded, st));
    if (by_degree && n > 0) {
      if (overlap) {
        // The copies wait for the stream's earlier work (which may still read
        // the staging buffer); piece k's degree pass waits for piece k.
        TB_CUDA(cudaEventRecord(up.events[0], st));
        TB_CUDA(cudaStreamWaitEvent(up.copy_stream, up.events[0], 0));
        const uint64_t piece = ceil_div<uint64_t>(E, pieces);
        for (uint64_t k = 0; k < pieces; ++k) {
          const uint64_t i0 = k * piece, i1 = std::min<uint64_t>(E, i0 + piece);
          if (i0 >= i1) break;
          upload_entries(in, i0, i1, up.copy_stream);
          TB_CUDA(cudaEventRecord(up.events[k + 1], up.copy_stream));
          TB_CUDA(cudaStreamWaitEvent(st, up.events[k + 1], 0));
          if (i1 == E && up.uploaded) TB_CUDA(cudaEventRecord(up.uploaded, st));
          degree_pass(in, i0, i1, deg, &stats->err, st);
        }
      } else {
        degree_pass(in, 0, E, deg, &stats->err, st);
      }
      rank_by_degree(deg, E, 0, n, in.voff, in.G, 0, in.G, rb, rank, graph_of_rank, rw, st);
    } else if (in.G && n > 0) {
      k_identity_graph_of<<<grid_for(n), kThreads, 0, st>>>(n, in.voff, in.G, graph_of_rank);
      TB_LAUNCH_CHECK();
    }
  }
  // Phase 2: orient, rows, sort + dedup per row, CSR + bit rows.
  run_rows(ar, in, rank, cnt, off, nbig, st, out, stats, rp);
}

}  // namespace tb
