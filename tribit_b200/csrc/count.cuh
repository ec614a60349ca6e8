// Counting kernels over a prepared graph (see prep.cuh).
//
// Triangles = sum over u, over v in N+(u), of |N+(u) & N+(v)|: each triangle
// is counted once, at its lowest-ranked vertex. This is the quantity the
// reference accumulates as sum popc(U(u, blk) & L(v, blk)) in
// compute_binary_popcount_mma_9 (tribit.cu:519-586), whose per-lane binary
// searches and one-row-in-eight b1 MMA tiles it replaces.
//
// Work is scheduled in two levels. The dispatcher assigns every 32-row block
// of the oriented graph one counting variant (row-block features -> plain
// thresholds or the learned MLP). Each variant's rows are then cut into
// pieces of at most piece_width neighbours, so one heavy row is spread
// over many warps; the variant kernels are persistent and pull pieces from a
// device cursor.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "arena.h"
#include "prep.cuh"

namespace tb {

constexpr int kNumFeatures = 16;
constexpr int kTileMaxK = 64;  // bit-tile variant: row blocks spanning at most this many column blocks
constexpr int kFeatSpan = 13;  // feature index of log2(1 + column-block span)
constexpr uint32_t kMinPieceWidth = 32;  // piece_width is a multiple of 32, at least this
// Plain dispatcher: a row block goes to the merge variant when its neighbours'
// bit rows average at least this many times its own rows' length. Set once from
// a sweep over RMAT-18..24, planted partition, Chung-Lu and Erdos-Renyi graphs.
// On today's merge pieces 0.25, 0.75 and 1.5 count RMAT-24 in 35.6, 37.2 and 47.3
// ms, RMAT-22 in 6.17, 6.65 and 11.1, planted in 1.59, 1.59 and 1.55, Erdos-Renyi in
// 0.83, 0.81 and 0.80 and the 4,096-graph batch in 34.4, 32.1 and 31.3.
constexpr float kDefaultMergeRatio = 0.75f;

// Piece lists: one per variant, the heavy rows' (too many bit blocks for a
// warp's table: a CTA per piece) and the wide rows' (too many for the heavy
// phase's 32 KiB as well: kernel k_rows_wide).
enum { kListHeavy = TRIBIT_NUM_VARIANTS, kListWide, kPieceLists };
// piece_off: where each list starts in `pieces` (and where the last ends), the
// hub pass's CTA pieces, all its pieces and its edges, then the row blocks with
// pieces of each variant.
enum { kOffHubCta = kPieceLists + 1, kOffHubAll, kOffHubEdges, kOffRowBlocks };
static_assert(kOffRowBlocks + TRIBIT_NUM_VARIANTS == kScheduleWords, "piece_off's words in DeviceStats");

// What the hub builder keeps of a vertex: its bit row, (blocks it spans << 32) |
// length, 0 for a vertex that is no hub; and, apart from it (the row words are
// only read while edges are walked, and stay in the L1), a pair of counters:
// while candidates are counted, their number and the blocks their walks would
// save; then the next place in its in-list for a bit-row tail (from the front)
// and the last one taken for a column tail (from the back).
struct HubTable {
  uint64_t* info = nullptr;  // n + 1; null: no hub pass
  uint2* cur = nullptr;      // n + 1
};

struct Schedule {
  uint32_t num_row_blocks = 0;
  uint8_t* variant_of = nullptr;   // device, per row block
  uint64_t* pieces = nullptr;      // device, (row << 32) | first neighbour, one segment per piece list
  uint64_t piece_cap = 0;
  uint32_t* piece_off = nullptr;   // device, kScheduleWords words in DeviceStats (see kOff*)
  uint64_t* counts = nullptr;      // device, kPieceLists * nrb + 1: pieces per (list, row block), scanned
  uint64_t* scan_tmp = nullptr;
  float* features = nullptr;       // device, nrb x kNumFeatures
  // Hub pass of the merge variant (absent when taken without hubs).
  uint32_t* eflag = nullptr;       // device, bit per CSR position: edge counted by the hub pass
  uint64_t eflag_words = 0;
  HubTable hub;                    // device
  uint32_t* in_off = nullptr;      // device, n + 1: in-list of hub v at [in_off[v], in_off[v+1]); then, from
                                   // n + 1 on, 2(n + 1) piece counts scanned with it (CTA, warp pieces)
  uint64_t* inl = nullptr;         // device: (first block of u's tail << 32) | tail length
  uint64_t inl_cap = 0;            // entries inl (and inrow) hold
  uint32_t* inrow = nullptr;       // device: u of each in-list entry (timing mode only: its own buffer)
  uint64_t* hub_pieces = nullptr;  // device: (v << 32) | first in-list entry; CTA pieces, then warp pieces
  uint64_t* hub_pieces2 = nullptr; // device: the pieces in hub order, before the wave sort
  uint8_t* piece_wave = nullptr;   // device: digit of each piece (its list and the wave of its first tail)
  uint32_t* wave_lo = nullptr;     // device: first row of each wave, then n
  uint32_t* wave_bk = nullptr;     // device: bit-row start of each wave's first row
  uint32_t* wave_cp = nullptr;     // device: CSR position of each wave's first row
  uint32_t* wave_cnt = nullptr;    // device: pieces per (list, wave), scanned to positions
  uint32_t* hub_scan_tmp = nullptr;
  bool hubs = true;                // build the hub lists for merge row blocks
  bool hubs_active = false;        // set by build_pieces
  bool hub_rows = false;           // also write each in-list entry's row (read by the timing mode only)
  uint32_t piece_width = 64;       // neighbours per piece (tuned)
  float tile_min_nnz = 64.f;       // plain dispatcher: fewest edges for a bit-tile row block (tuned)
  float merge_ratio = kDefaultMergeRatio;  // plain dispatcher: merge where neighbours' bit rows are this much longer
  int tile_engine = TRIBIT_TILES_TCGEN05;  // bit-tile product: tcgen05 kind::i8 or b1 mma.sync
  const void* model = nullptr;     // device MLP parameters for learned dispatch
};

// Per-launch configuration chosen by the autotuner (or defaults).
struct CountConfig {
  int ctas_per_sm = 0;  // 0 = default
  int num_sms = 148;
  unsigned long long* block_ns = nullptr;  // optional: per-row-block warp-cycles (SM cycles x warps busy)
  cudaEvent_t variant_start = nullptr;     // optional (timing mode): these events bracket
  cudaEvent_t variant_stop = nullptr;      // all counting kernels
  uint32_t tile_wait_polls = 1u << 22;     // tcgen05 tiles: mbarrier polls before a wait gives up
  int tile_test_no_commit = 0;             // failure-detection test: tile MMAs never committed
  bool queue = false;                      // TRIBIT_LAUNCH_QUEUE (not in the timing mode)
};

// TRIBIT_LAUNCH_AUTO takes the queue kernel up to this many entries, where the
// boundaries between kernels weigh most (plain dispatch, queue and kernels:
// RMAT-16 90 and 154 us, RMAT-18 234 and 293, RMAT-20, 2^24 entries, 1,170 and
// 1,237). Beyond, it depends on the graph: RMAT-22 6.31 and 6.64 ms, RMAT-24 37.35
// and 37.22, but planted partition of 2 million vertices 1.88 and 1.58, Erdos-Renyi
// of 2^25 entries 2.17 and 2.11.
constexpr uint64_t kQueueMaxEntries = 1ull << 24;

// hubs: also take the hub-pass arrays (about 8 bytes per entry and 36 per vertex). stats: the
// prepared graph's, which holds the schedule's words (null when measuring).
Schedule take_schedule(Arena& ar, uint64_t n, uint64_t E, DeviceStats* stats, bool hubs = true);

// Sends the row blocks dispatched to the merge variant to the bitmap sweep.
void merge_blocks_to_bitmap(Schedule& s, cudaStream_t st);

// Computes row-block features, the per-block variant (mode: TRIBIT_DISPATCH_*),
// and the per-variant piece lists. full_features adds the neighbour-side
// features (one extra pass over the edges) the learned dispatcher needs.
void build_schedule(const GraphView& g, Schedule& s, int mode, bool full_features, cudaStream_t st);

// Row-block features (full adds the neighbour-side ones) and the plain or
// forced variant for every row block; build_schedule = this + build_pieces.
void compute_features(const GraphView& g, Schedule& s, int mode, bool full_features, cudaStream_t st);

// Re-derives the piece lists after variant_of was rewritten (learned dispatch).
void build_pieces(const GraphView& g, Schedule& s, cudaStream_t st);

struct LaunchInfo {
  uint64_t ctas = 0;     // CTAs over all counting kernels
  uint32_t kernels = 0;  // kernel launches
};

// Launches every counting kernel; the exact count lands in stats->triangles
// (and per_graph[g] in batch mode).
LaunchInfo launch_count(const GraphView& g, const Schedule& s, DeviceStats* stats, unsigned long long* per_graph,
                        const CountConfig& cfg, cudaStream_t st);

}  // namespace tb
