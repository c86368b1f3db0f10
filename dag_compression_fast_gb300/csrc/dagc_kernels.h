// Host-side declarations of the dagc kernel launchers (implemented in the .cu
// files). Plain C++: the orchestrator (dagc.cpp) includes this header only.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "dagc_hash.h"  // DAGC_HD

namespace dagc {

// ------------------------------------------------------------ error bits ----
// Kernels never trap: they OR one of these into the call's error word and
// carry on with a defined (if meaningless) value so that every wait still ends.
enum : uint32_t {
    kErrBadInput = 1u,      // fragment code >= 2^(3*depth)
    kErrCollision = 2u,     // equal 64-bit hash, different node
    kErrTimeout = 4u,       // a bounded wait ran out
    kErrCapacity = 8u,      // an upper bound on a buffer was exceeded
    kErrNotRooted = 16u,    // level 0 does not hold exactly one node
    kErrMergeRoot = 32u,    // a sub-DAG root hash missing from the merged level
    kErrFallback = 64u,     // the hash-set dedup could not hold a level: rerun with the radix form
};

constexpr uint32_t kEmptyChild = 0xFFFFFFFFu;


// ---------------------------------------------------------------- sort ----
constexpr int kSortThreads = 256;
// Digit-pass tiles hold 256 threads x (8..16) keys.
constexpr int kSortTile = 2048;
constexpr int kRadixBits = 8;       // default digit width
constexpr int kMaxRadixBits = 11;   // widest digit a keys-only pass takes
constexpr int kMaxPasses = 8;
constexpr int kSortHistWords = 8192;  // one sort's histograms: passes x 2^(widest digit)

DAGC_HD uint32_t sort_tiles(uint64_t n) { return (uint32_t)((n + kSortTile - 1) / kSortTile); }
// Look-back status words of one digit pass for n keys, enough for every pass
// shape: tiles of at least 2048 keys with 256 digits, or of at least 4096
// keys with up to 2048 digits.
DAGC_HD uint64_t sort_status_words(uint64_t n) { return ((n + 4095) / 4096 + 1) * 2048; }

// Digits of a sort over bits [lo, hi) in `passes` passes: widths differ by at
// most one, the wider ones first; pass i covers bits [shift, shift + bits).
DAGC_HD int sort_passes_r(int lo_bit, int hi_bit, int radix_bits) {
    return hi_bit > lo_bit ? (hi_bit - lo_bit + radix_bits - 1) / radix_bits : 0;
}
DAGC_HD void pass_digit(int lo_bit, int hi_bit, int passes, int i, int* shift, int* bits) {
    const int b = hi_bit - lo_bit, w = b / passes, extra = b % passes;
    *bits = w + (i < extra ? 1 : 0);
    *shift = lo_bit + i * w + (i < extra ? i : extra);
}
// Histogram words between consecutive passes: 2^(widest digit).
DAGC_HD int pass_hist_stride(int lo_bit, int hi_bit, int passes) {
    const int b = hi_bit - lo_bit;
    return passes > 0 ? 1 << ((b + passes - 1) / passes) : 0;
}
// Number of digit passes for a bit range at the default width.
DAGC_HD int sort_passes(int lo_bit, int hi_bit) { return sort_passes_r(lo_bit, hi_bit, kRadixBits); }

// Device count pointer convention: when d_n is non-null the kernels read the
// element count from device memory (written by an earlier kernel) and n is an
// upper bound used only to size the grid; otherwise n is the count.
struct SortArgs {
    const uint64_t* keys_in;
    uint64_t* keys_out;
    uint64_t* keys_alt;       // ping-pong buffer (n elements)
    const uint32_t* vals_in;  // null with with_values -> values are 0..n-1
    uint32_t* vals_out;
    uint32_t* vals_alt;
    bool with_values;
    uint64_t n;               // count or upper bound (see d_n)
    const uint64_t* d_n;
    int lo_bit, hi_bit;
    int radix_bits;           // widest digit (8..11; keys only above 8); 0 = 8
    int validate_bits;        // > 0: flag keys with bits >= validate_bits set
    uint32_t* hist;           // kSortHistWords words, zeroed
    uint32_t* status[2];      // 2 x sort_status_words(n) words; status[0] zeroed on entry
    uint32_t* tile_counters;  // kMaxPasses words, zeroed
    uint32_t* err;
    int grid_hist, grid_pass; // persistent grid sizes
    int shape;                // digit-pass kernel shape (a key shape or a pair shape)
    // Gate: when non-null, every kernel of the sort does nothing unless
    // *gate == gate_run (a path chosen on the device, see GroupArgs).
    const uint32_t* gate; uint32_t gate_run;
    // Segmented input (batched chunks): when seg_offsets is non-null, the key at
    // position i of keys_in belongs to segment s with seg_offsets[s] <= i <
    // seg_offsets[s+1] (seg_count + 1 ascending entries) and is sorted as the
    // composite (s << seg_shift) | key. Only the histogram and the first pass
    // read keys_in; they build the composite, later passes move it.
    const uint64_t* seg_offsets;
    uint32_t seg_count;
    int seg_shift;
    // Failure-path test hooks (zero in production): a lower limit on the
    // look-back waits (0 = kSpinLimit), and a first digit pass whose tile 0
    // never publishes its counts, so that the waits of the tiles after it run
    // out and the sort reports kErrTimeout.
    uint32_t spin_limit;
    int stall_first_tile;
};

// Digit-pass kernel shapes. Keys-only sorts: (items per thread, minimum
// resident CTAs per SM, which caps registers, equal-digit matching: ballots,
// match.any, alternating, shared-memory atomicOr); each is
// built for every digit width 8..kMaxRadixBits. Key/value sorts: 8-bit
// digits. The autotuner and dagc options pick a shape and a width per sort.
constexpr int kNumKeyShapes = 9;
constexpr int kNumPairShapes = 10;
constexpr int kNumSortShapes = kNumPairShapes;
int sort_shape_items(int shape, bool with_values);
// Resident CTAs per SM of a shape at a digit width (occupancy query) for grid sizing.
int occupancy_sort_shape(int shape, bool with_values, int radix_bits = kRadixBits);
int occupancy_sort_histogram();
// Whether a (shape, width) plan can sort bits [lo, hi): histogram room and
// look-back status room.
bool sort_plan_valid(int shape, bool with_values, int radix_bits, int lo_bit, int hi_bit);

// Where the result lands: keys_out always (the pass sequence is arranged so).
void launch_sort(const SortArgs& a, cudaStream_t s);
// The same, one launch at a time: histogram (+ copy when there is no digit),
// then digit pass i for i in [0, sort_plan_passes(a)).
int sort_plan_passes(const SortArgs& a);
void launch_sort_histogram(const SortArgs& a, cudaStream_t s);
void launch_sort_pass(const SortArgs& a, int i, cudaStream_t s);
void sort_configure();  // sets shared-memory attributes once per device
// Autotuner input: n pseudo-random keys with bits only in [lo_bit, hi_bit).
void launch_fill_tune_keys(uint64_t* out, uint64_t n, int lo_bit, int hi_bit, uint64_t seed, cudaStream_t s);

// ---------------------------------------------------------- DAG kernels ----
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;
DAGC_HD uint32_t scan_tiles(uint64_t n) { return (uint32_t)((n + kScanTile - 1) / kScanTile); }
// leaf_build takes 8192 sorted keys per tile (its per-tile arrays, sized by
// scan_tiles, are large enough).
constexpr int kLeafTile = 8192;
DAGC_HD uint32_t leaf_tiles(uint64_t n) { return (uint32_t)((n + kLeafTile - 1) / kLeafTile); }

// Fused unique + 4x4x4 leaf build over fragments sorted by (code >> 6):
// parents[p] = code >> 6 and leaves[p] = OR of 1 << (code & 63) per distinct
// parent; *d_out_n = number of parents.
struct LeafBuildArgs {
    const uint64_t* sorted; const uint64_t* d_n; uint64_t n_bound;
    // Batched input: sorted keys are (segment << seg_shift) | local code; the
    // global code is (seg_code[segment] << seg_shift) | local code.
    const uint64_t* seg_code; int seg_shift;
    uint64_t* parents; uint64_t* leaves; uint64_t out_capacity; uint64_t* d_out_n;
    uint64_t* lead_or; uint64_t* lead_run;  // per tile: OR of keys continuing an earlier run, its run id
    uint64_t* status; uint32_t* tile_counter; uint32_t* err; int grid;
    const uint32_t* gate; uint32_t gate_run;  // as in SortArgs
};
void launch_leaf_build(const LeafBuildArgs& a, cudaStream_t s);  // two launches (build + fix-up)

// Fragment grouping by hash (group.cu): the same parents and leaf masks as
// the fragment sort + leaf build, for inputs with many fragments per brick.
constexpr double kGroupMinRedundancy = 8.0;  // fragments per distinct brick that make grouping pay
constexpr int kGroupSketchRegs = 4096;
constexpr int kGroupPartLog = 11;                        // fine partitions counted by the sketch pass
constexpr int kGroupMaxParts = 1 << kGroupPartLog;
constexpr int kGroupPartSlotsLog = 12;                   // shared-memory table of one partition
constexpr int kGroupPartSlots = 1 << kGroupPartSlotsLog;
constexpr double kGroupMaxBricksPerPart = 0.45 * kGroupPartSlots;  // most bricks per table (load 0.45)
constexpr float kGroupTargetBricksPerPart = 1536.0f;     // partitions chosen for ~this many (load ~0.3)
constexpr uint64_t kGroupMaxBricks = (uint64_t)kGroupMaxParts * kGroupPartSlots;
constexpr int kGroupMaxChunks = 512;                     // CTAs of the sketch and scatter passes
constexpr uint64_t kGroupScratchBytes = kGroupMaxBricks * 8;  // the brick masks
struct GroupArgs {
    const uint64_t* frags; uint64_t n;
    const uint64_t* seg_offsets; uint32_t seg_count; int seg_shift;  // batched input (as in SortArgs)
    const uint64_t* seg_code;                                         // chunk Morton index per segment
    int validate_bits;
    int mode;                  // 1: choose by the sketch, 2: always group (tests)
    int narrow;                // every key below 2^37 (bricks below 2^31): 32-bit hashes and table keys
    int chunks;                // CTAs of the scatter: chunk c = [c*L, (c+1)*L), L = ceil(n / chunks)
    uint32_t* sketch;          // kGroupSketchRegs words, zero: the probe's distinct-brick sketch
    float probe_max_distinct;  // grouping when the probe's sample shows at most this many distinct bricks
    uint64_t* cursor;          // kGroupMaxParts: partition p's next free position in its slab
    uint32_t* path;            // [0] 1 grouping, 0 sort path; [1] log2 partitions; [2] log2 table slots; [3] slab size
    uint64_t* d_grouped;       // path[0] among the call's counts
    uint64_t* parts;           // partition slabs (group_shape's slab_total fragment keys)
    uint64_t* overflow; uint64_t overflow_cap;  // fragments past their slab's end, any partition
    uint64_t* overflow_count;  // zero on entry
    uint32_t* part_over;       // kGroupMaxParts flags, zero on entry: the partition spilled
    uint64_t* bricks; uint32_t* idx; uint64_t* masks; uint64_t cap;  // brick list (unsorted), masks[idx]
    // Or, when non-null (unbatched input): the direct-mapped table of all
    // bricks and its block counters (DirectArgs), which puts them in order.
    uint64_t* table; uint32_t* block_count;
    uint64_t* d_count;         // bricks found
    const uint64_t* sorted_bricks; const uint32_t* sorted_idx;      // after the brick sort
    uint64_t* parents; uint64_t* leaves;
    uint32_t* err;
};
void group_configure(int sms);
int group_chunks(uint64_t n);                                      // `chunks` for n fragments
// Room for the partition slabs of n fragments, and the probe's limit (host
// side, before the call).
void group_shape(uint64_t n, uint64_t* slab_total, float* probe_max_distinct);
void launch_group_probe(const GroupArgs& a, cudaStream_t s);
void launch_group_plan(const GroupArgs& a, cudaStream_t s);      // picks the path
void launch_group_scatter(const GroupArgs& a, cudaStream_t s);
void launch_group_aggregate(const GroupArgs& a, cudaStream_t s);
void launch_group_gather(const GroupArgs& a, cudaStream_t s);

// Leaves by a direct-mapped table of the whole brick space (direct.cu).
constexpr int kDirectBlockLog = 6;            // 64 bricks per block
constexpr uint32_t kDirectScanBlocks = 4096;  // up to here (depth 8) the compaction sums the block counts itself
constexpr uint32_t kDirectPlanTile = 4096;    // blocks per tile of the plan
constexpr int kDirectMaxDepth = 11;           // a table of 8^9 entries: 1 GB
DAGC_HD uint64_t direct_blocks(int depth) {
    return ((1ull << (3 * (depth - 2))) + (1ull << kDirectBlockLog) - 1) >> kDirectBlockLog;
}
DAGC_HD uint64_t direct_entries(int depth) { return direct_blocks(depth) << kDirectBlockLog; }  // whole blocks
DAGC_HD uint64_t direct_plan_tiles(int depth) { return direct_blocks(depth) / kDirectPlanTile + 1; }
struct DirectArgs {
    const uint64_t* frags; uint64_t n;
    int code_bits;          // 3 * depth: codes are below 2^code_bits
    uint32_t mark_rows;     // rows of 32 fragments that a warp marks at a time (launch_direct_mark)
    uint64_t* table;        // a leaf mask per brick (direct_entries), zero on entry and exit
    uint32_t blocks;
    uint32_t* block_count;  // bricks per block, zero on entry
    uint2* list; uint64_t* d_blocks;             // occupied blocks: (block, bricks before it), and how many
    uint64_t* status; uint32_t* tile_counter;    // of the plan: zero on entry
    uint64_t* parents; uint64_t* leaves; uint64_t out_capacity; uint64_t* d_out_n;
    uint32_t* err;
    const uint32_t* gate;   // non-null: the compaction does nothing unless *gate == 1 (grouping, GroupArgs::path)
};
void direct_configure(int sms);
// The fragments into the table; the table's bricks out in order. Both return
// the number of launches.
int launch_direct_mark(const DirectArgs& a, cudaStream_t s);
int launch_direct_compact(const DirectArgs& a, cudaStream_t s);

// Batched form: every chunk's leaves in one persistent launch (chunks.cu).
// A chunk's local bricks (local code >> 6) fall in 2^bin_bits bins of at most
// 2^kChunkDirectBits bricks, direct-mapped in shared memory.
constexpr int kChunkThreads = 512;
constexpr int kChunkTile = 8192;       // fragments per tile (a COUNT / SCATTER item is a run of tiles)
constexpr int kChunkDirectBits = 13;   // bricks of one bin
constexpr int kChunkMaxBinBits = 11;   // bins per chunk (chunk depth <= 10)
constexpr int kChunkGroupBins = 32;    // most bins per LEAVES item
struct ChunkArgs {
    const uint64_t* frags;                          // chunk-local codes, chunks back to back
    const uint64_t* seg_offsets; const uint64_t* seg_code;  // k + 1 offsets, k Morton indices (device)
    uint32_t k; int chunk_depth; int seg_shift;     // seg_shift = 3 * chunk_depth
    int bin_bits;                                   // chunk_bin_bits(chunk_depth)
    uint32_t run_tiles;                             // tiles per COUNT / SCATTER item (chunk_run_tiles)
    const uint32_t* item_off;                       // k + 1: first COUNT (and SCATTER) item of each chunk (device)
    uint32_t items;                                 // item_off[k] (host copy, for the grid only)
    uint32_t group_bins, groups_per_chunk;          // bins per LEAVES item (chunk_group_bins), items per chunk
    uint32_t* hist; uint32_t* cursor;               // k << bin_bits each, hist zero
    uint32_t* done;                                 // 3k: COUNT items done, SCATTER items done, starts known (zero)
    uint32_t* work;                                 // item counter (zero)
    uint32_t* scratch;                              // fragments' local codes by bin (n)
    uint64_t* stage_parent; uint64_t* stage_mask;   // n each: each item's bricks at its fragment offset
    uint32_t* group_bricks; uint64_t* group_src; uint32_t* group_dst;  // per LEAVES item
    uint64_t* parents; uint64_t* leaves; uint64_t out_capacity; uint64_t* d_out_n;
    uint32_t* err;
};
void chunk_configure(int sms);
int chunk_run_tiles(uint64_t n);
uint32_t chunk_group_bins(uint64_t k, uint32_t bins);
int chunk_bin_bits(int chunk_depth);  // -> bins of at most 2^kChunkDirectBits bricks
void launch_chunk_leaves(const ChunkArgs& a, cudaStream_t s);  // three launches

// Unique over (key, perm) sorted by key: uid = rank of the key among distinct
// keys; map[perm[i]] = uid; for the first of each run, out_keys[uid] = key and
// payloads are gathered from perm. With node payloads (masks/children) the
// run members are compared in full (collision check).
//
// Every kernel that produces a count is given the capacity of its outputs: it
// never writes past it, clamps the count (and ids) it publishes to it and
// flags kErrCapacity, so that later kernels stay inside their buffers even on
// rejected input.
struct UniqueArgs {
    const uint64_t* keys; const uint32_t* perm; const uint64_t* d_n; uint64_t n_bound;
    const uint8_t* masks; const uint32_t* children;  // null for leaves
    uint32_t* map;
    uint64_t* out_keys; uint8_t* out_masks; uint32_t* out_children;
    uint64_t out_capacity;
    uint64_t* d_out_n;
    uint64_t* status; uint32_t* tile_counter; uint32_t* err; int grid;
};
void launch_unique(const UniqueArgs& a, cudaStream_t s);

// Level dedup by hash set + ordering of the distinct keys (dedup.cu the leaf
// masks, levels.cu the node levels): same outputs as sort pairs + unique_runs on
// (key, item) for one level.
constexpr uint32_t kDedupPerBucket = 256;            // expected distinct keys per bucket (node hashes)
constexpr uint32_t kDedupTopBitCap = 1024;           // bucket room (128-256 expected)
constexpr uint32_t kDedupMaxBuckets = 16384;
constexpr uint64_t kDedupMaxItems = 1ull << 24;
constexpr uint64_t kDedupMaxUnique = (uint64_t)kDedupMaxBuckets * kDedupPerBucket;
// Bucket entries for up to uniq_cap distinct keys: the buckets for n items
// (a power of two, n / 256 <= buckets < 2n / 256) hold fewer than 8n entries.
DAGC_HD uint64_t dedup_bucket_area(uint64_t uniq_cap) {
    const uint64_t a = 8 * uniq_cap > kDedupTopBitCap ? 8 * uniq_cap : kDedupTopBitCap;
    const uint64_t most = (uint64_t)kDedupMaxBuckets * kDedupTopBitCap;
    return a < most ? a : most;
}
// Buckets of a node level of n items (they only grow with n): a power of two.
DAGC_HD uint32_t node_buckets(uint64_t n) {
    uint32_t b = 1;
    while ((uint64_t)b * kDedupPerBucket < n && b < kDedupMaxBuckets) b <<= 1;
    return b;
}
// Table slots for n items. Leaf masks repeat (about one distinct mask per ten
// bricks): 1.25 n slots, at most 0.8 full even when every mask is distinct,
// small enough to stay largely in the L2. Up to kLeafSparseMax of them the
// table is in the L2 anyway and the insert's time is its longest probe chain, a
// round trip per two slots: 4 n slots (25k distinct masks of 36k bricks: the
// insert takes 12 us, 25 with 1.25 n). Node hashes are about half distinct
// and each probe step is a dependent round trip: 2 n slots at sizes beyond the
// L2, where emptier tables cost more than they save, 4 n and 8 n below
// (kNodeSparseMax, kNodeEmptyMax nodes; 12k nodes of a 512^3 terrain: the
// insert takes 10 us, 29 with 2 n). At least 1024 slots, a multiple of 32.
constexpr uint64_t kLeafSparseMax = 1ull << 20;
constexpr uint64_t kNodeSparseMax = 1ull << 20, kNodeEmptyMax = 1ull << 17;
DAGC_HD uint64_t table_size_for(uint64_t n, bool leaf_masks) {
    const uint64_t want = leaf_masks ? (n <= kLeafSparseMax ? 4 * n : n + (n >> 2))
                                     : (n <= kNodeEmptyMax ? 8 * n : n <= kNodeSparseMax ? 4 * n : 2 * n);
    return want < 1024 ? 1024 : (want + 31) & ~31ull;
}
// Slots that hold any count of up to `items` items.
DAGC_HD uint64_t node_slots_upto(uint64_t items) {
    uint64_t most = table_size_for(items, false);
    const uint64_t a = table_size_for(items < kNodeEmptyMax ? items : kNodeEmptyMax, false);
    const uint64_t b = table_size_for(items < kNodeSparseMax ? items : kNodeSparseMax, false);
    if (a > most) most = a;
    return b > most ? b : most;
}
DAGC_HD uint64_t leaf_slots_upto(uint64_t items) {
    const uint64_t sparse = table_size_for(items < kLeafSparseMax ? items : kLeafSparseMax, true);
    const uint64_t all = table_size_for(items, true);
    return all > sparse ? all : sparse;
}
struct DedupState {
    unsigned long long u;  // distinct keys found (zero on entry)
};
// Ordering of the distinct leaf masks: up to kLeafRankMax of them are ranked
// at once, more go through buckets between samples (half as many buckets up to
// kLeafMidMax).
constexpr uint32_t kLeafRankMax = 8192;
constexpr uint32_t kLeafBuckets = 2048;
constexpr uint64_t kLeafMidMax = 1ull << 18;
struct LeafOrder {
    uint32_t count[kLeafBuckets];  // keys per bucket, zero on entry
    uint64_t splitter[kLeafBuckets];
};
// Most keys of one bucket (10 bytes of shared memory each) when the list may
// hold uniq_cap: the mean is at most 256 up to kLeafMidMax, then uniq_cap / 2048.
DAGC_HD uint32_t leaf_keys_for(uint64_t uniq_cap) { return uniq_cap <= kLeafMidMax ? 2048u : 8192u; }
struct DedupArgs {
    const uint64_t* keys; const uint64_t* d_n;  // the bricks' leaf masks
    uint64_t item_cap;
    // Table of table_cap slots, 16 bytes each so that a
    // slot's key and aux share a sector: table_key[2s] = key, 0 = empty (all
    // 0 on entry and exit); table_aux[2s] = representative item | unique id
    // << 32 (table_aux = table_key + 1).
    uint64_t* table_key; uint64_t* table_aux; uint64_t table_cap;
    uint32_t* item_slot;
    uint64_t* uniq_key; uint32_t* uniq_slot; uint64_t uniq_cap;  // the unique list and its slots
    LeafOrder* leaf; uint32_t leaf_keys;                         // its ordering; leaf_keys_for(uniq_cap)
    uint4* bucket; uint64_t bucket_area;                         // bucket entries: key (two words), slot
    DedupState* state;
    uint64_t* out_keys; uint64_t out_capacity;
    uint64_t* d_out_n;
    uint32_t* map;  // item -> unique id
    uint32_t* err;
};
void dedup_configure(int sms);
// Insert into the table and the unique list; order the list into the leaf array
// and assign the unique ids (returns the number of launches); then map.
void launch_dedup_insert(const DedupArgs& a, cudaStream_t s);
int launch_leaf_order(const DedupArgs& a, cudaStream_t s);
void launch_dedup_map(const DedupArgs& a, cudaStream_t s);

// Node levels of the hash-set form (levels.cu): nodes of a level, in the order
// of their codes.
constexpr int kNodeLevels = 19;  // levels of the deepest DAG
struct NodeArrays {
    uint64_t* hash;
    uint8_t* mask;     // children present
    uint32_t* first;   // index of the first child among the level below's nodes (or bricks); the others follow it
    // Or (first null; the union of several DAGs): all eight children as indices
    // among the level below's items, kEmptyChild where there is none.
    uint32_t* children;
};
struct NodesArgs {
    const uint64_t* child_codes; const uint64_t* child_hashes;  // of every child (not only the distinct ones)
    const uint64_t* d_n; uint64_t n_bound;
    uint64_t* node_codes; NodeArrays out; uint64_t out_capacity;
    uint64_t* d_out_n;
    uint64_t tail_max;  // up to this many children the level is left to the tail
    uint64_t* status; uint32_t* tile_counter; uint32_t* err;
};
void launch_extract_nodes(const NodesArgs& a, cudaStream_t s);
// Every level from the largest one of at most kTailCap children up to the root.
struct TailNodesLevel {
    const uint64_t* child_codes; const uint64_t* child_hashes; const uint64_t* d_child_n;
    NodeArrays out; uint64_t capacity;
    uint64_t* d_nodes;
};
struct TailNodesArgs {
    int levels;
    TailNodesLevel lv[kNodeLevels];  // root first
    uint32_t* err;
};
void launch_tail_nodes(const TailNodesArgs& a, cudaStream_t s);
// Dedup of consecutive levels at once, into one table and one set of buckets.
struct GroupLevel {
    NodeArrays nodes; const uint64_t* d_n;
    uint64_t* out_keys; uint8_t* out_masks; uint32_t* out_children; uint64_t capacity;
    uint64_t* d_out_n;
};
constexpr uint64_t kGroupItems = 1ull << 24;  // levels share a group while their bounds add up to this
struct GroupDedupArgs {
    int levels;
    GroupLevel lv[kNodeLevels];    // the group's levels, the one nearest the root first
    const uint32_t* child_map;     // unique ids of the items below the group's last level
    uint32_t* map;                 // null, or the unique ids of the first level's nodes (the next group's child_map)
    uint64_t* table_key; uint64_t* table_aux; uint64_t table_cap;  // as DedupArgs
    uint32_t* item_slot; uint64_t slot_cap;
    uint32_t* bucket_count; uint32_t bucket_cap;                   // zero on entry and exit
    uint4* bucket; uint64_t bucket_area;                           // kDedupTopBitCap entries each: key (two words), slot, representative
    uint64_t uniq_cap;
    uint32_t* err;
};
// Union of several DAGs: their levels' nodes and leaves one after another, as
// the items of the leaf dedup and of launch_group_dedup.
struct MergeArgs {
    uint32_t k; int levels;          // inputs, node levels
    // Per input: hashes, children, masks, leaves (device pointers), all inputs'
    // hashes first; then per input and level the level's first node; then per
    // level (the leaves last) and input, k + 1 each: its first item.
    const uint64_t* table;
    uint64_t level0[kNodeLevels + 2];   // items before each level (the leaves after the last; then the total)
    NodeArrays out[kNodeLevels];
    uint64_t* leaves;
    uint64_t* d_n[kNodeLevels + 1];     // item counts to set: levels, then leaves
    // Roots: the map of level 0 (or of the leaves), then per input its root's id and hash.
    const uint32_t* root_map; uint32_t* root_uid; uint64_t* root_hash;
    uint32_t* err;
};
void launch_merge_gather(const MergeArgs& a, cudaStream_t s);
void launch_merge_roots(const MergeArgs& a, cudaStream_t s);
void levels_configure(int sms);
uint64_t group_slot_items(uint64_t n);  // item_slot entries of a level of n nodes
int launch_group_dedup(const GroupDedupArgs& a, uint64_t items_bound, cudaStream_t s);  // returns the number of launches

// One level of the radix form: nodes with their child ids and hashes.
struct ExtractArgs {
    const uint64_t* child_codes; const uint32_t* child_map; const uint64_t* d_n; uint64_t n_bound;
    const uint64_t* child_hashes;  // unique child hashes (or leaf masks), indexed by child id
    uint64_t* node_codes; uint8_t* node_masks; uint32_t* node_children; uint64_t* node_hashes;
    uint64_t out_capacity;
    uint64_t* d_out_n;
    uint64_t* status; uint32_t* tile_counter; uint32_t* err; int grid;
};
void launch_extract(const ExtractArgs& a, cudaStream_t s);

// Headless tracer (trace.cu): one primary ray per pixel through the final
// word layout of a depth-`depth` DAG (depth >= 3).
struct TraceArgs {
    const uint32_t* words; uint64_t n_words; int depth;
    uint32_t debug_level, width, height;
    double camera[3], ray_min[3], ray_ddx[3], ray_ddy[3];
    // ray_min - camera, ray_ddx and ray_ddy as float32 pairs, and a bound of
    // what makes up a ray's components (set by launch_trace).
    float base[6], ddx[6], ddy[6], magnitude;
    uint32_t* colors;  // width * height, row-major
    uint64_t* hits;    // optional: Morton code of the voxel hit, ~0 for a miss
    uint32_t* err;
};
void launch_trace(const TraceArgs& a, cudaStream_t s);

// Triangle voxelizer (voxelize.cu).
constexpr int kVoxGL = 0;   // the reference's GL rule: one voxel per covered pixel of the dominant view
constexpr int kVoxSAT = 1;  // every voxel the triangle touches (separating axis test)
struct VoxArgs {
    const double* vertices; uint64_t n_tri;  // 9 doubles per triangle
    double aabb[6];                          // box mapped onto the grid: min xyz, max xyz
    double scale[3];                         // 2^depth / extent (set by launch_voxelize)
    int per;                                 // triangles per warp (set by launch_voxelize)
    int depth, mode;
    uint64_t* codes; uint64_t capacity;
    uint64_t* d_total;                       // fragments produced (may exceed capacity)
    uint64_t* status; uint32_t* tile_counter; uint32_t* err;  // status: voxelize_tiles + 1 words, zero
};
void voxelize_configure();
void launch_voxelize(const VoxArgs& a, int grid, cudaStream_t s);
uint64_t voxelize_tiles(uint64_t n_tri, int mode);

// The radix form's top levels in one single-CTA launch: every level l <= first_level has at
// most kTailCap nodes, so extract + hash + sort + unique run in shared memory.
constexpr int kTailThreads = 1024;
constexpr int kTailCap = 4096;
constexpr int kMaxTailLevels = 8;
constexpr int kTailChildCap = 8192;  // most children of the tail's first level
struct TailLevelOut {
    uint64_t* hashes; uint8_t* masks; uint32_t* children; uint64_t capacity;
    uint64_t* d_nodes; uint64_t* d_unique;
};
struct TailArgs {
    int first_level;
    const uint64_t* child_codes; const uint32_t* child_map; const uint64_t* child_hashes;
    const uint64_t* d_child_n;
    TailLevelOut lv[kMaxTailLevels];
    uint32_t* err;
};
void launch_tail(const TailArgs& a, cudaStream_t s);

// Final layout: word position of every node (exclusive scan of popc+1 over all
// levels concatenated), then headers, child pointers and leaves.
// Node levels root first: level l holds nodes [lv_off[l], lv_off[l + 1]) of
// the concatenated numbering, their masks at lv_masks[l] and children (8 per
// node, ids in level l + 1 or leaf ids) at lv_children[l]: slices of one
// DAG's arrays, or a call's separate per-level pools.
constexpr int kFinalMaxLevels = 24;
struct FinalArgs {
    const uint8_t* lv_masks[kFinalMaxLevels];
    const uint32_t* lv_children[kFinalMaxLevels];
    uint64_t lv_off[kFinalMaxLevels + 1];
    int num_levels;
    uint64_t num_nodes;  // lv_off[num_levels]
    // Positions before the host knows the counts: when non-null, the nodes per
    // level on the device, and lv_off is not read.
    const uint64_t* d_level_n;
    const uint64_t* leaves; uint64_t num_leaves;
    uint32_t* word_pos;  // num_nodes + 1
    uint64_t* d_total;   // exact 64-bit sum of node words
    uint32_t* words;
    uint64_t* status; uint32_t* tile_counter; uint32_t* err; int grid_scan, grid_write;
};
void launch_final_positions(const FinalArgs& a, cudaStream_t s);
void launch_final_write(const FinalArgs& a, cudaStream_t s);

// Gathers / copies used by the merge and the compaction of level outputs.
void launch_remap_children(const uint32_t* in, const uint32_t* map, uint32_t* out, uint64_t n_nodes,
                           cudaStream_t s);
void launch_iota_offset(uint32_t* out, uint64_t n, uint32_t offset, cudaStream_t s);

// Several device-to-device copies in one launch (a DAG's levels out of the
// call's scratch): each copy moves 16, 8, 4 or 1 bytes per thread step,
// whichever its addresses and size allow.
struct CopySeg {
    const void* src;
    void* dst;
    uint64_t bytes;
};
constexpr int kMaxCopySegs = 64;
constexpr uint64_t kCopyPiece = 32768;  // bytes per CTA: eight 16-byte units per thread
struct CopyTable {
    CopySeg seg[kMaxCopySegs];
    uint32_t first_cta[kMaxCopySegs + 1];  // filled by launch_copy_segments
    int count;
    uint64_t* lit_dst;  // and up to 24 words given by value (a DAG's level offsets)
    uint64_t lit[24];
    int lit_count;
};
void launch_copy_segments(const CopyTable& t, cudaStream_t s);
// n words to pinned host memory (a call's counts).
void launch_publish(const uint64_t* in, uint64_t* host, uint32_t n, cudaStream_t s);

void kernels_configure();

// Resident CTAs per SM of the persistent kernels (for grid sizing).
enum KernelId { kKernelLeafBuild = 0, kKernelExtract = 1, kKernelUnique = 2, kKernelFinalScan = 3, kKernelFinalWrite = 4 };
int occupancy_kernel(int which);

}  // namespace dagc
