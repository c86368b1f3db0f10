// The node levels of the hash-set form, for sm_103a. Replaces, per level, the
// reference's ExtractLevel + ComputeHashes (src/DAGCompression.cu:916-974,
// :827-833, :765-774) and SortLevel (:864-914): one node per distinct child
// code >> 3, its hash, the distinct hashes in ascending order with their masks
// and child ids.
//
// A node's hash needs its children's hashes, not their ids, so the levels fall
// into two parts:
//
//   extract_nodes, one launch per level, bottom up: from the children's sorted
//   codes and their hashes (the leaf masks below the last level), both read in
//   order, the nodes' codes and hashes, child masks and first child;
//   tail_nodes: the same for every level from the first one of at most
//   kTailCap children up to the root, in one CTA;
//
//   then, for a whole group of levels at once (all of them, unless the bounds
//   are large):
//   nodes_insert  every node's hash into its level's part of the hash table
//                 (linear probing, atomicCAS); the first inserter is the
//                 hash's representative and appends it to the bucket of its
//                 top bits;
//   nodes_order   ranks each bucket: the distinct hashes in order, and their
//                 ids and representatives to the table;
//   nodes_finish  every node reads its id and its children's ids through the
//                 table; representatives write their mask and children at
//                 their id, the others are compared with theirs in full.
//
// Nothing here waits for the leaves' order until nodes_finish, so the first
// part can run beside it. When each level was deduplicated before the next was
// extracted (four launches per level, and the tail's sorts one after another),
// the levels of a 512^3 terrain took 107 us, now 68 (and half of that beside the
// leaves: the call 217 -> 143 by that step); of the 8192^3 soup 2.36 ms, now 1.64.

#include "dagc_device.cuh"
#include "dagc_kernels.h"
#include "dagc_launch.h"

#include <algorithm>

namespace dagc {
namespace {

// ------------------------------------------------------------- extraction --
constexpr int kXThreads = 256;
constexpr int kXWarps = kXThreads / 32;
constexpr int kXRows = kScanTile / kXThreads;  // rows of 256 children per tile
constexpr int kXHalo = 7;                      // children of the tile's last node in the next tile
static_assert(kXRows * kXWarps == 64, "two counts per lane of the scanning warp");

struct NodesSmem {
    uint64_t codes[kScanTile + 8];
    uint64_t hash[kScanTile + 8];
    uint16_t head[kScanTile];     // first child of each node that starts in the tile, in order
    uint32_t cnt[64];             // heads per row and warp, then the heads before
    uint32_t slot, heads;
    uint64_t p_base;
};

// The node whose first child is at i of (codes, hash), with children below
// `end` of the arrays: its mask and hash. Codes ascend, so a node's children
// are in slot order.
__device__ __forceinline__ uint64_t node_hash(const uint64_t* codes, const uint64_t* hash, uint32_t i, uint32_t end,
                                              uint32_t* mask) {
    const uint64_t par = codes[i] >> 3;
    uint32_t m = 0;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k)
        if (i + k < end && (codes[i + k] >> 3) == par) m |= 1u << (uint32_t)(codes[i + k] & 7);
    uint64_t h[8];
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) h[c] = (m >> c) & 1u ? hash[i + __popc(m & ((1u << c) - 1u))] : 0ull;
    *mask = m;
    return hash_children(h);
}

// What bounds it: at large levels the barriers of a tile around its look-back
// (20 bytes read per child, 21 written per node); at small ones its chain of
// round trips.
__global__ void __launch_bounds__(kXThreads, 4) extract_nodes(NodesArgs a) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    NodesSmem& S = *reinterpret_cast<NodesSmem*>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t count = *a.d_n, n = count < a.n_bound ? count : a.n_bound;
    if (n <= a.tail_max) return;  // the tail takes this level and those above it
    const uint32_t ntiles = scan_tiles(n);
    if (blockIdx.x >= ntiles) return;  // grids are sized by an upper bound on n
    bool overflow = false;
    while (true) {
        if (tid == 0) S.slot = atomicAdd(a.tile_counter, 1u);
        __syncthreads();
        const uint32_t tile = S.slot;
        if (tile >= ntiles) break;
        const uint64_t base = (uint64_t)tile * kScanTile;
        const uint32_t tile_n = (uint32_t)(n - base < (uint64_t)kScanTile ? n - base : (uint64_t)kScanTile);
        // The tile and the few children after it that may belong to its last node.
        const uint32_t have = (uint32_t)(n - base < (uint64_t)(kScanTile + kXHalo) ? n - base : (uint64_t)(kScanTile + kXHalo));
        uint64_t c[kXRows], h[kXRows];
#pragma unroll
        for (int k = 0; k < kXRows; ++k) {
            const uint32_t i = k * kXThreads + tid;
            if (i < tile_n) { c[k] = a.child_codes[base + i]; h[k] = a.child_hashes[base + i]; }
        }
        if (tid < kXHalo && kScanTile + tid < have) {
            S.codes[kScanTile + tid] = a.child_codes[base + kScanTile + tid];
            S.hash[kScanTile + tid] = a.child_hashes[base + kScanTile + tid];
        }
        const uint64_t before = base > 0 ? a.child_codes[base - 1] >> 3 : ~0ull;
#pragma unroll
        for (int k = 0; k < kXRows; ++k) {
            const uint32_t i = k * kXThreads + tid;
            if (i < tile_n) { S.codes[i] = c[k]; S.hash[i] = h[k]; }
        }
        __syncthreads();
        uint32_t heads[kXRows];
#pragma unroll
        for (int k = 0; k < kXRows; ++k) {
            const uint32_t i = k * kXThreads + tid;
            const bool head = i < tile_n && (c[k] >> 3) != (i ? S.codes[i - 1] >> 3 : before);
            heads[k] = __ballot_sync(0xFFFFFFFFu, head);
            if (lane == 0) S.cnt[k * kXWarps + warp] = __popc(heads[k]);
        }
        __syncthreads();
        if (warp == 0) {
            const uint32_t n0 = S.cnt[2 * lane], n1 = S.cnt[2 * lane + 1];
            uint32_t x = n0 + n1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            S.cnt[2 * lane] = x - n0 - n1;
            S.cnt[2 * lane + 1] = x - n1;
            const uint32_t total = __shfl_sync(0xFFFFFFFFu, x, 31);
            if (lane == 0) S.heads = total;
            const uint64_t pb = sv_lookback(a.status, tile, total, a.err);
            if (lane == 0) S.p_base = pb;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kXRows; ++k)
            if ((heads[k] >> lane) & 1u)
                S.head[S.cnt[k * kXWarps + warp] + __popc(heads[k] & lanemask_lt())] = (uint16_t)(k * kXThreads + tid);
        __syncthreads();
        const uint32_t total = S.heads;
        const uint64_t p_base = S.p_base;
        for (uint32_t x = tid; x < total; x += kXThreads) {
            const uint64_t p = p_base + x;
            if (p >= a.out_capacity) { overflow = true; break; }
            const uint32_t i = S.head[x];
            uint32_t mask;
            const uint64_t hv = node_hash(S.codes, S.hash, i, have, &mask);
            a.node_codes[p] = S.codes[i] >> 3;
            a.out.hash[p] = hv;
            a.out.mask[p] = (uint8_t)mask;
            a.out.first[p] = (uint32_t)(base + i);
        }
        if (tid == 0 && base + tile_n == n) {
            const uint64_t cnt = p_base + total;
            *a.d_out_n = cnt < a.out_capacity ? cnt : a.out_capacity;
        }
        __syncthreads();
    }
    if (overflow) atomicOr(a.err, kErrCapacity);
}

// ------------------------------------------------------------------- tail --
// Children and nodes of a level in shared memory; the nodes are the next
// level's children.
struct TailNodesSmem {
    uint64_t code[2][kTailCap], hash[2][kTailCap];
    uint16_t first[kTailCap];
    uint32_t cnt[kTailCap / 32];  // heads per row and warp
};
static_assert(sizeof(TailNodesSmem) <= 227 * 1024, "tail state fits one CTA's shared memory");
constexpr int kTailRows = kTailCap / kTailThreads;

// One level of at most 32 children, by one warp: a lane per child, then a lane
// per node. Returns the number of nodes.
__device__ __forceinline__ uint32_t tail_level_warp(TailNodesSmem& S, int from, uint32_t nc, const TailNodesLevel& out) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t* codes = S.code[from];
    const bool head = lane < nc && (lane == 0 || (codes[lane] >> 3) != (codes[lane - 1] >> 3));
    const uint32_t heads = __ballot_sync(0xFFFFFFFFu, head);
    if (head) S.first[__popc(heads & lanemask_lt())] = (uint16_t)lane;
    __syncwarp();
    const uint32_t n = __popc(heads);
    if (lane < n && lane < out.capacity) {
        const uint32_t i = S.first[lane];
        uint32_t mask;
        const uint64_t hv = node_hash(codes, S.hash[from], i, nc, &mask);
        S.code[from ^ 1][lane] = codes[i] >> 3;
        S.hash[from ^ 1][lane] = hv;
        out.out.hash[lane] = hv;
        out.out.mask[lane] = (uint8_t)mask;
        out.out.first[lane] = i;
    }
    __syncwarp();
    return n;
}

// Bound by latency: three barriers per level, none once a level has at most 32
// children (one warp does the rest).
__global__ void __launch_bounds__(kTailThreads) tail_nodes(TailNodesArgs a) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TailNodesSmem& S = *reinterpret_cast<TailNodesSmem*>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // The first level: the largest one whose children fit (every warp looks).
    uint64_t cnt_l = 0;
    if ((int)lane < a.levels) cnt_l = *a.lv[lane].d_child_n;
    const uint32_t fit = __ballot_sync(0xFFFFFFFFu, cnt_l > 0 && cnt_l <= (uint64_t)kTailCap);
    if (!fit) return;  // no child of any level: nothing was extracted
    const int first = 31 - __clz(fit);
    uint32_t nc = (uint32_t)__shfl_sync(0xFFFFFFFFu, cnt_l, first);
    const uint64_t* gc = a.lv[first].child_codes;
    const uint64_t* gh = a.lv[first].child_hashes;
#pragma unroll
    for (int k = 0; k < kTailRows; ++k) {
        const uint32_t i = k * kTailThreads + tid;
        if (i < nc) { S.code[0][i] = gc[i]; S.hash[0][i] = gh[i]; }
    }
    __syncthreads();
    bool overflow = false;
    int from = 0, l = first;
    for (; l >= 0 && nc > 32; --l, from ^= 1) {
        const TailNodesLevel& out = a.lv[l];
        const uint64_t* codes = S.code[from];
        uint32_t heads[kTailRows];
#pragma unroll
        for (int k = 0; k < kTailRows; ++k) {
            const uint32_t i = k * kTailThreads + tid;
            const bool head = i < nc && (i == 0 || (codes[i] >> 3) != (codes[i - 1] >> 3));
            heads[k] = __ballot_sync(0xFFFFFFFFu, head);
            if (lane == 0) S.cnt[k * 32 + warp] = __popc(heads[k]);
        }
        __syncthreads();
        // Every warp scans the counts (kTailRows per lane, rows before warps).
        uint32_t v[kTailRows], sum = 0;
#pragma unroll
        for (int q = 0; q < kTailRows; ++q) { v[q] = S.cnt[lane * kTailRows + q]; sum += v[q]; }
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
            if (lane >= (uint32_t)o) x += y;
        }
        const uint32_t n = __shfl_sync(0xFFFFFFFFu, x, 31);
        x -= sum;
#pragma unroll
        for (int k = 0; k < kTailRows; ++k) {
            // Heads before (row k, this warp): entry k * 32 + warp.
            const uint32_t e = k * 32 + warp;
            uint32_t before = x;
#pragma unroll
            for (int q = 0; q < kTailRows; ++q)
                if ((uint32_t)q < e % kTailRows) before += v[q];
            before = __shfl_sync(0xFFFFFFFFu, before, e / kTailRows);
            if ((heads[k] >> lane) & 1u) S.first[before + __popc(heads[k] & lanemask_lt())] = (uint16_t)(k * kTailThreads + tid);
        }
        __syncthreads();
        for (uint32_t p = tid; p < n; p += kTailThreads) {
            if (p >= out.capacity) { overflow = true; break; }
            const uint32_t i = S.first[p];
            uint32_t mask;
            const uint64_t hv = node_hash(codes, S.hash[from], i, nc, &mask);
            S.code[from ^ 1][p] = codes[i] >> 3;
            S.hash[from ^ 1][p] = hv;
            out.out.hash[p] = hv;
            out.out.mask[p] = (uint8_t)mask;
            out.out.first[p] = i;
        }
        nc = n < out.capacity ? n : (uint32_t)out.capacity;
        if (tid == 0) *out.d_nodes = nc;
        __syncthreads();
    }
    if (warp == 0) {
        for (; l >= 0; --l, from ^= 1) {
            const TailNodesLevel& out = a.lv[l];
            const uint32_t n = tail_level_warp(S, from, nc, out);
            if (n > out.capacity) overflow = true;
            nc = n < out.capacity ? n : (uint32_t)out.capacity;
            if (lane == 0) *out.d_nodes = nc;
        }
    }
    if (overflow) atomicOr(a.err, kErrCapacity);
}

// ------------------------------------------------------------------ dedup --
// The group's levels on the device: nodes, and where each level's 128-item
// chunks, buckets and table slots start.
constexpr int kGIlp = 4;                  // items per lane in flight
constexpr uint32_t kGChunk = 32 * kGIlp;  // items of a warp and round, of one level
struct GroupSmem {
    uint32_t n[kNodeLevels];
    uint32_t chunk0[kNodeLevels + 1], bucket0[kNodeLevels + 1];
    uint64_t table0[kNodeLevels + 1];
    int shift[kNodeLevels];               // bucket of a hash: hash >> shift
    uint32_t ok;
};
static_assert(kNodeLevels < 32, "a lane per level");

// The whole CTA; false when the group does not fit its table or buckets (every
// kernel of the group then returns; nodes_insert flags it).
__device__ __forceinline__ bool load_group(const GroupDedupArgs& a, GroupSmem& G) {
    if (threadIdx.x < 32) {
        const uint32_t l = threadIdx.x;
        uint64_t n = 0;
        uint32_t nb = 0;
        int shift = 64;
        uint64_t slots = 0;
        bool fits = true;
        if ((int)l < a.levels) {
            n = *a.lv[l].d_n;
            if (n > a.lv[l].capacity) n = a.lv[l].capacity;
            fits = n <= kDedupMaxItems;
            if (n) {
                nb = topbit_buckets(n, &shift);
                slots = table_size_for(n, false);
            }
        }
        uint32_t chunks = (uint32_t)((n + kGChunk - 1) / kGChunk), c = chunks, b = nb;
        uint64_t t = slots;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t yc = __shfl_up_sync(0xFFFFFFFFu, c, o), yb = __shfl_up_sync(0xFFFFFFFFu, b, o);
            const uint64_t yt = __shfl_up_sync(0xFFFFFFFFu, t, o);
            if (l >= (uint32_t)o) { c += yc; b += yb; t += yt; }
        }
        if ((int)l < a.levels) {
            G.n[l] = (uint32_t)n;
            G.shift[l] = shift;
            G.chunk0[l + 1] = c;
            G.bucket0[l + 1] = b;
            G.table0[l + 1] = t;
        }
        if (l == 0) { G.chunk0[0] = 0; G.bucket0[0] = 0; G.table0[0] = 0; }
        const bool all = __all_sync(0xFFFFFFFFu, fits);
        const uint32_t nbt = __shfl_sync(0xFFFFFFFFu, b, 31);
        const uint64_t tt = __shfl_sync(0xFFFFFFFFu, t, 31);
        const uint32_t ct = __shfl_sync(0xFFFFFFFFu, c, 31);
        if (l == 0)
            G.ok = all && tt <= a.table_cap && (uint64_t)nbt * kDedupTopBitCap <= a.bucket_area && nbt <= a.bucket_cap &&
                   (uint64_t)ct * kGChunk <= a.slot_cap;
    }
    __syncthreads();
    return G.ok != 0;
}
__device__ __forceinline__ int level_of_chunk(const GroupSmem& G, int levels, uint32_t c) {
    int l = 0;
    while (l + 1 < levels && c >= G.chunk0[l + 1]) ++l;
    return l;
}

// Large levels are bound by the table's random accesses (a slot and the next
// one per probe, an atomicCAS per new hash), small ones by the chain of a
// probe, a claim and a bucket reservation. Each lane runs kGIlp probe chains
// side by side; levels of up to 2^20 nodes claim at once (one round trip),
// larger ones read first (L2 atomic throughput).
__global__ void __launch_bounds__(256, 4) nodes_insert(GroupDedupArgs a) {
    pdl_prologue();
    __shared__ GroupSmem G;
    if (!load_group(a, G)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(a.err, kErrFallback);
        return;
    }
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    bool full = false;
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < G.chunk0[a.levels]; c += warps) {
        const int l = level_of_chunk(G, a.levels, c);
        const uint32_t n = G.n[l], i0 = (c - G.chunk0[l]) * kGChunk + lane;
        const uint32_t S = (uint32_t)(G.table0[l + 1] - G.table0[l]);
        uint64_t* keys = a.table_key + 2 * G.table0[l];
        const uint64_t* hashes = a.lv[l].nodes.hash;
        const bool read_first = n > kDedupClaimFirstMax;
        uint64_t h[kGIlp];
        uint32_t s[kGIlp];
        bool pend[kGIlp], won[kGIlp];
#pragma unroll
        for (int k = 0; k < kGIlp; ++k) {
            const uint32_t i = i0 + k * 32;
            pend[k] = i < n;
            won[k] = false;
            h[k] = pend[k] ? hashes[i] : 0;  // hashes are never 0 (an empty slot)
            s[k] = (uint32_t)home_slot(h[k], S);
        }
        for (uint32_t round = 0; round < S; ++round) {
            bool claim[kGIlp];
            uint64_t cur[kGIlp], nxt[kGIlp];
#pragma unroll
            for (int k = 0; k < kGIlp; ++k) {
                claim[k] = pend[k];
                cur[k] = 0;
                nxt[k] = 0;
            }
            if (read_first) {
#pragma unroll
                for (int k = 0; k < kGIlp; ++k) {
                    if (!pend[k]) continue;
                    cur[k] = ld_relaxed(keys + 2ull * s[k]);
                    nxt[k] = ld_relaxed(keys + 2ull * next_slot(s[k], S));
                }
                // In probe order: a match ends the search; the first empty
                // slot is claimed; two other keys move the probe on by two.
#pragma unroll
                for (int k = 0; k < kGIlp; ++k) {
                    if (!pend[k]) continue;
                    if (cur[k] == h[k]) { pend[k] = claim[k] = false; continue; }
                    if (cur[k] == 0) continue;
                    s[k] = next_slot(s[k], S);
                    if (nxt[k] == h[k]) { pend[k] = claim[k] = false; continue; }
                    if (nxt[k] != 0) { s[k] = next_slot(s[k], S); claim[k] = false; }
                }
            }
#pragma unroll
            for (int k = 0; k < kGIlp; ++k)
                if (claim[k]) cur[k] = atomicCAS((unsigned long long*)(keys + 2ull * s[k]), 0ull, (unsigned long long)h[k]);
            bool any = false;
#pragma unroll
            for (int k = 0; k < kGIlp; ++k) {
                if (!pend[k]) continue;
                if (claim[k] && (cur[k] == 0 || cur[k] == h[k])) { won[k] = cur[k] == 0; pend[k] = false; continue; }
                if (claim[k]) s[k] = next_slot(s[k], S);
                any = true;
            }
            if (!any) break;
        }
        // Every winner's bucket slot is reserved before any is used.
        uint32_t bslot[kGIlp], b[kGIlp];
#pragma unroll
        for (int k = 0; k < kGIlp; ++k) {
            b[k] = G.bucket0[l] + (G.shift[l] >= 64 ? 0u : (uint32_t)(h[k] >> G.shift[l]));
            bslot[k] = won[k] ? atomicAdd(a.bucket_count + b[k], 1u) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kGIlp; ++k) {
            const uint32_t i = i0 + k * 32;
            if (i >= n) continue;
            if (pend[k]) full = true;  // cannot happen at half load; rerun rather than guess
            const uint32_t slot = (uint32_t)G.table0[l] + s[k];
            a.item_slot[(uint64_t)G.chunk0[l] * kGChunk + i] = pend[k] ? 0xFFFFFFFFu : slot;
            if (!won[k]) continue;
            if (bslot[k] < kDedupTopBitCap)
                a.bucket[(uint64_t)b[k] * kDedupTopBitCap + bslot[k]] = make_uint4((uint32_t)h[k], (uint32_t)(h[k] >> 32), slot, i);
            else
                full = true;
        }
    }
    if (full) atomicOr(a.err, kErrFallback);
}

// Each CTA takes a contiguous range of the group's buckets; a bucket's keys are
// distinct, so a key's rank is the number of smaller keys in its bucket. The
// hashes are uniform: the kOSub sub-buckets of their next bits hold a few keys
// each, and only those are compared (238 keys per bucket in the 8192^3 soup's
// largest level: 139 us comparing whole buckets, now 92). Slot, representative
// and id go out as one 16-byte store that also empties the slot.
constexpr int kOThreads = 256;
constexpr int kOSubLog = 6;
constexpr uint32_t kOSub = 1u << kOSubLog;
__global__ void __launch_bounds__(kOThreads) nodes_order(GroupDedupArgs a) {
    pdl_prologue();
    __shared__ GroupSmem G;
    __shared__ uint64_t key[kDedupTopBitCap];
    __shared__ uint16_t ord[kDedupTopBitCap];  // keys in sub-bucket order
    __shared__ uint32_t sub_cnt[kOSub], sub0[kOSub + 1];
    __shared__ uint32_t red[kOThreads / 32];
    if (!load_group(a, G)) return;
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint32_t nb = G.bucket0[a.levels];
    const uint32_t b0 = (uint32_t)((uint64_t)nb * blockIdx.x / gridDim.x);
    const uint32_t b1 = (uint32_t)((uint64_t)nb * (blockIdx.x + 1) / gridDim.x);
    if (b0 >= b1) return;
    int l = 0;
    while (b0 >= G.bucket0[l + 1]) ++l;
    // Keys in the level's buckets before this range (8 independent loads per
    // thread in flight).
    uint32_t part = 0;
    for (uint32_t x0 = G.bucket0[l]; x0 < b0; x0 += 8 * kOThreads) {
        uint32_t c[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const uint32_t x = x0 + u * kOThreads + tid;
            c[u] = x < b0 ? a.bucket_count[x] : 0u;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) part += min(c[u], kDedupTopBitCap);
    }
    part = __reduce_add_sync(0xFFFFFFFFu, part);
    if (lane == 0) red[warp] = part;
    __syncthreads();
    uint64_t start = 0;
    for (int w = 0; w < kOThreads / 32; ++w) start += red[w];
    uint4* slot4 = reinterpret_cast<uint4*>(a.table_key);
    bool bad = false;
    for (uint32_t b = b0; b < b1; ++b) {
        while (b >= G.bucket0[l + 1]) { ++l; start = 0; }
        const GroupLevel& lv = a.lv[l];
        const uint32_t cnt = min(a.bucket_count[b], kDedupTopBitCap);
        const uint4* ent = a.bucket + (uint64_t)b * kDedupTopBitCap;
        // Sub-bucket of a key: the bits after the bucket's.
        const int sub_shift = G.shift[l] - kOSubLog;
        __syncthreads();  // the previous bucket's keys are no longer read
        if (tid < kOSub) sub_cnt[tid] = 0;
        __syncthreads();
        for (uint32_t j = tid; j < cnt; j += kOThreads) {
            const uint4 e = ent[j];
            const uint64_t k = (uint64_t)e.x | (uint64_t)e.y << 32;
            key[j] = k;
            atomicAdd(&sub_cnt[(uint32_t)(k >> sub_shift) & (kOSub - 1)], 1u);
        }
        __syncthreads();
        if (warp == 0) {
            const uint32_t n0 = sub_cnt[2 * lane], n1 = sub_cnt[2 * lane + 1];
            uint32_t x = n0 + n1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            const uint32_t s0 = x - n0 - n1;
            sub_cnt[2 * lane] = sub0[2 * lane] = s0;
            sub_cnt[2 * lane + 1] = sub0[2 * lane + 1] = s0 + n0;
            if (lane == 31) sub0[kOSub] = x;
        }
        __syncthreads();
        for (uint32_t j = tid; j < cnt; j += kOThreads)
            ord[atomicAdd(&sub_cnt[(uint32_t)(key[j] >> sub_shift) & (kOSub - 1)], 1u)] = (uint16_t)j;
        __syncthreads();
        for (uint32_t x = tid; x < cnt; x += kOThreads) {
            const uint32_t j = ord[x];
            const uint2 e = *reinterpret_cast<const uint2*>(&ent[j].z);  // slot, representative
            const uint64_t k = key[j];
            const uint32_t s = (uint32_t)(k >> sub_shift) & (kOSub - 1), s1 = sub0[s + 1];
            uint32_t r = sub0[s];
            for (uint32_t y = sub0[s]; y < s1; ++y) r += key[ord[y]] < k;
            const uint64_t uid = start + r;
            if (uid < lv.capacity && e.x < a.table_cap) {
                lv.out_keys[uid] = k;
                slot4[e.x] = make_uint4(0u, 0u, e.y, (uint32_t)uid);  // empty for the next group (nodes_finish reads only aux)
            } else {
                bad = true;
            }
        }
        start += cnt;
        if (tid == 0 && b + 1 == G.bucket0[l + 1]) {  // the level's last bucket
            if (start > a.uniq_cap) atomicOr(a.err, kErrFallback);
            *lv.d_out_n = start < lv.capacity ? start : lv.capacity;
        }
    }
    if (bad) atomicOr(a.err, kErrCapacity);
}

// A node's child ids by slot, of the items below it: through the map of the
// level below the group for its lowest level, else through the table. The
// children are consecutive items, or (kRefs) any.
template <bool kRefs>
__device__ __forceinline__ void child_ids(const GroupDedupArgs& a, const GroupSmem& G, int l, uint32_t i, uint32_t mask,
                                          uint32_t (&id)[8]) {
    const NodeArrays& nodes = a.lv[l].nodes;
    uint32_t item[8];
    if (kRefs) {
        const uint4* p = reinterpret_cast<const uint4*>(nodes.children + (uint64_t)i * 8);
        const uint4 c0 = p[0], c1 = p[1];
        item[0] = c0.x; item[1] = c0.y; item[2] = c0.z; item[3] = c0.w;
        item[4] = c1.x; item[5] = c1.y; item[6] = c1.z; item[7] = c1.w;
    } else {
        const uint32_t first = nodes.first[i];
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c)
            item[c] = (mask >> c) & 1u ? first + __popc(mask & ((1u << c) - 1u)) : kEmptyChild;
    }
    if (l + 1 == a.levels) {
#pragma unroll
        for (uint32_t c = 0; c < 8; ++c) id[c] = item[c] != kEmptyChild ? a.child_map[item[c]] : kEmptyChild;
        return;
    }
    const uint32_t* slots = a.item_slot + (uint64_t)G.chunk0[l + 1] * kGChunk;
    uint32_t s[8];
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) s[c] = item[c] != kEmptyChild ? slots[item[c]] : 0xFFFFFFFFu;
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c)
        id[c] = s[c] < a.table_cap ? reinterpret_cast<const uint32_t*>(a.table_aux)[4ull * s[c] + 1] : kEmptyChild;
}

// Bound by random reads: per node its slot's aux word and, as somebody's child,
// one more. (Each node is a child once, so no map of a level is needed but for
// the group above.)
template <bool kRefs>
__global__ void __launch_bounds__(256) nodes_finish(GroupDedupArgs a) {
    pdl_prologue();
    __shared__ GroupSmem G;
    if (!load_group(a, G)) return;
    // The bucket counters, read by nodes_order, start the next group at zero.
    for (uint32_t b = blockIdx.x * blockDim.x + threadIdx.x; b < G.bucket0[a.levels]; b += gridDim.x * blockDim.x)
        a.bucket_count[b] = 0;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    bool collision = false;
    for (uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < G.chunk0[a.levels]; c += warps) {
        const int l = level_of_chunk(G, a.levels, c);
        const GroupLevel& lv = a.lv[l];
        const uint32_t n = G.n[l], i0 = (c - G.chunk0[l]) * kGChunk + lane;
        const uint32_t* slots = a.item_slot + (uint64_t)G.chunk0[l] * kGChunk;
        uint32_t s[kGIlp], mask[kGIlp];
        uint64_t aux[kGIlp];
#pragma unroll
        for (int k = 0; k < kGIlp; ++k) {
            const uint32_t i = i0 + k * 32;
            s[k] = i < n ? slots[i] : 0xFFFFFFFFu;
            mask[k] = i < n ? lv.nodes.mask[i] : 0u;
        }
#pragma unroll
        for (int k = 0; k < kGIlp; ++k) aux[k] = s[k] < a.table_cap ? a.table_aux[2ull * s[k]] : ~0ull;
#pragma unroll
        for (int k = 0; k < kGIlp; ++k) {
            const uint32_t i = i0 + k * 32, rep = (uint32_t)aux[k], uid = (uint32_t)(aux[k] >> 32);
            if (i >= n) continue;
            // Ids stay inside the next level's arrays even when a fallback or
            // an error discards this call.
            if (l == 0 && a.map) a.map[i] = uid < lv.capacity ? uid : (uint32_t)(lv.capacity - 1);
            if (s[k] >= a.table_cap || rep >= n || uid >= lv.capacity) continue;  // flagged by the insert or the order
            uint32_t id[8];
            child_ids<kRefs>(a, G, l, i, mask[k], id);
            if (rep == i) {
                lv.out_masks[uid] = (uint8_t)mask[k];
                uint4* d4 = reinterpret_cast<uint4*>(lv.out_children + (uint64_t)uid * 8);
                d4[0] = make_uint4(id[0], id[1], id[2], id[3]);
                d4[1] = make_uint4(id[4], id[5], id[6], id[7]);
            } else {
                uint32_t other[8];
                const uint32_t m = lv.nodes.mask[rep];
                child_ids<kRefs>(a, G, l, rep, m, other);
                collision |= m != mask[k];
#pragma unroll
                for (int q = 0; q < 8; ++q) collision |= id[q] != other[q];
            }
        }
    }
    if (collision) atomicOr(a.err, kErrCollision);
}

// ------------------------------------------------------------------ union --
// The input of item j (off ascending, k + 1 entries).
__device__ __forceinline__ uint32_t input_of(const uint64_t* off, uint32_t k, uint64_t j) {
    uint32_t lo = 0, hi = k;  // off[lo] <= j < off[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(off + mid) <= j) lo = mid; else hi = mid;
    }
    return lo;
}
struct MergeTable {
    const uint64_t *hashes, *children, *masks, *leaves, *first, *item;
    __device__ explicit MergeTable(const MergeArgs& a)
        : hashes(a.table), children(a.table + a.k), masks(a.table + 2ull * a.k), leaves(a.table + 3ull * a.k),
          first(a.table + 4ull * a.k), item(a.table + (4ull + a.levels) * a.k) {}
    __device__ const uint64_t* items(const MergeArgs& a, int l) const { return item + (uint64_t)l * (a.k + 1); }
};

// Every node of every input: hash and mask as they are, children as items of
// the level below. A hash or leaf of 0 would mark an empty slot of the table:
// those go to the radix form.
__global__ void __launch_bounds__(256) merge_gather(MergeArgs a) {
    pdl_prologue();
    const MergeTable t(a);
    if (blockIdx.x == 0 && (int)threadIdx.x <= a.levels) *a.d_n[threadIdx.x] = a.level0[threadIdx.x + 1] - a.level0[threadIdx.x];
    const uint64_t total = a.level0[a.levels + 1];
    bool zero = false;
    for (uint64_t g = (uint64_t)blockIdx.x * 256 + threadIdx.x; g < total; g += (uint64_t)gridDim.x * 256) {
        int l = 0;
        while (l < a.levels && g >= a.level0[l + 1]) ++l;
        const uint64_t j = g - a.level0[l];
        const uint64_t* off = t.items(a, l);
        const uint32_t i = input_of(off, a.k, j);
        const uint64_t r = j - __ldg(off + i);
        if (l == a.levels) {
            const uint64_t leaf = reinterpret_cast<const uint64_t*>(__ldg(t.leaves + i))[r];
            a.leaves[j] = leaf;
            zero |= leaf == 0;
            continue;
        }
        const uint64_t src = __ldg(t.first + (uint64_t)i * a.levels + l) + r;
        const uint32_t below = (uint32_t)__ldg(t.items(a, l + 1) + i);
        const uint64_t h = reinterpret_cast<const uint64_t*>(__ldg(t.hashes + i))[src];
        const uint4* c = reinterpret_cast<const uint4*>(__ldg(t.children + i)) + 2 * src;
        uint4 c0 = c[0], c1 = c[1];
        auto up = [&](uint32_t& x) { if (x != kEmptyChild) x += below; };
        up(c0.x); up(c0.y); up(c0.z); up(c0.w);
        up(c1.x); up(c1.y); up(c1.z); up(c1.w);
        a.out[l].hash[j] = h;
        a.out[l].mask[j] = reinterpret_cast<const uint8_t*>(__ldg(t.masks + i))[src];
        uint4* d = reinterpret_cast<uint4*>(a.out[l].children + 8 * j);
        d[0] = c0;
        d[1] = c1;
        zero |= h == 0;
    }
    if (zero) atomicOr(a.err, kErrFallback);
}

__global__ void __launch_bounds__(256) merge_roots(MergeArgs a) {
    pdl_prologue();
    const MergeTable t(a);
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < a.k; i += gridDim.x * 256) {
        const uint64_t j = t.items(a, 0)[i];
        const bool any = t.items(a, 0)[i + 1] > j;
        a.root_uid[i] = any ? a.root_map[j] : kEmptyChild;
        a.root_hash[i] = any ? (a.levels ? a.out[0].hash[j] : a.leaves[j]) : 0ull;
    }
}

int g_levels_sms = 152, g_extract_ctas = 4;

}  // namespace

void levels_configure(int sms) {
    g_levels_sms = sms > 0 ? sms : 152;
    cudaFuncSetAttribute(extract_nodes, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(NodesSmem));
    cudaFuncSetAttribute(tail_nodes, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TailNodesSmem));
    int occ = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, extract_nodes, kXThreads, sizeof(NodesSmem)) != cudaSuccess)
        cudaGetLastError();
    g_extract_ctas = occ > 0 ? occ : 1;
}

uint64_t group_slot_items(uint64_t n) { return (n + kGChunk - 1) / kGChunk * kGChunk; }

void launch_extract_nodes(const NodesArgs& a, cudaStream_t s) {
    const uint64_t tiles = scan_tiles(a.n_bound), most = (uint64_t)g_extract_ctas * g_levels_sms;
    launch_pdl(extract_nodes, dim3((unsigned)(tiles < most ? (tiles ? tiles : 1) : most)), dim3(kXThreads), sizeof(NodesSmem), s, a);
}
void launch_tail_nodes(const TailNodesArgs& a, cudaStream_t s) {
    launch_pdl(tail_nodes, dim3(1), dim3(kTailThreads), sizeof(TailNodesSmem), s, a);
}
int launch_group_dedup(const GroupDedupArgs& a, uint64_t items_bound, cudaStream_t s) {
    const uint64_t want = (items_bound + 255) / 256, most = 8ull * g_levels_sms;
    const unsigned g = (unsigned)(want < most ? (want ? want : 1) : most);
    launch_pdl(nodes_insert, dim3(g), dim3(256), 0, s, a);
    const uint64_t buckets = items_bound / 128 + a.levels;
    launch_pdl(nodes_order, dim3((unsigned)(buckets < most ? buckets : most)), dim3(kOThreads), 0, s, a);
    if (a.lv[0].nodes.children) launch_pdl(nodes_finish<true>, dim3(g), dim3(256), 0, s, a);
    else launch_pdl(nodes_finish<false>, dim3(g), dim3(256), 0, s, a);
    return 3;
}

void launch_merge_gather(const MergeArgs& a, cudaStream_t s) {
    const uint64_t want = (a.level0[a.levels + 1] + 255) / 256, most = 8ull * g_levels_sms;
    launch_pdl(merge_gather, dim3((unsigned)(want < most ? (want ? want : 1) : most)), dim3(256), 0, s, a);
}
void launch_merge_roots(const MergeArgs& a, cudaStream_t s) {
    launch_pdl(merge_roots, dim3((a.k + 255) / 256), dim3(256), 0, s, a);
}

}  // namespace dagc
