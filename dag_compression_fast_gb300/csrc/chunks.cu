// Batched form: the leaves of many chunks in one persistent launch, for
// sm_103a. Replaces, for dagc_create_batched, the fragment sort + unique +
// leaf build of every chunk (the reference runs SortKeys, SelectUnique and
// ReduceByKey once per subvolume, src/DAGCompression.cu:1026-1068, called per
// chunk from src/DAG_Compression_Fast.cpp:283-302).
//
// Every chunk's local brick space (bricks = local code >> 6, 3*chunk_depth - 6
// bits) is cut into 2^bin_bits bins of 2^D bricks each, D <= 13, so that one
// bin's leaf masks fit a direct-mapped array in shared memory, with a bitmap
// of the bricks present: the bricks of a bin come out in ascending order by
// walking the bitmap, with no sort. One
// persistent grid takes work items from a device counter, in this order:
//   COUNT(c, t)   a run of tiles of chunk c: the chunk's bin histogram; the
//                 last of c's COUNT items turns it into the bins' starts;
//   SCATTER(c, t) the same run of tiles, after c's starts: fragments to their
//                 bins (one global reservation per bin and tile). A tile is
//                 put in bin order in shared memory first, so that a bin's
//                 fragments leave as one run, while the next tile's are on
//                 their way; a local code of up to 31 bits is a 4-byte word
//                 from here on;
//   LEAVES(c, g)  up to 32 consecutive bins of chunk c, after all of c's SCATTER
//                 items: per bin, OR every fragment's voxel bit into its
//                 brick's mask, then emit the non-empty bricks in order (the
//                 next bin's first fragments on their way).
// Small chunks (one bin) skip COUNT and SCATTER: their LEAVES item reads the
// input. A CTA waits only on items taken before its own (taken by running
// CTAs that wait only on earlier items still), so the waits end; each is
// bounded anyway. Two small launches then pack the bricks of all items into
// one ascending list: a scan of the items' brick counts and a copy.
//
// What bounds it: the chain of barriers and round trips of each tile and bin, at
// 24 bytes of traffic per fragment (read for COUNT, read and 4 bytes written by
// SCATTER, 4 read by LEAVES). 256 chunks of 1024^3, 338M fragments, with the
// scan and the pack: 2.96 ms; 6.70 when every fragment left its SCATTER tile as
// a scattered 8-byte store and every voxel was ORed with an atomic, set or not.
// 318M, the persistent launch alone: 2.86 ms; 3.47 without the loads ahead and
// with a block scan per bin.

#include "dagc_device.cuh"
#include "dagc_kernels.h"
#include "dagc_launch.h"

namespace dagc {
namespace {

constexpr int kT = kChunkThreads;
constexpr int kMaxBins = 1 << kChunkMaxBinBits;
constexpr int kDirect = 1 << kChunkDirectBits;
constexpr int kPerThread = kChunkTile / kT;
static_assert(kChunkTile % kT == 0 && kDirect % kT == 0 && kMaxBins % kT == 0, "chunk shapes");

constexpr int kBitmapWords = kDirect / 32;
static_assert(2 * kBitmapWords <= kT, "a thread per word of both bitmaps");

struct ChunkSmem {
    union {
        struct {
            uint32_t cnt[kMaxBins];     // this tile's fragments per bin, then their offset in the tile
            uint32_t delta[kMaxBins];   // output position - tile position, per bin
            uint32_t stage[kChunkTile]; // the tile's codes in bin order
        } tile;
        struct {
            // One bin's leaf masks, by brick, as two 32-bit halves (native
            // shared atomics), and a bitmap of the bricks present; zero
            // between bins (the emission clears the masks it reads, and the
            // bitmap of the bin before: there are two, taken in turn).
            uint32_t masks[2 * kDirect];
            uint32_t present[2][kBitmapWords];
        } bin;
    };
    uint32_t bin_cnt[kChunkGroupBins];  // fragments of the LEAVES item's bins
    uint32_t scan[34];
    uint32_t item;
    uint32_t flag;
};

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Thread 0 waits (bounded) until *counter reaches target; then the CTA.
__device__ __forceinline__ void wait_counter(const uint32_t* counter, uint32_t target, uint32_t* err) {
    if (threadIdx.x == 0) {
        uint32_t it = 0;
        while (ld_acquire(counter) < target) {
            if (++it > kSpinLimit) { atomicOr(err, kErrTimeout); break; }
            backoff(it);
        }
    }
    __syncthreads();
}

// The chunk of a COUNT / SCATTER item (item_off ascending, k + 1 entries).
__device__ __forceinline__ uint32_t chunk_of_item(const uint32_t* item_off, uint32_t k, uint32_t t) {
    uint32_t lo = 0, hi = k;  // item_off[lo] <= t < item_off[hi]
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(item_off + mid) <= t) lo = mid; else hi = mid;
    }
    return lo;
}

__global__ void __launch_bounds__(kT, 2) chunk_leaves(ChunkArgs a) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ChunkSmem& S = *reinterpret_cast<ChunkSmem*>(smem_raw);
    const uint32_t tid = threadIdx.x;
    const uint32_t nb = 1u << a.bin_bits;
    const int lb = 3 * a.chunk_depth - 6;                    // local brick bits
    const int dbits = lb - a.bin_bits;                        // direct-mapped brick bits of a bin
    const uint32_t dsize = 1u << dbits;
    const uint64_t code_limit = 1ull << (3 * a.chunk_depth);
    // The item count comes from the device (item_off[k]): a recorded graph
    // replayed for other chunk sizes still sees the current one.
    const uint32_t runs = __ldg(a.item_off + a.k);
    const uint32_t total = 2 * runs + a.k * a.groups_per_chunk;
    const uint64_t run_len = (uint64_t)a.run_tiles * kChunkTile;
    const uint32_t lane = tid & 31, warp = tid >> 5;
    constexpr uint32_t kWarps = kT / 32;
    bool bad = false;
    bool clean = false;  // the bin arrays are zero (the tile arrays share their room)
    while (true) {
        if (tid == 0) S.item = atomicAdd(a.work, 1u);
        __syncthreads();
        const uint32_t item = S.item;
        __syncthreads();
        if (item >= total) break;
        if (item < runs) {
            // ----------------------------------------------------- COUNT ----
            clean = false;
            const uint32_t c = chunk_of_item(a.item_off, a.k, item);
            const uint32_t first = __ldg(a.item_off + c), items = __ldg(a.item_off + c + 1) - first;
            const uint64_t c1 = __ldg(a.seg_offsets + c + 1);
            const uint64_t f0 = __ldg(a.seg_offsets + c) + (item - first) * run_len;
            const uint64_t f1 = min(f0 + run_len, c1);
            uint32_t* hist = a.hist + (uint64_t)c * nb;
            for (uint32_t b = tid; b < nb; b += kT) S.tile.cnt[b] = 0;
            __syncthreads();
            constexpr int kIlp = 8;
            for (uint64_t i0 = f0 + tid; i0 < f1; i0 += kIlp * kT) {
                uint64_t code[kIlp];
#pragma unroll
                for (int q = 0; q < kIlp; ++q) code[q] = i0 + q * kT < f1 ? __ldg(a.frags + i0 + q * kT) : 0ull;
#pragma unroll
                for (int q = 0; q < kIlp; ++q) {
                    if (i0 + q * kT >= f1) continue;
                    if (code[q] >= code_limit) bad = true;
                    // (A code out of range goes where SCATTER puts it.)
                    atomicAdd(&S.tile.cnt[(uint32_t)(code[q] & (code_limit - 1)) >> (6 + dbits)], 1u);
                }
            }
            __syncthreads();
            for (uint32_t b = tid; b < nb; b += kT) {
                const uint32_t x = S.tile.cnt[b];
                if (x) atomicAdd(hist + b, x);
            }
            __threadfence();  // every thread's counts land before the item is marked done
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                S.flag = atomicAdd(a.done + c, 1u) == items - 1;
                __threadfence();
            }
            __syncthreads();
            if (S.flag) {
                // The chunk's last COUNT item: bin starts from the histogram.
                constexpr int kPer = kMaxBins / kT;
                uint32_t h[kPer], sum = 0, tot;
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    const uint32_t b = tid * kPer + q;
                    h[q] = b < nb ? ld_relaxed(hist + b) : 0u;
                    sum += h[q];
                }
                uint32_t run = block_exclusive_sum<uint32_t>(sum, S.scan, &tot);
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    const uint32_t b = tid * kPer + q;
                    if (b < nb) st_relaxed(a.cursor + (uint64_t)c * nb + b, run);
                    run += h[q];
                }
                __threadfence();
                __syncthreads();
                if (tid == 0) {
                    __threadfence();
                    atomicAdd(a.done + 2 * a.k + c, 1u);
                }
            }
            continue;
        }
        if (item < 2 * runs) {
            // --------------------------------------------------- SCATTER ----
            clean = false;
            const uint32_t t = item - runs;
            const uint32_t c = chunk_of_item(a.item_off, a.k, t);
            const uint64_t c0 = __ldg(a.seg_offsets + c), c1 = __ldg(a.seg_offsets + c + 1);
            const uint64_t f0 = c0 + (t - __ldg(a.item_off + c)) * run_len;
            const uint64_t f1 = min(f0 + run_len, c1);
            uint32_t* out = a.scratch + c0;
            const uint32_t room = (uint32_t)(c1 - c0);
            const int bin_shift = 6 + dbits;
            const uint32_t code_mask = (uint32_t)(code_limit - 1);  // the low 32 bits hold a code whole (3 * chunk_depth <= 31)
            uint32_t code[kPerThread], rank[kPerThread];
            uint32_t fn = (uint32_t)min((uint64_t)kChunkTile, f1 - f0);
#pragma unroll
            for (int q = 0; q < kPerThread; ++q)
                code[q] = q * kT + tid < fn ? (uint32_t)__ldcs(a.frags + f0 + q * kT + tid) & code_mask : 0u;
            for (uint32_t b = tid; b < nb; b += kT) S.tile.cnt[b] = 0;
            wait_counter(a.done + 2 * a.k + c, 1u, a.err);  // the bins' starts; also orders the zeros above
            for (uint64_t f = f0; f < f1; f += kChunkTile) {
#pragma unroll
                for (int q = 0; q < kPerThread; ++q)
                    if (q * kT + tid < fn) rank[q] = atomicAdd(&S.tile.cnt[code[q] >> bin_shift], 1u);
                __syncthreads();
                constexpr int kPer = kMaxBins / kT;
                uint32_t n[kPer], g[kPer], sum = 0, tot;
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    const uint32_t b = tid * kPer + q;
                    n[q] = b < nb ? S.tile.cnt[b] : 0u;
                    g[q] = n[q] ? atomicAdd(a.cursor + (uint64_t)c * nb + b, n[q]) : 0u;
                    sum += n[q];
                }
                uint32_t run = block_exclusive_sum<uint32_t>(sum, S.scan, &tot);
#pragma unroll
                for (int q = 0; q < kPer; ++q) {
                    const uint32_t b = tid * kPer + q;
                    if (b < nb) {
                        S.tile.cnt[b] = run;
                        S.tile.delta[b] = g[q] - run;
                    }
                    run += n[q];
                }
                __syncthreads();
#pragma unroll
                for (int q = 0; q < kPerThread; ++q)
                    if (q * kT + tid < fn) S.tile.stage[S.tile.cnt[code[q] >> bin_shift] + rank[q]] = code[q];
                __syncthreads();
                const uint32_t m = fn;
                const uint64_t next = f + kChunkTile;
                fn = next < f1 ? (uint32_t)min((uint64_t)kChunkTile, f1 - next) : 0u;
#pragma unroll
                for (int q = 0; q < kPerThread; ++q)
                    code[q] = q * kT + tid < fn ? (uint32_t)__ldcs(a.frags + next + q * kT + tid) & code_mask : 0u;
                for (uint32_t b = tid; b < nb; b += kT) S.tile.cnt[b] = 0;
#pragma unroll 4
                for (uint32_t q = tid; q < m; q += kT) {
                    const uint32_t x = S.tile.stage[q];
                    const uint32_t dst = S.tile.delta[x >> bin_shift] + q;
                    if (dst < room) out[dst] = x;
                    else bad = true;  // only after a timed-out wait
                }
                __syncthreads();
            }
            __threadfence();  // every thread's fragments land before the item is marked done
            __syncthreads();
            if (tid == 0) {
                __threadfence();
                atomicAdd(a.done + a.k + c, 1u);
            }
            continue;
        }
        // --------------------------------------------------------- LEAVES ----
        if (!clean) {
            for (uint32_t x = tid; x < 2u * kDirect; x += kT) S.bin.masks[x] = 0;
            if (tid < 2u * kBitmapWords) (&S.bin.present[0][0])[tid] = 0;
            clean = true;
        }
        const uint32_t gi = item - 2 * runs;
        const uint32_t c = gi / a.groups_per_chunk, g = gi % a.groups_per_chunk;
        const uint64_t c0 = __ldg(a.seg_offsets + c), c1 = __ldg(a.seg_offsets + c + 1);
        const uint32_t b0 = g * a.group_bins, b1 = min(nb, b0 + a.group_bins);
        const uint64_t pbase = __ldg(a.seg_code + c) << (a.seg_shift - 6);  // global brick of local brick 0
        const uint32_t* hist = a.hist + (uint64_t)c * nb;
        uint64_t gstart = c0;  // fragment offset of bin b0 (and of the group's bricks)
        if (nb > 1) {
            const uint32_t items = __ldg(a.item_off + c + 1) - __ldg(a.item_off + c);
            if (items) wait_counter(a.done + a.k + c, items, a.err);
            if (tid < b1 - b0) S.bin_cnt[tid] = ld_relaxed(hist + b0 + tid);
            // A bin's cursor ends at its start plus its count.
            if (items) gstart += ld_relaxed(a.cursor + (uint64_t)c * nb + b0) - ld_relaxed(hist + b0);
        }
        __syncthreads();
        // The first kIlp fragments per thread of a bin are fetched while the
        // bin before is emitted.
        constexpr int kIlp = 8;
        uint32_t code[kIlp];
        auto bin_count = [&](uint32_t b) -> uint64_t { return nb > 1 ? (uint64_t)S.bin_cnt[b - b0] : c1 - c0; };
        auto next_bin = [&](uint32_t b) -> uint32_t {  // the first nonempty bin from b on
            while (b < b1 && bin_count(b) == 0) ++b;
            return b;
        };
        auto fetch = [&](uint64_t from, uint64_t i0, uint64_t cnt) {
#pragma unroll
            for (int u = 0; u < kIlp; ++u) {
                const uint64_t i = i0 + (uint64_t)u * kT;
                code[u] = 0;
                if (i >= cnt) continue;
                if (nb > 1) {
                    code[u] = __ldcg(a.scratch + from + i);
                } else {
                    const uint64_t full = __ldg(a.frags + from + i);
                    if (full >= code_limit) bad = true;
                    code[u] = (uint32_t)full;
                }
            }
        };
        uint32_t running = 0, turn = 0;
        uint64_t fstart = gstart;
        uint32_t b = next_bin(b0);
        uint64_t cnt = b < b1 ? bin_count(b) : 0;
        if (fstart + cnt > c1) { bad = true; b = b1; }  // only after a timed-out wait
        if (b < b1) fetch(fstart, tid, cnt);
        while (b < b1) {
            // The voxel bit goes to its brick's low or high half where it is
            // not set yet (voxels repeat); the first bit of a half marks the
            // brick present.
            uint32_t* present = S.bin.present[turn];
            for (uint64_t i0 = tid;;) {
#pragma unroll
                for (int u = 0; u < kIlp; ++u) {
                    if (i0 + (uint64_t)u * kT >= cnt) continue;
                    const uint32_t e = (code[u] >> 6) & (dsize - 1);
                    uint32_t* half = &S.bin.masks[2 * e + ((code[u] >> 5) & 1u)];
                    const uint32_t bit = 1u << (code[u] & 31u);
                    const uint32_t seen = *reinterpret_cast<volatile uint32_t*>(half);
                    if (seen & bit) continue;
                    if (atomicOr(half, bit) == 0) atomicOr(&present[e >> 5], 1u << (e & 31));
                }
                i0 += kIlp * kT;
                if (i0 >= cnt) break;
                fetch(fstart, i0, cnt);
            }
            const uint32_t bin = b;
            fstart += cnt;
            b = next_bin(b + 1);
            cnt = b < b1 ? bin_count(b) : 0;
            if (fstart + cnt > c1) { bad = true; b = b1; }
            if (b < b1) fetch(fstart, tid, cnt);
            __syncthreads();
            // The bin's bricks in order: warp w emits bitmap words [16w, 16w +
            // 16), a lane per brick. Every warp counts the bricks before its
            // words, and all of them, from the bitmap.
            constexpr uint32_t kWordsPerWarp = kBitmapWords / kWarps;
            static_assert(kWordsPerWarp <= 32, "a lane per word of a warp");
            const uint32_t w0 = warp * kWordsPerWarp;
            const uint32_t own = lane < kWordsPerWarp ? present[w0 + lane] : 0u;
            uint32_t before = 0, all = 0;
#pragma unroll
            for (uint32_t x = lane; x < (uint32_t)kBitmapWords; x += 32) {
                const uint32_t n = __popc(present[x]);
                all += n;
                if (x < w0) before += n;
            }
            before = __reduce_add_sync(0xFFFFFFFFu, before);
            all = __reduce_add_sync(0xFFFFFFFFu, all);
            uint64_t out0 = gstart + running + before;
            for (uint32_t words = __ballot_sync(0xFFFFFFFFu, own != 0); words; words &= words - 1) {
                const uint32_t w = __ffs(words) - 1;
                const uint32_t bits = __shfl_sync(0xFFFFFFFFu, own, w);
                if ((bits >> lane) & 1u) {
                    const uint32_t e = (w0 + w) * 32 + lane;
                    const uint64_t m = (uint64_t)S.bin.masks[2 * e] | (uint64_t)S.bin.masks[2 * e + 1] << 32;
                    S.bin.masks[2 * e] = 0;
                    S.bin.masks[2 * e + 1] = 0;
                    const uint64_t o = out0 + __popc(bits & lanemask_lt());
                    if (o < c1) {
                        a.stage_parent[o] = pbase | ((uint64_t)bin << dbits) | e;
                        a.stage_mask[o] = m;
                    }
                }
                out0 += __popc(bits);
            }
            // The other bitmap, of the bin before, is no longer read.
            turn ^= 1u;
            if (tid < (uint32_t)kBitmapWords) S.bin.present[turn][tid] = 0;
            running += all;
            __syncthreads();
        }
        if (running) {
            if (tid < (uint32_t)kBitmapWords) S.bin.present[turn ^ 1u][tid] = 0;  // the last bin's
            __syncthreads();
        }
        if (tid == 0) {
            a.group_bricks[gi] = running;
            a.group_src[gi] = gstart;
        }
    }
    if (__syncthreads_or(bad) && tid == 0) atomicOr(a.err, kErrBadInput);
}

// Exclusive scan of the items' brick counts (one CTA; items in order) and
// the total, clamped to the output capacity.
__global__ void __launch_bounds__(1024) chunk_scan(ChunkArgs a) {
    pdl_prologue();
    __shared__ uint32_t scan[34];
    const uint32_t g = a.k * a.groups_per_chunk;
    uint64_t carry = 0;
    for (uint32_t b = 0; b < g; b += 1024) {
        const uint32_t i = b + threadIdx.x;
        const uint32_t v = i < g ? a.group_bricks[i] : 0u;
        uint32_t tot;
        const uint32_t ex = block_exclusive_sum<uint32_t>(v, scan, &tot);
        if (i < g) {
            const uint64_t d = carry + ex;
            a.group_dst[i] = d < 0xFFFFFFFFull ? (uint32_t)d : 0xFFFFFFFFu;
        }
        carry += tot;
    }
    if (threadIdx.x == 0) {
        if (carry > a.out_capacity) atomicOr(a.err, kErrCapacity);
        *a.d_out_n = carry < a.out_capacity ? carry : a.out_capacity;
    }
}

// Packs the items' bricks into the ascending list: a CTA moves kCopyTile
// consecutive output bricks (balanced whatever the items' sizes), each row of
// threads consecutive ones. The items of the tile are those from the last that
// starts at or before its first brick on; a thread follows its bricks through
// them. (184 us for 13M bricks when each thread moved a run of eight.)
constexpr int kCopyThreads = 256;
constexpr int kCopyPer = 8;
constexpr int kCopyTile = kCopyThreads * kCopyPer;
__global__ void __launch_bounds__(kCopyThreads) chunk_copy(ChunkArgs a) {
    pdl_prologue();
    const uint32_t g = a.k * a.groups_per_chunk;
    const uint64_t total = *a.d_out_n;
    for (uint64_t t0 = (uint64_t)blockIdx.x * kCopyTile; t0 < total; t0 += (uint64_t)gridDim.x * kCopyTile) {
        uint32_t lo = 0, hi = g;  // group_dst[lo] <= t0 < group_dst[hi] (ascending)
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__ldg(a.group_dst + mid) <= t0) lo = mid; else hi = mid;
        }
        uint32_t w = lo;
        uint64_t p[kCopyPer], m[kCopyPer];
#pragma unroll
        for (int q = 0; q < kCopyPer; ++q) {
            const uint64_t j = t0 + q * kCopyThreads + threadIdx.x;
            if (j >= total) continue;
            while (w + 1 < g && __ldg(a.group_dst + w + 1) <= j) ++w;
            const uint64_t src = __ldg(a.group_src + w) + (j - __ldg(a.group_dst + w));
            p[q] = a.stage_parent[src];
            m[q] = a.stage_mask[src];
        }
#pragma unroll
        for (int q = 0; q < kCopyPer; ++q) {
            const uint64_t j = t0 + q * kCopyThreads + threadIdx.x;
            if (j >= total) continue;
            a.parents[j] = p[q];
            a.leaves[j] = m[q];
        }
    }
}

int g_chunk_ctas = 0;

}  // namespace

void chunk_configure(int sms) {
    cudaFuncSetAttribute(chunk_leaves, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ChunkSmem));
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, chunk_leaves, kT, sizeof(ChunkSmem));
    g_chunk_ctas = (occ > 0 ? occ : 1) * (sms > 0 ? sms : 152);
}

int chunk_run_tiles(uint64_t n) {
    // Runs of up to four tiles (the next tile's fragments are fetched while one
    // is written), but at least two per resident CTA.
    const uint64_t runs = n / ((uint64_t)kChunkTile * 2 * (g_chunk_ctas > 0 ? g_chunk_ctas : 1));
    return (int)(runs < 1 ? 1 : (runs < 4 ? runs : 4));
}

uint32_t chunk_group_bins(uint64_t k, uint32_t bins) {
    // Enough items that the fullest (an item's bins come one after another) is
    // a small part of a CTA's share: 16 per resident CTA where the bins allow
    // (150 chunks of 256^3, 32 bins each: 119 us with one bin per item, 185
    // with all of a chunk's).
    const uint64_t per = k * bins / (16ull * (g_chunk_ctas > 0 ? g_chunk_ctas : 1));
    return (uint32_t)(per < 1 ? 1 : (per < kChunkGroupBins ? per : kChunkGroupBins));
}

int chunk_bin_bits(int chunk_depth) {
    const int lb = 3 * chunk_depth - 6;
    return lb > kChunkDirectBits ? lb - kChunkDirectBits : 0;
}

void launch_chunk_leaves(const ChunkArgs& a, cudaStream_t s) {
    const uint64_t items = 2ull * a.items + (uint64_t)a.k * a.groups_per_chunk;
    const int grid = (int)(items < (uint64_t)g_chunk_ctas ? (items ? items : 1) : g_chunk_ctas);
    launch_pdl(chunk_leaves, dim3(grid), dim3(kT), sizeof(ChunkSmem), s, a);
    launch_pdl(chunk_scan, dim3(1), dim3(1024), 0, s, a);
    // The brick total is on the device: the grid covers the bound and extra
    // CTAs leave at once.
    const uint64_t blocks = (a.out_capacity + kCopyTile - 1) / kCopyTile;
    launch_pdl(chunk_copy, dim3((unsigned)(blocks < 4096 ? (blocks ? blocks : 1) : 4096)), dim3(kCopyThreads), 0, s, a);
}

}  // namespace dagc
