// Leaves by a direct-mapped table of the whole brick space, for sm_103a: the
// same sorted parents and leaf masks as the fragment sort + leaf build
// (src/DAGCompression.cu:1026-1068: SortKeys, SelectUnique, ReduceByKey) and
// the grouping of group.cu, without a sort and without a hash.
//
// The volume's 8^(depth - 2) bricks (code >> 6) are the entries of a table of
// leaf masks that the context keeps, all zero between calls:
//
//   direct_mark     every fragment ORs its voxel bit into its brick's entry
//                   (and checks its code's range); the first fragment of a
//                   brick counts it for its block of 64 entries;
//   direct_plan     (above kDirectScanBlocks blocks) the blocks that hold a
//                   brick, in order, with the number of bricks before each;
//   direct_compact  reads the occupied blocks: their nonzero entries, which
//                   are in ascending brick order by position, go out as
//                   (parent, mask), and their entries are zero again.
//
// Blocks of 64 entries (512 bytes): where bricks lie apart (a triangle soup at
// depth 11, 0.56M bricks over the whole volume) larger ones read mostly empty
// entries: with 512 entries per block, 77 us of the 1 GB table.
//
// The brick order is the table's, so nothing of the N fragments is moved or
// sorted: they are read once, and what is written is 16 bytes per brick. The
// grouping (group.cu) of deeper or larger volumes puts its bricks, one store
// each, in the same table instead of sorting them.

#include "dagc_device.cuh"
#include "dagc_kernels.h"
#include "dagc_launch.h"

#include <algorithm>

namespace dagc {
namespace {

constexpr int kMarkThreads = 256;
constexpr int kMarkIlp = 8;  // rows of 32 fragments per warp in flight
constexpr int kBlockLog = kDirectBlockLog;
constexpr int kBlockRows = (1 << kBlockLog) / 32;  // rows of 32 entries per block
constexpr int kWarpBlocks = 8;                     // blocks per warp and step: 16 loads per lane in flight

// An entry through the L1: a stale value only shows fewer bits than are set,
// which costs an OR that changes nothing.
__device__ __forceinline__ uint64_t ld_cached(const uint64_t* p) {
    uint64_t v;
    asm volatile("ld.global.ca.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// What bounds it: the fragments' read and, per fragment, one random 8-byte
// access of the table in the L2. An entry is read first and ORed only where
// the bit is missing: repeated voxels (1 to 4 per voxel in the workloads) and
// crowded bricks then cost a cached load instead of an atomic that queues
// behind the others of its address. Only an entry seen empty takes the atomic
// that returns the old value (its first setter counts the brick); the others
// take the reduction.
//
// Fragments in order (a voxelizer's, a sorted list) put whole rows, and many
// warps at a time, on the same few entries, whose atomics queue in the L2. A
// row of at most kMarkRuns runs of equal bricks therefore makes one access per
// run, and consecutive rows of one brick one between them: a warp takes up to
// kMarkIlp consecutive rows at a time (one where that does not fill the GPU).
// This kernel, us, with an access per fragment / so: 1M sorted fragments that
// fill a 32^3 grid 170 / 13, the same shuffled 82 / 57; 4M, 64 per voxel in order,
// 256^3, 215 / 21; 33M in a slab of 512^3, sorted 455 / 133, shuffled 248 / 243;
// 2.3M, four per brick of 1024^3, sorted 38 / 39, shuffled 49 / 47.
constexpr int kMarkRuns = 8;

// ORs `bits` into a brick's entry (depth 10 at most: bricks below 2^24), whose
// value `cur`, just read, lacks some of them.
__device__ __forceinline__ void mark(const DirectArgs& a, uint32_t brick, uint64_t bits, uint64_t cur) {
    unsigned long long* e = reinterpret_cast<unsigned long long*>(a.table + brick);
    if (cur == 0) {
        if (atomicOr(e, (unsigned long long)bits) == 0) atomicAdd(a.block_count + (brick >> kBlockLog), 1u);
    } else {
        atomicOr(e, (unsigned long long)bits);
    }
}

__global__ void __launch_bounds__(kMarkThreads) direct_mark(DirectArgs a) {
    pdl_prologue();
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t rows = a.mark_rows, step = (uint64_t)gridDim.x * kMarkThreads * rows;
    bool bad = false;
    // Uniform trip count over a warp: every lane takes part in the shuffles.
    for (uint64_t w0 = ((uint64_t)blockIdx.x * kMarkThreads + threadIdx.x - lane) * rows; w0 < a.n; w0 += step) {
        uint64_t bits[kMarkIlp];  // the fragments, then their voxel bits
        uint32_t brick[kMarkIlp];
#pragma unroll
        for (int k = 0; k < kMarkIlp; ++k) {
            const uint64_t i = w0 + lane + k * 32;
            bits[k] = (uint32_t)k < rows && i < a.n ? __ldcs(a.frags + i) : ~0ull;
        }
        bool whole_before = false;  // the row before is one run
#pragma unroll
        for (int k = 0; k < kMarkIlp; ++k) {
            if ((uint32_t)k >= rows) break;
            const uint64_t code = bits[k];
            const bool ok = !(code >> a.code_bits);
            bad |= !ok && w0 + lane + k * 32 < a.n;
            brick[k] = ok ? (uint32_t)(code >> 6) : 0xFFFFFFFFu;
            bits[k] = ok ? 1ull << (code & 63) : 0ull;
            const uint32_t left = __shfl_up_sync(0xFFFFFFFFu, brick[k], 1);
            const uint32_t heads = __ballot_sync(0xFFFFFFFFu, lane == 0 || brick[k] != left);
            const bool whole = heads == 1u;
            if (__popc(heads) <= kMarkRuns) {
                // The lanes of this one's run: from its head to before the next.
                const uint32_t head = 31 - __clz(heads & ((2u << lane) - 1u));
                const uint32_t after = heads & ~((2u << lane) - 1u);
                const uint32_t run = (after ? (after & (0u - after)) - 1u : 0xFFFFFFFFu) & ~((1u << head) - 1u);
                const uint32_t lo = __reduce_or_sync(run, (uint32_t)bits[k]);
                const uint32_t hi = __reduce_or_sync(run, (uint32_t)(bits[k] >> 32));
                bits[k] = lane == head ? (uint64_t)hi << 32 | lo : 0ull;
                if (k > 0 && whole && whole_before && brick[k] == brick[k - 1]) {
                    bits[k] |= bits[k - 1];
                    bits[k - 1] = 0;
                }
            }
            whole_before = whole;
        }
        uint64_t cur[kMarkIlp];
#pragma unroll
        for (int k = 0; k < kMarkIlp; ++k)
            cur[k] = (uint32_t)k < rows && bits[k] ? ld_cached(a.table + brick[k]) : ~0ull;
#pragma unroll
        for (int k = 0; k < kMarkIlp; ++k)
            if ((cur[k] & bits[k]) != bits[k]) mark(a, brick[k], bits[k], cur[k]);
    }
    if (bad) atomicOr(a.err, kErrBadInput);
}

// The occupied blocks in order and the bricks before each: tiles of 4096
// counters, one look-back value for both sums (blocks above, bricks below).
constexpr int kPlanThreads = 256;
constexpr int kPlanPer = 16;
static_assert(kPlanThreads * kPlanPer == kDirectPlanTile, "plan tile");

__global__ void __launch_bounds__(kPlanThreads) direct_plan(DirectArgs a) {
    pdl_prologue();
    __shared__ uint64_t scan[34];
    __shared__ uint32_t slot;
    __shared__ uint64_t base_s;
    const uint32_t tid = threadIdx.x;
    if (a.gate && *a.gate != 1u) return;
    const uint32_t tiles = (a.blocks + kDirectPlanTile - 1) / kDirectPlanTile;
    while (true) {
        if (tid == 0) slot = atomicAdd(a.tile_counter, 1u);
        __syncthreads();
        const uint32_t tile = slot;
        if (tile >= tiles) break;
        const uint32_t b0 = tile * kDirectPlanTile + tid * kPlanPer;
        uint32_t c[kPlanPer];
        uint64_t sum = 0;
#pragma unroll
        for (int q = 0; q < kPlanPer; q += 4) {
            uint4 v = make_uint4(0, 0, 0, 0);  // a.blocks is a multiple of 4 here (a power of 8)
            if (b0 + q < a.blocks) v = *reinterpret_cast<const uint4*>(a.block_count + b0 + q);
            c[q] = v.x; c[q + 1] = v.y; c[q + 2] = v.z; c[q + 3] = v.w;
        }
#pragma unroll
        for (int q = 0; q < kPlanPer; ++q) sum += c[q] ? (1ull << 32) + c[q] : 0ull;
        uint64_t total;
        const uint64_t excl = block_exclusive_sum<uint64_t>(sum, scan, &total);
        if (tid < 32) {
            const uint64_t b = sv_lookback(a.status, tile, total, a.err);
            if (tid == 0) base_s = b;
        }
        __syncthreads();
        uint64_t at = base_s + excl;
#pragma unroll
        for (int q = 0; q < kPlanPer; ++q) {
            if (!c[q]) continue;
            const uint32_t pos = (uint32_t)(at >> 32);
            if (pos < a.blocks) a.list[pos] = make_uint2(b0 + q, (uint32_t)at);
            at += (1ull << 32) + c[q];
        }
        if (tid == 0 && tile == tiles - 1) {
            const uint64_t all = base_s + total;
            const uint64_t bricks = all & 0xFFFFFFFFull;
            *a.d_blocks = all >> 32 < a.blocks ? all >> 32 : a.blocks;
            *a.d_out_n = bricks < a.out_capacity ? bricks : a.out_capacity;
        }
        __syncthreads();
    }
}

// A warp takes kWarpBlocks blocks per step: of the list, or (up to
// kDirectScanBlocks blocks) the next ones of the table, whose CTA then sums
// the counters before its 64 blocks itself: at most 16 KB from the L2 per CTA,
// cheaper than another launch.
template <bool kList>
__global__ void __launch_bounds__(256) direct_compact(DirectArgs a) {
    pdl_prologue();
    __shared__ uint32_t red[8], cnt[8];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (a.gate && *a.gate != 1u) return;
    constexpr uint32_t kCtaBlocks = 8 * kWarpBlocks;
    const uint64_t count = kList ? *a.d_blocks : (uint64_t)a.blocks;
    const uint64_t step = (uint64_t)gridDim.x * kCtaBlocks;
    bool overflow = false;
    for (uint64_t g = (uint64_t)blockIdx.x * kCtaBlocks; g < count; g += step) {  // uniform over the CTA
        // Lane j < kWarpBlocks: the warp's block j and the bricks before it.
        const uint64_t x = g + warp * kWarpBlocks + lane;
        const bool own = lane < (uint32_t)kWarpBlocks && x < count;
        uint32_t block = 0, base = 0;
        bool occupied = own;
        if (kList) {
            if (own) {
                const uint2 e = a.list[x];
                block = e.x;
                base = e.y;
            }
        } else {
            const uint32_t mine = own ? a.block_count[x] : 0u;
            uint32_t part = 0, incl = mine;
            for (uint32_t b = tid; b < g; b += 256) part += a.block_count[b];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, incl, o);
                if (lane >= (uint32_t)o) incl += y;
            }
            if (lane == 31) { red[warp] = part; cnt[warp] = incl; }
            __syncthreads();
            uint32_t all = 0;
            for (uint32_t w = 0; w < 8; ++w) {
                base += red[w] + (w < warp ? cnt[w] : 0u);
                all += red[w] + cnt[w];
            }
            if (g + kCtaBlocks >= count && tid == 0) *a.d_out_n = all < a.out_capacity ? all : a.out_capacity;
            __syncthreads();
            block = (uint32_t)x;
            base += incl - mine;
            occupied = mine != 0;
        }
        const uint32_t live = __ballot_sync(0xFFFFFFFFu, occupied);
        uint64_t m[kWarpBlocks][kBlockRows];
#pragma unroll
        for (int j = 0; j < kWarpBlocks; ++j) {
            const uint64_t e0 = ((uint64_t)__shfl_sync(0xFFFFFFFFu, block, j) << kBlockLog) + lane;
#pragma unroll
            for (int k = 0; k < kBlockRows; ++k) m[j][k] = (live >> j) & 1u ? ld_relaxed(a.table + e0 + k * 32) : 0ull;
        }
#pragma unroll
        for (int j = 0; j < kWarpBlocks; ++j) {
            const uint64_t e0 = ((uint64_t)__shfl_sync(0xFFFFFFFFu, block, j) << kBlockLog) + lane;
            uint64_t out = __shfl_sync(0xFFFFFFFFu, base, j);
#pragma unroll
            for (int k = 0; k < kBlockRows; ++k) {
                const uint32_t has = __ballot_sync(0xFFFFFFFFu, m[j][k] != 0);
                if (m[j][k]) {
                    const uint64_t o = out + __popc(has & lanemask_lt());
                    a.table[e0 + k * 32] = 0;  // empty for the next call
                    if (o < a.out_capacity) {
                        a.parents[o] = e0 + k * 32;
                        a.leaves[o] = m[j][k];
                    } else {
                        overflow = true;
                    }
                }
                out += __popc(has);
            }
        }
    }
    if (overflow) atomicOr(a.err, kErrCapacity);
}

int g_direct_sms = 152;

}  // namespace

void direct_configure(int sms) { g_direct_sms = sms > 0 ? sms : 152; }

int launch_direct_mark(const DirectArgs& args, cudaStream_t s) {
    DirectArgs a = args;
    const uint64_t most = 8ull * g_direct_sms;
    // A row per warp where that does not fill the GPU, up to eight.
    const uint64_t full = most * kMarkThreads;
    a.mark_rows = (uint32_t)std::min<uint64_t>(kMarkIlp, std::max<uint64_t>(1, (a.n + full - 1) / full));
    const uint64_t per = (uint64_t)kMarkThreads * a.mark_rows, want = (a.n + per - 1) / per;
    launch_pdl(direct_mark, dim3((unsigned)(want < most ? (want ? want : 1) : most)), dim3(kMarkThreads), 0, s, a);
    return 1;
}

int launch_direct_compact(const DirectArgs& a, cudaStream_t s) {
    const uint64_t most = 8ull * g_direct_sms;
    const uint64_t ctas = (a.blocks + 8 * kWarpBlocks - 1) / (8 * kWarpBlocks);
    if (a.blocks <= kDirectScanBlocks) {
        launch_pdl(direct_compact<false>, dim3((unsigned)ctas), dim3(256), 0, s, a);
        return 1;
    }
    const uint64_t tiles = (a.blocks + kDirectPlanTile - 1) / kDirectPlanTile;
    launch_pdl(direct_plan, dim3((unsigned)(tiles < most ? tiles : most)), dim3(kPlanThreads), 0, s, a);
    launch_pdl(direct_compact<true>, dim3((unsigned)(ctas < most ? ctas : most)), dim3(256), 0, s, a);
    return 2;
}

}  // namespace dagc
