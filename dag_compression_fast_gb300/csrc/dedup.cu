// Deduplication of the leaf masks by hash set + ordering of the distinct ones,
// for sm_103a (the node levels: levels.cu). Replaces the reference's SortLevel
// (src/DAGCompression.cu:864-914) of the leaves: sort (mask, index) pairs, flag
// runs, scan, scatter to unique ids. Same result: the distinct masks in
// ascending order and a map brick -> unique id. Instead of eight 8-bit radix
// passes over every brick, the distinct masks are found first and only those
// are ordered:
//
//   dedup_insert   every brick inserts its mask into an open-addressing table
//                  (linear probing, atomicCAS on the mask); the first inserter
//                  of a mask records itself as the slot's representative and
//                  appends the mask and its slot to the unique list;
//   leaf_rank      (the masks are far from uniform) ranks the unique list, or
//                  where it is long a sample of it, by counting smaller masks;
//                  a list ranked whole is done: each mask goes to its rank in
//                  the leaf array and its rank to its slot (its unique id);
//   leaf_scatter   else the masks (with their slots) go to the buckets between
//                  every fourth sample;
//   leaf_order     and each bucket's masks are ranked and written so;
//   dedup_map      every brick reads its unique id through its slot; a mask's
//                  representative empties its slot.
//
// What the fixed sizes cannot hold (table, unique list, a bucket) sets
// kErrFallback, and the caller reruns the call with the radix-sort form.

#include "dagc_device.cuh"
#include "dagc_kernels.h"
#include "dagc_launch.h"

#include <algorithm>

namespace dagc {
namespace {

__device__ __forceinline__ uint64_t unique_count(const DedupArgs& a) {
    const uint64_t u = a.state->u;
    return u < a.uniq_cap ? u : a.uniq_cap;
}

// Items per lane in flight at once (independent probe chains).
constexpr int kIlp = 4;

__global__ void __launch_bounds__(256, 4) dedup_insert(DedupArgs a) {
    pdl_prologue();
    const uint64_t n = *a.d_n;
    const uint64_t S = table_size_for(n, true);
    const uint32_t S32 = (uint32_t)S;
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t gtid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t gsize = (uint64_t)gridDim.x * blockDim.x;
    if (S > a.table_cap || n > a.item_cap) {
        if (gtid == 0) atomicOr(a.err, kErrFallback);
        return;
    }
    uint32_t* aux = reinterpret_cast<uint32_t*>(a.table_aux);  // slot s: [4s] representative, [4s+1] unique id
    const uint64_t warps = gsize / 32;
    const uint64_t warp = gtid / 32;
    bool bad = false, full = false;
    // Each lane takes kIlp items (32 apart) per round and runs their probe
    // chains side by side. A probe reads the slot first and only an empty
    // slot takes an atomicCAS: duplicated keys (common leaf masks) would
    // otherwise serialise on their slot's atomics.
    for (uint64_t base = warp * 32 * kIlp; base < n; base += warps * 32 * kIlp) {
        uint64_t h[kIlp];
        uint32_t s[kIlp];  // slot indices (tables hold fewer than 2^32 slots)
        bool live[kIlp], won[kIlp];
#pragma unroll
        for (int k = 0; k < kIlp; ++k) {
            const uint64_t i = base + k * 32 + lane;
            won[k] = false;
            live[k] = i < n;
            h[k] = live[k] ? a.keys[i] : 0;
            if (live[k] && h[k] == 0) { bad = true; live[k] = false; }  // 0 marks an empty slot
            s[k] = (uint32_t)home_slot(h[k], S);
        }
        bool found[kIlp];
#pragma unroll
        for (int k = 0; k < kIlp; ++k) found[k] = false;
        // Leaf masks repeat (many items per key): read first, claim only an
        // empty slot. The read takes a slot and the one after it (two loads in
        // flight, usually one sector), so that a key displaced by one slot, or
        // an empty slot right after an occupied one, costs no second round
        // trip. Each round issues every pending item's reads, then every
        // claim, back to back (no result is used before the last one is
        // issued).
        for (uint64_t round = 0; round < S; ++round) {
            bool pend[kIlp], claim[kIlp];
            uint64_t cur[kIlp], nxt[kIlp];
#pragma unroll
            for (int k = 0; k < kIlp; ++k) {
                pend[k] = live[k] && !won[k] && !found[k];
                claim[k] = pend[k];
                cur[k] = 0;
                nxt[k] = 0;
            }
#pragma unroll
            for (int k = 0; k < kIlp; ++k) {
                if (pend[k]) {
                    cur[k] = ld_relaxed(a.table_key + 2ull * s[k]);
                    nxt[k] = ld_relaxed(a.table_key + 2ull * next_slot(s[k], S32));
                }
            }
            // In probe order: a match ends the search; the first empty
            // slot is claimed; two other keys move the probe on by two.
#pragma unroll
            for (int k = 0; k < kIlp; ++k) {
                if (!pend[k]) continue;
                if (cur[k] == h[k]) { found[k] = true; claim[k] = false; continue; }
                if (cur[k] == 0) continue;
                s[k] = next_slot(s[k], S32);
                if (nxt[k] == h[k]) { found[k] = true; claim[k] = false; continue; }
                if (nxt[k] != 0) { s[k] = next_slot(s[k], S32); claim[k] = false; }
            }
#pragma unroll
            for (int k = 0; k < kIlp; ++k)
                if (claim[k]) cur[k] = atomicCAS((unsigned long long*)(a.table_key + 2ull * s[k]), 0ull, (unsigned long long)h[k]);
            bool any = false;
#pragma unroll
            for (int k = 0; k < kIlp; ++k) {
                if (!pend[k] || found[k]) continue;
                if (!claim[k]) { any = true; continue; }  // both slots held other keys
                if (cur[k] == 0) won[k] = true;
                else if (cur[k] == h[k]) found[k] = true;
                else { s[k] = next_slot(s[k], S32); any = true; }
            }
            if (!any) break;
        }
#pragma unroll
        for (int k = 0; k < kIlp; ++k) {
            const uint64_t i = base + k * 32 + lane;
            if (i < n) {
                const bool placed = live[k] && (won[k] || found[k]);
                if (live[k] && !placed) full = true;  // cannot happen: tables are at most 0.8 full; rerun rather than guess
                a.item_slot[i] = placed ? s[k] : 0xFFFFFFFFu;
            }
        }
        // Winners append to the unique list: one atomic per warp for all its
        // item rows. Every lane takes part in the ballots and shuffles.
        uint32_t wm[kIlp];
        uint32_t wtotal = 0;
#pragma unroll
        for (int k = 0; k < kIlp; ++k) {
            wm[k] = __ballot_sync(0xFFFFFFFFu, won[k]);
            wtotal += __popc(wm[k]);
        }
        uint64_t pos0 = 0;
        if (lane == 0 && wtotal)
            pos0 = atomicAdd((unsigned long long*)&a.state->u, (unsigned long long)wtotal);
        pos0 = __shfl_sync(0xFFFFFFFFu, pos0, 0);
#pragma unroll
        for (int k = 0; k < kIlp; ++k) {
            if (won[k]) {
                const uint64_t i = base + k * 32 + lane;
                const uint64_t pos = pos0 + __popc(wm[k] & lanemask_lt());
                aux[4ull * s[k]] = (uint32_t)i;
                if (pos < a.uniq_cap) {
                    a.uniq_key[pos] = h[k];
                    a.uniq_slot[pos] = s[k];
                } else {
                    full = true;
                }
            }
            pos0 += __popc(wm[k]);
        }
    }
    if (bad) atomicOr(a.err, kErrBadInput);
    if (full) atomicOr(a.err, kErrFallback);
}

// ------------------------------------------- ordering the leaf masks ----
// The distinct masks are any 64-bit values (a few bits set, or nearly all), so
// their buckets come from a sample of them. Three launches whatever their
// number; the first form, a radix sort of the list (eight digit passes and a
// histogram, each gated on a one-CTA form for short lists, then a probe of the
// table per key for its slot), was twelve, mostly latency.
// Kernel times before / now (us): 200 masks (32^3 shell) 50 / 4; 25k (512^3
// terrain) 116 / 28; 40k (2048^3 terrain) 106 / 31; 1.08M (8192^3 soup) 192 / 152.

// Samples and buckets for u distinct masks. Up to kLeafRankMax every mask is a
// "sample" and its rank is final. Else a bucket holds the keys between every
// fourth sample: its size is a gamma distribution of shape 4, with a mean of at
// most 256 keys up to 2^18 masks, 2048 at the list's limit.
__device__ __forceinline__ void leaf_shape(uint64_t u, uint32_t* samples, uint32_t* buckets) {
    if (u <= kLeafRankMax) { *samples = (uint32_t)u; *buckets = 0; }
    else if (u <= kLeafMidMax) { *samples = kLeafRankMax / 2; *buckets = kLeafBuckets / 2; }
    else { *samples = kLeafRankMax; *buckets = kLeafBuckets; }
}
// Position of sample i in the unique list (all different: u >= samples, which
// are a power of two unless they are all of the list).
__device__ __forceinline__ uint64_t sample_pos(uint32_t i, uint64_t u, uint32_t samples) {
    return samples == u ? (uint64_t)i : ((uint64_t)i * u) >> (31 - __clz(samples));
}

// Entry room per bucket: eight times the mean or more, up to the shared memory
// of leaf_order (four times the mean at the list's limit).
__device__ __forceinline__ uint32_t leaf_bucket_cap(const DedupArgs& a, uint32_t buckets) {
    const uint64_t room = a.bucket_area / buckets;
    return (uint32_t)(room < a.leaf_keys ? room : a.leaf_keys);
}

constexpr int kRankThreads = 1024;
constexpr int kRankPer = kRankThreads / 32;  // keys per CTA and round, a warp each
constexpr int kRankCtas = 128;

// Every CTA holds all the samples in shared memory and ranks its share of them,
// a warp to a key: the samples' square over the GPU (8192: 67M comparisons).
// Few large CTAs, since each fetches every sample, a sector apiece (256 CTAs of
// 256 threads: 17 us for 4096 samples, 40 for 8192; these take 9 and 23).
__global__ void __launch_bounds__(kRankThreads) leaf_rank(DedupArgs a) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* key = reinterpret_cast<uint64_t*>(smem_raw);  // kLeafRankMax
    const uint64_t u = unique_count(a);
    if (blockIdx.x == 0 && threadIdx.x == 0) *a.d_out_n = u < a.out_capacity ? u : a.out_capacity;
    uint32_t ns, nb;
    leaf_shape(u, &ns, &nb);
    if (blockIdx.x * kRankPer >= ns) return;
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < ns; i += kRankThreads) key[i] = a.uniq_key[sample_pos(i, u, ns)];
    __syncthreads();
    uint32_t* aux = reinterpret_cast<uint32_t*>(a.table_aux);
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t i = blockIdx.x * kRankPer + (threadIdx.x >> 5); i < ns; i += gridDim.x * kRankPer) {
        const uint64_t k = key[i];
        uint32_t r = 0;
#pragma unroll 8
        for (uint32_t x = lane; x < ns; x += 32) r += key[x] < k;
        r = __reduce_add_sync(0xFFFFFFFFu, r);
        if (lane != 0) continue;
        if (nb == 0) {
            if (r < a.out_capacity) {
                a.out_keys[r] = k;
                aux[4ull * a.uniq_slot[i] + 1] = r;
            } else {
                atomicOr(a.err, kErrCapacity);
            }
        } else if (r % (ns / nb) == 0) {
            a.leaf->splitter[r / (ns / nb)] = k;
        }
    }
}

// Bucket b holds the keys from splitter b (b = 0: any) up to splitter b + 1.
constexpr int kLeafIlp = 4;
__global__ void __launch_bounds__(512) leaf_scatter(DedupArgs a) {
    pdl_prologue();
    __shared__ uint64_t spl[kLeafBuckets];
    const uint64_t u = unique_count(a);
    uint32_t ns, nb;
    leaf_shape(u, &ns, &nb);
    const uint64_t per = 512ull * kLeafIlp;
    if (nb == 0 || blockIdx.x * per >= u) return;
    for (uint32_t i = threadIdx.x; i < nb; i += 512) spl[i] = a.leaf->splitter[i];
    __syncthreads();
    const uint32_t cap = leaf_bucket_cap(a, nb);
    bool full = false;
    for (uint64_t i0 = blockIdx.x * per + threadIdx.x; i0 < u; i0 += gridDim.x * per) {
        uint64_t k[kLeafIlp];
        uint32_t s[kLeafIlp], b[kLeafIlp], pos[kLeafIlp];
#pragma unroll
        for (int q = 0; q < kLeafIlp; ++q) {
            const uint64_t i = i0 + q * 512;
            k[q] = i < u ? a.uniq_key[i] : 0;
            s[q] = i < u ? a.uniq_slot[i] : 0;
            b[q] = 0;
        }
        // The last splitter not above the key, among the nb - 1 after the first.
        for (uint32_t half = nb / 2; half > 0; half /= 2) {
#pragma unroll
            for (int q = 0; q < kLeafIlp; ++q)
                if (spl[b[q] + half] <= k[q]) b[q] += half;
        }
#pragma unroll
        for (int q = 0; q < kLeafIlp; ++q) pos[q] = i0 + q * 512 < u ? atomicAdd(&a.leaf->count[b[q]], 1u) : 0u;
#pragma unroll
        for (int q = 0; q < kLeafIlp; ++q) {
            if (i0 + q * 512 >= u) continue;
            if (pos[q] < cap) {
                a.bucket[(uint64_t)b[q] * cap + pos[q]] = make_uint4((uint32_t)k[q], (uint32_t)(k[q] >> 32), s[q], 0u);
            } else {
                full = true;  // a bucket past its room (a very uneven sample)
            }
        }
    }
    if (full) atomicOr(a.err, kErrFallback);
}

// Each CTA takes a range of buckets. A bucket's keys are put in sub-buckets
// between kSub of them (ranked by counting) and ranked by counting within those:
// some 20 shared-memory reads per key whatever the bucket's size (counting over
// whole buckets, 264 keys on average at 1.08M masks, took four times as long as
// the radix sort).
constexpr uint32_t kSub = 64;
constexpr uint32_t kSubMin = 96;  // up to here a bucket is counted whole

// Room for 2048 keys per bucket (20 KB): 256 threads; for 8192 (80 KB, two CTAs
// per SM): 512.
template <int kOrderThreads>
__global__ void __launch_bounds__(kOrderThreads) leaf_order(DedupArgs a) {
    pdl_prologue();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* key = reinterpret_cast<uint64_t*>(smem_raw);              // leaf_keys
    uint16_t* ord = reinterpret_cast<uint16_t*>(key + a.leaf_keys);     // keys in sub-bucket order
    __shared__ uint64_t spl[kSub];
    __shared__ uint32_t cnt[kSub], sub0[kSub + 1];
    __shared__ uint32_t red[kOrderThreads / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint64_t u = unique_count(a);
    uint32_t ns, nb;
    leaf_shape(u, &ns, &nb);
    const uint32_t b0 = (uint32_t)((uint64_t)nb * blockIdx.x / gridDim.x);
    const uint32_t b1 = (uint32_t)((uint64_t)nb * (blockIdx.x + 1) / gridDim.x);
    if (b0 >= b1) return;
    uint32_t part = 0;
    for (uint32_t x = tid; x < b0; x += kOrderThreads) part += a.leaf->count[x];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xFFFFFFFFu, part, o);
    if (lane == 0) red[warp] = part;
    __syncthreads();
    uint64_t start = 0;
    for (int w = 0; w < kOrderThreads / 32; ++w) start += red[w];
    const uint32_t cap = leaf_bucket_cap(a, nb);
    uint32_t* aux = reinterpret_cast<uint32_t*>(a.table_aux);
    bool bad = false;
    auto put = [&](const uint4* ent, uint32_t j, uint64_t k, uint64_t uid) {
        const uint32_t slot = ent[j].z;
        if (uid < a.out_capacity && slot < a.table_cap) {
            a.out_keys[uid] = k;
            aux[4ull * slot + 1] = (uint32_t)uid;
        } else {
            bad = true;
        }
    };
    auto sub_of = [&](uint64_t k) {  // the last of spl not above k, among those after the first
        uint32_t s = 0;
#pragma unroll
        for (uint32_t half = kSub / 2; half > 0; half /= 2)
            if (spl[s + half] <= k) s += half;
        return s;
    };
    for (uint32_t b = b0; b < b1; ++b) {
        const uint32_t total = a.leaf->count[b], c = min(total, cap);  // beyond: flagged by leaf_scatter
        const uint4* ent = a.bucket + (uint64_t)b * cap;
        __syncthreads();  // the bucket before is no longer read
        for (uint32_t j = tid; j < c; j += kOrderThreads) {
            const uint4 e = ent[j];
            key[j] = (uint64_t)e.x | (uint64_t)e.y << 32;
        }
        if (tid < kSub) cnt[tid] = 0;
        __syncthreads();
        if (c <= kSubMin) {
            if (tid < c) {
                const uint64_t k = key[tid];
                uint32_t r = 0;
#pragma unroll 8
                for (uint32_t x = 0; x < c; ++x) r += key[x] < k;
                put(ent, tid, k, start + r);
            }
            start += total;
            continue;
        }
        if (tid < kSub) {
            const uint64_t k = key[tid * c / kSub];
            uint32_t r = 0;
#pragma unroll 8
            for (uint32_t x = 0; x < kSub; ++x) r += key[x * c / kSub] < k;
            spl[r] = k;
        }
        __syncthreads();
        for (uint32_t j = tid; j < c; j += kOrderThreads) atomicAdd(&cnt[sub_of(key[j])], 1u);
        __syncthreads();
        if (warp == 0) {
            const uint32_t n0 = cnt[2 * lane], n1 = cnt[2 * lane + 1];
            uint32_t x = n0 + n1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                if (lane >= (uint32_t)o) x += y;
            }
            const uint32_t s0 = x - n0 - n1;
            cnt[2 * lane] = sub0[2 * lane] = s0;
            cnt[2 * lane + 1] = sub0[2 * lane + 1] = s0 + n0;
            if (lane == 31) sub0[kSub] = x;
        }
        __syncthreads();
        for (uint32_t j = tid; j < c; j += kOrderThreads) ord[atomicAdd(&cnt[sub_of(key[j])], 1u)] = (uint16_t)j;
        __syncthreads();
        for (uint32_t i = tid; i < c; i += kOrderThreads) {
            const uint32_t j = ord[i];
            const uint64_t k = key[j];
            const uint32_t s = sub_of(k), s0 = sub0[s], s1 = sub0[s + 1];
            uint32_t r = s0;
            for (uint32_t x = s0; x < s1; ++x) r += key[ord[x]] < k;
            put(ent, j, k, start + r);
        }
        start += total;
    }
    if (bad) atomicOr(a.err, kErrCapacity);
}

__global__ void __launch_bounds__(256) dedup_map(DedupArgs a) {
    pdl_prologue();
    const uint64_t n = *a.d_n;
    if (table_size_for(n, true) > a.table_cap || n > a.item_cap) return;  // insert did nothing
    const uint32_t last = a.out_capacity ? (uint32_t)(a.out_capacity - 1) : 0u;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    // kIlp items per thread per round, their slot reads in flight together.
    for (uint64_t i0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += stride * kIlp) {
        uint32_t s[kIlp];
        uint64_t aux[kIlp];
#pragma unroll
        for (int k = 0; k < kIlp; ++k) {
            const uint64_t i = i0 + k * stride;
            s[k] = i < n ? a.item_slot[i] : 0xFFFFFFFFu;
        }
#pragma unroll
        for (int k = 0; k < kIlp; ++k) aux[k] = s[k] < a.table_cap ? a.table_aux[2 * (uint64_t)s[k]] : 0;
#pragma unroll
        for (int k = 0; k < kIlp; ++k) {
            const uint64_t i = i0 + k * stride;
            if (i >= n) continue;
            uint32_t uid = 0;
            if (s[k] < a.table_cap) {
                const uint32_t rep = (uint32_t)aux[k];
                uid = (uint32_t)(aux[k] >> 32);
                if (rep == (uint32_t)i) a.table_key[2 * (uint64_t)s[k]] = 0;  // empty for the node levels
            }
            // Ids stay inside the next level's arrays even when a fallback or
            // an error discards this call.
            a.map[i] = uid <= last ? uid : last;
        }
    }
}

int g_sms = 152;

}  // namespace

void dedup_configure(int sms) {
    cudaFuncSetAttribute(leaf_rank, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kLeafRankMax * 8));
    cudaFuncSetAttribute(leaf_order<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(leaf_keys_for(kDedupMaxUnique) * 10));
    g_sms = sms > 0 ? sms : 152;
}

namespace {
int item_grid(const DedupArgs& a) {
    const uint64_t want = (a.item_cap + 255) / 256;
    const int g = 8 * g_sms;  // full occupancy: 8 CTAs of 256 threads per SM
    return (int)(want < (uint64_t)g ? (want > 0 ? want : 1) : g);
}
}  // namespace

void launch_dedup_insert(const DedupArgs& a, cudaStream_t s) {
    launch_pdl(dedup_insert, dim3(item_grid(a)), dim3(256), 0, s, a);
}

int launch_leaf_order(const DedupArgs& a, cudaStream_t s) {
    const int ranks = (int)std::min<uint64_t>((a.uniq_cap + kRankPer - 1) / kRankPer, kRankCtas);
    launch_pdl(leaf_rank, dim3(ranks), dim3(kRankThreads), std::min<uint64_t>(a.uniq_cap, kLeafRankMax) * 8, s, a);
    if (a.uniq_cap <= kLeafRankMax) return 1;  // no list is longer
    const uint64_t want = (a.uniq_cap + 512 * kLeafIlp - 1) / (512 * kLeafIlp);
    launch_pdl(leaf_scatter, dim3((unsigned)std::min<uint64_t>(want, 2ull * g_sms)), dim3(512), 0, s, a);
    if (a.uniq_cap <= kLeafMidMax)
        launch_pdl(leaf_order<256>, dim3(kLeafBuckets / 2), dim3(256), a.leaf_keys * 10, s, a);
    else
        launch_pdl(leaf_order<512>, dim3(2 * g_sms), dim3(512), a.leaf_keys * 10, s, a);
    return 3;
}

void launch_dedup_map(const DedupArgs& a, cudaStream_t s) {
    launch_pdl(dedup_map, dim3(item_grid(a)), dim3(256), 0, s, a);
}

}  // namespace dagc
