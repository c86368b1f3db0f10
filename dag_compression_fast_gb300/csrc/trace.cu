// Headless DAG tracer for sm_103a: primary rays through the final uint32 DAG
// layout, written to device buffers (a colour per pixel and the Morton code of
// the voxel hit) instead of the reference's OpenGL surface
// (src/DAGTracer.cu:297-427, FDAGTracer::ResolvePaths :429-443). It reads
// exactly the layout CreateFinalDAG writes (src/DAGCompression.cu:1550-1610),
// so it doubles as an end-to-end check of that format.
//
// The traversal is the reference's: a per-ray stack of (node word index, child
// mask, children still to visit), children visited in the order given by the
// ray's direction signs, each child's intersection found with the slab test
// around the node's centre (epsilon 1e-4 near the splitting planes), the last
// two levels read from the 64-bit leaf. Float arithmetic follows the
// reference's operation order; this file is compiled with --fmad=false, so
// every operation is one IEEE rounding and the result is reproducible on the
// CPU.
//
// A ray's direction is normalised in float64 (the rule), of which this part
// does 2 operations per SM and clock. It is computed in pairs of float32
// instead, with an error bound, and only where a float32 rounding lies within
// the bound does the float64 form decide (ray_direction). The rest is bound by
// the instructions of a step (half of them compares and selects on the ALU
// pipe, 23 of 32 lanes busy) and the last rays of a frame. The whole call,
// 1920x1080 on the 2048^3 terrain: 337 us with float64 throughout; 309 with the
// pairs; 252 with one-step ascents, positions in voxels and the error word in
// pinned memory. Blocks of 32 to 256 rays, 4 or 8 wide, make no difference.
//
// Reads of the word array are bounds-checked and each ray stops after
// kTraceMaxSteps descents: a malformed array sets kErrBadInput, never a read
// outside it.

#include "dagc_device.cuh"
#include "dagc_kernels.h"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace dagc {
namespace {

constexpr uint32_t kTraceMaxSteps = 1u << 22;
constexpr int kTraceThreads = 128;
constexpr int kTraceMaxDepth = 21;  // the deepest DAG the library builds

// The reference's maximum and minimum; kTame: no operand is NaN, and the
// machine's own differ at most in the sign of a zero, which no later
// operation tells apart.
template <bool kTame>
__device__ __forceinline__ float max_ref(float a, float b) { return kTame ? fmaxf(a, b) : a > b ? a : b; }
template <bool kTame>
__device__ __forceinline__ float min_ref(float a, float b) { return kTame ? fminf(a, b) : a < b ? a : b; }

// Children of the node at `pos` (its corner, in voxels), half its edge
// `radius`, that the ray crosses.
template <bool kTame>
__device__ __forceinline__ uint32_t crossed_children(bool root, uint32_t half_edge, const uint32_t pos[3], float3 org,
                                                     float3 dir, float3 inv) {
    const float radius = float(half_edge);
    const float3 cr = make_float3(radius + float(pos[0]) - org.x, radius + float(pos[1]) - org.y,
                                  radius + float(pos[2]) - org.z);
    const float3 tmid = make_float3(cr.x * inv.x, cr.y * inv.y, cr.z * inv.z);
    const float3 slab = make_float3(radius * fabsf(inv.x), radius * fabsf(inv.y), radius * fabsf(inv.z));
    const float tmin = max_ref<kTame>(max_ref<kTame>(tmid.x - slab.x, max_ref<kTame>(tmid.y - slab.y, tmid.z - slab.z)), 0.0f);
    const float tmax = min_ref<kTame>(tmid.x + slab.x, min_ref<kTame>(tmid.y + slab.y, tmid.z + slab.z));
    if (root && tmin >= tmax) return 0;
    // The child holding the midpoint of the ray's span inside the node...
    const float half = 0.5f * (tmin + tmax);
    uint32_t mask = 1u << ((half * dir.x >= cr.x ? 4 : 0) + (half * dir.y >= cr.y ? 2 : 0) +
                           (half * dir.z >= cr.z ? 1 : 0));
    // ... and, where the ray crosses a splitting plane inside the span, the
    // children on both sides of it (both, near another plane).
    const float eps = 1e-4f;
    if (tmin <= tmid.x && tmid.x <= tmax) {
        const float py = tmid.x * dir.y, pz = tmid.x * dir.z;
        const uint32_t a = (py >= cr.y - eps ? 0xCCu : 0u) | (py <= cr.y + eps ? 0x33u : 0u);
        const uint32_t b = (pz >= cr.z - eps ? 0xAAu : 0u) | (pz <= cr.z + eps ? 0x55u : 0u);
        mask |= a & b;
    }
    if (tmin <= tmid.y && tmid.y <= tmax) {
        const float px = tmid.y * dir.x, pz = tmid.y * dir.z;
        const uint32_t c = (px >= cr.x - eps ? 0xF0u : 0u) | (px <= cr.x + eps ? 0x0Fu : 0u);
        const uint32_t d = (pz >= cr.z - eps ? 0xAAu : 0u) | (pz <= cr.z + eps ? 0x55u : 0u);
        mask |= c & d;
    }
    if (tmin <= tmid.z && tmid.z <= tmax) {
        const float px = tmid.z * dir.x, py = tmid.z * dir.y;
        const uint32_t e = (px >= cr.x - eps ? 0xF0u : 0u) | (px <= cr.x + eps ? 0x0Fu : 0u);
        const uint32_t f = (py >= cr.y - eps ? 0xCCu : 0u) | (py <= cr.y + eps ? 0x33u : 0u);
        mask |= e & f;
    }
    return mask;
}

__device__ __forceinline__ uint32_t murmur32(uint32_t h) {
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}

__device__ __forceinline__ uint32_t channel(uint32_t v) {
    const float c = float(v & 0xFFu) / 255.0f;
    return uint32_t(fminf(1.0f, fmaxf(0.0f, c)) * 255.0f);
}

// Stack entry: node word index | child mask << 32 | children to visit << 40.
__device__ __forceinline__ uint64_t pack(uint32_t index, uint32_t cm, uint32_t vm) {
    return (uint64_t)index | (uint64_t)cm << 32 | (uint64_t)vm << 40;
}

// ------------------------------------------------ pairs of float32 values ----
// hi + lo, |lo| <= ulp(hi) / 2: the usual error-free sums and products (Dekker
// 1971, Knuth) with fmaf.
struct F2 { float hi, lo; };
__device__ __forceinline__ F2 quick_sum(float a, float b) { const float s = a + b; return {s, b - (s - a)}; }  // |a| >= |b|
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
    const float s = a.hi + b.hi, t = s - a.hi;
    const float e = (a.hi - (s - t)) + (b.hi - t);
    return quick_sum(s, e + (a.lo + b.lo));
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
    const float p = a.hi * b.hi, e = fmaf(a.hi, b.hi, -p);
    return quick_sum(p, fmaf(a.hi, b.lo, fmaf(a.lo, b.hi, e)));
}
__device__ __forceinline__ F2 f2_scale(F2 a, float b) {
    const float p = a.hi * b;
    return quick_sum(p, fmaf(a.lo, b, fmaf(a.hi, b, -p)));
}

// The rule (src/DAGTracer.cu:310-318): direction normalised in double, then float.
__device__ __noinline__ float3 ray_direction_exact(const TraceArgs& a, uint32_t px, uint32_t py) {
    const double vx = a.ray_min[0] + double(px) * a.ray_ddx[0] + double(py) * a.ray_ddy[0] - a.camera[0];
    const double vy = a.ray_min[1] + double(px) * a.ray_ddx[1] + double(py) * a.ray_ddy[1] - a.camera[1];
    const double vz = a.ray_min[2] + double(px) * a.ray_ddx[2] + double(py) * a.ray_ddy[2] - a.camera[2];
    const double s = 1 / sqrt(vx * vx + vy * vy + vz * vz);
    return make_float3(float(s * vx), float(s * vy), float(s * vz));
}

// The same value. With T a bound of the magnitudes that make up a component of
// v (so that the rule's v is off by less than 2^-50 T), the pairs hold v to
// 2^-45 T, its square sum and the reciprocal root to relative
// 2^-44 + 2^-44 T/|v|, and so the direction to 2^-42.5 T/|v|. A component whose
// rounding to float32 is the same on both sides of 2^-41 T/|v| is the rule's.
__device__ __forceinline__ float3 ray_direction(const TraceArgs& a, uint32_t px, uint32_t py) {
    const float x = (float)px, y = (float)py, T = a.magnitude;
    F2 v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
        v[k] = f2_add(f2_add({a.base[2 * k], a.base[2 * k + 1]}, f2_scale({a.ddx[2 * k], a.ddx[2 * k + 1]}, x)),
                      f2_scale({a.ddy[2 * k], a.ddy[2 * k + 1]}, y));
    const F2 n2 = f2_add(f2_add(f2_mul(v[0], v[0]), f2_mul(v[1], v[1])), f2_mul(v[2], v[2]));
    // 1 / sqrt(n2): the approximation r0 (error below 2^-21), then
    // r0 * (1 + d / 2 + 3 d^2 / 8) with d = 1 - n2 * r0^2.
    const float r0 = rsqrtf(n2.hi);
    const F2 t = f2_mul(n2, f2_mul({r0, 0.0f}, {r0, 0.0f}));
    const float d = (1.0f - t.hi) - t.lo;
    const F2 r = quick_sum(r0, r0 * d * fmaf(0.375f, d, 0.5f));
    const float err = 0x1p-41f * T * r0;
    float out[3];
    bool sure = T > 0.0f && n2.hi >= T * T * 0x1p-24f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const F2 c = f2_mul(v[k], r);
        out[k] = c.hi;
        sure = sure && c.hi + (c.lo + err) == c.hi && c.hi + (c.lo - err) == c.hi;
    }
    if (!sure) return ray_direction_exact(a, px, py);
    return make_float3(out[0], out[1], out[2]);
}

// The child bytes of a leaf half that are not zero, one bit each: the sum
// carries into a byte's top bit unless its low seven are zero, and the product
// moves the four top bits together.
__device__ __forceinline__ uint32_t nonzero_bytes(uint32_t x) {
    const uint32_t t = (((x & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | x) & 0x80808080u;
    return ((t >> 7) * 0x01020408u) >> 24;
}

struct Ray {
    uint32_t pos[3];       // the voxel hit
    uint32_t debug_index;
    bool hit, ok;
};

// One ray. kNarrow: the words' indices fit 32 bits. kTame: no infinity or NaN
// comes up (trace_rays).
template <bool kNarrow, bool kTame>
__device__ __forceinline__ Ray walk(const TraceArgs& a, float3 org, float3 dir, float3 inv) {
    using Index = typename std::conditional<kNarrow, uint32_t, uint64_t>::type;
    const int depth = a.depth, leaf_level = depth - 2;
    const uint32_t* w = a.words;
    const Index nw = (Index)a.n_words;
    bool ok = true;
    auto word = [&](Index i) -> uint32_t {
        if (i >= nw) { ok = false; return 0; }
        return __ldg(w + i);
    };
    const uint32_t order = (dir.x < 0.f ? 4u : 0u) + (dir.y < 0.f ? 2u : 0u) + (dir.z < 0.f ? 1u : 0u);
    const uint32_t debug_at = (uint32_t)(depth - 2) - a.debug_level;  // level entered when the index is noted

    // The levels above that have children left (their bits in `live`), for
    // the ascent in one step.
    uint64_t stack[kTraceMaxDepth];
    uint32_t live = 0;
    uint32_t pos[3] = {0, 0, 0};
    uint32_t debug_index = 0, leaf_lo = 0, leaf_hi = 0;
    int level = 0;
    uint32_t edge = 1u << depth;  // of a node at `level`
    uint32_t index = 0;
    uint32_t cm = word(0) & 0xFFu;
    uint32_t vm = cm & crossed_children<kTame>(true, edge >> 1, pos, org, dir, inv);
    bool hit = false;
    for (uint32_t step = 0;; ++step) {
        if (step >= kTraceMaxSteps) { ok = false; break; }
        if (!vm) {
            // Ascend to the deepest level with a child left.
            if (!live) { pos[0] = pos[1] = pos[2] = 0; break; }
            level = 31 - __clz(live);
            const uint64_t e = stack[level];
            index = (uint32_t)e;
            cm = (uint32_t)(e >> 32) & 0xFFu;
            vm = (uint32_t)(e >> 40) & 0xFFu;
            edge = 1u << (depth - level);
            pos[0] &= 0u - edge;
            pos[1] &= 0u - edge;
            pos[2] &= 0u - edge;
        }
        // Next child in the ray's order: the first set bit of vm after
        // relabelling the children by child ^ order.
        uint32_t seen = vm;
        if (order & 1u) seen = ((seen & 0x55u) << 1) | ((seen >> 1) & 0x55u);
        if (order & 2u) seen = ((seen & 0x33u) << 2) | ((seen >> 2) & 0x33u);
        if (order & 4u) seen = ((seen & 0x0Fu) << 4) | (seen >> 4);
        const uint32_t child = (uint32_t)(__ffs(seen) - 1) ^ order;
        vm &= ~(1u << child);
        edge >>= 1;
        if (child & 4u) pos[0] |= edge;
        if (child & 2u) pos[1] |= edge;
        if (child & 1u) pos[2] |= edge;
        const uint32_t bit = 1u << level;
        live &= ~bit;
        if (vm) {
            stack[level] = pack(index, cm, vm);
            live |= bit;
        }
        ++level;
        if ((uint32_t)level == debug_at) debug_index = index;
        if (level == depth) { hit = true; break; }
        if (level <= leaf_level) {
            const uint32_t ptr = word((Index)index + (Index)(__popc(cm & ((1u << child) - 1u)) + 1));
            if (level < leaf_level) {
                index = ptr;
                cm = word(index) & 0xFFu;
            } else {
                leaf_lo = word(ptr);
                leaf_hi = word((Index)ptr + 1);
                // Sub-block b of the leaf is byte b of the 64-bit mask.
                cm = nonzero_bytes(leaf_lo) | nonzero_bytes(leaf_hi) << 4;
            }
        } else {
            cm = (((child & 4u) ? leaf_hi : leaf_lo) >> ((child & 3u) * 8)) & 0xFFu;
        }
        vm = cm & crossed_children<kTame>(false, edge >> 1, pos, org, dir, inv);
        if (!ok) break;
    }
    return {{pos[0], pos[1], pos[2]}, debug_index, hit, ok};
}

template <bool kNarrow>
__global__ void __launch_bounds__(kTraceThreads) trace_rays(TraceArgs a) {
    const uint32_t px = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t py = blockIdx.y * blockDim.y + threadIdx.y;
    if (px >= a.width || py >= a.height) return;
    const int depth = a.depth;
    const float3 org = make_float3(float(a.camera[0]), float(a.camera[1]), float(a.camera[2]));
    const float3 dir = ray_direction(a, px, py);
    // 1 / double(dir), rounded to float: the float32 quotient is the same (a
    // double holds more than twice a float's bits, and no quotient of a
    // component below 2 is subnormal).
    const float3 inv = make_float3(__frcp_rn(dir.x), __frcp_rn(dir.y), __frcp_rn(dir.z));
    // With a camera below 1e15 and no component below 1e-10, no product of the
    // walk exceeds 1e26.
    const bool tame = fminf(fabsf(dir.x), fminf(fabsf(dir.y), fabsf(dir.z))) > 1e-10f &&
                      fabsf(org.x) < 1e15f && fabsf(org.y) < 1e15f && fabsf(org.z) < 1e15f &&
                      fabsf(dir.x) + fabsf(dir.y) + fabsf(dir.z) < 4.0f;
    const Ray ray = tame ? walk<kNarrow, true>(a, org, dir, inv) : walk<kNarrow, false>(a, org, dir, inv);
    const uint32_t* path = ray.pos;
    const uint32_t debug_index = ray.debug_index;
    const bool hit = ray.hit, ok = ray.ok;
    const uint64_t pix = (uint64_t)py * a.width + px;
    a.colors[pix] = a.debug_level == 0xFFFFFFFFu ? channel(path[0]) | channel(path[1]) << 8 | channel(path[2]) << 16
                                                 : murmur32(debug_index);
    if (a.hits) {
        uint64_t code = ~0ull;
        if (hit) {
            code = 0;
            for (int b = 0; b < depth; ++b)
                code |= (uint64_t)((path[0] >> b) & 1u) << (3 * b + 2) | (uint64_t)((path[1] >> b) & 1u) << (3 * b + 1) |
                        (uint64_t)((path[2] >> b) & 1u) << (3 * b);
        }
        a.hits[pix] = code;
    }
    if (!ok) atomicOr(a.err, kErrBadInput);
}

}  // namespace

void launch_trace(const TraceArgs& args, cudaStream_t s) {
    // The direction's float32 pairs; magnitude 0 (float64 for every ray) where
    // they would leave the range in which float32 products are exact.
    TraceArgs a = args;
    double most = 0.0;
    bool finite = true;
    for (int k = 0; k < 3; ++k) {
        const double v[3] = {a.ray_min[k] - a.camera[k], a.ray_ddx[k], a.ray_ddy[k]};
        float* to[3] = {a.base + 2 * k, a.ddx + 2 * k, a.ddy + 2 * k};
        for (int q = 0; q < 3; ++q) {
            finite = finite && std::fabs(v[q]) < 1e15;
            to[q][0] = (float)v[q];
            to[q][1] = (float)(v[q] - (double)to[q][0]);
        }
        most = std::max(most, std::fabs(a.ray_min[k]) + std::fabs(a.camera[k]) + a.width * std::fabs(v[1]) +
                                  a.height * std::fabs(v[2]));
    }
    a.magnitude = finite && most > 1e-6 && most < 1e15 && a.width < (1u << 24) && a.height < (1u << 24)
                      ? (float)(most * 1.0001)
                      : 0.0f;
    const dim3 block(8, kTraceThreads / 8);
    const dim3 grid((a.width + block.x - 1) / block.x, (a.height + block.y - 1) / block.y);
    if (a.n_words <= 0xFFFFFFF0ull) trace_rays<true><<<grid, block, 0, s>>>(a);
    else trace_rays<false><<<grid, block, 0, s>>>(a);
}

}  // namespace dagc
