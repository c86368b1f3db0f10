// Triangle voxelizer for sm_103a: the fragment producer in front of the DAG
// path. Restates in CUDA the reference's OpenGL voxelization pass
// (src/Voxelizer.cpp:254-369 with Shaders/GeometryShader.glsl and
// Shaders/FragmentShader.glsl), which cannot run on a compute-only box, and
// writes Morton codes to a device buffer, ready for dagc_create.
//
// Two rules:
//   kVoxGL  the reference's: each triangle is projected on the plane of its
//           dominant axis (face normal scaled by the box half-size), every
//           pixel (voxel column) the projection touches is covered
//           (conservative rasterisation), and each covered pixel emits ONE
//           voxel, at the smallest of the plane depths sampled at the pixel
//           centre and corners (truncated, clamped to the grid). float32.
//   kVoxSAT every voxel whose cube the triangle touches, by the separating
//           axis test (Akenine-Moller 2001); float64. The 26-connected
//           surface used for the triangle-soup workload.
//
// Tiles of kVoxTile triangles, a run of them to each warp: its lanes set up one
// triangle each (the constants go to shared memory), then the warp tests them
// one by one, lanes striding over the bounding box (rows of pixels / voxel
// columns), so that large triangles spread over 32 lanes. The hits found while
// counting are kept (packed local positions, per warp) and only their codes are
// left to compute, 32 at a time over all of the warp's triangles, once the
// tiles' counts have given the output offsets through a single decoupled
// look-back. The output order is fixed: triangles in input order, each
// triangle's fragments in bounding-box order. A call without room for codes
// only counts. This file is compiled with --fmad=false: every float operation
// rounds once, as in the CPU oracle (but for the explicit fmaf of the SAT
// filter, whose error bound covers it).
//
// Each form is bound by the arithmetic per candidate (2.7 instructions per SM
// and clock of 4). A counting and a writing call together, 500k triangles, depth
// 12, the GL rule: 2640 us when every lane of the warp repeated the setup and a
// second pass repeated the tests; 684 with one setup by 64 of 256 threads, a
// third of whose time was barriers, and four integer divisions a lane to start
// each box; now 515. 60k triangles, depth 11, the SAT rule: 57 ms in float64
// throughout (of which this part does 2 operations per SM and clock), 0.90 ms
// with the filter, now 0.75.

#include "dagc_device.cuh"
#include "dagc_kernels.h"

#include <type_traits>

namespace dagc {
namespace {

constexpr int kVoxThreads = 128;
constexpr int kVoxWarps = kVoxThreads / 32;
// Most triangles of a tile, and of a warp (consecutive ones): fewer when the
// tiles would be too few for the GPU (voxelize_per).
constexpr int kVoxTile = 64;
constexpr int kVoxPer = kVoxTile / kVoxWarps;
// Tiles below which a warp takes fewer triangles: 8 CTAs on each of 152 SMs
// for the SAT rule (3000 triangles: 299 us for both calls against 748 with 16 a
// warp), 4 for the GL rule, whose triangles are a tenth of the work.
constexpr uint64_t kVoxMinTilesGl = 608, kVoxMinTilesSat = 1216;
// Hits kept per warp from the count to the emission: the triangle in the
// warp's run and the local position, packed.
constexpr int kVoxKeep = 768;
constexpr int kKeepShift = 28;
static_assert(kVoxPer <= 32 && kVoxPer <= 1 << (32 - kKeepShift), "a lane and an id per triangle");

__device__ __forceinline__ uint32_t spread10(uint32_t x) {
    x &= 0x3FFu;
    x = (x | x << 16) & 0x030000FFu;
    x = (x | x << 8) & 0x0300F00Fu;
    x = (x | x << 4) & 0x030C30C3u;
    return (x | x << 2) & 0x09249249u;
}
// The low 11 bits of x, each moved to three times its place.
__device__ __forceinline__ uint64_t spread11(uint32_t x) {
    x &= 0x7FFu;
    const uint64_t top = (uint64_t)(x >> 10) << 30;
    x = (x | x << 16) & 0x030000FFu;
    x = (x | x << 8) & 0x0300F00Fu;
    x = (x | x << 4) & 0x030C30C3u;
    x = (x | x << 2) & 0x09249249u;
    return top | x;
}
__device__ __forceinline__ uint64_t spread21(uint32_t x) { return spread11(x & 0x3FFu) | spread11((x >> 10) & 0x7FFu) << 30; }
// Ten bits of the three coordinates interleave in 32-bit words; G is the same
// for all lanes.
__device__ __forceinline__ uint64_t morton3(uint32_t x, uint32_t y, uint32_t z, int G) {
    if (G > 1 << 20) return spread21(x) << 2 | spread21(y) << 1 | spread21(z);
    const uint32_t lo = spread10(x) << 2 | spread10(y) << 1 | spread10(z);
    if (G <= 1 << 10) return lo;
    const uint32_t hi = spread10(x >> 10) << 2 | spread10(y >> 10) << 1 | spread10(z >> 10);
    return (uint64_t)hi << 30 | lo;
}

// A box of candidates (nz fastest), walked by the lanes of a warp 32 at a time.
// Set up once per triangle: how far 32 candidates on is, and the reciprocals
// that give a lane's first position: (i + 0.5) / n is at least 0.5 / n from a
// whole number, far more than its rounding for i < 32.
struct Box {
    uint32_t nx, ny, nz;
    uint32_t dx, dy, dz;
    float ry, rz;
    __device__ void set(uint32_t x, uint32_t y, uint32_t z) {
        nx = x; ny = y; nz = z;
        if (x == 0 || y == 0 || z == 0) return;
        dz = 32 % z;
        const uint32_t rows = 32 / z;
        dy = x == 1 ? rows : rows % y;  // one layer: the rows past its last end the walk
        dx = rows / y;
        ry = 1.0f / (float)y;
        rz = 1.0f / (float)z;
    }
};

// ---------------------------------------------------------------- GL rule --
struct GlTri {
    int axis;
    float U[3], V[3], W[3];
    float dwdu, dwdv;
    float nx[3], ny[3], dk[3];
    int i0, j0;
    Box box;  // (1, rows, columns); no columns: empty
};

__device__ __forceinline__ int lo_cell(float m, float Gf) {
    const int i = (int)floorf(fminf(fmaxf(m, -1.0f), Gf));
    return i < 0 ? 0 : i;
}
__device__ __forceinline__ int hi_cell(float m, float Gf, int G) {
    const int i = (int)floorf(fminf(fmaxf(m, -1.0f), Gf));
    return i > G - 1 ? G - 1 : i;
}
__device__ __forceinline__ int clamp_cell(float z, int G) {
    const int k = (int)fminf(fmaxf(z, -1.0f), (float)G);
    return k < 0 ? 0 : (k > G - 1 ? G - 1 : k);
}

__device__ void gl_setup(const double* P, const double* aabb, int depth, GlTri& t) {
    const int G = 1 << depth;
    const float Gf = (float)G;
    float p[3][3], mn[3], mx[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a) p[k][a] = (float)P[3 * k + a];
#pragma unroll
    for (int a = 0; a < 3; ++a) { mn[a] = (float)aabb[a]; mx[a] = (float)aabb[3 + a]; }
    const float e1[3] = {p[1][0] - p[0][0], p[1][1] - p[0][1], p[1][2] - p[0][2]};
    const float e2[3] = {p[2][0] - p[0][0], p[2][1] - p[0][1], p[2][2] - p[0][2]};
    const float c[3] = {e1[1] * e2[2] - e1[2] * e2[1], e1[2] * e2[0] - e1[0] * e2[2], e1[0] * e2[1] - e1[1] * e2[0]};
    const float len = sqrtf(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
    float nd[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) nd[a] = fabsf((c[a] / len) * ((mx[a] - mn[a]) * 0.5f));
    t.axis = nd[0] >= nd[2] ? (nd[0] >= nd[1] ? 0 : 1) : (nd[1] >= nd[2] ? 1 : 2);
    // View axes: X -> (u, v, w) = (z, y, x), Y -> (x, z, y), Z -> (y, x, z).
    const int ua = t.axis == 0 ? 2 : (t.axis == 1 ? 0 : 1);
    const int va = t.axis == 0 ? 1 : (t.axis == 1 ? 2 : 0);
    const int wa = t.axis;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        float g[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) g[a] = (p[k][a] - mn[a]) * (Gf / (mx[a] - mn[a]));
        t.U[k] = g[ua];
        t.V[k] = g[va];
        t.W[k] = g[wa];
    }
    const float e1u = t.U[1] - t.U[0], e1v = t.V[1] - t.V[0], e1w = t.W[1] - t.W[0];
    const float e2u = t.U[2] - t.U[0], e2v = t.V[2] - t.V[0], e2w = t.W[2] - t.W[0];
    const float det = e1u * e2v - e2u * e1v;
    bool empty = !(det != 0.0f) || !isfinite(det);
    t.dwdu = (e1w * e2v - e2w * e1v) / det;
    t.dwdv = (e2w * e1u - e1w * e2u) / det;
    const float sgn = det > 0.0f ? 1.0f : -1.0f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const int k1 = k == 2 ? 0 : k + 1;
        t.nx[k] = -(t.V[k1] - t.V[k]) * sgn;
        t.ny[k] = (t.U[k1] - t.U[k]) * sgn;
        t.dk[k] = fmaxf(t.nx[k], 0.0f) + fmaxf(t.ny[k], 0.0f);
    }
    t.i0 = lo_cell(fminf(t.U[0], fminf(t.U[1], t.U[2])), Gf);
    const int i1 = hi_cell(fmaxf(t.U[0], fmaxf(t.U[1], t.U[2])), Gf, G);
    t.j0 = lo_cell(fminf(t.V[0], fminf(t.V[1], t.V[2])), Gf);
    const int j1 = hi_cell(fmaxf(t.V[0], fmaxf(t.V[1], t.V[2])), Gf, G);
    if (t.i0 > i1 || t.j0 > j1) empty = true;
    t.box.set(1, (uint32_t)(j1 - t.j0 + 1), empty ? 0u : (uint32_t)(i1 - t.i0 + 1));
}

// Is pixel (i, j) covered?
__device__ __forceinline__ bool gl_covered(const GlTri& t, int i, int j) {
    bool covered = true;
#pragma unroll
    for (int k = 0; k < 3; ++k)
        covered = covered && t.nx[k] * ((float)i - t.U[k]) + t.ny[k] * ((float)j - t.V[k]) + t.dk[k] >= 0.0f;
    return covered;
}
// The Morton code of a covered pixel's voxel.
__device__ __forceinline__ uint64_t gl_code(const GlTri& t, int i, int j, int G) {
    const float zc = t.W[0] + t.dwdu * (((float)i + 0.5f) - t.U[0]) + t.dwdv * (((float)j + 0.5f) - t.V[0]);
    const float hx = 0.5f * t.dwdu, hy = 0.5f * t.dwdv;
    const int s0 = clamp_cell(zc, G);
    const int s1 = clamp_cell(zc + hx + hy, G), s2 = clamp_cell(zc + hx - hy, G);
    const int s3 = clamp_cell(zc - hx + hy, G), s4 = clamp_cell(zc - hx - hy, G);
    const int k = min(min(min(s0, s1), min(s2, s3)), s4);
    // View axes back: X (u, v, w) = (z, y, x), Y (x, z, y), Z (y, x, z).
    const uint32_t u = (uint32_t)i, v = (uint32_t)j, w = (uint32_t)k;
    return morton3(t.axis == 0 ? w : t.axis == 1 ? u : v, t.axis == 0 ? v : t.axis == 1 ? w : u,
                   t.axis == 0 ? u : t.axis == 1 ? v : w, G);
}

// --------------------------------------------------------------- SAT rule --
struct D3 { double x, y, z; };
__device__ __forceinline__ D3 dsub(D3 a, D3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ D3 dcross(D3 a, D3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ double ddot(D3 a, D3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double dmin(double a, double b) { return b < a ? b : a; }  // std::min
__device__ __forceinline__ double dmax(double a, double b) { return a < b ? b : a; }  // std::max

// Triangle (a, b, d) against the cube of half-size h around c: 9 edge-cross
// axes, the 3 box normals, the triangle normal; touching counts as overlap.
__device__ bool tri_box(D3 c, double h, D3 a, D3 b, D3 d) {
    const D3 v0 = dsub(a, c), v1 = dsub(b, c), v2 = dsub(d, c);
    const D3 e[3] = {dsub(v1, v0), dsub(v2, v1), dsub(v0, v2)};
    const D3 ax[3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
#pragma unroll
    for (int i = 0; i < 3; ++i) {
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const D3 axis = dcross(ax[i], e[j]);
            const double p0 = ddot(axis, v0), p1 = ddot(axis, v1), p2 = ddot(axis, v2);
            const double mn = dmin(p0, dmin(p1, p2));
            const double mx = dmax(p0, dmax(p1, p2));
            const double r = h * (fabs(axis.x) + fabs(axis.y) + fabs(axis.z));
            if (mn > r || mx < -r) return false;
        }
    }
    if (dmin(v0.x, dmin(v1.x, v2.x)) > h || dmax(v0.x, dmax(v1.x, v2.x)) < -h) return false;
    if (dmin(v0.y, dmin(v1.y, v2.y)) > h || dmax(v0.y, dmax(v1.y, v2.y)) < -h) return false;
    if (dmin(v0.z, dmin(v1.z, v2.z)) > h || dmax(v0.z, dmax(v1.z, v2.z)) < -h) return false;
    const D3 nrm = dcross(e[0], e[1]);
    const double dist = ddot(nrm, v0);
    const double r = h * (fabs(nrm.x) + fabs(nrm.y) + fabs(nrm.z));
    return fabs(dist) <= r;
}

__device__ __forceinline__ D3 sat_vertex(const double* P, const double* aabb, const double* scale, int k) {
    return {(P[3 * k + 0] - aabb[0]) * scale[0], (P[3 * k + 1] - aabb[1]) * scale[1], (P[3 * k + 2] - aabb[2]) * scale[2]};
}
// The rule itself, for one voxel: float64, in the oracle's order.
__device__ __noinline__ bool sat_exact(const VoxArgs& a, uint64_t tri, int64_t x, int64_t y, int64_t z) {
    const double* P = a.vertices + 9 * tri;
    const D3 c{(double)x + 0.5, (double)y + 0.5, (double)z + 0.5};
    return tri_box(c, 0.5, sat_vertex(P, a.aabb, a.scale, 0), sat_vertex(P, a.aabb, a.scale, 1),
                   sat_vertex(P, a.aabb, a.scale, 2));
}

// A triangle's float32 filter. Its tests are tri_box's, rewritten for a fixed
// triangle and a moving voxel centre c: the triangle's projection on an axis is
// separated from the cube's when |axis . c - mid| > half, with mid and half
// from the triangle alone. Coordinates are relative to an integer origin near
// the box's centre; K bounds every |coordinate| and |c|. With u = 2^-24, the
// float32 coordinates are off by uK, the edges by 4uK, an edge axis's
// axis . c by 14uK^2, its mid and half by 24uK^2 (the cross products with unit
// vectors are single components); the normal by 50uK^2, normal . c and its mid
// by 250uK^3 each; the float64 rule itself by less than a unit of these. So
// beyond half + 128uK^2 (1024uK^3 for the normal) an axis separates for sure,
// below half minus that it does not; a voxel that no axis separates for sure
// and some axis leaves open is decided by sat_exact. The three box normals
// never separate a voxel of the bounding box. K above 2^16, or not a number:
// every voxel by sat_exact.
struct SatTri {
    float e[3][3];                                  // edges v1 - v0, v2 - v1, v0 - v2
    float mid[3][3], out[3][3], in[3][3];           // per box axis i and edge j
    float n[3], nmid, nout, nin;
    int x0, y0, z0;                                  // bounding box origin
    Box box;                                         // and extents (0: empty)
    int ox, oy, oz;                                  // the filter's origin
    bool exact;
};

__device__ __forceinline__ int64_t cell_floor(double m, double G) { return (int64_t)floor(dmin(dmax(m, -1.0), G)); }

__device__ void sat_setup(const VoxArgs& args, uint64_t tri, SatTri& t) {
    const double* P = args.vertices + 9 * tri;
    const double G = (double)((int64_t)1 << args.depth);
    const int64_t Gi = (int64_t)1 << args.depth;
    const D3 v[3] = {sat_vertex(P, args.aabb, args.scale, 0), sat_vertex(P, args.aabb, args.scale, 1),
                     sat_vertex(P, args.aabb, args.scale, 2)};
    const D3 a = v[0], b = v[1], c = v[2];
    int64_t x0 = cell_floor(dmin(a.x, dmin(b.x, c.x)), G), x1 = cell_floor(dmax(a.x, dmax(b.x, c.x)), G);
    int64_t y0 = cell_floor(dmin(a.y, dmin(b.y, c.y)), G), y1 = cell_floor(dmax(a.y, dmax(b.y, c.y)), G);
    int64_t z0 = cell_floor(dmin(a.z, dmin(b.z, c.z)), G), z1 = cell_floor(dmax(a.z, dmax(b.z, c.z)), G);
    x0 = x0 < 0 ? 0 : x0; y0 = y0 < 0 ? 0 : y0; z0 = z0 < 0 ? 0 : z0;
    x1 = x1 > Gi - 1 ? Gi - 1 : x1; y1 = y1 > Gi - 1 ? Gi - 1 : y1; z1 = z1 > Gi - 1 ? Gi - 1 : z1;
    const int nx = x1 >= x0 ? (int)(x1 - x0 + 1) : 0;
    const int ny = y1 >= y0 ? (int)(y1 - y0 + 1) : 0;
    const int nz = z1 >= z0 ? (int)(z1 - z0 + 1) : 0;
    t.box.set((uint32_t)nx, (uint32_t)ny, (uint32_t)nz);
    t.x0 = (int)x0; t.y0 = (int)y0; t.z0 = (int)z0;
    t.exact = true;
    if (nx == 0 || ny == 0 || nz == 0) return;
    t.ox = t.x0 + nx / 2;
    t.oy = t.y0 + ny / 2;
    t.oz = t.z0 + nz / 2;
    float f[3][3];
    float K = (float)(max(nx, max(ny, nz)) / 2 + 2);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        f[k][0] = (float)(v[k].x - (double)t.ox);
        f[k][1] = (float)(v[k].y - (double)t.oy);
        f[k][2] = (float)(v[k].z - (double)t.oz);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            if (!(fabsf(f[k][x]) <= 65536.0f)) return;  // far outside the grid, or not a number
            K = fmaxf(K, fabsf(f[k][x]) + 1.0f);
        }
    }
    if (!(K <= 65536.0f)) return;
    t.exact = false;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        t.e[0][x] = f[1][x] - f[0][x];
        t.e[1][x] = f[2][x] - f[1][x];
        t.e[2][x] = f[0][x] - f[2][x];
    }
    const float slack = 0x1p-17f * K * K;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        // Box axis i crossed with edge e: components y = -e_z, z = e_y in the
        // cyclic order (i, y, z) of the coordinates.
        const int y = (i + 1) % 3, z = (i + 2) % 3;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const float ey = t.e[j][y], ez = t.e[j][z];
            // The edge's two ends project alike; the third vertex is j + 2.
            const int o = (j + 2) % 3;
            const float p = ey * f[j][z] - ez * f[j][y], q = ey * f[o][z] - ez * f[o][y];
            const float half = 0.5f * (fabsf(ey) + fabsf(ez)) + 0.5f * fabsf(p - q);
            t.mid[i][j] = 0.5f * (p + q);
            t.out[i][j] = half + slack;
            t.in[i][j] = half - slack;
        }
    }
    float r = 0.0f, d = 0.0f;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int y = (i + 1) % 3, z = (i + 2) % 3;
        t.n[i] = t.e[0][y] * t.e[1][z] - t.e[0][z] * t.e[1][y];
        r += 0.5f * fabsf(t.n[i]);
        d += t.n[i] * f[0][i];
    }
    const float nslack = 0x1p-14f * K * K * K;
    t.nmid = d;
    t.nout = r + nslack;
    t.nin = r - nslack;
}

// Whether voxel (x, y, z) of the bounding box is hit.
__device__ __forceinline__ bool sat_hit(const VoxArgs& a, uint64_t tri, const SatTri& t, int x, int y, int z) {
    bool open = t.exact;
    if (!t.exact) {
        const float c[3] = {(float)(x - t.ox) + 0.5f, (float)(y - t.oy) + 0.5f, (float)(z - t.oz) + 0.5f};
        const float s = fabsf(fmaf(t.n[0], c[0], fmaf(t.n[1], c[1], t.n[2] * c[2])) - t.nmid);
        if (s > t.nout) return false;
        open = s > t.nin;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int u = (i + 1) % 3, w = (i + 2) % 3;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const float q = fabsf(fmaf(t.e[j][u], c[w], -(t.e[j][w] * c[u])) - t.mid[i][j]);
                if (q > t.out[i][j]) return false;
                open |= q > t.in[i][j];
            }
        }
    }
    return !open || sat_exact(a, tri, x, y, z);
}

// ------------------------------------------------------------------ kernel --
template <int kMode>
struct VoxSmem {
    typename std::conditional<kMode == kVoxGL, GlTri, SatTri>::type tri[kVoxTile];
    uint64_t warp_total[kVoxWarps];
    uint64_t base;
    uint32_t kept[kVoxWarps][kVoxKeep];
    uint32_t slot;
};

// The code of candidate (x, y, z) of a triangle's box.
template <int kMode, typename Tri>
__device__ __forceinline__ uint64_t code_of(const Tri& t, uint32_t x, uint32_t y, uint32_t z, int G) {
    if constexpr (kMode == kVoxGL) return gl_code(t, t.i0 + (int)z, t.j0 + (int)y, G);
    else return morton3((uint32_t)t.x0 + x, (uint32_t)t.y0 + y, (uint32_t)t.z0 + z, G);
}

// The warp tests a triangle, lanes striding over its box in order. kEmit: the
// hits' codes go out from `pos` on. Otherwise they are counted and, where
// `keep` is set, kept from `at` on with the triangle's id; *keep is cleared
// once one does not fit. Every lane runs the same trip count, so each ballot
// is made by all 32 lanes.
template <int kMode, bool kEmit, typename Tri>
__device__ __forceinline__ uint64_t warp_triangle(const VoxArgs& a, const Tri& tri_s, uint64_t tri, uint32_t id, uint64_t pos,
                                                  uint32_t* kept, uint32_t at, bool* keep) {
    const uint32_t lane = threadIdx.x & 31;
    const Box box = tri_s.box;
    const uint64_t area = (uint64_t)box.nx * box.ny * box.nz;
    if (area == 0) return 0;
    // What the GL tests read fits registers; the SAT's 45 words stay shared.
    typename std::conditional<kMode == kVoxGL, const Tri, const Tri&>::type t = tri_s;
    const int G = 1 << a.depth;
    if (!kEmit && (kMode == kVoxGL ? (box.ny | box.nz) >> 14 : (box.nx | box.ny) >> 9 | box.nz >> 10)) *keep = false;
    const bool keeps = !kEmit && *keep;
    // The lane's position moves on without a division.
    const uint32_t row = (uint32_t)(((float)lane + 0.5f) * box.rz);
    uint32_t z = lane - row * box.nz, y = row, x = 0;
    if constexpr (kMode != kVoxGL) {
        x = (uint32_t)(((float)row + 0.5f) * box.ry);
        y = row - x * box.ny;
    }
    uint64_t n = 0;
    for (uint64_t b = 0; b < area; b += 32) {
        bool hit = b + lane < area;
        if constexpr (kMode == kVoxGL) hit = hit && gl_covered(t, t.i0 + (int)z, t.j0 + (int)y);
        else hit = hit && sat_hit(a, tri, t, t.x0 + (int)x, t.y0 + (int)y, t.z0 + (int)z);
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, hit);
        if (hit) {
            const uint64_t o = n + __popc(m & lanemask_lt());
            if constexpr (kEmit) {
                if (pos + o < a.capacity) a.codes[pos + o] = code_of<kMode>(t, x, y, z, G);
            } else if (keeps && at + o < (uint64_t)kVoxKeep) {
                kept[at + o] = id << kKeepShift | (kMode == kVoxGL ? y << 14 | z : x << 19 | y << 10 | z);
            }
        }
        n += __popc(m);
        z += box.dz;
        y += box.dy;
        x += box.dx;
        if (z >= box.nz) { z -= box.nz; ++y; }
        if constexpr (kMode != kVoxGL)
            if (y >= box.ny) { y -= box.ny; ++x; }
    }
    if (!kEmit && at + n > (uint64_t)kVoxKeep) *keep = false;
    return n;
}

template <int kMode>
__global__ void __launch_bounds__(kVoxThreads, 8) voxelize(VoxArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    VoxSmem<kMode>& S = *reinterpret_cast<VoxSmem<kMode>*>(smem_raw);
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = 1 << a.depth;
    const uint32_t per = (uint32_t)a.per;
    const uint64_t ntiles = (a.n_tri + per * kVoxWarps - 1) / (per * kVoxWarps);
    auto* tris = S.tri + warp * kVoxPer;  // the warp's own: no barrier between setup, tests and emission
    uint32_t* kept = S.kept[warp];
    while (true) {
        if (tid == 0) S.slot = atomicAdd(a.tile_counter, 1u);
        __syncthreads();
        const uint64_t tile = S.slot;
        if (tile >= ntiles) break;
        const uint64_t t0 = (tile * kVoxWarps + warp) * per;
        const uint32_t mine = t0 >= a.n_tri ? 0u : (uint32_t)(a.n_tri - t0 < per ? a.n_tri - t0 : per);
        if (lane < mine) {
            if constexpr (kMode == kVoxGL) gl_setup(a.vertices + 9 * (t0 + lane), a.aabb, a.depth, tris[lane]);
            else sat_setup(a, t0 + lane, tris[lane]);
        }
        __syncwarp();
        uint64_t count = 0;
        bool keep = a.capacity != 0;
        for (uint32_t k = 0; k < mine; ++k)
            count += warp_triangle<kMode, false>(a, tris[k], t0 + k, k, 0, kept, keep ? (uint32_t)count : 0u, &keep);
        if (lane == 0) S.warp_total[warp] = count;
        __syncthreads();
        if (warp == 0) {
            uint64_t total = 0;
#pragma unroll
            for (int w = 0; w < kVoxWarps; ++w) total += S.warp_total[w];
            const uint64_t b = sv_lookback(a.status, (uint32_t)tile, total, a.err);
            if (lane == 0) {
                S.base = b;
                if (tile == ntiles - 1) *a.d_total = b + total;
            }
        }
        __syncthreads();
        uint64_t base = S.base;
        for (uint32_t w = 0; w < warp; ++w) base += S.warp_total[w];
        if (base >= a.capacity) continue;
        if (keep) {
            // Every hit was kept: all lanes take hits, of whichever triangle.
            for (uint32_t j = lane; j < (uint32_t)count; j += 32) {
                const uint32_t e = kept[j];
                const auto& t = tris[e >> kKeepShift];
                uint64_t code;
                if constexpr (kMode == kVoxGL) code = code_of<kMode>(t, 0, (e >> 14) & 0x3FFFu, e & 0x3FFFu, G);
                else code = code_of<kMode>(t, (e >> 19) & 0x1FFu, (e >> 10) & 0x1FFu, e & 0x3FFu, G);
                if (base + j < a.capacity) a.codes[base + j] = code;
            }
            __syncwarp();
        } else {
            for (uint32_t k = 0; k < mine; ++k) {
                bool unused = false;
                base += warp_triangle<kMode, true>(a, tris[k], t0 + k, k, base, kept, 0u, &unused);
            }
        }
    }
}

// Triangles per warp.
int voxelize_per(uint64_t n_tri, int mode) {
    const uint64_t tiles = mode == kVoxGL ? kVoxMinTilesGl : kVoxMinTilesSat;
    int per = kVoxPer;
    while (per > 1 && n_tri < tiles * kVoxWarps * per) per >>= 1;
    return per;
}

}  // namespace

void voxelize_configure() {
    cudaFuncSetAttribute(voxelize<kVoxGL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(VoxSmem<kVoxGL>));
    cudaFuncSetAttribute(voxelize<kVoxSAT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(VoxSmem<kVoxSAT>));
}

void launch_voxelize(const VoxArgs& args, int grid, cudaStream_t s) {
    VoxArgs a = args;
    a.per = voxelize_per(a.n_tri, a.mode);
    for (int k = 0; k < 3; ++k) a.scale[k] = (double)((int64_t)1 << a.depth) / (a.aabb[3 + k] - a.aabb[k]);
    if (a.mode == kVoxGL) voxelize<kVoxGL><<<grid, kVoxThreads, sizeof(VoxSmem<kVoxGL>), s>>>(a);
    else voxelize<kVoxSAT><<<grid, kVoxThreads, sizeof(VoxSmem<kVoxSAT>), s>>>(a);
}

uint64_t voxelize_tiles(uint64_t n_tri, int mode) {
    const uint64_t tile = (uint64_t)voxelize_per(n_tri, mode) * kVoxWarps;
    return (n_tri + tile - 1) / tile;
}

}  // namespace dagc
