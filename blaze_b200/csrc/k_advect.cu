// k_advect.cu — RK3 semi-Lagrangian advection with tricubic interpolation
// (reference src/FluidSolver.cu:431-456, launched for T, U, V, W at 942-945).
//
// A node's trace reads about 120 values (three velocity samples of up to 24,
// one tricubic sample of 64), which makes the pass bound by the L1 cache's data
// path and by instruction issue.  Two kernels:
//  - k_advect_tile, for grids of enough tiles to fill the SMs several times
//    (kTileGrids): a CTA copies the neighbourhood its traces can reach, 40 x 16 x
//    16 nodes of each field for 32 x 8 x 8 nodes, into shared memory, where a
//    sample is one index plus compile-time offsets: two thirds of the
//    instructions.  The tile's origin follows the displacement at the CTA's centre
//    (tile_follow); margins of 4 nodes cover the stages' spread, to 12 cells a step,
//    and the variation of the flow across the CTA.  A sample that leaves the tile
//    reads global memory (out of line).  What the tile loses to k_advect is fast
//    flow whose samples are far apart: a shear of 120 cells a step across 128^3
//    takes 1120 us (917), at 256^3 4870 (4520).  The tile repeats the field's edge
//    nodes beyond its sides, which is what the tricubic's clamped stencil reads, so
//    samples have no edge cases.
//    The last faces of each axis (i = W, j = H, k = D) have blocks of their own.
//  - k_advect, a thread per node and all four fields, from global memory: on a
//    small grid one wave of 1024-thread CTAs that first copy a tile waits longer.
// In both, positions are kept in cells, so no sample multiplies by 1/dx; the first
// stage samples the velocity at the field's own node, where the trilinear weights
// are 0 and 1/2 (33 values for the four fields instead of 96; nodes at the
// domain's sides take the general sample); and the integer and fractional parts
// of a coordinate come from one add of 2^23 rounded down, not from conversions,
// which share a quarter-rate pipe.
// Measured, us (before: every sample general, from global memory): 256^3 2086
// (2648), 128^3 312 (362), 64^3 52 (59 with the density scalar, now 58).
// What bounds the tile kernel: shared-memory wavefronts, 87 % of the peak, two
// per load, since a warp's samples cross a cell boundary somewhere and then two
// of them meet in a bank.
#include "kernels.cuh"

namespace blz {

// The cell of a clamped coordinate and the position inside it.
struct Coord { int i; float f; };

// WIDE: an axis of 2^23 nodes or more.

template <bool WIDE>
__device__ __forceinline__ Coord coord(float c, int n) {
    c = clamp_coord(c, n);
    if (WIDE) {
        const int i = (int)c;
        return {i, c - (float)i};
    }
    const float t = __fadd_rd(c, 8388608.0f);              // 2^23 + floor(c)
    return {__float_as_int(t) & 0x7fffff, c - (t - 8388608.0f)};
}

__device__ __forceinline__ float at(const float *__restrict__ a, int e) { return __ldg(a + e); }

__device__ __forceinline__ float mix(float a, float b, float f) { return fmaf(f, b - a, a); }

// Trilinear sample (src/Grid.h:94-108) from the three coordinates' cells;
// sy, sz: row and plane strides.
__device__ __forceinline__ float tri(const float *__restrict__ a, int sy, int sz, Coord x, Coord y, Coord z) {
    const int q = x.i + sy * y.i + sz * z.i;
    const int q1 = q + sy, q2 = q + sz, q3 = q1 + sz;
    const float r0 = mix(at(a, q), at(a, q + 1), x.f), r1 = mix(at(a, q1), at(a, q1 + 1), x.f);
    const float r2 = mix(at(a, q2), at(a, q2 + 1), x.f), r3 = mix(at(a, q3), at(a, q3 + 1), x.f);
    return mix(mix(r0, r1, y.f), mix(r2, r3, y.f), z.f);
}

struct Vel { const float *__restrict__ u, *__restrict__ v, *__restrict__ w; int W, H, D; };

// Velocity (world units) at a position in cells.
template <bool WIDE>
__device__ __forceinline__ float3 vel_at(const Vel &f, float px, float py, float pz) {
    const Coord xc = coord<WIDE>(px - 0.5f, f.W), yc = coord<WIDE>(py - 0.5f, f.H), zc = coord<WIDE>(pz - 0.5f, f.D);
    const Coord xf = coord<WIDE>(px, f.W + 1), yf = coord<WIDE>(py, f.H + 1), zf = coord<WIDE>(pz, f.D + 1);
    const int rT = f.W, rU = rT + 1;
    return make_float3(tri(f.u, rU, rU * f.H, xf, yc, zc), tri(f.v, rT, rT * (f.H + 1), xc, yf, zc),
                       tri(f.w, rT, rT * f.H, xc, yc, zf));
}

// vel_at out of line: near the domain's sides and outside a tile.
template <bool WIDE>
__device__ __noinline__ float3 vel_side(Vel f, float px, float py, float pz) { return vel_at<WIDE>(f, px, py, pz); }

// Velocity at node (i, j, k) of a field: AXIS -1 the cell centres, 0, 1, 2 the
// U, V, W faces.
template <int AXIS, bool WIDE>
__device__ __forceinline__ float3 vel_node(const Vel &f, int i, int j, int k, float px, float py, float pz) {
    const bool in = (AXIS == 0 ? i >= 1 && i < f.W : i < f.W - 1) && (AXIS == 1 ? j >= 1 && j < f.H : j < f.H - 1) &&
                    (AXIS == 2 ? k >= 1 && k < f.D : k < f.D - 1);
    if (!in) return vel_side<WIDE>(f, px, py, pz);
    const int rT = f.W, rU = rT + 1, pT = rT * f.H, pU = rU * f.H, pV = rT * (f.H + 1);
    const int qu = i + rU * j + pU * k, qv = i + rT * j + pV * k, qw = i + rT * j + pT * k;
    auto mean2 = [](const float *a, int q, int s) { return 0.5f * (at(a, q) + at(a, q + s)); };
    auto mean4 = [](const float *a, int q, int lo, int up) {     // over (-lo, 0) x (0, up)
        return 0.25f * ((at(a, q - lo) + at(a, q)) + (at(a, q - lo + up) + at(a, q + up)));
    };
    if (AXIS == 0) return make_float3(at(f.u, qu), mean4(f.v, qv, 1, rT), mean4(f.w, qw, 1, pT));
    if (AXIS == 1) return make_float3(mean4(f.u, qu, rU, 1), at(f.v, qv), mean4(f.w, qw, rT, pT));
    if (AXIS == 2) return make_float3(mean4(f.u, qu, pU, 1), mean4(f.v, qv, pV, rT), at(f.w, qw));
    return make_float3(mean2(f.u, qu, 1), mean2(f.v, qv, rT), mean2(f.w, qw, pT));
}

// Departure point, in cells, of the trace that arrives at (px, py, pz), where the
// velocity is k1, with trilinear velocity samples vel(x, y, z): RK3 (stages at
// 0.5 dt and 0.75 dt, weights 2/9, 3/9, 4/9; FluidSolver.cu:431-456), forward
// Euler (392-407) or midpoint RK2 (409-429).  r = dt / dx.
template <int SCHEME, typename F>
__device__ __forceinline__ float3 trace(float r, float px, float py, float pz, float3 k1, F vel) {
    if (SCHEME == BLZ_ADVECT_EULER) return make_float3(px - r * k1.x, py - r * k1.y, pz - r * k1.z);
    const float h1 = 0.5f * r;
    const float3 k2 = vel(px - h1 * k1.x, py - h1 * k1.y, pz - h1 * k1.z);
    if (SCHEME == BLZ_ADVECT_RK2) return make_float3(px - r * k2.x, py - r * k2.y, pz - r * k2.z);
    const float h2 = 0.75f * r;
    const float3 k3 = vel(px - h2 * k2.x, py - h2 * k2.y, pz - h2 * k2.z);
    const float a = 2.0f / 9.0f, b = 3.0f / 9.0f, c = 4.0f / 9.0f;
    return make_float3(px - r * (a * k1.x + b * k2.x + c * k3.x), py - r * (a * k1.y + b * k2.y + c * k3.y),
                       pz - r * (a * k1.z + b * k2.z + c * k3.z));
}

// The same from global memory, for node (i, j, k) of a field: AXIS -1 the cell
// centres, 0, 1, 2 the U, V, W faces.
template <int SCHEME, int AXIS, bool WIDE>
__device__ __forceinline__ float3 departure(const Vel &f, float r, int i, int j, int k) {
    const float px = (float)i + (AXIS == 0 ? 0.0f : 0.5f), py = (float)j + (AXIS == 1 ? 0.0f : 0.5f);
    const float pz = (float)k + (AXIS == 2 ? 0.0f : 0.5f);
    return trace<SCHEME>(r, px, py, pz, vel_node<AXIS, WIDE>(f, i, j, k, px, py, pz),
                         [&](float x, float y, float z) { return vel_at<WIDE>(f, x, y, z); });
}

// Weights of the Lagrange cubic on nodes -1, 0, 1, 2 (src/Grid.h:148-163).
struct Cubic { float w0, w1, w2, w3; };
__device__ __forceinline__ Cubic cubic(float s) {
    const float s2 = s * s, s3 = s2 * s;
    return {-1.0f / 3.0f * s + 0.5f * s2 - 1.0f / 6.0f * s3, 1.0f - s2 + 0.5f * (s3 - s), s + 0.5f * (s2 - s3),
            1.0f / 6.0f * (s3 - s)};
}
template <bool CLAMP>
__device__ __forceinline__ float apply(const Cubic &c, float q0, float q1, float q2, float q3) {
    const float v = c.w0 * q0 + c.w1 * q1 + c.w2 * q2 + c.w3 * q3;
    return CLAMP ? fmaxf(v, 0.0f) : v;
}

// Separable tricubic (x, then y, then z) of a w x h x d field at a position in
// cells less the field's offsets, with edge-clamped stencil indices; CLAMP
// zeroes negatives after every 1-D stage (src/Grid.h:165-222).
template <bool CLAMP, bool WIDE>
__device__ __forceinline__ float tricubic(const float *__restrict__ a, int w, int h, int d, float gx, float gy,
                                          float gz) {
    const Coord x = coord<WIDE>(gx, w), y = coord<WIDE>(gy, h), z = coord<WIDE>(gz, d);
    const Cubic cx = cubic(x.f), cy = cubic(y.f), cz = cubic(z.f);
    const int sy = w, sz = w * h;
    // steps from node 1 to nodes 0 and 3 along y and z (0 and one node where clamped)
    const int y0 = y.i > 0 ? sy : 0, y3 = y.i < h - 2 ? 2 * sy : sy;
    const int z0 = z.i > 0 ? sz : 0, z3 = z.i < d - 2 ? 2 * sz : sz;
    const int q = x.i + sy * y.i + sz * z.i;
    const int x0 = x.i > 0 ? 1 : 0, x3 = x.i < w - 2 ? 2 : 1;
    auto row = [&](int r) { return apply<CLAMP>(cx, at(a, r - x0), at(a, r), at(a, r + 1), at(a, r + x3)); };
    auto plane = [&](int p) { return apply<CLAMP>(cy, row(p - y0), row(p), row(p + sy), row(p + y3)); };
    return apply<CLAMP>(cz, plane(q - z0), plane(q), plane(q + sz), plane(q + z3));
}

struct AdvectArrays {
    const float *__restrict__ T, *__restrict__ U, *__restrict__ V, *__restrict__ W, *__restrict__ D;
    float *__restrict__ Tn, *__restrict__ Un, *__restrict__ Vn, *__restrict__ Wn, *__restrict__ Dn;
};

// One face of U, V or W (AXIS) from global memory.
template <int SCHEME, int AXIS, bool WIDE>
__device__ __forceinline__ void node_face(const Vel &f, const AdvectArrays &a, float r, int i, int j, int k) {
    const float3 q = departure<SCHEME, AXIS, WIDE>(f, r, i, j, k);
    if (AXIS == 0)
        a.Un[lin(i, j, k, f.W + 1, f.H)] = tricubic<false, WIDE>(f.u, f.W + 1, f.H, f.D, q.x, q.y - 0.5f, q.z - 0.5f);
    else if (AXIS == 1)
        a.Vn[lin(i, j, k, f.W, f.H + 1)] = tricubic<false, WIDE>(f.v, f.W, f.H + 1, f.D, q.x - 0.5f, q.y, q.z - 0.5f);
    else
        a.Wn[lin(i, j, k, f.W, f.H)] = tricubic<false, WIDE>(f.w, f.W, f.H, f.D + 1, q.x - 0.5f, q.y - 0.5f, q.z);
}

// ---- tile ----
constexpr int kTX = 32, kTY = 8, kTZ = 8;              // nodes of a CTA
constexpr int kMargin = 4;
constexpr int kSX = kTX + 2 * kMargin, kSY = kTY + 2 * kMargin, kSZ = kTZ + 2 * kMargin;
constexpr int kTileNodes = kSX * kSY * kSZ;
constexpr int kAdvThreads = 1024;

// The shared tile: arrays U, V, W, T (, density) of kTileNodes, and its origin.
struct Tile { const float *s; int ox, oy, oz; };
enum { kTileU, kTileV, kTileW, kTileT, kTileD };

__device__ __forceinline__ float tile_tri(const float *a, int q, float fx, float fy, float fz) {
    const float *p = a + q;
    const float r0 = mix(p[0], p[1], fx), r1 = mix(p[kSX], p[kSX + 1], fx);
    const float r2 = mix(p[kSX * kSY], p[kSX * kSY + 1], fx), r3 = mix(p[kSX * kSY + kSX], p[kSX * kSY + kSX + 1], fx);
    return mix(mix(r0, r1, fy), mix(r2, r3, fy), fz);
}

// Velocity at a position in cells; from global memory when the tile does not
// cover it.
__device__ __forceinline__ float3 tile_vel(const Tile &t, const Vel &f, float px, float py, float pz) {
    const Coord xc = coord<false>(px - 0.5f, f.W), yc = coord<false>(py - 0.5f, f.H), zc = coord<false>(pz - 0.5f, f.D);
    const Coord xf = coord<false>(px, f.W + 1), yf = coord<false>(py, f.H + 1), zf = coord<false>(pz, f.D + 1);
    const int x0 = xc.i - t.ox, x1 = xf.i - t.ox, y0 = yc.i - t.oy, y1 = yf.i - t.oy, z0 = zc.i - t.oz, z1 = zf.i - t.oz;
    // every index in [0, size - 2]; centre and face indices are at most one apart
    const bool in = (unsigned)x0 < kSX - 1u && (unsigned)x1 < kSX - 1u && (unsigned)y0 < kSY - 1u &&
                    (unsigned)y1 < kSY - 1u && (unsigned)z0 < kSZ - 1u && (unsigned)z1 < kSZ - 1u;
    if (!in) return vel_side<false>(f, px, py, pz);
    const int qc = z0 * kSY, qy = (qc + y0) * kSX;
    return make_float3(tile_tri(t.s + kTileU * kTileNodes, qy + x1, xf.f, yc.f, zc.f),
                       tile_tri(t.s + kTileV * kTileNodes, (qc + y1) * kSX + x0, xc.f, yf.f, zc.f),
                       tile_tri(t.s + kTileW * kTileNodes, (z1 * kSY + y0) * kSX + x0, xc.f, yc.f, zf.f));
}

// Velocity at node (i, j, k) of a field (AXIS as in vel_node), local index q in
// the tile.
template <int AXIS>
__device__ __forceinline__ float3 tile_vel_node(const Tile &t, const Vel &f, int i, int j, int k, float px, float py,
                                                float pz) {
    const bool in = (AXIS == 0 ? i >= 1 && i < f.W : i < f.W - 1) && (AXIS == 1 ? j >= 1 && j < f.H : j < f.H - 1) &&
                    (AXIS == 2 ? k >= 1 && k < f.D : k < f.D - 1);
    const int x = i - t.ox, y = j - t.oy, z = k - t.oz;
    // the node and its neighbours one lower and one higher lie in the tile
    if (!in || (unsigned)(x - 1) >= kSX - 2u || (unsigned)(y - 1) >= kSY - 2u || (unsigned)(z - 1) >= kSZ - 2u)
        return vel_side<false>(f, px, py, pz);
    const int q = (z * kSY + y) * kSX + x;
    constexpr int X = 1, Y = kSX, Z = kSX * kSY;
    const float *u = t.s + kTileU * kTileNodes + q, *v = t.s + kTileV * kTileNodes + q, *w = t.s + kTileW * kTileNodes + q;
    auto mean2 = [](const float *p, int s) { return 0.5f * (p[0] + p[s]); };
    auto mean4 = [](const float *p, int lo, int up) {      // over (-lo, 0) x (0, up)
        return 0.25f * ((p[-lo] + p[0]) + (p[up - lo] + p[up]));
    };
    if (AXIS == 0) return make_float3(u[0], mean4(v, X, Y), mean4(w, X, Z));
    if (AXIS == 1) return make_float3(mean4(u, Y, X), v[0], mean4(w, Y, Z));
    if (AXIS == 2) return make_float3(mean4(u, Z, X), mean4(v, Z, Y), w[0]);
    return make_float3(mean2(u, X), mean2(v, Y), mean2(w, Z));
}

template <bool CLAMP>
__device__ __noinline__ float tricubic_side(const float *__restrict__ a, int w, int h, int d, float gx, float gy,
                                            float gz) {
    return tricubic<CLAMP, false>(a, w, h, d, gx, gy, gz);
}

// tricubic on array `s` of the tile, from global memory (a) where the stencil
// leaves it.
template <bool CLAMP>
__device__ __forceinline__ float tile_tricubic(const Tile &t, const float *s, const float *__restrict__ a, int w, int h,
                                               int d, float gx, float gy, float gz) {
    const Coord x = coord<false>(gx, w), y = coord<false>(gy, h), z = coord<false>(gz, d);
    const int lx = x.i - 1 - t.ox, ly = y.i - 1 - t.oy, lz = z.i - 1 - t.oz;
    if ((unsigned)lx >= kSX - 3u || (unsigned)ly >= kSY - 3u || (unsigned)lz >= kSZ - 3u)
        return tricubic_side<CLAMP>(a, w, h, d, gx, gy, gz);
    const Cubic cx = cubic(x.f), cy = cubic(y.f), cz = cubic(z.f);
    const float *p = s + (lz * kSY + ly) * kSX + lx;
    float zs[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        float ys[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float *r = p + (k * kSY + j) * kSX;
            ys[j] = apply<CLAMP>(cx, r[0], r[1], r[2], r[3]);
        }
        zs[k] = apply<CLAMP>(cy, ys[0], ys[1], ys[2], ys[3]);
    }
    return apply<CLAMP>(cz, zs[0], zs[1], zs[2], zs[3]);
}

template <int SCHEME, int AXIS>
__device__ __forceinline__ float3 tile_departure(const Tile &t, const Vel &f, float r, int i, int j, int k) {
    const float px = (float)i + (AXIS == 0 ? 0.0f : 0.5f), py = (float)j + (AXIS == 1 ? 0.0f : 0.5f);
    const float pz = (float)k + (AXIS == 2 ? 0.0f : 0.5f);
    const float3 k1 = tile_vel_node<AXIS>(t, f, i, j, k, px, py, pz);
    return trace<SCHEME>(r, px, py, pz, k1, [&](float x, float y, float z) { return tile_vel(t, f, x, y, z); });
}

// One node of one field (FIELD 0: T and the density, 1, 2, 3: U, V, W).
template <int SCHEME, bool DENS, int FIELD>
__device__ __forceinline__ void tile_node(const Tile &t, const Vel &f, const AdvectArrays &a, float r, int i, int j, int k) {
    const float3 q = tile_departure<SCHEME, FIELD - 1>(t, f, r, i, j, k);
    if (FIELD == 0) {
        const int e = i + f.W * (j + f.H * k);
        a.Tn[e] = tile_tricubic<true>(t, t.s + kTileT * kTileNodes, a.T, f.W, f.H, f.D, q.x - 0.5f, q.y - 0.5f, q.z - 0.5f);
        if (DENS)
            a.Dn[e] = tile_tricubic<true>(t, t.s + kTileD * kTileNodes, a.D, f.W, f.H, f.D, q.x - 0.5f, q.y - 0.5f, q.z - 0.5f);
    } else if (FIELD == 1) {
        a.Un[i + (f.W + 1) * (j + f.H * k)] = tile_tricubic<false>(t, t.s + kTileU * kTileNodes, f.u, f.W + 1, f.H, f.D,
                                                                   q.x, q.y - 0.5f, q.z - 0.5f);
    } else if (FIELD == 2) {
        a.Vn[i + f.W * (j + (f.H + 1) * k)] = tile_tricubic<false>(t, t.s + kTileV * kTileNodes, f.v, f.W, f.H + 1, f.D,
                                                                   q.x - 0.5f, q.y, q.z - 0.5f);
    } else {
        a.Wn[i + f.W * (j + f.H * k)] = tile_tricubic<false>(t, t.s + kTileW * kTileNodes, f.w, f.W, f.H, f.D + 1,
                                                             q.x - 0.5f, q.y - 0.5f, q.z);
    }
}

// How far the tile's origin follows the displacement d at its centre, before it is
// rounded: three quarters of it, between the trace's stages and its end, as long as
// the end then stays within the margin less the tricubic's one cell; in faster flow
// to two to three cells short of the end, whose samples are the most.  Uniform flow
// of 16 and 25 cells a step, us: 128^3 344 and 355, 256^3 2339 and 2430 (at three
// quarters 413 and 410, 3145 and 3148; every sample general, from global memory: 355
// and 350, 2604 and 2586).
__device__ __forceinline__ float tile_follow(float d) {
    const float m = fabsf(d);
    return copysignf(0.25f * m <= (float)(kMargin - 1) ? 0.75f * m : m - ((float)kMargin - 1.5f), d);
}

template <int SCHEME, bool DENS>
__global__ void __launch_bounds__(kAdvThreads, 1) k_advect_tile(Geom g, AdvectArrays a, int nx, int ny, int ntiles) {
    extern __shared__ float tile_s[];
    const Vel f{a.U, a.V, a.W, g.W, g.H, g.D};
    const float r = g.dt * g.inv_dx;
    if ((int)blockIdx.x >= ntiles) {
        // the last faces of each axis: U at i = W, V at j = H, W at k = D
        int e = ((int)blockIdx.x - ntiles) * kAdvThreads + threadIdx.x;
        const int nu = g.H * g.D, nv = g.W * g.D, nw = g.W * g.H;
        if (e < nu) node_face<SCHEME, 0, false>(f, a, r, g.W, e % g.H, e / g.H);
        else if ((e -= nu) < nv) node_face<SCHEME, 1, false>(f, a, r, e % g.W, g.H, e / g.W);
        else if ((e -= nv) < nw) node_face<SCHEME, 2, false>(f, a, r, e % g.W, e / g.W, g.D);
        return;
    }
    const int bx = blockIdx.x % nx, by = blockIdx.x / nx % ny, bz = blockIdx.x / (nx * ny);
    const int i0 = bx * kTX, j0 = by * kTY, k0 = bz * kTZ;
    Tile t;
    t.s = tile_s;
    {
        const int ci = min(i0 + kTX / 2, g.W - 1), cj = min(j0 + kTY / 2, g.H - 1), ck = min(k0 + kTZ / 2, g.D - 1);
        // within the bounds that keep the origin's arithmetic in range whatever the
        // velocity (0 for a NaN)
        auto shift = [&](float v, int n) {
            const float d = tile_follow(-r * v);
            return d == d ? __float2int_rn(fmaxf(fminf(d, (float)n), -(float)n)) : 0;
        };
        t.ox = i0 - kMargin + shift(__ldg(a.U + ci + (g.W + 1) * (cj + g.H * ck)), g.W);
        t.oy = j0 - kMargin + shift(__ldg(a.V + ci + g.W * (cj + (g.H + 1) * ck)), g.H);
        t.oz = k0 - kMargin + shift(__ldg(a.W + ci + g.W * (cj + g.H * ck)), g.D);
    }
    constexpr int kIters = (kTileNodes + kAdvThreads - 1) / kAdvThreads;
    static_assert(kTileNodes % kAdvThreads == 0, "whole rounds of the tile copy");
#pragma unroll 5
    for (int n = 0; n < kIters; ++n) {
        const int e = threadIdx.x + n * kAdvThreads;
        const int x = e % kSX, yz = e / kSX, y = yz % kSY, z = yz / kSY;
        const int i = max(t.ox + x, 0), j = max(t.oy + y, 0), k = max(t.oz + z, 0);
        const int ic = min(i, g.W - 1), jc = min(j, g.H - 1), kc = min(k, g.D - 1);   // cells; a face axis has one more
        const int c = ic + g.W * (jc + g.H * kc);
        tile_s[kTileU * kTileNodes + e] = __ldg(a.U + (min(i, g.W) + (g.W + 1) * (jc + g.H * kc)));
        tile_s[kTileV * kTileNodes + e] = __ldg(a.V + (ic + g.W * (min(j, g.H) + (g.H + 1) * kc)));
        tile_s[kTileW * kTileNodes + e] = __ldg(a.W + (ic + g.W * (jc + g.H * min(k, g.D))));
        tile_s[kTileT * kTileNodes + e] = __ldg(a.T + c);
        if (DENS) tile_s[kTileD * kTileNodes + e] = __ldg(a.D + c);
    }
    __syncthreads();
    const int i = i0 + (threadIdx.x & 31), j = j0 + ((threadIdx.x >> 5) & 7);
    if (i >= g.W || j >= g.H) return;
    constexpr int kStep = kAdvThreads / (kTX * kTY), kNodes = kTZ / kStep;       // planes apart; nodes a thread
    const int kb = k0 + (threadIdx.x >> 8);
    // field by field, so that the CTA's warps share a field's code
#pragma unroll 1
    for (int n = 0; n < kNodes; ++n) if (kb + n * kStep < g.D) tile_node<SCHEME, DENS, 0>(t, f, a, r, i, j, kb + n * kStep);
#pragma unroll 1
    for (int n = 0; n < kNodes; ++n) if (kb + n * kStep < g.D) tile_node<SCHEME, DENS, 1>(t, f, a, r, i, j, kb + n * kStep);
#pragma unroll 1
    for (int n = 0; n < kNodes; ++n) if (kb + n * kStep < g.D) tile_node<SCHEME, DENS, 2>(t, f, a, r, i, j, kb + n * kStep);
#pragma unroll 1
    for (int n = 0; n < kNodes; ++n) if (kb + n * kStep < g.D) tile_node<SCHEME, DENS, 3>(t, f, a, r, i, j, kb + n * kStep);
}

// A thread per node, its four fields one after another, samples from global
// memory.
template <int SCHEME, bool DENS, bool WIDE>
__global__ void __launch_bounds__(256) k_advect(Geom g, AdvectArrays a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i > g.W || j > g.H || k > g.D) return;
    const Vel f{a.U, a.V, a.W, g.W, g.H, g.D};
    const float r = g.dt * g.inv_dx;
    if (i < g.W && j < g.H && k < g.D) {          // T and the density scalar share one backtrace
        const float3 q = departure<SCHEME, -1, WIDE>(f, r, i, j, k);
        const size_t e = lin(i, j, k, g.W, g.H);
        a.Tn[e] = tricubic<true, WIDE>(a.T, g.W, g.H, g.D, q.x - 0.5f, q.y - 0.5f, q.z - 0.5f);
        if (DENS) a.Dn[e] = tricubic<true, WIDE>(a.D, g.W, g.H, g.D, q.x - 0.5f, q.y - 0.5f, q.z - 0.5f);
    }
    if (j < g.H && k < g.D) node_face<SCHEME, 0, WIDE>(f, a, r, i, j, k);
    if (i < g.W && k < g.D) node_face<SCHEME, 1, WIDE>(f, a, r, i, j, k);
    if (i < g.W && j < g.H) node_face<SCHEME, 2, WIDE>(f, a, r, i, j, k);
}

// Tiles from which on the tile kernel is the faster: six waves on 148 SMs.  128^3
// (1024 tiles) 312 us against 333; 112 x 112 x 104 (728 tiles) 228 us, 0.175 ns a
// cell, where k_advect takes 0.16 at 96^3.
constexpr int kTileGrids = 888;

constexpr int tile_smem(bool dens) { return (dens ? 5 : 4) * kTileNodes * (int)sizeof(float); }

template <int SCHEME>
static cudaError_t prepare_scheme(bool dens) {
    return dens ? allow_smem((const void *)k_advect_tile<SCHEME, true>, tile_smem(true))
                : allow_smem((const void *)k_advect_tile<SCHEME, false>, tile_smem(false));
}

static bool wide(const Geom &g) { return g.W >= (1 << 23) - 1 || g.H >= (1 << 23) - 1 || g.D >= (1 << 23) - 1; }
static dim3 tiles(const Geom &g) { return dim3((g.W + kTX - 1) / kTX, (g.H + kTY - 1) / kTY, (g.D + kTZ - 1) / kTZ); }
static bool tiled(const Geom &g) {
    const dim3 t = tiles(g);
    return !wide(g) && (int)(t.x * t.y * t.z) >= kTileGrids;
}

cudaError_t advect_prepare(const Geom &g, int scheme, bool dens) {
    if (!tiled(g)) return cudaSuccess;
    return scheme == BLZ_ADVECT_EULER ? prepare_scheme<BLZ_ADVECT_EULER>(dens)
           : scheme == BLZ_ADVECT_RK2 ? prepare_scheme<BLZ_ADVECT_RK2>(dens) : prepare_scheme<BLZ_ADVECT_RK3>(dens);
}

template <int SCHEME, bool DENS>
static void launch_scheme(const Geom &g, const AdvectArrays &a, cudaStream_t st) {
    if (!tiled(g)) {
        if (wide(g)) k_advect<SCHEME, DENS, true><<<face_grid(g), face_block(), 0, st>>>(g, a);
        else k_advect<SCHEME, DENS, false><<<face_grid(g), face_block(), 0, st>>>(g, a);
        return;
    }
    constexpr int smem = tile_smem(DENS);
    allow_smem((const void *)k_advect_tile<SCHEME, DENS>, smem);
    const dim3 t = tiles(g);
    const int n = (int)(t.x * t.y * t.z);
    const long long last = (long long)g.H * g.D + (long long)g.W * g.D + (long long)g.W * g.H;
    k_advect_tile<SCHEME, DENS><<<n + (unsigned)((last + kAdvThreads - 1) / kAdvThreads), kAdvThreads, smem, st>>>(
        g, a, (int)t.x, (int)t.y, n);
}

void launch_advect(const Geom &g, const float *T, const float *U, const float *V, const float *W,
                   float *Tn, float *Un, float *Vn, float *Wn, cudaStream_t st, int scheme, const float *D,
                   float *Dn) {
    const AdvectArrays a{T, U, V, W, D, Tn, Un, Vn, Wn, Dn};
    const bool dens = D && Dn;
    if (scheme == BLZ_ADVECT_EULER)
        dens ? launch_scheme<BLZ_ADVECT_EULER, true>(g, a, st) : launch_scheme<BLZ_ADVECT_EULER, false>(g, a, st);
    else if (scheme == BLZ_ADVECT_RK2)
        dens ? launch_scheme<BLZ_ADVECT_RK2, true>(g, a, st) : launch_scheme<BLZ_ADVECT_RK2, false>(g, a, st);
    else
        dens ? launch_scheme<BLZ_ADVECT_RK3, true>(g, a, st) : launch_scheme<BLZ_ADVECT_RK3, false>(g, a, st);
}

} // namespace blz
