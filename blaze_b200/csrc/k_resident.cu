// k_resident.cu — red-black Gauss-Seidel sweeps of a grid that stays on chip
// for the whole batch of sweeps (reference src/FluidSolver.cu:517-599).
//
// A grid of up to about 2.1 million cells (148 SMs) is small enough for the
// SMs' registers and shared memory: one cooperative launch loads p and rhs
// once, runs any number of sweeps and writes p once.  What bounds the small
// grids otherwise is the launch of every half sweep (2 us each in a graph,
// 4 us from the host, whatever the size); here a sweep costs one exchange of
// boundary cells between neighbouring SMs through L2 and the update itself.
//
// Layout.  A CTA owns TY rows and TZ planes of full width; a thread owns one
// quad (four packed cells of a colour, both colours) of two adjacent rows in
// RZ consecutive planes, p in registers and rhs in shared memory.  The z
// neighbours and the y neighbour inside the pair are the thread's own
// registers; the other y neighbours and the z neighbours beyond the RZ planes
// come from shared memory, where every thread publishes what it has updated;
// the x neighbour past the quad comes from a shuffle when rows do not straddle
// warps and the last warp is full, else from shared memory.  Pairs start at
// even rows and RZ and TZ are even, so the row parity of every update is a
// compile-time constant.
//
// One exchange per sweep.  The shared tile carries a border two cells deep of
// the neighbouring CTAs' black cells (zero past the domain's sides).  In the
// red half sweep the CTA also updates the one-cell ring of red cells around
// its own, redundantly with its neighbours, so that the black half sweep has
// every red value it needs; only black cells travel.  Exchanging both colours,
// one cell deep, after each half sweep costs a second trip through L2, which
// is most of a small grid's sweep (64^3: 2.5 us a sweep).
//
// Exchange.  Border cells are sent as {value, epoch, value, epoch} in 16-byte
// stores to a buffer the neighbouring CTA polls: every 8 bytes carry their own
// epoch, so a reader that sees the epoch has the value and no fence or flag
// round trip is needed.  A CTA's threads share out the quads to send and those
// to receive (tables in shared memory, formed at the start), after a barrier:
// polling warps slow the shared-memory reads of updating ones down.  Two
// buffers by epoch parity suffice: a CTA sends epoch e after the barrier that
// followed its reading of e - 1, which its neighbour sent after the barrier
// that followed the reading of e - 2 from the slot e overwrites.  The epochs go
// on from launch to launch (kept per CTA in device memory).
//
// Every wait is bounded (kResWaitNs); a thread that gives up records it, stops
// waiting for the rest of the launch and keeps sending, so the other CTAs do
// not wait for it, and the solver reports BLZ_ERR_TIMEOUT.
//
// Widths that are not multiples of 8 (RAGGED): the last quad of a row is partly
// pad, which the count 0 keeps at 0, and rows are read and written cell by cell,
// once per batch of sweeps.  The counts per lane cost the update 10 to 20 %
// (100^3 3.6 us a sweep, 96^3 2.75); one cell per thread takes 13.8 there.
//
// The operations per cell are gs_quad's, so the bits are those of the segment
// kernel's sweeps.
//
// Measured, us per sweep (in brackets the fastest launch shape of the segment
// kernel in a CUDA graph): 32^3 1.6 (3.8), 64^3 1.8 (4.0), 128 x 64 x 64 2.4,
// 96^3 2.75, 120 x 100 x 84 3.3 (5.3), 128^3 4.0 (6.7).  What bounds it now:
// the trip through L2 (0.4 to 0.6 us one way between two SMs) and the length of
// the instruction chains between the barriers; at 128^3 half of a sweep is the
// two updates (shared-memory wavefronts at 41 % of their peak over a launch, issue at
// 30 %).
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "gs.cuh"
#include "kernels.cuh"

namespace blz {

constexpr unsigned long long kResWaitNs = 1000ull * 1000ull * 1000ull;   // 1 s; a normal wait takes a microsecond

// Dynamic shared memory a CTA may have.  Every kernel's limit is set to this one
// value, once: the limit belongs to the kernel and not to a launch, so a grid's own
// need would lower it between another thread's setting and launch.
constexpr int kResSmem = 226 * 1024;
// Threads a CTA may have: RZ = 2 keeps 32 values of p in registers, RZ = 4
// keeps 64.
template <int RZ> constexpr int res_threads() { return RZ == 2 ? 384 : 256; }
// Border quads a thread polls at a time: as many as a thread has on the small
// tiles (two at most), and all six of a 128^3 grid's.  More loads in flight than
// needed lengthen every poll: 64^3 takes 1.79 us a sweep with 2, 1.91 with 6;
// 128^3 4.02 with 6, 4.55 with 2.
constexpr int kResRecv2 = 2, kResRecv4 = 6;      // RZ = 2 and 4
// Threads that share out the exchange and the ring: those without cells of
// their own, where they have two border quads each or fewer, else all.
__host__ __device__ inline int res_sharers(int threads, int tile, int border) {
    return 2 * (threads - tile) >= border ? threads - tile : threads;
}

// Border quads a CTA receives in one exchange: two cells deep along y and z,
// and the four edges of the box (one cell).
__host__ __device__ inline int res_border(int TY, int TZ, int Wq) { return 4 * (TY + TZ + 1) * Wq; }

struct ResParams {
    int NY, NZ, TY, TZ;
    uint4 *halo;                 // receive buffers: per CTA and epoch parity, 2 uint4 per border quad
    unsigned *epoch;             // one per CTA
    int *err;                    // set when a wait gave up (mapped host memory)
};

__device__ __forceinline__ unsigned long long res_now() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ void ll_store(uint4 *p, float a, float b, unsigned e) {
    asm volatile("st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(__float_as_uint(a)), "r"(e),
                 "r"(__float_as_uint(b)), "r"(e)
                 : "memory");
}
__device__ __forceinline__ uint4 ll_load(const uint4 *p) {
    uint4 v;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}

// The b-th border quad row of a CTA: its row y and plane z in the tile's
// coordinates, the CTA it belongs to (dy, dz) and its place in the border of
// that CTA's border list when the direction is turned round.
struct Border { int y, z, dy, dz, back; };
__device__ __forceinline__ Border res_border_row(int b, int TY, int TZ) {
    const int n = TY + TZ;
    if (b >= 4 * n) {                                    // edges: (-, -), (+, -), (-, +), (+, +)
        const int c = b - 4 * n, dy = c & 1 ? 1 : -1, dz = c & 2 ? 1 : -1;
        return {dy > 0 ? TY : -1, dz > 0 ? TZ : -1, dy, dz, 4 * n + (3 - c)};
    }
    // layer (0: next to the tile), side, place along it; the row a CTA sends as
    // layer l to one side is the layer l of the other side there
    const int layer = b / (2 * n), r = b % (2 * n);
    if (r < 2 * TZ) {
        const int hi = r / TZ, z = r % TZ;
        return {hi ? TY + layer : -1 - layer, z, hi ? 1 : -1, 0, hi ? b - TZ : b + TZ};
    }
    const int hi = (r - 2 * TZ) / TY, y = (r - 2 * TZ) % TY;
    return {y, hi ? TZ + layer : -1 - layer, 0, hi ? 1 : -1, hi ? b - TY : b + TY};
}

// One packed row quad from global memory.  RAGGED: rows of W / 2 cells that are
// not whole quads (nor 16-byte aligned); the lanes past the row read 0.
template <bool RAGGED>
__device__ __forceinline__ float4 res_load(const float *p, int lanes) {
    if (!RAGGED) return __ldcg(reinterpret_cast<const float4 *>(p));
    float4 v = make_float4(__ldcg(p), 0.f, 0.f, 0.f);
    if (lanes > 1) v.y = __ldcg(p + 1);
    if (lanes > 2) v.z = __ldcg(p + 2);
    if (lanes > 3) v.w = __ldcg(p + 3);
    return v;
}
template <bool RAGGED>
__device__ __forceinline__ void res_store(float *p, float4 v, int lanes) {
    if (!RAGGED) { *reinterpret_cast<float4 *>(p) = v; return; }
    p[0] = v.x;
    if (lanes > 1) p[1] = v.y;
    if (lanes > 2) p[2] = v.z;
    if (lanes > 3) p[3] = v.w;
}

// gs_quad with a count per lane: `in` inside the row, `end` in the cell at the
// row's end (lane 0 of its first quad where s = 0, the last valid lane of its
// last where s = 1), 0 past it, so that the pad stays 0.
__device__ __forceinline__ float4 res_quad_ragged(float scale, int s, float4 r, float4 o, float xe, float4 ym, float4 yp,
                                                  float4 zm, float4 zp, float2 in, float2 end, bool first, bool last,
                                                  int lanes) {
    auto pick = [&](int t) {
        const bool at_end = s == 0 ? first && t == 0 : last && t == lanes - 1;
        return t >= lanes ? make_float2(0.0f, 0.0f) : at_end ? end : in;
    };
    const float2 d0 = pick(0), d1 = pick(1), d2 = pick(2), d3 = pick(3);
    const f2_t sc = f2(scale, scale);
    const f2_t xl01 = s == 0 ? f2(xe, o.x) : f2(o.x, o.y), xl23 = s == 0 ? f2(o.y, o.z) : f2(o.z, o.w);
    const f2_t xr01 = s == 0 ? f2(o.x, o.y) : f2(o.y, o.z), xr23 = s == 0 ? f2(o.z, o.w) : f2(o.w, xe);
    const f2_t a = gs_pair(sc, f2(r.x, r.y), xl01, xr01, f2(ym.x, ym.y), f2(yp.x, yp.y), f2(zm.x, zm.y),
                           f2(zp.x, zp.y), f2(d0.x, d1.x), f2(d0.y, d1.y));
    const f2_t b = gs_pair(sc, f2(r.z, r.w), xl23, xr23, f2(ym.z, ym.w), f2(yp.z, yp.w), f2(zm.z, zm.w),
                           f2(zp.z, zp.w), f2(d2.x, d3.x), f2(d2.y, d3.y));
    float4 out;
    f2_split(a, out.x, out.y);
    f2_split(b, out.z, out.w);
    return out;
}

// The CTA `cta` of a grid's.
template <int RZ, bool WARPROW, bool RAGGED>
__device__ __forceinline__ void res_sweeps(const Geom &g, const SolveParams &sp, const float *__restrict__ rhs_r,
                                           const float *__restrict__ rhs_b, float *p_r, float *p_b, int sweeps,
                                           const ResParams &rs, int cta) {
    extern __shared__ __align__(16) float4 sm[];
    __shared__ float2 inv[8];
    constexpr int NR = RZ == 2 ? kResRecv2 : kResRecv4;
    const int Wh = g.W >> 1, Wq = (Wh + 3) >> 2, TY = rs.TY, TZ = rs.TZ, NRP = TY >> 1, nthr = blockDim.x;
    const int by = cta % rs.NY, bz = cta / rs.NY;
    const int mq = threadIdx.x % Wq, rp = (threadIdx.x / Wq) % NRP, zg = threadIdx.x / (Wq * NRP);
    const bool live = zg * RZ < TZ;                      // threads beyond the tile only exchange
    const int jA = by * TY + 2 * rp, k0 = bz * TZ + zg * RZ;
    const bool okA = live && jA < g.H, okB = live && jA + 1 < g.H;
    const int pl = Wh * g.H, gA = 4 * mq + Wh * jA + pl * k0;    // element offset of row A, plane k0
    const bool first = mq == 0, last = mq == Wq - 1;
    const int tail = Wh - 4 * (Wq - 1), lanes = last ? tail : 4;     // valid cells of the last quad; of this thread's
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    // Shared memory: p of both colours on planes -2..TZ+1 and rows -2..TY+1;
    // rhs of the tile; rhs of the red ring; the tables.
    const int prow = Wq, pplane = (TY + 4) * Wq, pcol = (TZ + 4) * pplane;
    const int rplane = TY * Wq, rcol = TZ * rplane, ring = 2 * (TY + TZ) * Wq, border = res_border(TY, TZ, Wq);
    auto quad = [&](int y, int z, int m) { return m + prow * (y + 2) + pplane * (z + 2); };
    const int own = live ? quad(2 * rp, zg * RZ, mq) : 0;
    float4 *const rhs = sm + 2 * pcol + (live ? mq + Wq * (2 * rp + TY * zg * RZ) : 0);
    float4 *const ring_rhs = sm + 2 * pcol + 2 * rcol;
    int *const t_dst = reinterpret_cast<int *>(ring_rhs + 2 * ring); // border quad: its place in the tile (-1: none)
    int *const t_src = t_dst + border, *const t_to = t_src + border; // what is sent for it and where to
    float4 *const ring_den = ring_rhs + ring;                        // reciprocals (hi, lo) inside the quad and at the row's end
    int *const t_cell = t_to + border;                               // ring quad: parity, at its row's end (x neighbour missing), last quad

    for (int q = threadIdx.x; q < 2 * pcol; q += nthr) sm[q] = zero4;
    if (threadIdx.x < 8)
        inv[threadIdx.x] = threadIdx.x ? make_float2(inv_count((float)threadIdx.x), inv_count_lo((float)threadIdx.x))
                                       : make_float2(0.0f, 0.0f);
    const bool dir = sp.dirichlet;
    auto has = [&](bool neighbour, bool open) { return neighbour || (dir && open) ? 1 : 0; };
    auto count_y = [&](int j) { return has(j > 0, sp.open.ylo) + has(j < g.H - 1, sp.open.yhi); };
    auto count_z = [&](int k) { return has(k > 0, sp.open.zlo) + has(k < g.D - 1, sp.open.zhi); };
    const int x_lo = dir && sp.open.xlo ? 0 : 1, x_hi = dir && sp.open.xhi ? 0 : 1;   // a row end's count is less by
    __syncthreads();
    for (int q = threadIdx.x; q < border; q += nthr) {
        const int m = q % Wq;
        const Border b = res_border_row(q / Wq, TY, TZ);
        const bool ok = by + b.dy >= 0 && by + b.dy < rs.NY && bz + b.dz >= 0 && bz + b.dz < rs.NZ;
        // the border's cell in the grid, and the cell sent in its place: the
        // mirror image of the border's place, in this tile
        const int j = by * TY + b.y, k = bz * TZ + b.z;
        const int sy = b.dy ? (b.dy > 0 ? 2 * TY - 1 - b.y : -1 - b.y) : b.y;
        const int sz = b.dz ? (b.dz > 0 ? 2 * TZ - 1 - b.z : -1 - b.z) : b.z;
        const bool in = ok && j < g.H && k < g.D;
        t_dst[q] = in ? quad(b.y, b.z, m) : -1;
        t_src[q] = quad(sy, sz, m);
        t_to[q] = ok && by * TY + sy < g.H && bz * TZ + sz < g.D
                      ? 4 * border * (cta + b.dy + b.dz * rs.NY) + b.back * Wq + m : -1;
        // The border's first black values come from p itself: no CTA writes p
        // before every neighbour has sent its first sweep's.
        const long long e = 4 * m + (long long)Wh * j + (long long)pl * k;
        const int valid = m == Wq - 1 ? tail : 4;
        if (in) sm[pcol + quad(b.y, b.z, m)] = res_load<RAGGED>(p_b + e, valid);
        if (q < ring) {
            const int s = (j + k) & 1, n = 2 + count_y(j) + count_z(k);
            const int end = n - (s ? (m == Wq - 1 ? x_hi : 0) : (m == 0 ? x_lo : 0));
            t_cell[q] = in ? s | ((s ? m == Wq - 1 : m == 0) ? 2 : 0) | (m == Wq - 1 ? 4 : 0) : -1;
            if (in) {
                ring_rhs[q] = res_load<RAGGED>(rhs_r + e, valid);
                ring_den[q] = make_float4(inv_count((float)n), inv_count_lo((float)n), inv_count((float)end),
                                          inv_count_lo((float)end));
            }
        }
    }
    float4 p[2][2][RZ];                                  // [colour][row][plane]
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int w = 0; w < 2; ++w)
#pragma unroll
            for (int z = 0; z < RZ; ++z) {
                const int o = gA + w * Wh + z * pl;
                p[c][w][z] = zero4;
                if (live) rhs[c * rcol + z * rplane + w * Wq] = zero4;
                if ((w ? okB : okA) && k0 + z < g.D) {
                    p[c][w][z] = res_load<RAGGED>((c ? p_b : p_r) + o, lanes);
                    rhs[c * rcol + z * rplane + w * Wq] = res_load<RAGGED>((c ? rhs_b : rhs_r) + o, lanes);
                    if (c == 1) sm[pcol + own + w * prow + z * pplane] = p[c][w][z];
                }
            }
    // Neighbour counts: of each row without its z neighbours, of each plane's z
    // neighbours, and what a row's end cell has less; their reciprocals (hi, lo
    // of div_hl) come from a table, which takes fewer registers than every
    // quad's and serves the domain's sides alike.  Entry 0: cells outside the
    // grid (the last CTA's rows and planes past it), whose update is 0 * num,
    // so that the update has no branches and its quads overlap.
    int cy[2], cz[RZ];
#pragma unroll
    for (int w = 0; w < 2; ++w) cy[w] = (w ? okB : okA) ? 2 + count_y(jA + w) : -8;
#pragma unroll
    for (int z = 0; z < RZ; ++z) cz[z] = k0 + z < g.D ? count_z(k0 + z) : -8;
    const int c_lo = first ? x_lo : 0, c_hi = last ? x_hi : 0;
    __syncthreads();
    // Where the exchange's and the ring's work goes to threads without cells of
    // their own it overlaps the update.
    const int tile = Wq * NRP * (TZ / RZ), nsh = res_sharers(nthr, tile, border);
    const int share = nsh == nthr ? (int)threadIdx.x : (int)threadIdx.x - tile;        // < 0: none
    const unsigned e0 = rs.epoch[cta];
    bool dead = false;
    __syncthreads();

    auto update = [&](auto c_t) __attribute__((always_inline)) {
        constexpr int c = decltype(c_t)::value, o = 1 - c;
        const float4 *so = sm + o * pcol + own;
        float4 *sc = sm + c * pcol + own;
        float4 zm[2], zp[2];
#pragma unroll
        for (int w = 0; w < 2; ++w) {
            zm[w] = so[w * prow - pplane];
            zp[w] = so[w * prow + RZ * pplane];
        }
#pragma unroll
        for (int z = 0; z < RZ; ++z) {
            const float4 ym = so[z * pplane - prow], yp = so[z * pplane + 2 * prow];
#pragma unroll
            for (int w = 0; w < 2; ++w) {
                const int s = (c + z + w) & 1;           // row A at plane k0: parity c
                float xe;
                const float4 x = p[o][w][z];
                if (WARPROW) {
                    const float v = s == 0 ? __shfl_up_sync(0xffffffffu, x.w, 1) : __shfl_down_sync(0xffffffffu, x.x, 1);
                    xe = (s == 0 ? first : last) ? 0.0f : v;
                } else {
                    const float *q = reinterpret_cast<const float *>(so + w * prow + z * pplane);
                    xe = (s == 0 ? first : last) ? 0.0f : s == 0 ? q[-1] : q[4];
                }
                const int n = cy[w] + cz[z];
                const float2 in = inv[max(n, 0)], end = inv[max(n - (s == 0 ? c_lo : c_hi), 0)];
                const float4 b = rhs[c * rcol + z * rplane + w * Wq], y0 = w ? p[o][0][z] : ym, y1 = w ? yp : p[o][1][z];
                const float4 z0 = z ? p[o][w][z - 1] : zm[w], z1 = z < RZ - 1 ? p[o][w][z + 1] : zp[w];
                float4 v;
                if (RAGGED) {
                    v = res_quad_ragged(sp.scale, s, b, x, xe, y0, y1, z0, z1, in, end, first, last, lanes);
                } else {
                    const QuadDen d = s == 0 ? QuadDen{end.y, end.x, in.y, in.x, in.y, in.x}
                                             : QuadDen{in.y, in.x, in.y, in.x, end.y, end.x};
                    v = gs_quad_pk(sp.scale, s, b, x, xe, y0, y1, z0, z1, d);
                }
                p[c][w][z] = v;
                sc[w * prow + z * pplane] = v;
            }
        }
    };
    // The red ring: this thread's share of the neighbours' red cells next to
    // the tile.
    auto update_ring = [&]() __attribute__((always_inline)) {
#pragma unroll 1
        for (int q = share; q < ring; q += nsh) {
            const int cell = t_cell[q];
            if (cell < 0) continue;
            const int at = t_dst[q], s = cell & 1;
            const float4 *b = sm + pcol + at;
            const float4 n = ring_den[q];
            const float xe = cell & 2 ? 0.0f : reinterpret_cast<const float *>(b)[s ? 4 : -1];
            const float4 z0 = b[-pplane], z1 = b[pplane], y0 = b[-prow], y1 = b[prow];
            if (RAGGED) {
                const bool q_last = cell & 4;
                sm[at] = res_quad_ragged(sp.scale, s, ring_rhs[q], *b, xe, y0, y1, z0, z1, make_float2(n.x, n.y),
                                         make_float2(n.z, n.w), s == 0 && (cell & 2), s == 1 && q_last, q_last ? tail : 4);
            } else {
                const QuadDen d = s ? QuadDen{n.y, n.x, n.y, n.x, n.w, n.z} : QuadDen{n.w, n.z, n.y, n.x, n.y, n.x};
                sm[at] = gs_quad(sp.scale, s, ring_rhs[q], *b, xe, y0, y1, z0, z1, d);
            }
        }
    };
    // Exchanges: after every sweep but the last, whose black cells nobody reads
    // here; a single sweep has one all the same, so that no CTA writes p while
    // a neighbour still reads its first border from it.
    const int exchanges = sweeps > 1 ? sweeps - 1 : 1;
    for (int n = 0; n < sweeps; ++n) {
        if (live) update(std::integral_constant<int, 0>{});
        if (share >= 0) update_ring();
        __syncthreads();
        if (live) update(std::integral_constant<int, 1>{});
        if (n >= exchanges) break;
        __syncthreads();
        const unsigned e = e0 + (unsigned)n + 1u;
        uint4 *out = rs.halo + (e & 1u) * 2 * border;
        const uint4 *in = out + (size_t)cta * 4 * border;
        float4 *sb = sm + pcol;
#pragma unroll 1
        for (int q = share >= 0 ? share : border; q < border; q += nsh) {
            const int to = t_to[q];
            if (to < 0) continue;
            const float4 v = sb[t_src[q]];
            ll_store(out + to, v.x, v.y, e);
            ll_store(out + to + border, v.z, v.w, e);
        }
        unsigned long long t0 = 0;
        for (int q0 = share >= 0 ? share : border; q0 < border; q0 += NR * nsh) {
            int dst[NR];
            unsigned pend = 0;
#pragma unroll
            for (int i = 0; i < NR; ++i) {
                const int q = q0 + i * nsh;
                dst[i] = q < border ? t_dst[q] : -1;
                if (dst[i] >= 0) pend |= 1u << i;
            }
            for (int spin = 1; pend && !dead; ++spin) {
                uint4 lo[NR], hi[NR];
#pragma unroll
                for (int i = 0; i < NR; ++i)
                    if (pend >> i & 1u) {
                        lo[i] = ll_load(in + q0 + i * nsh);
                        hi[i] = ll_load(in + q0 + i * nsh + border);
                    }
#pragma unroll
                for (int i = 0; i < NR; ++i)
                    if ((pend >> i & 1u) && lo[i].y == e && lo[i].w == e && hi[i].y == e && hi[i].w == e) {
                        sb[dst[i]] = make_float4(__uint_as_float(lo[i].x), __uint_as_float(lo[i].z),
                                                 __uint_as_float(hi[i].x), __uint_as_float(hi[i].z));
                        pend &= ~(1u << i);
                    }
                if ((spin & 255) == 0) {
                    const unsigned long long t = res_now();
                    if (t0 == 0) t0 = t;
                    else if (t - t0 > kResWaitNs) { dead = true; *rs.err = 1; }
                }
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int c = 0; c < 2; ++c)
#pragma unroll
        for (int w = 0; w < 2; ++w)
#pragma unroll
            for (int z = 0; z < RZ; ++z)
                if ((w ? okB : okA) && k0 + z < g.D)
                    res_store<RAGGED>((c ? p_b : p_r) + gA + w * Wh + z * pl, p[c][w][z], lanes);
    if (threadIdx.x == 0) rs.epoch[cta] = e0 + (unsigned)exchanges;
}

template <int RZ, bool WARPROW, bool RAGGED>
__global__ void __launch_bounds__(res_threads<RZ>(), 1)
k_rbgs_resident(Geom g, SolveParams sp, const float *__restrict__ rhs_r, const float *__restrict__ rhs_b,
                float *p_r, float *p_b, int sweeps, ResParams rs) {
    res_sweeps<RZ, WARPROW, RAGGED>(g, sp, rhs_r, rhs_b, p_r, p_b, sweeps, rs, (int)blockIdx.x);
}

// The same for several grids side by side, each on CTAs of its own: one wave of
// a batch (plan below).  Grids that have stopped do nothing.  Sixteen grids of
// 48^3 to 96^3 cells, 8.7 million in all, take four waves and 20.5 us per sweep
// of all of them; temporal-blocking tiles take 23.4, the segment kernel 32.  A
// wave's SMs hold close to all the cells they can; its time is the exchange
// (about 2 us) and the update of the fullest SM.
template <int RZ>
__global__ void __launch_bounds__(res_threads<RZ>(), 1)
k_batch_resident(const __grid_constant__ ResidentWave w, const BatchCtl *__restrict__ ctl, int sweeps) {
    int i = 0;
    while (i + 1 < w.n && (int)blockIdx.x >= w.grid[i + 1].cta0) ++i;
    const ResidentGrid &q = w.grid[i];
    if (!ctl[q.sim].active) return;
    const ResParams rs{q.NY, q.NZ, q.TY, q.TZ, static_cast<uint4 *>(q.halo), q.epoch, w.err};
    const int cta = (int)blockIdx.x - q.cta0;
    if (q.warprow) res_sweeps<RZ, true, false>(q.g, q.sp, q.rhs_r, q.rhs_b, q.p_r, q.p_b, sweeps, rs, cta);
    else res_sweeps<RZ, false, false>(q.g, q.sp, q.rhs_r, q.rhs_b, q.p_r, q.p_b, sweeps, rs, cta);
}

namespace {

struct Shape { int RZ, NY, NZ, TY, TZ, threads; };

int quads_of(const Geom &g) { return ((g.W >> 1) + 3) >> 2; }      // quads per packed row

int sm_count() {
    static std::atomic<int> cache[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (cache[dev] == 0) {
        int n = 0, coop = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
        cache[dev] = coop && n > 0 ? n : -1;
    }
    return cache[dev];
}

// SMs that the current context holds: a context made for a part of the device's
// has fewer.
int context_sms() {
    static const auto current = driver_function<CUresult (*)(CUcontext *)>("cuCtxGetCurrent");
    static const auto resource =
        driver_function<CUresult (*)(CUcontext, CUdevResource *, CUdevResourceType)>("cuCtxGetDevResource");
    CUcontext ctx = nullptr;
    CUdevResource r = {};
    if (!current || !resource || current(&ctx) != CUDA_SUCCESS || !ctx ||
        resource(ctx, &r, CU_DEV_RESOURCE_TYPE_SM) != CUDA_SUCCESS)
        return sm_count();
    return std::min(sm_count(), (int)r.sm.smCount);
}

size_t smem_of(int Wq, int TY, int TZ) {
    const size_t ring = (size_t)2 * (TY + TZ) * Wq;
    return ((size_t)2 * (TY + 4) * (TZ + 4) * Wq + (size_t)2 * TY * TZ * Wq + 2 * ring) * sizeof(float4) +
           (3 * (size_t)res_border(TY, TZ, Wq) + ring) * sizeof(int);
}

// The split of a grid over at most `sms` SMs, one CTA each: the fewest cells
// per CTA with its ring, then the smallest boundary.  rz: 2 or 4 planes per
// thread, 0 for either.
bool shape_of(const Geom &g, int sms, int rz, Shape *out) {
    const int Wq = quads_of(g);
    if (sms <= 0 || Wq > 256) return false;
    long long best = -1;
    for (int RZ = 2; RZ <= 4; RZ += 2) {
        if (rz && rz != RZ) continue;
        const int cap = RZ == 2 ? res_threads<2>() : res_threads<4>();
        for (int TY = 2; TY <= g.H + 1; TY += 2) {
            const int NY = (g.H + TY - 1) / TY;
            if (NY > sms) continue;
            const int nzmax = sms / NY;
            int TZ = (g.D + nzmax - 1) / nzmax;
            TZ = (TZ + RZ - 1) / RZ * RZ;
            const int threads = Wq * (TY / 2) * (TZ / RZ);
            if (threads > cap || smem_of(Wq, TY, TZ) > (size_t)kResSmem) continue;
            const int border = res_border(TY, TZ, Wq);
            const int block = std::min(cap, (threads + border + 31) & ~31);
            if (block < threads) continue;
            const long long cost = ((long long)2 * TY * TZ + 2 * (TY + TZ)) * 1000 + (TY + TZ) * 4 + RZ;
            if (best >= 0 && cost >= best) continue;
            best = cost;
            *out = {RZ, NY, (g.D + TZ - 1) / TZ, TY, TZ, block};
        }
    }
    return best >= 0;
}

template <class... P, class... A>
cudaError_t launch_coop(void (*k)(P...), int ctas, int threads, size_t smem, cudaStream_t st, const A &...args) {
    cudaError_t e = allow_smem((const void *)k, kResSmem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(ctas, 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeCooperative;
    at[0].val.cooperative = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k, P(args)...);
    if (e != cudaSuccess) cudaGetLastError();            // the caller has it; the next check of a launch must not
    return e;
}

bool warp_rows(int Wq, const Shape &s) {
    return Wq <= 32 && 32 % Wq == 0 && (Wq * (s.TY / 2) * (s.TZ / s.RZ)) % 32 == 0;
}

} // namespace

bool resident_supported(const Geom &g) {
    Shape s;
    return shape_of(g, sm_count(), 0, &s) && s.NY * s.NZ <= context_sms();
}

static size_t halo_quads(const Geom &g, const Shape &s) {
    return (size_t)s.NY * s.NZ * 4 * res_border(s.TY, s.TZ, quads_of(g));
}

size_t resident_bytes(const Geom &g) {
    Shape s;
    if (!shape_of(g, sm_count(), 0, &s)) return 0;
    return halo_quads(g, s) * sizeof(uint4) + (size_t)s.NY * s.NZ * sizeof(unsigned);
}

typedef void (*ResidentKernel)(Geom, SolveParams, const float *, const float *, float *, float *, int, ResParams);
static ResidentKernel resident_kernel(const Geom &g, const Shape &s) {
    const bool ragged = (g.W & 7) != 0, warprow = warp_rows(quads_of(g), s);
    if (s.RZ == 2)
        return ragged ? k_rbgs_resident<2, false, true> : warprow ? k_rbgs_resident<2, true, false> : k_rbgs_resident<2, false, false>;
    return ragged ? k_rbgs_resident<4, false, true> : warprow ? k_rbgs_resident<4, true, false> : k_rbgs_resident<4, false, false>;
}

cudaError_t resident_prepare(const Geom &g, int *sms) {
    Shape s;
    if (!shape_of(g, sm_count(), 0, &s)) return cudaErrorInvalidValue;
    const ResidentKernel k = resident_kernel(g, s);
    cudaError_t e = allow_smem((const void *)k, kResSmem);
    int per_sm = 0;
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, s.threads, smem_of(quads_of(g), s.TY, s.TZ));
    *sms = per_sm > 0 ? (s.NY * s.NZ + per_sm - 1) / per_sm : 0;
    return e == cudaSuccess && per_sm == 0 ? cudaErrorInvalidValue : e;
}

cudaError_t launch_resident(const Geom &g, const SolveParams &sp, const float *rhs_r, const float *rhs_b, float *p_r,
                            float *p_b, int sweeps, const ResidentWork &res, cudaStream_t st) {
    Shape s;
    if (!res.work || !res.err || sweeps < 1 || !shape_of(g, sm_count(), 0, &s)) return cudaErrorInvalidValue;
    const int ctas = s.NY * s.NZ, Wq = quads_of(g);
    ResParams rs{s.NY, s.NZ, s.TY, s.TZ, static_cast<uint4 *>(res.work), nullptr, res.err};
    rs.epoch = reinterpret_cast<unsigned *>(rs.halo + halo_quads(g, s));
    const size_t smem = smem_of(Wq, s.TY, s.TZ);
    return launch_coop(resident_kernel(g, s), ctas, s.threads, smem, st, g, sp, rhs_r, rhs_b, p_r, p_b, sweeps, rs);
}

// A batch's grids in waves of one launch each.  Every grid first gets the fewest
// CTAs it fits on, largest grids first into the first wave with room; a wave's
// time is its slowest grid's, so the SMs that are left go to the grids with the
// most cells per CTA.  Two planes per thread where that takes no more waves than
// four.  False where a grid does not fit.
bool batch_resident_plan(const BatchSim *sims, int n, std::vector<ResidentWave> *waves, size_t *bytes) {
    const int sms = context_sms();
    struct Item { int sim, ctas; Shape s; };
    auto work_of = [&](const Item &x) { return (long long)quads_of(sims[x.sim].g) * (x.s.TY * x.s.TZ + x.s.TY + x.s.TZ); };
    std::vector<std::vector<Item>> best;
    for (int rz = 4; rz >= 2; rz -= 2) {
        std::vector<Item> items;
        for (int i = 0; i < n; ++i) {
            Item x{i, 0, {}};
            if ((sims[i].g.W & 7) != 0 || !shape_of(sims[i].g, sms, rz, &x.s)) break;
            for (int c = 1; !shape_of(sims[i].g, c, rz, &x.s);) ++c;
            x.ctas = x.s.NY * x.s.NZ;
            items.push_back(x);
        }
        if ((int)items.size() < n) continue;
        std::stable_sort(items.begin(), items.end(), [](const Item &a, const Item &b) { return a.ctas > b.ctas; });
        std::vector<std::vector<Item>> plan;
        std::vector<int> used;
        for (const Item &x : items) {
            size_t w = 0;
            while (w < plan.size() && (used[w] + x.ctas > sms || (int)plan[w].size() == kWaveGrids)) ++w;
            if (w == plan.size()) { plan.emplace_back(); used.push_back(0); }
            plan[w].push_back(x);
            used[w] += x.ctas;
        }
        if (best.empty() || plan.size() <= best.size()) best = plan;
    }
    if (best.empty()) return false;
    waves->clear();
    *bytes = 0;
    for (auto &wave : best) {
        int used = 0;
        for (const Item &x : wave) used += x.ctas;
        for (bool grown = true; grown;) {
            grown = false;
            Item &x = *std::max_element(wave.begin(), wave.end(),
                                        [&](const Item &a, const Item &b) { return work_of(a) < work_of(b); });
            for (int c = x.ctas + 1; c <= x.ctas + sms - used && !grown; ++c) {
                Item y = x;
                if (!shape_of(sims[x.sim].g, c, x.s.RZ, &y.s)) continue;
                y.ctas = y.s.NY * y.s.NZ;
                if (work_of(y) >= work_of(x)) continue;
                used += y.ctas - x.ctas;
                x = y;
                grown = true;
            }
        }
        ResidentWave w{};
        for (const Item &x : wave) {
            const BatchSim &b = sims[x.sim];
            const Shape &s = x.s;
            ResidentGrid &q = w.grid[w.n++];
            q = {b.g, b.sp, b.rhs_r, b.rhs_b, b.p_r, b.p_b, reinterpret_cast<void *>(*bytes), nullptr, s.NY, s.NZ, s.TY, s.TZ,
                 x.sim, w.ctas, warp_rows(quads_of(b.g), s) ? 1 : 0};
            *bytes += halo_quads(b.g, s) * sizeof(uint4);
            q.epoch = reinterpret_cast<unsigned *>(*bytes);
            *bytes += ((size_t)x.ctas * sizeof(unsigned) + 15) & ~(size_t)15;
            w.ctas += x.ctas;
            w.RZ = s.RZ;
            w.smem = std::max(w.smem, smem_of(quads_of(b.g), s.TY, s.TZ));
        }
        waves->push_back(w);
    }
    return true;
}

cudaError_t batch_resident_bind(std::vector<ResidentWave> *waves, void *work, int *err) {
    for (ResidentWave &w : *waves) {
        w.err = err;
        for (int i = 0; i < w.n; ++i) {
            w.grid[i].halo = static_cast<char *>(work) + reinterpret_cast<size_t>(w.grid[i].halo);
            w.grid[i].epoch = reinterpret_cast<unsigned *>(static_cast<char *>(work) + reinterpret_cast<size_t>(w.grid[i].epoch));
        }
    }
    const cudaError_t e = allow_smem((const void *)k_batch_resident<2>, kResSmem);
    return e != cudaSuccess ? e : allow_smem((const void *)k_batch_resident<4>, kResSmem);
}

cudaError_t launch_batch_resident(const std::vector<ResidentWave> &waves, const BatchCtl *ctl, int sweeps, cudaStream_t st) {
    for (const ResidentWave &w : waves) {
        const cudaError_t e = w.RZ == 2 ? launch_coop(k_batch_resident<2>, w.ctas, res_threads<2>(), w.smem, st, w, ctl, sweeps)
                                        : launch_coop(k_batch_resident<4>, w.ctas, res_threads<4>(), w.smem, st, w, ctl, sweeps);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

} // namespace blz
