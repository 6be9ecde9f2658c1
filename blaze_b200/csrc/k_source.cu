// k_source.cu — particle sourcing (reference src/FluidSolver.cu:57-116 and
// Grid::sphereToGrid / cubicPulse, src/Grid.h:309-335), as a gather.
//
// The reference clears four back buffers over the whole grid, splats every
// particle with float atomics and copies |back| > 1e-5 into the front
// buffers (three full-grid passes, order-dependent sums).  Here the host bins
// the particles by 8^3 blocks of cells (the records come from host memory
// anyway) and each bin is one CTA: every cell sums the cubic pulses of the
// particles overlapping its bin in particle order and writes the front buffer
// once where |sum| > 1e-5.  No atomics, no accumulator buffers, no clear
// pass, and the sums are bitwise reproducible.
#include "kernels.cuh"

namespace blz {

__device__ __forceinline__ float cubic_pulse(float x, float w) {   // Grid.h:309-313
    if (x > w) return 0.0f;
    x /= w;
    return 1.0f - x * x * (3.0f - 2.0f * x);
}

// One CTA per (active bin, field), one thread per cell; a warp owns 8 x 4 cells
// of one plane of the bin.  What bounds the pass is the chain of particles a
// cell has to sum in order, so the chain is cut down to the particles that
// reach the warp's own cells: the particle's box in the bin is staged as three
// 8-bit axis masks, each lane tests one particle of a group of 32 against the
// warp's rows and plane, and only the balloted ones (about a sixth of the bin's)
// are evaluated.  A field per CTA instead of per loop iteration makes four or
// five times as many independent chains.  The order of a cell's sum is the
// bin list's.  Measured: 20,000 particles in 100 bins of a 128^3 grid 64 us,
// 2,000 particles with density in 79 bins 14 us (every particle evaluated for
// every field by one CTA per bin: 552 and 113 us).
constexpr int kSplatChunk = 256;

__global__ void __launch_bounds__(512)
k_splat_gather(Geom g, const float *__restrict__ rec8, const int *__restrict__ boxes,
               const int *__restrict__ bin_start, const int *__restrict__ bin_list,
               const int *__restrict__ active, int nbx, int nby, float *__restrict__ T,
               float *__restrict__ U, float *__restrict__ V, float *__restrict__ W,
               const float *__restrict__ dens, float *__restrict__ Dn) {
    __shared__ float4 s_pos[kSplatChunk];         // object-space position, radius
    __shared__ float s_val[kSplatChunk];
    __shared__ unsigned s_mask[kSplatChunk];      // x, y, z bits of the bin's cells in the box
    const int f = blockIdx.y;                     // T, U, V, W, density
    const int b = active[blockIdx.x];
    const int bx = b % nbx, by = (b / nbx) % nby, bz = b / (nbx * nby);
    const int i = bx * kSplatBin + threadIdx.x, j = by * kSplatBin + threadIdx.y, k = bz * kSplatBin + threadIdx.z;
    const int tid = threadIdx.x + kSplatBin * (threadIdx.y + kSplatBin * threadIdx.z);
    const float ox = f == 1 ? 0.0f : 0.5f, oy = f == 2 ? 0.0f : 0.5f, oz = f == 3 ? 0.0f : 0.5f;
    const float cx = ((float)i + ox) * g.dx, cy = ((float)j + oy) * g.dx, cz = ((float)k + oz) * g.dx;
    const unsigned cell = (1u << threadIdx.x) | (256u << threadIdx.y) | (65536u << threadIdx.z);
    const unsigned rows = 0xfu << (8 + 4 * (threadIdx.y >> 2)), plane = 65536u << threadIdx.z;
    const int lane = tid & 31;
    float acc = 0.0f;
    const int p0 = bin_start[b], p1 = bin_start[b + 1];
    // bits [lo - o, hi - o) of the bin's eight cells along one axis
    auto axis_bits = [](int lo, int hi, int o) -> unsigned {
        const int l = min(max(lo - o, 0), kSplatBin), h = min(max(hi - o, 0), kSplatBin);
        return h > l ? ((1u << h) - 1u) & ~((1u << l) - 1u) : 0u;
    };
    for (int base = p0; base < p1; base += kSplatChunk) {
        const int n = min(kSplatChunk, p1 - base);
        if (tid < kSplatChunk) {
            unsigned m = 0u;
            if (tid < n) {
                const int p = bin_list[base + tid];
                const float4 r0 = *reinterpret_cast<const float4 *>(rec8 + 8 * (size_t)p);
                const float4 r1 = *reinterpret_cast<const float4 *>(rec8 + 8 * (size_t)p + 4);
                const int2 *bb = reinterpret_cast<const int2 *>(boxes + (size_t)p * kSplatBoxInts + 6 * f);
                const int2 xb = bb[0], yb = bb[1], zb = bb[2];
                const unsigned mx = axis_bits(xb.x, xb.y, bx * kSplatBin), my = axis_bits(yb.x, yb.y, by * kSplatBin),
                               mz = axis_bits(zb.x, zb.y, bz * kSplatBin);
                if (mx && my && mz) m = mx | my << 8 | mz << 16;
                s_pos[tid] = make_float4(r0.x - g.dmin[0], g.dsize[1] - (r0.y - g.dmin[1]), r0.z - g.dmin[2],
                                         r1.z / 2.0f);
                s_val[tid] = f == 0 ? r1.w : f == 1 ? r0.w : f == 2 ? -r1.x : f == 3 ? r1.y : dens[p];   // V flips (Grid.h:331)
            }
            s_mask[tid] = m;
        }
        __syncthreads();
        for (int q0 = 0; q0 < n; q0 += 32) {
            const unsigned mine = s_mask[q0 + lane];
            unsigned hits = __ballot_sync(0xffffffffu, (mine & rows) && (mine & plane));
            while (hits) {
                const int q = q0 + __ffs(hits) - 1;
                hits &= hits - 1;
                if ((s_mask[q] & cell) != cell) continue;
                const float4 r = s_pos[q];
                const float mask = cubic_pulse(len3(r.x - cx, r.y - cy, r.z - cz), r.w);
                if (mask > 0.0f) acc += s_val[q] * mask;
            }
        }
        __syncthreads();
    }
    // set_source_from_back_to_front_kernel (FluidSolver.cu:99-116)
    float *const out = f == 0 ? T : f == 1 ? U : f == 2 ? V : f == 3 ? W : Dn;
    const int w = g.W + (f == 1), h = g.H + (f == 2), d = g.D + (f == 3);
    if (i < w && j < h && k < d && fabsf(acc) > 1e-5f) out[lin(i, j, k, w, h)] = acc;
}

// One CTA per bin for all fields: for scattered particles, a few in each bin.  What
// counts then is the number of CTAs and the one chain of loads that each begins
// with, not the sum: 2,000 particles all over a 256^3 grid (4,900 bins) take 36 us
// and 20,000 take 214 us here, 101 and 539 us with a CTA per bin and field.
constexpr int kScatteredChunk = 64;

__global__ void __launch_bounds__(512)
k_splat_scattered(Geom g, const float *__restrict__ rec8, const int *__restrict__ boxes,
               const int *__restrict__ bin_start, const int *__restrict__ bin_list,
               const int *__restrict__ active, int nbx, int nby, float *__restrict__ T,
               float *__restrict__ U, float *__restrict__ V, float *__restrict__ W,
               const float *__restrict__ dens, float *__restrict__ Dn) {
    __shared__ float s_rec[kScatteredChunk * 9];
    __shared__ int s_box[kScatteredChunk * kSplatBoxInts];
    const int b = active[blockIdx.x];
    const int bx = b % nbx, by = (b / nbx) % nby, bz = b / (nbx * nby);
    const int i = bx * kSplatBin + threadIdx.x, j = by * kSplatBin + threadIdx.y, k = bz * kSplatBin + threadIdx.z;
    const int tid = threadIdx.x + kSplatBin * (threadIdx.y + kSplatBin * threadIdx.z);
    const float ox[4] = {0.5f, 0.0f, 0.5f, 0.5f}, oy[4] = {0.5f, 0.5f, 0.0f, 0.5f}, oz[4] = {0.5f, 0.5f, 0.5f, 0.0f};
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f}, acc_d = 0.0f;
    const int p0 = bin_start[b], p1 = bin_start[b + 1];
    const int nthr = blockDim.x * blockDim.y * blockDim.z;
    for (int base = p0; base < p1; base += kScatteredChunk) {
        const int n = min(kScatteredChunk, p1 - base);
        for (int t = tid; t < n * 8; t += nthr)
            s_rec[9 * (t / 8) + t % 8] = rec8[(size_t)bin_list[base + t / 8] * 8 + t % 8];
        if (Dn)
            for (int t = tid; t < n; t += nthr) s_rec[9 * t + 8] = dens[bin_list[base + t]];
        for (int t = tid; t < n * kSplatBoxInts; t += nthr)
            s_box[t] = boxes[(size_t)bin_list[base + t / kSplatBoxInts] * kSplatBoxInts + t % kSplatBoxInts];
        __syncthreads();
        for (int q = 0; q < n; ++q) {
            const float *r = s_rec + 9 * q;
            const float radius = r[6] / 2.0f;
            const float px = r[0] - g.dmin[0], py = g.dsize[1] - (r[1] - g.dmin[1]), pz = r[2] - g.dmin[2];
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                const int *bb = s_box + kSplatBoxInts * q + 6 * f;   // imin, imax, jmin, jmax, kmin, kmax (empty if skipped)
                if (i < bb[0] || i >= bb[1] || j < bb[2] || j >= bb[3] || k < bb[4] || k >= bb[5]) continue;
                const float value = f == 0 ? r[7] : r[2 + f];
                const float ddx = px - ((float)i + ox[f]) * g.dx;
                const float ddy = py - ((float)j + oy[f]) * g.dx;
                const float ddz = pz - ((float)k + oz[f]) * g.dx;
                const float mask = cubic_pulse(len3(ddx, ddy, ddz), radius);
                if (mask > 0.0f) acc[f] += f == 2 ? -value * mask : value * mask;   // V flips (Grid.h:331)
            }
            if (Dn) {                                     // density: T's geometry, its own box and value
                const int *bb = s_box + kSplatBoxInts * q + 24;
                if (i >= bb[0] && i < bb[1] && j >= bb[2] && j < bb[3] && k >= bb[4] && k < bb[5]) {
                    const float ddx = px - ((float)i + 0.5f) * g.dx;
                    const float ddy = py - ((float)j + 0.5f) * g.dx;
                    const float ddz = pz - ((float)k + 0.5f) * g.dx;
                    const float mask = cubic_pulse(len3(ddx, ddy, ddz), radius);
                    if (mask > 0.0f) acc_d += r[8] * mask;
                }
            }
        }
        __syncthreads();
    }
    // set_source_from_back_to_front_kernel (FluidSolver.cu:99-116)
    if (i < g.W && j < g.H && k < g.D && fabsf(acc[0]) > 1e-5f) T[lin(i, j, k, g.W, g.H)] = acc[0];
    if (i <= g.W && j < g.H && k < g.D && fabsf(acc[1]) > 1e-5f) U[lin(i, j, k, g.W + 1, g.H)] = acc[1];
    if (i < g.W && j <= g.H && k < g.D && fabsf(acc[2]) > 1e-5f) V[lin(i, j, k, g.W, g.H + 1)] = acc[2];
    if (i < g.W && j < g.H && k <= g.D && fabsf(acc[3]) > 1e-5f) W[lin(i, j, k, g.W, g.H)] = acc[3];
    if (Dn && i < g.W && j < g.H && k < g.D && fabsf(acc_d) > 1e-5f) Dn[lin(i, j, k, g.W, g.H)] = acc_d;
}

// Which of the two: waves of CTAs times a wave's time in us, four CTAs per SM that
// sum every particle for every field here, three per SM and a thirtieth of the sum
// there (measured: 1 to 13 particles in 130 to 4,900 bins).
bool splat_scattered(int bins, long long entries, int fields) {
    const double a = bins > 0 ? (double)entries / bins : 0.0;
    return ((bins + 591) / 592) * (3.3 + 0.95 * a) < ((bins * (long long)fields + 443) / 444) * (2.3 + 0.07 * a);
}

void launch_splat_gather(const Geom &g, const float *rec8, const int *boxes, const int *bin_start,
                         const int *bin_list, const int *active, int n_active, bool scattered, int nbx, int nby,
                         float *T, float *U, float *V, float *W, cudaStream_t st, const float *dens, float *Dn) {
    if (n_active <= 0) return;
    const dim3 b(kSplatBin, kSplatBin, kSplatBin);
    if (scattered)
        k_splat_scattered<<<n_active, b, 0, st>>>(g, rec8, boxes, bin_start, bin_list, active, nbx, nby, T, U, V, W, dens, Dn);
    else
        k_splat_gather<<<dim3(n_active, Dn ? 5 : 4), b, 0, st>>>(g, rec8, boxes, bin_start, bin_list, active, nbx, nby, T, U,
                                                                 V, W, dens, Dn);
}

} // namespace blz
