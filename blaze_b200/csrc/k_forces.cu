// k_forces.cu — cooldown, drag, vorticity confinement, buoyancy, wind and
// turbulence (reference src/FluidSolver.cu:118-390), in gather form.
//
// The reference scatters confinement and pseudo-curl forces with float
// atomics (FluidSolver.cu:242-247, 287-292).  Here every face gathers the
// contributions of its two adjacent cells, which makes the pass deterministic
// and free of atomics.  Drag, vorticity, buoyancy and wind only touch a face's
// own value, so they are fused into one in-place face pass.
#include <algorithm>

#include "kernels.cuh"

namespace blz {

dim3 face_block() { return dim3(32, 4, 2); }
dim3 face_grid(const Geom &g) {
    const dim3 b = face_block();
    return dim3((g.W + 1 + b.x - 1) / b.x, (g.H + 1 + b.y - 1) / b.y, (g.D + 1 + b.z - 1) / b.z);
}

static dim3 cell_grid(const Geom &g) {
    const dim3 b = face_block();
    return dim3((g.W + b.x - 1) / b.x, (g.H + b.y - 1) / b.y, (g.D + b.z - 1) / b.z);
}

// temperature_cooldown_kernel / apply_drag_kernel (FluidSolver.cu:118-140).
__global__ void k_scale(float *__restrict__ a, size_t n, float s) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        a[i] *= s;
}

void launch_scale(float *a, size_t n, float s, cudaStream_t st) {
    const int threads = 256;
    const int blocks = (int)std::min<size_t>((n + threads - 1) / threads, 148 * 16);
    k_scale<<<blocks, threads, 0, st>>>(a, n, s);
}

__device__ __forceinline__ bool vort_active(const Geom &g, int i, int j, int k) {
    return i >= 2 && j >= 2 && k >= 2 && i <= g.W - 3 && j <= g.H - 3 && k <= g.D - 3;
}

// Sample weight of the last node where a coordinate n - 1 is clamped to
// n - 1.001 (clamp_coord): the sample there is a mix of the last two nodes.
__device__ __forceinline__ float end_weight(int n) { return clamp_coord((float)(n - 1), n) - (float)(n - 2); }
__device__ __forceinline__ float end_mix(float inner, float last, float w) { return inner * (1.0f - w) + last * w; }

// computeVorticity (FluidSolver.cu:174-201) for cells 1..n-2 in each axis
// (centred differences of trilinear samples at the neighbouring cell
// centres), |omega|, and for cells 2..n-3 omega clamped to the local speed
// (FluidSolver.cu:203-228): what the confinement force reads.  The samples lie
// at cell centres, where the trilinear weights are 0 and 1/2, so a sample is
// the mean of the cell's two faces; only where a neighbour is the last cell of
// an axis does the coordinate clamp mix in 0.001 of the cell before it (the
// cell itself, end_mix).  The velocities are read through the drag factor
// (applied in memory by k_face_forces) and T is cooled in place on the way.
// One cell per thread, every load independent: marching planes with the
// column in registers issues a third fewer loads but waits for memory once per
// plane (328 us at 256^3).  Measured at 256^3: 188 us, 670 MB in all; one pass of
// general trilinear samples for omega, a second for the force and four scaling
// passes took 472 + 320 + 128 us.
__global__ void __launch_bounds__(256)
k_vorticity(Geom g, float *__restrict__ T, const float *__restrict__ U, const float *__restrict__ V,
            const float *__restrict__ W, float cool, float drag, float tiny, float *__restrict__ mag,
            float *__restrict__ wx, float *__restrict__ wy, float *__restrict__ wz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i >= g.W || j >= g.H || k >= g.D) return;
    const int rT = g.W, pT = rT * g.H, rU = rT + 1, pU = rU * g.H, pV = rT * (g.H + 1);
    const int q = i + rT * j + pT * k, qu = i + rU * j + pU * k, qv = i + rT * j + pV * k;
    if (cool != 1.0f) T[q] *= cool;
    if (i < 1 || j < 1 || k < 1 || i > g.W - 2 || j > g.H - 2 || k > g.D - 2) return;
    // cell-centre velocity of the cell whose lower face is element e
    auto mean = [&](const float *p, int e, int step) {
        return 0.5f * (__fmul_rn(__ldg(p + e), drag) + __fmul_rn(__ldg(p + (e + step)), drag));
    };
    const float uc = mean(U, qu, 1), vc = mean(V, qv, rT), wc = mean(W, q, pT);
    float u_y = mean(U, qu + rU, 1), u_z = mean(U, qu + pU, 1), v_x = mean(V, qv + 1, rT), v_z = mean(V, qv + pV, rT);
    float w_x = mean(W, q + 1, pT), w_y = mean(W, q + rT, pT);
    const float u_y0 = mean(U, qu - rU, 1), u_z0 = mean(U, qu - pU, 1);
    const float v_x0 = mean(V, qv - 1, rT), v_z0 = mean(V, qv - pV, rT);
    const float w_x0 = mean(W, q - 1, pT), w_y0 = mean(W, q - rT, pT);
    if (i == g.W - 2) { const float e = end_weight(g.W); v_x = end_mix(vc, v_x, e); w_x = end_mix(wc, w_x, e); }
    if (j == g.H - 2) { const float e = end_weight(g.H); u_y = end_mix(uc, u_y, e); w_y = end_mix(wc, w_y, e); }
    if (k == g.D - 2) { const float e = end_weight(g.D); u_z = end_mix(uc, u_z, e); v_z = end_mix(vc, v_z, e); }
    const float h = 0.5f * g.inv_dx;
    const float ox = (w_y - w_y0 - (v_z - v_z0)) * h;
    const float oy = (u_z - u_z0 - (w_x - w_x0)) * h;
    const float oz = (v_x - v_x0 - (u_y - u_y0)) * h;
    const float m = len3(ox, oy, oz);
    mag[q] = m;
    if (!vort_active(g, i, j, k)) return;
    const float speed = len3(uc, vc, wc), onorm = m + tiny;
    const float c = onorm > speed ? speed / onorm : 1.0f;
    wx[q] = ox * c; wy[q] = oy * c; wz[q] = oz * c;
}

void launch_vorticity(const Geom &g, float *T, const float *U, const float *V, const float *W, float cool, float drag,
                      const ForceParams &fp, float *mag, float *wx, float *wy, float *wz, cudaStream_t st) {
    k_vorticity<<<cell_grid(g), face_block(), 0, st>>>(g, T, U, V, W, cool, drag, fp.tiny, mag, wx, wy, wz);
}

// One in-place pass over every face: drag, confinement gather (FluidSolver.cu:
// 203-248: the half increment 0.5 dt eps dx (grad|omega| x omega) of both
// cells, for 2 <= i <= W-3, same for j, k), then buoyancy (add_buoyancy_kernel,
// FluidSolver.cu:142-156), then the wind relaxation in the two-voxel slabs at
// both ends of the wind axis (add_wind_kernel, FluidSolver.cu:337-390) — the
// reference's order.  A face needs one component of each of its two cells'
// forces, six loads a component, most of them in L1; a tile that forms every
// force once and passes it on through shuffles and shared memory, marching
// planes, took 440 us at 256^3 for waiting on memory at every plane's barrier.
// Measured at 256^3: 286 us (394 us with the force read from memory and T
// sampled by the general trilinear).
template <bool VORT>
__global__ void __launch_bounds__(256)
k_face_forces(Geom g, float *__restrict__ U, float *__restrict__ V, float *__restrict__ W,
              const float *__restrict__ T, const float *__restrict__ mag, const float *__restrict__ wx,
              const float *__restrict__ wy, const float *__restrict__ wz, ForceParams fp, float drag,
              const float *__restrict__ Dn) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i > g.W || j > g.H || k > g.D) return;
    const bool fu = j < g.H && k < g.D, fv = i < g.W && k < g.D, fw = i < g.W && j < g.H;
    const int rT = g.W, pT = rT * g.H, rU = rT + 1;
    const int q = i + rT * j + pT * k, qu = i + rU * j + rU * g.H * k, qv = i + rT * j + rT * (g.H + 1) * k;
    float u = fu ? U[qu] : 0.0f, v = fv ? V[qv] : 0.0f, w = fw ? W[q] : 0.0f, lift = 0.0f;
    if (fv && fp.buoy_on) {
        // The face lies midway between two cell centres; at the domain's
        // sides the sample is clamped (trilinear).
        auto at_face = [&](const float *a) -> float {
            if (i < g.W - 1 && j >= 1 && j < g.H && k < g.D - 1) return 0.5f * (__ldg(a + (q - rT)) + __ldg(a + q));
            return trilinear(fT(a, g), g.inv_dx, ((float)i + 0.5f) * g.dx, (float)j * g.dx, ((float)k + 0.5f) * g.dx);
        };
        lift = fp.beta * at_face(T);
        if (fp.dens_on) lift -= fp.alpha * at_face(Dn);   // target mode: the density's weight pulls down
    }
    u = __fmul_rn(u, drag);
    v = __fmul_rn(v, drag);
    w = __fmul_rn(w, drag);
    if (VORT) {
        const float s = 0.5f * g.inv_dx, sc = fp.conf * g.dx, h = 0.5f * g.dt;
        // gradient of |omega| along one axis, and a force component
        // h eps dx (ga ob - gb oa), at cell c
        auto grad = [&](int c, int step) { return (__ldg(mag + (c + step)) - __ldg(mag + (c - step))) * s; };
        auto force = [&](float ga, float ob, float gb, float oa) { return h * (sc * (ga * ob - gb * oa)); };
        auto fx = [&](int c) { return force(grad(c, rT), __ldg(wz + c), grad(c, pT), __ldg(wy + c)); };
        auto fy = [&](int c) { return force(grad(c, pT), __ldg(wx + c), grad(c, 1), __ldg(wz + c)); };
        auto fz = [&](int c) { return force(grad(c, 1), __ldg(wy + c), grad(c, rT), __ldg(wx + c)); };
        const bool self = vort_active(g, i, j, k);
        if (vort_active(g, i - 1, j, k)) u += fx(q - 1);
        if (vort_active(g, i, j - 1, k)) v += fy(q - rT);
        if (vort_active(g, i, j, k - 1)) w += fz(q - pT);
        if (self) { u += fx(q); v += fy(q); w += fz(q); }
    }
    if (fp.buoy_on) v += g.dt * (lift * fp.grav);
    if (fp.wind_on && (fp.wind_along_x ? (i < 2 || i >= g.W - 1) : (k < 2 || k >= g.D - 1))) {
        const float one_m = 1.0f - g.dt;
        float nU = 0.0f, nV = 0.0f, nW = 0.0f;
        if (fp.wind_turb_amp != 0.0f) {
            const float x = (float)i * g.dx, y = (float)j * g.dx, z = (float)k * g.dx + fp.wind_offset;
            nU = fp.wind_turb_amp * perlin(x, y, z, fp.wind_freq, 123);
            nV = fp.wind_turb_amp * perlin(x, y, z, fp.wind_freq, 456);
            nW = fp.wind_turb_amp * perlin(x, y, z, fp.wind_freq, 789);
        }
        u = u * one_m + (fp.wind_amp * ((fp.wind_along_x ? fp.wind_dir_sign : 0.0f) + nU)) * g.dt;
        v = v * one_m + (fp.wind_amp * nV) * g.dt;
        w = w * one_m + (fp.wind_amp * ((fp.wind_along_x ? 0.0f : fp.wind_dir_sign) + nW)) * g.dt;
    }
    if (fu) U[qu] = u;
    if (fv) V[qv] = v;
    if (fw) W[q] = w;
}

void launch_face_forces(const Geom &g, float *U, float *V, float *W, const float *T, const float *mag,
                        const float *wx, const float *wy, const float *wz, const ForceParams &fp, float drag,
                        cudaStream_t st, const float *Dn) {
    if (fp.vort_on)
        k_face_forces<true><<<face_grid(g), face_block(), 0, st>>>(g, U, V, W, T, mag, wx, wy, wz, fp, drag, Dn);
    else
        k_face_forces<false><<<face_grid(g), face_block(), 0, st>>>(g, U, V, W, T, mag, wx, wy, wz, fp, drag, Dn);
}

__device__ __forceinline__ float fit01(float v, float a, float b, float lo, float hi) {
    return fmaxf(fminf((v - a) / (b - a), 1.0f), 0.0f) * (hi - lo) + lo;   // FluidSolver.cu:250-252
}

// compute_turbulence_kernel (FluidSolver.cu:295-335): masked Perlin noise per
// face; the noise lattice position is the face index plus a time offset.  The
// masks sample T and the speed at the face: away from the domain's sides every
// sample is a mean of two or four values, at the sides the clamped trilinear
// sample.  Measured at 128^3: 132 us (203 us with trilinear samples throughout
// and a branch per lattice gradient).
__global__ void __launch_bounds__(256)
k_turb_noise(Geom g, const float *__restrict__ T, const float *__restrict__ U, const float *__restrict__ V,
             const float *__restrict__ W, float *__restrict__ nU, float *__restrict__ nV, float *__restrict__ nW,
             ForceParams fp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i > g.W || j > g.H || k > g.D) return;
    const float r = g.inv_dx, fi = (float)i, fj = (float)j, fk = (float)k, dx = g.dx;
    const bool xi = i >= 1 && i < g.W, yi = j >= 1 && j < g.H, zi = k >= 1 && k < g.D;   // between two cells
    const bool xc = i < g.W - 1, yc = j < g.H - 1, zc = k < g.D - 1;                     // centre sample unclamped
    const int rT = g.W, pT = rT * g.H, rU = rT + 1, pU = rU * g.H, pV = rT * (g.H + 1);
    const int q = i + rT * j + pT * k, qu = i + rU * j + pU * k, qv = i + rT * j + pV * k;
    auto mean2 = [](const float *p, int e, int s) { return 0.5f * (__ldg(p + (e - s)) + __ldg(p + e)); };
    auto mean4 = [](const float *p, int e, int lo, int up) {          // over (-lo, 0) x (0, up)
        return 0.25f * (__ldg(p + (e - lo)) + __ldg(p + e) + __ldg(p + (e - lo + up)) + __ldg(p + (e + up)));
    };
    auto temp_mask = [&](float x) { return fit01(x, fp.tr0, fp.tr1, 1.0f, 0.0f); };
    auto speed_mask = [&](float x, float y, float z) { return fit01(len3(x, y, z), fp.vr0, fp.vr1, 0.0f, 1.0f); };
    auto side_mask = [&](float px, float py, float pz) {
        return temp_mask(trilinear(fT(T, g), r, px, py, pz)) *
               speed_mask(trilinear(fU(U, g), r, px, py, pz), trilinear(fV(V, g), r, px, py, pz),
                          trilinear(fW(W, g), r, px, py, pz));
    };
    if (j < g.H && k < g.D) {
        const float m = xi && yc && zc ? temp_mask(mean2(T, q, 1)) * speed_mask(__ldg(U + qu), mean4(V, qv, 1, rT), mean4(W, q, 1, pT))
                                       : side_mask(fi * dx, (fj + 0.5f) * dx, (fk + 0.5f) * dx);
        nU[qu] =
            m == 0.0f ? 0.0f : m * fp.turb_amp * perlin(fi + fp.turb_offset, fj, fk, fp.turb_freq, 123);
    }
    if (i < g.W && k < g.D) {
        const float m = yi && xc && zc ? temp_mask(mean2(T, q, rT)) * speed_mask(mean4(U, qu, rU, 1), __ldg(V + qv), mean4(W, q, rT, pT))
                                       : side_mask((fi + 0.5f) * dx, fj * dx, (fk + 0.5f) * dx);
        nV[qv] =
            m == 0.0f ? 0.0f : m * fp.turb_amp * perlin(fi, fj + fp.turb_offset, fk, fp.turb_freq, 123);
    }
    if (i < g.W && j < g.H) {
        const float m = zi && xc && yc ? temp_mask(mean2(T, q, pT)) * speed_mask(mean4(U, qu, pU, 1), mean4(V, qv, pV, rT), __ldg(W + q))
                                       : side_mask((fi + 0.5f) * dx, (fj + 0.5f) * dx, fk * dx);
        nW[q] =
            m == 0.0f ? 0.0f : m * fp.turb_amp * perlin(fi, fj, fk + fp.turb_offset, fp.turb_freq, 123);
    }
}

void launch_turb_noise(const Geom &g, const float *T, const float *U, const float *V,
                       const float *W, float *nU, float *nV, float *nW, const ForceParams &fp,
                       cudaStream_t st) {
    k_turb_noise<<<face_grid(g), face_block(), 0, st>>>(g, T, U, V, W, nU, nV, nW, fp);
}

// Pseudo-curl of the noise field at every cell (add_curl_noise_kernel,
// FluidSolver.cu:271-293), rescaled to the cell's mean noise speed and
// multiplied by 0.5*dt.  dudx and dwdz subtract the V noise, as the
// reference does (lines 276, 278).  A pass of its own, so that the square
// roots and divisions of a cell are done once and not for each of its faces:
// 15 us and 20 us for the sum at 128^3, 50 us in one pass that forms four curls
// per thread.
__global__ void __launch_bounds__(256)
k_turb_curl(Geom g, const float *__restrict__ nU, const float *__restrict__ nV, const float *__restrict__ nW,
            float tiny, float *__restrict__ cx_out, float *__restrict__ cy_out, float *__restrict__ cz_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i >= g.W || j >= g.H || k >= g.D) return;
    const int rT = g.W, pT = rT * g.H, rU = rT + 1;
    const int q = i + rT * j + pT * k, qu = i + rU * j + rU * g.H * k, qv = i + rT * j + rT * (g.H + 1) * k;
    const float u0 = __ldg(nU + qu), u1 = __ldg(nU + (qu + 1));
    const float v0 = __ldg(nV + qv), v1 = __ldg(nV + (qv + rT));
    const float w0 = __ldg(nW + q), w1 = __ldg(nW + (q + pT));
    // Explicit roundings: where the differences are equal (e.g. masked-out
    // noise on three faces) the curl must be exactly zero.  A contracted
    // fma(a, s, -b*s) leaves a rounding residue instead, which the
    // normalisation below inflates to the full noise speed in an arbitrary
    // direction.
    const float dudx = __fmul_rn(__fsub_rn(u1, v0), g.inv_dx);
    const float dvdy = __fmul_rn(__fsub_rn(v1, v0), g.inv_dx);
    const float dwdz = __fmul_rn(__fsub_rn(w1, v0), g.inv_dx);
    const float cx = __fsub_rn(dvdy, dwdz), cy = __fsub_rn(dwdz, dudx), cz = __fsub_rn(dudx, dvdy);
    const float avg = len3((u0 + u1) / 2.0f, (v0 + v1) / 2.0f, (w0 + w1) / 2.0f);
    const float den = len3(cx, cy, cz) + tiny;
    const float h = 0.5f * g.dt;
    cx_out[q] = h * (avg * cx / den);
    cy_out[q] = h * (avg * cy / den);
    cz_out[q] = h * (avg * cz / den);
}

// Adds each face's two cells' pseudo-curls.
__global__ void __launch_bounds__(256)
k_turb_add(Geom g, float *__restrict__ U, float *__restrict__ V, float *__restrict__ W,
           const float *__restrict__ cx, const float *__restrict__ cy, const float *__restrict__ cz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z * blockDim.z + threadIdx.z;
    if (i > g.W || j > g.H || k > g.D) return;
    const bool self = i < g.W && j < g.H && k < g.D;
    const int rT = g.W, pT = rT * g.H, rU = rT + 1;
    const int q = i + rT * j + pT * k;
    auto add = [&](float *f, int e, const float *c, bool lower, int step) {
        float x = f[e];
        if (lower) x += __ldg(c + (q - step));
        if (self) x += __ldg(c + q);
        f[e] = x;
    };
    if (j < g.H && k < g.D) add(U, i + rU * j + rU * g.H * k, cx, i >= 1, 1);
    if (i < g.W && k < g.D) add(V, i + rT * j + rT * (g.H + 1) * k, cy, j >= 1, rT);
    if (i < g.W && j < g.H) add(W, q, cz, k >= 1, pT);
}

void launch_turb_apply(const Geom &g, float *U, float *V, float *W, const float *nU, const float *nV, const float *nW,
                       const ForceParams &fp, float *cx, float *cy, float *cz, cudaStream_t st) {
    k_turb_curl<<<cell_grid(g), face_block(), 0, st>>>(g, nU, nV, nW, fp.tiny, cx, cy, cz);
    k_turb_add<<<face_grid(g), face_block(), 0, st>>>(g, U, V, W, cx, cy, cz);
}

__global__ void k_perlin(const float *__restrict__ pos3, int n, float scale, int seed,
                         float *__restrict__ out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) out[t] = perlin(pos3[3 * t], pos3[3 * t + 1], pos3[3 * t + 2], scale, seed);
}

void launch_perlin(const float *pos3, int n, float scale, int seed, float *out, cudaStream_t st) {
    if (n > 0) k_perlin<<<(n + 255) / 256, 256, 0, st>>>(pos3, n, scale, seed, out);
}

} // namespace blz
