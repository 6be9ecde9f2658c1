// gs.cuh — the Gauss-Seidel update of four packed cells, shared by every sweep
// kernel so that all perform the same rounded operations per cell.
#pragma once
#include "kernels.cuh"

namespace blz {

// Quotient num/den for the neighbour count den in {1..6} as
// RN(num * hi + RN(num * lo)), hi = RN(1/den) and lo = RN(1/den - hi): two
// instructions on the FMA pipe instead of an IEEE division (a reciprocal and
// an int-to-float conversion per cell on the XU pipe) or a remainder-
// corrected product (three).  The result is within about half an ulp of the
// quotient and, unlike num * RN(1/den) alone, carries no bias: RN(1/3),
// RN(1/5) and RN(1/6) are all slightly large, and a sweep that scaled every
// update by 1 + 3e-8 would converge to the solution of A - 1.8e-7 I, whose
// smooth modes differ from A's by parts in 10^4 at 256^3.
__device__ __forceinline__ float inv_count(float den) {
    return den == 6.0f ? 1.0f / 6.0f : den == 5.0f ? 0.2f : den == 4.0f ? 0.25f
         : den == 3.0f ? 1.0f / 3.0f : den == 2.0f ? 0.5f : 1.0f;
}
__device__ __forceinline__ float inv_count_lo(float den) {
    return den == 6.0f ? -4.967053879312289e-09f : den == 5.0f ? -2.9802322831784522e-09f
         : den == 3.0f ? -9.934107758624577e-09f : 0.0f;
}
__device__ __forceinline__ float div_hl(float num, float hi, float lo) {
    return __fmaf_rn(num, hi, __fmul_rn(num, lo));
}
__device__ __forceinline__ float div_count(float num, float den) {
    return div_hl(num, inv_count(den), inv_count_lo(den));
}

__device__ __forceinline__ float4 ld4(const float *p) { return __ldg(reinterpret_cast<const float4 *>(p)); }

// Neighbour counts' reciprocals (hi, lo of div_hl) of a quad: the count is
// the same for every cell of the quad except the one at a row end (cell 0
// when the row's cells sit at even i and the quad starts the row, cell 3
// when odd and it ends the row), so they are formed three times per quad.
struct QuadDen {
    float l0, i0, lb, ib, l3, i3;
};

__device__ __forceinline__ QuadDen quad_den(const SolveParams &sp, int s, bool first, bool last, bool has_ym,
                                            bool has_yp, bool has_zm, bool has_zp) {
    const bool dir = sp.dirichlet;
    QuadDen q;
    const float db = 2.0f + (has_ym ? 1.0f : (dir && sp.open.ylo ? 1.0f : 0.0f)) +
                     (has_yp ? 1.0f : (dir && sp.open.yhi ? 1.0f : 0.0f)) +
                     (has_zm ? 1.0f : (dir && sp.open.zlo ? 1.0f : 0.0f)) +
                     (has_zp ? 1.0f : (dir && sp.open.zhi ? 1.0f : 0.0f));
    const float d0 = (s == 0 && first) ? db - 1.0f + (dir && sp.open.xlo ? 1.0f : 0.0f) : db;
    const float d3 = (s == 1 && last) ? db - 1.0f + (dir && sp.open.xhi ? 1.0f : 0.0f) : db;
    q.ib = inv_count(db);
    q.i0 = inv_count(d0);
    q.i3 = inv_count(d3);
    q.lb = inv_count_lo(db);
    q.l0 = inv_count_lo(d0);
    q.l3 = inv_count_lo(d3);
    return q;
}

// Updates four consecutive packed cells m0..m0+3 of one row given their
// neighbour counts: o is the other colour at the same packed indices, xe its
// value just outside the segment (m0-1 when the row's cells sit at even i,
// m0+4 when odd), ym/yp/zm/zp the other colour in rows j-1, j+1 and planes
// k-1, k+1.  A missing neighbour arrives as 0 (the caller passes zero4 and
// xe = 0), so the sum is branch free and in the reference's order.
__device__ __forceinline__ float4 gs_quad(float scale, int s, float4 r, float4 o, float xe, float4 ym, float4 yp,
                                          float4 zm, float4 zp, const QuadDen &q) {
    float xl[4], xr[4];
    if (s == 0) {
        xl[0] = xe; xl[1] = o.x; xl[2] = o.y; xl[3] = o.z;
        xr[0] = o.x; xr[1] = o.y; xr[2] = o.z; xr[3] = o.w;
    } else {
        xl[0] = o.x; xl[1] = o.y; xl[2] = o.z; xl[3] = o.w;
        xr[0] = o.y; xr[1] = o.z; xr[2] = o.w; xr[3] = xe;
    }
    const float ra[4] = {r.x, r.y, r.z, r.w};
    const float yma[4] = {ym.x, ym.y, ym.z, ym.w}, ypa[4] = {yp.x, yp.y, yp.z, yp.w};
    const float zma[4] = {zm.x, zm.y, zm.z, zm.w}, zpa[4] = {zp.x, zp.y, zp.z, zp.w};
    float out[4];
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        // every rounding explicit, so the packed form (gs_quad_pk) has the
        // same bits
        float num = __fmaf_rn(scale, ra[t], xl[t]);
        num = __fadd_rn(num, xr[t]);
        num = __fadd_rn(num, yma[t]);
        num = __fadd_rn(num, ypa[t]);
        num = __fadd_rn(num, zma[t]);
        num = __fadd_rn(num, zpa[t]);
        const float hi = t == 0 ? q.i0 : t == 3 ? q.i3 : q.ib;
        const float lo = t == 0 ? q.l0 : t == 3 ? q.l3 : q.lb;
        out[t] = div_hl(num, hi, lo);
    }
    return make_float4(out[0], out[1], out[2], out[3]);
}

// gs_quad on Blackwell's paired FP32 instructions: cells (0,1) and (2,3) of
// the quad go through one fma/add/mul.rn.f32x2 each, every lane rounded as
// IEEE FP32, in gs_quad's order, so the bits equal gs_quad's.
typedef unsigned long long f2_t;
__device__ __forceinline__ f2_t f2(float lo, float hi) {
    f2_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void f2_split(f2_t v, float &lo, float &hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2_t f2_fma(f2_t a, f2_t b, f2_t c) {
    f2_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2_t f2_add(f2_t a, f2_t b) {
    f2_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2_t f2_mul(f2_t a, f2_t b) {
    f2_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

__device__ __forceinline__ f2_t gs_pair(f2_t scale2, f2_t r, f2_t xl, f2_t xr, f2_t ym, f2_t yp, f2_t zm, f2_t zp,
                                        f2_t hi, f2_t lo) {
    f2_t num = f2_fma(scale2, r, xl);
    num = f2_add(num, xr);
    num = f2_add(num, ym);
    num = f2_add(num, yp);
    num = f2_add(num, zm);
    num = f2_add(num, zp);
    return f2_fma(num, hi, f2_mul(num, lo));
}

__device__ __forceinline__ float4 gs_quad_pk(float scale, int s, float4 r, float4 o, float xe, float4 ym, float4 yp,
                                             float4 zm, float4 zp, const QuadDen &q) {
    const f2_t sc = f2(scale, scale);
    const f2_t xl01 = s == 0 ? f2(xe, o.x) : f2(o.x, o.y), xl23 = s == 0 ? f2(o.y, o.z) : f2(o.z, o.w);
    const f2_t xr01 = s == 0 ? f2(o.x, o.y) : f2(o.y, o.z), xr23 = s == 0 ? f2(o.z, o.w) : f2(o.w, xe);
    const f2_t a = gs_pair(sc, f2(r.x, r.y), xl01, xr01, f2(ym.x, ym.y), f2(yp.x, yp.y), f2(zm.x, zm.y),
                           f2(zp.x, zp.y), f2(q.i0, q.ib), f2(q.l0, q.lb));
    const f2_t b = gs_pair(sc, f2(r.z, r.w), xl23, xr23, f2(ym.z, ym.w), f2(yp.z, yp.w), f2(zm.z, zm.w),
                           f2(zp.z, zp.w), f2(q.ib, q.i3), f2(q.lb, q.l3));
    float4 out;
    f2_split(a, out.x, out.y);
    f2_split(b, out.z, out.w);
    return out;
}

} // namespace blz
