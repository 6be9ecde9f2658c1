// unet_conv.cu — 3x3x3 convolution as an implicit GEMM on the tcgen05
// tensor cores (BF16 operands, FP32 accumulation in tensor memory).
//
// Activations are channels-last with a one-voxel zero halo on every side:
// element (x, y, z, c) of a W x H x D x C tensor sits at
// ((z+1)*Hp + (y+1))*Wp + (x+1)) * C + c with Wp = W+2, Hp = H+2, plus
// kSlack zero voxels before and after the tensor.  Weights are [27][Cout][Cin]
// (tap = (dz+1)*9 + (dy+1)*3 + (dx+1)), bias FP32 [Cout].
//
// One CTA computes M = 128 consecutive voxels of the padded plane z (its
// interior rows) for all N = Cout outputs.  For each 16-channel chunk of the
// input it stages the 9 input rows (dy, dz) of 130 voxels once, in the
// canonical K-major layout of the UMMA operand descriptor (8-voxel core
// matrices of 16 B rows, 128 B apart; the two 8-channel halves 2080 B
// apart).  Because a voxel's row is exactly 16 B at a linear position, the
// A operand of tap (dx, dy, dz) is the same block seen 16*(dx+1) B further
// on: 27 MMAs of M=128 x N x K=16 read one staged block.  The halo makes
// the zero padding of the convolution a plain memory read.
#include <algorithm>
#include <atomic>

#include <cuda_bf16.h>

#include "kernels.cuh"

namespace blz {

namespace {

constexpr int kConvM = 128;
constexpr int kRowVox = kConvM + 2;                 // 130 voxels per staged row
constexpr int kKgBytes = kRowVox * 16;              // one 8-channel half of a row
constexpr int kRowBytes = 2 * kKgBytes;             // 4160 B per staged row (16 ch)
constexpr int kABytes = 9 * kRowBytes;              // 37440 B

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory descriptor: K-major, no swizzle (canonical layout
// ((8,m),2):((1,SBO),LBO) in 16-byte units), descriptor version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;                          // version
    return d;                                        // base offset 0, layout SWIZZLE_NONE
}

// Instruction descriptor, kind::f16: D FP32, A and B BF16, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

__device__ __forceinline__ void st_shared_zero16(uint32_t dst) {
    asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(dst), "r"(0u) : "memory");
}

__device__ __forceinline__ unsigned long long conv_now_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// A commit group of one tile's MMAs completes in microseconds.
constexpr unsigned long long kConvWaitNs = 10ull * 1000ull * 1000ull;

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity, int *err) {
    // Bounded in time (device global timer, read only when the first tries
    // fail: the read is slow): gives up after kConvWaitNs, records the timeout
    // and returns.
    unsigned long long t0 = 0;
    for (;;) {
        for (int it = 0; it < 64; ++it) {
            uint32_t done;
            asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
                         " selp.u32 %0, 1, 0, p;\n}\n"
                         : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
            if (done) return true;
        }
        const unsigned long long t = conv_now_ns();
        if (t0 == 0) t0 = t;
        else if (t - t0 > kConvWaitNs) break;
    }
    if (err) atomicExch(err, 1);
    return false;
}

} // namespace

template <int N, bool RELU, bool OUT_F32>
__global__ void __launch_bounds__(128, 1)
k_conv3d_tc(int W, int H, int D, int cin, int out_stride, int out_offset, const __nv_bfloat16 *__restrict__ x,
            const __nv_bfloat16 *__restrict__ w, const float *__restrict__ bias, void *__restrict__ y,
            const __nv_bfloat16 *__restrict__ aux, int *err) {
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *sA = smem;
    unsigned char *sB = smem + kABytes;
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_base;
    constexpr int kCols = N < 32 ? 32 : N;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int Wp = W + 2, Hp = H + 2;
    const long long plane = (long long)Wp * Hp;
    const int z = blockIdx.y;
    const long long P0 = (long long)Wp + (long long)kConvM * blockIdx.x;   // first voxel of the tile

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const uint32_t aS = smem_u32(sA), bS = smem_u32(sB), mb = smem_u32(&mbar);
    constexpr uint32_t idesc = umma_idesc_bf16(kConvM, N);
    const int chunks = cin / 16;
    bool ok = true;
    for (int c = 0; c < chunks && ok; ++c) {
        // Stage the 9 input rows (dz, dy) of this 16-channel chunk: row r =
        // (dz + 1) * 3 + (dy + 1) holds 16-byte chunks (kg, v) at kg *
        // kKgBytes + v * 16, from voxel v of that row ...
#pragma unroll
        for (int r = 0; r < 9; ++r) {
            const int dz = r / 3 - 1, dy = r % 3 - 1;
            const __nv_bfloat16 *rs =
                x + ((long long)(z + 1 + dz) * plane + P0 - 1 + (long long)dy * Wp) * cin + c * 16;
            for (int e = tid; e < 2 * kRowVox; e += 128) {
                const int kg = e & 1, v = e >> 1;
                cp_async16(aS + r * kRowBytes + kg * kKgBytes + v * 16, rs + (long long)v * cin + kg * 8);
            }
        }
        // ... and the 27 taps' weights of the chunk (B: N x 16, K-major).
        for (int e = tid; e < 27 * N * 2; e += 128) {
            const int t = e / (N * 2), rem = e % (N * 2);
            const int n = rem >> 1, kg = rem & 1;
            cp_async16(bS + t * N * 32 + kg * N * 16 + n * 16, w + ((size_t)t * N + n) * cin + c * 16 + kg * 8);
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // a tap's operands: the block's descriptors plus constant offsets
            // in the 16-byte address field (addresses below 2^18 bytes, so
            // the field never carries)
            const uint64_t a_desc0 = umma_desc(aS, kKgBytes, 128), b_desc0 = umma_desc(bS, N * 16, 128);
#pragma unroll
            for (int t = 0; t < 27; ++t) {
                const int dz = t / 9 - 1, dy = (t / 3) % 3 - 1, dx = t % 3 - 1;
                const int r = (dz + 1) * 3 + (dy + 1);
                const uint64_t ad = a_desc0 + (uint64_t)((r * kRowBytes + (dx + 1) * 16) >> 4);
                const uint64_t bd = b_desc0 + (uint64_t)((t * N * 32) >> 4);
                const uint32_t acc = (c > 0 || t > 0) ? 1u : 0u;
                asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                             " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                             ::"r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(acc) : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(mb) : "memory");
        }
        // The staged block is reused by the next chunk only once the MMAs
        // that read it have completed.
        // (CTA-uniform outcome, so the .sync.aligned TMEM loads below never
        // run in a divergent warp.)
        ok = __syncthreads_and(mbar_wait(mb, (uint32_t)(c & 1), err)) != 0;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
        // Epilogue: warp w owns TMEM lanes 32w..32w+31 = voxels of the tile.
        const long long P = P0 + 32 * warp + lane;
        const int xp = (int)(P % Wp), yp = (int)(P / Wp);
        const bool inside = xp >= 1 && xp <= W && yp >= 1 && yp <= H;
        const long long outv = (long long)(z + 1) * plane + P;
#pragma unroll
        for (int n0 = 0; n0 < N; n0 += 16) {
            uint32_t r[16];
            const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)n0;
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                           "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
                           "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                         : "r"(taddr) : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (inside) {
                float v[16];
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    v[q] = __uint_as_float(r[q]) + (bias ? __ldg(bias + n0 + q) : 0.0f);
                    if (RELU) v[q] = fmaxf(v[q], 0.0f);
                }
                const long long o = outv * out_stride + out_offset + n0;
                if (aux) {
                    // Backward through a ReLU: keep the gradient where the
                    // forward activation was positive.
                    const uint4 a0 = __ldg(reinterpret_cast<const uint4 *>(aux + o));
                    const uint4 a1 = __ldg(reinterpret_cast<const uint4 *>(aux + o) + 1);
                    const __nv_bfloat16 *ah0 = reinterpret_cast<const __nv_bfloat16 *>(&a0);
                    const __nv_bfloat16 *ah1 = reinterpret_cast<const __nv_bfloat16 *>(&a1);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        if (!(__bfloat162float(ah0[q]) > 0.0f)) v[q] = 0.0f;
                        if (!(__bfloat162float(ah1[q]) > 0.0f)) v[8 + q] = 0.0f;
                    }
                }
                if (OUT_F32) {
                    float4 *dst = reinterpret_cast<float4 *>(static_cast<float *>(y) + o);
#pragma unroll
                    for (int q = 0; q < 4; ++q) dst[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                } else {
                    __nv_bfloat162 h[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
                    uint4 *dst = reinterpret_cast<uint4 *>(static_cast<__nv_bfloat16 *>(y) + o);
                    dst[0] = *reinterpret_cast<uint4 *>(&h[0]);
                    dst[1] = *reinterpret_cast<uint4 *>(&h[4]);
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols) : "memory");
}

int conv3d_smem_bytes(int cout) { return kABytes + 27 * cout * 32; }

// ---------------------------------------------------------------------------
// z-marching variant for the layers of 16 to 128 input and output channels.  A
// CTA keeps the layer's weights resident and walks a tile of 8 x 16 voxels (x, y)
// through `zs` output planes.
//
// What bounds such a layer is the number of MMAs: with 16 output channels one
// of 128 x 16 x 16 takes as long as one three times as wide, since both read the
// same 128 x 16 operand of voxels.  So each staged block, the 16-channel chunk c
// of input plane p, is used once, for the three output planes it reaches: an
// MMA per (dy, dx) with N = 3 Cout, the weights of dz = +1, 0, -1 side by side
// and the accumulators of output planes p - 1, p, p + 1 side by side in a TMEM
// ring of R planes.  9 MMAs instead of 27 (10, since a new plane's first one
// overwrites while the others add).  Chunk c runs 2 c planes behind chunk 0, so
// every output still adds its taps in the general kernel's order, chunk by chunk
// and tap by tap, and has its bits.
//
// A tile of 8 x 16 voxels instead of 128 in a row reads 1.4 input voxels per
// output voxel and plane, not 3, and its block arrives by TMA as one box of 10 x
// 18 voxels of 32 bytes in the K-major layout of the 32-byte swizzle, which is a
// function of the shared address (slots are whole periods of it), 320 bytes from
// row to row: tap (dy, dx) is the same block seen 320 dy + 32 dx bytes on.
//
// Warps: four read finished accumulators out of TMEM, add bias / ReLU and store;
// one issues the MMAs (the whole warp runs the loop, so descriptors are uniform
// values, and an elected lane issues); one issues the copies.  They hand over
// through mbarriers only: full / empty per ring slot, done / free per accumulator.
// Every wait is bounded in time; a wait that gives up sets the error flag and ends
// that warp's loop, which ends the others' at their next wait; before the CTA
// ends, the MMA warp waits for its last commit and the copy warp for every copy
// it issued.
//
// Layers whose weights do not fit (64 or 128 channels in, 64 or 128 out) are cut
// by output channels: a CTA takes N of them, so the input is staged cout / N
// times, mostly from L2.
//
// Measured, us: 16 -> 16 and 32 -> 16 at 256^3 317 and 538, 32 -> 32 and 64 -> 32
// at 128^3 130 and 290 (an MMA per tap and output plane on 128 voxels of a row: 738,
// 1994, 298 and, general kernel, 1146); by parts, 64 -> 64 and 128 -> 64 at 64^3
// 81 and 252 (general kernel about 228 and 456).  What bounds it is the MMA warp: a block
// costs it about 900 cycles of waits, descriptors and 9 or 10 MMAs, with the
// copies taken out as with them.  So small layers share an SM, up to four CTAs
// (16 -> 16: 460 us with two; at 192^3 an SM then issues an MMA every 66 cycles,
// the tensor pipe is active 34 % of the time and the fullest unit is the L1, 77 %);
// the usual case of three planes inside the ring has its own path with
// constant descriptors, and an elected lane issues (64 -> 32: 360 us without the
// two).  The swizzle's 32-byte runs against 16-byte ones: 343 against 367 (16 ->
// 16, before the last two).
// ---------------------------------------------------------------------------
constexpr int kZmWorkers = 128;                           // epilogue warps 0-3
constexpr int kZmThreads = kZmWorkers + 64;               // + the MMA warp + the copy warp
constexpr int kZmTX = 8, kZmTY = 16;                      // tile (x, y)
constexpr int kZmRow = (kZmTX + 2) * 32;                  // bytes of one row of a block, 16 channels a voxel
constexpr int kZmBytes = (kZmTY + 2) * kZmRow;            // a block: 10 x 18 voxels
constexpr int kZmBlock = (kZmBytes + 1023) / 1024 * 1024; // ring slots, whole periods of the swizzle
constexpr int zm_room(int ctas) { return ctas == 1 ? 227 * 1024 - 1024 : 228 * 1024 / ctas - 1024 - 512; }   // dynamic bytes a CTA
constexpr int kZmMaxSlots = 12;

template <int N, int CIN> struct Zm {
    static constexpr int CH = CIN / 16;
    static constexpr int kWeights = 27 * CH * N * 32;
    // output planes in flight: 3 for a plane's own MMAs, 2 per later chunk, and
    // at least 3 being read out; a power of two
    static constexpr int R = 2 * (CH - 1) + 6 <= 8 ? 8 : 2 * (CH - 1) + 6 <= 16 ? 16 : 32;
    static constexpr int kCols = R * N;
    // CTAs per SM, as many as tensor memory and shared memory with four ring
    // slots or more hold
    static constexpr int slots(int ctas) { return (zm_room(ctas) - kWeights - 1024) / kZmBlock; }
    static constexpr int kPerSm = kCols * 4 <= 512 && slots(4) >= 4 ? 4 : kCols * 3 <= 512 && slots(3) >= 4 ? 3
                                  : kCols * 2 <= 512 && slots(2) >= 4 ? 2 : 1;
    static constexpr int kRoom = slots(kPerSm);
    static constexpr int SL = kRoom < kZmMaxSlots ? kRoom : kZmMaxSlots;
    static constexpr int kSmem = kWeights + 1024 + SL * kZmBlock;
    static_assert(kCols <= 512 && SL >= 4, "TMEM columns and ring slots");
};

// One lane of a converged warp.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred q;\n elect.sync _|q, 0xffffffff;\n selp.u32 %0, 1, 0, q;\n}\n" : "=r"(p));
    return p != 0;
}
// One tcgen05.mma; descriptors as 32-bit halves (offsets only move the address
// field, in the low half).
__device__ __forceinline__ void zm_mma(uint32_t d, uint32_t a, uint32_t a_hi, uint32_t b, uint32_t b_hi,
                                       uint32_t idesc, uint32_t acc) {
    asm volatile("{\n .reg .pred p;\n .reg .b64 da, db;\n setp.ne.b32 p, %6, 0;\n"
                 " mov.b64 da, {%1, %2};\n mov.b64 db, {%3, %4};\n"
                 " tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n}\n"
                 ::"r"(d), "r"(a), "r"(a_hi), "r"(b), "r"(b_hi), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void zm_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

template <int N, int CIN, bool RELU>
__global__ void __launch_bounds__(kZmThreads, Zm<N, CIN>::kPerSm)
k_conv3d_zm(int W, int H, int D, int zs, int parts, int out_stride, int out_offset,
            const __grid_constant__ CUtensorMap xmap,
            const __nv_bfloat16 *__restrict__ w, const float *__restrict__ bias, __nv_bfloat16 *__restrict__ y,
            const __nv_bfloat16 *__restrict__ aux, int *err) {
    extern __shared__ __align__(128) unsigned char smem[];
    typedef Zm<N, CIN> Z;
    constexpr int CH = Z::CH, R = Z::R, SL = Z::SL;
    constexpr int kTap = 3 * N * 32;                      // bytes of one (chunk, dy, dx)'s weights
    __shared__ __align__(8) uint64_t full[SL], empty[SL], accf[R], acce[R], fin;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int Wp = W + 2, Hp = H + 2;
    const int part = blockIdx.z % parts, cout = parts * N;      // this CTA's output channels: part N .. part N + N - 1
    const int X0 = blockIdx.x * kZmTX, Y0 = blockIdx.y * kZmTY, z0 = (int)(blockIdx.z / parts) * zs;
    w += (size_t)part * N * CIN;
    if (bias) bias += part * N;
    out_offset += part * N;
    const int nz = (z0 + zs < D ? z0 + zs : D) - z0;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base)), "r"(Z::kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        auto init = [](uint64_t *b, int n) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(n) : "memory");
        };
        for (int s = 0; s < SL; ++s) { init(&full[s], 1); init(&empty[s], 1); }
        for (int b = 0; b < R; ++b) { init(&accf[b], 1); init(&acce[b], kZmWorkers); }
        init(&fin, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t aS = (smem_u32(smem) + 1023u) & ~1023u;     // the ring, then the weights
    const uint32_t bS = aS + (uint32_t)(SL * kZmBlock);
    // Weights: per (chunk, dy, dx) 3 N rows of 16 channels, K-major: the rows of
    // output plane p - 1 (dz = +1), p (0), p + 1 (-1).
    for (int e = tid; e < 27 * CH * N * 2; e += kZmThreads) {
        const int kg = e & 1, n = (e >> 1) % N, ct = (e >> 1) / N;          // ct = ch * 27 + tap
        const int ch = ct / 27, t = ct % 27, o = 2 - t / 9, t9 = t % 9;
        cp_async16(bS + (ch * 9 + t9) * kTap + kg * 3 * N * 16 + (o * N + n) * 16,
                   w + ((size_t)t * cout + n) * CIN + ch * 16 + kg * 8);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmem_base, 0);
    // Blocks in order: round s takes chunk c of input plane z0 - 1 + s - 2 c, for
    // the planes z0 - 1 .. z0 + nz.
    const int rounds = nz + 2 + 2 * (CH - 1);
    auto in_range = [&](int p) { return p >= z0 - 1 && p <= z0 + nz; };

    if (warp < 4) {
        // ---- epilogue: this thread's voxel of the tile is TMEM lane tid ----
        const int xv = X0 + (tid & 7), yv = Y0 + (tid >> 3);
        const bool inside = xv < W && yv < H;
        const long long plane = (long long)Wp * Hp, Pv = (long long)(yv + 1) * Wp + xv + 1;
        bool ok = true;
#pragma unroll 1
        for (int it = 0; it < nz && ok; ++it) {
            const int slot = it & (R - 1);
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&accf[slot]), (uint32_t)((it / R) & 1), err));
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const long long outv = (long long)(z0 + it + 1) * plane + Pv;
#pragma unroll
            for (int n0 = 0; n0 < N; n0 += 16) {
                uint32_t r[16];
                const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(slot * N + n0);
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                               "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
                               "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                             : "r"(taddr) : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (n0 + 16 == N) {
                    // read out: the buffer may be overwritten
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acce[slot])) : "memory");
                }
                if (inside) {
                    float v[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        v[q] = __uint_as_float(r[q]) + (bias ? __ldg(bias + n0 + q) : 0.0f);
                        if (RELU) v[q] = fmaxf(v[q], 0.0f);
                    }
                    const long long o = outv * out_stride + out_offset + n0;
                    if (aux) {
                        const uint4 a0 = __ldg(reinterpret_cast<const uint4 *>(aux + o));
                        const uint4 a1 = __ldg(reinterpret_cast<const uint4 *>(aux + o) + 1);
                        const __nv_bfloat16 *ah0 = reinterpret_cast<const __nv_bfloat16 *>(&a0);
                        const __nv_bfloat16 *ah1 = reinterpret_cast<const __nv_bfloat16 *>(&a1);
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            if (!(__bfloat162float(ah0[q]) > 0.0f)) v[q] = 0.0f;
                            if (!(__bfloat162float(ah1[q]) > 0.0f)) v[8 + q] = 0.0f;
                        }
                    }
                    __nv_bfloat162 h[8];
#pragma unroll
                    for (int q = 0; q < 8; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
                    uint4 *dst = reinterpret_cast<uint4 *>(y + o);
                    dst[0] = *reinterpret_cast<uint4 *>(&h[0]);
                    dst[1] = *reinterpret_cast<uint4 *>(&h[4]);
                }
            }
        }
    } else if (warp == 4) {
        // ---- MMA warp ----
        // Every operand address stays below 2^18 bytes, so adding an offset's
        // 16-byte units to the 14-bit address field never carries.
        const uint64_t a_desc0 = umma_desc(aS, 16, kZmRow) | (uint64_t)6 << 61, b_desc0 = umma_desc(bS, 3 * N * 16, 128);
        const uint32_t a_lo = (uint32_t)a_desc0, a_hi = (uint32_t)(a_desc0 >> 32);
        const uint32_t b_lo = (uint32_t)b_desc0, b_hi = (uint32_t)(b_desc0 >> 32);
        const bool lead = elect_one();
        bool ok = true;
        int n = 0, slot = 0;                              // blocks taken; the next one's ring slot
        uint32_t phase = 0;
#pragma unroll 1
        for (int s = 0; s < rounds && ok; ++s)
#pragma unroll 1
            for (int c = 0; c < CH; ++c) {
                const int p = z0 - 1 + s - 2 * c;
                if (!in_range(p)) continue;
                bool done = mbar_wait(smem_u32(&full[slot]), phase, err);
                // output planes lo .. hi as iterations of this CTA; the last is
                // new where chunk 0 meets it for the first time
                const int lo = p - 1 < z0 ? 0 : p - 1 - z0, hi = p + 1 > z0 + nz - 1 ? nz - 1 : p + 1 - z0;
                const bool fresh = c == 0 && hi == p + 1 - z0;
                if (fresh && hi >= R)
                    done = mbar_wait(smem_u32(&acce[hi & (R - 1)]), (uint32_t)((hi / R - 1) & 1), err) && done;
                if (!__all_sync(0xffffffffu, done)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t ad0 = a_lo + (uint32_t)((slot * kZmBlock) >> 4);
                // weights' rows start at output plane p - 1
                const uint32_t bd0 = b_lo + (uint32_t)((c * 9 * kTap + (lo + z0 - (p - 1)) * N * 16) >> 4);
                // the ring's end may split the columns of lo .. hi: `head` planes
                // up to it, the rest from its start
                const int first = lo & (R - 1), count = hi - lo + 1, head = first + count > R ? R - first : count;
                const uint32_t d0 = tmem + (uint32_t)(first * N);
                auto idesc = [&](int planes) { return umma_idesc_bf16(kConvM, 0) + ((uint32_t)(planes * N / 8) << 17); };
                auto offset = [&](int planes) { return (uint32_t)(planes * N); };        // weights' rows, 16 bytes each
                auto tap = [&](int t) { return (uint32_t)(((t / 3) * kZmRow + (t % 3) * 32) >> 4); };
                if (lead) {
                    // tap 0 of a new plane overwrites, the other planes' add
                    if (hi - lo == 2 && first <= R - 3) {          // three planes, inside the ring
                        constexpr uint32_t id3 = umma_idesc_bf16(kConvM, 3 * N);
                        if (fresh) {
                            zm_mma(d0, ad0, a_hi, bd0, b_hi, umma_idesc_bf16(kConvM, 2 * N), 1u);
                            zm_mma(d0 + 2 * N, ad0, a_hi, bd0 + offset(2), b_hi, umma_idesc_bf16(kConvM, N), 0u);
                        } else {
                            zm_mma(d0, ad0, a_hi, bd0, b_hi, id3, 1u);
                        }
#pragma unroll
                        for (int t = 1; t < 9; ++t)
                            zm_mma(d0, ad0 + tap(t), a_hi, bd0 + (uint32_t)((t * kTap) >> 4), b_hi, id3, 1u);
                    } else {
                        int t0 = 0;
                        if (fresh) {
                            const int old = count - 1, h = head < old ? head : old;
                            if (h > 0) zm_mma(d0, ad0, a_hi, bd0, b_hi, idesc(h), 1u);
                            if (old > h) zm_mma(tmem, ad0, a_hi, bd0 + offset(h), b_hi, idesc(old - h), 1u);
                            zm_mma(tmem + (uint32_t)((hi & (R - 1)) * N), ad0, a_hi, bd0 + offset(old), b_hi, idesc(1), 0u);
                            t0 = 1;
                        }
                        const uint32_t id0 = idesc(head), id1 = idesc(count - head), bd1 = bd0 + offset(head);
                        if (head == count) {
                            if (t0 == 0) zm_mma(d0, ad0, a_hi, bd0, b_hi, id0, 1u);
#pragma unroll
                            for (int t = 1; t < 9; ++t)
                                zm_mma(d0, ad0 + tap(t), a_hi, bd0 + (uint32_t)((t * kTap) >> 4), b_hi, id0, 1u);
                        } else {
#pragma unroll 1
                            for (int t = t0; t < 9; ++t) {
                                zm_mma(d0, ad0 + tap(t), a_hi, bd0 + (uint32_t)((t * kTap) >> 4), b_hi, id0, 1u);
                                zm_mma(tmem, ad0 + tap(t), a_hi, bd1 + (uint32_t)((t * kTap) >> 4), b_hi, id1, 1u);
                            }
                        }
                    }
                    zm_commit(smem_u32(&empty[slot]));
                    if (c == CH - 1 && p - 1 >= z0) zm_commit(smem_u32(&accf[(p - 1 - z0) & (R - 1)]));
                }
                ++n;
                if (++slot == SL) { slot = 0; phase ^= 1u; }
            }
        // The last MMAs complete before the accumulator columns are released,
        // also when a wait gave up (bounded wait).
        if (n > 0) {
            if (lead) zm_commit(smem_u32(&fin));
            mbar_wait(smem_u32(&fin), 0, nullptr);
        }
    } else if (lane == 0) {
        // ---- copy warp ----
        int n = 0, slot = 0;
        uint32_t phase = 1;                               // a fresh barrier's previous phase has completed
        bool ok = true;
        for (int s = 0; s < rounds && ok; ++s)
            for (int c = 0; c < CH; ++c) {
                const int p = z0 - 1 + s - 2 * c;
                if (!in_range(p)) continue;
                if (!mbar_wait(smem_u32(&empty[slot]), phase, err)) { ok = false; break; }
                const uint32_t bar = smem_u32(&full[slot]);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(kZmBytes) : "memory");
                asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                             " [%0], [%1, {%2, %3, %4, %5}], [%6];"
                             ::"r"(aS + (uint32_t)(slot * kZmBlock)), "l"(reinterpret_cast<uint64_t>(&xmap)), "r"(16 * c),
                               "r"(X0), "r"(Y0), "r"(p + 1), "r"(bar)
                             : "memory");
                ++n;
                if (++slot == SL) { slot = 0; phase ^= 1u; }
            }
        // No copy may land after the CTA ends (done already unless a wait gave up).
        for (int q = n - 1; q >= 0 && q >= n - SL; --q)
            mbar_wait(smem_u32(&full[q % SL]), (uint32_t)((q / SL) & 1), nullptr);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Z::kCols) : "memory");
}

// Tensor map of a padded channels-last activation x (CIN channels, W+2 x
// H+2 x D+2 voxels from x): dims (channel, x, y, z), box (16, 10, 18, 1): one
// 16-channel chunk of a tile with its border, 32-byte swizzle.  The innermost
// coordinate of every copy is a multiple of 16, so every copy starts 32-byte
// aligned; voxels past the tensor read as zeros.
static bool zm_tensor_map(CUtensorMap *m, const __nv_bfloat16 *x, const ConvDesc &cd) {
    TensorMapEncodeFn enc = tensor_map_encoder();
    if (!enc || (reinterpret_cast<uintptr_t>(x) & 15) != 0) return false;
    const cuuint64_t Wp = (cuuint64_t)cd.W + 2, Hp = (cuuint64_t)cd.H + 2, Dp = (cuuint64_t)cd.D + 2;
    const cuuint64_t C = (cuuint64_t)cd.cin;
    const cuuint64_t dims[4] = {C, Wp, Hp, Dp};
    const cuuint64_t strides[3] = {C * 2, Wp * C * 2, Wp * Hp * C * 2};
    const cuuint32_t box[4] = {16, kZmTX + 2, kZmTY + 2, 1};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16 *>(x), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int conv_sm_count() {
    static std::atomic<int> cache[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (cache[dev] == 0) {
        int n = 0;
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        cache[dev] = n > 0 ? n : 148;
    }
    return cache[dev];
}

template <int N, int CIN, bool RELU>
static cudaError_t launch_zm(const ConvDesc &cd, const __nv_bfloat16 *x, const __nv_bfloat16 *w, const float *bias,
                             void *y, const __nv_bfloat16 *aux, int *err, cudaStream_t st) {
    typedef Zm<N, CIN> Z;
    cudaError_t e = allow_smem((const void *)k_conv3d_zm<N, CIN, RELU>, Z::kSmem);
    if (e != cudaSuccess) return e;
    CUtensorMap xm;
    if (!zm_tensor_map(&xm, x, cd)) return cudaErrorNotSupported;
    // Output planes per CTA: the least time of a whole number of waves, a CTA of
    // zs planes taking zs + 2 + 2 (CH - 1) rounds and about 6 more to start.
    const int parts = cd.cout / N;
    const long long tiles = (long long)((cd.W + kZmTX - 1) / kZmTX) * ((cd.H + kZmTY - 1) / kZmTY) * parts;
    const long long room = (long long)conv_sm_count() * Z::kPerSm;
    int zs = 0;
    long long best = 0;
    for (int v = 4; v <= 64; v <<= 1) {
        const long long ctas = tiles * ((cd.D + v - 1) / v), cost = (ctas + room - 1) / room * (v + 2 * Z::CH + 6);
        if (zs == 0 || cost < best) { zs = v; best = cost; }
    }
    const dim3 grid((unsigned)((cd.W + kZmTX - 1) / kZmTX), (unsigned)((cd.H + kZmTY - 1) / kZmTY),
                    (unsigned)(parts * ((cd.D + zs - 1) / zs)));
    const int os = cd.out_stride > 0 ? cd.out_stride : cd.cout;
    k_conv3d_zm<N, CIN, RELU><<<grid, kZmThreads, Z::kSmem, st>>>(cd.W, cd.H, cd.D, zs, parts, os, cd.out_offset, xm, w, bias,
                                                                  static_cast<__nv_bfloat16 *>(y), aux, err);
    return cudaGetLastError();
}

// The z-marching kernel: BF16 output and a pair of channel counts whose weights
// and accumulators fit.
static bool zm_dispatch(const ConvDesc &cd, const __nv_bfloat16 *x, const __nv_bfloat16 *w, const float *bias,
                        void *y, const __nv_bfloat16 *aux, int *err, cudaStream_t st, cudaError_t *res) {
    if (cd.out_f32) return false;
#define BLZ_ZM(OUT, NN, CC)                                                                         \
    if (cd.cout == OUT && cd.cin == CC) {                                                           \
        *res = cd.relu ? launch_zm<NN, CC, true>(cd, x, w, bias, y, aux, err, st)                   \
                       : launch_zm<NN, CC, false>(cd, x, w, bias, y, aux, err, st);                 \
        return true;                                                                                \
    }
    BLZ_ZM(16, 16, 16)
    BLZ_ZM(16, 16, 32)
    BLZ_ZM(32, 32, 16)
    BLZ_ZM(32, 32, 32)
    BLZ_ZM(32, 32, 64)
    BLZ_ZM(64, 64, 32)
    // weights past shared memory: by parts of the output channels
    BLZ_ZM(64, 32, 64)
    BLZ_ZM(128, 32, 64)
    BLZ_ZM(64, 16, 128)
    BLZ_ZM(128, 16, 128)
#undef BLZ_ZM
    return false;
}

template <int N, bool RELU, bool F32>
static cudaError_t launch_n(const ConvDesc &cd, const __nv_bfloat16 *x, const __nv_bfloat16 *w, const float *bias,
                            void *y, const __nv_bfloat16 *aux, int *err, cudaStream_t st) {
    const int smem = conv3d_smem_bytes(N);
    cudaError_t e = allow_smem((const void *)k_conv3d_tc<N, RELU, F32>, smem);
    if (e != cudaSuccess) return e;
    const long long interior = (long long)(cd.W + 2) * cd.H;
    const dim3 grid((unsigned)((interior + kConvM - 1) / kConvM), (unsigned)cd.D);
    const int os = cd.out_stride > 0 ? cd.out_stride : cd.cout;
    k_conv3d_tc<N, RELU, F32><<<grid, 128, smem, st>>>(cd.W, cd.H, cd.D, cd.cin, os, cd.out_offset, x, w, bias, y,
                                                        aux, err);
    return cudaGetLastError();
}

cudaError_t launch_conv3d(const ConvDesc &cd, const __nv_bfloat16 *x, const __nv_bfloat16 *w, const float *bias,
                          void *y, int *err, cudaStream_t st, const __nv_bfloat16 *aux) {
    if (cd.cin % 16 || cd.cin <= 0 || cd.out_offset % 8 || (cd.out_stride > 0 && cd.out_stride % 8) ||
        (aux && cd.out_f32))
        return cudaErrorInvalidValue;
    cudaError_t res = cudaSuccess;
    if (zm_dispatch(cd, x, w, bias, y, aux, err, st, &res)) return res;
#define BLZ_CONV_CASE(NN)                                                                        \
    if (cd.cout == NN) {                                                                         \
        if (cd.out_f32) return cd.relu ? launch_n<NN, true, true>(cd, x, w, bias, y, aux, err, st) \
                                       : launch_n<NN, false, true>(cd, x, w, bias, y, aux, err, st); \
        return cd.relu ? launch_n<NN, true, false>(cd, x, w, bias, y, aux, err, st)             \
                       : launch_n<NN, false, false>(cd, x, w, bias, y, aux, err, st);          \
    }
    BLZ_CONV_CASE(16)
    BLZ_CONV_CASE(32)
    BLZ_CONV_CASE(64)
    BLZ_CONV_CASE(128)
#undef BLZ_CONV_CASE
    return cudaErrorInvalidValue;
}

// ---------------------------------------------------------------------------
// 2x2x2 stride-2 transposed convolution on the tensor cores.  Fine voxel
// (2x+a, 2y+b, 2z+c) = bias + W[a + 2b + 4c] . x[x, y, z], so the 8 parities
// of a coarse voxel are one GEMM row: one CTA takes M = 128 consecutive
// padded coarse voxels of interior plane z (its interior rows, as the 3x3x3
// kernels tile a plane) and computes D[128 x 8 COUT] = X[128 x CIN] W^T with
// W in BF16 [8][COUT][CIN] (GEMM row n = par * COUT + co), K = 16 per MMA,
// N = 8 COUT split into MMAs of at most 256 columns.  Operands are staged
// once by cp.async in the canonical K-major layouts of the 3x3x3 kernels
// (A: [chunk][kg][voxel][8], B: [chunk][kg][n][8]); one thread issues the
// MMAs and commits them to an mbarrier (bounded wait); the epilogue reads
// each parity's COUT columns from TMEM, adds the bias and stores BF16 into
// the fine voxel's channels [0, COUT) of a tensor with channel stride ys.
//
// Persistent: as many CTAs as the SMs' tensor memory holds, the weights staged
// once each and the next tile's voxels while this one's are read out.  What
// bounds it is the output, 16 channels of 32 (with the skip half) per fine voxel
// at 256^3, whose 32-byte sectors one store fills.  32 -> 16 to 256^3 196 us, 64 ->
// 32 to 128^3 54, 128 -> 64 to 64^3 21; a CTA per tile that staged, multiplied and
// read out in turn, with 16-byte stores: 390, 106 and 37.
// ---------------------------------------------------------------------------
template <int CIN, int COUT> struct UpShape {
    static constexpr int N = 8 * COUT, CH = CIN / 16;
    static constexpr int kAChunk = 2 * kConvM * 16;      // [kg][voxel][8] of one 16-channel chunk
    static constexpr int kBChunk = 2 * N * 16;           // [kg][n][8] of one 16-channel chunk
    static constexpr int kABytes = CH * kAChunk;
    static constexpr int SMEM = 2 * kABytes + CH * kBChunk;
    static constexpr int kPerSm = 512 / N;               // CTAs an SM's tensor memory holds
    static_assert(kPerSm * (SMEM + 1024) <= 227 * 1024, "shared memory for as many");
};

// 16 BF16 outputs of a voxel: one 32-byte store, which fills its sector, where
// the tensor's layout allows it.
__device__ __forceinline__ void st_bf16x16(__nv_bfloat16 *dst, const uint32_t v[8], bool wide) {
    if (wide) {
        asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                     ::"l"(dst), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                     : "memory");
    } else {
        reinterpret_cast<uint4 *>(dst)[0] = make_uint4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<uint4 *>(dst)[1] = make_uint4(v[4], v[5], v[6], v[7]);
    }
}
static bool wide_stores(const void *y, int stride, int offset) {
    return (reinterpret_cast<uintptr_t>(y) & 31) == 0 && stride % 16 == 0 && offset % 16 == 0;
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(128, 1)
k_upconv_tc(int W, int H, int D, const __nv_bfloat16 *__restrict__ x, const __nv_bfloat16 *__restrict__ w,
            const float *__restrict__ bias, __nv_bfloat16 *__restrict__ y, int ys, int wide, int *err) {
    typedef UpShape<CIN, COUT> S;
    constexpr int N = S::N, CH = S::CH, kAChunk = S::kAChunk, kBChunk = S::kBChunk;
    constexpr int NMMA = N > 256 ? 256 : N;              // columns per MMA
    constexpr int kCols = N;                              // 128, 256 or 512: a power of two
    constexpr uint32_t idesc = umma_idesc_bf16(kConvM, NMMA);
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ __align__(16) float sbias[COUT];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int Wp = W + 2, Hp = H + 2;
    const long long plane = (long long)Wp * Hp;
    const int tiles_x = (Wp * H + kConvM - 1) / kConvM, tiles = tiles_x * D;

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base)), "r"(kCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int e = tid; e < COUT; e += 128) sbias[e] = bias[e];
    const uint32_t aS = smem_u32(smem), bS = aS + (uint32_t)(2 * S::kABytes);
    // Tile t: 128 voxels of interior coarse plane t / tiles_x.  A: 16-byte chunk
    // (c, kg) of voxel v at c kAChunk + kg 2048 + v 16.
    auto stage = [&](int t, uint32_t dst) {
        const int z = t / tiles_x;
        const __nv_bfloat16 *xs = x + ((long long)(z + 1) * plane + Wp + (long long)kConvM * (t - z * tiles_x)) * CIN;
        for (int e = tid; e < CH * 2 * kConvM; e += 128) {
            const int kc = e % (2 * CH), v = e / (2 * CH);      // a voxel's chunks side by side: whole lines
            cp_async16(dst + (kc >> 1) * kAChunk + (kc & 1) * (kConvM * 16) + v * 16, xs + (long long)v * CIN + kc * 8);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // B: 16-byte chunk (c, kg) of row n at bS + c kBChunk + kg N 16 + n 16.
    for (int e = tid; e < CH * 2 * N; e += 128) {
        const int c = e / (2 * N), r = e % (2 * N), kg = r & 1, n = r >> 1;
        cp_async16(bS + c * kBChunk + kg * (N * 16) + n * 16, w + (size_t)n * CIN + c * 16 + kg * 8);
    }
    int tile = blockIdx.x;
    if (tile < tiles) stage(tile, aS);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    const long long Wf = 2LL * W + 2, Hf = 2LL * H + 2;
    uint32_t tmem = 0;
    bool ok = true;
#pragma unroll 1
    for (int it = 0; tile < tiles && ok; ++it, tile += gridDim.x) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // staged, and the previous tile read out of tensor memory
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem = tmem_base;
        const uint32_t aT = aS + (uint32_t)((it & 1) * S::kABytes);
        if (tid == 0) {
#pragma unroll
            for (int c = 0; c < CH; ++c) {
#pragma unroll
                for (int h = 0; h < N / NMMA; ++h) {
                    const uint64_t ad = umma_desc(aT + c * kAChunk, kConvM * 16, 128);
                    const uint64_t bd = umma_desc(bS + c * kBChunk + h * NMMA * 16, N * 16, 128);
                    const uint32_t accum = c > 0 ? 1u : 0u;
                    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                                 ::"r"(tmem + (uint32_t)(h * NMMA)), "l"(ad), "l"(bd), "r"(idesc), "r"(accum)
                                 : "memory");
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(smem_u32(&mbar)) : "memory");
        }
        // the other buffer's MMAs completed before the last epilogue
        if (tile + (int)gridDim.x < tiles) stage(tile + gridDim.x, aS + (uint32_t)(((it & 1) ^ 1) * S::kABytes));
        // CTA-uniform outcome, so the .sync.aligned TMEM loads never run in a
        // divergent warp.
        ok = __syncthreads_and(mbar_wait(smem_u32(&mbar), (uint32_t)(it & 1), err)) != 0;
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // warp w owns TMEM lanes 32w..32w+31 = voxels of the tile
        const int z = tile / tiles_x, Pv = Wp + kConvM * (tile - z * tiles_x) + 32 * warp + lane;
        const int yv = Pv / Wp, xv = Pv - yv * Wp;
        const bool inside = xv >= 1 && xv <= W && yv >= 1 && yv <= H;
        const int cx = xv - 1, cy = yv - 1;
#pragma unroll 1
        for (int n2 = 0; n2 < N; n2 += 32) {              // two runs of 16 columns: (parity, 16 channels)
            uint32_t r[32];
            const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)n2;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t *q = r + 16 * h;
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                             : "=r"(q[0]), "=r"(q[1]), "=r"(q[2]), "=r"(q[3]), "=r"(q[4]), "=r"(q[5]), "=r"(q[6]),
                               "=r"(q[7]), "=r"(q[8]), "=r"(q[9]), "=r"(q[10]), "=r"(q[11]), "=r"(q[12]),
                               "=r"(q[13]), "=r"(q[14]), "=r"(q[15])
                             : "r"(taddr + 16u * h) : "memory");
            }
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (inside) {
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int n = n2 + 16 * h, par = n / COUT, n0 = n % COUT;
                    const long long f = ((long long)(2 * z + (par >> 2) + 1) * Hf + (2 * cy + ((par >> 1) & 1) + 1)) * Wf +
                                        (2 * cx + (par & 1) + 1);
                    uint32_t v[8];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 bq = *reinterpret_cast<const float4 *>(sbias + n0 + 4 * q);
                        const uint32_t *u = r + 16 * h + 4 * q;
                        const __nv_bfloat162 lo = __floats2bfloat162_rn(__uint_as_float(u[0]) + bq.x, __uint_as_float(u[1]) + bq.y);
                        const __nv_bfloat162 hi = __floats2bfloat162_rn(__uint_as_float(u[2]) + bq.z, __uint_as_float(u[3]) + bq.w);
                        v[2 * q] = *reinterpret_cast<const uint32_t *>(&lo);
                        v[2 * q + 1] = *reinterpret_cast<const uint32_t *>(&hi);
                    }
                    st_bf16x16(y + f * ys + n0, v, wide != 0);
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kCols) : "memory");
}

template <int CIN, int COUT>
static cudaError_t launch_up_tc(int W, int H, int D, const __nv_bfloat16 *x, const __nv_bfloat16 *w,
                                const float *bias, __nv_bfloat16 *y, int ys, int *err, cudaStream_t st) {
    typedef UpShape<CIN, COUT> S;
    cudaError_t e = allow_smem((const void *)k_upconv_tc<CIN, COUT>, S::SMEM);
    if (e != cudaSuccess) return e;
    const long long tiles = ((long long)(W + 2) * H + kConvM - 1) / kConvM * D;
    const long long room = (long long)conv_sm_count() * S::kPerSm;
    k_upconv_tc<CIN, COUT><<<(unsigned)std::min(tiles, room), 128, S::SMEM, st>>>(W, H, D, x, w, bias, y, ys,
                                                                                  wide_stores(y, ys, 0), err);
    return cudaGetLastError();
}

cudaError_t launch_upconv_tc(int W, int H, int D, int cin, int cout, const __nv_bfloat16 *x,
                             const __nv_bfloat16 *w, const float *bias, __nv_bfloat16 *y, int ys, int *err,
                             cudaStream_t st) {
    if (ys % 8 != 0) return cudaErrorInvalidValue;
    if (cin == 32 && cout == 16) return launch_up_tc<32, 16>(W, H, D, x, w, bias, y, ys, err, st);
    if (cin == 64 && cout == 32) return launch_up_tc<64, 32>(W, H, D, x, w, bias, y, ys, err, st);
    if (cin == 128 && cout == 64) return launch_up_tc<128, 64>(W, H, D, x, w, bias, y, ys, err, st);
    return cudaErrorNotSupported;
}

// ---------------------------------------------------------------------------
// Data gradient of the transposed convolution on the tensor cores:
//   gx[v][ci] = (x[v][ci] > 0) * sum over (par, co) of gy[fine(v, par)][co] * W[par][co][ci],
// a GEMM of M = 128 padded coarse voxels (the tile of k_upconv_tc), K =
// 8 COUT (parity, channel) and N = CIN.  A is gy gathered at the fine voxels
// in the K-major layout of the 3x3x3 kernels ([k group][voxel][8], zero for
// halo voxels); B is the BF16 weights in the MN-major layout ([ci group]
// [k][8], k rows 16 B apart), re-laid from [8][COUT][CIN] while staging.
// The parities go in chunks of PC (all 8, or 4 for 128 -> 64, so that a
// chunk fits in shared memory), each chunk's MMAs committed to the mbarrier
// and waited on (bounded) before the next chunk is staged.  The epilogue
// masks by the forward activation and stores BF16.
// ---------------------------------------------------------------------------
template <int CIN, int COUT>
struct UpDgradShape {
    static constexpr int PC = CIN == 128 ? 4 : 8;         // parities per chunk
    static constexpr int KC = PC * COUT;                   // K per chunk
    static constexpr int ABYTES = KC * kConvM * 2;         // KC / 8 slabs of 128 voxels x 16 B
    static constexpr int BBYTES = KC * CIN * 2;
    static constexpr int SMEM = ABYTES + BBYTES;
    static_assert(SMEM <= 227 * 1024, "chunk exceeds shared memory");
    static_assert(CIN % 16 == 0 && CIN <= 256, "N = CIN must be a multiple of 16, at most 256");
};

template <int CIN, int COUT>
__global__ void __launch_bounds__(128, 1)
k_upconv_dgrad_tc(int W, int H, int D, const __nv_bfloat16 *__restrict__ gy, int gs,
                  const __nv_bfloat16 *__restrict__ w, const __nv_bfloat16 *__restrict__ act,
                  __nv_bfloat16 *__restrict__ gx, int *err) {
    using S = UpDgradShape<CIN, COUT>;
    constexpr int KC = S::KC, NG = COUT / 8;
    // kind::f16, D FP32, A and B BF16, A K-major, B MN-major
    constexpr uint32_t idesc = umma_idesc_bf16(kConvM, CIN) | (1u << 16);
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int Wp = W + 2, Hp = H + 2;
    const long long plane = (long long)Wp * Hp;
    const int z = blockIdx.y;                                              // interior coarse plane
    const long long P0 = (long long)Wp + (long long)kConvM * blockIdx.x;   // first voxel of the tile

    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base)), "r"(CIN < 32 ? 32 : CIN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&mbar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;
    const uint32_t aS = smem_u32(smem), bS = aS + (uint32_t)S::ABYTES;
    // thread tid gathers voxel P0 + tid of the tile
    const long long P = P0 + tid;
    const int yv = (int)(P / Wp), xv = (int)(P - (long long)yv * Wp);
    const bool inside = xv >= 1 && xv <= W && yv >= 1 && yv <= H;
    const long long Wf = 2LL * W + 2, Hf = 2LL * H + 2;
    bool ok = true;
    constexpr int NCH = 8 / S::PC;
#pragma unroll 1
    for (int c = 0; c < NCH && ok; ++c) {
        // A: k group kg = (parity, 8 channels) of voxel tid at aS + kg 2048 + tid 16
#pragma unroll 4
        for (int kg = 0; kg < KC / 8; ++kg) {
            const int par = c * S::PC + kg / NG, g = kg % NG;
            const uint32_t dst = aS + kg * (kConvM * 16) + tid * 16;
            if (inside) {
                const long long f = ((long long)(2 * z + (par >> 2) + 1) * Hf + (2 * (yv - 1) + ((par >> 1) & 1) + 1)) * Wf +
                                    (2 * (xv - 1) + (par & 1) + 1);
                cp_async16(dst, gy + f * gs + g * 8);
            } else {
                st_shared_zero16(dst);
            }
        }
        // B: chunk (k, ci group ng) of W row c KC + k at bS + (ng KC + k) 16
        for (int e = tid; e < KC * (CIN / 8); e += 128) {
            const int k = e / (CIN / 8), ng = e % (CIN / 8);
            cp_async16(bS + (ng * KC + k) * 16, w + (size_t)(c * KC + k) * CIN + ng * 8);
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t ad0 = umma_desc(aS, kConvM * 16, 128), bd0 = umma_desc(bS, 128, KC * 16);
#pragma unroll
            for (int s = 0; s < KC / 16; ++s) {
                const uint64_t ad = ad0 + (uint64_t)((2 * s * kConvM * 16) >> 4);
                const uint64_t bd = bd0 + (uint64_t)((s * 256) >> 4);
                const uint32_t accum = (c > 0 || s > 0) ? 1u : 0u;
                asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                             " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                             ::"r"(tmem), "l"(ad), "l"(bd), "r"(idesc), "r"(accum) : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(smem_u32(&mbar)) : "memory");
        }
        // The staged chunk is overwritten only once its MMAs completed.
        ok = __syncthreads_and(mbar_wait(smem_u32(&mbar), (uint32_t)(c & 1), err)) != 0;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok) {
        // TMEM lane tid = 32 warp + lane is this thread's own voxel P
        const long long vc = (long long)(z + 1) * plane + P;
#pragma unroll 1
        for (int n0 = 0; n0 < CIN; n0 += 16) {
            uint32_t r[16];
            const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)n0;
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                         : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                           "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
                           "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                         : "r"(taddr) : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (inside) {
                const uint4 a0 = __ldg(reinterpret_cast<const uint4 *>(act + vc * CIN + n0));
                const uint4 a1 = __ldg(reinterpret_cast<const uint4 *>(act + vc * CIN + n0) + 1);
                const __nv_bfloat16 *ah0 = reinterpret_cast<const __nv_bfloat16 *>(&a0);
                const __nv_bfloat16 *ah1 = reinterpret_cast<const __nv_bfloat16 *>(&a1);
                __nv_bfloat162 hv[8];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float a = __bfloat162float(q < 4 ? ah0[2 * q] : ah1[2 * q - 8]) > 0.0f
                                        ? __uint_as_float(r[2 * q]) : 0.0f;
                    const float b = __bfloat162float(q < 4 ? ah0[2 * q + 1] : ah1[2 * q - 7]) > 0.0f
                                        ? __uint_as_float(r[2 * q + 1]) : 0.0f;
                    hv[q] = __floats2bfloat162_rn(a, b);
                }
                uint4 *dst = reinterpret_cast<uint4 *>(gx + vc * CIN + n0);
                dst[0] = *reinterpret_cast<uint4 *>(&hv[0]);
                dst[1] = *reinterpret_cast<uint4 *>(&hv[4]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(CIN < 32 ? 32 : CIN)
                     : "memory");
}

template <int CIN, int COUT>
static cudaError_t launch_up_dgrad(int W, int H, int D, const __nv_bfloat16 *gy, int gs, const __nv_bfloat16 *w,
                                   const __nv_bfloat16 *act, __nv_bfloat16 *gx, int *err, cudaStream_t st) {
    constexpr int smem = UpDgradShape<CIN, COUT>::SMEM;
    cudaError_t e = allow_smem((const void *)k_upconv_dgrad_tc<CIN, COUT>, smem);
    if (e != cudaSuccess) return e;
    const long long interior = (long long)(W + 2) * H;
    const dim3 grid((unsigned)((interior + kConvM - 1) / kConvM), (unsigned)D);
    k_upconv_dgrad_tc<CIN, COUT><<<grid, 128, smem, st>>>(W, H, D, gy, gs, w, act, gx, err);
    return cudaGetLastError();
}

cudaError_t launch_upconv_dgrad_tc(int W, int H, int D, int cin, int cout, const __nv_bfloat16 *gy, int gs,
                                   const __nv_bfloat16 *w, const __nv_bfloat16 *act, __nv_bfloat16 *gx, int *err,
                                   cudaStream_t st) {
    if (gs % 8 != 0) return cudaErrorInvalidValue;
    if (cin == 32 && cout == 16) return launch_up_dgrad<32, 16>(W, H, D, gy, gs, w, act, gx, err, st);
    if (cin == 64 && cout == 32) return launch_up_dgrad<64, 32>(W, H, D, gy, gs, w, act, gx, err, st);
    if (cin == 128 && cout == 64) return launch_up_dgrad<128, 64>(W, H, D, gy, gs, w, act, gx, err, st);
    return cudaErrorNotSupported;
}

// ---------------------------------------------------------------------------
// Weight gradients on the tensor cores.  For the 3x3x3 convolution
//   dW[tap][co][ci] = sum over voxels P of gy[P][co] * x[P + off(tap)][ci],
// a GEMM whose reduction (K) runs over voxels.  Both tensors are channels
// last, so 8 channels of one voxel are one 16-byte row, and a block of
// voxels staged row by row is already an operand in the MN-major, no-swizzle
// layout: core matrices of 8 voxels (K) x 8 channels (M or N), 8-voxel groups
// LBO = 128 B apart, 8-channel groups SBO apart.  With K blocks of KB voxels:
//   A (M = 128): 16 eight-channel groups (r, g) of x over the 9 row offsets
//     r = (dz, dy), each a window of KB + 2 voxels staged from one voxel
//     early; tap dx reads the same window 16 * (dx + 1) bytes further on;
//   B (N = Cout): gy over the KB voxels;
//   three accumulators (dx) of Cout columns in TMEM.
// The K range is the padded voxels from the first interior row to the last;
// gy is zero on the halo, so halo voxels add nothing.  For the 2x2x2
// transposed convolution (8 parities)
//   dW[par][co][ci] = sum over coarse voxels v of gy[fine(v, par)][co] * x[v][ci]:
//   A (M = 128): 16 groups (par, co group) of gy gathered at the fine voxels
//     (zero for halo voxels), B (N = Cin): x over the KB coarse voxels.
// A CTA owns one M tile (blockIdx.y) and a run of K blocks (blockIdx.x),
// double buffered: block i + 1 is staged by cp.async before the MMAs of block
// i are issued, so its loads are in flight while they run (issuing the MMAs
// first exposes every block's load latency and measured 10 % slower).  One
// thread issues the MMAs; each buffer's commit arrives on its own mbarrier,
// waited on (bounded in time) before the buffer is restaged.  The CTA's sums
// are added to dW with FP32 atomics.
// ---------------------------------------------------------------------------
constexpr int kWgKB = 128;                 // voxels per K block; the up gather has one per thread
static_assert(kWgKB + 2 <= BLZ_CONV_SLACK, "the last K block's window must stay inside the slack");

struct WgTcArgs {
    const __nv_bfloat16 *x;
    int xs;                                // layer input (conv) / coarse input (up), channel stride
    const __nv_bfloat16 *gy;
    int gys, gyoff;                        // output gradient: channel stride, first channel
    int W, H, D;                           // dims of the K loop's level (up: the coarse one)
    long long pbeg;                        // first padded voxel of the K range
    int nkb, kb_per;                       // K blocks in all, per CTA
    float *dw;
    int *err;
};

template <int MODE, int CIN, int CO>
struct WgShape {
    static constexpr int AW = MODE == 0 ? kWgKB + 2 : kWgKB;   // staged voxels per A group
    static constexpr int GA = AW * 16;                         // bytes per A group
    static constexpr int NGA = (MODE == 0 ? CIN : CO) / 8;     // A groups per row offset / parity
    static constexpr int NGALL = (MODE == 0 ? 9 : 8) * NGA;
    static constexpr int MTILES = (NGALL + 15) / 16;
    static constexpr int N = MODE == 0 ? CO : CIN;
    static constexpr int NGB = N / 8;
    static constexpr int GB = kWgKB * 16;
    static constexpr int ABYTES = 16 * GA, BUF = ABYTES + NGB * GB;
    static constexpr int NACC = MODE == 0 ? 3 : 1;
    static constexpr int COLS = NACC * N <= 32 ? 32 : NACC * N <= 64 ? 64 : NACC * N <= 128 ? 128
                                                    : NACC * N <= 256 ? 256 : 512;
    static_assert(NACC * N <= 512, "accumulators exceed tensor memory");
    static_assert(N % 16 == 0 && N <= 256, "MN-major B needs N a multiple of 16, at most 256");
};

template <int MODE, int CIN, int CO>
__global__ void __launch_bounds__(128, 1) k_wgrad_tc(WgTcArgs a) {
    using S = WgShape<MODE, CIN, CO>;
    constexpr int KB = kWgKB, N = S::N, NGA = S::NGA;
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t mbar[2];
    __shared__ uint32_t tmem_base;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int mt = blockIdx.y;
    const long long Wp = a.W + 2, Hp = a.H + 2, plane = Wp * Hp;
    const int kb0 = blockIdx.x * a.kb_per;
    const int nk = min(a.kb_per, a.nkb - kb0);
    const uint32_t s0 = smem_u32(smem);
    const uint32_t mb0 = smem_u32(&mbar[0]);
    auto mb = [&](int b) { return mb0 + 8u * (uint32_t)b; };

    // A groups that hold no row (conv tiles past the 9th row offset) stay zero.
    for (int e = tid; e < 2 * S::BUF / 16; e += 128) st_shared_zero16(s0 + e * 16);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_u32(&tmem_base)), "r"(S::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb(0)) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb(1)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_base;

    auto stage = [&](int kb, int buf) {
        const uint32_t sa = s0 + buf * S::BUF, sb = sa + S::ABYTES;
        const long long P0 = a.pbeg + (long long)kb * KB;
        if constexpr (MODE == 0) {
            // local row offset lr holds groups lr * NGA .. lr * NGA + NGA - 1;
            // element e of its window is voxel e / NGA, group e % NGA
            constexpr int NR = 16 / NGA, PER = S::AW * NGA;
#pragma unroll
            for (int lr = 0; lr < NR; ++lr) {
                const int r = mt * NR + lr;
                if (r >= 9) break;
                const __nv_bfloat16 *src =
                    a.x + (P0 - 1 + (long long)(r / 3 - 1) * plane + (long long)(r % 3 - 1) * Wp) * a.xs;
                for (int e = tid; e < PER; e += 128) {
                    const int v = e / NGA, g = e & (NGA - 1);
                    cp_async16(sa + (lr * NGA + g) * S::GA + v * 16, src + v * a.xs + g * 8);
                }
            }
            const __nv_bfloat16 *gb = a.gy + P0 * a.gys + a.gyoff;
            for (int e = tid; e < S::NGB * KB; e += 128) {
                const int g = e & (S::NGB - 1), v = e / S::NGB;
                cp_async16(sb + g * S::GB + v * 16, gb + v * a.gys + g * 8);
            }
        } else {
            // thread tid gathers coarse voxel P0 + tid's 16 groups
            const long long P = P0 + tid;
            const long long zc = P / plane, rem = P - zc * plane;
            const long long yc = rem / Wp, xc = rem - yc * Wp;
            const bool inside = zc >= 1 && zc <= a.D && yc >= 1 && yc <= a.H && xc >= 1 && xc <= a.W;
            const long long Wf = 2LL * a.W + 2, Hf = 2LL * a.H + 2;
#pragma unroll 4
            for (int lg = 0; lg < 16; ++lg) {
                const int grp = mt * 16 + lg, par = grp / NGA, g = grp % NGA;
                const uint32_t dst = sa + lg * S::GA + tid * 16;
                if (inside) {
                    const long long f = ((2 * zc - 1 + (par >> 2)) * Hf + (2 * yc - 1 + ((par >> 1) & 1))) * Wf +
                                        (2 * xc - 1 + (par & 1));
                    cp_async16(dst, a.gy + f * a.gys + a.gyoff + g * 8);
                } else {
                    st_shared_zero16(dst);
                }
            }
            for (int e = tid; e < S::NGB * KB; e += 128) {
                const int g = e % S::NGB, v = e / S::NGB;
                cp_async16(sb + g * S::GB + v * 16, a.x + (P0 + v) * a.xs + g * 8);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    // kind::f16, D FP32, A and B BF16, both MN-major
    constexpr uint32_t idesc = umma_idesc_bf16(128, N) | (1u << 15) | (1u << 16);
    bool ok = true;
    int issued = 0;                                      // MMA batches committed
    if (nk > 0) stage(kb0, 0);
    for (int i = 0; i < nk; ++i) {
        const int buf = i & 1;
        if (i + 1 < nk) {
            // buffer buf ^ 1 was last read by the MMAs of block i - 1
            if (i >= 1) ok = __syncthreads_and(mbar_wait(mb(buf ^ 1), ((i - 1) >> 1) & 1, a.err)) != 0;
            if (!ok) break;
            stage(kb0 + i + 1, buf ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t sa = s0 + buf * S::BUF, sb = sa + S::ABYTES;
            const uint64_t ad0 = umma_desc(sa, 128, S::GA), bd0 = umma_desc(sb, 128, S::GB);
#pragma unroll
            for (int kk = 0; kk < KB / 16; ++kk) {
                const uint64_t bd = bd0 + (uint64_t)((kk * 256) >> 4);
#pragma unroll
                for (int d = 0; d < S::NACC; ++d) {
                    const uint64_t ad = ad0 + (uint64_t)((kk * 256 + (MODE == 0 ? d * 16 : 0)) >> 4);
                    const uint32_t acc = (i > 0 || kk > 0) ? 1u : 0u;
                    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                                 " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                                 ::"r"(tmem + (uint32_t)(d * N)), "l"(ad), "l"(bd), "r"(idesc), "r"(acc)
                                 : "memory");
                }
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(mb(buf)) : "memory");
        }
        ++issued;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // The last commit completes after every MMA issued before it.
    if (issued > 0)
        ok = __syncthreads_and(mbar_wait(mb((issued - 1) & 1), ((issued - 1) >> 1) & 1, a.err) && ok) != 0;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok && issued == nk && nk > 0) {
        // TMEM lane m = A row: group m / 8, channel m % 8 of it.
        const int m = 32 * warp + lane, grp = mt * 16 + (m >> 3), c8 = m & 7;
        const bool valid = grp < S::NGALL;
        const int hi = grp / NGA, ch = (grp % NGA) * 8 + c8;   // conv: (row offset, ci); up: (parity, co)
#pragma unroll 1
        for (int d = 0; d < S::NACC; ++d) {
#pragma unroll 1
            for (int n0 = 0; n0 < N; n0 += 16) {
                uint32_t r[16];
                const uint32_t taddr = tmem + ((uint32_t)(32 * warp) << 16) + (uint32_t)(d * N + n0);
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                             : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                               "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]),
                               "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                             : "r"(taddr) : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (valid) {
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        const int n = n0 + q;
                        const size_t o = MODE == 0 ? ((size_t)(3 * hi + d) * CO + n) * CIN + ch
                                                   : ((size_t)hi * CO + ch) * CIN + n;
                        atomicAdd(a.dw + o, __uint_as_float(r[q]));
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(S::COLS) : "memory");
}

template <int MODE, int CIN, int CO>
static cudaError_t launch_wg_tc(WgTcArgs a, cudaStream_t st) {
    using S = WgShape<MODE, CIN, CO>;
    constexpr int smem = 2 * S::BUF;
    cudaError_t e = allow_smem((const void *)k_wgrad_tc<MODE, CIN, CO>, smem);
    if (e != cudaSuccess) return e;
    const long long Wp = a.W + 2, plane = Wp * (a.H + 2);
    a.pbeg = plane + Wp;                                  // first interior row
    const long long pend = (long long)(a.D + 1) * plane - Wp;   // past the last interior row
    const long long nkb = (pend - a.pbeg + kWgKB - 1) / kWgKB;
    if (nkb >= (1LL << 30)) return cudaErrorInvalidValue;
    // about two CTAs per SM, at least four K blocks each
    const long long want = (2 * 148 + S::MTILES - 1) / S::MTILES;
    long long per = (nkb + want - 1) / want;
    if (per < 4) per = 4;
    a.nkb = (int)nkb;
    a.kb_per = (int)per;
    const dim3 grid((unsigned)((nkb + per - 1) / per), (unsigned)S::MTILES);
    k_wgrad_tc<MODE, CIN, CO><<<grid, 128, smem, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_wgrad_tc(int up, int W, int H, int D, int cin, int cout, const __nv_bfloat16 *x, int xs,
                            const __nv_bfloat16 *gy, int gys, int gyoff, float *dw, int *err, cudaStream_t st) {
    if (xs % 8 != 0 || gys % 8 != 0 || gyoff % 8 != 0) return cudaErrorInvalidValue;
    WgTcArgs a{x, xs, gy, gys, gyoff, W, H, D, 0, 0, 0, dw, err};
    if (up) {
        if (cin == 32 && cout == 16) return launch_wg_tc<1, 32, 16>(a, st);
        if (cin == 64 && cout == 32) return launch_wg_tc<1, 64, 32>(a, st);
        if (cin == 128 && cout == 64) return launch_wg_tc<1, 128, 64>(a, st);
        return cudaErrorNotSupported;
    }
#define BLZ_WG(ci, co) if (cin == ci && cout == co) return launch_wg_tc<0, ci, co>(a, st)
    BLZ_WG(16, 16); BLZ_WG(16, 32); BLZ_WG(32, 16); BLZ_WG(32, 32); BLZ_WG(32, 64);
    BLZ_WG(64, 32); BLZ_WG(64, 64); BLZ_WG(64, 128); BLZ_WG(128, 64); BLZ_WG(128, 128);
#undef BLZ_WG
    return cudaErrorNotSupported;
}

} // namespace blz

namespace {
__device__ int g_conv_timeout;          // set by a convolution whose MMA wait gave up
}

extern "C" int blz_conv3d(const blz_conv_desc *d, const void *x, const void *w, const float *bias, void *y,
                          void *cuda_stream) {
    using namespace blz;
    if (!d || !x || !w || !bias || !y) return BLZ_ERR_ARG;
    if (d->W < 1 || d->H < 1 || d->D < 1 || d->cin <= 0 || d->cin % 16 ||
        (d->cout != 16 && d->cout != 32 && d->cout != 64 && d->cout != 128)) {
        set_thread_error("blz_conv3d: need cin % 16 == 0 and cout in {16, 32, 64, 128}");
        return BLZ_ERR_ARG;
    }
    int *flag = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void **)&flag, g_conv_timeout);
    if (e == cudaSuccess) e = cudaMemsetAsync(flag, 0, sizeof(int), (cudaStream_t)cuda_stream);
    const ConvDesc cd{d->W, d->H, d->D, d->cin, d->cout, d->relu, d->out_f32, d->cout, 0};
    if (e == cudaSuccess)
        e = launch_conv3d(cd, static_cast<const __nv_bfloat16 *>(x), static_cast<const __nv_bfloat16 *>(w), bias, y,
                          flag, (cudaStream_t)cuda_stream);
    int timeout = 0;
    if (e == cudaSuccess) e = cudaMemcpyAsync(&timeout, flag, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)cuda_stream);
    if (e == cudaSuccess) e = cudaStreamSynchronize((cudaStream_t)cuda_stream);
    if (e != cudaSuccess) {
        set_thread_error(cudaGetErrorString(e));
        return BLZ_ERR_CUDA;
    }
    if (timeout) {
        set_thread_error("blz_conv3d: tensor-core completion wait timed out");
        return BLZ_ERR_TIMEOUT;
    }
    return BLZ_OK;
}
