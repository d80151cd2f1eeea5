// Far-history contraction on the 5th-generation tensor cores (tcgen05), split precision.
//
// For a block of BN upcoming steps starting at n0, the history older than the block enters
// every step of the block through a dense product
//     C[i][j] = sum_{t < n0} A[i][t] * W[t][j],   A[i][t] = D_t[i] (node i, increment t),
//                                                  W[t][j] = w[n0 + j - t] (Toeplitz weights),
// M = nodes, N = BN = 64 steps, K = n0. This is the reference's mode-1 far-history tile
// product (fr_do.cpp:173-235, wmma 16x16x16 half/float), rebuilt for sm_103a:
//   * A and W are stored as 16-bit hi/lo pairs (fp16 with power-of-two scaling, or bf16);
//     three products A_hi W_hi + A_hi W_lo + A_lo W_hi run as kind::f16 MMAs
//     (M=128, N=64, K=16) accumulating in FP32 in TMEM;
//   * every 256 history columns the TMEM accumulator is folded into float-float (hi, lo)
//     registers by the epilogue warps while the MMA warp fills the other TMEM buffer; the
//     CTA's result is written as FP64 partial sums C[split][j][row];
//   * operands arrive by TMA (cp.async.bulk.tensor, 128-byte swizzle) into a 4-stage ring
//     guarded by mbarriers; no multicast.
// Warp roles (192 threads): warp 0 TMA producer, warp 1 TMEM allocator + MMA issuer,
// warps 2-5 epilogue (TMEM lane quadrant = warp % 4).
// Every wait is bounded (2 s of %globaltimer); on timeout the kernel raises
// DEVERR_MBAR_TIMEOUT, stops issuing, drains its own copies (bounded) and frees its TMEM.
#include <algorithm>
#include <cuda.h>
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernels.cuh"
#include "tc_far.cuh"

namespace fpde {
namespace tc {

constexpr int BM = 128, BN = 64, BK = 64;
constexpr int STAGES = 4;
constexpr int CHUNK_KT = 4;                          // k-tiles per TMEM accumulation chunk
constexpr int A_BYTES = BM * BK * 2;                 // 16 KB
constexpr int W_BYTES = BN * BK * 2;                 // 8 KB
constexpr int STAGE_BYTES = 2 * A_BYTES + 2 * W_BYTES;
constexpr int TMEM_COLS = 128;                       // two 64-column fp32 accumulators
constexpr int THREADS = 192;
constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + 256;
constexpr unsigned long long WAIT_NS = 2000000000ull;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long gtimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait on the phase with the given parity. After a timeout (abort_s) no wait of the CTA waits again. The
// epilogue warps go on with whatever they read, since TMEM loads, shuffles and votes take a warp as a whole and
// a lane that left alone would keep the others waiting; one vote on abort_s per item drops their results.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, unsigned *flags, volatile int *abort_s)
{
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = gtimer();
    while (true) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort_s) return false;
        if (gtimer() - t0 > WAIT_NS) {
            atomicOr(flags, DEVERR_MBAR_TIMEOUT);
            *abort_s = 1;
            return false;
        }
    }
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *tm, int x, int y, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(smem_u32(dst)), "l"((uint64_t)tm), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// K-major operand tile, 128-byte swizzle: rows of 128 B, 8-row atoms of 1024 B (SBO).
__device__ __forceinline__ uint64_t sdesc_sw128(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);        // start address
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused for SW128 K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                // stride byte offset: 8 rows x 128 B
    d |= (uint64_t)1 << 46;                          // descriptor version (tcgen05)
    d |= (uint64_t)2 << 61;                          // SWIZZLE_128B
    return d;
}

// Instruction descriptor, kind::f16: D f32, A/B fp16 (0) or bf16 (1), both K-major.
__host__ __device__ constexpr uint32_t idesc_f16(int bf16, int M, int N)
{
    return (1u << 4) | ((uint32_t)bf16 << 7) | ((uint32_t)bf16 << 10) | ((uint32_t)(N >> 3) << 17) |
           ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma(uint32_t dtm, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
        ::"r"(dtm), "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
}
// Same MMA with both smem descriptors given as (low, high) 32-bit words: the high words are
// constant and the low words differ from a stage's base only by the operand offset >> 4 (the
// 14-bit start-address field cannot carry: shared memory ends below 256 KB), so the issuing
// thread forms each descriptor with one integer add.
__device__ __forceinline__ void umma_lo(uint32_t dtm, uint32_t alo, uint32_t blo, uint32_t dhi, uint32_t idesc,
                                        uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .b64 da, db;\n\t.reg .pred p;\n\t"
        "mov.b64 da, {%1, %3};\n\t"
        "mov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %4, p;\n\t}\n"
        ::"r"(dtm), "r"(alo), "r"(blo), "r"(dhi), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void umma_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v)
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *v)
{
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __uint_as_float(r[k]);
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// Four floats from shared memory, not moved ahead of other volatile operations.
__device__ __forceinline__ float4 lds4(const float *p)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(smem_u32(p)));
    return v;
}
// After the wait: no use of the loaded values is scheduled before it.
template <int N>
__device__ __forceinline__ void tmem_loaded(float *v)
{
#pragma unroll
    for (int k = 0; k < N; ++k) asm volatile("" : "+f"(v[k]));
}

struct __align__(64) FarMaps {
    CUtensorMap a_hi, a_lo, w_hi, w_lo;
};

// grid = (row tiles, K splits); split y covers k-tiles [y*kt_per, min((y+1)*kt_per, kt_total)).
__global__ void __launch_bounds__(THREADS, 1)
    k_far_tc(const __grid_constant__ FarMaps maps, double *__restrict__ C, int64_t ldc_split, int64_t ldc_col,
             int64_t rows, int kt_total, int kt_per, uint32_t idesc, double out_scale,
             const double *__restrict__ out_scale_ptr, unsigned *flags)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *stage_base = smem;
    uint64_t *bars = (uint64_t *)(smem + STAGES * STAGE_BYTES);
    uint64_t *full = bars, *empty = bars + STAGES, *tfull = bars + 2 * STAGES, *tempty = bars + 2 * STAGES + 2;
    uint64_t *mma_done = bars + 2 * STAGES + 4;
    volatile uint32_t *tmem_slot = (volatile uint32_t *)(bars + 2 * STAGES + 5);
    volatile int *abort_s = (volatile int *)(bars + 2 * STAGES + 6);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = blockIdx.x, split = blockIdx.y;
    const int kt0 = split * kt_per;
    const int kt1 = min(kt0 + kt_per, kt_total);
    const int nkt = max(0, kt1 - kt0);
    const int nchunks = (nkt + CHUNK_KT - 1) / CHUNK_KT;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], 128); }
        mbar_init(mma_done, 1);
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void *)tmem_slot)),
                     "r"(TMEM_COLS));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 0) {
        // ------------------------------------------------ TMA producer
        if (lane == 0) {
            int issued = 0;
            for (int it = 0; it < nkt; ++it) {
                const int s = it % STAGES;
                const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                if (!mbar_wait(&empty[s], ph ^ 1u, flags, abort_s)) break;
                uint8_t *st = stage_base + s * STAGE_BYTES;
                mbar_expect_tx(&full[s], STAGE_BYTES);
                const int x = (kt0 + it) * BK, y = mt * BM;
                tma_load_2d(st, &maps.a_hi, x, y, &full[s]);
                tma_load_2d(st + A_BYTES, &maps.a_lo, x, y, &full[s]);
                tma_load_2d(st + 2 * A_BYTES, &maps.w_hi, x, 0, &full[s]);
                tma_load_2d(st + 2 * A_BYTES + W_BYTES, &maps.w_lo, x, 0, &full[s]);
                ++issued;
            }
            // Drain: every issued stage's copy must land before the CTA exits.
            for (int it = (issued > STAGES ? issued - STAGES : 0); it < issued; ++it) {
                const int s = it % STAGES;
                const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                unsigned long long t0 = gtimer();
                while (!mbar_try_wait(&full[s], ph) && gtimer() - t0 < WAIT_NS) {}
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        if (lane == 0) {
            int it = 0;
            for (int c = 0; c < nchunks && !*abort_s; ++c) {
                const int buf = c & 1;
                const uint32_t use = (uint32_t)(c >> 1);
                if (!mbar_wait(&tempty[buf], (use & 1u) ^ 1u, flags, abort_s)) break;
                tc_fence_after();
                const uint32_t dtm = tmem + (uint32_t)(buf * BN);
                const int kend = min(nkt, (c + 1) * CHUNK_KT);
                bool ok = true;
                for (int first = 1; it < kend; ++it, first = 0) {
                    const int s = it % STAGES;
                    const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                    if (!mbar_wait(&full[s], ph, flags, abort_s)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t st = smem_u32(stage_base + s * STAGE_BYTES);
                    const uint32_t a_hi = st, a_lo = st + A_BYTES, w_hi = st + 2 * A_BYTES,
                                   w_lo = st + 2 * A_BYTES + W_BYTES;
#pragma unroll
                    for (int k = 0; k < BK / 16; ++k) {
                        const uint32_t off = (uint32_t)(k * 32);     // 16 elements x 2 B along K
                        const uint32_t acc = (first && k == 0) ? 0u : 1u;
                        umma(dtm, sdesc_sw128(a_hi + off), sdesc_sw128(w_hi + off), idesc, acc);
                        umma(dtm, sdesc_sw128(a_hi + off), sdesc_sw128(w_lo + off), idesc, 1u);
                        umma(dtm, sdesc_sw128(a_lo + off), sdesc_sw128(w_hi + off), idesc, 1u);
                    }
                    umma_commit(&empty[s]);                 // frees the stage when these MMAs finish
                }
                if (!ok) break;
                umma_commit(&tfull[buf]);                   // chunk accumulator ready
            }
            // Every MMA of this CTA must have finished before its TMEM is released.
            umma_commit(mma_done);
            const unsigned long long t0 = gtimer();
            while (!mbar_try_wait(mma_done, 0) && gtimer() - t0 < WAIT_NS) {}
        }
    } else {
        // ------------------------------------------------ epilogue (warps 2..5)
        const int q = warp & 3;                            // TMEM lane quadrant of this warp
        const int64_t row = (int64_t)mt * BM + q * 32 + lane;
        float hi[BN], lo[BN];
#pragma unroll
        for (int j = 0; j < BN; ++j) { hi[j] = 0.f; lo[j] = 0.f; }
        for (int c = 0; c < nchunks; ++c) {
            const int buf = c & 1;
            const uint32_t use = (uint32_t)(c >> 1);
            mbar_wait(&tfull[buf], use & 1u, flags, abort_s);
            tc_fence_after();
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * BN);
            float v[BN];
            tmem_ld16(taddr + 0, v);
            tmem_ld16(taddr + 16, v + 16);
            tmem_ld16(taddr + 32, v + 32);
            tmem_ld16(taddr + 48, v + 48);
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive(&tempty[buf]);
#pragma unroll
            for (int j = 0; j < BN; ++j) {                 // float-float accumulation (TwoSum)
                const float s = hi[j] + v[j];
                const float bb = s - hi[j];
                const float e = (hi[j] - (s - bb)) + (v[j] - bb);
                hi[j] = s;
                lo[j] += e;
            }
        }
        if (*abort_s == 0 && row < rows && nchunks > 0) {
            if (out_scale_ptr) out_scale *= *out_scale_ptr;
            double *out = C + (int64_t)split * ldc_split + row;
#pragma unroll
            for (int j = 0; j < BN; ++j) out[(int64_t)j * ldc_col] = ((double)hi[j] + (double)lo[j]) * out_scale;
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
    }
}

// ------------------------------------------------------------------------------------
// Exact-slice variant (three bf16 slices per operand).
// A[i][t] = (a0 + a1' + a2') * 2^pA[i][kt], W[j][t] = (w0 + w1' + w2') * 2^pW[j][kt] with
// a0, w0 integers of at most 8 bits and a1' = a1 2^-8, a2' = a2 2^-16 (a1, a2 integers of
// at most 8 bits), per node (or step) and 64-column k-tile. Per k-tile the products
//   X0  = sum a0 w0                                  (integers < 2^16, 64 of them < 2^22:
//                                                    exact in the FP32 accumulator)
//   X12 = sum a0 w1' + a1' w0 + a0 w2' + a1' w1' + a2' w0     (2^-8 below X0)
// go to two TMEM accumulators; the epilogue scales both by 2^(pA+pW) every k-tile and folds them
// into a float-float pair (hi, lo): X0 by an error-free TwoSum into hi, X12 (2^-8 of X0) added
// into lo together with that sum's rounding error. The leading product is therefore free of
// accumulation error, whatever the rounding of the tensor core's FP32 adder, and the FP32
// rounding of lo stays near 2^-31 of the partial per k-tile.
// What bounds it: the fold. A 128 x 128 k-tile (NG = 2) takes 24 MMAs of 64 cycles and 2,300 cycles of
// shared memory, the fold of its two accumulators 3,000 (nine packed operations per column pair and 128 KB
// out of TMEM); loads and MMAs hide behind it. One column at a time, its scale by a shuffle, in 168
// registers it took 4,300. 16 epilogue warps of 32 columns were slower (3,250). At 65,536 rows, 256 steps
// and 2,560 columns a launch takes 459 us (625 before).
constexpr int THREADS3 = 64 + 8 * 32;                         // TMA warp, MMA warp, 8 epilogue warps

// Shape of the three-slice kernel for NG weight groups (64 steps each) per item: one MMA of
// N = 64 NG columns reads the item's history tile once for all NG groups, so the shared-memory
// traffic per group (TMA writes + MMA operand reads) falls with NG.
template <int NG>
struct Far3Cfg {
    static constexpr int N = BN * NG;                         // MMA N: steps per item
    static constexpr int WB = N * BK * 2;                     // one weight slice of a stage
    static constexpr int STAGE = 3 * A_BYTES + 3 * WB;        // 72 KB (NG 1), 96 KB (NG 2)
    static constexpr int STAGES = NG == 1 ? 3 : 2;
    static constexpr int TMEM = 4 * N;                        // 2 buffers x (X0, X12)
    static constexpr int COLS = N / 2;                        // columns per epilogue warp
    static constexpr int CH = 16;                             // columns per TMEM read batch
    static constexpr int EW = 8;                              // epilogue warps
    // A warpgroup for TMA and MMA, the others for the epilogue. At NG = 2 the epilogue takes the registers
    // that the first warpgroup gives back (the shares add up to what the block is launched with).
    static constexpr int THREADS = 128 + 32 * EW;
    static constexpr int REGS = 168, REGS_ISSUE = 40, REGS_FOLD = 232;   // NG = 2
    static_assert(NG != 2 || (128 * REGS_ISSUE + 32 * EW * REGS_FOLD <= THREADS * REGS && THREADS * REGS <= 65536),
                  "register shares");
    static constexpr int SCALES = EW * 2 * COLS * 4;          // per epilogue warp: two k-tiles' column scales
    static constexpr int SMEM = 1024 + STAGES * STAGE + SCALES + 256;
};

// Where a k-tile's boxes and scales are: row-major slices ([rows][ld], scales [rows][ldp]) or tile-major
// ones ([k-tile][rows][64], scales [k-tile][rows]), in which a box is one contiguous 16 KB.
struct Far3Layout {
    int x_kt, ya_kt, yw_kt;                                   // box coordinates per k-tile
    int64_t pa_row, pa_kt, pw_row, pw_kt;                     // strides of the scales
};

struct __align__(64) FarMaps3 {
    CUtensorMap a[3], w[3], w2[3];                            // w: 64-row weight boxes, w2: 128-row
};

// 2^e as a float for e in [-127, 127], from the bits (exact; e = -127 is the subnormal 2^-127).
__device__ __forceinline__ float pow2f(int e)
{
    return e >= -126 ? __int_as_float((e + 127) << 23) : __int_as_float(0x00400000);
}

// Two floats in one 64-bit register, one instruction per operation on both: the folds of the accumulators
// are bound by issue slots and by the latency of their dependent operations, not by the FP32 lanes.
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float x, float y)
{
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 unpack2(f32x2 v)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b)
{
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c)
{
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// a - b: exactly one multiply-add (a packed subtract costs two more instructions for the signs).
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) { return fma2(b, 0xBF800000BF800000ull, a); }
// a += b, returns the rounding error (TwoSum); and with b = v sc exactly (sc a power of two).
__device__ __forceinline__ f32x2 two_sum2(f32x2 &a, f32x2 b)
{
    const f32x2 s = add2(a, b), nb = sub2(a, s);        // -(what of b went into s)
    const f32x2 e = add2(sub2(a, add2(s, nb)), add2(b, nb));
    a = s;
    return e;
}
__device__ __forceinline__ f32x2 two_sum2(f32x2 &a, f32x2 v, f32x2 sc)
{
    const f32x2 s = fma2(v, sc, a), nb = sub2(a, s);
    const f32x2 e = add2(sub2(a, add2(s, nb)), fma2(v, sc, nb));
    a = s;
    return e;
}

// Persistent: gridDim.x CTAs (at most one per SM) walk the items (128-row tile mt, k-split ks,
// weight-group set gi of NG groups) = blockIdx.x, blockIdx.x + gridDim.x, ...; the TMA producer,
// the MMA issuer and the epilogue follow the same static sequence of k-tiles, so the pipeline runs
// on across item boundaries and TMEM is allocated once. Every item writes its partial (zeros if
// its k range is empty).
template <int NG>
__global__ void __launch_bounds__(Far3Cfg<NG>::THREADS, 1)
    k_far_tc3(const __grid_constant__ FarMaps3 maps, double *__restrict__ C, int64_t ldc_split, int64_t ldc_col,
              int64_t rows, int kt_begin, int kt_total, int kt_per, int n_split, uint32_t idesc,
              const int8_t *__restrict__ pA, const float *__restrict__ pW, const Far3Layout ly,
              const int *__restrict__ wcol, int n_sets, int grp0, int64_t ldc_grp, unsigned *flags)
{
    using Cfg = Far3Cfg<NG>;
    constexpr int STAGES = Cfg::STAGES, STAGE_BYTES3 = Cfg::STAGE, N = Cfg::N, COLS = Cfg::COLS, CH = Cfg::CH;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *stage_base = smem;
    float *scales = (float *)(smem + STAGES * STAGE_BYTES3);
    uint64_t *bars = (uint64_t *)(smem + STAGES * STAGE_BYTES3 + Cfg::SCALES);
    uint64_t *full = bars, *empty = bars + STAGES, *tfull = bars + 2 * STAGES, *tempty = bars + 2 * STAGES + 2;
    uint64_t *mma_done = bars + 2 * STAGES + 4;
    volatile uint32_t *tmem_slot = (volatile uint32_t *)(bars + 2 * STAGES + 5);
    volatile int *abort_s = (volatile int *)(bars + 2 * STAGES + 6);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_mt = (int)(rows / BM);
    const int n_items = n_mt * n_split * n_sets;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], 32 * Cfg::EW); }
        mbar_init(mma_done, 1);
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void *)tmem_slot)),
                     "r"(Cfg::TMEM));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp < 4) {
        if constexpr (NG == 2) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::REGS_ISSUE));
        if (warp == 0) {
            if (lane == 0) {                                   // TMA producer
                const CUtensorMap *wm = NG == 1 ? maps.w : maps.w2;
                int g = 0;
                bool ok = true;
                for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                    const int gi = item % n_sets, mk = item / n_sets;
                    const int mt = mk / n_split, ks = mk % n_split;
                    const int kt0 = kt_begin + ks * kt_per, kt1 = min(kt0 + kt_per, kt_total);
                    for (int kt = kt0; kt < kt1; ++kt, ++g) {
                        const int s = g % STAGES;
                        const uint32_t ph = (uint32_t)(g / STAGES) & 1u;
                        if (!mbar_wait(&empty[s], ph ^ 1u, flags, abort_s)) { ok = false; break; }
                        uint8_t *st = stage_base + s * STAGE_BYTES3;
                        mbar_expect_tx(&full[s], STAGE_BYTES3);
                        const int x = kt * ly.x_kt, y = kt * ly.ya_kt + mt * BM;
                        const int yw = kt * ly.yw_kt + ((wcol ? wcol[mt] : 0) + grp0 + NG * gi) * BN;
#pragma unroll
                        for (int q = 0; q < 3; ++q) tma_load_2d(st + q * A_BYTES, &maps.a[q], x, y, &full[s]);
#pragma unroll
                        for (int q = 0; q < 3; ++q) tma_load_2d(st + 3 * A_BYTES + q * Cfg::WB, &wm[q], x, yw, &full[s]);
                    }
                }
                for (int it = (g > STAGES ? g - STAGES : 0); it < g; ++it) {   // own copies in flight
                    const int s = it % STAGES;
                    const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
                    unsigned long long t0 = gtimer();
                    while (!mbar_try_wait(&full[s], ph) && gtimer() - t0 < WAIT_NS) {}
                }
            }
        } else if (warp == 1) {
            if (lane == 0) {                                   // MMA issuer: one k-tile per chunk
                int g = 0;
                bool ok = true;
                for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                    const int ks = (item / n_sets) % n_split;
                    const int kt0 = kt_begin + ks * kt_per, kt1 = min(kt0 + kt_per, kt_total);
                    for (int kt = kt0; kt < kt1 && !*abort_s; ++kt, ++g) {
                        const int buf = g & 1;
                        const uint32_t use = (uint32_t)(g >> 1);
                        if (!mbar_wait(&tempty[buf], (use & 1u) ^ 1u, flags, abort_s)) { ok = false; break; }
                        tc_fence_after();
                        const int s = g % STAGES;
                        const uint32_t ph = (uint32_t)(g / STAGES) & 1u;
                        if (!mbar_wait(&full[s], ph, flags, abort_s)) { ok = false; break; }
                        tc_fence_after();
                        const uint32_t x0 = tmem + (uint32_t)(buf * 2 * N), x12 = x0 + N;
                        const uint64_t dst = sdesc_sw128(smem_u32(stage_base + s * STAGE_BYTES3));
                        const uint32_t dlo = (uint32_t)dst, dhi = (uint32_t)(dst >> 32);
                        constexpr uint32_t A1 = A_BYTES >> 4, A2 = 2 * A_BYTES >> 4;
                        constexpr uint32_t W0 = 3 * A_BYTES >> 4, W1 = W0 + (Cfg::WB >> 4), W2 = W0 + (2 * Cfg::WB >> 4);
#pragma unroll
                        for (int k = 0; k < BK / 16; ++k) {
                            const uint32_t o = dlo + (uint32_t)(k * 2);      // +32 bytes per K=16 step
                            const uint32_t acc = k ? 1u : 0u;
                            umma_lo(x0, o, o + W0, dhi, idesc, acc);
                            umma_lo(x12, o, o + W1, dhi, idesc, acc);
                            umma_lo(x12, o + A1, o + W0, dhi, idesc, 1u);
                            umma_lo(x12, o, o + W2, dhi, idesc, 1u);
                            umma_lo(x12, o + A1, o + W1, dhi, idesc, 1u);
                            umma_lo(x12, o + A2, o + W0, dhi, idesc, 1u);
                        }
                        umma_commit(&empty[s]);
                        umma_commit(&tfull[buf]);
                    }
                }
                umma_commit(mma_done);
                const unsigned long long t0 = gtimer();
                while (!mbar_try_wait(mma_done, 0) && gtimer() - t0 < WAIT_NS) {}
            }
        }
    } else {
        if constexpr (NG == 2) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::REGS_FOLD));
        // epilogue warps: warp w reads TMEM lane quadrant w % 4 (the hardware's rule) and
        // folds columns [c0, c0 + COLS) with c0 = COLS * (w / 4 - 1)
        const int q = warp & 3;
        const int c0 = COLS * ((warp >> 2) - 1);
        int g = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            const int gi = item % n_sets, mk = item / n_sets;
            const int mt = mk / n_split, ks = mk % n_split;
            const int kt0 = kt_begin + ks * kt_per, kt1 = min(kt0 + kt_per, kt_total);
            const int64_t row = (int64_t)mt * BM + q * 32 + lane;
            const int64_t row_c = row < rows ? row : rows - 1;
            // this lane's row exponents and its columns' (c0 + 32u + lane) weight-tile scales; the
            // next k-tile's set is loaded while the current one is folded (both miss L1 often:
            // shared memory takes most of it); the column scales go through the warp's two rows of
            // shared memory, from where each four reach all lanes with one load
            constexpr int NU = COLS / 32;
            float *wrow = scales + (warp - 4) * (2 * COLS);
            const int8_t *pAr = pA + row_c * ly.pa_row;
            const float *pWl = pW + ((int64_t)((wcol ? wcol[mt] : 0) + grp0 + NG * gi) * BN + c0 + lane) * ly.pw_row;
            int e_nx = kt0 < kt1 ? (int)pAr[kt0 * ly.pa_kt] : 0;
            float w_nx[NU];
#pragma unroll
            for (int u = 0; u < NU; ++u) w_nx[u] = kt0 < kt1 ? __ldg(pWl + 32 * u * ly.pw_row + kt0 * ly.pw_kt) : 0.f;
            f32x2 hi[COLS / 2], lo[COLS / 2];             // columns 2j, 2j + 1
#pragma unroll
            for (int j = 0; j < COLS / 2; ++j) hi[j] = lo[j] = 0ull;
            for (int kt = kt0; kt < kt1; ++kt, ++g) {
                const int buf = g & 1;
                const uint32_t use = (uint32_t)(g >> 1);
                const int e_cur = e_nx;
                float *wcur = wrow + buf * COLS;          // last read two k-tiles ago
#pragma unroll
                for (int u = 0; u < NU; ++u) wcur[32 * u + lane] = w_nx[u];
                __syncwarp();
                if (kt + 1 < kt1) {
                    e_nx = (int)pAr[(kt + 1) * ly.pa_kt];
#pragma unroll
                    for (int u = 0; u < NU; ++u) w_nx[u] = __ldg(pWl + 32 * u * ly.pw_row + (kt + 1) * ly.pw_kt);
                }
                mbar_wait(&tfull[buf], use & 1u, flags, abort_s);
                tc_fence_after();
                // 2^pA * 2^pW: a product of powers of two, exact while it stays normal
                const float sa1 = pow2f(e_cur);
                const f32x2 sa = pack2(sa1, sa1);
                const uint32_t tb = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * 2 * N + c0);
                // batches of CH columns of both accumulators, the next one in flight while one is folded
                constexpr int NB = COLS / CH;
                float v0[2][CH], v1[2][CH];
                tmem_ld16(tb, v0[0]);
                tmem_ld16(tb + N, v1[0]);
#pragma unroll
                for (int h = 0; h < NB; ++h) {
                    float *x0 = v0[h & 1], *x12 = v1[h & 1];
                    tmem_ld_wait();
                    tmem_loaded<CH>(x0);
                    tmem_loaded<CH>(x12);
                    if (h + 1 < NB) {
                        tmem_ld16(tb + CH * (h + 1), v0[(h + 1) & 1]);
                        tmem_ld16(tb + N + CH * (h + 1), v1[(h + 1) & 1]);
                    } else {
                        tc_fence_before();
                        mbar_arrive(&tempty[buf]);
                    }
#pragma unroll
                    for (int jj = 0; jj < CH; jj += 4) {
                        const float4 w = lds4(wcur + CH * h + jj);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int j = (CH * h + jj) / 2 + u, i = jj + 2 * u;
                            const f32x2 sc = mul2(sa, u ? pack2(w.z, w.w) : pack2(w.x, w.y));
                            // X0 (exact integer sum) enters hi by TwoSum; X12, 2^-8 of it, goes straight
                            // into lo with the rounding error (FP32 rounding of lo is ~2^-31 of hi per
                            // k-tile)
                            const f32x2 e = two_sum2(hi[j], pack2(x0[i], x0[i + 1]), sc);
                            lo[j] = fma2(pack2(x12[i], x12[i + 1]), sc, add2(lo[j], e));
                        }
                    }
                }
            }
            ok = __all_sync(0xffffffffu, *abort_s == 0);
            if (ok && row < rows) {                   // float pairs: no FP64 work here
                // column c of the item is step c % 64 of group NG gi + c / 64, i.e. at
                // C + (NG gi) ldc_grp + c ldc_col (ldc_grp = 64 ldc_col)
                float2 *out = reinterpret_cast<float2 *>(C + (int64_t)ks * ldc_split + (int64_t)NG * gi * ldc_grp + row) +
                              (int64_t)c0 * ldc_col;
#pragma unroll
                for (int j = 0; j < COLS / 2; ++j) {
                    const float2 h = unpack2(hi[j]), l = unpack2(lo[j]);
                    out[(int64_t)(2 * j) * ldc_col] = make_float2(h.x, l.x);
                    out[(int64_t)(2 * j + 1) * ldc_col] = make_float2(h.y, l.y);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::TMEM));
    }
}

// ------------------------------------------------------------------------------------
// FP64 form (seven bf16 slices per operand). A[i][t] = 2^pA[i][t/64] sum_s a_s 2^-9s with integer digits
// |a_s| <= 256 (base 512, balanced: 63 bits from a row block's largest value down), W likewise per (step,
// 64-lag tile). This is the scheme of splitting FP64 operands into slices whose products a lower-
// precision matrix unit sums without rounding (Ozaki, Ogita, Oishi, Rump 2012). Per 64-column k-tile the
// products of level L = s + t,
//     X_L = sum a_s w_t 2^-9L,   |X_L| 2^9L <= (L + 1) 2^22,
// are exact in FP32 accumulators for L = 0 .. 3 (and for 4 unless its digits conspire: the bound is 1.25
// 2^24); levels 5 and 6 share one (rounded 2^-60 below X_0) and higher ones are dropped (2^-60 of a
// k-tile's largest term each): 28 products. With six slices and 21 products (levels 0 to 5) the sums were
// 1.5 times further from exact ones than the FP64 chain's, with six and 26 products 1.1 to 1.2 times (small
// increments beside a block's largest lost bits). The epilogue adds the six accumulators into three
// floats (h, m, l) per output by error-free sums, and the result leaves as FP64. Against exact sums its
// rms error is that of an FP64 multiply-add chain over the same terms (1.01 times, increments over seven
// decades); with levels 4 to 6 in one accumulator it would be 1.04 times.
// What bounds it: no one unit. A k-tile of 128 rows x 64 steps takes 112 MMAs (M = 128, N = 64, K = 16)
// that read 6 KB each next to 168 KB of TMA writes: 6,600 cycles of shared memory at 128 B per cycle; the
// tensor cores' own time is 3,600, the fold's 4,000 on the FP32 pipes and 3,000 of TMEM reads, HBM's 5,000.
// Measured 10,600: the FP64 pipe would take 320,000. At 65,536 rows the product over one k-tile takes 50 us,
// over ten 231 us. On the way: 8 epilogue warps of 32 columns, their conversions to FP64 with branches, and
// two stages of node-major slices took 102 and 302 us; the conversions alone 58 of each.
// Operands come as 32-column half tiles (64-byte swizzle), contiguous in memory: three stages of the history
// (it comes from HBM), two of the weights (they come from L2). 16-column stages of 32-byte swizzle let more
// be in flight, but were slower (26 %). The six accumulators of 64 columns rotate through eight TMEM slots,
// the widest level first, so that a k-tile's MMAs start while the one before is folded.
constexpr int F7_BK = 32;
constexpr int F7_A = BM * F7_BK * 2, F7_W = BN * F7_BK * 2;   // one slice of a stage: 8 KB, 4 KB
constexpr int F7_STA = 7 * F7_A, F7_STW = 7 * F7_W;           // a stage: 56 KB of history, 28 KB of weights
constexpr int F7_NA = 3, F7_NW = 2, F7_SLOTS = 8, F7_LEV = 6;
constexpr int F7_SMEM = 1024 + F7_NA * F7_STA + F7_NW * F7_STW + 256;
static_assert(F7_SMEM <= 227 * 1024, "shared memory");
constexpr int F7_COLS = 16, F7_EW = 4 * (BN / F7_COLS);       // columns per epilogue warp, epilogue warps
constexpr int F7_THREADS = 128 + 32 * F7_EW;                  // a TMA, an MMA and two idle warps, the epilogue

struct __align__(64) FarMaps7 {
    CUtensorMap a[7], w[7];
};

__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFFu) >> 4);        // start address
    d |= (uint64_t)1 << 16;                          // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(512 >> 4) << 32;                 // stride byte offset: 8 rows x 64 B
    d |= (uint64_t)1 << 46;                          // descriptor version (tcgen05)
    d |= (uint64_t)4 << 61;                          // SWIZZLE_64B
    return d;
}

// x 2^e for a finite x (e in a range where 2^e is normal), exact unless the result leaves FP64's range
__device__ __forceinline__ double scale_f64(double x, int e)
{
    const int hi = __double2hiint(x), f = (hi >> 20) & 0x7FF;
    if (f + e > 0 && f + e < 0x7FF && f > 0 && f < 0x7FF) return __hiloint2double(hi + e * (1 << 20), __double2loint(x));
    return scalbn(x, e);
}

struct Far7Args {
    double *C;
    int64_t ldc_split, ldc_col, rows;
    int kt_end, kt_per, n_split;                     // k-tiles [0, kt_end); the block's index is kt_end
    const int16_t *pA;                               // [k-tile][rows]
    const int16_t *eA;                               // [rows]: largest pA of the row so far
    int w_rows;                                      // 64 per weight tile
    const float *sW;                                 // [weight tiles][n_delta][64]: 2^(pW - eW)
    const int16_t *eW;                               // [weight tiles][64]: largest pW of the step
    int n_delta;
    const int *wcol;
    uint32_t idesc;
    unsigned *flags;
};

__global__ void __launch_bounds__(F7_THREADS, 1) k_far_tc7(const __grid_constant__ FarMaps7 maps, const Far7Args p)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *smw = smem + F7_NA * F7_STA;                  // the weights' stages
    uint64_t *bars = (uint64_t *)(smw + F7_NW * F7_STW);
    uint64_t *full = bars, *empty = full + F7_NA, *fullw = empty + F7_NA, *emptyw = fullw + F7_NW;
    uint64_t *sfull = emptyw + F7_NW, *sempty = sfull + F7_SLOTS, *mma_done = sempty + F7_SLOTS;
    volatile uint32_t *tmem_slot = (volatile uint32_t *)(mma_done + 1);
    volatile int *abort_s = (volatile int *)(mma_done + 2);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n_items = (int)(p.rows / BM) * p.n_split;
    if (threadIdx.x == 0) {
        for (int s = 0; s < F7_NA; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
        for (int s = 0; s < F7_NW; ++s) { mbar_init(&fullw[s], 1); mbar_init(&emptyw[s], 1); }
        for (int s = 0; s < F7_SLOTS; ++s) { mbar_init(&sfull[s], 1); mbar_init(&sempty[s], 32 * F7_EW); }
        mbar_init(mma_done, 1);
        *abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32((const void *)tmem_slot)),
                     "r"(F7_SLOTS * BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // the splits of a row tile differ in length when they do not divide the k-tiles: the rotation gives every
    // CTA each of them in turn where the grid is a multiple of their count
    auto k_range = [&](int item, int &mt, int &ks, int &k0, int &k1) {
        mt = item / p.n_split;
        ks = (item + (gridDim.x % p.n_split ? 0 : item / gridDim.x)) % p.n_split;
        k0 = ks * p.kt_per;
        k1 = min(k0 + p.kt_per, p.kt_end);
    };

    if (warp == 0) {
        if (lane == 0) {                                   // TMA producer: half tiles
            int g = 0, ga = 0, mt, ks, k0, k1;
            bool ok = true;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                k_range(item, mt, ks, k0, k1);
                const int yw = (p.wcol ? p.wcol[mt] : 0) * BN;
                for (int h = 2 * k0; h < 2 * k1; ++h, ++g) {
                    const int s = g % F7_NA, sw = g % F7_NW;
                    if (!mbar_wait(&empty[s], ((uint32_t)(g / F7_NA) & 1u) ^ 1u, p.flags, abort_s)) { ok = false; break; }
                    uint8_t *st = smem + s * F7_STA;
                    mbar_expect_tx(&full[s], F7_STA);
                    const int ya = h * (int)p.rows + mt * BM;
#pragma unroll
                    for (int q = 0; q < 7; ++q) tma_load_2d(st + q * F7_A, &maps.a[q], 0, ya, &full[s]);
                    ++ga;
                    if (!mbar_wait(&emptyw[sw], ((uint32_t)(g / F7_NW) & 1u) ^ 1u, p.flags, abort_s)) { ok = false; break; }
                    st = smw + sw * F7_STW;
                    mbar_expect_tx(&fullw[sw], F7_STW);
                    // the weights depend on the distance between the block and the k-tile only
                    const int y = (2 * (p.kt_end - (h >> 1) - 1) + (h & 1)) * p.w_rows + yw;
#pragma unroll
                    for (int q = 0; q < 7; ++q) tma_load_2d(st + q * F7_W, &maps.w[q], 0, y, &fullw[sw]);
                }
            }
            auto landed = [&](uint64_t *bar, int n, int stages) {   // own copies in flight
                for (int it = (n > stages ? n - stages : 0); it < n; ++it) {
                    const unsigned long long t0 = gtimer();
                    while (!mbar_try_wait(&bar[it % stages], (uint32_t)(it / stages) & 1u) && gtimer() - t0 < WAIT_NS) {}
                }
            };
            landed(full, ga, F7_NA);
            landed(fullw, g, F7_NW);
        }
    } else if (warp == 1) {
        if (lane == 0) {                                   // MMA issuer
            int g = 0, c = 0, mt, ks, k0, k1;              // half tiles, TMEM slots used so far
            bool ok = true;
            for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
                k_range(item, mt, ks, k0, k1);
                for (int h = 2 * k0; h < 2 * k1 && ok && !*abort_s; ++h, ++g) {
                    const int s = g % F7_NA, sw = g % F7_NW;
                    if (!mbar_wait(&full[s], (uint32_t)(g / F7_NA) & 1u, p.flags, abort_s) ||
                        !mbar_wait(&fullw[sw], (uint32_t)(g / F7_NW) & 1u, p.flags, abort_s)) { ok = false; break; }
                    tc_fence_after();
                    const bool second = h & 1;
                    const uint64_t dst = sdesc_sw64(smem_u32(smem + s * F7_STA));
                    const uint32_t dlo = (uint32_t)dst, dhi = (uint32_t)(dst >> 32);
                    const uint32_t wlo = (uint32_t)sdesc_sw64(smem_u32(smw + sw * F7_STW));
                    // accumulator 0: levels 6 and 5; 1 .. 5: levels 4 .. 0
#pragma unroll
                    for (int l = 0; l < F7_LEV; ++l) {
                        const int sl = (c + l) % F7_SLOTS;
                        if (!second) {
                            if (!mbar_wait(&sempty[sl], ((uint32_t)((c + l) / F7_SLOTS) & 1u) ^ 1u, p.flags, abort_s)) { ok = false; break; }
                            tc_fence_after();
                        }
                        const uint32_t x = tmem + (uint32_t)(sl * BN);
                        bool acc = second;
#pragma unroll
                        for (int lev = l == 0 ? 6 : 5 - l; lev >= 5 - l; --lev)
#pragma unroll
                            for (int sa = 0; sa <= lev; ++sa)
#pragma unroll
                                for (int k = 0; k < F7_BK / 16; ++k) {
                                    umma_lo(x, dlo + (uint32_t)(k * 2 + (sa * F7_A >> 4)),
                                            wlo + (uint32_t)(k * 2 + ((lev - sa) * F7_W >> 4)), dhi, p.idesc, acc ? 1u : 0u);
                                    acc = true;
                                }
                        if (second) umma_commit(&sfull[sl]);
                    }
                    umma_commit(&empty[s]);
                    umma_commit(&emptyw[sw]);
                    if (second) c += F7_LEV;
                }
            }
            umma_commit(mma_done);
            const unsigned long long t0 = gtimer();
            while (!mbar_try_wait(mma_done, 0) && gtimer() - t0 < WAIT_NS) {}
        }
    } else if (warp >= 4) {
        // epilogue warps: TMEM lane quadrant warp % 4, columns c0 .. c0 + F7_COLS - 1
        const int q = warp & 3, c0 = F7_COLS * ((warp >> 2) - 1);
        int c = 0, mt, ks, k0, k1;
        bool ok = true;
        for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            k_range(item, mt, ks, k0, k1);
            const int64_t row = (int64_t)mt * BM + q * 32 + lane;
            const int wt = p.wcol ? p.wcol[mt] : 0;
            const int16_t *pAr = p.pA + row;
            const int eA = p.eA[row];
            const float *sW = p.sW + (int64_t)wt * p.n_delta * BN + c0;
            constexpr int NP = F7_COLS / 2;
            f32x2 hh[NP], mm[NP], ll[NP];                     // columns 2j, 2j + 1
#pragma unroll
            for (int j = 0; j < NP; ++j) hh[j] = mm[j] = ll[j] = 0ull;
            int e_nx = k0 < k1 ? (int)pAr[k0 * p.rows] : 0;
            for (int kt = k0; kt < k1; ++kt, c += F7_LEV) {
                const float sa1 = pow2f(max(e_nx - eA, -127));
                const f32x2 sa = pack2(sa1, sa1);
                if (kt + 1 < k1) e_nx = pAr[(kt + 1) * p.rows];
                const float4 *w4 = reinterpret_cast<const float4 *>(sW + (int64_t)(p.kt_end - kt - 1) * BN);
                // not unrolled: the levels share two bodies (into m, into h), which have to stay in the
                // instruction cache (unrolled, the warps waited for instructions most of the time)
#pragma unroll 1
                for (int l = 0; l < F7_LEV; ++l) {
                    const int sl = (c + l) % F7_SLOTS;
                    mbar_wait(&sfull[sl], (uint32_t)((c + l) / F7_SLOTS) & 1u, p.flags, abort_s);
                    tc_fence_after();
                    const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(sl * BN + c0);
                    float v[F7_COLS];
                    tmem_ld16(ta, v);
                    tmem_ld_wait();
                    tmem_loaded<F7_COLS>(v);
                    tc_fence_before();
                    mbar_arrive(&sempty[sl]);
#pragma unroll
                    for (int k = 0; k < F7_COLS / 4; ++k) {
                        const float4 x = __ldg(w4 + k);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int j = 2 * k + u;
                            const f32x2 sc = mul2(sa, u ? pack2(x.z, x.w) : pack2(x.x, x.y));   // powers of two
                            const f32x2 y = pack2(v[2 * j], v[2 * j + 1]);
                            if (l <= 3)                                       // levels 6 + 5, 4, 3, 2
                                ll[j] = add2(ll[j], two_sum2(mm[j], y, sc));
                            else                                              // levels 1, 0
                                ll[j] = add2(ll[j], two_sum2(mm[j], two_sum2(hh[j], y, sc)));
                        }
                    }
                }
            }
            ok = __all_sync(0xffffffffu, *abort_s == 0);
            if (ok) {
                const int16_t *eW = p.eW + (int64_t)wt * BN + c0;
                double *out = p.C + (int64_t)ks * p.ldc_split + row + (int64_t)c0 * p.ldc_col;
                // the usual exponents: the result's own exponent moves, without its edge cases
                const int ew = eW[lane % F7_COLS] == PE7_ZERO ? 0 : eW[lane % F7_COLS], ea = eA == PE7_ZERO ? 0 : eA;
                const int lo = ea + __reduce_min_sync(0xffffffffu, ew), hi = ea + __reduce_max_sync(0xffffffffu, ew);
                const bool usual = __all_sync(0xffffffffu, lo > -800 && hi < 800);
                auto value = [&](int j, double (&d)[2]) {
                    const float2 h = unpack2(hh[j]), m = unpack2(mm[j]), l = unpack2(ll[j]);
                    d[0] = f2d_bits(h.x) + (f2d_bits(m.x) + f2d_bits(l.x));
                    d[1] = f2d_bits(h.y) + (f2d_bits(m.y) + f2d_bits(l.y));
                };
                if (usual) {
#pragma unroll
                    for (int j = 0; j < NP; ++j) {
                        double d[2];
                        value(j, d);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int e = ea + __shfl_sync(0xffffffffu, ew, 2 * j + u), dh = __double2hiint(d[u]);
                            out[(int64_t)(2 * j + u) * p.ldc_col] =
                                __hiloint2double(dh & 0x7FF00000 ? dh + e * (1 << 20) : 0, __double2loint(d[u]));
                        }
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < NP; ++j) {
                        double d[2];
                        value(j, d);
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int e = ea + __shfl_sync(0xffffffffu, ew, 2 * j + u);
                            out[(int64_t)(2 * j + u) * p.ldc_col] =
                                eA == PE7_NONFINITE ? __longlong_as_double(0x7FF8000000000000ll) : scale_f64(d[u], e);
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(F7_SLOTS * BN));
    }
}

// ---------------------------------------------------------------- host side

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)p;
    }
    return fn;
}

// 2D tensor map over a row-major [rows][cols] array of 16-bit values, box 64 (or 32) cols x box_rows.
static int make_map(CUtensorMap *tm, const void *base, int64_t rows, int64_t cols, int box_rows, int box_cols = BK)
{
    EncodeTiledFn enc = encode_fn();
    if (!enc) return set_error(FPDE_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is not available");
    if ((cols * 2) % 16 != 0 || ((uintptr_t)base % 16) != 0)
        return set_error(FPDE_ERR_ARG, "tensor map: row pitch and base must be 16-byte aligned");
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)(cols * 2)};
    cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    cuuint32_t es[2] = {1, 1};
    CUresult r = enc(tm, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(base), dims, strides, box, es,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == BK ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return set_error(FPDE_ERR_ARG, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return FPDE_OK;
}

}  // namespace tc

int far_plan_init(FarPlan *p, const void *a_hi, const void *a_lo, int64_t rows, int64_t lda, const void *w_hi,
                  const void *w_lo, int64_t ldw, int bf16)
{
    if (rows % tc::BM != 0 || lda % tc::BK != 0 || ldw % tc::BK != 0)
        return set_error(FPDE_ERR_ARG, "far contraction: rows must be a multiple of 128, pitches of 64");
    static_assert(sizeof(tc::FarMaps) <= sizeof(p->maps), "map storage");
    tc::FarMaps *m = (tc::FarMaps *)p->maps;
    int rc;
    if ((rc = tc::make_map(&m->a_hi, a_hi, rows, lda, tc::BM)) || (rc = tc::make_map(&m->a_lo, a_lo, rows, lda, tc::BM)) ||
        (rc = tc::make_map(&m->w_hi, w_hi, tc::BN, ldw, tc::BN)) || (rc = tc::make_map(&m->w_lo, w_lo, tc::BN, ldw, tc::BN)))
        return rc;
    p->rows = rows;
    p->idesc = tc::idesc_f16(bf16 ? 1 : 0, tc::BM, tc::BN);
    cudaError_t e = smem_opt_in((const void *)tc::k_far_tc, tc::SMEM_BYTES);
    if (e != cudaSuccess) return set_error(FPDE_ERR_CUDA, "far kernel smem attribute: %s", cudaGetErrorString(e));
    return FPDE_OK;
}

int far_plan3_init(FarPlan3 *p, const void *const a[3], int64_t rows, int64_t lda, const void *const w[3],
                   int64_t ldw, int w_tiles, bool tiled)
{
    if (rows % tc::BM != 0 || lda % tc::BK != 0 || ldw % tc::BK != 0)
        return set_error(FPDE_ERR_ARG, "far contraction: rows must be a multiple of 128, pitches of 64");
    static_assert(sizeof(tc::FarMaps3) <= sizeof(p->maps), "map storage");
    tc::FarMaps3 *m = (tc::FarMaps3 *)p->maps;
    int rc;
    const int64_t w_rows = (int64_t)tc::BN * (w_tiles > 0 ? w_tiles : 1);
    const int64_t ra = tiled ? rows * (lda / tc::BK) : rows, rw = tiled ? w_rows * (ldw / tc::BK) : w_rows;
    const int64_t ca = tiled ? tc::BK : lda, cw = tiled ? tc::BK : ldw;
    for (int q = 0; q < 3; ++q) {
        if ((rc = tc::make_map(&m->a[q], a[q], ra, ca, tc::BM))) return rc;
        if ((rc = tc::make_map(&m->w[q], w[q], rw, cw, tc::BN))) return rc;
        // 128-row weight boxes (two groups per item) exist only when the slices hold two tiles
        if (w_rows >= 2 * tc::BN) {
            if ((rc = tc::make_map(&m->w2[q], w[q], rw, cw, 2 * tc::BN))) return rc;
        } else {
            m->w2[q] = m->w[q];
        }
    }
    p->rows = rows;
    p->w_rows = w_rows;
    p->tiled = tiled;
    p->idesc = tc::idesc_f16(1, tc::BM, tc::BN);
    p->idesc2 = tc::idesc_f16(1, tc::BM, 2 * tc::BN);
    cudaError_t e = smem_opt_in((const void *)tc::k_far_tc3<1>, tc::Far3Cfg<1>::SMEM);
    if (e == cudaSuccess) e = smem_opt_in((const void *)tc::k_far_tc3<2>, tc::Far3Cfg<2>::SMEM);
    if (e != cudaSuccess) return set_error(FPDE_ERR_CUDA, "far kernel smem attribute: %s", cudaGetErrorString(e));
    return FPDE_OK;
}

int far3_launch(cudaStream_t st, const FarPlan3 *p, int k_cols, double *C, int64_t ldc_split, int64_t ldc_col,
                int splits, const int8_t *pA, const float *pW, int64_t ldp, unsigned *flags, const int *wcol,
                int k_begin, int n_grp, int grp0)
{
    if (n_grp < 1 || grp0 < 0 || (int64_t)(grp0 + n_grp) * tc::BN > p->w_rows)
        return set_error(FPDE_ERR_ARG, "far contraction: weight rows out of range");
    if (k_cols % tc::BK != 0 || k_begin % tc::BK != 0 || k_begin < 0 || k_begin > k_cols)
        return set_error(FPDE_ERR_ARG, "far contraction: K range must be in multiples of 64");
    if (k_cols == k_begin) return FPDE_OK;
    const int kt_total = k_cols / tc::BK, kt_begin = k_begin / tc::BK;
    if (splits < 1) splits = 1;
    if (splits > FAR_MAX_SPLITS) splits = FAR_MAX_SPLITS;
    const int kt_per = (kt_total - kt_begin + splits - 1) / splits;   // every split is written, possibly with zeros
    // Two weight groups per item (one N = 128 MMA reads the history tile once for both) when the
    // groups pair up; the item sets of one (row tile, split) are consecutive items, and a grid that
    // is a multiple of their count keeps them on neighbouring CTAs for the whole walk, so the
    // history tiles they share stream from HBM once and are re-read from L2.
    const int ng = (n_grp % 2 == 0) ? 2 : 1;
    const int n_sets = n_grp / ng;
    const int64_t items = (p->rows / tc::BM) * splits * n_sets;
    const int sms = device_sm_count();
    int64_t grid = std::min<int64_t>(items, sms);
    if (grid > n_sets) grid -= grid % n_sets;
    const tc::FarMaps3 *m = (const tc::FarMaps3 *)p->maps;
    const int64_t ldc_grp = (int64_t)tc::BN * ldc_col;
    const tc::Far3Layout ly = p->tiled ? tc::Far3Layout{0, (int)p->rows, (int)p->w_rows, 1, p->rows, 1, p->w_rows}
                                       : tc::Far3Layout{tc::BK, 0, 0, ldp, 1, ldp, 1};
    if (ng == 2)
        tc::k_far_tc3<2><<<(unsigned)grid, tc::Far3Cfg<2>::THREADS, tc::Far3Cfg<2>::SMEM, st>>>(
            *m, C, ldc_split, ldc_col, p->rows, kt_begin, kt_total, kt_per, splits, p->idesc2, pA, pW, ly, wcol,
            n_sets, grp0, ldc_grp, flags);
    else
        tc::k_far_tc3<1><<<(unsigned)grid, tc::Far3Cfg<1>::THREADS, tc::Far3Cfg<1>::SMEM, st>>>(
            *m, C, ldc_split, ldc_col, p->rows, kt_begin, kt_total, kt_per, splits, p->idesc, pA, pW, ly, wcol,
            n_sets, grp0, ldc_grp, flags);
    FPDE_LAUNCHED(1);
    return FPDE_OK;
}

int far_plan7_init(FarPlan7 *p, const void *const a[7], int64_t rows, int n_tiles, const void *const w[7], int w_tiles)
{
    if (rows % tc::BM != 0) return set_error(FPDE_ERR_ARG, "far contraction: rows must be a multiple of 128");
    static_assert(sizeof(tc::FarMaps7) <= sizeof(p->maps), "map storage");
    tc::FarMaps7 *m = (tc::FarMaps7 *)p->maps;
    int rc;
    for (int q = 0; q < 7; ++q)
        if ((rc = tc::make_map(&m->a[q], a[q], 2 * n_tiles * rows, tc::F7_BK, tc::BM, tc::F7_BK)) ||
            (rc = tc::make_map(&m->w[q], w[q], (int64_t)2 * n_tiles * tc::BN * w_tiles, tc::F7_BK, tc::BN, tc::F7_BK)))
            return rc;
    p->rows = rows;
    p->idesc = tc::idesc_f16(1, tc::BM, tc::BN);
    cudaError_t e = smem_opt_in((const void *)tc::k_far_tc7, tc::F7_SMEM);
    if (e != cudaSuccess) return set_error(FPDE_ERR_CUDA, "far kernel smem attribute: %s", cudaGetErrorString(e));
    return FPDE_OK;
}

int far7_launch(cudaStream_t st, const FarPlan7 *p, const Hist7 &h, int k_cols, double *C, int64_t ldc_split,
                int64_t ldc_col, int splits, unsigned *flags, const int *wcol)
{
    if (k_cols % tc::BK != 0 || k_cols < 0)
        return set_error(FPDE_ERR_ARG, "far contraction: K range must be in multiples of 64");
    if (k_cols == 0) return FPDE_OK;
    tc::Far7Args a;
    a.kt_end = k_cols / tc::BK;
    if (a.kt_end > h.n_delta) return set_error(FPDE_ERR_ARG, "far contraction: weight tiles out of range");
    splits = std::max(1, std::min(splits, FAR_MAX_SPLITS));
    a.kt_per = (a.kt_end + splits - 1) / splits;                   // every split is written, possibly with zeros
    a.n_split = splits;
    a.C = C; a.ldc_split = ldc_split; a.ldc_col = ldc_col; a.rows = p->rows;
    a.pA = h.pA; a.eA = h.eA; a.w_rows = tc::BN * h.w_tiles; a.sW = h.sW; a.eW = h.eW; a.n_delta = h.n_delta; a.wcol = wcol;
    a.idesc = p->idesc; a.flags = flags;
    const int64_t items = (p->rows / tc::BM) * splits;
    const unsigned grid = (unsigned)std::min<int64_t>(items, device_sm_count());
    tc::k_far_tc7<<<grid, tc::F7_THREADS, tc::F7_SMEM, st>>>(*(const tc::FarMaps7 *)p->maps, a);
    FPDE_LAUNCHED(1);
    return FPDE_OK;
}

int far_splits(int kt_total, int64_t rows)
{
    // Splits of K only for balance of the persistent grid (one CTA per SM): the fewest splits
    // whose items fill the SMs within 5% (each split keeps at least 2 k-tiles).
    const int sms = device_sm_count();
    const int64_t tiles = rows / tc::BM;
    int best = 1;
    double best_waste = 1e30;
    for (int s = 1; s <= FAR_MAX_SPLITS && (s == 1 || kt_total / s >= 2); ++s) {
        const int64_t items = tiles * s;
        const double waves = (double)items / sms, full = (double)((items + sms - 1) / sms);
        const double waste = full / waves;
        if (waste < best_waste - 1e-9) { best_waste = waste; best = s; }
        if (waste <= 1.05) break;
    }
    return best;
}

int far_launch(cudaStream_t st, const FarPlan *p, int k_cols, double *C, int64_t ldc_split, int64_t ldc_col,
               int splits, double out_scale, const double *out_scale_ptr, unsigned *flags)
{
    if (k_cols % tc::BK != 0) return set_error(FPDE_ERR_ARG, "far contraction: K must be a multiple of 64");
    if (k_cols == 0) return FPDE_OK;
    const int kt_total = k_cols / tc::BK;
    if (splits < 1) splits = 1;
    if (splits > FAR_MAX_SPLITS) splits = FAR_MAX_SPLITS;
    const int kt_per = (kt_total + splits - 1) / splits;
    splits = (kt_total + kt_per - 1) / kt_per;
    dim3 grid((unsigned)(p->rows / tc::BM), (unsigned)splits);
    const tc::FarMaps *m = (const tc::FarMaps *)p->maps;
    tc::k_far_tc<<<grid, tc::THREADS, tc::SMEM_BYTES, st>>>(*m, C, ldc_split, ldc_col, p->rows, kt_total, kt_per,
                                                           p->idesc, out_scale, out_scale_ptr, flags);
    FPDE_LAUNCHED(1);
    return FPDE_OK;
}

}  // namespace fpde

using namespace fpde;

extern "C" int fpde_far_contract(fpde_ctx *ctx, const void *a_hi, const void *a_lo, int64_t rows, int64_t lda,
                                 const void *w_hi, const void *w_lo, int64_t ldw, int k_cols, int bf16,
                                 double out_scale, double *C, int splits)
{
    clear_error();
    int rc = ctx_enter(ctx);
    if (rc) return rc;
    FPDE_CHECK_ARG(a_hi && a_lo && w_hi && w_lo && C && rows > 0 && k_cols >= 0, "bad arguments");
    FPDE_CHECK_ARG(k_cols <= lda && k_cols <= ldw, "K beyond the operand pitch");
    FarPlan plan;
    if ((rc = far_plan_init(&plan, a_hi, a_lo, rows, lda, w_hi, w_lo, ldw, bf16))) return rc;
    const int kt_total = k_cols / 64;
    if (splits <= 0) splits = far_splits(kt_total, rows);
    if ((rc = far_launch(ctx->stream, &plan, k_cols, C, rows * 64, rows, splits, out_scale, nullptr, ctx->d_flags)))
        return rc;
    FPDE_CUDA(cudaStreamSynchronize(ctx->stream));
    return ctx_check_flags(ctx, "far contraction");
}

namespace fpde {
// Weight-tile exponents -> their scales 2^e (the far kernel takes the scales).
__global__ void k_exp_to_scale(const int8_t *e, float *s, int64_t n)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) s[i] = tc::pow2f((int)e[i]);
}
// In place: float-pair slots of a far contraction -> FP64 values.
__global__ void k_ff_to_double(double *C, int64_t n)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) C[i] = ff_to_double(C[i]);
}
}  // namespace fpde

extern "C" int fpde_far_contract3(fpde_ctx *ctx, const void *const a[3], int64_t rows, int64_t lda,
                                  const void *const w[3], int64_t ldw, int k_cols, const int8_t *pA,
                                  const int8_t *pW, int64_t ldp, double *C, int splits)
{
    clear_error();
    int rc = ctx_enter(ctx);
    if (rc) return rc;
    FPDE_CHECK_ARG(a && w && a[0] && a[1] && a[2] && w[0] && w[1] && w[2] && pA && pW && C, "null argument");
    FPDE_CHECK_ARG(rows > 0 && k_cols >= 0 && k_cols <= lda && k_cols <= ldw && ldp * 64 >= k_cols, "bad shape");
    FarPlan3 plan;
    if ((rc = far_plan3_init(&plan, a, rows, lda, w, ldw, 1, false))) return rc;
    if (splits <= 0) splits = far_splits(k_cols / 64, rows);
    if (splits > FAR_MAX_SPLITS) splits = FAR_MAX_SPLITS;
    float *pWs = nullptr;
    const int64_t nw = 64 * ldp;
    if (dev_alloc((void **)&pWs, (size_t)nw * sizeof(float))) return FPDE_ERR_NOMEM;
    k_exp_to_scale<<<(unsigned)((nw + 255) / 256), 256, 0, ctx->stream>>>(pW, pWs, nw);
    FPDE_LAUNCHED(1);
    rc = far3_launch(ctx->stream, &plan, k_cols, C, rows * 64, rows, splits, pA, pWs, ldp, ctx->d_flags);
    if (rc) {
        cudaStreamSynchronize(ctx->stream);
        dev_free(pWs);
        return rc;
    }
    const int64_t n = (int64_t)splits * 64 * rows;
    if (k_cols > 0) {
        k_ff_to_double<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(C, n);
        FPDE_LAUNCHED(1);
    }
    FPDE_CUDA(cudaStreamSynchronize(ctx->stream));
    dev_free(pWs);
    return ctx_check_flags(ctx, "far contraction (three slices)");
}
