// Block preparation of the split-precision path (per block of 64 steps):
//   k_absmax  : largest |increment| of the finished block (for the fp16 scale)
//   k_convert : FP64 increments (time-major ring, 64 rows of P) -> 16-bit hi/lo pairs in the
//               node-major history used as the K-major A operand, scaled by 2^sexp
//   k_wgen    : Toeplitz weight tile W[j][t] = w[n0+j-t] * 2^(kexp - sexp(t)), split hi/lo,
//               and the output scale 2^-kexp of the contraction
// The power-of-two scales keep fp16 operands inside its normal range; they are exact, and
// A*W keeps its value up to the single global factor 2^kexp undone in the epilogue.
// bf16 has float's exponent range and runs unscaled (sexp = kexp = 0).
// Three slices (k_convert3, k_wgen3) and seven slices (k_convert7, k_wgen7) are exact digits with a block
// exponent each, stored k-tile by k-tile; k_near64_pre and k_near64 sum a block's own rows in FP64.
#include <algorithm>
#include <cmath>
#include <vector>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "common.cuh"
#include "kernels.cuh"
#include "tc_far.cuh"

namespace fpde {

__global__ void k_absmax(const double *__restrict__ x, int64_t n, unsigned long long *slot)
{
    double m = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        m = fmax(m, fabs(x[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    __shared__ double red[32];
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < 32) {
        m = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (threadIdx.x == 0 && m > 0.0) atomicMax(slot, (unsigned long long)__double_as_longlong(m));
    }
}

__device__ __forceinline__ int scale_exp_from_max(unsigned long long bits)
{
    const double m = __longlong_as_double((long long)bits);
    if (!(m > 0.0)) return 0;
    const int e = ilogb(m) + 1;           // m < 2^e
    return 14 - e;                        // scaled max < 2^14
}

__device__ __forceinline__ void split16(double v, int bf16, uint16_t &h, uint16_t &l)
{
    if (bf16) {
        __nv_bfloat16 hb = __double2bfloat16(v);
        __nv_bfloat16 lb = __double2bfloat16(v - (double)__bfloat162float(hb));
        h = __bfloat16_as_ushort(hb);
        l = __bfloat16_as_ushort(lb);
    } else {
        __half hh = __double2half(v);
        __half lh = __double2half(v - (double)__half2float(hh));
        h = __half_as_ushort(hh);
        l = __half_as_ushort(lh);
    }
}

// One CTA per 64 nodes: transpose a 64 (rows of the ring) x 64 (nodes) FP64 tile through
// shared memory and write each node's 64 new history columns as 16-byte vectors.
__global__ void __launch_bounds__(256) k_convert(const double *__restrict__ ring, int64_t P, int64_t nvalid,
                                                 const unsigned long long *__restrict__ slot, int *__restrict__ exps,
                                                 int blk, uint16_t *__restrict__ hi, uint16_t *__restrict__ lo,
                                                 int64_t ld, int64_t col0, int bf16)
{
    __shared__ double tile[64][65];
    const int64_t node0 = (int64_t)blockIdx.x * 64;
    const int sexp = bf16 ? 0 : scale_exp_from_max(*slot);
    const double sc = ldexp(1.0, sexp);
    if (blockIdx.x == 0 && threadIdx.x == 0) exps[blk] = sexp;
    for (int e = threadIdx.x; e < 64 * 64; e += 256) {
        const int r = e >> 6, c = e & 63;
        const int64_t node = node0 + c;
        tile[c][r] = node < nvalid ? ring[(int64_t)r * P + node] * sc : 0.0;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 64 * 8; e += 256) {
        const int c = e >> 3, g = e & 7;                 // node c, columns 8g..8g+7
        const int64_t node = node0 + c;
        if (node >= nvalid) continue;
        uint16_t h[8], l[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) split16(tile[c][8 * g + k], bf16, h[k], l[k]);
        uint4 vh, vl;
        vh.x = h[0] | ((uint32_t)h[1] << 16); vh.y = h[2] | ((uint32_t)h[3] << 16);
        vh.z = h[4] | ((uint32_t)h[5] << 16); vh.w = h[6] | ((uint32_t)h[7] << 16);
        vl.x = l[0] | ((uint32_t)l[1] << 16); vl.y = l[2] | ((uint32_t)l[3] << 16);
        vl.z = l[4] | ((uint32_t)l[5] << 16); vl.w = l[6] | ((uint32_t)l[7] << 16);
        *(uint4 *)(hi + node * ld + col0 + 8 * g) = vh;
        *(uint4 *)(lo + node * ld + col0 + 8 * g) = vl;
    }
}

// grid = (ceil(n0/256), 64): row j of the weight tile, columns t < n0.
__global__ void __launch_bounds__(256) k_wgen(const double *__restrict__ wlag, int n0, const int *__restrict__ exps,
                                              uint16_t *__restrict__ whi, uint16_t *__restrict__ wlo, int64_t ldw,
                                              int bf16, double *__restrict__ out_scale)
{
    __shared__ int s_kexp;
    if (threadIdx.x < 32) {
        int kmax = -100000;
        if (!bf16) {
            for (int b = threadIdx.x; b < n0 / 64; b += 32) {
                const double wm = wlag[n0 - 64 * b - 63];            // largest weight of block b
                const int ew = (wm > 0.0) ? ilogb(wm) + 1 : -100000; // wm < 2^ew
                kmax = max(kmax, ew - exps[b]);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) kmax = max(kmax, __shfl_xor_sync(0xffffffffu, kmax, o));
        }
        if (threadIdx.x == 0) s_kexp = bf16 ? 0 : (kmax > -100000 ? 14 - kmax : 0);
    }
    __syncthreads();
    const int kexp = s_kexp;
    const int j = blockIdx.y;
    const int t = blockIdx.x * 256 + threadIdx.x;
    if (blockIdx.x == 0 && j == 0 && threadIdx.x == 0) *out_scale = ldexp(1.0, -kexp);
    if (t >= n0) return;
    const double v = wlag[n0 + j - t] * ldexp(1.0, kexp - (bf16 ? 0 : exps[t >> 6]));
    uint16_t h, l;
    split16(v, bf16, h, l);
    whi[(int64_t)j * ldw + t] = h;
    wlo[(int64_t)j * ldw + t] = l;
}

// ---- exact three-slice form (bf16): x 2^-pe = a0 + a1 2^-8 + a2 2^-16 (+ rounding at 2^-16),
// |x| < 2^(pe+8), with integer a0 (|a0| <= 256) and a1, a2 (|.| <= 128); the exponent pe is
// stored per (node, 64-column block) for the history and per (step j, k-tile) for the
// weights.
// Integer form of the slicing (no FP64 arithmetic; GB300's FP64 pipe is narrow):
// v = rint(x * 2^(16 - pe)) from the double's bits, |v| <= 2^24, then balanced base-256
// digits v = a0 2^16 + a1 2^8 + a2 with |a0| <= 256, |a1|, |a2| <= 128.
__device__ __forceinline__ long long fixed16(double x, int pe)
{
    const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
    const int ex = (int)((bits >> 52) & 0x7FF);
    if (ex == 0) return 0;                               // zero / subnormal: below the 2^-16 grid
    const long long mant = (long long)((bits & 0xFFFFFFFFFFFFFull) | (1ull << 52));
    const int sh = (ex - 1075) + 16 - pe;                // value * 2^(16-pe) = mant * 2^sh
    long long v;
    if (sh >= 0) {
        v = sh > 10 ? (1ll << 62) : (mant << sh);        // out of range: caller's exponent prevents it
    } else if (sh < -62) {
        v = 0;
    } else {
        const int r = -sh;
        const long long q = mant >> r;
        const long long rem = mant & ((1ll << r) - 1);
        const long long half = 1ll << (r - 1);
        v = q + ((rem > half || (rem == half && (q & 1))) ? 1 : 0);   // round half to even
    }
    return (bits >> 63) ? -v : v;
}
__device__ __forceinline__ void digits3(long long v, uint16_t &s0, uint16_t &s1, uint16_t &s2)
{
    const int iv = (int)v;                               // |v| <= 2^24
    const int a0 = (iv + 32768) >> 16;
    const int r1 = iv - a0 * 65536;                      // [-32768, 32767]
    const int a1 = (r1 + 128) >> 8;
    const int a2 = r1 - a1 * 256;                        // [-128, 127]
    s0 = __bfloat16_as_ushort(__float2bfloat16((float)a0));
    s1 = __bfloat16_as_ushort(__float2bfloat16((float)a1 * (1.0f / 256.0f)));
    s2 = __bfloat16_as_ushort(__float2bfloat16((float)a2 * (1.0f / 65536.0f)));
}
// Block exponent from the largest magnitude: |x| < 2^(pe + 8).
__device__ __forceinline__ int exp_of_maxbits(unsigned long long mbits)
{
    const int ex = (int)((mbits >> 52) & 0x7FF);
    if (ex == 0) return 0;
    const int p = (ex - 1023) + 1 - 8;
    return p < -127 ? -127 : (p > 127 ? 127 : p);
}

// Four adjacent lanes per node, each with 16 of the node's 64 increments of the finished block
// (time-major ring: for each row the lanes of a warp read eight consecutive nodes). The block
// exponent is the maximum over the four lanes (shuffles); each lane then writes its 16 columns of
// the three slices. Sixteen values per thread keep the registers low and many nodes' loads in
// flight (one thread per node with all 64 values had left the kernel latency-bound).
constexpr int CONV_LANES = 4, CONV_ROWS = 64 / CONV_LANES;
__global__ void __launch_bounds__(256) k_convert3(const double *__restrict__ ring, int64_t P, int64_t nvalid,
                                                  uint16_t *__restrict__ h0, uint16_t *__restrict__ h1,
                                                  uint16_t *__restrict__ h2, int64_t rows,
                                                  int8_t *__restrict__ pA, int blk)
{
    const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t node = gt / CONV_LANES;
    const int part = (int)(gt % CONV_LANES);
    const bool live = node < nvalid;
    const int r0 = part * CONV_ROWS;
    unsigned long long v[CONV_ROWS];
    unsigned long long mb = 0;
    const unsigned long long *src = (const unsigned long long *)ring + (live ? node : 0);
#pragma unroll
    for (int r = 0; r < CONV_ROWS; ++r) {
        v[r] = live ? __ldcg(src + (int64_t)(r0 + r) * P) : 0ull;
        const unsigned long long m0 = v[r] & 0x7FFFFFFFFFFFFFFFull;
        mb = m0 > mb ? m0 : mb;
    }
#pragma unroll
    for (int o = 1; o < CONV_LANES; o <<= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, mb, o, CONV_LANES);
        mb = other > mb ? other : mb;
    }
    if (!live) return;
    const int pe = exp_of_maxbits(mb);
    if (part == 0) pA[blk * rows + node] = (int8_t)pe;
#pragma unroll
    for (int g = 0; g < CONV_ROWS / 8; ++g) {
        uint16_t a[8], b[8], c[8];
#pragma unroll
        for (int k = 0; k < 8; ++k)
            digits3(fixed16(__longlong_as_double((long long)v[8 * g + k]), pe), a[k], b[k], c[k]);
        uint4 va, vb, vc;
        va.x = a[0] | ((uint32_t)a[1] << 16); va.y = a[2] | ((uint32_t)a[3] << 16);
        va.z = a[4] | ((uint32_t)a[5] << 16); va.w = a[6] | ((uint32_t)a[7] << 16);
        vb.x = b[0] | ((uint32_t)b[1] << 16); vb.y = b[2] | ((uint32_t)b[3] << 16);
        vb.z = b[4] | ((uint32_t)b[5] << 16); vb.w = b[6] | ((uint32_t)b[7] << 16);
        vc.x = c[0] | ((uint32_t)c[1] << 16); vc.y = c[2] | ((uint32_t)c[3] << 16);
        vc.z = c[4] | ((uint32_t)c[5] << 16); vc.w = c[6] | ((uint32_t)c[7] << 16);
        const int64_t o = (blk * rows + node) * 64 + r0 + 8 * g;
        *(uint4 *)(h0 + o) = va;
        *(uint4 *)(h1 + o) = vb;
        *(uint4 *)(h2 + o) = vc;
    }
}

// grid = (n0/64 + n_grp - 1 k-tiles, 64 n_grp steps r, columns), 64 threads:
// W[c*64*n_grp + r][t] = w_c[n0 + r - t] for the k-tile (one weight tile per column of an
// ensemble; one column for a line or a grid). Row r (of weight group r/64) gets the columns
// t < n0 + 64 (r/64): every lag n0 + r - t it holds is at least 1. With n_grp > 1 the groups past
// the first serve the steps of the later blocks of a super-block starting at n0, the columns
// past n0 their contraction over the super-block's own history.
__global__ void __launch_bounds__(64) k_wgen3(const double *__restrict__ wlag_all, int64_t wstride, int n0,
                                              uint16_t *__restrict__ w0, uint16_t *__restrict__ w1,
                                              uint16_t *__restrict__ w2, float *__restrict__ pW, int n_grp,
                                              int kt_lim)
{
    __shared__ double red[2];
    const int kt = blockIdx.x, r = blockIdx.y;
    if (kt >= n0 / 64 + r / 64 || kt >= kt_lim) return;  // the whole CTA (uniform)
    const int j = r + 64 * n_grp * blockIdx.z;
    const double *wlag = wlag_all + (int64_t)blockIdx.z * wstride;
    const int64_t row = (int64_t)kt * (64 * n_grp * gridDim.z) + j;   // of the tile-major slices
    const int t = kt * 64 + threadIdx.x;
    const double v = wlag[n0 + r - t];
    double m = fabs(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = fmax(red[0], red[1]);
    const int pe = exp_of_maxbits((unsigned long long)__double_as_longlong(m));
    if (threadIdx.x == 0)                                // the scale 2^pe, exact (pe in [-127, 127])
        pW[row] = pe >= -126 ? __int_as_float((pe + 127) << 23) : __int_as_float(0x00400000);
    uint16_t a, b, c;
    digits3(fixed16(v, pe), a, b, c);
    w0[row * 64 + threadIdx.x] = a;
    w1[row * 64 + threadIdx.x] = b;
    w2[row * 64 + threadIdx.x] = c;
}

// ---- seven-slice form: x 2^-pe = sum_s a_s 2^-9s, |x| < 2^(pe+8), balanced base-512 digits |a_s| <= 256
// of the 63-bit integer v = rint(x 2^(54-pe)); each digit is stored as the bf16 value a_s 2^-9s (exact). Blocks
// below the normal range keep the exponent of its lower end; one with an infinity or a NaN has PE7_NONFINITE and
// zero digits, and every sum of its row is NaN.
__device__ __forceinline__ int exp7_of_maxbits(unsigned long long mbits)
{
    const int ex = (int)((mbits >> 52) & 0x7FF);
    return mbits == 0 ? PE7_ZERO : ex == 0x7FF ? PE7_NONFINITE : max(ex, 1) - 1023 + 1 - 8;
}
__device__ __forceinline__ void digits7(unsigned long long bits, int pe, uint16_t (&s)[7])
{
    const int ex = (int)((bits >> 52) & 0x7FF);
    const long long mant = (long long)(bits & 0xFFFFFFFFFFFFFull) | (ex ? 1ll << 52 : 0ll);
    long long v = 0;
    if (mant != 0) {
        const int r = pe + 1021 - max(ex, 1);        // >= -9: within 9 binary orders of the largest, exact
        if (r <= 0) v = mant << min(-r, 9);
        else if (r < 62) {
            const long long q = mant >> r, rem = mant & ((1ll << r) - 1), half = 1ll << (r - 1);
            v = q + ((rem > half || (rem == half && (q & 1))) ? 1 : 0);   // round half to even
        }
        if (bits >> 63) v = -v;
    }
#pragma unroll
    for (int k = 6; k >= 1; --k) {
        const int a = (int)((v + 256) & 511) - 256;
        v = (v - a) >> 9;
        s[k] = __bfloat16_as_ushort(__float2bfloat16((float)a * __int_as_float((127 - 9 * k) << 23)));
    }
    s[0] = __bfloat16_as_ushort(__float2bfloat16((float)(int)v));
}
struct Slices7 { uint16_t *p[7]; };

// Eight adjacent lanes per node, each with 8 of the node's 64 increments (as k_convert3); also the
// row's largest block exponent so far.
constexpr int CONV7_LANES = 8, CONV7_ROWS = 64 / CONV7_LANES;
__global__ void __launch_bounds__(256) k_convert7(const double *__restrict__ rows64, int64_t P, int64_t nvalid, Slices7 out,
                                                  int64_t rows, int16_t *__restrict__ pA, int blk,
                                                  int16_t *__restrict__ eA)
{
    const int64_t gt = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t node = gt / CONV7_LANES;
    const int part = (int)(gt % CONV7_LANES);
    const bool live = node < nvalid;
    const int r0 = part * CONV7_ROWS;
    unsigned long long v[CONV7_ROWS], mb = 0;
    const unsigned long long *src = (const unsigned long long *)rows64 + (live ? node : 0);
#pragma unroll
    for (int r = 0; r < CONV7_ROWS; ++r) {
        v[r] = live ? __ldcg(src + (int64_t)(r0 + r) * P) : 0ull;
        const unsigned long long m0 = v[r] & 0x7FFFFFFFFFFFFFFFull;
        mb = m0 > mb ? m0 : mb;
    }
#pragma unroll
    for (int o = 1; o < CONV7_LANES; o <<= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, mb, o, CONV7_LANES);
        mb = other > mb ? other : mb;
    }
    if (!live) return;
    const int pe = exp7_of_maxbits(mb);
    if (part == 0) {
        pA[blk * rows + node] = (int16_t)pe;
        eA[node] = (int16_t)(blk == 0 ? pe : max((int)eA[node], pe));
    }
    uint16_t d[CONV7_ROWS][7];
#pragma unroll
    for (int k = 0; k < CONV7_ROWS; ++k) digits7(v[k], pe, d[k]);
    const int64_t o = ((2 * blk + r0 / 32) * rows + node) * 32 + r0 % 32;
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        uint4 x;
        x.x = d[0][q] | ((uint32_t)d[1][q] << 16); x.y = d[2][q] | ((uint32_t)d[3][q] << 16);
        x.z = d[4][q] | ((uint32_t)d[5][q] << 16); x.w = d[6][q] | ((uint32_t)d[7][q] << 16);
        *(uint4 *)(out.p[q] + o) = x;
    }
}

// grid (weight tiles, 64 steps j), 64 threads: every distance's tile of step j, two passes (the largest
// exponent first). The tiles, one per column of an ensemble, take the x axis: y ends at 65,535.
__global__ void __launch_bounds__(64) k_wgen7(const double *__restrict__ wlag_all, int64_t wstride, Slices7 out,
                                              int n_delta, float *__restrict__ sW, int16_t *__restrict__ eW)
{
    __shared__ unsigned long long red[2];
    const int j = blockIdx.y, c = threadIdx.x;
    const double *w = wlag_all + (int64_t)blockIdx.x * wstride;
    auto tile_exp = [&](int d) {
        unsigned long long m = (unsigned long long)__double_as_longlong(fabs(w[64 * d + j - c]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long x = __shfl_xor_sync(0xffffffffu, m, o);
            m = x > m ? x : m;
        }
        __syncthreads();
        if ((c & 31) == 0) red[c >> 5] = m;
        __syncthreads();
        return exp7_of_maxbits(red[0] > red[1] ? red[0] : red[1]);
    };
    int emax = PE7_ZERO;
    for (int d = 1; d <= n_delta; ++d) emax = max(emax, tile_exp(d));
    if (c == 0) eW[(int64_t)blockIdx.x * 64 + j] = (int16_t)emax;
    for (int d = 1; d <= n_delta; ++d) {
        const int pe = tile_exp(d);
        if (c == 0) {
            const int e = max(pe - emax, -126);
            sW[((int64_t)blockIdx.x * n_delta + d - 1) * 64 + j] = __int_as_float((e + 127) << 23);
        }
        uint16_t s[7];
        digits7((unsigned long long)__double_as_longlong(w[64 * d + j - c]), pe, s);
        const int64_t o = (((int64_t)2 * (d - 1) + c / 32) * (64 * (int64_t)gridDim.x) + 64 * (int64_t)blockIdx.x + j) * 32 + c % 32;
#pragma unroll
        for (int q = 0; q < 7; ++q) out.p[q][o] = s[q];
    }
}

// Near history of a 64-step block in FP64, one node per thread, in sub-blocks of 8 steps: k_near64_pre adds
// the block's rows before j0 to the far sums of the steps j0 .. j0 + 7 (out[u] = init[u] + sum_{r < j0}
// w[j0 + u - r] D_r), k_near64 a step's own sub-block rows (S = init + sum_{j0 <= r < j} w[j - r] D_r); the
// order of the sums is that of one pass over the rows. FP64-pipe bound: one multiply-add per row and step.
// k_near64_pre keeps the pipe 96 % busy. Read again for every step the rows bound it instead: 19.9 us per
// step for 284,000 nodes (20.6 in one pass per step), 14.0 for 96 columns of 200 to 5,000 nodes (16.7).
// CTAs of 64 nodes give the SMs equal shares (512 nodes: 22.2 and 17.5 in one pass).
constexpr int N64_T = 64;
__global__ void __launch_bounds__(N64_T) k_near64(const double *__restrict__ rows, int64_t P, int j,
                                                  const double *__restrict__ wlag, int64_t wstride,
                                                  const int *__restrict__ cta_col, const double *__restrict__ init,
                                                  double *__restrict__ S)
{
    const int64_t i = (int64_t)blockIdx.x * N64_T + threadIdx.x;
    if (i >= P) return;
    const double *w = wlag;
    if (cta_col) w += (int64_t)cta_col[blockIdx.x / (512 / N64_T)] * wstride;      // a 512-node group's column
    double s = init ? __ldcs(init + i) : 0.0;
    const int r = j - j % NEAR_SUB;
    double v[NEAR_SUB];
#pragma unroll
    for (int u = 0; u < NEAR_SUB; ++u) v[u] = r + u < j ? __ldcg(rows + (int64_t)(r + u) * P + i) : 0.0;
#pragma unroll
    for (int u = 0; u < NEAR_SUB; ++u)
        if (r + u < j) s = fma(__ldg(w + (j - r - u)), v[u], s);
    S[i] = s;
}

__global__ void __launch_bounds__(N64_T) k_near64_pre(const double *__restrict__ rows, int64_t P, int j0,
                                                      const double *__restrict__ wlag, int64_t wstride,
                                                      const int *__restrict__ cta_col, const double *init, double *out)
{
    const int64_t i = (int64_t)blockIdx.x * N64_T + threadIdx.x;
    if (i >= P) return;
    const double *w = wlag;
    if (cta_col) w += (int64_t)cta_col[blockIdx.x / (512 / N64_T)] * wstride;
    double s[NEAR_SUB];
#pragma unroll
    for (int u = 0; u < NEAR_SUB; ++u) s[u] = init ? init[(int64_t)u * P + i] : 0.0;
    for (int r = 0; r < j0; r += NEAR_SUB) {             // j0 is a multiple of NEAR_SUB
        double v[NEAR_SUB];
#pragma unroll
        for (int q = 0; q < NEAR_SUB; ++q) v[q] = __ldcg(rows + (int64_t)(r + q) * P + i);
#pragma unroll
        for (int q = 0; q < NEAR_SUB; ++q)
#pragma unroll
            for (int u = 0; u < NEAR_SUB; ++u) s[u] = fma(__ldg(w + (j0 + u - r - q)), v[q], s[u]);
    }
#pragma unroll
    for (int u = 0; u < NEAR_SUB; ++u) out[(int64_t)u * P + i] = s[u];
}

int launch_near64_pre(cudaStream_t st, const double *rows, int64_t P, int j0, const double *wlag, const double *init,
                      double *out, const int *cta_col, int64_t wstride)
{
    k_near64_pre<<<(unsigned)((P + N64_T - 1) / N64_T), N64_T, 0, st>>>(rows, P, j0, wlag, wstride, cta_col, init, out);
    FPDE_LAUNCHED(1);
    return FPDE_OK;
}

int launch_near64(cudaStream_t st, const double *rows, int64_t P, int j, const double *wlag, const double *init,
                  double *S, const int *cta_col, int64_t wstride)
{
    k_near64<<<(unsigned)((P + N64_T - 1) / N64_T), N64_T, 0, st>>>(rows, P, j, wlag, wstride, cta_col, init, S);
    FPDE_LAUNCHED(1);
    return FPDE_OK;
}

bool slices7_hold(const double *w, int64_t lags)
{
    constexpr double NEAR = 256.0, ALL = 1099511627776.0;          // 2^8, 2^40
    if (lags < 1) return true;
    std::vector<double> a(lags), hi(lags), lo(lags);
    for (int64_t l = 0; l < lags; ++l) {
        a[l] = std::fabs(w[l + 1]);
        if (!(a[l] >= 2.2250738585072014e-308) || !std::isfinite(a[l])) return false;
    }
    const auto all = std::minmax_element(a.begin(), a.end());
    if (*all.second > ALL * *all.first) return false;
    // extremes of [l, l + 63]: from l to its group's end and from the next group's start to l + 63
    for (int64_t l = lags - 1; l >= 0; --l) {
        const bool end = l == lags - 1 || l % 64 == 63;
        hi[l] = end ? a[l] : std::max(a[l], hi[l + 1]);
        lo[l] = end ? a[l] : std::min(a[l], lo[l + 1]);
    }
    double h = 0.0, m = 0.0;
    for (int64_t l = 0; l < lags; ++l) {
        h = l % 64 == 0 ? a[l] : std::max(h, a[l]);
        m = l % 64 == 0 ? a[l] : std::min(m, a[l]);
        const int64_t first = std::max<int64_t>(l - 63, 0);
        if (std::max(h, hi[first]) > NEAR * std::min(m, lo[first])) return false;
    }
    return true;
}

int hist7_alloc(cudaStream_t st, Hist7 *h, FarPlan7 *p, int64_t nodes, int64_t P, int max_steps, int w_tiles, int far_parts)
{
    h->rows = (nodes + 127) / 128 * 128;
    h->n_delta = (max_steps - 1) / 64;
    h->w_tiles = w_tiles;
    // one allocation: eighteen cost a line's creation 0.2 ms
    size_t total = 0;
    auto place = [&](size_t bytes) {
        const size_t at = total;
        total += (bytes + 255) / 256 * 256;
        return at;
    };
    const size_t n_a = (size_t)h->rows * h->n_delta, n_w = (size_t)w_tiles * 64 * h->n_delta;
    size_t at_a[7], at_w[7];
    for (int q = 0; q < 7; ++q) {
        at_a[q] = place(n_a * 128);
        at_w[q] = place(n_w * 128);
    }
    const size_t at_pA = place(n_a * sizeof(int16_t)), at_eA = place((size_t)h->rows * sizeof(int16_t)),
                 at_eW = place((size_t)w_tiles * 64 * sizeof(int16_t)), at_sW = place(n_w * sizeof(float)),
                 at_ring = place((size_t)64 * P * sizeof(double)),
                 at_far = place((size_t)far_parts * 64 * P * sizeof(double));
    size_t avail = 0, all = 0;
    FPDE_CUDA(cudaMemGetInfo(&avail, &all));
    if (total > avail / 2) return set_error(FPDE_ERR_NOMEM, "digit slices: %zu bytes of %zu free", total, avail);
    int rc = dev_alloc(&h->base, total);
    if (!rc) {
        char *p0 = (char *)h->base;
        for (int q = 0; q < 7; ++q) {
            h->a[q] = (uint16_t *)(p0 + at_a[q]);
            h->w[q] = (uint16_t *)(p0 + at_w[q]);
        }
        h->pA = (int16_t *)(p0 + at_pA);
        h->eA = (int16_t *)(p0 + at_eA);
        h->eW = (int16_t *)(p0 + at_eW);
        h->sW = (float *)(p0 + at_sW);
        h->ring = (double *)(p0 + at_ring);
        h->far = (double *)(p0 + at_far);
    }
    if (!rc) {
        const void *a[7], *w[7];
        for (int q = 0; q < 7; ++q) { a[q] = h->a[q]; w[q] = h->w[q]; }
        rc = far_plan7_init(p, a, h->rows, h->n_delta, w, w_tiles);
    }
    // rows past the nodes are never converted: their (unused) sums only need readable exponents. On the
    // context's stream: it does not wait for the default one, where a clear could still be queued when the
    // first blocks are converted
    if (!rc && (cudaMemsetAsync(h->pA, 0, (size_t)h->rows * h->n_delta * sizeof(int16_t), st) != cudaSuccess ||
                cudaMemsetAsync(h->eA, 0, (size_t)h->rows * sizeof(int16_t), st) != cudaSuccess))
        rc = set_error(FPDE_ERR_CUDA, "digit slices: clearing the exponents failed");
    if (rc) hist7_free(h);
    return rc;
}

void hist7_free(Hist7 *h)
{
    dev_free(h->base);
    *h = Hist7();
}

int hist7_weights(cudaStream_t st, const Hist7 &h, const double *wlag, int64_t wstride)
{
    Slices7 o;
    for (int q = 0; q < 7; ++q) o.p[q] = h.w[q];
    k_wgen7<<<dim3((unsigned)h.w_tiles, 64), 64, 0, st>>>(wlag, wstride, o, h.n_delta, h.sW, h.eW);
    FPDE_LAUNCHED(1);
    return FPDE_OK;
}

int hist7_convert(cudaStream_t st, const Hist7 &h, const double *rows64, int64_t P, int64_t nvalid, int64_t n0)
{
    Slices7 o;
    for (int q = 0; q < 7; ++q) o.p[q] = h.a[q];
    const int64_t threads = nvalid * CONV7_LANES;
    k_convert7<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(rows64, P, nvalid, o, h.rows, h.pA, (int)(n0 / 64) - 1,
                                                                  h.eA);
    FPDE_LAUNCHED(1);
    return FPDE_OK;
}

int launch_block_prep3(cudaStream_t st, const SplitPrep3 &p, int64_t n0, bool weights)
{
    if (n0 >= 64) {
        const int blk = (int)(n0 / 64) - 1;
        const int64_t threads = p.nvalid * CONV_LANES;
        k_convert3<<<(unsigned)((threads + 255) / 256), 256, 0, st>>>(p.ring, p.P, p.nvalid, p.hist[0], p.hist[1],
                                                                      p.hist[2], p.rows, p.pA, blk);
        FPDE_LAUNCHED(1);
    }
    if (weights && n0 / 64 + (p.n_grp > 0 ? p.n_grp : 1) - 1 > 0) {
        const int ng = p.n_grp > 0 ? p.n_grp : 1;
        dim3 g((unsigned)(n0 / 64 + ng - 1), 64 * ng, (unsigned)(p.ncols > 0 ? p.ncols : 1));
        // columns stop at the slices' pitch: a later block of the super-block exists only below the
        // step capacity, so its contraction never reaches past it
        const int kt_lim = (int)std::min<int64_t>(p.ld / 64, p.ldp);
        k_wgen3<<<g, 64, 0, st>>>(p.wlag, p.wstride, (int)n0, p.w[0], p.w[1], p.w[2], p.pW, ng, kt_lim);
        FPDE_LAUNCHED(1);
    }
    return FPDE_OK;
}

int launch_block_prep(cudaStream_t st, const SplitPrep &p, int64_t n0)
{
    const int blk = (int)(n0 / 64) - 1;          // the block that has just finished
    if (!p.bf16) {
        FPDE_CUDA(cudaMemsetAsync(p.slots + blk, 0, sizeof(unsigned long long), st));
        k_absmax<<<512, 256, 0, st>>>(p.ring, 64 * p.P, p.slots + blk);
        FPDE_LAUNCHED(1);
    }
    k_convert<<<(unsigned)((p.nvalid + 63) / 64), 256, 0, st>>>(p.ring, p.P, p.nvalid, p.slots + blk, p.exps, blk,
                                                                p.hist_hi, p.hist_lo, p.ld, n0 - 64, p.bf16);
    FPDE_LAUNCHED(1);
    dim3 g((unsigned)((n0 + 255) / 256), 64);
    k_wgen<<<g, 256, 0, st>>>(p.wlag, (int)n0, p.exps, p.w_hi, p.w_lo, p.ld, p.bf16, p.out_scale);
    FPDE_LAUNCHED(1);
    return FPDE_OK;
}

}  // namespace fpde
