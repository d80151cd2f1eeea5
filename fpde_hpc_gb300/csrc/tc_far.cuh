// Far-history tensor-core contraction (tc_far.cu): plan and launch helpers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace fpde {

constexpr int FAR_MAX_SPLITS = 4;   // K splits (FP64 partial slices) per contraction
constexpr int FAR_MAX_SUPER = 4;    // 64-step weight groups per far super-block

struct FarPlan {
    alignas(64) unsigned char maps[4 * 128];   // four CUtensorMap (a_hi, a_lo, w_hi, w_lo)
    int64_t rows = 0;
    uint32_t idesc = 0;
};

// a_hi/a_lo: [rows][lda] 16-bit (rows % 128 == 0, lda % 64 == 0); w_hi/w_lo: [64][ldw].
int far_plan_init(FarPlan *p, const void *a_hi, const void *a_lo, int64_t rows, int64_t lda, const void *w_hi,
                  const void *w_lo, int64_t ldw, int bf16);
// C[split*ldc_split + j*ldc_col + row] = out_scale * sum over the split's K range.
// out_scale_ptr (device, may be null) multiplies out_scale at run time.
int far_launch(cudaStream_t st, const FarPlan *p, int k_cols, double *C, int64_t ldc_split, int64_t ldc_col,
               int splits, double out_scale, const double *out_scale_ptr, unsigned *flags);
int far_splits(int kt_total, int64_t rows);

// Exact-slice variant: three bf16 slices per operand, per-(row, k-tile) exponents pA (int8) and
// per-(j, k-tile) scales pW = 2^e (float: the epilogue multiplies by them without rebuilding each
// power of two). Tile-major (what the engines keep): slices [ld/64][rows][64], pA [k-tile][rows], pW
// [k-tile][w_rows]. Row-major (the public contraction): slices [rows][ld], pA and pW [rows][ldp].
struct FarPlan3 {
    alignas(64) unsigned char maps[9 * 128];
    int64_t rows = 0;
    int64_t w_rows = 0;                        // rows of the W slices (64 per weight tile)
    bool tiled = true;
    uint32_t idesc = 0, idesc2 = 0;            // MMA instruction descriptors for N = 64 and 128
};
// w_tiles: number of 64-row weight tiles in the W slices (columns of an ensemble; 1 otherwise).
int far_plan3_init(FarPlan3 *p, const void *const a[3], int64_t rows, int64_t lda, const void *const w[3],
                   int64_t ldw, int w_tiles = 1, bool tiled = true);
// Writes each partial as a float pair (hi, lo) into the 8-byte slot of C (the fold's float-
// float value; hi + lo is exact in FP64): read it with ff_to_double.
// wcol (device, may be null): per 128-row tile the weight tile (column of an ensemble) it uses,
// whose 64 rows start at row wcol[tile] * 64 of the W slices and of pW.
// k_begin (a multiple of 64): the contraction covers history columns [k_begin, k_cols) only
// (a restricted history window); the splits divide that range.
// n_grp, grp0: every row tile is contracted against the n_grp weight tiles grp0 .. grp0+n_grp-1
// (64 steps each, W rows (grp0+g)*64 ..; plus wcol's tile) and writes group g's 64 steps at
// C + g*64*ldc_col: one launch covers n_grp*64 upcoming steps (a super-block).
int far3_launch(cudaStream_t st, const FarPlan3 *p, int k_cols, double *C, int64_t ldc_split, int64_t ldc_col,
                int splits, const int8_t *pA, const float *pW, int64_t ldp, unsigned *flags,
                const int *wcol = nullptr, int k_begin = 0, int n_grp = 1, int grp0 = 0);

// FP64 form (seven slices of 9 bits; tc_far.cu): slices, exponents and weight tables of a history. The
// weights w[n0 + j - t] of a block at n0 depend on its distance from a k-tile only, so their tiles
// (distance 1 .. n_delta blocks) are formed once.
struct Hist7 {
    void *base = nullptr;  // the one allocation that holds all of them
    // half-tile-major slices: a box of the product (128 nodes or 64 steps x 32 columns) is contiguous
    uint16_t *a[7] = {};   // [2 n_delta half blocks][rows][32]
    uint16_t *w[7] = {};   // [2 n_delta][w_tiles 64][32]: column c of distance d, half c / 32: lag 64 d + j - c
    int16_t *pA = nullptr, *eA = nullptr;      // [n_delta][rows] exponents per (block, node); [rows] largest so far
    int16_t *eW = nullptr;                     // [w_tiles][64] largest exponent of the step's weights
    float *sW = nullptr;                       // [w_tiles][n_delta][64] 2^(exponent - eW)
    double *ring = nullptr, *far = nullptr;    // the block's FP64 rows [64][P], far sums [far_parts][64][P]
    int64_t rows = 0;
    int n_delta = 0, w_tiles = 1;
};
constexpr int PE7_ZERO = -4096, PE7_NONFINITE = 4096;   // exponents of an all-zero block, of one with Inf or NaN
struct FarPlan7 {
    alignas(64) unsigned char maps[14 * 128];
    int64_t rows = 0;
    uint32_t idesc = 0;
};
// Allocate for `nodes` rows and max_steps columns, free. One allocation, made last by the creations, so that
// FPDE_ERR_NOMEM leaves nothing behind and the FP64 rows can take its place (other errors are errors). It is
// also returned where the slices would take more than half of the free memory: they need 14 bytes per node and
// step against the rows' 8, and a second object of the size has to fit as it does with rows.
int hist7_alloc(cudaStream_t st, Hist7 *h, FarPlan7 *p, int64_t nodes, int64_t P, int max_steps, int w_tiles, int far_parts);
void hist7_free(Hist7 *h);
// Weight tiles from w[lag] (w_tiles rows of wstride values, lag < 64 n_delta + 64), once.
int hist7_weights(cudaStream_t st, const Hist7 &h, const double *wlag, int64_t wstride);
// The finished block [n0 - 64, n0) of increments (64 rows of P) into the slices.
int hist7_convert(cudaStream_t st, const Hist7 &h, const double *rows64, int64_t P, int64_t nvalid, int64_t n0);
// Whether the slices hold the sums of the lag weights w[1 .. lags] with FP64's accuracy. A block's increments
// and a tile's weights are fixed-point numbers of 62 bits below the largest, so a small product keeps
// few bits beside a large increment; that is no loss while the large one enters the same sum with a weight that
// is not much smaller, and it is one where it carries none (a window) or hardly any. So: no weight is 0, any
// 64 neighbouring ones lie within a factor of 2^8 (1 at most 45 for Caputo weights of any order in (0, 1)) and all
// within 2^40 (the accumulators' floats reach 2^-100 below the largest block and tile). A window of 3 lags in
// which increments fell by 1.4 binary orders per step was off by 0.93 of the state, weights of 2^-l by 5e-9.
bool slices7_hold(const double *w, int64_t lags);
// out[u P + i] = init[u P + i] + sum_{0 <= r < j0} w[j0 + u - r] rows_r[i], u < 8, in FP64; init may be null (0)
// or out itself. j0 is a multiple of 8. Per-column weights with cta_col.
int launch_near64_pre(cudaStream_t st, const double *rows, int64_t P, int j0, const double *wlag, const double *init,
                      double *out, const int *cta_col = nullptr, int64_t wstride = 0);
// S[i] = init[i] + sum_{j - j % 8 <= r < j} w[j - r] rows_r[i] in FP64 (init may be null).
int launch_near64(cudaStream_t st, const double *rows, int64_t P, int j, const double *wlag, const double *init,
                  double *S, const int *cta_col = nullptr, int64_t wstride = 0);
int far_plan7_init(FarPlan7 *p, const void *const a[7], int64_t rows, int n_tiles, const void *const w[7], int w_tiles);
// C[split ldc_split + j ldc_col + row] = sum over the split's share of columns [0, k_cols) of
// A[row][t] w[k_cols + j - t], j < 64, in FP64.
int far7_launch(cudaStream_t st, const FarPlan7 *p, const Hist7 &h, int k_cols, double *C, int64_t ldc_split,
                int64_t ldc_col, int splits, unsigned *flags, const int *wcol = nullptr);

// float -> double from the bits (integer instructions only; exact for every float).
__device__ __forceinline__ double f2d_bits(float x)
{
    const uint32_t b = (uint32_t)__float_as_int(x);
    const bool tiny = (b & 0x7F800000u) == 0;               // zero or subnormal: scaled by 2^64 first
    const uint32_t y = tiny ? (uint32_t)__float_as_int(__fmul_rn(x, 18446744073709551616.f)) : b, m = y & 0x7FFFFFFFu;
    uint32_t hi = (m >> 3) + (tiny ? (896u - 64u) << 20 : m >= 0x7F800000u ? 1792u << 20 : 896u << 20);
    hi = (m == 0 ? 0u : hi) | (b & 0x80000000u);
    return __hiloint2double((int)hi, (int)(y << 29));
}
// A far-contraction slot (float pair) as one double: hi + lo, exact.
__device__ __forceinline__ double ff_to_double(double slot)
{
    const float2 v = *reinterpret_cast<const float2 *>(&slot);
    return f2d_bits(v.x) + f2d_bits(v.y);
}

}  // namespace fpde
