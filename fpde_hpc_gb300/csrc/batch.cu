// Ensemble of independent 1D Caputo columns (fpde_batch_*): many lines of different length,
// order and coefficients advanced together, two or three kernels per time step for the whole ensemble.
//
// Layout in HBM: the columns' nodes are concatenated, column c occupying
// [off_c, off_c + P_c) with P_c = N_c + 1 rounded up to 512, so that every CTA of the
// history sum (256 threads x 2 nodes) lies inside one column. The increments are one
// time-major table D[t][sum_c P_c]; padding nodes stay zero.
//
// Per time step n:
//   1. k_batch_partial : part[ks][q] = sum_t w_c[n-t] D_t[q], the column's lag weights picked
//                        per CTA (one flat grid over all nodes: balanced by construction)
//   2. k_batch_sweep   : Thomas (fpde_hpc_1d.cpp al1/bt1/U1 :4002-4027, :4585-4590, :4683-4724) inside
//                        every chunk of up to 1,024 nodes of a column from zero carries: the chunk's
//                        solution, its last y and first u; the column's last chunk to finish solves
//                        the column's chunk-level recurrences for every chunk's carries
//   3. k_batch_join    : u = u^chunk + c_in KF + c_out CB, writing U and D_n (columns of at most 1,024
//                        intervals, all of them: done by the sweep)
// FP64 where the digit slices and weight tiles fit and every column's weights allow them: step 1 becomes k_far_tc7 per 64-step block, k_near64_pre
// per 8 steps and k_near64 per step, as for the 3D grids.
// Split path (FPDE_PREC_SPLIT_BF16X3): step 1 becomes, per 64-step block, the exact
// three-slice tensor-core contraction of all history before the block with one weight tile
// per column (tc_far.cu; each 128-row tile picks its column's tile), and per step the near
// history in float-float from a 64-row float-pair ring (k_near_pre_ff, k_near_history_sub); the solve
// writes each increment to that ring and to the FP64 one the conversion reads.
// The alpha recurrence is time-invariant and precomputed on the host per column.
#include <algorithm>
#include <cmath>
#include <map>
#include <string>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "graph_cache.cuh"
#include "scan.cuh"
#include "tc_far.cuh"
#include "ff.cuh"

namespace fpde {

struct ColInfo {
    int64_t off;              // first node of the column in the concatenated node space
    int N;                    // intervals (nodes 0..N; nodes 0..N-1 are swept)
    int chunk0, nchunk;       // the column's chunks
    double lam, g0, gN, dLN, AlN;
    int rkind;
    int pad;
};
struct ChunkInfo {
    int64_t off;              // first node in the concatenated node space (a multiple of 512)
    int n, col, idx;          // nodes, column, position in the column
    int pad;
};

// col_lag (may be null): the lags each column keeps under restricted summing; rows older than
// n - col_lag[c] carry zero weights and are skipped (adding a zero-weight term changes nothing).
__global__ void __launch_bounds__(256) k_batch_partial(const double2 *__restrict__ D, int64_t P2, int n,
                                                       const double *__restrict__ wall, int64_t wstride,
                                                       int64_t woff, const int *__restrict__ cta_col,
                                                       const int *__restrict__ col_lag, double2 *__restrict__ part)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int ks = blockIdx.y, KS = gridDim.y;
    const int t0 = (int)((int64_t)n * ks / KS), t1 = (int)((int64_t)n * (ks + 1) / KS);
    if (i >= P2) return;
    const int c = cta_col[blockIdx.x];
    const double *wt = wall + (int64_t)c * wstride + woff;                       // wt[t] = w_c[n - t]
    double ax = 0.0, ay = 0.0;
    int t = col_lag ? max(t0, n - col_lag[c]) : t0;
    for (; t + 8 <= t1; t += 8) {
        double2 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = __ldcs(D + (int64_t)(t + u) * P2 + i);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const double w = __ldg(wt + t + u);
            ax = fma(w, v[u].x, ax);
            ay = fma(w, v[u].y, ay);
        }
    }
    for (; t < t1; ++t) {
        const double2 v = __ldcs(D + (int64_t)t * P2 + i);
        const double w = __ldg(wt + t);
        ax = fma(w, v.x, ax);
        ay = fma(w, v.y, ay);
    }
    part[(int64_t)ks * P2 + i] = make_double2(ax, ay);
}

// One step of every column, cut into chunks of CN nodes so that the work per CTA is even whatever the
// columns' lengths (one CTA per column left most SMs idle behind the longest columns: 153 us per step
// for 512 columns of 2.1 M nodes, and its segments were read with strides of up to 256 bytes). Bound
// by the FP64 pipe: 6 operations per node for the sweeps, about 1.5 for the scans, 3 to finish.
// Measured on that ensemble: sweep 56 us (FP64 pipe 59 % busy; six CTAs per SM, four took 60 us),
// join 18 us.
constexpr int CT = 128, CW = CT / 32;    // threads of a chunk
constexpr int CQ = 8;                    // nodes per thread
constexpr int CN = CT * CQ;              // nodes per chunk

// 8 consecutive doubles at a 16-byte aligned address
__device__ __forceinline__ void load8(const double *p, double (&v)[CQ])
{
#pragma unroll
    for (int k = 0; k < CQ; k += 2) {
        const double2 x = __ldcg(reinterpret_cast<const double2 *>(p + k));
        v[k] = x.x;
        v[k + 1] = x.y;
    }
}

struct BatchSweepArgs {
    const ColInfo *cols;
    const ChunkInfo *chunks;
    const double *ga, *g, *al;           // gA, g, Al per node (0, 0, Al[1] at a column's first node)
    const double *lane;                  // [12][chunks CT]: 5 forward level products, prefix, 5 backward, suffix
    const double *warp;                  // [chunks][2][CW]: the warps' forward and backward products
    int64_t nlane;                       // chunks CT
    const double *part;
    int KS;
    int64_t pstride;
    double *U;
    double *Y;                           // the chunk's zero-carry solution
    double *agg;                         // [chunks][2]: last y, first u; then the chunk's carries c_in, c_out
    const double *cmap;                  // [chunks][3]: product of gA, and KF, CB at the chunk's first node
    double *uN;                          // per column: U[N-1] before the step, then U[N] after it
    unsigned *count;                     // per column: chunks done in this step
    const double *CB;                    // single-chunk columns: as in BatchJoinArgs
    double *Drow;
    float2 *Drowf;
};

// The right end (U1 :4685-4719) from y at node N-1 and the old U[N-1].
__device__ __forceinline__ double batch_right_end(const ColInfo &c, double yN, double uNm1)
{
    if (c.rkind == FPDE_BC_DIRICHLET) return c.gN;
    if (fabs(yN) > 1e-15) return (fabs(1.0 - c.AlN) > 1e-15) ? (yN + c.gN * c.dLN) / (1.0 - c.AlN) : uNm1;
    return (fabs(1.0 - c.AlN) > 1e-15) ? 0.0 : uNm1;
}

// One warp: the chunk-level recurrences of a column (at most 17 chunks up to 16,384 intervals, one per
// lane). agg[k] (last y, first u of chunk k from zero carries) becomes chunk k's carries.
__device__ void batch_carries(const ColInfo &c, int col, const BatchSweepArgs &p, int lane)
{
    const int nch = c.nchunk, per = (nch + 31) / 32;
    const int a = min(lane * per, nch), b = min(a + per, nch);
    double *ag = p.agg + 2 * (int64_t)c.chunk0;
    const double *cm = p.cmap + 3 * (int64_t)c.chunk0;
    double P = 1.0, X = 0.0;                             // y after this lane's chunks = P y_before + X
    for (int k = a; k < b; ++k) {
        const double pk = __ldg(cm + 3 * k);
        X = fma(pk, X, __ldcg(ag + 2 * k));
        P *= pk;
    }
    warp_scan_up(P, X, lane);
    const double yN = __shfl_sync(FULL, X, 31);          // Bt[N]
    double y = __shfl_up_sync(FULL, X, 1);
    if (lane == 0) y = 0.0;
    double Q = 1.0, V = 0.0;                             // u at this lane's first chunk = Q u_after + V
    for (int k = a; k < b; ++k) {
        const double yl = __ldcg(ag + 2 * k), v = fma(__ldg(cm + 3 * k + 1), y, __ldcg(ag + 2 * k + 1));
        V = fma(Q, v, V);
        Q *= __ldg(cm + 3 * k + 2);
        __stcg(ag + 2 * k, y);                           // c_in
        __stcg(ag + 2 * k + 1, v);
        y = fma(__ldg(cm + 3 * k), y, yl);
    }
    const double uN = batch_right_end(c, yN, __ldcg(p.uN + col));
    warp_scan_down(Q, V, lane);
    double u = __shfl_down_sync(FULL, fma(Q, uN, V), 1);          // u after this lane's chunks
    if (lane == 31) u = uN;
    for (int k = b - 1; k >= a; --k) {
        const double v = __ldcg(ag + 2 * k + 1);
        __stcg(ag + 2 * k + 1, u);                       // c_out
        u = fma(__ldg(cm + 3 * k + 2), u, v);
    }
    if (lane == 0) __stcg(p.uN + col, uN);
}

// The scans' products are time-invariant and come from tables, so a scan level is one shuffle and one
// multiply-add; carries enter by a second sweep (the same operation count as adding responses,
// without their loads). ONE: every column is one chunk, which then needs no other's carries and finishes the
// step itself, to the same bits as the join. Without that, ensembles of short columns took longer than with one
// CTA per column (split, 400 steps, per step: 8 columns of 70 nodes 16.7 us against 13.9, 64 of 500 19.0
// against 17.4); with it 12.4 and 12.7.
template <bool ONE>
__global__ void __launch_bounds__(CT, ONE ? 4 : 6) k_batch_sweep(BatchSweepArgs p)
{
    __shared__ double sX[2][CW], s_end[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const ChunkInfo ch = p.chunks[blockIdx.x];
    const ColInfo *c = p.cols + ch.col;
    const int i0 = tid * CQ, cnt = min(max(ch.n - i0, 0), CQ);
    const int64_t q = ch.off + (cnt > 0 ? i0 : 0);
    const int64_t T = (int64_t)blockIdx.x * CT + tid;
    double h[CQ], ga[CQ], al[CQ], uo[ONE ? CQ : 1];
    {
        double u[CQ], g[CQ], s[CQ];
        load8(p.U + q, u);
        load8(p.g + q, g);
        load8(p.ga + q, ga);
        load8(p.al + q, al);
#pragma unroll
        for (int k = 0; k < CQ; ++k) s[k] = 0.0;
        if (p.KS > 0) load8(p.part + q, s);
        for (int r = 1; r < p.KS; ++r) {
            double v[CQ];
            load8(p.part + (int64_t)r * p.pstride + q, v);
#pragma unroll
            for (int k = 0; k < CQ; ++k) s[k] += v[k];
        }
        const double lam = c->lam;
#pragma unroll
        for (int k = 0; k < CQ; ++k) h[k] = g[k] * fma(lam, u[k], -s[k]);       // -g Om
        if (ch.idx == 0 && tid == 0) h[0] = c->g0;                             // Bt[1]
        if constexpr (ONE) {
#pragma unroll
            for (int k = 0; k < CQ; ++k) uo[k] = u[k];
            if (tid == 0) s_end[1] = __ldcg(p.U + ch.off + ch.n - 1);
        } else if (tid == 0 && ch.idx == c->nchunk - 1) {
            p.uN[ch.col] = __ldcg(p.U + ch.off + ch.n - 1);
        }
    }
    const double *lp = p.lane + T, *wp = p.warp + (int64_t)blockIdx.x * (2 * CW);
    double pf[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) pf[k] = __ldg(lp + k * p.nlane);
    // forward: y_i = gA y_{i-1} + h_i
    double x = 0.0;
#pragma unroll
    for (int k = 0; k < CQ; ++k)
        if (k < cnt) x = fma(ga[k], x, h[k]);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const double xp = __shfl_up_sync(FULL, x, 1 << k);
        if (lane >= (1 << k)) x = fma(pf[k], xp, x);
    }
    double xe = __shfl_up_sync(FULL, x, 1);
    if (lane == 0) xe = 0.0;
    if (lane == 31) sX[0][warp] = x;
    __syncthreads();
    double cw = 0.0;
    for (int w = 0; w < warp; ++w) cw = fma(__ldg(wp + w), cw, sX[0][w]);
    x = fma(pf[5], cw, xe);                                                    // y before this thread's nodes
#pragma unroll
    for (int k = 0; k < CQ; ++k)
        if (k < cnt) h[k] = x = fma(ga[k], x, h[k]);                           // y
    if (cnt > 0 && i0 + cnt == ch.n) {
        if constexpr (ONE) s_end[0] = x;
        else p.agg[2 * (int64_t)blockIdx.x] = x;
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) pf[k] = __ldg(lp + (6 + k) * p.nlane);
    // backward: u_i = Al u_{i+1} + y_i
    x = 0.0;
#pragma unroll
    for (int k = CQ - 1; k >= 0; --k)
        if (k < cnt) x = fma(al[k], x, h[k]);
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        const double xn = __shfl_down_sync(FULL, x, 1 << k);
        if (lane + (1 << k) < 32) x = fma(pf[k], xn, x);
    }
    xe = __shfl_down_sync(FULL, x, 1);
    if (lane == 31) xe = 0.0;
    if (lane == 0) sX[1][warp] = x;
    __syncthreads();
    cw = 0.0;
    for (int w = CW - 1; w > warp; --w) cw = fma(__ldg(wp + CW + w), cw, sX[1][w]);
    x = fma(pf[5], cw, xe);                                                    // u after this thread's nodes
#pragma unroll
    for (int k = CQ - 1; k >= 0; --k)
        if (k < cnt) h[k] = x = fma(al[k], x, h[k]);                           // u^chunk
    if constexpr (ONE) {
        const double uN = batch_right_end(*c, s_end[0], s_end[1]);
        double cb[CQ];
        load8(p.CB + q, cb);
#pragma unroll
        for (int k = 0; k < CQ; ++k) {
            h[k] = fma(uN, cb[k], h[k]);                                       // the new state, then its increment
            uo[k] = h[k] - uo[k];
        }
        if (cnt == CQ) {
#pragma unroll
            for (int k = 0; k < CQ; k += 2) {
                *reinterpret_cast<double2 *>(p.U + q + k) = make_double2(h[k], h[k + 1]);
                *reinterpret_cast<double2 *>(p.Drow + q + k) = make_double2(uo[k], uo[k + 1]);
                if (p.Drowf) {
                    const float2 f0 = d2ff(uo[k]), f1 = d2ff(uo[k + 1]);
                    *reinterpret_cast<float4 *>(p.Drowf + q + k) = make_float4(f0.x, f0.y, f1.x, f1.y);
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < CQ; ++k)
                if (k < cnt) {
                    p.U[q + k] = h[k];
                    p.Drow[q + k] = uo[k];
                    if (p.Drowf) p.Drowf[q + k] = d2ff(uo[k]);
                }
        }
        if (tid == 0) {
            const int64_t e = ch.off + ch.n;
            const double d = uN - p.U[e];
            p.U[e] = uN;
            p.Drow[e] = d;
            if (p.Drowf) p.Drowf[e] = d2ff(d);
        }
        return;
    }
    if (tid == 0) p.agg[2 * (int64_t)blockIdx.x + 1] = x;
    if (cnt == CQ) {
#pragma unroll
        for (int k = 0; k < CQ; k += 2) *reinterpret_cast<double2 *>(p.Y + q + k) = make_double2(h[k], h[k + 1]);
    } else {
#pragma unroll
        for (int k = 0; k < CQ; ++k)
            if (k < cnt) p.Y[q + k] = h[k];
    }
    // the column's last chunk to get here joins them
    __threadfence();
    __syncthreads();
    if (warp != 0) return;
    unsigned done = 0;
    if (lane == 0) done = atomicAdd(p.count + ch.col, 1u);
    done = __shfl_sync(FULL, done, 0);
    if (done != (unsigned)c->nchunk - 1) return;
    __threadfence();
    if (lane == 0) p.count[ch.col] = 0;                                        // for the next step
    batch_carries(*c, ch.col, p, lane);
}

struct BatchJoinArgs {
    const ColInfo *cols;
    const int *cta_col;
    const double *KF, *CB;               // per node: responses of the chunk's solution to its carries
    const double *Y, *agg, *uN;
    double *U, *Drow;
    float2 *Drowf;                       // split path: the float-pair ring row
};

// 512 nodes (of one chunk) per CTA, two per thread; bound by memory (56 bytes per node).
__global__ void __launch_bounds__(256) k_batch_join(BatchJoinArgs p)
{
    const int col = p.cta_col[blockIdx.x];
    const ColInfo *c = p.cols + col;
    const int64_t q = (int64_t)blockIdx.x * 512 + 2 * threadIdx.x;
    const int i = (int)(q - c->off), N = c->N;
    if (i > N) return;
    const int64_t k = c->chunk0 + min(i / CN, c->nchunk - 1);
    const double cin = __ldg(p.agg + 2 * k), cout = __ldg(p.agg + 2 * k + 1);
    const double2 ub = __ldcs(reinterpret_cast<const double2 *>(p.Y + q)), kf = __ldg(reinterpret_cast<const double2 *>(p.KF + q)),
                  cb = __ldg(reinterpret_cast<const double2 *>(p.CB + q)), uo = *reinterpret_cast<const double2 *>(p.U + q);
    double2 u = make_double2(fma(cout, cb.x, fma(cin, kf.x, ub.x)), fma(cout, cb.y, fma(cin, kf.y, ub.y)));
    if (i == N) u.x = p.uN[col];
    if (i + 1 == N) u.y = p.uN[col];
    const double dx = u.x - uo.x, dy = u.y - uo.y;
    if (i < N) {
        *reinterpret_cast<double2 *>(p.U + q) = u;
        *reinterpret_cast<double2 *>(p.Drow + q) = make_double2(dx, dy);
        if (p.Drowf) {
            const float2 f0 = d2ff(dx), f1 = d2ff(dy);
            *reinterpret_cast<float4 *>(p.Drowf + q) = make_float4(f0.x, f0.y, f1.x, f1.y);
        }
    } else {
        p.U[q] = u.x;
        p.Drow[q] = dx;
        if (p.Drowf) p.Drowf[q] = d2ff(dx);
    }
}

}  // namespace fpde

using namespace fpde;

struct fpde_batch {
    fpde_ctx *ctx = nullptr;
    int n_cols = 0, max_steps = 0;
    int64_t Ptot = 0;
    std::vector<int64_t> off;
    std::vector<int> N;
    double *ga = nullptr, *g = nullptr, *al = nullptr;
    double *KF = nullptr, *CB = nullptr;      // per node: the chunk's responses to its carries
    double *lane = nullptr, *warp = nullptr, *cmap = nullptr;   // scan products, chunk-level maps
    double *agg = nullptr, *uN = nullptr;
    unsigned *count = nullptr;
    ChunkInfo *chunks = nullptr;
    int n_chunks = 0;
    double *U = nullptr, *U0 = nullptr, *Y = nullptr, *D = nullptr, *part = nullptr, *wall = nullptr;
    ColInfo *cols = nullptr;
    int *cta_col = nullptr;
    int *col_lag = nullptr;                   // restricted summing: lags kept per column (null: all)
    // FP64 with the far history of every 64-step block in seven bf16 slices (else the rows of D)
    bool x7 = false;
    Hist7 h7;
    FarPlan7 plan7;
    // split path
    bool split = false;
    int64_t ld16 = 0, ldp = 0, LW = 0;
    uint16_t *h3[3] = {nullptr, nullptr, nullptr}, *w3[3] = {nullptr, nullptr, nullptr};
    int8_t *pA = nullptr;
    float *pW = nullptr;
    double *ring = nullptr, *cfar = nullptr, *wlag = nullptr, *Sn = nullptr;
    float2 *ringf = nullptr, *wff = nullptr;  // the ring and every column's lag weights as float pairs
    float2 *pre = nullptr;                    // near-history sums of the current 8-step sub-block
    int *wcol = nullptr;
    FarPlan3 plan3;
    int64_t n_done = 0;
    GraphCache<int> graphs;                        // captured runs (at least GRAPH_MIN_STEPS steps)
};

namespace fpde {

static int batch_enqueue(fpde_batch *b, cudaStream_t st, int64_t n0, int steps, int64_t *nk)
{
    int64_t k = 0;
    int rc;
    for (int64_t n = n0; n < n0 + steps; ++n) {
        int KS = 0;
        const double *part = b->part;
        double *Drow;
        float2 *Drowf = nullptr;                                     // split: the float-pair ring row
        if (b->x7) {
            const int64_t nb0 = n - n % 64;
            const int j = (int)(n - nb0);
            if (j == 0 && nb0 > 0) {
                if ((rc = hist7_convert(st, b->h7, b->ring, b->Ptot, b->Ptot, nb0))) return rc;
                if ((rc = far7_launch(st, &b->plan7, b->h7, (int)nb0, b->cfar, (int64_t)64 * b->Ptot, b->Ptot, 1,
                                      b->ctx->d_flags, b->wcol)))
                    return rc;
                k += 2;
            }
            if (n >= 1) {                                            // far sums + the block's earlier rows
                // the rows before the step's 8-step sub-block go into its far sums once per sub-block
                const int j0 = j - j % NEAR_SUB;
                double *far = b->cfar + (int64_t)j * b->Ptot;
                if (j == j0 && j0 > 0) {
                    if ((rc = launch_near64_pre(st, b->ring, b->Ptot, j0, b->wlag, nb0 > 0 ? far : nullptr, far,
                                                b->cta_col, b->LW)))
                        return rc;
                    ++k;
                }
                if ((rc = launch_near64(st, b->ring, b->Ptot, j, b->wlag, nb0 > 0 || j0 > 0 ? far : nullptr, b->part,
                                        b->cta_col, b->LW)))
                    return rc;
                ++k;
                KS = 1;
            }
            Drow = b->ring + (int64_t)j * b->Ptot;
        } else if (!b->split) {
            if (n >= 1) {
                KS = choose_splits((int)n, b->Ptot);
                dim3 grid((unsigned)(b->Ptot / 512), (unsigned)KS);
                k_batch_partial<<<grid, 256, 0, st>>>((const double2 *)b->D, b->Ptot / 2, (int)n, b->wall,
                                                      b->max_steps + 1, b->max_steps - n, b->cta_col,
                                                      b->col_lag, (double2 *)b->part);
                FPDE_LAUNCHED(1);
                ++k;
            }
            Drow = b->D + n * b->Ptot;
        } else {
            const int64_t nb0 = n - n % 64;
            const int j = (int)(n - nb0);
            int splits = 0;
            if (nb0 > 0) {
                splits = far_splits((int)(nb0 / 64), b->Ptot);
                if (j == 0) {                                        // far history t < nb0, per column
                    SplitPrep3 sp;
                    sp.ring = b->ring; sp.P = b->Ptot; sp.nvalid = b->Ptot; sp.ld = b->ld16; sp.rows = b->Ptot; sp.wlag = b->wlag;
                    for (int q = 0; q < 3; ++q) { sp.hist[q] = b->h3[q]; sp.w[q] = b->w3[q]; }
                    sp.pA = b->pA; sp.pW = b->pW; sp.ldp = b->ldp; sp.ncols = b->n_cols; sp.wstride = b->LW;
                    if ((rc = launch_block_prep3(st, sp, nb0))) return rc;
                    k += 2;
                    if ((rc = far3_launch(st, &b->plan3, (int)nb0, b->cfar, (int64_t)64 * b->Ptot, b->Ptot, splits,
                                          b->pA, b->pW, b->ldp, b->ctx->d_flags, b->wcol)))
                        return rc;
                    ++k;
                }
            }
            if (n >= 1) {
                // rows older than the step's 8-step sub-block (and the far partials) once per sub-block
                const int j0 = j - j % NEAR_SUB;
                const bool use_pre = splits > 0 || j0 > 0;
                if (use_pre && j == j0) {
                    if ((rc = launch_near_pre_ff(st, b->ringf, b->Ptot, j0, b->wff, b->cfar, splits, 1, b->pre,
                                                 b->cta_col, b->LW)))
                        return rc;
                    ++k;
                }
                if ((rc = launch_near_history_sub(st, b->ringf, b->Ptot, j, b->wff, b->Sn, use_pre ? b->pre : nullptr,
                                                  b->cta_col, b->LW)))
                    return rc;
                ++k;
                KS = 1;
                part = b->Sn;
            }
            Drow = b->ring + (int64_t)j * b->Ptot;
            Drowf = b->ringf + (int64_t)j * b->Ptot;
        }
        BatchSweepArgs sa;
        sa.cols = b->cols; sa.chunks = b->chunks; sa.ga = b->ga; sa.g = b->g; sa.al = b->al;
        sa.lane = b->lane; sa.warp = b->warp; sa.nlane = (int64_t)b->n_chunks * CT;
        sa.part = part; sa.KS = KS; sa.pstride = b->Ptot; sa.U = b->U; sa.Y = b->Y; sa.agg = b->agg; sa.cmap = b->cmap;
        sa.uN = b->uN; sa.count = b->count;
        sa.CB = b->CB; sa.Drow = Drow; sa.Drowf = Drowf;
        if (b->n_chunks == b->n_cols) {                              // every column is one chunk
            k_batch_sweep<true><<<b->n_chunks, CT, 0, st>>>(sa);
            FPDE_LAUNCHED(1);
            ++k;
            continue;
        }
        k_batch_sweep<false><<<b->n_chunks, CT, 0, st>>>(sa);
        FPDE_LAUNCHED(1);
        BatchJoinArgs ja;
        ja.cols = b->cols; ja.cta_col = b->cta_col; ja.KF = b->KF; ja.CB = b->CB;
        ja.Y = b->Y; ja.agg = b->agg; ja.uN = b->uN; ja.U = b->U; ja.Drow = Drow; ja.Drowf = Drowf;
        k_batch_join<<<(unsigned)(b->Ptot / 512), 256, 0, st>>>(ja);
        FPDE_LAUNCHED(1);
        k += 2;
    }
    *nk = k;
    return FPDE_OK;
}

}  // namespace fpde

extern "C" {

int fpde_batch_destroy(fpde_batch *b)
{
    if (!b) return FPDE_OK;
    if (b->ctx) {
        cudaSetDevice(b->ctx->device);
        cudaStreamSynchronize(b->ctx->stream);
    }
    b->graphs.clear();
    if (b->x7) b->ring = b->cfar = nullptr;                            // parts of the slices' allocation
    for (double *p : {b->ga, b->g, b->al, b->lane, b->warp, b->cmap, b->agg, b->uN, b->KF, b->CB, b->U, b->U0, b->Y, b->D,
                      b->part, b->wall, b->ring, b->cfar, b->wlag, b->Sn})
        dev_free(p);
    for (int q = 0; q < 3; ++q) {
        dev_free(b->h3[q]);
        dev_free(b->w3[q]);
    }
    hist7_free(&b->h7);
    dev_free(b->pA);
    dev_free(b->pW);
    dev_free(b->ringf);
    dev_free(b->pre);
    dev_free(b->wff);
    dev_free(b->wcol);
    dev_free(b->cols);
    dev_free(b->chunks);
    dev_free(b->count);
    dev_free(b->cta_col);
    dev_free(b->col_lag);
    delete b;
    return FPDE_OK;
}

int fpde_batch_create(fpde_ctx *ctx, const fpde_column_desc *cols, int n_cols, int max_steps, int precision,
                      fpde_batch **out)
{
    clear_error();
    FPDE_CHECK_ARG(out && cols && n_cols > 0, "bad arguments");
    *out = nullptr;
    int rc = ctx_enter(ctx);
    if (rc) return rc;
    FPDE_CHECK_ARG(max_steps > 0, "max_steps must be positive");
    FPDE_CHECK_ARG(precision == FPDE_PREC_FP64 || precision == FPDE_PREC_SPLIT_BF16X3,
                   "ensemble: precision must be FP64 or the exact three-slice split");
    for (int c = 0; c < n_cols; ++c) {
        const fpde_column_desc &d = cols[c];
        FPDE_CHECK_ARG(d.N >= 2 && d.N <= (1 << 24), "column N out of range");
        FPDE_CHECK_ARG(d.A && d.B && d.Rlap && d.u0, "column arrays missing");
        FPDE_CHECK_ARG(d.lag_weights || (d.alpha > 0.0 && d.alpha < 1.0), "alpha must be in (0, 1)");
        FPDE_CHECK_ARG(d.tau > 0.0, "tau must be positive");
        FPDE_CHECK_ARG((d.left_kind == 0 || d.left_kind == 1) && (d.right_kind == 0 || d.right_kind == 1),
                       "bad boundary kind");
        FPDE_CHECK_ARG(std::isfinite(d.restrict_eps) && d.restrict_eps >= 0.0, "restrict_eps must be >= 0");
    }
    // restricted summing per column (time_summing :4117-4131, newest first): the lags before the
    // first one whose kb = w tau / Da falls below restrict_eps; later lags get weight 0
    std::vector<int> lag_keep(n_cols, max_steps);
    bool any_restrict = false;
    for (int c = 0; c < n_cols; ++c) {
        const fpde_column_desc &d = cols[c];
        if (d.restrict_eps <= 0.0) continue;
        const double kkk0 = d.lag_weights ? 0.0 : l1_interval_weight(d.alpha, 0.0, d.tau);
        std::vector<double> kbl(max_steps);
        for (int64_t j = 1; j <= max_steps; ++j) {
            const double w = d.lag_weights ? d.lag_weights[j] : d.Da * (kkk0 * l1_lag(d.alpha, j)) / d.tau;
            kbl[j - 1] = w * d.tau / d.Da;
        }
        int keep = max_steps;
        fpde_restricted_lags(kbl.data(), max_steps, d.restrict_eps, &keep);
        lag_keep[c] = keep;
        any_restrict = any_restrict || keep < max_steps;
    }
    clear_error();
    fpde_batch *b = new fpde_batch();
    b->ctx = ctx;
    b->n_cols = n_cols;
    b->max_steps = max_steps;
    b->off.resize(n_cols);
    b->N.resize(n_cols);
    int64_t tot = 0;
    for (int c = 0; c < n_cols; ++c) {
        b->off[c] = tot;
        b->N[c] = (int)cols[c].N;
        tot += (cols[c].N + 1 + 511) / 512 * 512;
    }
    b->Ptot = tot;
    std::vector<double> hga(tot, 0.0), hg(tot, 0.0), hal(tot, 0.0), hU(tot, 0.0);
    std::vector<double> hKF(tot, 0.0), hCB(tot, 0.0), hlane, hwarp, hmap;
    std::vector<ChunkInfo> hch;
    for (int c = 0; c < n_cols; ++c)
        for (int64_t a = 0; a < cols[c].N; a += CN) {
            ChunkInfo ci;
            ci.off = b->off[c] + a;
            ci.n = (int)std::min<int64_t>(CN, cols[c].N - a);
            ci.col = c;
            ci.idx = (int)(a / CN);
            ci.pad = 0;
            hch.push_back(ci);
        }
    b->n_chunks = (int)hch.size();
    const int64_t nlane = (int64_t)hch.size() * CT;
    hlane.assign((size_t)12 * nlane, 1.0);
    hwarp.assign(hch.size() * 2 * CW, 1.0);
    hmap.assign(hch.size() * 3, 1.0);
    int chunk0 = 0;
    std::vector<double> hw((size_t)n_cols * (max_steps + 1), 0.0);
    std::vector<ColInfo> hc(n_cols);
    std::vector<int> cta_col(tot / 512);
    for (int c = 0; c < n_cols; ++c) {
        const fpde_column_desc &d = cols[c];
        const int64_t N = d.N, o = b->off[c];
        double lam, lamR, kkk0 = 0.0;
        if (d.lag_weights) {
            lam = lamR = d.lag_weights[0];
        } else {                                                   // Om1 :4191, R :3120
            kkk0 = l1_interval_weight(d.alpha, 0.0, d.tau);
            lam = d.Da * (kkk0 / d.tau);
            lamR = d.Da * kkk0 / d.tau;
        }
        double Al = d.left_kind == FPDE_BC_FLUX ? 1.0 : 0.0;         // Al[1]
        hal[o] = Al;
        for (int64_t i = 1; i < N; ++i) {
            Al = d.B[i] / ((d.Rlap[i] + lamR) - d.A[i] * Al);        // Al[i+1]
            hal[o + i] = Al;
            hg[o + i] = Al / d.B[i];
            hga[o + i] = hg[o + i] * d.A[i];
        }
        for (int64_t i = 0; i <= N; ++i) hU[o + i] = d.u0[i];
        ColInfo &ci = hc[c];
        ci.off = o;
        ci.N = (int)N;
        ci.chunk0 = chunk0;
        ci.nchunk = (int)((N + CN - 1) / CN);
        ci.lam = lam;
        ci.g0 = d.left_value;
        ci.gN = d.right_value;
        ci.dLN = d.dLN;
        ci.AlN = Al;
        ci.rkind = d.right_kind;
        ci.pad = 0;
        for (int k = 0; k < ci.nchunk; ++k, ++chunk0) {              // time-invariant products of the chunk
            const int64_t a0 = o + (int64_t)k * CN, b0 = a0 + hch[chunk0].n;
            double pr = 1.0;
            for (int64_t i = a0; i < b0; ++i) { pr *= hga[i]; hKF[i] = pr; }
            hmap[(size_t)chunk0 * 3] = pr;
            double kf = 0.0, cb = 1.0;                                  // backward sweep of the prefix products, suffix of al
            for (int64_t i = b0 - 1; i >= a0; --i) {
                kf = hal[i] * kf + hKF[i];
                cb = hal[i] * cb;
                hKF[i] = kf;
                hCB[i] = cb;
            }
            hmap[(size_t)chunk0 * 3 + 1] = kf;
            hmap[(size_t)chunk0 * 3 + 2] = cb;
            double Pt[CT], Qt[CT];
            for (int t = 0; t < CT; ++t) {
                Pt[t] = Qt[t] = 1.0;
                for (int64_t i = a0 + (int64_t)t * CQ; i < std::min(a0 + (int64_t)(t + 1) * CQ, b0); ++i) {
                    Pt[t] *= hga[i];
                    Qt[t] *= hal[i];
                }
            }
            for (int w = 0; w < CW; ++w) {
                const double *pw = Pt + 32 * w, *qw = Qt + 32 * w;
                double F[32], B[32];                                   // running level products
                for (int l = 0; l < 32; ++l) { F[l] = pw[l]; B[l] = qw[l]; }
                const int64_t T0 = (int64_t)chunk0 * CT + 32 * w;
                for (int s = 0; s < 5; ++s) {
                    for (int l = 0; l < 32; ++l) {
                        hlane[(size_t)s * nlane + T0 + l] = F[l];
                        hlane[(size_t)(6 + s) * nlane + T0 + l] = B[l];
                    }
                    for (int l = 31; l >= (1 << s); --l) F[l] *= F[l - (1 << s)];
                    for (int l = 0; l + (1 << s) < 32; ++l) B[l] *= B[l + (1 << s)];
                }
                double pe = 1.0, qe = 1.0;
                for (int l = 0; l < 32; ++l) {
                    hlane[(size_t)5 * nlane + T0 + l] = pe;
                    pe *= pw[l];
                    hlane[(size_t)11 * nlane + T0 + 31 - l] = qe;
                    qe *= qw[31 - l];
                }
                hwarp[(size_t)chunk0 * 2 * CW + w] = pe;
                hwarp[(size_t)chunk0 * 2 * CW + CW + w] = qe;
            }
        }
        double *w = hw.data() + (size_t)c * (max_steps + 1);          // w[m] = w_c[max_steps - m]
        for (int64_t m = 0; m < max_steps; ++m) {
            const int64_t j = max_steps - m;
            w[m] = j > lag_keep[c] ? 0.0
                                   : d.lag_weights ? d.lag_weights[j] : d.Da * (kkk0 * l1_lag(d.alpha, j)) / d.tau;
        }
        for (int64_t q = o / 512; q < (o + (N + 1 + 511) / 512 * 512) / 512; ++q) cta_col[q] = c;
    }
    const bool split = precision == FPDE_PREC_SPLIT_BF16X3;
    b->split = split;
    b->LW = (int64_t)max_steps + 64 + 1;
    std::vector<double> hwl;                                           // split: w_c[lag], lag < LW
    std::vector<int> hwcol;                                            // column of each 128-row tile
    // FP64 runs of more than a block also take the tables (up to 4 GB of weight tiles, 56 KB per column
    // and distance)
    bool want7 = !split && max_steps > 64 && (int64_t)n_cols * ((max_steps - 1) / 64) * 57344 <= (4ll << 30);
    if (split || want7) {
        hwl.assign((size_t)n_cols * b->LW, 0.0);
        hwcol.assign(tot / 128, 0);
        for (int c = 0; c < n_cols; ++c) {
            const fpde_column_desc &d = cols[c];
            const double kkk0 = d.lag_weights ? 0.0 : l1_interval_weight(d.alpha, 0.0, d.tau);
            for (int64_t j = 1; j < b->LW; ++j)
                hwl[(size_t)c * b->LW + j] = j > lag_keep[c] ? 0.0
                                             : d.lag_weights ? (j <= max_steps ? d.lag_weights[j] : 0.0)
                                                             : d.Da * (kkk0 * l1_lag(d.alpha, j)) / d.tau;
            const int64_t o = b->off[c], Pc = (cols[c].N + 1 + 511) / 512 * 512;
            for (int64_t q = o / 128; q < (o + Pc) / 128; ++q) hwcol[q] = c;
        }
    }
    for (int c = 0; c < n_cols && want7; ++c) want7 = slices7_hold(hwl.data() + (size_t)c * b->LW, max_steps - 1);
    const size_t tb = (size_t)tot * sizeof(double);
    bool fail = dev_alloc((void **)&b->ga, tb) || dev_alloc((void **)&b->g, tb) || dev_alloc((void **)&b->al, tb) ||
                dev_alloc((void **)&b->lane, hlane.size() * sizeof(double)) ||
                dev_alloc((void **)&b->warp, hwarp.size() * sizeof(double)) ||
                dev_alloc((void **)&b->cmap, hmap.size() * sizeof(double)) ||
                dev_alloc((void **)&b->agg, hch.size() * 2 * sizeof(double)) ||
                dev_alloc((void **)&b->uN, (size_t)n_cols * sizeof(double)) ||
                dev_alloc((void **)&b->count, (size_t)n_cols * sizeof(unsigned)) ||
                dev_alloc((void **)&b->chunks, hch.size() * sizeof(ChunkInfo)) || dev_alloc((void **)&b->U, tb) ||
                dev_alloc((void **)&b->KF, tb) || dev_alloc((void **)&b->CB, tb) ||
                dev_alloc((void **)&b->U0, tb) || dev_alloc((void **)&b->Y, tb) ||
                dev_alloc((void **)&b->cols, hc.size() * sizeof(ColInfo)) ||
                dev_alloc((void **)&b->cta_col, cta_col.size() * sizeof(int)) ||
                (any_restrict && dev_alloc((void **)&b->col_lag, (size_t)n_cols * sizeof(int)));
    if (!fail && want7) {
        rc = dev_alloc((void **)&b->part, tb);
        if (!rc) rc = dev_alloc((void **)&b->wlag, hwl.size() * sizeof(double));
        if (!rc) rc = dev_alloc((void **)&b->wcol, hwcol.size() * sizeof(int));
        if (!rc) rc = hist7_alloc(ctx->stream, &b->h7, &b->plan7, tot, tot, max_steps, n_cols, 1);
        if (rc && rc != FPDE_ERR_NOMEM) {
            std::string keep = fpde_last_error_string();
            fpde_batch_destroy(b);
            return set_error(rc, "%s", keep.c_str());
        }
        b->x7 = rc == FPDE_OK;
        b->ring = b->h7.ring;
        b->cfar = b->h7.far;
        clear_error();
        if (!b->x7) {                                                  // FP64 rows instead (8 bytes against 14)
            dev_free(b->part);
            dev_free(b->wlag);
            dev_free(b->wcol);
            b->part = b->wlag = nullptr;
            b->wcol = nullptr;
        }
    }
    if (!fail && !b->x7 && !split) {
        fail = dev_alloc((void **)&b->D, (size_t)max_steps * tb) || dev_alloc((void **)&b->part, (size_t)KS_MAX * tb) ||
               dev_alloc((void **)&b->wall, hw.size() * sizeof(double));
    } else if (!fail && split) {
        b->ld16 = ((int64_t)max_steps + 63) / 64 * 64;
        b->ldp = b->ld16 / 64;
        const int64_t wrows = (int64_t)n_cols * 64;
        for (int q = 0; q < 3 && !fail; ++q)
            fail = dev_alloc((void **)&b->h3[q], (size_t)tot * b->ld16 * 2) ||
                   dev_alloc((void **)&b->w3[q], (size_t)wrows * b->ld16 * 2);
        fail = fail || dev_alloc((void **)&b->pA, (size_t)tot * b->ldp) ||
               dev_alloc((void **)&b->pW, (size_t)wrows * b->ldp * sizeof(float)) || dev_alloc((void **)&b->ring, (size_t)64 * tb) ||
               dev_alloc((void **)&b->cfar, (size_t)FAR_MAX_SPLITS * 64 * tb) ||
               dev_alloc((void **)&b->wlag, hwl.size() * sizeof(double)) || dev_alloc((void **)&b->Sn, tb) ||
               dev_alloc((void **)&b->ringf, (size_t)64 * tot * sizeof(float2)) ||
               dev_alloc((void **)&b->pre, (size_t)NEAR_SUB * tot * sizeof(float2)) ||
               dev_alloc((void **)&b->wff, hwl.size() * sizeof(float2)) ||
               dev_alloc((void **)&b->wcol, hwcol.size() * sizeof(int));
        if (!fail) {
            const void *a3[3] = {b->h3[0], b->h3[1], b->h3[2]}, *w3[3] = {b->w3[0], b->w3[1], b->w3[2]};
            int rcp = far_plan3_init(&b->plan3, a3, tot, b->ld16, w3, b->ld16, n_cols);
            if (rcp) {
                std::string keep = fpde_last_error_string();
                fpde_batch_destroy(b);
                return set_error(rcp, "%s", keep.c_str());
            }
        }
    }
    if (fail) {
        std::string keep = fpde_last_error_string();
        fpde_batch_destroy(b);
        return set_error(FPDE_ERR_NOMEM, "%s", keep.c_str());
    }
    cudaStream_t st = ctx->stream;
    cudaMemcpyAsync(b->ga, hga.data(), tb, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->g, hg.data(), tb, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->al, hal.data(), tb, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->lane, hlane.data(), hlane.size() * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->warp, hwarp.data(), hwarp.size() * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->cmap, hmap.data(), hmap.size() * sizeof(double), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->chunks, hch.data(), hch.size() * sizeof(ChunkInfo), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->KF, hKF.data(), tb, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->CB, hCB.data(), tb, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->U, hU.data(), tb, cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->U0, hU.data(), tb, cudaMemcpyHostToDevice, st);
    cudaMemsetAsync(b->Y, 0, tb, st);
    cudaMemsetAsync(b->count, 0, (size_t)n_cols * sizeof(unsigned), st);
    if (b->x7) {
        cudaMemsetAsync(b->ring, 0, (size_t)64 * tb, st);
        cudaMemcpyAsync(b->wlag, hwl.data(), hwl.size() * sizeof(double), cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(b->wcol, hwcol.data(), hwcol.size() * sizeof(int), cudaMemcpyHostToDevice, st);
        if ((rc = hist7_weights(st, b->h7, b->wlag, b->LW))) {
            cudaStreamSynchronize(st);
            std::string keep = fpde_last_error_string();
            fpde_batch_destroy(b);
            return set_error(rc, "%s", keep.c_str());
        }
    } else if (!split) {
        cudaMemsetAsync(b->D, 0, (size_t)max_steps * tb, st);
        cudaMemcpyAsync(b->wall, hw.data(), hw.size() * sizeof(double), cudaMemcpyHostToDevice, st);
    } else {
        const int64_t wrows = (int64_t)n_cols * 64;
        for (int q = 0; q < 3; ++q) {
            cudaMemsetAsync(b->h3[q], 0, (size_t)tot * b->ld16 * 2, st);
            cudaMemsetAsync(b->w3[q], 0, (size_t)wrows * b->ld16 * 2, st);
        }
        cudaMemsetAsync(b->pA, 0, (size_t)tot * b->ldp, st);
        cudaMemsetAsync(b->pW, 0, (size_t)wrows * b->ldp * sizeof(float), st);
        cudaMemsetAsync(b->ring, 0, (size_t)64 * tb, st);
        cudaMemsetAsync(b->cfar, 0, (size_t)FAR_MAX_SPLITS * 64 * tb, st);
        cudaMemcpyAsync(b->wlag, hwl.data(), hwl.size() * sizeof(double), cudaMemcpyHostToDevice, st);
        std::vector<float2> hwff(hwl.size());            // w = hi + lo, hi the nearest float
        for (size_t q = 0; q < hwl.size(); ++q) {
            const float hi = (float)hwl[q];
            hwff[q] = make_float2(hi, (float)(hwl[q] - (double)hi));
        }
        cudaMemcpyAsync(b->wff, hwff.data(), hwff.size() * sizeof(float2), cudaMemcpyHostToDevice, st);
        cudaMemsetAsync(b->ringf, 0, (size_t)64 * tot * sizeof(float2), st);
        cudaMemcpyAsync(b->wcol, hwcol.data(), hwcol.size() * sizeof(int), cudaMemcpyHostToDevice, st);
    }
    cudaMemcpyAsync(b->cols, hc.data(), hc.size() * sizeof(ColInfo), cudaMemcpyHostToDevice, st);
    cudaMemcpyAsync(b->cta_col, cta_col.data(), cta_col.size() * sizeof(int), cudaMemcpyHostToDevice, st);
    if (b->col_lag) cudaMemcpyAsync(b->col_lag, lag_keep.data(), (size_t)n_cols * sizeof(int), cudaMemcpyHostToDevice, st);
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        fpde_batch_destroy(b);
        return set_error(FPDE_ERR_CUDA, "batch setup: %s", cudaGetErrorString(e));
    }
    *out = b;
    return FPDE_OK;
}

int fpde_batch_run(fpde_batch *b, int steps)
{
    clear_error();
    FPDE_CHECK_ARG(b && steps >= 0, "bad arguments");
    int rc = ctx_enter(b->ctx);
    if (rc) return rc;
    if (steps == 0) return FPDE_OK;
    if (b->n_done + steps > b->max_steps)
        return set_error(FPDE_ERR_CAPACITY, "run of %d steps exceeds the history capacity %d", steps, b->max_steps);
    if (steps < GRAPH_MIN_STEPS) {                 // short runs: enqueued directly, no graph
        int64_t nk = 0;
        if ((rc = batch_enqueue(b, b->ctx->stream, b->n_done, steps, &nk))) return rc;
    } else {
        auto *g = b->graphs.find(b->n_done, steps);
        if (!g) {
            rc = b->graphs.capture(b->n_done, steps,
                                   [&](cudaStream_t cs, int64_t *nk, int *) { return batch_enqueue(b, cs, b->n_done, steps, nk); },
                                   &g);
            if (rc) return rc;
        }
        FPDE_CUDA(cudaGraphLaunch(g->exec, b->ctx->stream));
        count_launches(g->launches);
    }
    b->n_done += steps;
    return FPDE_OK;
}

int fpde_batch_get_state(fpde_batch *b, int col, double *u, int on_device)
{
    clear_error();
    FPDE_CHECK_ARG(b && u && col >= 0 && col < b->n_cols, "bad arguments");
    int rc = ctx_enter(b->ctx);
    if (rc) return rc;
    FPDE_CUDA(cudaMemcpyAsync(u, b->U + b->off[col], (b->N[col] + 1) * sizeof(double),
                              on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, b->ctx->stream));
    FPDE_CUDA(cudaStreamSynchronize(b->ctx->stream));
    return FPDE_OK;
}

int fpde_batch_layout(const fpde_batch *b, int col, int64_t *offset, int64_t *N, int64_t *total)
{
    FPDE_CHECK_ARG(b && col >= 0 && col < b->n_cols, "bad arguments");
    if (offset) *offset = b->off[col];
    if (N) *N = b->N[col];
    if (total) *total = b->Ptot;
    return FPDE_OK;
}

int fpde_batch_reset(fpde_batch *b, const double *u_padded, int on_device)
{
    clear_error();
    FPDE_CHECK_ARG(b, "null argument");
    int rc = ctx_enter(b->ctx);
    if (rc) return rc;
    const double *src = u_padded ? u_padded : b->U0;
    const cudaMemcpyKind kind = (!u_padded || on_device) ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    FPDE_CUDA(cudaMemcpyAsync(b->U, src, b->Ptot * sizeof(double), kind, b->ctx->stream));
    if (u_padded && !on_device) FPDE_CUDA(cudaStreamSynchronize(b->ctx->stream));
    b->n_done = 0;
    return FPDE_OK;
}

int fpde_batch_solve_host(fpde_batch *b, const double *u0_padded_host, int steps, double *u_out_padded_host)
{
    clear_error();
    FPDE_CHECK_ARG(b && u0_padded_host && u_out_padded_host, "null argument");
    int rc = fpde_batch_reset(b, u0_padded_host, 0);
    if (rc) return rc;
    if ((rc = fpde_batch_run(b, steps))) return rc;
    FPDE_CUDA(cudaMemcpyAsync(u_out_padded_host, b->U, b->Ptot * sizeof(double), cudaMemcpyDeviceToHost,
                              b->ctx->stream));
    FPDE_CUDA(cudaStreamSynchronize(b->ctx->stream));
    return ctx_check_flags(b->ctx, "batch");
}

}  // extern "C"
