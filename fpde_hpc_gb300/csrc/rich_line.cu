// One time step of a 1D line with solution-dependent coefficients (the reference's Richards
// problem, analytic_test 0 of fpde_hpc_1d.cpp, on a column with the history): every node's A_/B/R
// (:3095-3142) from the closures KK / inv_dw_dh at the current values (suction P = -(U - Z),
// :2499-2500, :2529), the right-hand side Om = -(Da kkk0/tau) U + src + Da S (Om1 :4191, :4267),
// the surface condition of al1 / bc0 (:4004-4012, :4493-4500), the Thomas solve of al1 / bt1 / U1
// on those coefficients and the increment of the step.
//
//   k_rich_step  : the whole step in one cooperative launch over all SMs (lines of up to 256
//                  nodes per SM, about 38,900 intervals). The step is bound by the
//                  latency of dependent FP64 operations (a lone warp waits ~64 cycles for each, an
//                  SM issues one warp instruction per ~16 cycles), so the line is cut into one node
//                  per thread and as few warps per SM as the length allows.
//   k_rich_coefs + k_rich_thomas: longer lines; the solve in one CTA of 1,024 threads, each owning
//                  a segment of the line.
//
// The alpha recurrence Al[i+1] = B/(R - A Al[i]) is a Moebius map. In g = 1 - Al it reads
// g' = (A g + l) / (A g + B + l) with l = R - A - B (the local term): positive matrices
// [[A, l], [A, B + l]], whose products lose nothing to cancellation even where Al is close to 1 (the
// map in Al itself, [[0, B], [-A, R]], cancels there). Segments' products are combined by scans; the
// beta recurrence and the back substitution are affine maps, combined the same way.
#include <cuda_runtime.h>

#include "common.cuh"
#include "kernels.cuh"
#include "richards.cuh"
#include "ff.cuh"
#include "scan.cuh"

namespace fpde {

constexpr int RT = 1024;                  // threads of the solve

// A, B, R, Om at nodes 1..N-1; al[1], bt[1] from the surface condition.
__global__ void __launch_bounds__(256) k_rich_coefs(RichLineArgs p)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i > p.N) return;
    auto suction = [&](int q) { return -__dadd_rn(p.U[q], -p.Z[q]); };
    if (i == 0) {
        const double kk1 = rich_KK(suction(1), p.kform, p.ksat);
        const double Uc = __ddiv_rn(__dmul_rn(p.dL[0], p.E - 0.0), kk1);
        if (rich_inv_dw_dh(suction(0)) != RICH_SATURATED) {
            p.al[1] = 1.0;
            p.bt[1] = -Uc;
        } else {
            p.al[1] = 0.0;
            p.bt[1] = __ddiv_rn(__dmul_rn(-Uc, kk1), p.dL[0]);
        }
        return;
    }
    if (i >= p.N) return;
    const double Pm = suction(i - 1), Pi = suction(i);
    const double kkm = rich_KK(Pm, p.kform, p.ksat), kk = rich_KK(Pi, p.kform, p.ksat), iw = rich_inv_dw_dh(Pi);
    const double dq = p.dL[i], dm = p.dL[i - 1];
    const double dqq = __dmul_rn(dq, dq), dqm = __dmul_rn(dq, dm);
    p.cA[i] = __ddiv_rn(__dmul_rn(kkm, iw), dqm);
    p.cB[i] = __ddiv_rn(__dmul_rn(kk, iw), dqq);
    p.cR[i] = __dadd_rn(__dmul_rn(iw, __dadd_rn(__ddiv_rn(kk, dqq), __ddiv_rn(kkm, dqm))), p.lamR);
    double sv = 0.0;
    for (int k = 0; k < p.KS; ++k) sv += __ldcg(p.part + (int64_t)k * p.pstride + i);
    const double om = __dadd_rn(-__dmul_rn(p.lam, p.U[i]), p.src ? p.src[i] : 0.0);
    p.cOm[i] = __dadd_rn(om, sv);
}

struct Mob { double a, b, c, d; };                 // 2x2 matrix [[a, b], [c, d]]
struct Aff { double a, c; };                       // x -> a x + c

__device__ __forceinline__ Mob mob_mul(const Mob &x, const Mob &y)   // x y
{
    return {x.a * y.a + x.b * y.c, x.a * y.b + x.b * y.d, x.c * y.a + x.d * y.c, x.c * y.b + x.d * y.d};
}
// x 2^-e from the bits: integer instructions (results below the normal range become 0,
// which is below 2^-1022 of the matrix's largest entry).
__device__ __forceinline__ double scale_bits(double x, int e)
{
    const int hi = __double2hiint(x), f = (hi >> 20) & 0x7FF;
    return f - e <= 0 ? 0.0 : __hiloint2double(hi - (e << 20), __double2loint(x));
}
// Projective maps are unchanged by a common scale: keep the largest entry near 1 with an exact power
// of two, off the FP64 pipe. Entries are >= 0; a matrix with infinities or NaN stays as it is.
__device__ __forceinline__ Mob mob_norm(Mob m)
{
    const int s = max(max(__double2hiint(m.a) & 0x7FFFFFFF, __double2hiint(m.b) & 0x7FFFFFFF),
                      max(__double2hiint(m.c) & 0x7FFFFFFF, __double2hiint(m.d) & 0x7FFFFFFF)) >> 20;
    if (s > 0 && s < 0x7FF) {
        const int e = s - 1023;
        m.a = scale_bits(m.a, e); m.b = scale_bits(m.b, e); m.c = scale_bits(m.c, e); m.d = scale_bits(m.d, e);
    }
    return m;
}
__device__ __forceinline__ Aff aff_after(const Aff &later, const Aff &earlier)
{
    return {later.a * earlier.a, later.a * earlier.c + later.c};
}
__device__ __forceinline__ Mob shfl_up_mob(const Mob &m, int o)
{
    return {__shfl_up_sync(0xffffffffu, m.a, o), __shfl_up_sync(0xffffffffu, m.b, o),
            __shfl_up_sync(0xffffffffu, m.c, o), __shfl_up_sync(0xffffffffu, m.d, o)};
}
__device__ __forceinline__ Aff shfl_up_aff(const Aff &m, int o)
{
    return {__shfl_up_sync(0xffffffffu, m.a, o), __shfl_up_sync(0xffffffffu, m.c, o)};
}

// Inclusive scan over the CTA's threads in index order, combined as later * earlier.
__device__ Mob scan_mob(Mob v, Mob *warp_tot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Mob u = shfl_up_mob(v, o);
        if (lane >= o) v = mob_norm(mob_mul(v, u));
    }
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    if (warp == 0) {
        Mob w = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const Mob u = shfl_up_mob(w, o);
            if (lane >= o) w = mob_norm(mob_mul(w, u));
        }
        warp_tot[lane] = w;
    }
    __syncthreads();
    if (warp > 0) v = mob_norm(mob_mul(v, warp_tot[warp - 1]));
    __syncthreads();
    return v;
}
__device__ Aff scan_aff(Aff v, Aff *warp_tot)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const Aff u = shfl_up_aff(v, o);
        if (lane >= o) v = aff_after(v, u);
    }
    if (lane == 31) warp_tot[warp] = v;
    __syncthreads();
    if (warp == 0) {
        Aff w = warp_tot[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const Aff u = shfl_up_aff(w, o);
            if (lane >= o) w = aff_after(w, u);
        }
        warp_tot[lane] = w;
    }
    __syncthreads();
    if (warp > 0) v = aff_after(v, warp_tot[warp - 1]);
    __syncthreads();
    return v;
}

__global__ void __launch_bounds__(RT, 1) k_rich_thomas(RichLineArgs p)
{
    __shared__ Mob mtot[32];
    __shared__ Aff atot[32];
    // the matrix prefixes (phase 1) and the affine ones (phases 2 and 4) share one buffer: a
    // barrier separates the last read of the former from the first write of the latter
    __shared__ double pref[4 * RT];
    Mob *mincl = reinterpret_cast<Mob *>(pref);
    Aff *aincl = reinterpret_cast<Aff *>(pref);
    __shared__ double uN_s;
    const int t = threadIdx.x, N = p.N;
    const int seg = (N - 1 + RT - 1) / RT;
    const int i0 = 1 + t * seg, i1 = min(i0 + seg, N);          // nodes [i0, i1) of 1..N-1
    const double uold_last = p.U[N - 1];                         // before any write (U1 :4695-4718)
    const double al1 = p.al[1], bt1 = p.bt[1];
    // 1. alpha. In g = 1 - Al the recurrence reads g' = (A g + l) / (A g + B + l) with
    // l = R - A - B (the local term): a Moebius map with positive entries [[A, l], [A, B + l]], whose
    // products lose nothing to cancellation even where Al is close to 1 (the map in Al itself,
    // [[0, B], [-A, R]], cancels there). Segment products, a scan, then each segment in order.
    Mob m = {1.0, 0.0, 0.0, 1.0};
    for (int i = i0; i < i1; ++i) {
        const double A = p.cA[i], B = p.cB[i], l = (p.cR[i] - A) - B;
        m = mob_norm(mob_mul(Mob{A, l, A, B + l}, m));
    }
    mincl[t] = scan_mob(m, mtot);
    __syncthreads();
    double al = al1;
    if (t > 0) {
        const Mob e = mincl[t - 1];                              // segments 0 .. t-1
        const double g1 = 1.0 - al1;                             // exact: Al[1] is 0 or 1
        al = 1.0 - (e.a * g1 + e.b) / (e.c * g1 + e.d);
    }
    for (int i = i0; i < i1; ++i) {
        al = __ddiv_rn(p.cB[i], __dadd_rn(p.cR[i], -__dmul_rn(p.cA[i], al)));  // al1 :4026
        p.al[i + 1] = al;
    }
    __syncthreads();
    // 2. beta: Bt[i+1] = (Al[i+1]/B_i)(A_i Bt[i] - Om_i) (bt1 :4587-4589), affine in Bt[i]
    Aff f = {1.0, 0.0};
    for (int i = i0; i < i1; ++i) {
        const double g = p.al[i + 1] / p.cB[i];
        f = aff_after(Aff{g * p.cA[i], -g * p.cOm[i]}, f);
    }
    aincl[t] = scan_aff(f, atot);
    __syncthreads();
    double bt = bt1;
    if (t > 0) bt = aincl[t - 1].a * bt1 + aincl[t - 1].c;
    for (int i = i0; i < i1; ++i) {
        bt = __dmul_rn(__ddiv_rn(p.al[i + 1], p.cB[i]), __dadd_rn(__dmul_rn(p.cA[i], bt), -p.cOm[i]));
        p.bt[i + 1] = bt;
    }
    __syncthreads();
    // 3. right end (U1 :4685-4719)
    if (t == 0) {
        double uN;
        if (p.rkind == FPDE_BC_DIRICHLET) {
            uN = p.gN;
        } else {
            const double BtN = p.bt[N], AlN = p.al[N];
            if (fabs(BtN) > 1e-15)
                uN = (fabs(1.0 - AlN) > 1e-15) ? __ddiv_rn(__dadd_rn(BtN, __dmul_rn(p.gN, p.dLN)), 1.0 - AlN) : uold_last;
            else
                uN = (fabs(1.0 - AlN) > 1e-15) ? 0.0 : uold_last;
        }
        uN_s = uN;
    }
    __syncthreads();
    const double uN = uN_s;
    // 4. back substitution U_i = Al[i+1] U_{i+1} + Bt[i+1] from the right: segment t maps the
    // value at i1 to the one at i0; the scan runs over the segments in reverse order
    Aff h = {1.0, 0.0};
    for (int i = i1 - 1; i >= i0; --i) h = aff_after(Aff{p.al[i + 1], p.bt[i + 1]}, h);
    __syncthreads();
    aincl[RT - 1 - t] = h;                                       // reversed order
    __syncthreads();
    const Aff hr = aincl[t];
    __syncthreads();
    aincl[t] = scan_aff(hr, atot);
    __syncthreads();
    double u = uN;                                               // the value at node i1
    if (t < RT - 1) {
        const Aff e = aincl[RT - 2 - t];                         // segments t+1 .. last
        u = e.a * uN + e.c;
    }
    __syncthreads();
    if (t == 0) p.U[N] = uN;
    for (int i = i1 - 1; i >= i0; --i) {
        u = __dadd_rn(__dmul_rn(p.al[i + 1], u), p.bt[i + 1]);   // U1 :4723
        p.U[i] = u;
    }
    __syncthreads();
    if (t == 0) p.U[0] = __dadd_rn(__dmul_rn(al1, p.U[1]), bt1);
}


// ------------------------------------------------------------------ the step over all SMs

__device__ __forceinline__ double rslot_load(const double *p, bool &got)
{
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    if (v == SLOT_EMPTY) got = false;
    return __longlong_as_double((long long)v);
}
__device__ __forceinline__ void rslot_store_bits(double *p, unsigned long long v)
{
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
__device__ __forceinline__ void rslot_store(double *p, double v) { rslot_store_bits(p, slot_bits(v)); }

__device__ __forceinline__ Mob shfl_down_mob(const Mob &m, int o)
{
    return {__shfl_down_sync(FULL, m.a, o), __shfl_down_sync(FULL, m.b, o), __shfl_down_sync(FULL, m.c, o),
            __shfl_down_sync(FULL, m.d, o)};
}

// One step of a line in one cooperative launch: CTA c owns the 32 W nodes from 1 + 32 W c. Three
// roles: W solve warps (one node per lane: KK, the coefficients, the scans), W closure warps (the
// same nodes' inv_dw_dh, beside the longer KK chain) and one edge warp (KK of the node before the
// chunk; in CTA 0 the state of node 0 for the surface condition). Two exchanges of a few numbers
// per chunk join the chunks: the products of the alpha maps (every CTA then composes those before
// it), and the chunk's zero-carry sweeps with their responses (every CTA then solves the chunk-level
// recurrences). A slot is written once per launch and polled as a value (a 64-bit access is
// single-copy atomic); the launch uses the half of the slots that its sequence number's parity
// names and empties its own slots of the other half, which the launch before it used, so no
// launch needs a memset. Every wait is bounded (1 s, DEVERR_BARRIER_TIMEOUT).
// Bound by the latency of its FP64 chain (three dependent pows, about 60 scan and carry operations).
// N = 4,001, 400 steps on a GB300, per step with its history sum: 42 us; 295 us as k_rich_coefs (146 us:
// 15 pows per node on 16 SMs) + k_rich_thomas (144 us: one SM's FP64 pipe) + append.
template <int W>
__global__ void __launch_bounds__(32 * (2 * W + 1), 1) k_rich_step(RichLineArgs p)
{
    constexpr int C = 32 * W;                           // nodes per CTA
    __shared__ double sIw[C], sKK[C + 1], sEdge[2];     // sKK[k + 1]: node a + k; sKK[0]: node a - 1
    __shared__ double sT[W][4];                         // per warp: scan totals
    __shared__ double sCarry[4];                        // gamma_in, then y_in, u_out, U_N
    __shared__ unsigned long long s_seq;
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = blockIdx.x, G = gridDim.x, N = p.N;
    const int a = 1 + c * C;
    if (tid == 0) { s_seq = *((volatile unsigned long long *)p.seq) + 1; s_abort = 0; }
    const double uold_last = p.U[N - 1];                // read before any write of the launch
    auto suction = [&](int q) { return -__dadd_rn(p.U[q], -p.Z[q]); };

    if (warp >= 2 * W) {                                // edge warp
        if (lane == 0) sKK[0] = rich_KK(suction(a - 1), p.kform, p.ksat);
        if (lane == 1 && c == 0) sEdge[0] = rich_inv_dw_dh(suction(0)) != RICH_SATURATED ? 1.0 : 0.0;
    } else if (warp >= W) {                             // closure warps
        const int i = a + (warp - W) * 32 + lane;
        if (i < N) sIw[(warp - W) * 32 + lane] = rich_inv_dw_dh(suction(i));
    }
    const int k = warp * 32 + lane, i = a + k;          // solve warps: this lane's node
    const bool solve = warp < W, in = solve && i < N;
    double uo = 0.0, lo = 0.0, kk = 0.0, om = 0.0;
    if (in) {
        uo = p.U[i];
        lo = p.last[i];
        double sv = 0.0;                                // the history partials, four chains of loads
        double s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int q = 0;
        for (; q + 4 <= p.KS; q += 4) {
            const double *pp = p.part + (int64_t)q * p.pstride + i;
            sv += __ldcg(pp);
            s1 += __ldcg(pp + p.pstride);
            s2 += __ldcg(pp + 2 * p.pstride);
            s3 += __ldcg(pp + 3 * p.pstride);
        }
        for (; q < p.KS; ++q) sv += __ldcg(p.part + (int64_t)q * p.pstride + i);
        om = __dadd_rn(__dadd_rn(-__dmul_rn(p.lam, uo), p.src ? __ldg(p.src + i) : 0.0), (sv + s1) + (s2 + s3));
        kk = rich_KK(suction(i), p.kform, p.ksat);
        sKK[k + 1] = kk;
    }
    __syncthreads();
    const unsigned long long seq = s_seq;
    double *slots = p.slots + (seq & 1) * (size_t)(16 * G);
    if (warp == 2 * W && lane < 16)                     // empty this chunk's slots for the next launch
        rslot_store_bits(p.slots + ((seq & 1) ^ 1) * (size_t)(16 * G) + 16 * c + lane, SLOT_EMPTY);

    // ---- coefficients (A_/B/R) and the alpha maps; inclusive products over the CTA's nodes
    double cA = 0.0, cB = 1.0, cBl = 1.0;               // A, B, B + l
    Mob m = {1.0, 0.0, 0.0, 1.0};
    double al1 = 0.0, bt1 = 0.0;                        // Al[1], Bt[1] (CTA 0; the others get them)
    if (solve) {
        if (in) {
            const double kkm = sKK[k], iw = sIw[k];
            const double dq = __ldg(p.dL + i), dm = __ldg(p.dL + i - 1);
            const double dqq = __dmul_rn(dq, dq), dqm = __dmul_rn(dq, dm);
            cA = __ddiv_rn(__dmul_rn(kkm, iw), dqm);
            cB = __ddiv_rn(__dmul_rn(kk, iw), dqq);
            const double R = __dadd_rn(__dmul_rn(iw, __dadd_rn(__ddiv_rn(kk, dqq), __ddiv_rn(kkm, dqm))), p.lamR);
            const double l = (R - cA) - cB;
            cBl = cB + l;
            m = mob_norm(Mob{cA, l, cA, cBl});
        }
        if (c == 0 && warp == 0) {                      // surface condition (al1 :4004-4012, bc0 :4493-4500)
            const double kk1 = sKK[1], Uc = __ddiv_rn(__dmul_rn(p.dL[0], p.E - 0.0), kk1);
            if (sEdge[0] != 0.0) {
                al1 = 1.0;
                bt1 = -Uc;
            } else {
                al1 = 0.0;
                bt1 = __ddiv_rn(__dmul_rn(-Uc, kk1), p.dL[0]);
            }
            if (lane == 0) { rslot_store(slots + 4, al1); rslot_store(slots + 5, bt1); }
        }
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const Mob u = shfl_up_mob(m, o);
            if (lane >= o) m = mob_norm(mob_mul(m, u));
        }
        if (W > 1 && lane == 31) { sT[warp][0] = m.a; sT[warp][1] = m.b; sT[warp][2] = m.c; sT[warp][3] = m.d; }
    }
    if (W > 1) {                                        // products of the warps before this one
        __syncthreads();
        if (warp == 0) {
            Mob w = {1.0, 0.0, 0.0, 1.0};
            if (lane < W) w = Mob{sT[lane][0], sT[lane][1], sT[lane][2], sT[lane][3]};
#pragma unroll
            for (int o = 1; o < W; o <<= 1) {
                const Mob u = shfl_up_mob(w, o);
                if (lane >= o) w = mob_norm(mob_mul(w, u));
            }
            if (lane < W) { sT[lane][0] = w.a; sT[lane][1] = w.b; sT[lane][2] = w.c; sT[lane][3] = w.d; }
        }
        __syncthreads();
        if (solve && warp > 0)
            m = mob_norm(mob_mul(m, Mob{sT[warp - 1][0], sT[warp - 1][1], sT[warp - 1][2], sT[warp - 1][3]}));
    }
    if (warp == W - 1 && lane == 31) {
        double *s = slots + 16 * c;
        rslot_store(s, m.a); rslot_store(s + 1, m.b); rslot_store(s + 2, m.c); rslot_store(s + 3, m.d);
    }
    // ---- exchange 1, warp 0: gamma before this chunk from the maps of the chunks before it
    if (warp == 0) {
        Mob v[5];
        double e0 = 0.0, e1 = 0.0;
        bool ok = true;
        const unsigned long long t0 = gtimer_ns();
        while (true) {
            bool got = true;
#pragma unroll
            for (int t = 0; t < 5; ++t) {
                const int q = 5 * lane + t;
                v[t] = Mob{1.0, 0.0, 0.0, 1.0};
                if (q < c) {
                    const double *s = slots + 16 * q;
                    v[t].a = rslot_load(s, got); v[t].b = rslot_load(s + 1, got);
                    v[t].c = rslot_load(s + 2, got); v[t].d = rslot_load(s + 3, got);
                }
            }
            e0 = rslot_load(slots + 4, got);
            e1 = rslot_load(slots + 5, got);
            if (__all_sync(FULL, got)) break;
            if (gtimer_ns() - t0 > 1000000000ull) { ok = false; break; }
        }
        ok = __all_sync(FULL, ok);
        if (!ok) {
            if (lane == 0) { atomicOr(p.flags, DEVERR_BARRIER_TIMEOUT); s_abort = 1; }
        } else {
            Mob w = v[0];
#pragma unroll
            for (int t = 1; t < 5; ++t)
                if (5 * lane + t < c) w = mob_norm(mob_mul(v[t], w));
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {          // lane 0: all lanes, later maps on the left
                const Mob u = shfl_down_mob(w, o);
                if (lane + o < 32) w = mob_norm(mob_mul(u, w));
            }
            al1 = e0;
            bt1 = e1;
            if (lane == 0) {
                const double g1 = 1.0 - al1;            // exact: Al[1] is 0 or 1
                sCarry[0] = c == 0 ? g1 : (w.a * g1 + w.b) / (w.c * g1 + w.d);
                sCarry[1] = al1;
                sCarry[2] = bt1;
            }
        }
    }
    __syncthreads();
    if (s_abort) return;

    // ---- zero-carry sweeps of the chunk. Forward y_i = g (A y_{i-1} - Om) as (P, X) prefixes; backward
    // u_i = Al u_{i+1} + y_i as u_i = Q u_out + Ub + K y_in (suffixes over Q = prod Al, Ub from X, K from P)
    double al = 0.0, P = 1.0, X = 0.0;
    if (solve) {
        // Al[i+1] = B/(A g_i + B + l) with g_i = (E.a g + E.b)/(E.c g + E.d), E the maps of the chunk's
        // nodes before i: one division, and no 1 - g_{i+1}, which would cancel where Al is small
        Mob E = shfl_up_mob(m, 1);
        if (lane == 0)
            E = warp > 0 ? Mob{sT[warp - 1][0], sT[warp - 1][1], sT[warp - 1][2], sT[warp - 1][3]}
                         : Mob{1.0, 0.0, 0.0, 1.0};
        if (in) {
            const double g = sCarry[0], top = fma(E.a, g, E.b), bot = fma(E.c, g, E.d);
            al = cB * bot / fma(cA, top, cBl * bot);
            const double gg = al / cB;
            P = gg * cA;
            X = -gg * om;
        }
        warp_scan_up(P, X, lane);
    }
    if (W > 1) {
        __syncthreads();                                // the alpha maps in sT have been read
        if (solve && lane == 31) { sT[warp][0] = P; sT[warp][1] = X; }
        __syncthreads();
        if (warp == 0) {
            double Pw = lane < W ? sT[lane][0] : 1.0, Xw = lane < W ? sT[lane][1] : 0.0;
            warp_scan_up(Pw, Xw, lane);
            if (lane < W) { sT[lane][2] = Pw; sT[lane][3] = Xw; }
        }
        __syncthreads();
        if (solve && warp > 0) {
            X = fma(P, sT[warp - 1][3], X);
            P = P * sT[warp - 1][2];
        }
    }
    const double yP = P, yX = X;                        // inclusive prefixes: y_i = yX + yP y_in
    double Q = in ? al : 1.0, Ub = in ? X : 0.0, K = in ? P : 0.0;
    if (solve) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double Qn = __shfl_down_sync(FULL, Q, o), Un = __shfl_down_sync(FULL, Ub, o),
                         Kn = __shfl_down_sync(FULL, K, o);
            if (lane + o < 32) { Ub = fma(Q, Un, Ub); K = fma(Q, Kn, K); Q = Q * Qn; }
        }
    }
    if (W > 1) {
        __syncthreads();
        if (solve && lane == 0) { sT[warp][0] = Q; sT[warp][1] = Ub; sT[warp][2] = K; }
        __syncthreads();
        if (solve) {                                    // the warps after this one, nearest last
            double Qs = 1.0, Us = 0.0, Ks = 0.0;
            for (int w = W - 1; w > warp; --w) {
                Us = fma(sT[w][0], Us, sT[w][1]);
                Ks = fma(sT[w][0], Ks, sT[w][2]);
                Qs *= sT[w][0];
            }
            Ub = fma(Q, Us, Ub);
            K = fma(Q, Ks, K);
            Q = Q * Qs;
        }
    }
    {
        double *s = slots + 16 * c + 8;
        if (warp == W - 1 && lane == 31) { rslot_store(s, yP); rslot_store(s + 1, yX); }
        if (tid == 0) { rslot_store(s + 2, Q); rslot_store(s + 3, Ub); rslot_store(s + 4, K); }
        if (solve && i == N - 1) rslot_store(s + 5, al);    // last chunk: Al[N] for the flux closure
    }
    // ---- exchange 2, warp 0: the chunk-level recurrences (every CTA the same, its own chunk's carries)
    if (warp == 0) {
        double cP[5], cX[5], cQ[5], cU[5], cK[5], alN = 0.0;
        bool ok = true;
        const unsigned long long t0 = gtimer_ns();
        while (true) {
            bool got = true;
#pragma unroll
            for (int t = 0; t < 5; ++t) {
                const int q = 5 * lane + t;
                cP[t] = cQ[t] = 1.0;
                cX[t] = cU[t] = cK[t] = 0.0;
                if (q < G) {
                    const double *s = slots + 16 * q + 8;
                    cP[t] = rslot_load(s, got); cX[t] = rslot_load(s + 1, got); cQ[t] = rslot_load(s + 2, got);
                    cU[t] = rslot_load(s + 3, got); cK[t] = rslot_load(s + 4, got);
                }
            }
            alN = rslot_load(slots + 16 * (G - 1) + 13, got);
            if (__all_sync(FULL, got)) break;
            if (gtimer_ns() - t0 > 1000000000ull) { ok = false; break; }
        }
        ok = __all_sync(FULL, ok);
        if (!ok) {
            if (lane == 0) { atomicOr(p.flags, DEVERR_BARRIER_TIMEOUT); s_abort = 1; }
        } else {
            double Pl = 1.0, Xl = 0.0;
#pragma unroll
            for (int t = 0; t < 5; ++t) { Xl = fma(cP[t], Xl, cX[t]); Pl *= cP[t]; }
            warp_scan_up(Pl, Xl, lane);
            const double yN = __shfl_sync(FULL, fma(Pl, sCarry[2], Xl), 31);     // Bt[N]
            double Pe = __shfl_up_sync(FULL, Pl, 1), Xe = __shfl_up_sync(FULL, Xl, 1);
            if (lane == 0) { Pe = 1.0; Xe = 0.0; }
            double yin[5];
            double y = fma(Pe, sCarry[2], Xe);
#pragma unroll
            for (int t = 0; t < 5; ++t) { yin[t] = y; y = fma(cP[t], y, cX[t]); }
            double uN;                                  // right end (U1 :4685-4719)
            if (p.rkind == FPDE_BC_DIRICHLET) {
                uN = p.gN;
            } else if (fabs(yN) > 1e-15) {
                uN = (fabs(1.0 - alN) > 1e-15) ? __ddiv_rn(__dadd_rn(yN, __dmul_rn(p.gN, p.dLN)), 1.0 - alN)
                                               : uold_last;
            } else {
                uN = (fabs(1.0 - alN) > 1e-15) ? 0.0 : uold_last;
            }
            double Ql = 1.0, Ul = 0.0, v[5];
#pragma unroll
            for (int t = 4; t >= 0; --t) {
                v[t] = fma(cK[t], yin[t], cU[t]);
                Ul = fma(cQ[t], Ul, v[t]);
                Ql *= cQ[t];
            }
            warp_scan_down(Ql, Ul, lane);
            double Qe = __shfl_down_sync(FULL, Ql, 1), Ue = __shfl_down_sync(FULL, Ul, 1);
            if (lane == 31) { Qe = 1.0; Ue = 0.0; }
            double u = fma(Qe, uN, Ue);
#pragma unroll
            for (int t = 4; t >= 0; --t) {
                if (5 * lane + t == c) {
                    sCarry[0] = yin[t];
                    sCarry[3] = u;
                }
                u = fma(cQ[t], u, v[t]);
            }
            if (lane == 0) sEdge[1] = uN;
        }
    }
    __syncthreads();
    if (s_abort) return;
    // ---- the new state, its increment and (split history) the increment as a float pair. The increment counts
    // from the last computed state, whatever the caller has written to U since (as k_append's)
    auto put = [&](int q, double un, double before) {
        const double d = un - before;
        p.U[q] = un;
        p.last[q] = un;
        p.Drow[q] = d;
        if (p.Drowf) p.Drowf[q] = d2ff(d);
    };
    double u = 0.0;
    if (in) {
        u = fma(Q, sCarry[3], fma(K, sCarry[0], Ub));
        put(i, u, lo);
        if (i == N - 1) put(N, sEdge[1], p.last[N]);
    }
    if (c == 0 && tid == 0) {
        put(0, __dadd_rn(__dmul_rn(sCarry[1], u), sCarry[2]), p.last[0]);   // Al[1] U[1] + Bt[1]
        *((volatile unsigned long long *)p.seq) = seq;  // every CTA has read it (it published)
    }
}

// Warps of solve nodes per CTA for a line of N intervals on `sms` SMs (one CTA per SM, at most 160
// chunks): the fewest, since fewer warps share an SM's FP64 pipe; 0 for lines it does not hold.
static int rich_step_warps(int N, int sms)
{
    const int g = sms < 160 ? sms : 160;
    for (int w = 1; w <= 8; w <<= 1)
        if ((int64_t)32 * w * g >= N - 1) return w;
    return 0;
}

size_t rich_slot_count(int N)
{
    const int w = rich_step_warps(N, device_sm_count());
    return w ? (size_t)2 * 16 * ((N - 1 + 32 * w - 1) / (32 * w)) : 0;
}

template <int W>
static cudaError_t launch_rich_step(cudaStream_t st, const RichLineArgs &a)
{
    const int G = (a.N - 1 + 32 * W - 1) / (32 * W);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(32 * (2 * W + 1));
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = G > 1 ? 1 : 0;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_rich_step<W>, a);
}

int launch_rich_line_step(cudaStream_t st, const RichLineArgs &a, int64_t *nk)
{
    if (a.N < 2) return set_error(FPDE_ERR_ARG, "richards line: N must be at least 2");
    if (const int w = a.slots ? rich_step_warps(a.N, device_sm_count()) : 0) {
        cudaError_t e = w == 1   ? launch_rich_step<1>(st, a)
                        : w == 2 ? launch_rich_step<2>(st, a)
                        : w == 4 ? launch_rich_step<4>(st, a)
                                 : launch_rich_step<8>(st, a);
        if (e != cudaSuccess) return set_error(FPDE_ERR_CUDA, "richards line launch: %s", cudaGetErrorString(e));
        count_launches(1);
        *nk += 1;
        return FPDE_OK;
    }
    k_rich_coefs<<<(unsigned)((a.N + 1 + 255) / 256), 256, 0, st>>>(a);
    FPDE_LAUNCHED(1);
    k_rich_thomas<<<1, RT, 0, st>>>(a);
    FPDE_LAUNCHED(1);
    *nk += 3;
    return a.Drowf ? launch_append_ff(st, a.U, a.last, a.Drow, a.Drowf, a.N + 1, a.pitch)
                   : launch_append(st, a.U, a.last, a.Drow, a.N + 1, a.pitch);
}

}  // namespace fpde
