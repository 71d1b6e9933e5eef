// pcg.cuh -- whole iterations of the mixed-precision CG on QplusQminus_eo in one
// cooperative launch, for lattices whose sweeps are shorter than the launches
// around them.
//
// The ordinary iteration is five dependent launches (mix_p of mixed.cuh, the
// four sweeps of pdslash.cuh with the vector updates and reductions fused in)
// and a residual read by the host one iteration behind the queue.  At 16^3x32 a
// sweep has 256 tiles for 148 SMs and takes a few microseconds, so the iteration
// is bound by the launches and by the host that queues them.  Here the blocks
// stay resident and step through the same five phases with a grid barrier
// between them; the four sweeps are one loop over one copy of the stencil (the
// epilogue is chosen per phase), so the instruction cache holds it.  The host is
// asked only when a right-hand side needs it: a reliable update, or a residual
// that is no number.
//
// The arithmetic, its order and the rule that judges an iteration's residual
// (one iteration after it, as the host does) are those of the ordinary path, so
// the iterates are bitwise the same: a reduction leaves one partial per warp,
// and after the barrier every block adds them up in the order of pk_finish_kernel
// and runs the same finisher on its own copy of the solver scalars, which
// saves the second barrier that one finishing block would need.
#pragma once

#include "c2q_host.h"
#include "gridbar.cuh"
#include "pdslash.cuh"

namespace c2q {

// what the slots' stencils of a launch on `ref`'s lattice and precision have in common (pdslash.cu)
void pk_stencil_args(const c2q_spinor_eo* ref, const c2q_gauge* g, int gkind, double kappa, PkStencil* st);

// Arrival counter, what the last launch did, and whether a barrier gave up.
struct PcgCtl {
    unsigned arrived;
    unsigned error;
    int iters;                  // iterations done
    int undecided;              // they ended at the limit
    double judged[PK_MAX_RHS];  // the residual the last iteration judged
    double maxrr[PK_MAX_RHS];
    int flag[PK_MAX_RHS];       // SolverScalars::flag when it was judged
};

struct PcgRhs {
    void *p, *t1, *t2;
    float *p_norm, *t1_norm, *t2_norm;
    void *rs, *xs;  // FP32
    SolverScalars* sc;
    double thr, maxrr;
};

struct PcgParams : PkStencil {
    PcgRhs f[PK_MAX_RHS];
    int nrhs, ntiles;
    EpiArgs e[4];       // per sweep
    double delta;
    int first;          // the solve's first iteration comes first: p is the residual, nothing to judge yet
    unsigned skip;      // bit r: the residual before the first iteration is a true one, not to be judged
    int iters;          // at most
    double* partials;   // one per warp, tile and right-hand side
    PcgCtl* ctl;
};

// The sums of all right-hand sides' partials (one per warp of each tile) into tot, by
// the whole block, in the order of pk_finish_kernel: partials j, j + 1024, ... per
// accumulator j, a tree over each 32 accumulators, a tree over those.
__device__ __forceinline__ void pcg_sums(const double* partials, int nparts, int nrhs, double* tot, double* smem)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int rhs = 0; rhs < nrhs; ++rhs) {
        double a[32 / PK_WARPS];
#pragma unroll
        for (int q = 0; q < 32 / PK_WARPS; ++q) {
            const int j = 32 * (PK_WARPS * q + warp) + lane;
            a[q]        = j < nparts ? __ldcg(partials + (size_t)j * nrhs + rhs) : 0.0;
        }
        for (int m = 1024; m < nparts; m += 1024)
#pragma unroll
            for (int q = 0; q < 32 / PK_WARPS; ++q) {
                const int j = m + 32 * (PK_WARPS * q + warp) + lane;
                if (j < nparts) a[q] += __ldcg(partials + (size_t)j * nrhs + rhs);
            }
#pragma unroll
        for (int q = 0; q < 32 / PK_WARPS; ++q)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) a[q] += __shfl_down_sync(0xffffffffu, a[q], o);
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < 32 / PK_WARPS; ++q) smem[PK_WARPS * q + warp] = a[q];
        __syncthreads();
        if (warp == 0) {
            double t = smem[lane];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
            if (lane == 0) tot[rhs] = t;
        }
        __syncthreads();
    }
}

template <int P, int NL>
__global__ void __launch_bounds__(PK_THREADS, PkStage<P, NL, 0>::MINB) pcg_kernel(const PcgParams prm)
{
    using S = PkStage<P, NL, 0>;
    extern __shared__ uint4 ring[];
    __shared__ SolverScalars sc[PK_MAX_RHS];
    __shared__ double prev[PK_MAX_RHS], maxrr[PK_MAX_RHS], judged[PK_MAX_RHS];
    __shared__ int prev_flag[PK_MAX_RHS], judged_flag[PK_MAX_RHS];
    __shared__ double smem[32], tot[PK_MAX_RHS];
    __shared__ int ok, stop;
    uint4* mine     = ring + threadIdx.x;
    uint4* s8       = mine + (size_t)((8 % S::STAGES) * S::CH) * PK_THREADS;
    uint4* s9       = mine + (size_t)((9 % S::STAGES) * S::CH) * PK_THREADS;
    const PkGeom& g = prm.g;
    const int nrhs = prm.nrhs, ss = g.ss;
    const int items = prm.ntiles * nrhs;
    const float hop = (float)prm.c.scale;
    unsigned target = 0;

    for (int r = threadIdx.x; r < nrhs; r += PK_THREADS) {
        sc[r]        = *prm.f[r].sc;
        prev[r]      = sc[r].resid;
        prev_flag[r] = sc[r].flag;
        maxrr[r]     = prm.f[r].maxrr;
        judged[r]    = 0.0;
        judged_flag[r] = 0;
    }
    if (threadIdx.x == 0) stop = 0;
    __syncthreads();

    int it = 0;
    while (it < prm.iters) {
        if (!(prm.first && it == 0)) {  // p = r + beta p (mix_p)
            for (int item = blockIdx.x; item < items; item += gridDim.x) {
                const int tile  = nrhs == 1 ? item : (int)((unsigned)item / (unsigned)nrhs);
                const int rhs   = item - tile * nrhs;
                const int j     = tile * PK_THREADS + threadIdx.x;
                const PcgRhs& F = prm.f[rhs];
                if (j >= g.H) continue;
                stage_spinor<P>(s8, F.p, F.p_norm, ss, j);
                stage_residual<P, NL, 8>(s8, F.rs, ss, j);
                stage_residual<P, NL, 9>(s9, F.rs, ss, j);
                cp_commit();
                cp_wait<0>();
                C2 pv[12];
                float2 ps;
                staged_operand<P>(s8, pv, &ps);
                const float br = (float)sc[rhs].beta[0], bi = (float)sc[rhs].beta[1];
                const float2 cr = mul2(bc2(br), ps), ci = mul2(bc2(bi), ps), nci = mul2(bc2(-bi), ps);
#pragma unroll
                for (int c = 0; c < 12; ++c) {
                    const C2 r = c2_from(as_f4(residual_chunk<P, NL>(s8, s9, c)), false);
                    const C2 b = pv[c];
                    pv[c]      = C2{fma2(b.re, cr, fma2(b.im, nci, r.re)), fma2(b.im, cr, fma2(b.re, ci, r.im))};
                }
                if constexpr (P == 16)
                    SlotF16::store(F.p, F.p_norm, ss, j, pv);
                else
                    SlotF32::store(F.p, ss, j, pv);
            }
            if (!grid_barrier(&prm.ctl->arrived, &prm.ctl->error, target += gridDim.x, &ok)) return;
        }
#pragma unroll 1
        for (int ph = 0; ph < 4; ++ph) {
            // 0: t1 = diag D p   1: t2 = g5 (diag p - D t1), |t2|^2 -> alpha
            // 2: t1 = diag D t2, x += alpha p   3: r -= alpha g5 (diag t2 - D t1), |r|^2 -> beta
            const bool axpy = ph & 1;
            for (int item = blockIdx.x; item < items; item += gridDim.x) {
                const int tile  = nrhs == 1 ? item : (int)((unsigned)item / (unsigned)nrhs);
                const int rhs   = item - tile * nrhs;
                const int j     = tile * PK_THREADS + threadIdx.x;
                const PcgRhs& F = prm.f[rhs];
                float2 dre      = bc2(0.f);
                if (j < g.H) {
                    const void* in    = ph == 0 ? F.p : axpy ? F.t1 : F.t2;
                    const float* in_n = ph == 0 ? F.p_norm : axpy ? F.t1_norm : F.t2_norm;
                    C2 acc[12];
                    pk_stencil<P, NL, PH_TG, S>(acc, prm, in, in_n, ph & 1, j, mine, [&](auto qc, uint4* st) {
                        if constexpr (decltype(qc)::value == 8) {
                            if (ph == 1 || ph == 2) stage_spinor<P>(st, F.p, F.p_norm, ss, j);
                            if (ph == 3) stage_spinor<P>(st, F.t2, F.t2_norm, ss, j);
                            if (ph >= 2) stage_residual<P, NL, 8>(st, ph == 2 ? F.xs : F.rs, ss, j);
                        } else {
                            if (ph >= 2) stage_residual<P, NL, 9>(st, ph == 2 ? F.xs : F.rs, ss, j);
                        }
                    });
                    if (axpy)
                        pk_epi_axpy<P>(acc, prm.e[ph], hop, s8);
                    else
                        pk_epi_diag(acc, prm.e[ph], hop);
                    if (ph != 3) {
                        void* out    = axpy ? F.t2 : F.t1;
                        float* out_n = axpy ? F.t2_norm : F.t1_norm;
                        if constexpr (P == 16)
                            SlotF16::store(out, out_n, ss, j, acc);
                        else
                            SlotF32::store(out, ss, j, acc);
                    }
                    if (ph == 1)
                        pk_self_dot(acc, dre);
                    else if (ph == 2)
                        pk_cg_solution<P, NL>(sc[rhs].alpha, static_cast<float4*>(F.xs), ss, j, s8, s9);
                    else if (ph == 3)
                        pk_cg_residual<P, NL>(acc, sc[rhs].alpha, static_cast<float4*>(F.rs), ss, j, s8, s9, dre);
                }
                if (axpy) pk_partial<DOT_SELF>(dre, bc2(0.f), bc2(0.f), prm.partials, tile, nrhs, rhs);
            }
            if (!grid_barrier(&prm.ctl->arrived, &prm.ctl->error, target += gridDim.x, &ok)) return;
            if (axpy) {
                pcg_sums(prm.partials, prm.ntiles * PK_WARPS, nrhs, tot, smem);
                for (int r = threadIdx.x; r < nrhs; r += PK_THREADS) {
                    const double v[2] = {tot[r], 0.0};
                    RedArgs ra;
                    ra.sc  = &sc[r];
                    ra.fin = ph == 1 ? FIN_CG_ALPHA : FIN_CG_BETA;
                    finish_apply<2>(ra, v);
                    if (ph == 3) {
                        // judge the residual of the iteration before this one
                        if (!(it == 0 && (prm.first || ((prm.skip >> r) & 1u)))) {
                            const double q = prev[r], rn = sqrt(q);
                            judged[r]      = q;
                            judged_flag[r] = prev_flag[r];
                            if (rn > maxrr[r]) maxrr[r] = rn;
                            if (q != q || prev_flag[r] || rn < prm.delta * maxrr[r] || q < prm.f[r].thr) stop = 1;
                        }
                        prev[r]      = sc[r].resid;
                        prev_flag[r] = sc[r].flag;
                    }
                }
                __syncthreads();
            }
        }
        ++it;
        if (stop) break;
    }
    if (blockIdx.x == 0) {
        for (int r = threadIdx.x; r < nrhs; r += PK_THREADS) {
            *prm.f[r].sc         = sc[r];
            prm.ctl->judged[r]   = judged[r];
            prm.ctl->maxrr[r]    = maxrr[r];
            prm.ctl->flag[r]     = judged_flag[r];
        }
        if (threadIdx.x == 0) {
            prm.ctl->iters     = it;
            prm.ctl->undecided = !stop;
        }
    }
}

}  // namespace c2q
