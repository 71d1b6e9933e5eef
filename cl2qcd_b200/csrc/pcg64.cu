// pcg64.cu -- the iterations of the FP64 CG on QplusQminus_eo between two
// residual refreshes in one cooperative launch, for small lattices.
//
// The ordinary iteration (solvers.cu) is six dependent launches, replayed as a
// graph at best, with one thread per site in a sweep: at 8^4 that is 16 blocks on
// 148 SMs, each thread a chain of eight hops, and the iteration is bound by
// the launches and that chain.  Here the blocks stay resident and step through
// five phases with a grid barrier between them, and a sweep gives each of the
// eight hops of 32 sites to a warp of its own: the hops' half spinors meet in
// shared memory, where six warps add them up, two components each.  As in the
// mixed-precision CG, alpha comes from |Q- p|^2 = (p, Q+Q- p) after the second
// sweep (Q+ is the adjoint of Q-), so the third sweep updates x and the last
// one the residual; every block adds up the tiles' partial sums itself, in the
// same order, and keeps its own copy of the scalars.
//
// Semantics of physics/algorithms/solvers/cg.cpp:277-400 between refreshes.
#include <cstring>

#include "c2q_host.h"
#include "dslash.cuh"
#include "gridbar.cuh"

namespace c2q {

namespace {

constexpr int T64      = 32;   // sites per tile
constexpr int THREADS64 = 256;  // one warp per hop

struct Ctl64 {
    unsigned arrived, error;
    int iters, stop;
    double judged;
};

struct Params64 {
    double2 *p, *t1, *t2, *r, *x;
    const double2* gauge;
    Geom g;
    HopCoef c;
    EpiArgs e[4];
    SolverScalars* sc;
    double* partials;
    Ctl64* ctl;
    int ntiles;
    int iters;        // at most
    int p_ready;      // the first iteration's p is up to date
    int lag;          // judge each residual one iteration later (skip: not at the first iteration), else
    int skip;         //   after the iterations whose number is a multiple of check_every
    int check_every;
    int iter0, min_iter;
    double thr;
};

using C = Cplx<double>;

// fields change within the kernel: never through the non-coherent path
__device__ __forceinline__ C ldc(const double2* p)
{
    const double2 v = __ldcg(p);
    return cmk(v.x, v.y);
}

// Hop (MU, BACK) of one site: k U (psi_a + c psi_p) for a = 0, 1 into h[6][T64].
template <int NL, int MU, bool BACK>
__device__ __forceinline__ void hop64(const Params64& prm, const double2* in, int par, int nb, int li, double2* h)
{
    using T          = Proj<MU>;
    constexpr int c0 = BACK ? NegUnit<T::c0>::value : T::c0;
    constexpr int c1 = BACK ? NegUnit<T::c1>::value : T::c1;
    const size_t st  = (size_t)prm.g.stride;
    C psi[12], u[9];
#pragma unroll
    for (int k = 0; k < 12; ++k) psi[k] = ldc(in + k * st + nb);
    const double2* lk = prm.gauge + (size_t)(((BACK ? 1 - par : par) * 4 + MU) * NL) * st + li;
#pragma unroll
    for (int k = 0; k < NL; ++k) {
        const double2 v = __ldg(lk + k * st);
        u[k]            = cmk(v.x, v.y);
    }
    if (NL == 6) reconstruct_row2(u);
    const C w = cmk(prm.c.re[MU][BACK], prm.c.im[MU][BACK]);
#pragma unroll
    for (int a = 0; a < 2; ++a) {
        C q[3];
        if (a == 0)
            project<double, 0, T::p0, c0>(q, psi);
        else
            project<double, 1, T::p1, c1>(q, psi);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            C s;
            if (!BACK) {
                s = cmul(u[3 * r], q[0]);
                cmac(s, u[3 * r + 1], q[1]);
                cmac(s, u[3 * r + 2], q[2]);
            } else {
                s = cmulc(u[r], q[0]);
                cmacc(s, u[3 + r], q[1]);
                cmacc(s, u[6 + r], q[2]);
            }
            s                      = cmul(s, w);
            h[(3 * a + r) * T64] = make_double2(s.re, s.im);
        }
    }
}

// sum over the hops of conj(unit) times the half spinors, for the lower spin
// row 2 + LOW: partner (a, c) pairs read off the projector table
template <int MU, int LOW>
__device__ __forceinline__ void low_add(C& acc, const double2* h, int col)
{
    using T         = Proj<MU>;
    constexpr int a = T::p0 == 2 + LOW ? 0 : 1;
    constexpr int c = a == 0 ? T::c0 : T::c1;
    const double2 f = h[(size_t)(12 * MU + 3 * a + col) * T64];      // forward hop 2 MU
    const double2 b = h[(size_t)(12 * MU + 6 + 3 * a + col) * T64];  // backward hop: -c
    acc             = acc + mul_unit<ConjUnit<c>::value>(cmk(f.x - b.x, f.y - b.y));
}

template <int NL>
__global__ void __launch_bounds__(THREADS64, 2) pcg64_kernel(const Params64 prm)
{
    __shared__ double2 half[8 * 6 * T64];
    __shared__ double smem[32];
    __shared__ SolverScalars sc;
    __shared__ double prev, judged;
    __shared__ int ok, stop;
    const Geom& g   = prm.g;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t st = (size_t)g.stride;
    const double hop = prm.c.scale;
    unsigned target  = 0;
    if (threadIdx.x == 0) {
        sc     = *prm.sc;
        prev   = sc.resid;
        judged = __longlong_as_double(-1LL);  // NaN: nothing judged
        stop   = 0;
    }
    __syncthreads();
    int it = 0;
    while (it < prm.iters) {
        if (!(it == 0 && prm.p_ready)) {  // p = r + beta p
            const C mb = cmk(-sc.beta[0], -sc.beta[1]);
            for (int tile = blockIdx.x; tile < prm.ntiles; tile += gridDim.x)
                for (int e = threadIdx.x; e < 12 * T64; e += THREADS64) {
                    const int i = tile * T64 + (e & (T64 - 1));
                    if (i >= g.seo) continue;
                    const size_t at = (size_t)(e / T64) * st + i;
                    const C v       = ldc(prm.r + at) - cmul(ldc(prm.p + at), mb);
                    prm.p[at]       = make_double2(v.re, v.im);
                }
            if (!grid_barrier(&prm.ctl->arrived, &prm.ctl->error, target += gridDim.x, &ok)) return;
        }
#pragma unroll 1
        for (int ph = 0; ph < 4; ++ph) {
            // 0: t1 = diag D p   1: t2 = g5 (diag p - D t1), |t2|^2 -> alpha
            // 2: t1 = diag D t2, x += alpha p   3: r -= alpha g5 (diag t2 - D t1), |r|^2 -> beta
            const double2* in = ph == 0 ? prm.p : ph == 2 ? prm.t2 : prm.t1;
            const int par     = ph & 1;
            const EpiArgs& e  = prm.e[ph];
            for (int tile = blockIdx.x; tile < prm.ntiles; tile += gridDim.x) {
                const int i = tile * T64 + lane;
                if (i < g.seo) {
                    int rest     = i / g.nsh;
                    const int xh = i - rest * g.nsh;
                    const int y  = rest % g.ns;
                    rest /= g.ns;
                    const int z = rest % g.ns;
                    const int t = rest / g.ns;
                    const int x = 2 * xh + ((par + y + z + t) & 1);
                    const int row = g.nsh, pl = g.nsh * g.ns;
                    double2* h = half + (size_t)warp * 6 * T64 + lane;
                    int n;
                    switch (warp) {
                        case 0: hop64<NL, 0, false>(prm, in, par, t + 1 == g.nt ? i - (g.nt - 1) * g.vs_h : i + g.vs_h, i, h); break;
                        case 1:
                            n = t == 0 ? i + (g.nt - 1) * g.vs_h : i - g.vs_h;
                            hop64<NL, 0, true>(prm, in, par, n, n, h);
                            break;
                        case 2: hop64<NL, 1, false>(prm, in, par, i - xh + ((x + 1 == g.ns ? 0 : x + 1) >> 1), i, h); break;
                        case 3:
                            n = i - xh + ((x == 0 ? g.ns - 1 : x - 1) >> 1);
                            hop64<NL, 1, true>(prm, in, par, n, n, h);
                            break;
                        case 4: hop64<NL, 2, false>(prm, in, par, y + 1 == g.ns ? i - (g.ns - 1) * row : i + row, i, h); break;
                        case 5:
                            n = y == 0 ? i + (g.ns - 1) * row : i - row;
                            hop64<NL, 2, true>(prm, in, par, n, n, h);
                            break;
                        case 6: hop64<NL, 3, false>(prm, in, par, z + 1 == g.ns ? i - (g.ns - 1) * pl : i + pl, i, h); break;
                        default:
                            n = z == 0 ? i + (g.ns - 1) * pl : i - pl;
                            hop64<NL, 3, true>(prm, in, par, n, n, h);
                            break;
                    }
                }
                __syncthreads();
                double dv[1] = {0.0};
                if (warp < 6 && i < g.seo) {
                    // components 3 a + col and 6 + 3 a + col of the site
                    const int a = warp / 3, col = warp - 3 * a;
                    const double2* h = half + lane;
                    C v[2] = {cmk(0.0, 0.0), cmk(0.0, 0.0)};
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const double2 s = h[(size_t)(6 * q + warp) * T64];
                        v[0]            = v[0] + cmk(s.x, s.y);
                    }
                    if (a == 0) {
                        low_add<0, 0>(v[1], h, col);
                        low_add<1, 0>(v[1], h, col);
                        low_add<2, 0>(v[1], h, col);
                        low_add<3, 0>(v[1], h, col);
                    } else {
                        low_add<0, 1>(v[1], h, col);
                        low_add<1, 1>(v[1], h, col);
                        low_add<2, 1>(v[1], h, col);
                        low_add<3, 1>(v[1], h, col);
                    }
                    const double al = sc.alpha[0], ai = sc.alpha[1];
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        const size_t at = (size_t)(6 * b + warp) * st + i;
                        const C f       = b == 0 ? cmk(e.f1re, e.f1im) : cmk(e.f2re, e.f2im);
                        if (!par) {
                            const C o  = cmul(cmk(f.re * hop, f.im * hop), v[b]);
                            prm.t1[at] = make_double2(o.re, o.im);
                            if (ph == 2) {  // x += alpha p
                                C xv = ldc(prm.x + at);
                                cmac(xv, cmk(al, ai), ldc(prm.p + at));
                                prm.x[at] = make_double2(xv.re, xv.im);
                            }
                        } else {
                            const C m = cmul(f, ldc((ph == 1 ? prm.p : prm.t2) + at));
                            C o       = cmk(m.re - hop * v[b].re, m.im - hop * v[b].im);
                            if (b == 1) o = cmk(-o.re, -o.im);  // g5
                            if (ph == 1) {
                                prm.t2[at] = make_double2(o.re, o.im);
                            } else {  // r -= alpha v
                                const C rv = ldc(prm.r + at);
                                o          = rv - cmul(o, cmk(al, ai));
                                prm.r[at]  = make_double2(o.re, o.im);
                            }
                            dv[0] += o.re * o.re + o.im * o.im;
                        }
                    }
                }
                if (par) {
                    block_sum<1>(dv, smem);
                    if (threadIdx.x == 0) prm.partials[tile] = dv[0];
                } else {
                    __syncthreads();  // the half spinors are read: the next tile may write its own
                }
            }
            if (!grid_barrier(&prm.ctl->arrived, &prm.ctl->error, target += gridDim.x, &ok)) return;
            if (par) {
                // one fixed order: thread j takes partials j, j + 256, ...
                double s[1] = {0.0};
                for (int m = threadIdx.x; m < prm.ntiles; m += THREADS64) s[0] += __ldcg(prm.partials + m);
                block_sum<1>(s, smem);
                if (threadIdx.x == 0) {
                    const double v[2] = {s[0], 0.0};
                    RedArgs ra;
                    ra.sc  = &sc;
                    ra.fin = ph == 1 ? FIN_CG_ALPHA : FIN_CG_BETA;
                    finish_apply<2>(ra, v);
                    if (ph == 3) {
                        const int iter = prm.iter0 + it;
                        const double q = prm.lag ? prev : sc.resid;
                        if (prm.lag ? !(it == 0 && prm.skip) : iter % prm.check_every == 0) {
                            judged = q;
                            if (q != q || (q < prm.thr && iter >= prm.min_iter)) stop = 1;
                        }
                        prev = sc.resid;
                    }
                }
                __syncthreads();
            }
        }
        ++it;
        if (stop) break;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        *prm.sc          = sc;
        prm.ctl->iters  = it;
        prm.ctl->stop   = stop;
        prm.ctl->judged = judged;
    }
}

int blocks64(c2q_ctx* ctx, const void* kern, int ntiles, int* blocks)
{
    int per_sm = 0, sms = 0;
    C2Q_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, THREADS64, 0));
    C2Q_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    *blocks = ntiles < per_sm * sms ? ntiles : per_sm * sms;
    return *blocks < 1 ? fail(ctx, C2Q_CUDA_ERROR, "cooperative CG: no resident block") : C2Q_OK;
}

int go64(c2q_ctx* ctx, const void* kern, int blocks, Params64& prm)
{
    C2Q_CUDA(ctx, cudaMemsetAsync(prm.ctl, 0, sizeof(Ctl64), ctx->stream));
    if (ctx->cooperative == C2Q_COOPERATIVE_TEST)  // arrived: -1
        C2Q_CUDA(ctx, cudaMemsetAsync(&prm.ctl->arrived, 0xFF, sizeof prm.ctl->arrived, ctx->stream));
    void* args[] = {&prm};
    C2Q_CUDA(ctx, cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(THREADS64), args, 0, ctx->stream));
    ctx->launches++;
    return C2Q_OK;
}

}  // namespace

// Lattices of at most this many eo sites take the cooperative iterations: a
// phase is then at most about two and a half waves of tiles.  A solve's time over its
// iterations (its fixed part included), against the ordinary launches replayed as a
// graph: 8^4 19.3 us against 46.4, 12^3x16 (13824 sites) 37.3 against 45.8, 12^3x24
// (20736) 51.2 against 50.0, 16^4 (32768) 60.8 against 52.6.
constexpr int PCG64_MAX_SITES = 24000;

bool pcg64_applies(const c2q_ctx* ctx, int op, const c2q_gauge* gf)
{
    // (per-launch timing wants the sweeps as launches of their own)
    if (op != C2Q_OP_QPLUSQMINUS_EO || ctx->profiling || !ctx->cooperative || gf->geom.seo > PCG64_MAX_SITES)
        return false;
    return adjoint_weights(gf);
}

int pcg64_run(c2q_ctx* ctx, const c2q_gauge* g, int gkind, const Pcg64Solve& S, Pcg64Result* out)
{
    gauge_reader(g, ctx);
    int rc = gauge_ensure(const_cast<c2q_gauge*>(g), gkind);
    if (rc) return rc;
    Params64 prm;
    memset(&prm, 0, sizeof prm);
    auto lanes = [](const c2q_spinor_eo* f) { return static_cast<double2*>(f->data); };
    prm.p      = lanes(S.p);
    prm.t1     = lanes(S.t1);
    prm.t2     = lanes(S.t2);
    prm.r      = lanes(S.r);
    prm.x      = lanes(S.x);
    prm.gauge  = static_cast<const double2*>(g->store[gkind].data);
    prm.g      = S.x->geom;
    prm.c      = hop_coef(g, S.kappa);
    const bool tm = S.action == C2Q_ACTION_TWISTEDMASS;
    const EpiArgs one{1, 0, 1, 0, 0};
    prm.e[0]        = tm ? diag_epi(S.mubar, C2Q_DIAG_M_TM_INVERSE_MINUS, 0) : one;
    prm.e[1]        = tm ? diag_epi(S.mubar, C2Q_DIAG_M_TM_MINUS, 1) : one;
    prm.e[2]        = tm ? diag_epi(S.mubar, C2Q_DIAG_M_TM_INVERSE, 0) : one;
    prm.e[3]        = tm ? diag_epi(S.mubar, C2Q_DIAG_M_TM, 1) : one;
    prm.ntiles      = (prm.g.seo + T64 - 1) / T64;
    prm.sc          = ctx->scalars;
    prm.iters       = S.iters;
    prm.p_ready     = S.p_ready;
    prm.lag         = S.lag;
    prm.skip        = S.skip;
    prm.check_every = S.check_every;
    prm.iter0       = S.iter0;
    prm.min_iter    = S.min_iter;
    prm.thr         = S.thr;
    // the control block after the partials
    rc = ensure_partials(ctx, (size_t)prm.ntiles + 16);
    if (rc) return rc;
    prm.partials = ctx->partials;
    prm.ctl      = reinterpret_cast<Ctl64*>(ctx->partials + prm.ntiles + (prm.ntiles & 1));
    const void* kern = gkind_is_r12(gkind) ? (const void*)pcg64_kernel<6> : (const void*)pcg64_kernel<9>;
    int blocks       = 0;
    rc               = blocks64(ctx, kern, prm.ntiles, &blocks);
    if (rc) return rc;
    // counted, but not tested for room: these iterates differ from the ordinary launches'
    // by rounding, and results do not depend on what else runs
    const CoopRoom share(ctx->device, blocks, 0);
    rc = go64(ctx, kern, blocks, prm);
    if (!rc) rc = pinned_copy(ctx, ctx->host_pinned_dev, 0, prm.ctl, 0, sizeof(Ctl64));
    if (rc) return rc;
    C2Q_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    Ctl64 c;
    memcpy(&c, ctx->host_pinned, sizeof c);
    out->gave_up = c.error || c.iters < 1;
    if (out->gave_up) ++ctx->barrier_giveups;
    out->iters  = c.iters;
    out->stop   = c.stop;
    out->judged = c.judged;
    return C2Q_OK;
}

}  // namespace c2q
