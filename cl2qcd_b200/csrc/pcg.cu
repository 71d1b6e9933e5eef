// pcg.cu -- host side of pcg.cuh: the cooperative launch that runs the
// iterations of the mixed-precision CG on small lattices.
#include <atomic>
#include <cstring>

#include "c2q_host.h"
#include "pcg.cuh"

namespace c2q {

template <int P, int NL>
static int pcg_resident(c2q_ctx* ctx, int* blocks)
{
    constexpr size_t smem = PkStage<P, NL, 0>::BYTES;
    const void* kern      = (const void*)pcg_kernel<P, NL>;
    C2Q_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0, sms = 0;
    C2Q_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, PK_THREADS, smem));
    C2Q_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device));
    *blocks = per_sm * sms;
    return C2Q_OK;
}

static std::atomic<int> coop_blocks[64];

bool coop_enter(int device, int blocks, int most)
{
    std::atomic<int>& in_flight = coop_blocks[device & 63];
    int now                     = in_flight.load(std::memory_order_relaxed);
    do {
        if (most && now + blocks > most) return false;
    } while (!in_flight.compare_exchange_weak(now, now + blocks, std::memory_order_relaxed));
    return true;
}

void coop_leave(int device, int blocks) { coop_blocks[device & 63].fetch_sub(blocks, std::memory_order_relaxed); }

int pcg_capacity(c2q_ctx* ctx, int prec, int gkind, const Geom& g, int* tiles, int* room)
{
    *tiles = (g.seo / 2 + PK_THREADS - 1) / PK_THREADS;
    *room  = 0;
    // (per-launch timing and a pinned sweep choice want the sweeps as launches of their own)
    if (ctx->profiling || ctx->force_choice >= 0 || !ctx->cooperative) return C2Q_OK;
    return prec == 16 ? (gkind_is_r12(gkind) ? pcg_resident<16, 6>(ctx, room) : pcg_resident<16, 9>(ctx, room))
                      : (gkind_is_r12(gkind) ? pcg_resident<32, 6>(ctx, room) : pcg_resident<32, 9>(ctx, room));
}

// where the control block lands in the context's pinned buffer (read_scalars uses its head)
constexpr int PCG_PINNED = 16;

size_t pcg_ctl_bytes() { return sizeof(PcgCtl); }

template <int P, int NL>
static int pcg_go(c2q_ctx* ctx, PcgParams& prm)
{
    constexpr size_t smem = PkStage<P, NL, 0>::BYTES;
    const void* kern      = (const void*)pcg_kernel<P, NL>;
    const int blocks      = prm.ntiles * prm.nrhs;  // pcg_capacity holds them all
    C2Q_CUDA(ctx, cudaMemsetAsync(prm.ctl, 0, sizeof(PcgCtl), ctx->stream));
    if (ctx->cooperative == C2Q_COOPERATIVE_TEST)  // arrived: -1
        C2Q_CUDA(ctx, cudaMemsetAsync(&prm.ctl->arrived, 0xFF, sizeof prm.ctl->arrived, ctx->stream));
    void* args[] = {&prm};
    C2Q_CUDA(ctx, cudaLaunchCooperativeKernel(kern, dim3(blocks), dim3(PK_THREADS), args, smem, ctx->stream));
    ctx->launches++;
    return C2Q_OK;
}

int pcg_launch(c2q_ctx* ctx, const c2q_gauge* g, int gkind, const PcgBatch& B)
{
    gauge_reader(g, ctx);
    PcgParams prm;
    memset(&prm, 0, sizeof prm);
    const c2q_spinor_eo* ref = B.p[0];
    const bool tm            = B.action == C2Q_ACTION_TWISTEDMASS;
    for (int r = 0; r < B.n; ++r) {
        PcgRhs& F = prm.f[r];
        F.p       = B.p[r]->data;
        F.p_norm  = B.p[r]->norm;
        F.t1      = B.t1[r]->data;
        F.t1_norm = B.t1[r]->norm;
        F.t2      = B.t2[r]->data;
        F.t2_norm = B.t2[r]->norm;
        F.rs      = B.rs[r]->data;
        F.xs      = B.xs[r]->data;
        F.sc      = B.sc[r];
        F.thr     = B.thr[r];
        F.maxrr   = B.maxrr[r];
        if (B.skip[r]) prm.skip |= 1u << r;
    }
    pk_stencil_args(ref, g, gkind, B.kappa, &prm);
    // Q+ Q-: the sweeps of Q- (minus factors), then those of Q+
    const EpiArgs one{1, 0, 1, 0, 0}, one5{1, 0, 1, 0, 1};
    prm.e[0]   = tm ? diag_epi(B.mubar, C2Q_DIAG_M_TM_INVERSE_MINUS, 0) : one;
    prm.e[1]   = tm ? diag_epi(B.mubar, C2Q_DIAG_M_TM_MINUS, 1) : one5;
    prm.e[2]   = tm ? diag_epi(B.mubar, C2Q_DIAG_M_TM_INVERSE, 0) : one;
    prm.e[3]   = tm ? diag_epi(B.mubar, C2Q_DIAG_M_TM, 1) : one5;
    prm.nrhs   = B.n;
    prm.ntiles = (prm.g.H + PK_THREADS - 1) / PK_THREADS;
    prm.delta  = B.delta;
    prm.first  = B.first;
    prm.iters  = B.iters;
    int rc     = ensure_partials(ctx, (size_t)prm.ntiles * PK_WARPS * B.n);
    if (rc) return rc;
    prm.partials = ctx->partials;
    prm.ctl      = static_cast<PcgCtl*>(B.ctl);
    if (ref->prec == 16)
        rc = gkind_is_r12(gkind) ? pcg_go<16, 6>(ctx, prm) : pcg_go<16, 9>(ctx, prm);
    else
        rc = gkind_is_r12(gkind) ? pcg_go<32, 6>(ctx, prm) : pcg_go<32, 9>(ctx, prm);
    if (rc) return rc;
    static_assert(sizeof(PcgCtl) <= (64 - PCG_PINNED) * sizeof(double), "the control block fits the pinned buffer");
    return pinned_copy(ctx, ctx->host_pinned_dev + PCG_PINNED, 0, prm.ctl, 0, sizeof(PcgCtl));
}

const int* pcg_undecided(const PcgBatch& B) { return &static_cast<const PcgCtl*>(B.ctl)->undecided; }

int pcg_collect(c2q_ctx* ctx, const PcgBatch& B, PcgResult* out)
{
    C2Q_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    PcgCtl c;
    memcpy(&c, ctx->host_pinned + PCG_PINNED, sizeof c);
    out->gave_up = c.error || c.iters < 1;
    if (out->gave_up) {
        ++ctx->barrier_giveups;
        return C2Q_OK;
    }
    out->iters     = c.iters;
    out->undecided = c.undecided;
    for (int r = 0; r < B.n; ++r) {
        out->judged[r] = c.judged[r];
        out->maxrr[r]  = c.maxrr[r];
        out->flag[r]   = c.flag[r];
    }
    return C2Q_OK;
}

}  // namespace c2q
