// c2q_host.h -- host-side objects behind the C ABI: context (stream, reduction
// scratch, device scalars), gauge fields in every storage precision, eo spinor
// fields, and the launch wrappers the solvers are built from.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <map>
#include <string>
#include <vector>

#include "../../include/cl2qcd_b200.h"
#include "c2q_internal.cuh"
#include "blas.cuh"
#include "pack.cuh"
#include "reduce.cuh"

namespace c2q {

struct Field;

// Storage of one gauge field in one precision / compression.
struct GaugeStore {
    void* data = nullptr;
    size_t bytes = 0;
};

}  // namespace c2q

struct c2q_ctx {
    int device        = 0;
    cudaStream_t stream = nullptr;
    bool own_stream   = false;
    std::string err;
    long long launches = 0;
    // reduction scratch (partials), the last-block ticket and result slots
    double* partials       = nullptr;
    size_t partials_cap    = 0;  // doubles
    unsigned* ticket       = nullptr;
    double* red_result     = nullptr;  // 8 doubles
    double* host_pinned    = nullptr;  // 64 doubles, pinned
    c2q::SolverScalars* scalars = nullptr;  // device solver scalars (one set per context)
    // staging buffer for AoS host <-> device transfers
    void* staging          = nullptr;
    size_t staging_cap     = 0;
    // freed blocks of gauge objects (link_free; guarded by that file's mutex)
    struct LinkBlock {
        void* p      = nullptr;
        size_t bytes = 0;
    };
    LinkBlock link_cache[256];
    c2q_ctx* next_ctx = nullptr;  // the process's contexts (also under that mutex)
    // ring of pinned buffers between pageable host arrays and the device (hostcopy.cu)
    void* hc_ring        = nullptr;
    cudaEvent_t hc_ev[4] = {};
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    cudaEvent_t ring_ev[4] = {};  // residual ring of the pipelined solvers
    // The pipelined solvers copy each iteration's residual into ring_dev on the
    // context's stream (device memory only) and forward it to pinned host memory
    // on `monitor`, so the solve never waits on a write across PCIe, which a large
    // transfer of another stream can hold up; ring_ev[k] completes when slot k
    // has reached the host, mon_ev[k] when it is in ring_dev.
    cudaStream_t monitor   = nullptr;
    cudaEvent_t mon_ev[4]  = {};
    double* ring_dev       = nullptr;  // 4 slots x 16 right-hand sides x 4 doubles
    // optional per-launch dslash timing (c2q_ctx_profile)
    bool profiling = false;
    struct Timed {
        cudaEvent_t a, b;
        int prec;
        double sites;
        double bytes;  // algorithmic bytes of the launch
    };
    std::vector<Timed> timed;
    std::vector<cudaEvent_t> event_pool;
    // link storage of the explicit operator entry points: 0 18-real, 1 12-real
    int rec12 = 0;
    // autotuner of the paired-site dslash: launch shape -> chosen configuration
    struct TuneEntry {
        int cfg;
        float us[5];  // per choice; 0 where a choice does not apply to the shape
    };
    std::map<std::vector<int>, TuneEntry> tune;
    bool autotune = true;
    // dependent launches of the solver-loop kernels (launch_dep); environment
    // C2Q_DEPENDENT_LAUNCH=0 turns them off for new contexts
    bool pdl = true;
    int force_choice = -1;  // >= 0: every paired-site sweep uses this choice where it applies
    // launch predicate of a device-driven solve (SolverScalars::halt): while set,
    // every reducing BLAS and dslash launch skips its work once *halt_dev != 0
    const int* halt_dev = nullptr;
    // the cooperative CG iterations (c2q_ctx_set_cooperative), and how many launches were
    // given up at a barrier
    int cooperative           = C2Q_COOPERATIVE_ON;
    long long barrier_giveups = 0;
    int sm_count  = 0;
    // pinned ring of the batched solvers: 4 slots x 16 right-hand sides x 4 doubles
    double* batch_ring = nullptr;
    // device aliases of the pinned host buffers above (small solver transfers are
    // copied by a one-block kernel through them, keeping them off the copy engines,
    // where a large transfer of another stream would hold them up)
    double* host_pinned_dev = nullptr;
    double* batch_ring_dev  = nullptr;
};

struct c2q_gauge {
    c2q_ctx* ctx = nullptr;
    c2q_lattice lat{};
    c2q::Geom geom{};
    c2q::HopCoef coef{};  // hop phases of the lattice (scale unset)
    // [0] FP64 18-real, [1] FP64 12-real, [2] FP32 18-real, [3] FP32 12-real, [4] FP16 12-real,
    // [5] FP16 18-real; [6..9] the FP32 / FP16 kinds of the field in the temporal gauge
    c2q::GaugeStore store[10];
    // temporal gauge: the transformation G(x) (FP64, [parity][9 lanes][stride])
    // and the weight of the T hop leaving the last time slice
    c2q::GaugeStore tg_transform;
    double tg_lam_re = 1.0, tg_lam_im = 0.0;
    // max |row 2 - conj(row0 x row1)| of the uploaded links (-1: not measured yet)
    double rec12_dev = -1.0;
    // a context other than its own has queued work on it (gauge_reader)
    mutable std::atomic<bool> foreign{false};
};

struct c2q_spinor_eo {
    c2q_ctx* ctx = nullptr;
    c2q_lattice lat{};
    c2q::Geom geom{};
    int prec   = 64;
    void* data = nullptr;
    float* norm = nullptr;  // FP16 only
    bool owned = true;
};

namespace c2q {

enum GaugeKind {
    G64 = 0, G64R12 = 1, G32 = 2, G32R12 = 3, G16R12 = 4, G16 = 5,
    G32TG = 6, G32R12TG = 7, G16R12TG = 8, G16TG = 9,  // the same in the temporal gauge
    GAUGE_KINDS = 10
};
inline bool gkind_is_tg(int k) { return k >= G32TG && k <= G16TG; }
inline bool gkind_is_r12(int k) { return k == G64R12 || k == G32R12 || k == G16R12 || k == G32R12TG || k == G16R12TG; }
// the temporal-gauge kind of a FP32 / FP16 kind
inline int gkind_tg(int k)
{
    return k == G32 ? G32TG : k == G32R12 ? G32R12TG : k == G16R12 ? G16R12TG : k == G16 ? G16TG : -1;
}

// ---- status plumbing ----
int fail(c2q_ctx* ctx, int code, const std::string& msg);
int cuda_fail(c2q_ctx* ctx, cudaError_t e, const char* where);
#define C2Q_CUDA(ctx, call)                                   \
    do {                                                      \
        cudaError_t _e = (call);                              \
        if (_e != cudaSuccess) return ::c2q::cuda_fail((ctx), _e, #call); \
    } while (0)

// ---- geometry / coefficients ----
bool make_geom(const c2q_lattice& lat, Geom* g);
bool same_lattice(const c2q_lattice& a, const c2q_lattice& b);
// A constant as the reference passes it in its build options (16 significant digits).
double as_build_option(double v);
// Hop coefficients for one launch: -kappa * boundary phase (and chemical potential on T).
HopCoef hop_coef(const c2q_lattice& lat, double kappa);
// the same for the gauge field's lattice, from the phases it keeps (forming them
// goes through the text of sixteen numbers, some microseconds of each launch)
HopCoef hop_coef(const c2q_gauge* g, double kappa);
EpiArgs diag_epi(double mubar, int which, int gamma5);

// gauge storage for operator sweeps at precision `prec` (FP16 links are always 12-real)
int gkind_for(int prec, int rec12);

// ---- fields ----
// Allocate a spinor field of storage precision `prec` (stream-ordered allocation).
// Its contents are undefined unless `clear`: work fields are written whole before
// they are read, and no kernel reads the padding after the last site.
int field_alloc(c2q_ctx* ctx, const c2q_lattice& lat, int prec, c2q_spinor_eo* f, bool clear = false);
void field_free(c2q_spinor_eo* f);
size_t field_bytes(const Geom& g, int prec);
// Memory of the gauge objects (links, derived copies, momenta).  A freed block stays
// with the context for the next request of the same size, so that a program that
// goes from one gauge field to the next pays for no new mappings and no device-wide
// frees; at most LINK_KEEP bytes are kept by all contexts of the process together.  All
// go back when any device allocation of the library finds no memory (device_alloc),
// before a server takes its budget from what is free, and a context's when it ends or
// is asked (c2q_ctx_trim).  link_free keeps a block only if `quiet`: no kernel may
// still use it; else it is freed, which waits for the device.
// Any thread may call these for any context (a solve on one context builds the copies
// of another's gauge field).
// (cudaMalloc'ed: the stream-ordered pool maps new memory several times slower,
// 35 ms against 6 ms for the copies of a first 32^3x64 field.)
constexpr size_t LINK_KEEP = (size_t)22 << 30;  // an eighth of a B200
cudaError_t link_alloc(c2q_ctx* ctx, void** p, size_t bytes);
void link_free(c2q_ctx* ctx, void* p, size_t bytes, bool quiet);
size_t link_trim(c2q_ctx* ctx);  // gives the kept blocks back; their bytes
size_t link_trim_device(int device);  // those of every context on the device
// cudaMalloc, and cudaMallocAsync on the context's stream; where memory has run out,
// once more after every context's kept blocks and the pool's unused memory went back
cudaError_t device_alloc(c2q_ctx* ctx, void** p, size_t bytes);
cudaError_t device_alloc_async(c2q_ctx* ctx, void** p, size_t bytes);
// Waits for the context's stream; whether nothing can use an object's memory any more.
// (Not for the device: a device is not to be synchronised while another thread captures
// a stream of it.)
inline bool stream_quiet(c2q_ctx* ctx) { return cudaStreamSynchronize(ctx->stream) == cudaSuccess; }
// Called where work of `ctx` that reads the links is queued: the block of a field that
// other contexts have read is not recycled (waiting for its own stream says nothing
// about theirs).
inline void gauge_reader(const c2q_gauge* g, const c2q_ctx* ctx)
{
    if (g->ctx != ctx) g->foreign.store(true, std::memory_order_relaxed);
}
int gauge_ensure(c2q_gauge* g, int kind);  // builds a lower-precision copy on first use
// frees every copy derived from the FP64 18-real links (rebuilt on next use)
int gauge_drop_derived(c2q_gauge* g);
// 12-real FP64 links are the same operator as the uploaded 18-real ones when
// row 2 of every link equals conj(row0 x row1) to this tolerance (unitarity.cu)
constexpr double REC12_EXACT_TOL = 1e-13;
bool rec12_exact(c2q_gauge* g);
// the FP64 links a solver's residuals use: 12-real only where they are the same operator
inline int gk64_for(const c2q_gauge* g, int rec12)
{
    return rec12 && rec12_exact(const_cast<c2q_gauge*>(g)) ? G64R12 : G64;
}

// ---- temporal gauge (tgauge.cu) ----
// The inner solves of the mixed-precision CG may run on the field transformed
// by G(x, t) = c^t prod_{t' < t} U_T(x, t') (c the forward T phase): every T
// link becomes the identity except the one leaving the last time slice, which
// becomes lambda W (W in SU(3), lambda = c^NT), all hop phases real.  Possible
// when the T weights are pure phases and the spatial ones real.
bool tg_applicable(const c2q_lattice& lat);
// the transformation G and lambda (first use)
int tg_ensure(c2q_gauge* g);
// the transformed links as an FP64 9-lane store (the layout of G64) in out
int tg_links_fp64(c2q_gauge* g, void* out);
// out (FP32) = G in (FP64), on the sites of parity 1 (those of the CG vectors)
int tg_to_inner(c2q_ctx* ctx, const c2q_gauge* g, c2q_spinor_eo* out, const c2q_spinor_eo* in);
// x (FP64) += G^dagger (xs + alpha p) (alpha from sc; sc null: xs only), xs = 0
int tg_accumulate(c2q_ctx* ctx, const c2q_gauge* g, c2q_spinor_eo* x, c2q_spinor_eo* xs, const c2q_spinor_eo* p,
                  const SolverScalars* sc);
int ensure_staging(c2q_ctx* ctx, size_t bytes);
// Host array -> device and back on the context's stream, at PCIe rate from and into
// pageable memory too (hostcopy.cu).  copy_to_host returns when the array is
// filled; copy_to_device may still be in flight, but has read a pageable array
// (a pinned one must stay valid until the stream has passed the copy).
int copy_to_device(c2q_ctx* ctx, void* dev, const void* host, size_t bytes);
int copy_to_host(c2q_ctx* ctx, void* host, const void* dev, size_t bytes);
// Small copies (multiples of 4 bytes) between device memory and the device alias
// of a pinned host buffer, by a one-block kernel on the context's stream:
// `height` rows of `width` bytes, rows `dpitch` / `spitch` bytes apart.
int pinned_copy(c2q_ctx* ctx, void* dst, size_t dpitch, const void* src, size_t spitch, size_t width,
                int height = 1, cudaStream_t stream = nullptr);
// Residual ring slot k (n rows of `width` bytes at src, row pitch spitch): into
// ring_dev on the context's stream, then to the pinned host buffer dst_host_dev
// (the device alias of a pinned slot) on the monitor stream; ring_ev[k % 4]
// completes when the host can read it.
// (src null: a kernel on the stream has filled ring_slot(ctx, k)).
inline double* ring_slot(c2q_ctx* ctx, int k) { return ctx->ring_dev + (size_t)(k % 4) * 16 * 4; }
int ring_push(c2q_ctx* ctx, int k, double* dst_host_dev, const void* src, size_t spitch, size_t width, int n);
int ensure_partials(c2q_ctx* ctx, size_t blocks);

template <int P>
inline SpinorPtr<P> sptr(const c2q_spinor_eo* f)
{
    return SpinorPtr<P>{f ? f->data : nullptr, f ? f->norm : nullptr, f ? f->geom.seo / 2 : 0};
}

// ---- launches (all stream-ordered on ctx->stream) ----
struct DotSpec {
    int mode = 0;  // DotMode
    const c2q_spinor_eo* y = nullptr;
    int fin = FIN_STORE_RESULT;
};

// One dslash parity sweep at the fields' storage precision P.
int launch_dslash(c2q_ctx* ctx, const c2q_gauge* g, int gkind, c2q_spinor_eo* out, const c2q_spinor_eo* in,
                  int out_parity, double kappa, int epi, const EpiArgs& e, const c2q_spinor_eo* x,
                  const DotSpec& dot);
struct BlasSpec {
    int op = 0;
    Coef a{0, 0, nullptr, 1}, b{0, 0, nullptr, 1};
    c2q_spinor_eo* out = nullptr;
    const c2q_spinor_eo *x = nullptr, *y = nullptr, *z = nullptr;
    const c2q_spinor_eo* w = nullptr;  // B_BICG_XR
    c2q_spinor_eo* out2    = nullptr;  // B_BICG_XR
    int dot = 0;
    int fin = FIN_STORE_RESULT;
    int fin_arg = 0;
};
int launch_blas(c2q_ctx* ctx, const BlasSpec& s);
int launch_cg_update(c2q_ctx* ctx, c2q_spinor_eo* x, c2q_spinor_eo* r, const c2q_spinor_eo* p,
                     const c2q_spinor_eo* v);
int launch_cg_p(c2q_ctx* ctx, c2q_spinor_eo* p, const c2q_spinor_eo* r);
int launch_convert(c2q_ctx* ctx, c2q_spinor_eo* out, const c2q_spinor_eo* in);

// A batch of right-hand sides for one sweep of the paired-site dslash
// (FP32 / FP16 fields, pdslash.cuh): per right-hand side r, out[r] = epilogue
// of the hopping term on in[r], with x[r] the EPI_AXPY operand, y[r] the DOT_Y
// partner and sc[r] the solver scalars its reduction finishes into.
constexpr int MAX_BATCH = PK_MAX_RHS;
struct PkBatch {
    int n = 0;
    c2q_spinor_eo* out[MAX_BATCH] = {};
    const c2q_spinor_eo* in[MAX_BATCH] = {};
    const c2q_spinor_eo* x[MAX_BATCH] = {};
    const c2q_spinor_eo* y[MAX_BATCH] = {};
    SolverScalars* sc[MAX_BATCH] = {};
    int out_parity = 0;
    double kappa = 0;
    int epi = 0;
    EpiArgs e{1, 0, 1, 0, 0};
    int dot_mode = 0;
    int fin = FIN_STORE_RESULT;
};
int launch_pdslash(c2q_ctx* ctx, const c2q_gauge* g, int gkind, const PkBatch& B);
// Batched fermion matrix on reduced-precision fields: out[r] = A in[r] for
// r < n, tmp1/tmp2 per right-hand side; optionally reduces <y[r], out[r]>
// into sc[r] with finisher `fin` (for QplusQminus_eo with y = in, as
// |Qminus_eo in|^2, which equals it because Qplus_eo = Qminus_eo^dagger).
// With r_update (QplusQminus_eo, y = in) the last sweep instead applies the CG
// residual update r[r] -= alpha A in[r] and reduces |r|^2 into sc[r] (FIN_CG_BETA);
// out[r] is then not written; with x_update as well, the third sweep applies the
// CG solution update x_update[r] += alpha in[r] (FP32 x_update).
int apply_operator_batch(c2q_ctx* ctx, int op, int n, c2q_spinor_eo* const* out, const c2q_gauge* g, int gkind,
                         const c2q_spinor_eo* const* in, double kappa, double mubar, int action,
                         c2q_spinor_eo* const* tmp1, c2q_spinor_eo* const* tmp2, int dot_mode,
                         const c2q_spinor_eo* const* y, int fin, SolverScalars* const* sc, int* sweeps,
                         c2q_spinor_eo* const* r_update = nullptr, c2q_spinor_eo* const* x_update = nullptr);
// Iterations of the mixed-precision CG on QplusQminus_eo in one cooperative
// launch (pcg.cuh), for the right-hand sides of a batch that share a field in
// the temporal gauge: from their search directions p, FP32 residuals rs and
// solution increments xs and device scalars sc, until one of them needs the
// host (a reliable update is due, or its residual is no number) or `iters` are
// done.  Bitwise the iterates of apply_operator_batch with mix_p.
struct PcgBatch {
    int n = 0;
    c2q_spinor_eo *p[MAX_BATCH] = {}, *t1[MAX_BATCH] = {}, *t2[MAX_BATCH] = {}, *rs[MAX_BATCH] = {},
                  *xs[MAX_BATCH] = {};
    SolverScalars* sc[MAX_BATCH] = {};
    double thr[MAX_BATCH] = {}, maxrr[MAX_BATCH] = {};
    bool skip[MAX_BATCH] = {};  // the residual before the first iteration is not to be judged
    double kappa = 0, mubar = 0, delta = 0;
    int action = 0, first = 0, iters = 0;
    void* ctl = nullptr;  // pcg_ctl_bytes() of device memory
};
struct PcgResult {
    bool gave_up;  // at a barrier: p, rs, xs and the scalars hold no one iteration's state
    int iters;     // done; the last one judged the residual of the one before
    bool undecided;  // they ended at the iteration limit
    double judged[MAX_BATCH], maxrr[MAX_BATCH];
    int flag[MAX_BATCH];
};
// *tiles: the blocks a right-hand side takes on a lattice of geometry g; *room: the blocks
// of the device, 0 where these iterations are not to be taken.  A batch takes them if
// every tile of every right-hand side has a resident block of its own (one
// wave).  With more, a phase runs a second, partly empty wave between two
// barriers and the ordinary launches are as fast or faster: FP16, a solve's time over its
// iterations, against the ordinary launches replayed as a graph, 16^3x32 (256 tiles, one
// wave of 444 blocks) 39 us against 48 us, 12^3x24 with five sources (405) 64.5 against
// 65.0; 16^3x32 with two sources (512) 89 against 71, 20^3x40 (625) 90 against 80, four sources
// at 16^3x32 133 against 111.
int pcg_capacity(c2q_ctx* ctx, int prec, int gkind, const Geom& g, int* tiles, int* room);
// Blocks of cooperative CG launches in flight on a device, all contexts together.  The
// hardware starts such a launch only once all its blocks have room, so grids that do
// not fit side by side run one after the other, and whatever is queued behind them
// waits: two 16^3x32 solves at a time took 20.7 ms each against 17.8 ms with launches of
// their own, a light request beside three of them up to 33 ms against 13 ms.  `most`
// blocks fit with what is in flight, or (most 0) they are counted without a test.
bool coop_enter(int device, int blocks, int most);
void coop_leave(int device, int blocks);
struct CoopRoom {  // a launch's share, given back when its results are in
    int device, blocks;
    bool got;
    CoopRoom(int device, int blocks, int most)
        : device(device), blocks(blocks), got(blocks > 0 && coop_enter(device, blocks, most))
    {
    }
    ~CoopRoom() { leave(); }
    void leave()
    {
        if (got) coop_leave(device, blocks);
        got = false;
    }
    CoopRoom(const CoopRoom&)            = delete;
    CoopRoom& operator=(const CoopRoom&) = delete;
};
size_t pcg_ctl_bytes();
// launch without waiting; collect waits for the stream, and so for what was queued since
int pcg_launch(c2q_ctx* ctx, const c2q_gauge* g, int gkind, const PcgBatch& B);
int pcg_collect(c2q_ctx* ctx, const PcgBatch& B, PcgResult* out);
// device memory, nonzero once the iterations have ended undecided
const int* pcg_undecided(const PcgBatch& B);
// Iterations of the FP64 CG on QplusQminus_eo in one cooperative launch
// (pcg64.cu), with the context's solver scalars: until a judged residual is
// below thr (from iteration min_iter on) or no number, or `iters` are done.
struct Pcg64Solve {
    c2q_spinor_eo *x, *r, *p, *t1, *t2;
    double kappa, mubar;
    int action;
    int iter0, iters, min_iter;
    int p_ready;      // p is up to date for the first iteration (a refresh set it)
    int lag;          // 1: judge each residual one iteration later (skip: not at the first iteration)
    int skip;
    int check_every;  // lag 0: judge iterations whose number is a multiple of this, at once
    double thr;
};
struct Pcg64Result {
    bool gave_up;  // at a barrier: x may hold a part of the last update, the rest no one iteration's state
    int iters, stop;
    double judged;
};
bool pcg64_applies(const c2q_ctx* ctx, int op, const c2q_gauge* g);
int pcg64_run(c2q_ctx* ctx, const c2q_gauge* g, int gkind, const Pcg64Solve& S, Pcg64Result* out);
// an event for per-launch profiling (from the context's pool)
cudaEvent_t profile_event(c2q_ctx* ctx);

// Fermion matrix application at the fields' precision.  tmp1/tmp2 are
// scratch fields of the same precision.  `dot` applies to the last sweep.
int apply_operator(c2q_ctx* ctx, int op, c2q_spinor_eo* out, const c2q_gauge* g, int gkind,
                   const c2q_spinor_eo* in, double kappa, double mubar, int action, c2q_spinor_eo* tmp1,
                   c2q_spinor_eo* tmp2, const DotSpec& dot, int* sweeps);

// Q+Q- in with the FP64 CG's vector updates fused in: alpha = omega / |Q- in|^2 after
// the second sweep ((in, Q+Q- in) where Q+ is the adjoint of Q-), x += alpha in in
// the third, r -= alpha Q+Q- in with |r|^2 -> beta in the last.
int apply_qpqm_cg(c2q_ctx* ctx, const c2q_gauge* g, int gkind, const c2q_spinor_eo* in, double kappa, double mubar,
                  int action, c2q_spinor_eo* tmp1, c2q_spinor_eo* tmp2, c2q_spinor_eo* x, c2q_spinor_eo* r,
                  int* sweeps);
// every backward hop weight is the conjugate of the forward one (no real chemical
// potential): Q+ is the adjoint of Q-
bool adjoint_weights(const c2q_gauge* g);

// Read back `n` doubles of device memory synchronously through pinned memory.
int read_scalars(c2q_ctx* ctx, const double* dev, int n, double* host);

}  // namespace c2q
