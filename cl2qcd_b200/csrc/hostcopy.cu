// hostcopy.cu -- transfers between pageable host arrays and the device.
//
// A copy from or to pageable memory runs through the driver's staging at the
// rate of one host thread (and, into fresh memory, of its page faults), a
// fraction of PCIe.  Here the array crosses in chunks through a small ring of
// pinned buffers of the context: several host threads copy one chunk while the
// copy engine moves the others.
#include <omp.h>

#include <algorithm>
#include <cstring>

#include "c2q_host.h"

namespace c2q {

// Ring of pinned buffers: 4 x 4 MiB keeps the engine busy while a chunk is
// being copied by the host; smaller arrays than two chunks take the plain copy.
constexpr size_t HC_CHUNK = (size_t)4 << 20;
constexpr int HC_RING     = 4;

static void parallel_copy(char* dst, const char* src, size_t n)
{
    constexpr size_t PIECE = (size_t)256 << 10;
    const long long pieces = (long long)((n + PIECE - 1) / PIECE);
    // eight fill PCIe; fewer where the caller's OpenMP setting or the process's cores say so
    const int threads = std::max(1, std::min({8, omp_get_num_procs(), omp_get_max_threads()}));
#pragma omp parallel for num_threads(threads) schedule(static)
    for (long long k = 0; k < pieces; ++k) {
        const size_t at = (size_t)k * PIECE;
        memcpy(dst + at, src + at, std::min(PIECE, n - at));
    }
}

// whether the ring serves this copy (and make the ring; without pinned memory for it the
// copy goes through the driver's staging)
static int use_ring(c2q_ctx* ctx, const void* host, size_t bytes, bool* ring)
{
    *ring = false;
    if (bytes < 2 * HC_CHUNK) return C2Q_OK;
    cudaPointerAttributes a;
    const cudaError_t e = cudaPointerGetAttributes(&a, host);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return C2Q_OK;
    }
    if (a.type != cudaMemoryTypeUnregistered) return C2Q_OK;  // pinned: the engine takes it as it is
    if (!ctx->hc_ring) {
        for (auto& ev : ctx->hc_ev)
            if (!ev) C2Q_CUDA(ctx, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming));
        if (cudaMallocHost(&ctx->hc_ring, HC_RING * HC_CHUNK) != cudaSuccess) {
            cudaGetLastError();
            ctx->hc_ring = nullptr;
            return C2Q_OK;
        }
    }
    *ring = true;
    return C2Q_OK;
}

int copy_to_device(c2q_ctx* ctx, void* dev, const void* host, size_t bytes)
{
    bool ring = false;
    int rc    = use_ring(ctx, host, bytes, &ring);
    if (rc) return rc;
    if (!ring) {
        C2Q_CUDA(ctx, cudaMemcpyAsync(dev, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
        return C2Q_OK;
    }
    const long long n = (long long)((bytes + HC_CHUNK - 1) / HC_CHUNK);
    for (long long k = 0; k < n; ++k) {
        const size_t at = (size_t)k * HC_CHUNK, m = std::min(HC_CHUNK, bytes - at);
        char* buf       = static_cast<char*>(ctx->hc_ring) + (size_t)(k % HC_RING) * HC_CHUNK;
        if (k >= HC_RING) C2Q_CUDA(ctx, cudaEventSynchronize(ctx->hc_ev[k % HC_RING]));
        parallel_copy(buf, static_cast<const char*>(host) + at, m);
        C2Q_CUDA(ctx, cudaMemcpyAsync(static_cast<char*>(dev) + at, buf, m, cudaMemcpyHostToDevice, ctx->stream));
        C2Q_CUDA(ctx, cudaEventRecord(ctx->hc_ev[k % HC_RING], ctx->stream));
    }
    // the ring may be written again by the next copy
    for (long long k = std::max(0LL, n - HC_RING); k < n; ++k)
        C2Q_CUDA(ctx, cudaEventSynchronize(ctx->hc_ev[k % HC_RING]));
    return C2Q_OK;
}

int copy_to_host(c2q_ctx* ctx, void* host, const void* dev, size_t bytes)
{
    bool ring = false;
    int rc    = use_ring(ctx, host, bytes, &ring);
    if (rc) return rc;
    if (!ring) {
        C2Q_CUDA(ctx, cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream));
        C2Q_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        return C2Q_OK;
    }
    const long long n = (long long)((bytes + HC_CHUNK - 1) / HC_CHUNK);
    auto issue        = [&](long long k) -> int {
        const size_t at = (size_t)k * HC_CHUNK, m = std::min(HC_CHUNK, bytes - at);
        char* buf       = static_cast<char*>(ctx->hc_ring) + (size_t)(k % HC_RING) * HC_CHUNK;
        C2Q_CUDA(ctx, cudaMemcpyAsync(buf, static_cast<const char*>(dev) + at, m, cudaMemcpyDeviceToHost, ctx->stream));
        C2Q_CUDA(ctx, cudaEventRecord(ctx->hc_ev[k % HC_RING], ctx->stream));
        return C2Q_OK;
    };
    for (long long k = 0; k < std::min<long long>(n, HC_RING) && !rc; ++k) rc = issue(k);
    for (long long k = 0; k < n && !rc; ++k) {
        const size_t at = (size_t)k * HC_CHUNK, m = std::min(HC_CHUNK, bytes - at);
        C2Q_CUDA(ctx, cudaEventSynchronize(ctx->hc_ev[k % HC_RING]));
        parallel_copy(static_cast<char*>(host) + at,
                      static_cast<const char*>(ctx->hc_ring) + (size_t)(k % HC_RING) * HC_CHUNK, m);
        if (k + HC_RING < n) rc = issue(k + HC_RING);
    }
    return rc;
}

}  // namespace c2q
