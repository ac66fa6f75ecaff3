// Device blocks to pageable host memory.
//
// A cudaMemcpy to memory that is not pinned runs through the driver's own staging on one thread, and
// the first touch of a fresh result's pages comes on top: 61 ms for the 136 MB of a 9,000-bus grid's
// sensitivities (2.2 GB/s), where the link needs 2.4 ms.  Here the block comes in 8 MB pieces through
// four pinned slots owned by the context, and up to eight host threads copy each piece out, with
// the sign the caller wants.  Bound: the host threads' copies into untouched memory.
#include <algorithm>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <mutex>
#include <thread>

#include "bpf_internal.cuh"

namespace bpf {

constexpr size_t kSlotDoubles = size_t(1) << 20;   // 8 MB
constexpr int kSlots = 4;
constexpr int kCopyThreads = 8;

static void copy_out(double *dst, const double *src, size_t len, bool negate) {
    if (!negate) {
        std::memcpy(dst, src, sizeof(double) * len);
        return;
    }
    for (size_t i = 0; i < len; i++) dst[i] = -src[i];
}

// What the copying threads and the issuing one share: how many threads copy (-1: not known yet), pieces that have
// arrived, and threads through with the latest.
struct CopyBoard {
    std::mutex mu;
    std::condition_variable cv;
    int threads = -1;
    size_t arrived = 0;
    bool stop = false;
    int done = 0;
};

}  // namespace bpf

using namespace bpf;

extern "C" bpf_status bpf_block_to_host(bpf_ctx *ctx, int n, int p, const double *X, int ldx, double *host, int negate) {
    if (!ctx) return BPF_ERR_INVALID_VALUE;
    if (n < 0 || p < 0 || (n > 0 && p > 0 && (!X || !host)))
        return set_error(ctx, BPF_ERR_INVALID_VALUE, "block_to_host: invalid argument");
    if (ldx < std::max(1, n)) return set_error(ctx, BPF_ERR_DIMENSION, "block_to_host: ldx < n");
    if (n == 0 || p == 0) return BPF_SUCCESS;
    const size_t total = (size_t)n * p;
    const bool linear = ldx == n || p == 1;
    // a piece: a run of the block where it is contiguous, else whole columns
    const size_t piece = linear ? kSlotDoubles : kSlotDoubles / n * n;
    if (total >= kSlotDoubles / 4 && piece > 0 && !ctx->stage) {
        void *s = nullptr;
        for (int k = 0; k < kSlots; k++)
            if (!ctx->ev_stage[k]) BPF_CUDA(ctx, cudaEventCreateWithFlags(&ctx->ev_stage[k], cudaEventDisableTiming));
        if (cudaMallocHost(&s, sizeof(double) * kSlots * kSlotDoubles) == cudaSuccess) ctx->stage = (double *)s;
        else cudaGetLastError();
    }
    if (total < kSlotDoubles / 4 || piece == 0 || !ctx->stage) {   // small, a huge column, or no pinned memory
        BPF_CUDA(ctx, cudaMemcpy2DAsync(host, sizeof(double) * n, X, sizeof(double) * ldx, sizeof(double) * n, p,
                                        cudaMemcpyDeviceToHost, ctx->stream));
        BPF_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
        if (negate)
            for (size_t i = 0; i < total; i++) host[i] = -host[i];
        return BPF_SUCCESS;
    }
    const size_t npieces = (total + piece - 1) / piece;
    auto issue = [&](size_t k) -> cudaError_t {
        double *slot = ctx->stage + (k % kSlots) * kSlotDoubles;
        const size_t at = k * piece, len = std::min(piece, total - at);
        cudaError_t e = linear ? cudaMemcpyAsync(slot, X + at, sizeof(double) * len, cudaMemcpyDeviceToHost, ctx->stream)
                               : cudaMemcpy2DAsync(slot, sizeof(double) * n, X + at / n * ldx, sizeof(double) * ldx,
                                                   sizeof(double) * n, len / n, cudaMemcpyDeviceToHost, ctx->stream);
        if (e == cudaSuccess) e = cudaEventRecord(ctx->ev_stage[k % kSlots], ctx->stream);
        return e;
    };
    CopyBoard b;
    auto part = [&](size_t k, int t, int nt) {   // thread t's share of piece k
        const size_t at = k * piece, len = std::min(piece, total - at);
        const size_t lo = len * t / nt, hi = len * (t + 1) / nt;
        copy_out(host + at + lo, ctx->stage + (k % kSlots) * kSlotDoubles + lo, hi - lo, negate != 0);
    };
    const int want = (int)std::max(1u, std::min((unsigned)kCopyThreads, std::thread::hardware_concurrency()));
    std::thread pool[kCopyThreads];
    int nt = 0;
    auto work = [&](int t) {
        for (size_t k = 0; k < npieces; k++) {
            int threads;
            {
                std::unique_lock<std::mutex> l(b.mu);
                b.cv.wait(l, [&]() { return b.stop || b.arrived > k; });
                if (b.stop) return;
                threads = b.threads;
            }
            part(k, t, threads);
            {
                std::lock_guard<std::mutex> l(b.mu);
                b.done++;
            }
            b.cv.notify_all();
        }
    };
    try {
        for (; nt < want; nt++) pool[nt] = std::thread(work, nt);
    } catch (const std::exception &) {
        // a thread limit, or no memory for one: those that started do it, or this one alone
    }
    {
        std::lock_guard<std::mutex> l(b.mu);
        b.threads = nt;
    }
    cudaError_t e = cudaSuccess;
    for (size_t k = 0; k < std::min<size_t>(kSlots, npieces) && e == cudaSuccess; k++) e = issue(k);
    for (size_t k = 0; k < npieces && e == cudaSuccess; k++) {
        e = cudaEventSynchronize(ctx->ev_stage[k % kSlots]);
        if (e != cudaSuccess) break;
        if (nt == 0) {
            part(k, 0, 1);
        } else {
            std::unique_lock<std::mutex> l(b.mu);
            b.done = 0;
            b.arrived = k + 1;
            b.cv.notify_all();
            b.cv.wait(l, [&]() { return b.done == nt; });
        }
        if (k + kSlots < npieces) e = issue(k + kSlots);
    }
    if (e != cudaSuccess) {
        std::lock_guard<std::mutex> l(b.mu);
        b.stop = true;
    }
    b.cv.notify_all();
    for (int t = 0; t < nt; t++) pool[t].join();
    if (e != cudaSuccess) return cuda_error(ctx, e, "block_to_host", __FILE__, __LINE__);
    return BPF_SUCCESS;
}
