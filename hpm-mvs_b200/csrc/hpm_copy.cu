/*
 * Staged copies of pageable host memory.
 *
 * A cudaMemcpyAsync of pageable memory goes through the driver's staging on
 * the calling thread: 11 GB/s in, and 5 GB/s out into pages that have not been
 * touched yet, with the GPU idle meanwhile (the driver lets one thread at a
 * time through it, so more threads in it change nothing).  Here a few threads
 * copy 1 MB chunks (smaller ones: 300 MB in 8.4 ms, with 512 KB 11.2, with
 * 256 KB 14.9) through their own pinned buffers (two each, so that a thread's
 * copy runs under its transfer); first touches of the destination are spread
 * over them as well.  11 images of 3200x2133 (300 MB) in: 27.0 -> 8.0 ms;
 * planes and costs of that size (137 MB) out: 23.5 -> 5.5 ms.  Small copies
 * take the plain way, where the threads cost more than they save (13 MB in:
 * 1.3 against 1.2 ms; 27 MB out into touched pages: 1.7 against 1.3 ms; 34 MB
 * in: 1.8 against 3.1; 38 MB out: 1.5 against 1.9), and so does pinned or
 * device memory, which needs no staging.
 *
 * The buffers are huge pages of the process, registered with the driver: 16 MB
 * in 1.2 ms, where cudaHostAlloc takes 10 to 25 and registering small pages 5.
 * That is still more than one copy of a few tens of MB saves (worth_it).
 */
#include <string.h>
#include <sys/mman.h>

#include <atomic>
#include <exception>
#include <new>
#include <thread>
#include <vector>

#include "hpm_capi_internal.h"
#include "hpm_copy.h"

namespace hpm {

namespace {
constexpr size_t kChunk = 1 << 20;
constexpr int kMaxThreads = 8, kSlots = 2;
constexpr size_t kMinIn = 16 << 20, kMinOut = 32 << 20;
constexpr size_t kWorth = 64 << 20;
constexpr size_t kHugePage = 2 << 20, kPinned = kMaxThreads * kSlots * kChunk;
}  // namespace

struct HostCopier {
    void *map = MAP_FAILED; /* kPinned and a huge page, for the alignment */
    char *pinned = nullptr; /* [kMaxThreads][kSlots][kChunk], once registered */
    cudaEvent_t done[kMaxThreads][kSlots] = {};
};

void host_copier_free(HostCopier *h)
{
    if (!h) return;
    for (auto &thread : h->done)
        for (cudaEvent_t &e : thread)
            if (e) {
                cudaEventSynchronize(e);
                cudaEventDestroy(e);
            }
    if (h->pinned) cudaHostUnregister(h->pinned);
    if (h->map != MAP_FAILED) munmap(h->map, kPinned + kHugePage);
    delete h;
}

namespace {

/* runs work(thread number) on up to `threads` threads, this one among them */
template <typename F>
void on_threads(int threads, F work)
{
    std::vector<std::thread> more;
    try {
        more.reserve(threads - 1);
        for (int t = 1; t < threads; ++t) more.emplace_back(work, t);
    } catch (const std::exception &) { /* fewer threads: the chunks are taken from one counter */
    }
    work(0);
    for (std::thread &t : more) t.join();
}

HostCopier *copier_of(hpm_ctx *c)
{
    if (c->copier) return c->copier;
    HostCopier *h = new (std::nothrow) HostCopier;
    if (!h) return nullptr;
    cudaError_t e = cudaErrorMemoryAllocation;
    h->map = mmap(nullptr, kPinned + kHugePage, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (h->map != MAP_FAILED) {
        char *p = (char *)h->map + (kHugePage - (size_t)h->map % kHugePage) % kHugePage;
        /* without huge pages it only takes longer; a child of this process
         * must not share pages that transfers write to */
        (void)madvise(p, kPinned, MADV_HUGEPAGE);
        (void)madvise(p, kPinned, MADV_DONTFORK);
        on_threads(kMaxThreads, [p](int t) { /* a huge page's zeroing per thread */
            for (size_t at = t * (kPinned / kMaxThreads); at < (t + 1) * (kPinned / kMaxThreads); at += kHugePage)
                *(volatile char *)(p + at) = 0;
        });
        e = cudaHostRegister(p, kPinned, cudaHostRegisterDefault);
        if (e == cudaSuccess) h->pinned = p;
    }
    for (int t = 0; t < kMaxThreads && e == cudaSuccess; ++t)
        for (int s = 0; s < kSlots && e == cudaSuccess; ++s)
            e = cudaEventCreateWithFlags(&h->done[t][s], cudaEventDisableTiming);
    if (e != cudaSuccess) { /* the plain copy needs neither */
        (void)cudaGetLastError();
        host_copier_free(h);
        return nullptr;
    }
    c->copier = h;
    return h;
}

/* Whether a copy of `bytes` pageable bytes, large enough for the threads, gets
 * pinned buffers to go through where the context has none yet: out of the
 * device it saves more than they cost; into it only a larger one does, or the
 * context's copies so far together. */
bool worth_it(hpm_ctx *c, size_t bytes, bool out)
{
    if (c->copier || out) return true;
    c->staged_so_far += bytes;
    return c->staged_so_far >= kWorth;
}

bool pageable(const void *p)
{
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        (void)cudaGetLastError();
        return false;
    }
    return at.type == cudaMemoryTypeUnregistered;
}

cudaError_t copy(hpm_ctx *c, const CopyItem *items, int n, bool out)
{
    std::vector<CopyItem> chunks;
    size_t staged = 0;
    const size_t least = out ? kMinOut : kMinIn;
    std::vector<char> stage;
    try {
        stage.resize(n);
        for (int i = 0; i < n; ++i) {
            stage[i] = pageable(out ? items[i].dst : items[i].src);
            if (stage[i]) staged += items[i].bytes;
        }
        if (staged >= least && (!worth_it(c, staged, out) || !copier_of(c))) staged = 0;
        if (staged >= least)
            for (int i = 0; i < n; ++i)
                for (size_t at = 0; stage[i] && at < items[i].bytes; at += kChunk)
                    chunks.push_back({(char *)items[i].dst + at, (const char *)items[i].src + at,
                                      items[i].bytes - at < kChunk ? items[i].bytes - at : kChunk});
    } catch (const std::bad_alloc &) {
        chunks.clear();
        staged = 0;
    }
    const bool threads_on = staged >= least;
    for (int i = 0; i < n; ++i) {
        if (threads_on && stage[i]) continue;
        const cudaError_t e = cudaMemcpyAsync(items[i].dst, items[i].src, items[i].bytes, cudaMemcpyDefault, c->stream);
        if (e != cudaSuccess) return e;
    }
    if (!threads_on) return cudaSuccess;
    HostCopier *h = c->copier;
    std::atomic<size_t> next{0};
    std::atomic<int> error{cudaSuccess};
    const int cores = (int)std::thread::hardware_concurrency();
    const int threads = cores < 4 ? 1 : (cores / 2 < kMaxThreads ? cores / 2 : kMaxThreads);
    on_threads(threads, [&](int t) {
        cudaError_t e = cudaSetDevice(c->device);
        CopyItem held[kSlots] = {};
        for (int s = 0; e == cudaSuccess; s = (s + 1) % kSlots) {
            char *buf = h->pinned + (size_t)(t * kSlots + s) * kChunk;
            /* the transfer that used this buffer last */
            e = cudaEventSynchronize(h->done[t][s]);
            if (e != cudaSuccess) break;
            if (held[s].bytes) memcpy(held[s].dst, buf, held[s].bytes);
            held[s].bytes = 0;
            const size_t i = error.load() == cudaSuccess ? next.fetch_add(1) : chunks.size();
            if (i >= chunks.size()) {
                bool more = false;
                for (const CopyItem &k : held) more = more || k.bytes != 0;
                if (!more) break;
                continue;
            }
            const CopyItem &k = chunks[i];
            if (out) {
                e = cudaMemcpyAsync(buf, k.src, k.bytes, cudaMemcpyDeviceToHost, c->stream);
                held[s] = k;
            } else {
                memcpy(buf, k.src, k.bytes);
                e = cudaMemcpyAsync(k.dst, buf, k.bytes, cudaMemcpyHostToDevice, c->stream);
            }
            if (e == cudaSuccess) e = cudaEventRecord(h->done[t][s], c->stream);
        }
        if (e != cudaSuccess) {
            int none = cudaSuccess;
            error.compare_exchange_strong(none, (int)e);
        }
    });
    return (cudaError_t)error.load();
}

}  // namespace

cudaError_t ctx_copy_in(hpm_ctx *c, const CopyItem *items, int n) { return copy(c, items, n, false); }

cudaError_t ctx_copy_out(hpm_ctx *c, const CopyItem *items, int n)
{
    const cudaError_t e = copy(c, items, n, true);
    const cudaError_t s = cudaStreamSynchronize(c->stream);
    return e != cudaSuccess ? e : s;
}

}  // namespace hpm
