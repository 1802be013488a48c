// Bulk transfers between caller memory (pageable) and the device: a ring of pinned slots, the copy engine on one
// side of it and a few host threads on the other.
//
// What bounds it: the bus (about 55 GB/s) as long as the host side keeps up.  One thread copies about 10 GB/s and takes the
// page faults of a fresh destination on top (0.25 us per 4 KB page), so a 34.6 MB snapshot as pageable copies moved
// 1.2 GB/s per direction; with the copies cut into 512 KB pieces and spread over the threads it takes 1.6 ms out and 1.2 ms
// back in (28 ms before), a quantize call of 8192 vectors 0.42 ms (1.0 ms before).
#ifdef __SSE2__
#include <emmintrin.h>
#endif
#include <string.h>

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <deque>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "bk_hostpipe.h"

namespace bk {

namespace {
constexpr int kSlots = 16;
constexpr size_t kSlotBytes = 512 << 10;
constexpr int kMaxThreads = 6;

#ifdef __SSE2__
inline void relax() { _mm_pause(); }

// Into a pinned slot the copy engine reads next: past the caches.  Lines that other cores hold dirty are fetched from
// them one by one, which held the engine to 4.5 GB/s on slots written with ordinary stores (52 GB/s from memory).
void copy_streaming(void *dst, const void *src, size_t n) {
    char *d = (char *)dst;
    const char *s = (const char *)src;
    while (n && ((uintptr_t)d & 15)) *d++ = *s++, n--;
    for (; n >= 64; n -= 64, d += 64, s += 64) {
        const __m128i a = _mm_loadu_si128((const __m128i *)s), b = _mm_loadu_si128((const __m128i *)s + 1);
        const __m128i c = _mm_loadu_si128((const __m128i *)s + 2), e = _mm_loadu_si128((const __m128i *)s + 3);
        _mm_stream_si128((__m128i *)d, a);
        _mm_stream_si128((__m128i *)d + 1, b);
        _mm_stream_si128((__m128i *)d + 2, c);
        _mm_stream_si128((__m128i *)d + 3, e);
    }
    while (n--) *d++ = *s++;
    _mm_sfence();
}
#else
inline void relax() { std::this_thread::yield(); }
void copy_streaming(void *dst, const void *src, size_t n) { memcpy(dst, src, n); }
#endif
}  // namespace

// Owned by one context and used by one thread at a time, like the context; the helpers end with it.
struct HostPipe {
    struct Task {
        void *dst;
        const void *src;
        size_t n;
        cudaEvent_t after;  // set: the source is complete once this event is
        bool to_slot;
        std::atomic<int> *done;
    };
    int device = 0;
    char *mem = nullptr;
    cudaEvent_t ev[kSlots] = {};
    std::atomic<int> done[kSlots];
    std::mutex m;
    std::condition_variable cv;
    std::deque<Task> q;
    std::atomic<int> waiting{0};  // tasks in q
    std::atomic<int> busy{0};     // tasks pushed and not finished
    std::atomic<int> err{0};      // first CUDA error a helper met
    bool stop = false;
    std::vector<std::thread> helpers;

    void run(const Task &t) {
        if (!t.src) {  // fault the page in; adding nothing is safe beside the copy that fills it
            __atomic_fetch_add((char *)t.dst, (char)0, __ATOMIC_RELAXED);
            busy.fetch_sub(1, std::memory_order_release);
            return;
        }
        const cudaError_t e = t.after ? cudaEventSynchronize(t.after) : cudaSuccess;
        if (e != cudaSuccess) err.store((int)e);  // (what the slot holds is an earlier transfer's)
        else if (t.to_slot) copy_streaming(t.dst, t.src, t.n);
        else memcpy(t.dst, t.src, t.n);
        t.done->store(1, std::memory_order_release);
        busy.fetch_sub(1, std::memory_order_release);
    }
    bool take(Task *t) {
        std::lock_guard<std::mutex> lk(m);
        if (q.empty()) return false;
        *t = q.front();
        q.pop_front();
        waiting.fetch_sub(1);
        return true;
    }
    void work() {
        cudaSetDevice(device);
        for (;;) {
            Task t;
            // the next task of a running transfer follows within microseconds: look for it before going to sleep
            for (int i = 0; i < 2000 && waiting.load(std::memory_order_relaxed) == 0; i++) relax();
            {
                std::unique_lock<std::mutex> lk(m);
                cv.wait(lk, [&] { return stop || !q.empty(); });
                if (q.empty()) return;
                t = q.front();
                q.pop_front();
                waiting.fetch_sub(1);
            }
            run(t);
        }
    }
    void push(const Task &t) {
        busy.fetch_add(1);
        try {
            std::lock_guard<std::mutex> lk(m);
            q.push_back(t);
            waiting.fetch_add(1);
        } catch (...) {  // no memory to queue it: now
            run(t);
            return;
        }
        cv.notify_one();
    }
    void finish(int slot) {  // wait for a slot's host copy, doing other copies meanwhile
        Task t;
        while (!done[slot].load(std::memory_order_acquire)) {
            if (take(&t)) run(t);
            else relax();
        }
    }
    // Page touches carry no flag of their own: none may outlive the call, whose caller owns the memory.
    void drain() {
        Task t;
        while (busy.load(std::memory_order_acquire) != 0) {
            if (take(&t)) run(t);
            else relax();
        }
    }
    char *slot(int i) { return mem + (size_t)i * kSlotBytes; }
};

void host_pipe_destroy(HostPipe *p) {
    if (!p) return;
    {
        std::lock_guard<std::mutex> lk(p->m);
        p->stop = true;
    }
    p->cv.notify_all();
    for (auto &t : p->helpers) t.join();
    for (auto &e : p->ev)
        if (e) cudaEventDestroy(e);
    if (p->mem) cudaFreeHost(p->mem);
    delete p;
}

bk_status out_of_memory(bk_ctx *ctx, const char *who) noexcept {
    try {
        return fail(ctx, BK_ERR_OOM, std::string(who) + ": host allocation failed");
    } catch (...) {
        return BK_ERR_OOM;
    }
}

static bk_status get_pipe(bk_ctx *ctx, HostPipe **out) {
    if (!ctx->pipe) {
        HostPipe *p;
        try {
            p = new HostPipe();  // (its queue allocates as well)
        } catch (const std::bad_alloc &) {
            return out_of_memory(ctx, "host pipe");
        }
        p->device = ctx->device;
        cudaError_t e = cudaMallocHost((void **)&p->mem, kSlots * kSlotBytes);
        for (int i = 0; i < kSlots && e == cudaSuccess; i++) e = cudaEventCreateWithFlags(&p->ev[i], cudaEventDisableTiming);
        if (e != cudaSuccess) {
            host_pipe_destroy(p);
            return cuda_fail(ctx, e, "host pipe");
        }
        const int n = (int)std::min<unsigned>(kMaxThreads, std::max(2u, std::thread::hardware_concurrency()) - 1);
        try {
            for (int i = 0; i < n; i++) p->helpers.emplace_back([p] { p->work(); });
        } catch (...) {
            // fewer helpers, or none: the calling thread does what is left
        }
        ctx->pipe = p;
    }
    *out = ctx->pipe;
    return BK_OK;
}

namespace {
// One slot's worth of host bytes and the device pieces that make it up.
struct Piece {
    char *host;
    size_t n;
    size_t first, count;  // in `parts`
};
struct Part {
    char *dev;
    size_t n;
};

// Cut the ranges into slots; ranges that follow one another in host memory share a slot.  False without memory for the lists.
bool cut(const HostSeg *segs, size_t n_seg, std::vector<Piece> &pieces, std::vector<Part> &parts) try {
    for (size_t i = 0; i < n_seg; i++) {
        size_t at = 0;
        while (at < segs[i].bytes) {
            char *h = (char *)segs[i].host + at;
            const bool join = !pieces.empty() && pieces.back().host + pieces.back().n == h && pieces.back().n < kSlotBytes;
            if (!join) pieces.push_back(Piece{h, 0, parts.size(), 0});
            Piece &p = pieces.back();
            const size_t n = std::min(segs[i].bytes - at, kSlotBytes - p.n);
            parts.push_back(Part{(char *)segs[i].dev + at, n});
            p.n += n;
            p.count++;
            at += n;
        }
    }
    return true;
} catch (const std::bad_alloc &) {
    return false;
}
}  // namespace

// Page-locked (or device-accessible) caller memory needs no slots.
static bool is_pinned(const void *host) {
    cudaPointerAttributes at{};
    const bool yes = cudaPointerGetAttributes(&at, host) == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();
    return yes;
}

// After an error: the copies that did go out still read or write the caller's memory and the slots.
static bk_status give_up(bk_ctx *ctx, cudaError_t e, const char *what) {
    cudaStreamSynchronize(ctx->stream);
    return cuda_fail(ctx, e, what);
}

// Without slots.
static bk_status copy_direct(bk_ctx *ctx, const HostSeg *segs, size_t n_seg, bool to_host) {
    for (size_t i = 0; i < n_seg; i++) {
        const cudaError_t e = to_host ? cudaMemcpyAsync(segs[i].host, segs[i].dev, segs[i].bytes, cudaMemcpyDeviceToHost, ctx->stream)
                                      : cudaMemcpyAsync(segs[i].dev, segs[i].host, segs[i].bytes, cudaMemcpyHostToDevice, ctx->stream);
        if (e != cudaSuccess) return give_up(ctx, e, to_host ? "copy to the host" : "copy to the device");
    }
    return sync_and_check(ctx);
}

bk_status host_pipe_d2h(bk_ctx *ctx, const HostSeg *segs, size_t n_seg) {
    if (n_seg > 0 && is_pinned(segs[0].host)) return copy_direct(ctx, segs, n_seg, true);
    HostPipe *p;
    bk_status st = get_pipe(ctx, &p);
    if (st != BK_OK) return st;
    std::vector<Piece> pieces;
    std::vector<Part> parts;
    if (!cut(segs, n_seg, pieces, parts)) return out_of_memory(ctx, "host pipe");
    // A fresh destination: fault its huge pages in on different threads first.  Copies of neighbouring pieces would fault on the
    // same page at once, and each clears 2 MB for it.
    for (size_t k = 0; k < pieces.size(); k++) {
        constexpr uintptr_t kHuge = 2 << 20;
        const uintptr_t page = ((uintptr_t)pieces[k].host + kHuge - 1) & ~(kHuge - 1);
        if (pieces.size() >= 8 && page < (uintptr_t)pieces[k].host + pieces[k].n) p->push(HostPipe::Task{(void *)page, nullptr, 0, nullptr, false, nullptr});
    }
    cudaError_t e = cudaSuccess;
    size_t i = 0;
    for (; i < pieces.size(); i++) {
        const int s = (int)(i % kSlots);
        if (i >= kSlots) p->finish(s);
        char *at = p->slot(s);
        for (size_t k = 0; k < pieces[i].count && e == cudaSuccess; k++) {
            const Part &pt = parts[pieces[i].first + k];
            e = cudaMemcpyAsync(at, pt.dev, pt.n, cudaMemcpyDeviceToHost, ctx->stream);
            at += pt.n;
        }
        if (e == cudaSuccess) e = cudaEventRecord(p->ev[s], ctx->stream);
        if (e != cudaSuccess) break;
        p->done[s].store(0);
        p->push(HostPipe::Task{pieces[i].host, p->slot(s), pieces[i].n, p->ev[s], false, &p->done[s]});
    }
    for (size_t k = i > kSlots ? i - kSlots : 0; k < i; k++) p->finish((int)(k % kSlots));
    p->drain();
    const cudaError_t helper = (cudaError_t)p->err.exchange(0);
    if (e == cudaSuccess) e = helper;
    return e != cudaSuccess ? give_up(ctx, e, "copy to the host") : sync_and_check(ctx);
}

bk_status host_pipe_h2d(bk_ctx *ctx, const HostSeg *segs, size_t n_seg) {
    if (n_seg > 0 && is_pinned(segs[0].host)) return copy_direct(ctx, segs, n_seg, false);
    HostPipe *p;
    bk_status st = get_pipe(ctx, &p);
    if (st != BK_OK) return st;
    std::vector<Piece> pieces;
    std::vector<Part> parts;
    if (!cut(segs, n_seg, pieces, parts)) return out_of_memory(ctx, "host pipe");
    cudaError_t e = cudaSuccess;
    size_t pushed = 0, issued = 0;
    while (issued < pieces.size() && e == cudaSuccess) {
        for (; pushed < pieces.size() && pushed - issued < kSlots && e == cudaSuccess; pushed++) {
            const int s = (int)(pushed % kSlots);
            if (pushed >= kSlots) {  // the slot's last copy to the device
                if (pushed > issued && cudaEventQuery(p->ev[s]) == cudaErrorNotReady) {
                    cudaGetLastError();
                    break;
                }
                e = cudaEventSynchronize(p->ev[s]);
            }
            p->done[s].store(0);
            p->push(HostPipe::Task{p->slot(s), pieces[pushed].host, pieces[pushed].n, nullptr, true, &p->done[s]});
        }
        const int s = (int)(issued % kSlots);
        p->finish(s);
        const char *at = p->slot(s);
        for (size_t k = 0; k < pieces[issued].count && e == cudaSuccess; k++) {
            const Part &pt = parts[pieces[issued].first + k];
            e = cudaMemcpyAsync(pt.dev, at, pt.n, cudaMemcpyHostToDevice, ctx->stream);
            at += pt.n;
        }
        if (e == cudaSuccess) e = cudaEventRecord(p->ev[s], ctx->stream);
        issued++;
    }
    for (; issued < pushed; issued++) p->finish((int)(issued % kSlots));  // (after an error)
    // the slots are the next transfer's: they must be read by then
    if (e == cudaSuccess && !pieces.empty()) e = cudaEventSynchronize(p->ev[(pieces.size() - 1) % kSlots]);
    return e != cudaSuccess ? give_up(ctx, e, "copy to the device") : BK_OK;
}

}  // namespace bk
