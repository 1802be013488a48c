// A stand-in for the CUDA runtime and for the rest of the library, enough to run the bulk host transfers (bk_hostpipe.cpp) and
// the snapshots (bk_snapshot.cpp) on the CPU, with copies that can be made to fail.  "Device" memory is host memory.  Copies are
// queued and happen when something waits for them, so that one that is still in flight when a call returns can be seen.
#include <cstdlib>
#include <cstring>
#include <deque>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "bk_hostpipe.h"

namespace {
struct Op {
    void *dst;
    const void *src;
    size_t n;
    cudaEvent_t ev;
};
std::recursive_mutex mu;
std::deque<Op> queue;
long n_copies, n_syncs, n_advice, fail_copy = -1, fail_sync = -1, fail_new = -1;
std::thread::id new_thread;
std::vector<std::pair<const char *, size_t>> pinned;
struct Event {
    bool done = true;
};
bool step() {  // the stream's next operation
    if (queue.empty()) return false;
    const Op o = queue.front();
    queue.pop_front();
    if (o.ev) reinterpret_cast<Event *>(o.ev)->done = true;
    else memcpy(o.dst, o.src, o.n);
    return true;
}
}  // namespace

void *operator new(size_t n) {
    if (fail_new >= 0 && std::this_thread::get_id() == new_thread && fail_new-- == 0) throw std::bad_alloc();
    if (void *p = malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { free(p); }
void operator delete(void *p, size_t) noexcept { free(p); }

extern "C" {
int madvise(void *, size_t, int) { return n_advice++, 0; }
cudaError_t cudaMallocHost(void **p, size_t n) { return *p = malloc(n), memset(*p, 0xee, n), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = reinterpret_cast<cudaEvent_t>(new Event()), cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete reinterpret_cast<Event *>(e), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    a->type = cudaMemoryTypeUnregistered;
    for (auto &r : pinned)
        if ((const char *)p >= r.first && (const char *)p < r.first + r.second) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (n_copies++ == fail_copy) return cudaErrorInvalidValue;
    queue.push_back(Op{dst, src, n, nullptr});
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    reinterpret_cast<Event *>(e)->done = false;
    queue.push_back(Op{nullptr, nullptr, 0, e});
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (n_syncs++ == fail_sync) return cudaErrorLaunchFailure;
    while (!reinterpret_cast<Event *>(e)->done && step()) {}
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (reinterpret_cast<Event *>(e)->done) return cudaSuccess;
    step();
    return cudaErrorNotReady;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    while (step()) {}
    return cudaSuccess;
}
}

namespace bk {
bk_status fail(bk_ctx *ctx, bk_status st, const std::string &msg) { return ctx ? (ctx->err = msg, st) : st; }
bk_status cuda_fail(bk_ctx *ctx, cudaError_t, const char *what) { return fail(ctx, BK_ERR_CUDA, what); }
bk_status sync_and_check(bk_ctx *ctx) { return cudaStreamSynchronize(ctx->stream), BK_OK; }
bk_status bind_device(bk_ctx *) { return BK_OK; }
RopeTable::~RopeTable() {}
}  // namespace bk

extern "C" {
// ---- the rest of the library, as far as the snapshots use it
static void rows(bk_cache *c, int l, int s, int p0, int n, void *k, float *kn, void *v, float *vn, bool out) {
    const size_t r0 = (size_t)p0 * c->cfg.n_kv, nr = (size_t)n * c->cfg.n_kv;
    auto cp = [&](void *host, void *dev, size_t b) {
        if (host && dev) out ? memcpy(host, dev, b) : memcpy(dev, host, b);
    };
    cp(k, c->k_rows(l, s) + r0 * c->k_row_bytes, nr * c->k_row_bytes);
    cp(v, c->v_rows(l, s) + r0 * c->v_row_bytes, nr * c->v_row_bytes);
    if (c->d_kn) cp(kn, c->k_norms(l, s) + r0, nr * 4);
    if (c->d_vn) cp(vn, c->v_norms(l, s) + r0, nr * 4);
}
bk_status bk_cache_download(bk_cache *c, int32_t l, int32_t s, int32_t p0, int32_t n, void *k, float *kn, void *v, float *vn) {
    return rows(c, l, s, p0, n, k, kn, v, vn, true), BK_OK;
}
bk_status bk_cache_upload(bk_cache *c, int32_t l, int32_t s, int32_t p0, int32_t n, const void *k, const float *kn, const void *v, const float *vn) {
    return rows(c, l, s, p0, n, const_cast<void *>(k), const_cast<float *>(kn), const_cast<void *>(v), const_cast<float *>(vn), false), BK_OK;
}
bk_status bk_cache_set_n_pos(bk_cache *c, int32_t l, int32_t s, int32_t n) { return c->n_pos[c->slab(l, s)] = n, BK_OK; }

// ---- for the tests
__attribute__((visibility("default"))) bk_ctx *fake_ctx() { return new bk_ctx(); }
__attribute__((visibility("default"))) void fake_ctx_free(bk_ctx *ctx) {
    bk::host_pipe_destroy(ctx->pipe);
    delete ctx;
}
__attribute__((visibility("default"))) void fake_plan(long copy, long sync, long alloc) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    n_copies = n_syncs = 0;
    fail_copy = copy, fail_sync = sync, fail_new = alloc;
    new_thread = std::this_thread::get_id();
}
__attribute__((visibility("default"))) long fake_advice() { return n_advice; }
__attribute__((visibility("default"))) void fake_pin(const void *p, size_t n) { pinned.emplace_back((const char *)p, n); }
__attribute__((visibility("default"))) long fake_in_flight() {
    std::lock_guard<std::recursive_mutex> lk(mu);
    long n = 0;
    for (auto &o : queue) n += o.ev == nullptr;
    while (step()) {}
    return n;
}
__attribute__((visibility("default"))) int fake_transfer(bk_ctx *ctx, int to_host, size_t n, void **host, void **dev, const size_t *bytes) {
    std::vector<bk::HostSeg> segs(n);
    for (size_t i = 0; i < n; i++) segs[i] = bk::HostSeg{host[i], dev[i], bytes[i]};
    return to_host ? bk::host_pipe_d2h(ctx, segs.data(), n) : bk::host_pipe_h2d(ctx, segs.data(), n);
}
__attribute__((visibility("default"))) bk_cache *fake_cache(bk_ctx *ctx, int n_layers, int n_seqs, int n_ctx, int bits, const int *n_pos, unsigned seed) {
    bk_cache *c = new bk_cache();
    c->ctx = ctx;
    c->cfg.n_layers = n_layers, c->cfg.n_seqs = n_seqs, c->cfg.n_ctx = n_ctx, c->cfg.n_kv = 4, c->cfg.hd = 256;
    c->cfg.mode.kind = BK_MODE_PLANAR, c->cfg.mode.bits = bits, c->cfg.mode.v_quant = 1;
    c->k_kind = c->v_kind = bk::ROW_PLANAR;
    c->k_row_bytes = c->v_row_bytes = 32 * bits;
    const size_t r = (size_t)n_layers * n_seqs * n_ctx * 4;
    c->d_k = (uint8_t *)malloc(r * c->k_row_bytes), c->d_v = (uint8_t *)malloc(r * c->v_row_bytes);
    c->d_kn = (float *)malloc(r * 4), c->d_vn = (float *)malloc(r * 4);
    for (size_t i = 0; i < r * c->k_row_bytes; i++) c->d_k[i] = (seed = seed * 1664525u + 1013904223u) >> 24, c->d_v[i] = seed >> 16;
    for (size_t i = 0; i < r; i++) c->d_kn[i] = seed = seed * 1664525u + 1013904223u, c->d_vn[i] = seed >> 7;
    for (int l = 0; l < n_layers; l++)
        for (int s = 0; s < n_seqs; s++) c->n_pos.push_back(s == 0 ? n_pos[l] : 0);
    return c;
}
__attribute__((visibility("default"))) void fake_cache_free(bk_cache *c) {
    free(c->d_k), free(c->d_v), free(c->d_kn), free(c->d_vn);
    delete c;
}
__attribute__((visibility("default"))) int fake_n_pos(bk_cache *c, int l, int s) { return c->n_pos[c->slab(l, s)]; }
// how often launches on these devices set a kernel up, when set-up number `fail_at` fails
__attribute__((visibility("default"))) int fake_set_ups(const int *devices, int n, int fail_at, int *failed) {
    bk::PerDevice per_device;
    int runs = 0;
    for (int i = 0; i < n; i++)
        failed[i] = per_device.once(devices[i], [&] { return runs++ == fail_at ? cudaErrorInvalidValue : cudaSuccess; }) != cudaSuccess;
    return runs;
}
}
