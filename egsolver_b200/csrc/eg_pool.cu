/*
 * eg_pool.cu -- device memory pool, idle streams and staged copies
 * (eg_pool.cuh).
 *
 * The singletons here are never destroyed: the CUDA context goes first at
 * process exit, and worker threads wait on their condition variable.
 */
#include "eg_pool.cuh"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <deque>
#include <functional>
#include <mutex>
#include <thread>
#include <vector>

#include <sys/mman.h>

#ifndef MADV_POPULATE_WRITE
#define MADV_POPULATE_WRITE 23
#endif

namespace eg {

namespace {

constexpr int kMaxDevices = 64;
constexpr unsigned long long kPoolKeep = 64ull << 20; /* idle device memory per device */
constexpr size_t kIdleLanes = 16, kIdleStages = 16;   /* per device; per process  */
constexpr size_t kHalf = kStageBlock;                   /* a staging buffer has two halves */
constexpr size_t kMapFrom = 128 << 10;                /* smaller arrays come from memory in use */
/* Threads of a large copy.  Transposes of 6.3 M entries (57 MB each way): 12.2
 * ms with one, 7.0-7.9 with 4, 6.5 with 8, 6.9-7.3 with 16.  It is too many for
 * smaller ones: of 300,000 entries 0.57 ms with one, 1.1 with 8, of 1 M 1.6
 * and 2.8. */
constexpr int kCopyThreads = 8;

std::mutex g_mu;
cudaMemPool_t g_pool[kMaxDevices];
std::vector<Lane *> *g_lanes[kMaxDevices];

cudaError_t pool_of(int device, cudaMemPool_t *out)
{
    if (device < 0 || device >= kMaxDevices) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_pool[device]) {
        cudaMemPoolProps pr;
        memset(&pr, 0, sizeof pr);
        pr.allocType = cudaMemAllocationTypePinned;
        pr.location.type = cudaMemLocationTypeDevice;
        pr.location.id = device;
        cudaError_t e = cudaMemPoolCreate(&g_pool[device], &pr);
        if (e != cudaSuccess) {
            g_pool[device] = nullptr;
            return e;
        }
        unsigned long long keep = kPoolKeep;
        cudaMemPoolSetAttribute(g_pool[device], cudaMemPoolAttrReleaseThreshold, &keep);
    }
    *out = g_pool[device];
    return cudaSuccess;
}

/* A pinned buffer of two halves, each with an event of its last copy. */
struct Stage {
    int device;
    char *p;
    cudaEvent_t ev[2];
    bool busy[2]; /* a copy from or to the half may still run */
};

std::vector<Stage *> *g_stages;

void stage_drop(Stage *s)
{
    if (s->p) cudaFreeHost(s->p);
    for (cudaEvent_t e : s->ev)
        if (e) cudaEventDestroy(e);
    delete s;
}

Stage *stage_take(int device)
{
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_stages)
            for (size_t i = g_stages->size(); i-- > 0;)
                if ((*g_stages)[i]->device == device) {
                    Stage *s = (*g_stages)[i];
                    g_stages->erase(g_stages->begin() + (long)i);
                    return s;
                }
    }
    Stage *s = new Stage();
    s->device = device;
    bool ok = cudaHostAlloc((void **)&s->p, 2 * kHalf, cudaHostAllocDefault) == cudaSuccess;
    for (int k = 0; k < 2 && ok; k++) ok = cudaEventCreateWithFlags(&s->ev[k], cudaEventDisableTiming) == cudaSuccess;
    if (ok) return s;
    cudaGetLastError();
    stage_drop(s);
    return nullptr;
}

/* A half may still be on its way to the device: whoever takes the buffer next
 * waits for its event before writing it. */
void stage_give(Stage *s)
{
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_stages) g_stages = new std::vector<Stage *>();
        if (g_stages->size() < kIdleStages) {
            g_stages->push_back(s);
            return;
        }
    }
    for (int k = 0; k < 2; k++)
        if (s->busy[k]) cudaEventSynchronize(s->ev[k]);
    stage_drop(s);
}

/* Threads that take jobs from a queue; the caller works too. */
struct Crew {
    std::mutex mu;
    std::condition_variable cv;
    std::deque<std::function<void()>> jobs;
    int threads = 0;
    Crew()
    {
        const int hw = (int)std::thread::hardware_concurrency();
        threads = std::max(0, std::min(kCopyThreads, hw) - 1);
        for (int t = 0; t < threads; t++)
            std::thread([this]() {
                for (;;) {
                    std::function<void()> f;
                    {
                        std::unique_lock<std::mutex> lk(mu);
                        cv.wait(lk, [this]() { return !jobs.empty(); });
                        f = std::move(jobs.front());
                        jobs.pop_front();
                    }
                    f();
                }
            }).detach();
    }
    /* Runs fn(0) .. fn(count - 1), fn(0) on the caller, and waits for all. */
    void run(int count, const std::function<void(int)> &fn)
    {
        struct Wait {
            std::mutex mu;
            std::condition_variable cv;
            int left;
        } w;
        w.left = count - 1;
        {
            std::lock_guard<std::mutex> lk(mu);
            for (int i = 1; i < count; i++)
                jobs.push_back([&w, &fn, i]() {
                    fn(i);
                    std::lock_guard<std::mutex> l(w.mu);
                    if (--w.left == 0) w.cv.notify_one();
                });
        }
        cv.notify_all();
        fn(0);
        std::unique_lock<std::mutex> lk(w.mu);
        w.cv.wait(lk, [&]() { return w.left == 0; });
    }
};

Crew &crew()
{
    static Crew *c = new Crew();
    return *c;
}

bool pageable(const void *p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

/* Maps the whole pages of a destination that is about to be written, in one
 * call: 0.5 us per page taken one fault at a time, and it runs while the copy
 * is on its way.  Where the system does not know it, memcpy faults as before. */
void map_pages(char *p, size_t bytes)
{
    const uintptr_t b = ((uintptr_t)p + 4095) & ~(uintptr_t)4095, e = ((uintptr_t)p + bytes) & ~(uintptr_t)4095;
    if (e > b) madvise((void *)b, e - b, MADV_POPULATE_WRITE);
}

/* One piece of a copy, at most half a staging buffer. */
struct Chunk {
    char *host, *dev;
    size_t bytes;
    bool map;
};

/* Copies chunks first, first + step, ... through one buffer: while one half is
 * in flight the other is filled or emptied. */
cudaError_t run_chunks(const std::vector<Chunk> &chunks, bool to_host, size_t first, size_t step, int device, cudaStream_t st)
{
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return e;
    Stage *s = stage_take(device);
    if (!s) return cudaErrorMemoryAllocation;
    const Chunk *held[2] = {nullptr, nullptr}; /* on its way to the host in each half */
    auto drain = [&](int k) {
        if (!s->busy[k]) return cudaSuccess;
        const cudaError_t x = cudaEventSynchronize(s->ev[k]);
        s->busy[k] = false;
        if (x == cudaSuccess && held[k]) memcpy(held[k]->host, s->p + (size_t)k * kHalf, held[k]->bytes);
        held[k] = nullptr;
        return x;
    };
    int k = 0;
    for (size_t i = first; i < chunks.size(); i += step, k ^= 1) {
        const Chunk &c = chunks[i];
        char *half = s->p + (size_t)k * kHalf;
        e = drain(k);
        if (e != cudaSuccess) break;
        if (to_host) {
            e = cudaMemcpyAsync(half, c.dev, c.bytes, cudaMemcpyDeviceToHost, st);
            held[k] = &c;
            if (c.map) map_pages(c.host, c.bytes);
        } else {
            memcpy(half, c.host, c.bytes);
            e = cudaMemcpyAsync(c.dev, half, c.bytes, cudaMemcpyHostToDevice, st);
        }
        if (e == cudaSuccess) e = cudaEventRecord(s->ev[k], st);
        s->busy[k] = e == cudaSuccess;
        if (e != cudaSuccess) break;
    }
    for (int j = 0; j < 2 && to_host; j++, k ^= 1) {
        const cudaError_t x = drain(k);
        if (e == cudaSuccess) e = x;
    }
    if (e != cudaSuccess) { /* no copy may still use the buffer */
        cudaStreamSynchronize(st);
        s->busy[0] = s->busy[1] = false;
    }
    stage_give(s);
    return e;
}

}  // namespace

cudaError_t copy_list(const CopyItem *items, int count, bool to_host, int device, cudaStream_t st)
{
    std::vector<Chunk> chunks;
    bool direct = false;
    cudaError_t e = cudaSuccess;
    for (int i = 0; i < count && e == cudaSuccess; i++) {
        const CopyItem &it = items[i];
        if (!it.bytes) continue;
        if (!pageable(it.host)) {
            e = to_host ? cudaMemcpyAsync(it.host, it.dev, it.bytes, cudaMemcpyDeviceToHost, st)
                        : cudaMemcpyAsync(it.dev, it.host, it.bytes, cudaMemcpyHostToDevice, st);
            direct = true;
            continue;
        }
        for (size_t at = 0; at < it.bytes; at += kHalf)
            chunks.push_back({(char *)it.host + at, (char *)it.dev + at, std::min(kHalf, it.bytes - at), it.bytes >= kMapFrom});
    }
    if (e == cudaSuccess && chunks.size() == 1) {
        e = run_chunks(chunks, to_host, 0, 1, device, st);
    } else if (e == cudaSuccess && !chunks.empty()) {
        Crew &c = crew();
        const int n = (int)std::min<size_t>(chunks.size(), (size_t)c.threads + 1);
        std::atomic<int> err(cudaSuccess);
        c.run(n, [&](int i) {
            const cudaError_t x = run_chunks(chunks, to_host, (size_t)i, (size_t)n, device, st);
            if (x != cudaSuccess) err = (int)x;
        });
        e = (cudaError_t)err.load();
    }
    if (direct || e != cudaSuccess) {
        const cudaError_t x = cudaStreamSynchronize(st);
        if (e == cudaSuccess) e = x;
    }
    return e;
}

cudaError_t pool_alloc(void **p, size_t bytes, int device, cudaStream_t st)
{
    cudaMemPool_t pool;
    *p = nullptr;
    cudaError_t e = pool_of(device, &pool);
    if (e == cudaSuccess) e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        cudaDeviceSynchronize();
        cudaMemPoolTrimTo(pool, 0);
        e = cudaMallocFromPoolAsync(p, bytes, pool, st);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        *p = nullptr;
    }
    return e;
}

void pool_free(void *p, cudaStream_t st)
{
    if (p) cudaFreeAsync(p, st);
}

size_t pool_idle(int device)
{
    cudaMemPool_t pool;
    unsigned long long held = 0, used = 0;
    if (pool_of(device, &pool) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &held) != cudaSuccess ||
        cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &used) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return held > used ? (size_t)(held - used) : 0;
}

Lane *lane_take(int device)
{
    if (device < 0 || device >= kMaxDevices) return nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (g_lanes[device] && !g_lanes[device]->empty()) {
            Lane *l = g_lanes[device]->back();
            g_lanes[device]->pop_back();
            return l;
        }
    }
    Lane *l = new Lane();
    memset(l, 0, sizeof *l);
    l->device = device;
    bool ok = cudaStreamCreateWithFlags(&l->st, cudaStreamNonBlocking) == cudaSuccess;
    for (int i = 0; i < 6 && ok; i++) ok = cudaEventCreate(&l->ev[i]) == cudaSuccess;
    if (ok) ok = cudaHostAlloc(&l->page, kLanePage, cudaHostAllocDefault) == cudaSuccess;
    if (ok) return l;
    cudaGetLastError();
    for (cudaEvent_t ev : l->ev)
        if (ev) cudaEventDestroy(ev);
    if (l->st) cudaStreamDestroy(l->st);
    delete l;
    return nullptr;
}

void lane_give(Lane *l)
{
    if (!l) return;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (!g_lanes[l->device]) g_lanes[l->device] = new std::vector<Lane *>();
        if (g_lanes[l->device]->size() < kIdleLanes) {
            g_lanes[l->device]->push_back(l);
            return;
        }
    }
    cudaStreamSynchronize(l->st);
    for (cudaEvent_t ev : l->ev) cudaEventDestroy(ev);
    cudaStreamDestroy(l->st);
    cudaFreeHost(l->page);
    delete l;
}

cudaError_t copy_to_host(void *dst, const void *dev, size_t bytes, int device, cudaStream_t st)
{
    const CopyItem it = {dst, (void *)dev, bytes};
    return copy_list(&it, 1, true, device, st);
}

cudaError_t copy_parts_to_device(void *dev, const CopyPart *parts, int count, size_t total, int device, cudaStream_t st)
{
    if (total > kHalf) {
        std::vector<CopyItem> items;
        for (int i = 0; i < count; i++) items.push_back({(void *)parts[i].src, (char *)dev + parts[i].at, parts[i].bytes});
        return copy_list(items.data(), count, false, device, st);
    }
    Stage *s = stage_take(device);
    if (!s) return cudaErrorMemoryAllocation;
    cudaError_t e = s->busy[0] ? cudaEventSynchronize(s->ev[0]) : cudaSuccess;
    s->busy[0] = false;
    for (int i = 0; i < count && e == cudaSuccess; i++) memcpy(s->p + parts[i].at, parts[i].src, parts[i].bytes);
    if (e == cudaSuccess) e = cudaMemcpyAsync(dev, s->p, total, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaEventRecord(s->ev[0], st);
    if (e == cudaSuccess) s->busy[0] = true;
    else cudaStreamSynchronize(st);
    stage_give(s);
    return e;
}

cudaError_t copy_block_to_host(const void *dev, size_t bytes, int device, cudaStream_t st,
                               const std::function<void(const char *)> &look)
{
    Stage *s = stage_take(device);
    if (!s) return cudaErrorMemoryAllocation;
    cudaError_t e = s->busy[0] ? cudaEventSynchronize(s->ev[0]) : cudaSuccess;
    s->busy[0] = false;
    if (e == cudaSuccess) e = cudaMemcpyAsync(s->p, dev, bytes, cudaMemcpyDeviceToHost, st);
    const cudaError_t x = cudaStreamSynchronize(st); /* also on an error: no copy may still use the buffer */
    if (e == cudaSuccess) e = x;
    if (e == cudaSuccess) look(s->p);
    stage_give(s);
    return e;
}

cudaError_t copy_to_device(void *dev, const void *src, size_t bytes, int device, cudaStream_t st)
{
    const CopyItem it = {(void *)src, dev, bytes};
    return copy_list(&it, 1, false, device, st);
}

}  // namespace eg
