// Host side of device memory: blocks kept between calls, and copies of pageable buffers
// staged through page-locked chunks by several threads.  Included by kssdgpu.cu inside its
// namespace.
#pragma once

// ------------------------------------------------------------------ device blocks
//
// An index build takes some twenty device arrays and gives half of them back before it
// returns.  cudaMalloc and cudaFree of each cost 0.3 to 0.7 ms (1.3 ms at 1 GB, and many
// times that on a host whose other processes allocate too), which was most of a small
// index's build: 64 genomes 6.2 ms, of which kernels 0.3.  Freed blocks are kept instead
// and handed out again for requests they fit (kssd_pool.h).  Kept: at most kPoolKeep bytes a
// device; blocks that two indexes in a row left unused are given back, all of them when an
// allocation fails and by kssdgpu_trim, and the rest of the library counts them as free memory.
// (cudaMallocAsync's pool was measured too: 6 ms per 500 MB that its reservation grows by.)
constexpr uint64_t kPoolKeep = 2ull << 30;

// Id of the calling thread's context, 0 where there is none.
uint64_t context_id()
{
    using GetId = int (*)(void *, unsigned long long *);
    static const GetId get = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<GetId>(f);
    }();
    unsigned long long id = 0;
    if (!get)
        return 0;
    if (get(nullptr, &id) != 0) {  // no context yet, or one that is gone
        if (cudaFree(nullptr) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        if (get(nullptr, &id) != 0)
            return 0;
    }
    return id;
}

struct CudaMemory {
    using Error = cudaError_t;
    static constexpr cudaError_t kOk = cudaSuccess, kNoMemory = cudaErrorMemoryAllocation;
    static uint64_t context() { return context_id(); }
    static cudaError_t alloc(void **p, size_t bytes)
    {
        const cudaError_t e = cudaMalloc(p, bytes);
        if (e == cudaErrorMemoryAllocation)
            cudaGetLastError();
        return e;
    }
    static void release(void *p) { cudaFree(p); }
};
using DevicePool = BlockPool<CudaMemory, kPoolKeep>;

// Never destroyed: at process exit the driver frees what it holds, in whatever order.
DevicePool &device_pool()
{
    static DevicePool *pool = new DevicePool();
    return *pool;
}

template <class T>
cudaError_t pool_malloc(T **p, size_t bytes)
{
    return device_pool().get(reinterpret_cast<void **>(p), bytes);
}
// As cudaFree: waits for the device first.
void pool_free(void *p)
{
    if (!p)
        return;
    cudaDeviceSynchronize();
    device_pool().put(p);
}
// After a synchronization that covers every use of the block.
void pool_free_idle(void *p) { device_pool().put(p); }

// Free device memory, the kept blocks (given up for any request) among it.
cudaError_t free_memory(uint64_t &bytes)
{
    size_t free_b = 0, total_b = 0;
    const cudaError_t e = cudaMemGetInfo(&free_b, &total_b);
    bytes = e == cudaSuccess ? free_b + device_pool().idle_bytes() : 0;
    return e;
}

// A block of exactly this size that is not kept (cudaFree it).
template <class T>
cudaError_t exact_malloc(T **p, size_t bytes)
{
    cudaError_t e = CudaMemory::alloc(reinterpret_cast<void **>(p), bytes);
    if (e == cudaErrorMemoryAllocation) {
        device_pool().trim();
        e = CudaMemory::alloc(reinterpret_cast<void **>(p), bytes);
    }
    return e;
}

// ------------------------------------------------------------------ staged copies
//
// A copy from or to pageable memory goes through the driver's own staging on one thread:
// 11 GB/s at 98 MB here, 5 GB/s into pages not touched before, against 55 GB/s from
// page-locked memory.  Copies of at least kStageMin bytes are cut into chunks that several
// threads move between the caller's buffer and page-locked chunks of their own, the DMA of
// one under the memcpy of the other.  The chunks (16 MB a context, page-locked on first use)
// are kept and are that context's alone, which frees them when it is reset; a second caller at
// the same time takes the driver's way.
constexpr size_t kStageMin = 2u << 20, kStageChunk = 1u << 20;
constexpr int kStageThreads = 8;

class Stager {
public:
    // Copies `bytes` between device memory and a host buffer on `st`; chunk(host, off, len)
    // moves one chunk to (IN) or from the page-locked chunk `host`.  false: not done here
    // (busy, no memory, no threads).  On return the host buffer is free / filled.
    template <bool IN, class Chunk>
    bool run(char *dev_ptr, size_t bytes, cudaStream_t st, const Chunk &chunk, cudaError_t &err)
    {
        std::unique_lock<std::mutex> lock(mu_, std::try_to_lock);
        if (!lock.owns_lock())
            return false;
        int dev = 0;
        if (cudaGetDevice(&dev) != cudaSuccess)
            return false;
        char *pinned = chunks(context_id());
        if (!pinned)
            return false;
        const size_t nchunks = (bytes + kStageChunk - 1) / kStageChunk;
        const int threads = (int)std::min<size_t>(
            {(size_t)kStageThreads, std::max<size_t>(1, std::thread::hardware_concurrency() / 2), (nchunks + 1) / 2});
        std::atomic<size_t> next{0};
        std::atomic<int> bad{(int)cudaSuccess};
        auto work = [&](int t) {
            cudaError_t e = cudaSetDevice(dev);
            cudaEvent_t ev[2] = {nullptr, nullptr};
            for (int i = 0; i < 2 && e == cudaSuccess; ++i)
                e = cudaEventCreateWithFlags(&ev[i], cudaEventDisableTiming);
            char *buf[2] = {pinned + (size_t)(2 * t) * kStageChunk, pinned + (size_t)(2 * t + 1) * kStageChunk};
            size_t off[2] = {0, 0}, len[2] = {0, 0};  // len: a DMA of the slot is under way
            for (int s = 0; e == cudaSuccess && bad.load() == (int)cudaSuccess; s ^= 1) {
                if (len[s]) {  // the slot's last DMA
                    e = cudaEventSynchronize(ev[s]);
                    if (e == cudaSuccess && !IN)
                        chunk(buf[s], off[s], len[s]);
                    len[s] = 0;
                }
                const size_t c = e == cudaSuccess ? next.fetch_add(1) : nchunks;
                if (c >= nchunks)
                    break;
                const size_t o = c * kStageChunk, n = std::min(kStageChunk, bytes - o);
                if (IN)
                    chunk(buf[s], o, n);
                e = IN ? cudaMemcpyAsync(dev_ptr + o, buf[s], n, cudaMemcpyHostToDevice, st)
                       : cudaMemcpyAsync(buf[s], dev_ptr + o, n, cudaMemcpyDeviceToHost, st);
                if (e == cudaSuccess)
                    e = cudaEventRecord(ev[s], st);
                off[s] = o;
                len[s] = n;
            }
            for (int s = 0; s < 2; ++s)
                if (len[s]) {
                    const cudaError_t e2 = cudaEventSynchronize(ev[s]);
                    if (e2 == cudaSuccess && e == cudaSuccess && !IN)
                        chunk(buf[s], off[s], len[s]);
                    if (e == cudaSuccess)
                        e = e2;
                }
            for (int i = 0; i < 2; ++i)
                if (ev[i])
                    cudaEventDestroy(ev[i]);
            if (e != cudaSuccess)
                bad.store((int)e);
        };
        std::vector<std::thread> team;
        try {
            team.reserve(threads);
            for (int t = 1; t < threads; ++t)
                team.emplace_back(work, t);
        } catch (const std::exception &) {
        }  // fewer threads: the others' chunks are this one's
        work(0);
        for (std::thread &t : team)
            t.join();
        err = (cudaError_t)bad.load();
        return true;
    }

    // Gives back the current context's chunks (none are in use while this holds the lock).
    void trim()
    {
        std::lock_guard<std::mutex> lock(mu_);
        const auto it = pinned_.find(context_id());
        if (it != pinned_.end()) {
            cudaFreeHost(it->second);
            pinned_.erase(it);
        }
    }

private:
    // The context's page-locked chunks, null where there are none.
    char *chunks(uint64_t context)
    {
        if (!context)
            return nullptr;
        try {
            void *&p = pinned_[context];
            if (!p && cudaHostAlloc(&p, kStageThreads * 2 * kStageChunk, cudaHostAllocDefault) != cudaSuccess) {
                cudaGetLastError();
                p = nullptr;
            }
            return static_cast<char *>(p);
        } catch (const std::bad_alloc &) {
            return nullptr;
        }
    }

    std::mutex mu_;
    std::map<uint64_t, void *> pinned_;
};

Stager &stager()
{
    static Stager *s = new Stager();
    return *s;
}

// Ordinary host memory (neither page-locked, managed nor of a device).
bool host_pageable(const void *p)
{
    cudaPointerAttributes a{};
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Host buffer -> device on `st` (as cudaMemcpyAsync of a pageable buffer: the buffer may be
// reused on return).
cudaError_t upload(void *dst, const void *src, size_t bytes, cudaStream_t st)
{
    cudaError_t e = cudaSuccess;
    if (bytes >= kStageMin && host_pageable(src) &&
        stager().run<true>((char *)dst, bytes, st,
                           [&](char *host, size_t off, size_t len) { memcpy(host, (const char *)src + off, len); }, e))
        return e;
    return bytes ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st) : cudaSuccess;
}

// Device -> host buffer behind the work on `st`; a staged copy is complete on return, any
// other when `st` has been synchronized.
cudaError_t download(void *dst, const void *src, size_t bytes, cudaStream_t st)
{
    cudaError_t e = cudaSuccess;
    if (bytes >= kStageMin && host_pageable(dst) &&
        stager().run<false>((char *)const_cast<void *>(src), bytes, st,
                            [&](char *host, size_t off, size_t len) { memcpy((char *)dst + off, host, len); }, e))
        return e;
    return bytes ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st) : cudaSuccess;
}
