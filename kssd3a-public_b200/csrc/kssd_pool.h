// Bookkeeping of device blocks that are kept between calls (plain C++; the memory itself is
// the Memory parameter's, CUDA's in kssd_hostmem.cuh).
//
// A block belongs to the context it was made in and is handed out in that context alone: a
// cudaDeviceReset frees every block with its context, and the next context's memory may lie at
// the same addresses.  Contexts are known by an id that no later one has again.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <new>
#include <unordered_map>
#include <utility>

// Memory: Error, kOk, kNoMemory; context() (0: unknown, nothing is kept), alloc(p, bytes),
// release(p).  At most `keep` bytes of idle blocks a context.
template <class Memory, uint64_t keep>
class BlockPool {
public:
    using Error = typename Memory::Error;

    Error get(void **p, size_t bytes)
    {
        *p = nullptr;
        const uint64_t id = Memory::context();
        if (!id)
            return Memory::alloc(p, std::max<size_t>(bytes, 1));
        // sizes in steps of an eighth of their power of two (at least 512 bytes), so that
        // requests a little apart use one another's blocks
        size_t step = 512;
        while (step * 16 < bytes)
            step <<= 1;
        const size_t size = (std::max<size_t>(bytes, 1) + step - 1) / step * step;
        try {
            std::lock_guard<std::mutex> lock(mu_);
            const auto it = idle_.lower_bound({id, size});
            if (it != idle_.end() && it->first.first == id && it->first.second <= size + size / 4) {
                live_[it->second.p] = Live{it->first.second, id};
                *p = it->second.p;
                context_[id].idle -= it->first.second;
                idle_.erase(it);
                return Memory::kOk;
            }
        } catch (const std::bad_alloc &) {
            return Memory::kNoMemory;
        }
        Error e = Memory::alloc(p, size);
        if (e == Memory::kNoMemory) {  // the kept blocks may be what is missing
            release(id, ~0ull);
            e = Memory::alloc(p, size);
            if (e == Memory::kNoMemory && size != bytes)
                e = Memory::alloc(p, std::max<size_t>(bytes, 1));
        }
        if (e == Memory::kOk) {
            try {
                std::lock_guard<std::mutex> lock(mu_);
                live_[*p] = Live{size, id};  // in place of a block that a lost context had there
            } catch (const std::bad_alloc &) {
            }  // unknown to put(): freed there
        }
        return e;
    }

    // p: a block whose device work has ended (the caller synchronized).
    void put(void *p)
    {
        if (!p)
            return;
        uint64_t id = 0;
        try {
            std::lock_guard<std::mutex> lock(mu_);
            const auto it = live_.find(p);
            if (it != live_.end()) {
                const Live b = it->second;
                id = b.id;
                live_.erase(it);
                Context &c = context_[b.id];
                if (c.idle + b.bytes <= keep) {
                    idle_.emplace(std::make_pair(b.id, b.bytes), Idle{p, c.epoch});
                    c.idle += b.bytes;
                    return;
                }
            }
        } catch (const std::bad_alloc &) {
        }
        if (!id || id == Memory::context())  // else it went with its context
            Memory::release(p);
    }

    // One index less: blocks of the current context that kAges of them in a row did not use go
    // back (kept for longer, they take the place of blocks that are of use: 2 GiB hold the arrays
    // of one or two indexes).
    void age()
    {
        const uint64_t id = Memory::context();
        uint64_t now;
        try {
            std::lock_guard<std::mutex> lock(mu_);
            now = ++context_[id].epoch;
        } catch (const std::bad_alloc &) {
            return;
        }
        if (now > kAges)
            release(id, now - kAges);
    }

    // Gives back all idle blocks of the current context.
    void trim() { release(Memory::context(), ~0ull); }

    // Their bytes.
    uint64_t idle_bytes()
    {
        const uint64_t id = Memory::context();
        std::lock_guard<std::mutex> lock(mu_);
        const auto it = context_.find(id);
        return it == context_.end() ? 0 : it->second.idle;
    }

    static constexpr uint64_t kAges = 2;

private:
    struct Live {
        size_t bytes;
        uint64_t id;
    };
    struct Idle {
        void *p;
        uint64_t epoch;
    };
    struct Context {
        uint64_t idle = 0, epoch = 0;
    };

    // Gives back the current context's blocks kept since before epoch `until`.
    void release(uint64_t id, uint64_t until)
    {
        std::lock_guard<std::mutex> lock(mu_);
        for (auto it = idle_.lower_bound({id, 0}); it != idle_.end() && it->first.first == id;) {
            if (it->second.epoch < until) {
                context_[id].idle -= it->first.second;
                Memory::release(it->second.p);
                it = idle_.erase(it);
            } else {
                ++it;
            }
        }
    }

    std::mutex mu_;
    std::unordered_map<void *, Live> live_;
    std::multimap<std::pair<uint64_t, size_t>, Idle> idle_;
    std::map<uint64_t, Context> context_;
};
