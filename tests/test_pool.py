"""The kept device blocks' bookkeeping over a fake of the device's memory (no GPU): blocks are
handed out in the context that they were made in and in no other, whatever addresses a later
context's memory has; idle blocks stay within their bound, age, and go when memory is short."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "kssd_pool.h"
#include <cstdio>
#include <cstdlib>
#include <set>

struct Fake {
    using Error = int;
    static constexpr int kOk = 0, kNoMemory = 2;
    static inline uint64_t id = 1;
    static inline size_t room = 1 << 20, used = 0;
    static inline char *next = (char *)4096;
    static inline std::map<void *, size_t> held;  // of the context `id`
    static inline int allocs = 0, frees = 0;
    static uint64_t context() { return id; }
    static int alloc(void **p, size_t n)
    {
        if (used + n > room)
            return kNoMemory;
        *p = next;
        next += n;
        used += n;
        held[*p] = n;
        ++allocs;
        return kOk;
    }
    static void release(void *p)
    {
        if (!held.count(p)) {
            std::printf("freed what is not held\n");
            std::exit(1);
        }
        used -= held[p];
        held.erase(p);
        ++frees;
    }
    static void reset()  // the context's memory goes; the next one's lies at the same addresses
    {
        ++id;
        used = 0;
        next = (char *)4096;
        held.clear();
    }
};

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

int main()
{
    BlockPool<Fake, 65536> pool;
    void *a, *b, *c, *d;
    CHECK(pool.get(&a, 1000) == 0 && pool.get(&b, 5000) == 0);
    pool.put(a);
    CHECK(pool.get(&c, 900) == 0 && c == a && Fake::allocs == 2);  // handed out again
    pool.put(c);
    pool.put(b);
    // a reset: nothing of before is handed out or given back
    Fake::reset();
    CHECK(pool.get(&c, 1000) == 0 && Fake::allocs == 3 && Fake::held.count(c));
    CHECK(c == a);  // at an old block's address
    CHECK(pool.get(&d, 5000) == 0 && Fake::allocs == 4 && Fake::held.count(d));
    CHECK(Fake::frees == 0);
    pool.put(c);
    CHECK(pool.get(&c, 1000) == 0 && c == a && Fake::allocs == 4);  // this context's
    // a block that was out during a reset, given back behind it: not freed, not handed out
    CHECK(pool.get(&b, 60000) == 0);
    Fake::reset();
    const int allocs = Fake::allocs;
    pool.put(b);
    CHECK(Fake::frees == 0);
    CHECK(pool.get(&b, 60000) == 0 && Fake::allocs == allocs + 1 && Fake::held.count(b));
    // the bound on what is kept: the second block is freed
    CHECK(pool.get(&c, 30000) == 0);
    pool.put(b);
    pool.put(c);
    CHECK(Fake::frees == 1);
    // unused for more than kAges ages: given back; of other contexts nothing
    CHECK(pool.idle_bytes() >= 60000);
    for (uint64_t i = 0; i <= pool.kAges; ++i) {
        CHECK(Fake::frees == 1);
        pool.age();
    }
    CHECK(Fake::frees == 2 && Fake::held.empty() && pool.idle_bytes() == 0);
    // at once
    CHECK(pool.get(&c, 30000) == 0);
    pool.put(c);
    pool.trim();
    CHECK(Fake::frees == 3 && Fake::held.empty() && pool.idle_bytes() == 0);
    // memory short: the idle blocks go first
    CHECK(pool.get(&a, 40000) == 0);
    pool.put(a);
    Fake::room = 50000;
    CHECK(pool.get(&b, 45000) == 0 && Fake::frees == 4);
    CHECK(pool.get(&c, 20000) == Fake::kNoMemory);
    // no context: plain allocations
    pool.put(b);
    Fake::id = 0;
    Fake::room = 1 << 20;
    CHECK(pool.get(&c, 45000) == 0 && c != b);
    pool.put(c);
    CHECK(!Fake::held.count(c));
    std::printf("ok\n");
    return 0;
}
"""


def test_blocks_stay_in_their_context(tmp_path):
    src = tmp_path / "pool.cpp"
    src.write_text(PROGRAM)
    exe = str(tmp_path / "pool")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Wextra", "-I",
                    os.path.join(ROOT, "kssd3a-public_b200", "csrc"), str(src), "-o", exe], check=True)
    run = subprocess.run([exe], capture_output=True, text=True)
    assert run.returncode == 0 and run.stdout == "ok\n", run.stdout
