// The pool of host size records (csrc/size_pool.h) without a GPU: fake memory,
// contexts by number.  Prints "ok".
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <thread>
#include <vector>

#include "size_pool.h"

#define CHECK(x) do { if (!(x)) { std::printf("%s:%d: %s\n", __FILE__, __LINE__, #x); std::exit(1); } } while (0)

using iso::SizePool;

int main() {
    std::atomic<int> slabs{0};
    const auto alloc = [&](size_t bytes) -> void* {
        ++slabs;
        CHECK(bytes == size_t(SizePool::SLAB) * SizePool::WORDS * 8);
        return std::malloc(bytes);
    };
    {  // threads that come and go, a call each: one slab
        SizePool pool;
        for (int i = 0; i < 300; ++i)
            std::thread([&] {
                long long* p = pool.lease(7, alloc);
                CHECK(p);
                p[0] = p[15] = 1;
                pool.release(7, p);
            }).join();
        CHECK(slabs == 1);
        // as many records at once as a slab holds, and one more; all cleared, none twice
        std::set<long long*> out;
        for (int i = 0; i <= SizePool::SLAB; ++i) {
            long long* p = pool.lease(7, alloc);
            CHECK(p && std::all_of(p, p + SizePool::WORDS, [](long long w) { return w == 0; }));
            for (long long* q : out) CHECK(p >= q + SizePool::WORDS || q >= p + SizePool::WORDS);
            CHECK(out.insert(p).second);
        }
        CHECK(slabs == 2);
        for (long long* p : out) pool.release(7, p);
        for (int i = 0; i < 2 * SizePool::SLAB; ++i) CHECK(pool.lease(7, alloc));
        CHECK(slabs == 2);
    }
    {  // another context: its own records; those of the first, which ended, stay untouched
        SizePool pool;
        slabs = 0;
        long long* a = pool.lease(1, alloc);
        a[3] = 42;
        pool.release(1, a);
        for (int i = 0; i < SizePool::SLAB; ++i) CHECK(pool.lease(2, alloc) != a);
        CHECK(slabs == 2 && a[3] == 42);
    }
    {  // no memory: nothing, and the next call works
        SizePool pool;
        slabs = 0;
        CHECK(!pool.lease(1, [](size_t) -> void* { return nullptr; }));
        long long* p = pool.lease(1, alloc);
        CHECK(p && slabs == 1);
    }
    {  // many threads at once: a record is one call's at a time
        SizePool pool;
        slabs = 0;
        std::vector<std::thread> ts;
        for (int t = 0; t < 8; ++t)
            ts.emplace_back([&, t] {
                for (int i = 0; i < 5000; ++i) {
                    long long* p = pool.lease(1, alloc);
                    CHECK(p && p[0] == 0);
                    p[0] = t + 1;
                    std::this_thread::yield();
                    CHECK(p[0] == t + 1);
                    pool.release(1, p);
                }
            });
        for (std::thread& t : ts) t.join();
        CHECK(slabs <= 8);  // a slab by each that found the pool empty at the start
    }
    {  // the end of a call: what is waited for, and what it returns
        long long words[4] = {5, 6, 7, 8}, out[4] = {};
        int waits = 0;
        bool good = true;
        const auto sync = [&] { ++waits; return good; };
        CHECK(iso::finish_sizes(0, 2, words, 3, out, sync) == 0 && waits == 1 && out[2] == 7 && out[3] == 0);
        out[0] = 0;
        CHECK(iso::finish_sizes(1, 2, words, 3, out, sync) == 1 && waits == 1);  // refused: nothing was launched
        CHECK(iso::finish_sizes(2, 2, words, 3, out, sync) == 2 && waits == 2);  // a launch failed: the rest waited for
        good = false;
        CHECK(iso::finish_sizes(0, 2, words, 3, out, sync) == 2 && waits == 3 && out[0] == 0);
    }
    std::printf("ok\n");
    return 0;
}
