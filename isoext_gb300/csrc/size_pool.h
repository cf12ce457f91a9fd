// Host records that a call's last kernel writes its sizes to (iso_*_sync),
// leased for one call at a time from a pool that all host threads share.
// Records come in slabs of pinned memory, so a new thread's first call costs a
// lock, not an allocation, and no thread's end frees (and so waits for) anything.
// The pool holds as many slabs as the most calls that ever ran at once need.  Memory
// belongs to the CUDA context it was allocated in and ends with it: records are
// kept by context id, and those of a context that has ended are not touched
// again.  Host code only (no CUDA header), so that it is tested without a GPU.
#pragma once

#include <cstddef>
#include <cstring>
#include <mutex>
#include <vector>

namespace iso {

class SizePool {
public:
    static constexpr int WORDS = 16;  // per record, 128 bytes: a line of its own
    static constexpr int SLAB = 64;   // records per allocation

    // A cleared record of context ctx; alloc(bytes) gives pinned memory of that
    // context (the current one), or nullptr: then so does lease.
    template <typename Alloc>
    long long* lease(unsigned long long ctx, Alloc alloc) noexcept {
        long long* p = take(ctx);
        if (!p) {
            long long* slab = static_cast<long long*>(alloc(size_t(SLAB) * WORDS * sizeof(long long)));
            if (!slab || !add(ctx, slab)) return nullptr;
            p = slab;
        }
        std::memset(p, 0, WORDS * sizeof(long long));
        return p;
    }

    void release(unsigned long long ctx, long long* p) noexcept {
        std::lock_guard<std::mutex> lk(mu_);
        for (Context& c : contexts_)
            if (c.id == ctx) c.free.push_back(p);  // within the capacity that add() reserved
    }

private:
    struct Context {
        unsigned long long id;
        size_t records;
        std::vector<long long*> free;
    };

    long long* take(unsigned long long ctx) noexcept {
        std::lock_guard<std::mutex> lk(mu_);
        for (Context& c : contexts_)
            if (c.id == ctx && !c.free.empty()) {
                long long* p = c.free.back();
                c.free.pop_back();
                return p;
            }
        return nullptr;
    }

    // A new slab's records but the first, which the caller takes.
    bool add(unsigned long long ctx, long long* slab) noexcept {
        try {
            std::lock_guard<std::mutex> lk(mu_);
            Context* at = nullptr;
            for (Context& c : contexts_)
                if (c.id == ctx) at = &c;
            if (!at) {
                contexts_.push_back(Context{ctx, 0, {}});
                at = &contexts_.back();
            }
            at->free.reserve(at->records + SLAB);
            at->records += SLAB;
            for (int i = 1; i < SLAB; ++i) at->free.push_back(slab + i * WORDS);
            return true;
        } catch (...) {  // no host memory: the slab is lost
            return false;
        }
    }

    std::mutex mu_;
    std::vector<Context> contexts_;
};

// Ends a waiting call whose launches returned rc: failed launches (rc ==
// launch_failed) can have kernels before them still queued, on the caller's
// buffers and on the record, so those are waited for before anyone uses either
// again; other failures launched nothing.  sync() -> whether the wait succeeded;
// the first n words are then copied to out.
template <typename Sync>
int finish_sizes(int rc, int launch_failed, const long long* words, int n, long long* out, Sync sync) {
    if (rc) {
        if (rc == launch_failed) sync();
        return rc;
    }
    if (!sync()) return launch_failed;
    for (int i = 0; i < n; ++i) out[i] = static_cast<const volatile long long*>(words)[i];
    return 0;
}

}  // namespace iso
