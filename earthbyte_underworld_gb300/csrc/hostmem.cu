// Reused host memory for large results: an allocator with the four functions of malloc, calloc, realloc and free.
//
// A fresh array's pages are faulted in while the device copy writes them, at about 20 GB/s against 190 GB/s into pages
// that are present, so a call that returns 150 MB took longer to fault than to compute.  A pool keeps freed blocks up
// to a limit and hands one out again where at least half of it is used.  Blocks come from malloc, so realloc is the C
// library's and a block's size is what malloc_usable_size says.  No call waits for another or runs foreign code: a
// block freed while another thread is inside goes to the C library, and one asked for meanwhile comes from it.
#include <malloc.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstdlib>
#include <mutex>
#include <new>
#include <vector>

#include "uwgpu.h"

struct uwgpu_hostmem {
    struct Block {
        void* p;
        size_t size;
    };
    std::mutex m;
    std::vector<Block> free;   // oldest first
    size_t held = 0, limit = 0, smallest = 0;

    void trim(size_t most) noexcept {
        size_t k = 0;
        for (; k < free.size() && held > most; ++k) {
            held -= free[k].size;
            std::free(free[k].p);
        }
        free.erase(free.begin(), free.begin() + (std::ptrdiff_t)k);
    }
};

namespace {

// Large fresh blocks ask for large pages exactly as numpy's own arrays do: from the next multiple of 4 KB, which a
// kernel with larger base pages refuses.
void* fresh(size_t size) noexcept {
    constexpr size_t kLarge = (size_t)4 << 20, kPage = 4096;
    void* p = std::malloc(size ? size : 1);
    if (p && size >= kLarge) {
        const size_t skip = kPage - (uintptr_t)p % kPage;
        (void)madvise(static_cast<char*>(p) + skip, size - skip, MADV_HUGEPAGE);
    }
    return p;
}

}  // namespace

extern "C" {

uwgpu_hostmem* uwgpu_hostmem_create(size_t limit, size_t smallest) {
    uwgpu_hostmem* h = new (std::nothrow) uwgpu_hostmem;
    if (h) {
        h->limit = limit;
        h->smallest = smallest;
    }
    return h;
}

void uwgpu_hostmem_limit(uwgpu_hostmem* h, size_t limit) {
    std::lock_guard<std::mutex> g(h->m);
    h->limit = limit;
    h->trim(limit);
}

void uwgpu_hostmem_release(uwgpu_hostmem* h) {
    std::lock_guard<std::mutex> g(h->m);
    h->trim(0);
}

size_t uwgpu_hostmem_held(uwgpu_hostmem* h, size_t* sizes, size_t count) {
    std::lock_guard<std::mutex> g(h->m);
    for (size_t k = 0; k < h->free.size() && k < count; ++k) sizes[k] = h->free[k].size;
    return h->free.size();
}

void* uwgpu_hostmem_malloc(uwgpu_hostmem* h, size_t size) {
    if (size >= h->smallest && h->m.try_lock()) {
        std::lock_guard<std::mutex> g(h->m, std::adopt_lock);
        size_t best = h->free.size();
        for (size_t k = 0; k < h->free.size(); ++k) {
            const size_t have = h->free[k].size;
            if (have >= size && have / 2 <= size && (best == h->free.size() || have < h->free[best].size)) best = k;
        }
        if (best < h->free.size()) {
            void* p = h->free[best].p;
            h->held -= h->free[best].size;
            h->free.erase(h->free.begin() + (std::ptrdiff_t)best);
            return p;
        }
    }
    return fresh(size);
}

void* uwgpu_hostmem_calloc(uwgpu_hostmem*, size_t count, size_t size) { return std::calloc(count ? count : 1, size ? size : 1); }

void* uwgpu_hostmem_realloc(uwgpu_hostmem*, void* p, size_t size) { return std::realloc(p, size ? size : 1); }

void uwgpu_hostmem_free(uwgpu_hostmem* h, void* p, size_t) {
    if (!p) return;
    const size_t size = malloc_usable_size(p);
    if (size >= h->smallest && size <= h->limit && h->m.try_lock()) {
        std::lock_guard<std::mutex> g(h->m, std::adopt_lock);
        if (size <= h->limit) {
            try {
                h->free.reserve(h->free.size() + 1);
                h->trim(h->limit - size);
                h->free.push_back({p, size});
                h->held += size;
                return;
            } catch (const std::bad_alloc&) {
            }
        }
    }
    std::free(p);
}

}  // extern "C"
