// The library's operator new, which fails after a number of allocations (below 0: never).
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <new>

static std::atomic<int64_t> allocs_left{-1};
extern "C" void fail_allocations_after(int64_t count) { allocs_left = count; }

void* operator new(size_t bytes) {
    if (allocs_left.load() >= 0 && allocs_left.fetch_sub(1) <= 0) {
        allocs_left = 0;
        throw std::bad_alloc();
    }
    if (void* p = std::malloc(bytes ? bytes : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
