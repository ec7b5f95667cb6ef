// parallel_ranges (cubokit_b200/csrc/host_ranges.h) where memory for its threads runs out: every item is still taken once.
// Run by tests/test_host_ranges.py.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <new>

#include "host_ranges.h"

static std::atomic<int> left{-1};  // allocations that still succeed; negative: all do

void *operator new(std::size_t n) {
    if (left >= 0 && left-- == 0) {
        left = 0;  // and none after it
        throw std::bad_alloc();
    }
    if (void *p = std::malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, std::size_t) noexcept { std::free(p); }

int main() {
    constexpr size_t kItems = 1003;
    for (int allowed = -1; allowed < 12; allowed++) {  // the vector, then one state per thread
        std::atomic<int> taken[kItems] = {};
        left = allowed;
        cubo::parallel_ranges(kItems, 100, [&](size_t first, size_t last) {
            for (size_t i = first; i < last; i++) taken[i]++;
        });
        left = -1;
        for (size_t i = 0; i < kItems; i++)
            if (taken[i] != 1) {
                std::printf("%d allocations: item %zu taken %d times\n", allowed, i, taken[i].load());
                return 1;
            }
    }
    return 0;
}
