// The staging memory of the object and probe transfers (cubokit_b200/csrc/host_staging.h): one size for every transfer of a
// plan, and pageable memory where none can be page-locked.  Run by tests/test_host_staging.py.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "host_staging.h"

static int allocations = 0, frees = 0;
static size_t limit = SIZE_MAX;  // larger requests fail

static void *allocate(size_t bytes) {
    if (bytes > limit) return nullptr;
    allocations++;
    return std::malloc(bytes);
}
static void release(void *p) {
    frees++;
    std::free(p);
}

#define REQUIRE(x) \
    if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; }

int main() {
    {
        cubo::HostStaging staging(allocate, release);
        // set_state, get_state and backward of one plan: one allocation
        const cubo::StagedState set(staging, 100, 3200), get(staging, 100, 3200), backward(staging, 100, 3200);
        REQUIRE(allocations == 1 && frees == 0);
        REQUIRE(backward.probe == set.probe && backward.object == get.object && backward.object == set.probe + 1600);
        REQUIRE((unsigned char *)backward.value == backward.object + 3200);
        // a larger plan that cannot be page-locked, then the first again
        limit = 5000;
        const cubo::StagedState large(staging, 100, 100000);
        REQUIRE(allocations == 1 && frees == 1);
        std::memset(large.probe, 1, 1600 + 100000);
        *large.value = 2.5;
        const cubo::StagedState again(staging, 100, 3200);
        REQUIRE(again.probe == large.probe && again.object == again.probe + 1600);
        REQUIRE((unsigned long long)again.probe % 16 == 0);
        const cubo::StagedState larger(staging, 100, 200000);
        std::memset(larger.probe, 1, 1600 + 200000);
        limit = SIZE_MAX;
        const cubo::StagedState largest(staging, 100, 300000);
        REQUIRE(allocations == 2 && frees == 1);
        std::memset(largest.probe, 1, 1600 + 300000);
    }
    REQUIRE(allocations == 2 && frees == 2);
    return 0;
}
