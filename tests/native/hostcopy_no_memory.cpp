// Host check of bld::HostCopy with a fake runtime whose copies are plain ones: copies in
// both directions while the memory for a worker thread runs out after 0, 1, 2 or more of
// them.  Prints the number of copies that came back changed.
#include <cstdio>
#include <cstdlib>
#include <new>
#include <vector>

#include "bld_hostcopy.h"

static thread_local int allocations_left = -1;   // of this thread; negative: no limit

void* operator new(size_t n) {
    if (allocations_left == 0) throw std::bad_alloc();
    if (allocations_left > 0) --allocations_left;
    if (void* p = malloc(n)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }

int main() {
    const size_t bytes = (size_t)5 << 20 | 12344;
    std::vector<unsigned char> from(bytes), to(bytes);
    for (size_t i = 0; i < bytes; ++i) from[i] = (unsigned char)(i * 2654435761u >> 13);
    bld::HostCopy& c = bld::HostCopy::get();
    c.add_user();
    int bad = 0;
    for (int left = 0; left < 5; ++left)
        for (bool up : {true, false}) {
            std::fill(to.begin(), to.end(), 0);
            allocations_left = left;
            const cudaError_t e = c.copy(to.data(), from.data(), bytes, up, nullptr, 0);
            allocations_left = -1;
            bad += e != cudaSuccess || to != from;
        }
    c.drop_user();
    printf("%d\n", bad);
    return 0;
}
