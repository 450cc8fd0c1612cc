// Host check of bld_util::opt_in with a fake runtime: two threads opt one kernel in for
// two grids at the same time, the one with the smaller block being the last to set its
// limit.  Prints the limit the kernel is left with, and the largest size asked for.
#include <cuda_runtime.h>

#include <cstdio>
#include <thread>

#include "bld_launch_util.cuh"

double2 h_wtab64[BLD_WTAB_SIZE];
float2 h_wtab32[BLD_WTAB_SIZE];

extern thread_local bool is_larger;   // of the fake: the calling thread asks for the larger size
extern int limit;                      // of the fake: the last size set

static void kernel() {}

int main() {
    const int larger = 67328, smaller = 65664;   // one kernel at two grid widths
    static std::atomic<int> done[64];
    cudaError_t e[2];
    std::thread a([&] { is_larger = true, e[0] = bld_util::opt_in(kernel, larger, done); });
    std::thread b([&] { e[1] = bld_util::opt_in(kernel, smaller, done); });
    a.join();
    b.join();
    printf("%d %d %d %d\n", (int)e[0], (int)e[1], limit, larger);
    return 0;
}
