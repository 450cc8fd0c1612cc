// How often the autotuner launches a candidate.
#pragma once

#include <algorithm>

namespace bld {

// A candidate is launched once to warm up, then `iters` times between two events.  The
// events tick in steps of about 2 us, so where those launches took less than 100 us (`ms`
// each) it is timed again over as many as take that, 12 at most.  Creating a small model is
// mostly this timing: with up to 40 launches and 200 us a candidate instead the first
// 16^2 x 8 model took 10.8 ms, now 8.6, and the first 64^2 x 32 one 16.2, now 13.3.  With half
// of that time for the kernels of 16 to 33 us the choice of z chunks was by chance (a step
// of two members of 53 x 135 x 23 378 or 403 us).
inline int tune_relaunches(float ms, int iters) {
    if (ms * iters >= 0.1f) return 0;
    return std::max(iters, std::min(12, (int)(0.1f / std::max(ms, 0.002f))));
}

}  // namespace bld
