// How often the autotuner launches a candidate.
#pragma once

#include <algorithm>

namespace bld {

// A candidate is launched once to warm up, then `iters` times between two events.  The
// events tick in steps of about 2 us, so where those launches took less than 100 us (`ms`
// each) it is timed again over as many as take 200 us, 12 at most.  Creating a small model is
// mostly this timing: with up to 40 launches a candidate (and the persistent projections on
// grids of one tile per SM) the first 16^2 x 8 LES took 10.5 ms and channel 5.9, now 9.2 and
// 4.6 (9.2 and 4.3 before the in-place kernels, 64^2 x 32 28.8 and now 12.4).  Fewer launches
// of the kernels of 16 to 33 us leave their z chunks to chance (a step of two members of
// 53 x 135 x 23 378 or 403 us, a right-hand side of 188 x 156 x 13 55 or 59).
inline int tune_relaunches(float ms, int iters) {
    if (ms * iters >= 0.1f) return 0;
    return std::max(iters, std::min(12, (int)(0.2f / std::max(ms, 0.002f))));
}

}  // namespace bld
