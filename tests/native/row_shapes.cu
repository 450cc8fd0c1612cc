// Prints the shape of every in-place x kernel: kind, points, double (0) or single (1)
// precision, radices, rows per block, threads, blocks per SM.
#include <cstdio>

#include "bld_xrow.h"

static void print(const char* kind, int points, bool fp32, const bld_row::Shape& s) {
    if (s.A) printf("%s,%d,%d,%d,%d,%d,%d,%d\n", kind, points, (int)fp32, s.A, s.B, s.NR, s.T, s.MINB);
}

int main() {
    for (bool fp32 : {false, true}) {
#define X(N) print("adv", N, fp32, bld_row::adv_shape(N, fp32));
        BLD_ROW_ADV_SIZES(X)
#undef X
#define X(N) print("sgs", N, fp32, bld_row::sgs_shape(N, fp32));
        BLD_ROW_SGS_SIZES(X)
#undef X
    }
    return 0;
}
