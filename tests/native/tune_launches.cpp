// Prints, per kernel time in microseconds, how often the autotuner launches it once more.
#include <cstdio>

#include "bld_tune.h"

int main() {
    for (int us = 0; us <= 60; ++us) printf("%d,%d\n", us, bld::tune_relaunches(us * 1e-3f, 3));
    return 0;
}
