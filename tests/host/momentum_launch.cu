// The momentum pass's launch under its targets-per-thread option.
// Arguments: particles, then option values to set in turn ("r": read the value
// and set it as it was read).  Prints the value read at the end and the targets a
// thread of the launch takes.
#include "fake_cuda.h"
#include <stdio.h>
#include <stdlib.h>
#include "asph_ctx.cuh"

int main(int argc, char** argv) {
    if (argc < 2) return 2;
    asph_ctx c;
    c.P.N = atoi(argv[1]);
    c.P.nx = c.P.ny = c.P.nz = 100;
    c.P.ncell = 1000000;
    if (asph_set_option(&c, ASPH_OPT_TARGETS_PER_THREAD, 0)) return 4;   // as asph_create leaves it
    int v = 0;
    for (int k = 2; k < argc; ++k) {
        if (argv[k][0] == 'r') {
            if (asph_get_option(&c, ASPH_OPT_TARGETS_PER_THREAD, &v)) return 3;
        } else {
            v = atoi(argv[k]);
        }
        if (asph_set_option(&c, ASPH_OPT_TARGETS_PER_THREAD, v)) return 4;
    }
    if (asph_get_option(&c, ASPH_OPT_TARGETS_PER_THREAD, &v)) return 3;
    launch_momentum(c.P, c.B, 0, 0, nullptr);
    if (fake_launches.size() != 1) return 5;
    const unsigned threads = fake_launches[0].grid.x * fake_launches[0].block.x;
    printf("%d %d\n", v, (int)((c.P.N + threads / 2) / threads));
    return 0;
}
