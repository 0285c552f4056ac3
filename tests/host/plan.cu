// The density pass's choice of a brick for a grid and a particle count, made on
// the host: prints the shape index (-1: the per-target path).  An exit by a
// signal is the planner's.
#include <stdio.h>
#include <stdlib.h>
#include "asph_ctx.cuh"

int main(int argc, char** argv) {
    if (argc != 5) return 2;
    asph_ctx c;
    c.P.nx = atoi(argv[1]); c.P.ny = atoi(argv[2]); c.P.nz = atoi(argv[3]);
    c.P.N = atoi(argv[4]);
    c.P.ncell = c.P.nx * c.P.ny * c.P.nz;
    c.B.shape = -1;
    int shape = -2;
    if (asph_get_option(&c, ASPH_OPT_PAIR_SHAPE, &shape)) return 3;
    printf("%d\n", shape);
    return 0;
}
