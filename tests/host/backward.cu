// The adjoint's backward when a segment cannot be recomputed (its graph capture is
// refused).  Argument: which of the three seed arrays are given, as bits.  Prints
// the backward's status, the copies it made from the seeds, and how many of them
// were still unfinished when it returned.
#include "fake_cuda.h"
#include <stdio.h>
#include <stdlib.h>
#include "asph_ctx.cuh"

int main(int argc, char** argv) {
    if (argc != 2) return 2;
    const int given = atoi(argv[1]);
    AsphParams p;
    if (asph_params_preset(&p, ASPH_PRESET_REFERENCE, 14, 14, 5)) return 3;
    asph_ctx* c = nullptr;
    asph_adj* a = nullptr;
    if (asph_create(&p, nullptr, &c)) return 4;
    c->initialised = true;
    if (asph_adj_create(c, 2, 1, &a)) return 5;
    if (asph_adj_forward(a)) {
        fprintf(stderr, "%s\n", asph_last_error());
        return 6;
    }
    const size_t N = (size_t)c->P.N;
    std::vector<float> qc(N), th(N), xyz(3 * N), out(N);
    fake_copies.clear();
    fake_waited = 0;
    fake_capture_fails = true;
    const int st = asph_adj_backward(a, given & 1 ? qc.data() : nullptr, given & 2 ? th.data() : nullptr,
                                     given & 4 ? xyz.data() : nullptr, out.data(), nullptr);
    int made = 0, unfinished = 0;
    for (size_t k = 0; k < fake_copies.size(); ++k) {
        if (fake_copies[k].kind != cudaMemcpyHostToDevice) continue;
        ++made;
        unfinished += k >= fake_waited;
    }
    printf("%d %d %d\n", st, made, unfinished);
    return 0;
}
