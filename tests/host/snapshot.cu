// Saves a context's state into a snapshot and restores it into a second
// context.  Arguments: the current device while each is made and used: first
// context, snapshot, save, second context, restore.  Prints launches and device
// copies of save and of restore, and whether the second context holds the state.
#include "fake_cuda.h"
#include <stddef.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>
#include "asph_ctx.cuh"

static size_t device_copies() {
    size_t n = 0;
    for (const FakeCopy& c : fake_copies) n += c.kind == cudaMemcpyDeviceToDevice;
    return n;
}

int main(int argc, char** argv) {
    if (argc != 6) return 2;
    int dev[5];
    for (int k = 0; k < 5; ++k) dev[k] = atoi(argv[k + 1]);
    AsphParams p;
    if (asph_params_preset(&p, ASPH_PRESET_REFERENCE, 14, 14, 5)) return 3;
    asph_ctx *a = nullptr, *b = nullptr;
    asph_snapshot* s = nullptr;
    fake_device = dev[0];
    if (asph_create(&p, nullptr, &a)) return 4;
    a->initialised = true;
    const size_t N = (size_t)a->P.N;
    for (size_t i = 0; i < 4 * N; ++i) ((float*)a->B.pos[a->B.pc])[i] = (float)i;
    for (size_t i = 0; i < N; ++i) a->B.surf[i] = (uint8_t)(i % 251);
    a->B.ctl->step = 17;
    a->B.ctl->epoch = 5;
    fake_device = dev[1];
    if (asph_snapshot_create(a, &s)) return 5;
    fake_device = dev[3];
    if (asph_create(&p, nullptr, &b)) return 4;
    b->B.ctl->epoch = 99;
    fake_launches.clear();
    fake_copies.clear();
    fake_device = dev[2];
    if (asph_snapshot_save(a, s)) return 6;
    const size_t l1 = fake_launches.size(), c1 = device_copies();
    fake_device = dev[4];
    if (asph_snapshot_restore(b, s)) return 7;
    const size_t l2 = fake_launches.size() - l1, c2 = device_copies() - c1;
    const bool same = !memcmp(a->B.pos[a->B.pc], b->B.pos[b->B.pc], N * 16) && !memcmp(a->B.surf, b->B.surf, N) &&
                      b->B.ctl->step == 17 && b->B.ctl->epoch == 99;
    printf("%zu %zu %zu %zu %d\n", l1, c1, l2, c2, (int)same);
    return 0;
}
