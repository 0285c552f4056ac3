// asph_pairs.cu — the two pair passes of the step, for sm_103a:
//   D  density (lagged Shepard) + EOS + microphysics (asph_h100.cu:286-402)
//   M  momentum + integration + rain sedimentation + CFL control
//      (asph_h100.cu:415-599, 1040-1078)
//
// Candidate set (identical to the reference): for target i, every particle
// listed by the cell table in the cells within +-2 of i's *current* cell,
// x/y wrapped, z clipped at the walls; the table is the one built at the
// last sort (positions have drifted since), distances are raw coordinate
// differences in cell units (no minimum image).  D and M see the same
// positions and table, so they accept the same pairs: D enumerates the
// candidates once and records each target's accepted neighbours (self
// excluded) in a slot-major list; M walks that list.
//
// D, brick path.  One CTA per Morton-aligned brick of BX x BY x BZ cells;
// the brick's targets are one contiguous span of the sorted order, a thread
// each.  The CTA copies the particles of every table cell within H cells of the
// brick into shared memory, bucketed row-major by region cell, so that each
// row of a target's 5 x 5 x 5 window is one contiguous span of slots.  A
// warp walks its targets' rows together, four candidates a step in fp16, queues
// what that test passes in a small per-thread list in shared memory, and
// drains the lists (float test, density sums, neighbour-list writes) together.
// What bounds the pass is instruction issue: about 75 candidates and 20
// neighbours per target at 0.6 particles per cell against 48 bytes.  Density per
// step at 2M, walk in float with a row advance in every step against this one:
// 0.6 per cell 511 -> 471 us, the same clustered 1018 -> 693 us, 8:1 cells
// 516 -> 435 us, one per cell 1191 -> 728 us (the reference's lattice 620 -> 432;
// there with the smaller brick and halo too); 475k 152 -> 132 us, 262k at one per cell
// 206 -> 131 us.  It issues on 60 % of the cycles with 31 of 32 lanes, and the
// shared-memory pipe is busy on 69 % (524k).
// H = 2 (the stencil) covers every target still in a cell of its brick; H = 3 also
// covers one cell of drift since the sort.  A region that overflows the
// staging capacity is split into its two Morton-aligned halves (each a
// contiguous sub-span of the targets with a smaller region), and a half
// that overflows once more; a target whose window leaves the staged region,
// and the targets of a quarter that still overflows, are queued for the
// deferred pass.
//
// Deferred pass.  One warp per queued target: the lanes read the window's
// cell ranges from the global table in parallel and test the candidates 32
// at a time in the reference's order, so the neighbour list comes out in
// that order.
//
// Global path.  One thread per target walking the cell table in global
// memory, the reference's loop structure; used for grids narrower than the
// staged region, and by M for a target whose list overflowed or was not
// produced on the current positions.
#include <cuda_fp16.h>
#include "asph_device.cuh"
#include "../../include/asph.h"

namespace asph {

constexpr int MAX_HALO = 3;      // widest staged halo (cells around a brick)
// Register cap of the brick kernel (its launch plan counts on it).  48 keep a
// fourth block of 320 threads per SM, but spill, and leave queues of 18 entries
// and little staging room; 56 do not spill and leave three blocks queues of 30 and
// regions that rarely split.  Density with 48 / 56 / 64: 466 / 471 / 470 us at 2M from
// the lattice, 802 / 693 / 692 clustered, 741 / 728 / 725 at one per cell, 436 / 435 /
// 466 with 8:1 cells; over 500 steps of the moist bubble 0.964 / 0.941 ms a step.
constexpr int DENSITY_REGS = 56;
constexpr int DLIST = 30;        // most queued accepted candidates per thread (D); a launch may use fewer
// The walk's fp16 test of a candidate.  Coordinates are within FCLAMP < 8
// cells of the region's centre, so their fp16 rounding is at most 2^-9 each
// (plus 1e-4 from forming them in float), a pair's distance is off by less than
// 2 sqrt(3) (2^-9 + 1e-4) = 0.0072, a pair with r < 2 has a rounded r^2 below
// 4.029, and the five fp16 roundings of forming it (2^-11 relative each) leave
// it below 4.0389.  The threshold is the next fp16 number above.
constexpr float FCLAMP = 7.9f;
constexpr float FTHR = 4.0390625f;
// Momentum blocks of 128 threads: a block ends with its slowest warp, and
// smaller blocks waste less of an SM on warps that wait for it (measured at
// 2M from init: 0.298 / 0.260 / 0.257 / 0.271 ms at 32 / 64 / 128 / 256).
constexpr int M_TPB = 128;
constexpr int M_MINB = 1024 / M_TPB;                     // resident blocks that keep 64 registers
// Rain cells per thread of a rain block: 1,024 cells a block, so that the
// rain advection adds few blocks (and few finished-block atomics) to the
// pass (momentum at 2M from init: 0.262 / 0.245 / 0.256 ms at 256 / 1,024 /
// 4,096 cells a block).
constexpr int M_RAIN_CELLS = 8;

template <int BX, int BY, int BZ, int H>
struct BrickGeom {
    static_assert((BX == BY && BY == BZ) || (BX == 2 * BY && BY == BZ) || (BX == BY && BX == 2 * BZ),
                  "brick must be a Morton-aligned key range");
    static_assert(H >= STENCIL && H <= MAX_HALO, "halo must cover the stencil");
    static constexpr int RX = BX + 2 * H, RY = BY + 2 * H, RZ = BZ + 2 * H;
    static constexpr int R = RX * RY * RZ;
    static constexpr int KEYS = BX * BY * BZ;
    static constexpr int LOG2K = KEYS >= 512 ? 9 : KEYS >= 256 ? 8 : KEYS >= 128 ? 7 : KEYS >= 64 ? 6
                               : KEYS >= 32 ? 5 : KEYS >= 16 ? 4 : 3;
    static_assert((1 << LOG2K) == KEYS, "brick key count is a power of two");
};

// The two Morton-aligned halves of a brick: the top bit of a brick-local
// key is z's for a cube, y's for BX = BY = 2 BZ and x's for BX = 2 BY = 2 BZ,
// so the lower half of the brick's keys is the half with the smaller
// coordinate along that axis, and each half is again a contiguous span of
// the sorted order.
template <int BX, int BY, int BZ>
struct BrickHalves {
    static constexpr bool cube = BX == BY && BY == BZ;
    static constexpr bool flat = BX == BY && BX == 2 * BZ;   // next split along y
    static constexpr int X = cube || flat ? BX : BX / 2;
    static constexpr int Y = flat ? BY / 2 : BY;
    static constexpr int Z = cube ? BZ / 2 : BZ;
    static constexpr int DX = BX - X, DY = BY - Y, DZ = BZ - Z;   // offset of the upper half
};

struct PairCfg {
    int nbx, nby, nbz, nbricks;
    int cap;            // staged particles that fit in shared memory
    int dlist;          // drain-queue depth of this launch (16 to DLIST)
    uint32_t qinv;      // 2^32 / bytes of a queue row, rounded up
};

namespace {

__device__ __forceinline__ int lower_bound_u32(const uint32_t* __restrict__ a, int n, uint32_t key) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&a[mid]) < key) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Exclusive scan of one int per thread over the block (any multiple of 32
// up to 1024 threads).
__device__ __forceinline__ int block_excl_scan_int(int v, int* s_warp, int* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nw ? s_warp[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) s_warp[lane] = w;
    }
    __syncthreads();
    const int off = warp ? s_warp[warp - 1] : 0;
    *total = s_warp[nw - 1];
    __syncthreads();
    return x - v + off;
}

// Walk the reference window of one target through the global cell table.
// At most ASPH_MAX_CANDIDATES candidates are visited: a denser window can
// only come from a blown-up state (the reference would spend quadratic
// time on it), so the run is stopped with ASPH_ERR_DENSE instead.
template <class F>
__device__ __forceinline__ void for_window_global(const Phys& P, const int2* __restrict__ range, DevCtl* ctl, float x,
                                                  float y, float z, F&& f) {
    const int ix = cell_ix(x, P.inv_dx, P.nx), iy = cell_ix(y, P.inv_dy, P.ny), iz = cell_ix(z, P.inv_dz, P.nz);
    const int z0 = max(iz - STENCIL, 0), z1 = min(iz + STENCIL, P.nz - 1);
    int budget = ASPH_MAX_CANDIDATES;
    for (int jz = z0; jz <= z1; ++jz)
        for (int jy = iy - STENCIL; jy <= iy + STENCIL; ++jy) {
            const int cy = wrapi(jy, P.ny);
            const int2* row = range + (size_t)(jz * P.ny + cy) * P.nx;
            for (int jx = ix - STENCIL; jx <= ix + STENCIL; ++jx) {
                const int2 rg = row[wrapi(jx, P.nx)];
                budget -= rg.y - rg.x;
                if (budget < 0) {
                    stop_run(ctl, ASPH_ERR_DENSE);
                    return;
                }
                for (int j = rg.x; j < rg.y; ++j) f(j);
            }
        }
}

// Region-local window of a target: returns false if it leaves the region.
template <int BX, int BY, int BZ, int H>
__device__ __forceinline__ bool local_window(const Phys& P, int ox, int oy, int oz, float x, float y, float z,
                                             int& lx, int& ly, int& zlo, int& zhi) {
    using G = BrickGeom<BX, BY, BZ, H>;
    const int ix = cell_ix(x, P.inv_dx, P.nx), iy = cell_ix(y, P.inv_dy, P.ny), iz = cell_ix(z, P.inv_dz, P.nz);
    lx = ix - (ox - H);
    lx += lx < 0 ? P.nx : 0; lx -= lx >= P.nx ? P.nx : 0;
    ly = iy - (oy - H);
    ly += ly < 0 ? P.ny : 0; ly -= ly >= P.ny ? P.ny : 0;
    const int rz0 = oz - H;
    zlo = max(iz - STENCIL, 0) - rz0;
    zhi = min(iz + STENCIL, P.nz - 1) - rz0;
    return lx >= STENCIL && lx < G::RX - STENCIL && ly >= STENCIL && ly < G::RY - STENCIL && zlo >= 0 &&
           zhi < G::RZ;
}

// Offsets of the staged region of a brick: s_off[l] = first slot of region
// cell l (row-major, H cells around the brick, x/y wrapped), s_off[R] =
// the total, and s_gidx[k] = the global index of every slot that fits.  A
// cell's particles take consecutive slots in index order.  Two threads take a row of cells, half of it each, all their table
// loads in flight: the threads' order is the slots' order, so one block scan
// of the threads' counts gives the offsets.
template <int BX, int BY, int BZ, int H>
__device__ int region_offsets(const Phys& P, const int2* __restrict__ range, int ox, int oy, int oz, int* s_off,
                              int* s_gidx, int cap, int* s_warp) {
    using G = BrickGeom<BX, BY, BZ, H>;
    constexpr int HX = G::RX / 2, HALVES = 2 * G::RY * G::RZ;
    const int T = blockDim.x;
    int carry = 0;
    for (int q0 = 0; q0 < HALVES; q0 += T) {
        const int q = q0 + threadIdx.x, row = q >> 1, x0 = (q & 1) * HX;
        int start[HX], cnt[HX];
        const int lz = row / G::RY, ly = row - lz * G::RY, gz = oz - H + lz;
        int gy = oy - H + ly;
        gy += gy < 0 ? P.ny : 0; gy -= gy >= P.ny ? P.ny : 0;
        const bool in = q < HALVES && gz >= 0 && gz < P.nz;
        const int2* const tab = range + (size_t)(gz * P.ny + gy) * P.nx;
        int run = 0;
#pragma unroll
        for (int c = 0; c < HX; ++c) {
            int gx = ox - H + x0 + c;
            gx += gx < 0 ? P.nx : 0; gx -= gx >= P.nx ? P.nx : 0;
            const int2 rg = in ? tab[gx] : make_int2(0, 0);
            start[c] = rg.x;
            cnt[c] = rg.y - rg.x;
        }
#pragma unroll
        for (int c = 0; c < HX; ++c) run += cnt[c];
        int total;
        int k = carry + block_excl_scan_int(run, s_warp, &total);
        carry += total;
        if (q < HALVES) {
            int* const o = s_off + row * G::RX + x0;
#pragma unroll
            for (int c = 0; c < HX; ++c) {
                o[c] = k;
                const int e = min(cnt[c], cap - k);   // slots beyond the capacity: the region is split
                for (int j = 0; j < e; ++j) s_gidx[k + j] = start[c] + j;
                k += cnt[c];
            }
        }
    }
    if (threadIdx.x == 0) s_off[G::R] = carry;
    __syncthreads();
    return carry;
}

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<uint32_t*>(&h); }
__device__ __forceinline__ __half2 h2_of(uint32_t b) { return *reinterpret_cast<__half2*>(&b); }
// fp16 cell coordinate from the region's centre.  Clamping brings points together, never apart.
__device__ __forceinline__ __half feat_coord(float x, float c, float inv) {
    return __float2half_rn(fminf(fmaxf((x - c) * inv, -FCLAMP), FCLAMP));
}

// Neighbour-list writer of one target (slot-major, coalesced over targets).
struct NbrOut {
    int* p;      // the next slot of target i's list
    size_t N;    // slot stride
    int n;
    __device__ __forceinline__ NbrOut(int* nbr, int n0, int N_, int i) : p(nbr + i), N((size_t)N_), n(n0) {}
    __device__ __forceinline__ void push(int j) {
        if (n < NBR_CAP) {
            *p = j;
            p += N;
        }
        ++n;
    }
    __device__ __forceinline__ void push_if(bool take, int j) {   // predicated, no branch
        asm volatile("{\n"
                     "  .reg .pred p, q;\n"
                     "  setp.ne.s32 p, %2, 0;\n"
                     "  setp.lt.and.s32 q, %1, %4, p;\n"
                     "  @q st.global.u32 [%0], %3;\n"
                     "  @q add.u64 %0, %0, %5;\n"
                     "  @p add.s32 %1, %1, 1;\n"
                     "}\n"
                     : "+l"(p), "+r"(n)
                     : "r"((int)take), "r"(j), "n"(NBR_CAP), "l"(N * 4)
                     : "memory");
    }
};

}  // namespace

// ===========================================================================
// D: density + EOS + microphysics, neighbour lists
// ===========================================================================
struct DArgs {
    const float4* pos;      // x, y, z, rho_old
    const int2* range;
    const uint32_t* skeys;  // sorted keys of the table's order
    const int2* spans;      // per brick: its span of targets in the sorted order
    DOut out;
    int* nbr;
    int* nbr_cnt;
    int* defer;             // targets queued for the deferred pass (count in ctl->defer_n)
    DevCtl* ctl;
};

// First index of a sorted array whose value is not below `key`, by a whole
// warp: 32 probes a round, so five dependent loads for 2M keys against 21.
__device__ __forceinline__ int lower_bound_warp(const uint32_t* __restrict__ a, int n, uint32_t key) {
    const int lane = threadIdx.x & 31;
    int lo = 0;
    for (;;) {
        const int step = (n - lo + 31) / 32;   // probes at lo, lo + step, ...
        const long long at = lo + (long long)lane * step;
        const int below = __popc(__ballot_sync(0xffffffffu, at < n && __ldg(&a[at < n ? at : 0]) < key));
        if (step <= 1) return lo + below;
        if (below == 0) return lo;
        const long long end = lo + (long long)below * step;   // the first probe not below, or past the end
        lo += (below - 1) * step + 1;
        n = end < n ? (int)end : n;
        if (lo >= n) return lo;
    }
}

// Every brick's span of targets in the sorted order: the brick is a
// Morton-aligned key range, found by search in the sorted keys (a warp for each
// end of a span).  The gather writes the same spans when a sort runs; this
// kernel serves sorted keys that the gather did not see (a restored state,
// another brick shape): 13 -> 4 us at 475k particles against a thread per
// brick and a binary search.
template <int BX, int BY, int BZ>
__global__ void k_brick_spans(const __grid_constant__ Phys P, const uint32_t* __restrict__ skeys, int2* spans,
                              PairCfg C) {
    using G = BrickGeom<BX, BY, BZ, STENCIL>;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, b = w >> 1, upper = w & 1;
    if (b >= C.nbricks) return;
    const int bxi = b % C.nbx, byi = (b / C.nbx) % C.nby, bzi = b / (C.nbx * C.nby);
    const uint32_t base = morton3((uint32_t)(bxi * BX), (uint32_t)(byi * BY), (uint32_t)(bzi * BZ));
    const int at = lower_bound_warp(skeys, P.N, base + (upper ? (uint32_t)G::KEYS : 0u));
    if ((threadIdx.x & 31) == 0) reinterpret_cast<int*>(spans + (base >> G::LOG2K))[upper] = at;
}

__device__ __forceinline__ DSum density_target_global(const Phys& P, const DArgs& A, int i, float4 pi, FF rr) {
    DSum s{0.f, 0.f, 0.f};
    NbrOut L{A.nbr, 0, P.N, i};
    for_window_global(P, A.range, A.ctl, pi.x, pi.y, pi.z, [&](int j) {
        const float4 pj = A.pos[j];
        const float r2 = r2_pair(P, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z);
        if (r2 < 4.0f) {
            dsum_add(s, r2, pj.w, rr);
            if (r2 >= 1e-12f) L.push(j);
        }
    });
    A.nbr_cnt[i] = L.n <= NBR_CAP ? L.n : -1;
    return s;
}

__global__ __launch_bounds__(256) void k_density_global(const __grid_constant__ Phys P,
                                                        const __grid_constant__ DArgs A) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (A.ctl->aborted || i >= P.N) return;
    const float dt = A.ctl->dt;
    const float4 pi = A.pos[i];
    const FF rr = snd_eval(P.snd_rho, P.snd_n, pi.z);
    const DSum s = density_target_global(P, A, i, pi, rr);
    density_eos_epilogue(P, A.out, i, pi, s, rr, dt);
}

// The density pass's dynamic shared memory (plan() sizes it).
struct DSmem {
    unsigned char* feat;      // at its start, so that a slot's offset fits a queue entry: per pair of slots 16
                              // bytes {x2, y2, z2, -}, fp16 cell coordinates from the region's centre; the
                              // pair after the last one that fits is far from everything
    float4* sp;               // staged particles: x, y, z, rho_old
    int* s_gidx;              // global index of a staged slot
    int* s_off;               // region cell -> first slot (R + 1)
    unsigned short* s_list;   // drain queue, dlist x T: 8 x slot
    int* s_warp;
    int* s_work;              // work items {ox, oy, oz, ts, te}: the root, then two per split level
};
constexpr int DENSITY_SPLITS = 2;   // an overflowing brick is split into halves, then quarters

// The work item at M.s_work + 5 * slot: the targets [ts, te) of the
// Morton-aligned brick with origin (ox, oy, oz) cells.  Stage the region,
// walk and drain.  A region that overflows the staging capacity is split
// into its two halves (each its own region and a contiguous sub-span of the
// targets), SPLITS times at most; targets the staged region still does not
// cover go to the deferred pass.  Work items live in shared memory, so
// nothing stays in registers across the first half's pass.
template <int BX, int BY, int BZ, int H, int SPLITS>
__device__ __forceinline__ void density_region(const Phys& P, const DArgs& A, const PairCfg& C, const DSmem& M,
                                               int slot) {
    using G = BrickGeom<BX, BY, BZ, H>;
    const int T = blockDim.x;
    // the work item was written by thread 0 before the call, and the shared
    // arrays of an earlier region are no longer read
    __syncthreads();
    const int* w = M.s_work + 5 * slot;
    const int ox = w[0], oy = w[1], oz = w[2], ts = w[3], te = w[4];
    const float dt = A.ctl->dt;
    float4* sp = M.sp;
    int* s_gidx = M.s_gidx;
    int* s_off = M.s_off;
    unsigned short* s_list = M.s_list;

    // ---- stage the region: counts, scan (row-major by region cell), copy
    const int total = region_offsets<BX, BY, BZ, H>(P, A.range, ox, oy, oz, s_off, s_gidx, C.cap, M.s_warp);
    const bool staged = total <= C.cap;
    if constexpr (SPLITS > 0) {
        if (!staged) {
            using S = BrickHalves<BX, BY, BZ>;
            const int c0 = 1 + 2 * (DENSITY_SPLITS - SPLITS);   // this level's two child slots
            if (threadIdx.x == 0) {
                atomicAdd(&A.ctl->split_n, 1u);
                const uint32_t half = morton3((uint32_t)ox, (uint32_t)oy, (uint32_t)oz) + (uint32_t)(G::KEYS / 2);
                const int mid = ts + lower_bound_u32(A.skeys + ts, te - ts, half);
                int* a = M.s_work + 5 * c0;
                a[0] = ox; a[1] = oy; a[2] = oz; a[3] = ts; a[4] = mid;
                a[5] = ox + S::DX; a[6] = oy + S::DY; a[7] = oz + S::DZ; a[8] = mid; a[9] = te;
            }
            density_region<S::X, S::Y, S::Z, H, SPLITS - 1>(P, A, C, M, c0);       // (starts with a barrier)
            density_region<S::X, S::Y, S::Z, H, SPLITS - 1>(P, A, C, M, c0 + 1);
            return;
        }
    }
    const float cx = ((float)ox + 0.5f * BX) * P.dx, cy0 = ((float)oy + 0.5f * BY) * P.dy,
                cz = ((float)oz + 0.5f * BZ) * P.dz;   // the region's centre
    if (staged) {
        // slots strided over the block, four loads in flight per thread
        for (int k0 = threadIdx.x; k0 < total; k0 += 4 * T) {
            float4 p[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k0 + u * T < total) p[u] = A.pos[s_gidx[k0 + u * T]];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                if (k0 + u * T < total) {
                    const int k = k0 + u * T;
                    sp[k] = p[u];
                    __half* const f = reinterpret_cast<__half*>(M.feat + (k >> 1) * 16) + (k & 1);
                    f[0] = feat_coord(p[u].x, cx, P.inv_dx);
                    f[2] = feat_coord(p[u].y, cy0, P.inv_dy);
                    f[4] = feat_coord(p[u].z, cz, P.inv_dz);
                }
        }
    }
    __syncthreads();

    // ---- targets, one warp-synchronous round of 32 targets at a time
    const int lane = threadIdx.x & 31;
    for (int base = ts + (threadIdx.x & ~31); base < te; base += T) {
        const int i = base + lane;
        const bool active = i < te;
        float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
        FF rr{0.f, 0.f};
        DSum s{0.f, 0.f, 0.f};
        int lx = 0, ly = 0, zlo = 0, zhi = -1;
        bool fast = false;
        if (active) {
            pi = A.pos[i];
            rr = snd_eval(P.snd_rho, P.snd_n, pi.z);
            fast = staged && local_window<BX, BY, BZ, H>(P, ox, oy, oz, pi.x, pi.y, pi.z, lx, ly, zlo, zhi);
        }
        // targets the staged region does not cover go to the deferred pass
        const unsigned dm = __ballot_sync(0xffffffffu, active && !fast);
        if (dm) {
            const int lead = __ffs(dm) - 1;
            unsigned at = 0;
            if (lane == lead) at = atomicAdd(&A.ctl->defer_n, (unsigned)__popc(dm));
            at = __shfl_sync(0xffffffffu, at, lead);
            if (active && !fast) A.defer[at + __popc(dm & ((1u << lane) - 1u))] = i;
        }
        NbrOut L{A.nbr, 0, P.N, i};
        // the lanes' queues are the columns of the dlist x T array, the next
        // entry of this lane at shared address qat, so a push is one predicated
        // store and one add
        unsigned short* const qlane = s_list + threadIdx.x;
        const uint32_t q0 = (uint32_t)__cvta_generic_to_shared(qlane), qstep = 2u * (uint32_t)T;
        uint32_t qat = q0;
        // All lanes drain their queues together, in lockstep and without
        // branches: an entry that fails the float test, and a lane whose queue has
        // ended (it reads slot 0), adds zero to the sums and stores nothing.
#define ASPH_DRAIN()                                                                      \
    do {                                                                                  \
        const int n_ = (int)(qat - q0) >> 1;                                              \
        const int nmax_ = __reduce_max_sync(0xffffffffu, n_);                             \
        for (int q_ = 0; q_ < nmax_; q_ += T) {                                           \
            const uint32_t a_ = q_ < n_ ? qlane[q_] : 0u;                                 \
            const float4 pj = *reinterpret_cast<const float4*>(spb + 2u * a_);            \
            const int j_ = *reinterpret_cast<const int*>(gib + (a_ >> 1));                \
            const float r2_ = r2_pair(P, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z);             \
            const bool near_ = q_ < n_ && r2_ < 4.0f;                                     \
            dsum_add_if(s, r2_, pj.w, rr, near_);                                         \
            L.push_if(near_ && r2_ >= 1e-12f, j_);                                        \
        }                                                                                 \
        qat = q0;                                                                         \
    } while (0)
        const unsigned char* const spb = reinterpret_cast<const unsigned char*>(sp);
        const unsigned char* const gib = reinterpret_cast<const unsigned char*>(s_gidx);
        // The walk: the window's rows one after another for the whole warp, four
        // candidates a step, two pairs of slots in fp16 (half2: seven
        // operations for a pair against ten each in float).  The loop's own cost (vote,
        // branch, queue bound) is a third of a step of one pair, and a row is
        // mostly two or three pairs: with two pairs a step (and 48 registers) density takes 466 against
        // 469 us at 2M, 741 against 822 at one per cell, 799 against 825 clustered
        // (438 against 441 the other way on the reference's unjittered lattice).  The fp16 test only
        // ever passes too many (FTHR); what passes is queued and takes the float test
        // in the drain.  A lane whose row has ended tests what follows and takes none.
        // Lanes of a warp have rows of much the same length (their windows
        // overlap), so waiting for the longest one costs less than letting each
        // lane run on into its next row, a dozen instructions more in every step.
        // The next row's span is read one row ahead: 893 -> 876 us clustered and 504 -> 466 even
        // with one pair a step and 48 registers; with two pairs and 56 it makes no difference
        // (468 against 468 us at 2M, 960 against 956 clustered without it).
        const __half2 xi2 = __half2half2(feat_coord(pi.x, cx, P.inv_dx));
        const __half2 yi2 = __half2half2(feat_coord(pi.y, cy0, P.inv_dy));
        const __half2 zi2 = __half2half2(feat_coord(pi.z, cz, P.inv_dz));
        const uint32_t thr = h2_bits(__float2half2_rn(FTHR));
        const int* ro = s_off + (zlo * G::RY + ly - STENCIL) * G::RX + lx - STENCIL;
        const int planes = fast ? zhi - zlo + 1 : 0;
        const int nplanes = __reduce_max_sync(0xffffffffu, planes);
        int room = C.dlist;   // entries that certainly fit in every lane's queue
        int kf = 0, ke = 0;   // the next row's slots, read one row ahead
        if (planes > 0) {
            kf = ro[0];
            ke = ro[2 * STENCIL + 1];
        }
        for (int jz = 0; jz < nplanes; ++jz) {
            for (int jy = 0; jy <= 2 * STENCIL; ++jy) {
                const int kfirst = kf * 8, kend = ke * 8;   // in 8-byte units of the features
                ro += G::RX;
                if (jy == 2 * STENCIL) ro += G::RX * G::RY - (2 * STENCIL + 1) * G::RX;
                kf = ke = 0;
                if (jz + (jy == 2 * STENCIL ? 1 : 0) < planes) {
                    kf = ro[0];
                    ke = ro[2 * STENCIL + 1];
                }
                int k = kfirst & ~15;
                while (__any_sync(0xffffffffu, k < kend)) {
                    const uint4 f = *reinterpret_cast<const uint4*>(M.feat + k);
                    const uint4 g = *reinterpret_cast<const uint4*>(M.feat + k + 16);
                    __half2 d = __hsub2(h2_of(f.x), xi2), e = __hsub2(h2_of(g.x), xi2);
                    __half2 r2 = __hmul2(d, d), s2 = __hmul2(e, e);
                    d = __hsub2(h2_of(f.y), yi2); e = __hsub2(h2_of(g.y), yi2);
                    r2 = __hfma2(d, d, r2); s2 = __hfma2(e, e, s2);
                    d = __hsub2(h2_of(f.z), zi2); e = __hsub2(h2_of(g.z), zi2);
                    r2 = __hfma2(d, d, r2); s2 = __hfma2(e, e, s2);
                    asm volatile("{\n"
                                 "  .reg .pred c, p, q, u, v;\n"
                                 "  .reg .b16 h;\n"
                                 "  .reg .b32 k1, k2, k3;\n"
                                 "  add.s32 k1, %4, 8;\n"
                                 "  add.s32 k2, %4, 16;\n"
                                 "  add.s32 k3, %4, 24;\n"
                                 "  setp.lt.s32 c, %4, %6;\n"
                                 "  setp.le.and.f16x2 p|q, %1, %3, c;\n"
                                 "  setp.ge.and.s32 p, %4, %5, p;\n"
                                 "  setp.lt.and.s32 q, k1, %6, q;\n"
                                 "  setp.lt.s32 c, k2, %6;\n"
                                 "  setp.le.and.f16x2 u|v, %2, %3, c;\n"
                                 "  setp.lt.and.s32 v, k3, %6, v;\n"
                                 "  cvt.u16.u32 h, %4;\n"
                                 "  @p st.shared.u16 [%0], h;\n"
                                 "  @p add.u32 %0, %0, %7;\n"
                                 "  cvt.u16.u32 h, k1;\n"
                                 "  @q st.shared.u16 [%0], h;\n"
                                 "  @q add.u32 %0, %0, %7;\n"
                                 "  cvt.u16.u32 h, k2;\n"
                                 "  @u st.shared.u16 [%0], h;\n"
                                 "  @u add.u32 %0, %0, %7;\n"
                                 "  cvt.u16.u32 h, k3;\n"
                                 "  @v st.shared.u16 [%0], h;\n"
                                 "  @v add.u32 %0, %0, %7;\n"
                                 "}\n"
                                 : "+r"(qat)
                                 : "r"(h2_bits(r2)), "r"(h2_bits(s2)), "r"(thr), "r"(k), "r"(kfirst), "r"(kend),
                                   "r"(qstep)
                                 : "memory");
                    k += 32;
                    room -= 4;
                    if (room < 4) {   // as far as the steps tell: take the real room, drain when there is little
                        room = C.dlist - (int)__umulhi(__reduce_max_sync(0xffffffffu, qat - q0), C.qinv);
                        if (room < 4) {
                            ASPH_DRAIN();
                            room = C.dlist;
                        }
                    }
                }
            }
        }
        ASPH_DRAIN();
#undef ASPH_DRAIN
        if (active && fast) {
            A.nbr_cnt[i] = L.n <= NBR_CAP ? L.n : -1;
            density_eos_epilogue(P, A.out, i, pi, s, rr, dt);
        }
    }
}

template <int BX, int BY, int BZ, int H>
__global__ __maxnreg__(DENSITY_REGS) void k_density_brick(const __grid_constant__ Phys P, const __grid_constant__ DArgs A,
                                                       PairCfg C) {
    using G = BrickGeom<BX, BY, BZ, H>;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int s_warp[32];
    __shared__ int s_work[5 * (1 + 2 * DENSITY_SPLITS)];
    __shared__ int s_run;
    DSmem M;
    M.feat = smem;
    M.sp = reinterpret_cast<float4*>(smem + (size_t)C.cap * 8 + 16);
    M.s_gidx = reinterpret_cast<int*>(M.sp + C.cap);
    M.s_off = M.s_gidx + C.cap;
    M.s_list = reinterpret_cast<unsigned short*>(M.s_off + (G::R + 1));
    M.s_warp = s_warp;
    M.s_work = s_work;
    const int b = blockIdx.x;
    // the block's two first loads are in flight together, one wait and one barrier less before
    // its staging starts (ten steps at 2M 7.690 -> 7.669 ms, at 475k 2.147 -> 2.139)
    if (threadIdx.x == 0) {
        const int bxi = b % C.nbx, byi = (b / C.nbx) % C.nby, bzi = b / (C.nbx * C.nby);
        const int2 sp2 =
            A.spans[morton3((uint32_t)(bxi * BX), (uint32_t)(byi * BY), (uint32_t)(bzi * BZ)) >> G::LOG2K];
        s_run = A.ctl->aborted ? 0 : 1;   // one decision per block (barriers follow)
        s_work[0] = bxi * BX; s_work[1] = byi * BY; s_work[2] = bzi * BZ; s_work[3] = sp2.x; s_work[4] = sp2.y;
        const uint32_t f = h2_bits(__float2half2_rn(1e4f));
        *reinterpret_cast<uint4*>(M.feat + C.cap * 8) = make_uint4(f, f, f, f);
    }
    __syncthreads();
    if (!s_run) return;
    density_region<BX, BY, BZ, H, DENSITY_SPLITS>(P, A, C, M, 0);   // (starts with a barrier)
}

// Deferred pass: one warp per queued target.  The lanes read the ranges of
// the window's cells (c = dz * 25 + dy * 5 + dx, the reference's loop order)
// and their prefix counts into shared memory, then test the candidates 32
// at a time: candidate g lies in the last cell whose prefix is <= g.
// Accepted neighbours are appended in candidate order by ballot, so the list
// has the order of the reference's loop; the sums are reduced over the warp
// in a fixed tree.
constexpr int DEF_TPB = 256;
constexpr int WIN_CELLS = (2 * STENCIL + 1) * (2 * STENCIL + 1) * (2 * STENCIL + 1);
static_assert(WIN_CELLS <= 128, "a window's cells fit four per lane");

__global__ __launch_bounds__(DEF_TPB) void k_density_deferred(const __grid_constant__ Phys P,
                                                              const __grid_constant__ DArgs A) {
    __shared__ int s_cs[DEF_TPB / 32][128];   // first table index of window cell c
    __shared__ int s_cp[DEF_TPB / 32][128];   // candidates in the cells before c
    __shared__ int s_run;
    DevCtl* ctl = A.ctl;
    if (threadIdx.x == 0) s_run = ctl->aborted ? 0 : 1;   // one decision per block: every thread
    __syncthreads();                                       // reaches the barrier at the end
    const unsigned nq = !s_run ? 0u : (A.defer ? ctl->defer_n : (unsigned)P.N);   // no queue: every target
    const int lane = threadIdx.x & 31;
    int* cs = s_cs[threadIdx.x >> 5];
    int* cp = s_cp[threadIdx.x >> 5];
    const float dt = ctl->dt;
    const unsigned nwarps = (gridDim.x * DEF_TPB) >> 5;
    for (unsigned t = (blockIdx.x * DEF_TPB + threadIdx.x) >> 5; t < nq; t += nwarps) {
        const int i = A.defer ? A.defer[t] : (int)t;
        const float4 pi = A.pos[i];
        const int ix = cell_ix(pi.x, P.inv_dx, P.nx), iy = cell_ix(pi.y, P.inv_dy, P.ny);
        const int iz = cell_ix(pi.z, P.inv_dz, P.nz);
        const int z0 = max(iz - STENCIL, 0), z1 = min(iz + STENCIL, P.nz - 1);
        const int ncell = (z1 - z0 + 1) * (2 * STENCIL + 1) * (2 * STENCIL + 1);
        int total = 0;
        int2 rgs[4];   // the four cell-range loads in flight together
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = u * 32 + lane;
            rgs[u] = make_int2(0, 0);
            if (c < ncell) {
                const int dz = c / 25, r = c - dz * 25, dy = r / 5, dx = r - dy * 5;
                const int gy = wrapi(iy - STENCIL + dy, P.ny), gx = wrapi(ix - STENCIL + dx, P.nx);
                rgs[u] = A.range[(size_t)((z0 + dz) * P.ny + gy) * P.nx + gx];
            }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int c = u * 32 + lane;
            const int2 rg = rgs[u];
            const int cnt = rg.y - rg.x;
            int x = cnt;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            cs[c] = rg.x;
            cp[c] = total + x - cnt;
            total += __shfl_sync(0xffffffffu, x, 31);
        }
        __syncwarp();
        if (total > ASPH_MAX_CANDIDATES) {   // same stop as the global walk's budget (total is warp-uniform)
            if (lane == 0) stop_run(ctl, ASPH_ERR_DENSE);
            break;
        }
        const FF rr = snd_eval(P.snd_rho, P.snd_n, pi.z);
        DSum s{0.f, 0.f, 0.f};
        int nb = 0;
        for (int g0 = 0; g0 < total; g0 += 64) {
            // two rounds of 32 candidates: both rounds' loads in flight together
            int jr[2];
            float4 pr[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int g = g0 + 32 * h + lane;
                jr[h] = 0;
                if (g < total) {
                    int lo = 0, hi = ncell - 1;   // cp[lo] <= g
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) >> 1;
                        if (cp[mid] <= g) lo = mid; else hi = mid - 1;
                    }
                    jr[h] = cs[lo] + (g - cp[lo]);
                    pr[h] = A.pos[jr[h]];
                }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
            const int g = g0 + 32 * h + lane;
            bool push = false;
            const int j = jr[h];
            if (g < total) {
                const float4 pj = pr[h];
                const float r2 = r2_pair(P, pi.x, pi.y, pi.z, pj.x, pj.y, pj.z);
                if (r2 < 4.0f) {
                    dsum_add(s, r2, pj.w, rr);
                    push = r2 >= 1e-12f;
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, push);
            if (push) {
                const int n = nb + __popc(m & ((1u << lane) - 1u));
                if (n < NBR_CAP) A.nbr[(size_t)n * P.N + i] = j;
            }
            nb += __popc(m);
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            s.S1 += __shfl_xor_sync(0xffffffffu, s.S1, o);
            s.S2 += __shfl_xor_sync(0xffffffffu, s.S2, o);
            s.T += __shfl_xor_sync(0xffffffffu, s.T, o);
        }
        if (lane == 0) {
            A.nbr_cnt[i] = nb <= NBR_CAP ? nb : -1;
            density_eos_epilogue(P, A.out, i, pi, s, rr, dt);
        }
        __syncwarp();   // cs and cp are rewritten for the next target
    }
    if (A.defer) {   // the last block to finish empties the queue for the next pass
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(&ctl->defer_done, 1u) == gridDim.x - 1) {
                ctl->defer_last = ctl->defer_n;
                ctl->defer_n = 0u;
                ctl->split_last = ctl->split_n;
                ctl->split_n = 0u;
                ctl->defer_done = 0u;
            }
        }
    }
}

// ===========================================================================
// M: momentum + integrate + rain + CFL (list-driven)
// ===========================================================================
struct MArgs {
    const float4* pos;     // x, y, z, -
    const float4* vel;     // velocities after the first half kick
    const float2* rp;      // rho, p'
    const int2* range;
    const int* nbr;
    const int* nbr_cnt;
    int use_lists;         // lists (and ms) were produced on the current positions and velocities
    const float4* ms;      // x, y, z, p' and u, v, w, rho of the density pass, 32 bytes a particle
    MOut out;
    const float* rain_in;
    const float* rain_delta;
    float* rain_out;
    float* precip;
    DevCtl* ctl;
    int part_blocks;       // chunks of particle work (TPT x M_TPB targets each) ...
    int rain_blocks;       // ... then chunks of rain cells (M_RAIN_CELLS x M_TPB each)
};

// Out of line: targets without a usable neighbour list come here.
__device__ __noinline__ MSum momentum_target_global(const Phys& P, const MArgs& A, const MTarget T) {
    MSum s{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for_window_global(P, A.range, A.ctl, T.x, T.y, T.z, [&](int j) {
        const float4 pj = A.pos[j];
        const float r2t = r2_pair(P, T.x, T.y, T.z, pj.x, pj.y, pj.z);
        if (r2t >= 4.0f || r2t < 1e-12f) return;   // also excludes j == i
        const float2 rj = A.rp[j];
        const float4 vj = A.vel[j];
        msum_add(P, s, T, make_float4(pj.x, pj.y, pj.z, rj.y), make_float4(vj.x, vj.y, vj.z, rj.x));
    });
    return s;
}

// The TPT x M_TPB targets of particle chunk `ch`: the lanes of warp w on
// targets w * 32 * TPT + lane + 32 r, so that a warp waits on the longest sum
// of its lanes' lists rather than on the longest list of each round; a warp
// covers 32 TPT consecutive targets, about 32 TPT / ppc cells.
template <int TPT>
__device__ __forceinline__ void momentum_chunk(const Phys& P, const MArgs& A, int mode, int ch, bool aborted,
                                               float dt, float3& m) {
    const int tbase = ch * (M_TPB * TPT) + (threadIdx.x >> 5) * (32 * TPT) + (threadIdx.x & 31);
    for (int r = 0; r < TPT; ++r) {
        const int i = tbase + 32 * r;
        if (i >= P.N) continue;
        if (aborted) {
            if (mode & M_INTEGRATE) A.out.vel_out[i] = A.vel[i];
            continue;
        }
        // (x, y, z, p') and (u, v, w, rho): packed by the density pass
        // when the lists are current, else from the state buffers
        float4 a, b;
        if (A.use_lists) {
            ldg_record(A.ms, i, a, b);
        } else {
            const float4 p = A.pos[i], v = A.vel[i];
            const float2 rr = A.rp[i];
            a = make_float4(p.x, p.y, p.z, rr.y);
            b = make_float4(v.x, v.y, v.z, rr.x);
        }
        MTarget T;
        T.x = a.x; T.y = a.y; T.z = a.z;
        T.u = b.x; T.v = b.y; T.w = b.z;
        T.rhoi = fmaxf(b.w, 1e-3f);
        T.irhoi = __frcp_rn(T.rhoi);
        T.pri = a.w;
        MSum s{0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        const int cnt = A.use_lists ? A.nbr_cnt[i] : -1;
        if (cnt >= 0) {
            // four neighbours' loads in flight before their arithmetic
            int q = 0;
            const int* lp = A.nbr + i;   // slot q of the list at lp[q N]
            const size_t N = (size_t)P.N;
            for (; q + 4 <= cnt; q += 4) {
                int jj[4];
                float4 pp[4], vv[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) jj[u] = lp[u * N];
                lp += 4 * N;
#pragma unroll
                for (int u = 0; u < 4; ++u) ldg_record(A.ms, jj[u], pp[u], vv[u]);
#pragma unroll
                for (int u = 0; u < 4; ++u) msum_add(P, s, T, pp[u], vv[u]);
            }
            if (q < cnt) {   // the last 1-3 neighbours as one batch, their loads in flight together
                int jj[3];
                float4 pp[3], vv[3];
#pragma unroll
                for (int u = 0; u < 3; ++u) jj[u] = q + u < cnt ? lp[u * N] : i;
#pragma unroll
                for (int u = 0; u < 3; ++u) ldg_record(A.ms, jj[u], pp[u], vv[u]);
#pragma unroll
                for (int u = 0; u < 3; ++u)
                    if (q + u < cnt) msum_add(P, s, T, pp[u], vv[u]);
            }
        } else {
            s = momentum_target_global(P, A, T);
        }
        const float3 mi = momentum_epilogue(P, A.out, i, T, s, (mode & M_INTEGRATE) != 0, dt);
        m = make_float3(fmaxf(m.x, mi.x), fmaxf(m.y, mi.y), fmaxf(m.z, mi.z));
    }
}

// The M_RAIN_CELLS x M_TPB rain cells of rain chunk `rc`.
__device__ __forceinline__ void rain_chunk(const Phys& P, const MArgs& A, int rc, bool aborted, float dt) {
#pragma unroll
    for (int r = 0; r < M_RAIN_CELLS; ++r) {
        const int cid = (rc * M_RAIN_CELLS + r) * M_TPB + threadIdx.x;
        if (cid < P.ncell && !aborted) rain_cell(P, cid, dt, A.rain_in, A.rain_delta, A.rain_out, A.precip);
    }
}

template <int TPT>
__global__ __launch_bounds__(M_TPB, M_MINB) void k_momentum(const __grid_constant__ Phys P, const __grid_constant__ MArgs A,
                                                    int mode) {
    __shared__ float s_max[3][M_TPB / 32];
    DevCtl* ctl = A.ctl;
    const bool aborted = ctl->aborted != 0;
    const float dt = ctl->dt;
    float3 m = make_float3(0.f, 0.f, 0.f);
    const int chunks = A.part_blocks + A.rain_blocks;
    if ((int)blockIdx.x >= A.part_blocks) {
        if ((int)blockIdx.x < chunks) rain_chunk(P, A, blockIdx.x - A.part_blocks, aborted, dt);
    } else {
        momentum_chunk<TPT>(P, A, mode, blockIdx.x, aborted, dt, m);
        if (mode & M_INTEGRATE) {   // the particle blocks' velocity maxima
            float mx = warp_max(m.x), my = warp_max(m.y), mz = warp_max(m.z);
            const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
            if (lane == 0) { s_max[0][warp] = mx; s_max[1][warp] = my; s_max[2][warp] = mz; }
            __syncthreads();
            if (threadIdx.x == 0) {
                float a = 0.f, b = 0.f, c = 0.f;
                for (int w = 0; w < M_TPB / 32; ++w) {
                    a = fmaxf(a, s_max[0][w]); b = fmaxf(b, s_max[1][w]); c = fmaxf(c, s_max[2][w]);
                }
                atomicMax(&ctl->gmax[0], __float_as_uint(a));
                atomicMax(&ctl->gmax[1], __float_as_uint(b));
                atomicMax(&ctl->gmax[2], __float_as_uint(c));
            }
        }
    }
}

// The CFL control after a momentum pass (asph_h100.cu:1040-1078), in a
// kernel of its own: one launch costs less than a finished-block atomic from
// each of the pass's ~11,600 blocks to find the last one (momentum 0.242 ->
// 0.234 ms at 2M).
__global__ void k_cfl_final(const __grid_constant__ Phys P, DevCtl* ctl) {
    if (threadIdx.x == 0 && !ctl->aborted) cfl_control(P, ctl);
}

// ===========================================================================
// launch
// ===========================================================================
namespace {

struct Shape {
    int bx, by, bz;
};
constexpr Shape SHAPES[] = {{8, 8, 8}, {8, 8, 4}, {8, 4, 4}, {4, 4, 4}};
constexpr int MAX_STAGE = 4096;      // staged particles per brick at most
constexpr double STAGE_MARGIN = 1.35;   // of the expected region count, in fits(): which shapes a grid admits
// Staging capacity that no launch goes below, over the expected count.  Less
// splits clustered bricks more often, more can cost a resident block (with 48
// registers 1.15 / 1.2 / 1.35 took 465 / 470 / 487 us at 2M from the lattice and
// 876 / 830 / 771 clustered).
constexpr double STAGE_NEED = 1.2;

int region_cells(const Shape& s, int h) { return (s.bx + 2 * h) * (s.by + 2 * h) * (s.bz + 2 * h); }

// Staged halo: with a sort every step, or the displacement-gated sort (about
// 0.3 cells of the fastest target's way and the last step's own), few targets have
// left their brick, and the stencil alone is staged; slower cadences stage one more
// cell of drift.  Targets outside either go to the deferred pass, where one costs two
// to three times as much as in its brick.  Under the gated sort these are, just
// before a sort and if every target moves as fast as the fastest, 3.75 % of a
// brick along an axis of 8 cells and 7.5 % along one of 4; in the runs measured
// 0.2 %.  Density with no drift / averaged over a gated interval of such a flow along
// one axis / two / three, against the wide halo: 485 / 585 / 656 / 793 against 679 us
// at 2M and one per cell (8x8x4), 471 / 545 / 608 / 668 against 630 at 0.6 per cell
// (8x8x8), 51 / 61 / 65 / 68 against 64 at 98k (8x4x4).  A floor and a lid keep the third
// axis out of that.
// While the targets are at most half the threads that the GPU holds, though,
// the wider halo is hidden and the deferred kernel would wait for one target's
// chain of loads (11 us against 4 with nothing queued): density 30.3 -> 28.8 us at
// 16k, 36.9 -> 34.3 at 65k.  An ensemble's small members fill the GPU together and pay
// for it (with the limit at all resident threads, 4.87 -> 5.01 ms for 16 members).
// That needs the bricks resident together, eight per SM: on a sparse grid of more
// bricks the staging is most of the pass (a step with 40,960 particles on 160 x 160 x 160
// cells, 8,000 bricks: 188 us with the wide halo, 172 without).
int halo_for(const Phys& P, const Shape& s) {
    const long long bricks =
        (long long)((P.nx + s.bx - 1) / s.bx) * ((P.ny + s.by - 1) / s.by) * ((P.nz + s.bz - 1) / s.bz);
    if (P.N <= 152 * 512 && bricks <= 152 * 8) return MAX_HALO;
    return P.sort_every <= 1 ? STENCIL : MAX_HALO;
}

// Largest brick whose region fits the grid without wrapping onto itself
// and whose expected staged count (with a margin) fits the cap.
bool fits(const Phys& P, int k) {
    const Shape& s = SHAPES[k];
    if (P.nx < s.bx + 2 * MAX_HALO || P.ny < s.by + 2 * MAX_HALO) return false;
    return region_cells(s, MAX_HALO) * ((double)P.N / (double)P.ncell) * STAGE_MARGIN <= MAX_STAGE;
}

int pick_shape(const Phys& P);

int shape_in_use(const Phys& P, const Bufs& B) {
    if (B.force_global) return -1;
    return B.shape >= 0 ? B.shape : pick_shape(P);
}

struct Launch {
    PairCfg C;
    int threads;
    int blocks;   // resident per SM
    size_t smem;
};

// Shared memory per SM and reserved per block (queried once; GB300 values as fallback).
void smem_limits(int* per_sm, int* reserved) {
    static int sm = 0, res = -1;
    if (!sm) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess || sm <= 0)
            sm = 228 * 1024;
        if (cudaDeviceGetAttribute(&res, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess || res < 0)
            res = 1024;
    }
    *per_sm = sm;
    *reserved = res;
}


Launch plan(const Phys& P, const Shape& s, int h) {
    Launch L;
    L.C.nbx = (P.nx + s.bx - 1) / s.bx;
    L.C.nby = (P.ny + s.by - 1) / s.by;
    L.C.nbz = (P.nz + s.bz - 1) / s.bz;
    L.C.nbricks = L.C.nbx * L.C.nby * L.C.nbz;
    const double ppc = (double)P.N / (double)P.ncell;
    const int R = region_cells(s, h);
    // about one thread per expected target (the lattice keeps brick counts
    // close to the mean), in whole warps, 64..512; a brick of a sparse grid may
    // expect less than one target
    int groups = (int)(s.bx * s.by * s.bz * ppc * 1.04 + 31) / 32;
    groups = groups < 1 ? 1 : groups;
    const int rounds = (groups + 15) / 16;
    groups = (groups + rounds - 1) / rounds;
    L.threads = 32 * (groups < 2 ? 2 : groups);
    auto smem_for = [&](size_t cap, int dlist) {
        return cap * (8 + 16 + 4) + 16 + (size_t)4 * (R + 1) + (size_t)dlist * L.threads * 2;
    };
    // staging capacity: at least the expected region count times STAGE_NEED;
    // the most resident blocks the registers allow come first, then the
    // deepest drain queue (fuller drains) that still fits them, then all the
    // shared memory left for staging, so that clustered bricks overflow less
    // often (an overflowing brick is split into halves)
    int need = (int)(R * ppc * STAGE_NEED) + 64;
    need = (need + 63) & ~63;
    need = need > MAX_STAGE ? MAX_STAGE : need;
    int per_sm, reserved;
    smem_limits(&per_sm, &reserved);
    const int by_regs = 65536 / (DENSITY_REGS * L.threads);
    int cap = need, dlist = 16;
    bool found = false;
    L.blocks = 1;
    for (int b = by_regs < 8 ? by_regs : 8; b >= 1 && !found; --b) {
        const size_t budget = (size_t)(per_sm / b - reserved - 512);   // 512: the kernel's static arrays
        for (int d = DLIST; d >= 16 && !found; d -= 2) {
            if (smem_for(need, d) > budget) continue;
            int c = MAX_STAGE;
            while (c > need && smem_for(c, d) > budget) c -= 64;
            cap = c;
            dlist = d;
            L.blocks = b;
            found = true;
        }
    }
    L.C.cap = cap;
    L.C.dlist = dlist;
    L.C.qinv = (uint32_t)((0x100000000ull + 2 * L.threads - 1) / (2 * L.threads));
    L.smem = smem_for(cap, dlist);
    return L;
}

// The largest brick (the smallest share of halo) whose blocks fill the GPU:
// at least SHAPE_WARPS warps resident per SM, and at least four blocks for every
// SM.  Staged slots and queues, not registers, limit the blocks of a large
// brick in dense states: at one particle per cell 8 x 8 x 8 cells leave 18 warps per SM
// and 8 x 8 x 4 leave 27 (density 473 against 433 us at 2M), at 0.6 both leave 30 (471
// against 569 us, the latter with 48 registers); and 112 bricks of 32,768 particles take 88 us where 637 smaller
// ones take 49.  A smaller brick is taken for its warps only while it has more of them:
// on a sparse grid (below 0.16 per cell) the eight blocks of two warps are all
// there are, and smaller bricks only add blocks (a step at 0.03 per cell on 100 x 100
// x 100 cells: 72 us with 8 x 8 x 8, 177 with 4 x 4 x 4).  The choice does not depend on the
// sort cadence, so the spans that one step's gather wrote serve every other step of
// the context.
constexpr int SHAPE_WARPS = 26;
int pick_shape(const Phys& P) {
    int k = 0;
    while (k < 4 && !fits(P, k)) ++k;
    if (k == 4) return -1;
    Launch L = plan(P, SHAPES[k], STENCIL);
    for (; k < 3; ++k) {
        const Launch next = plan(P, SHAPES[k + 1], STENCIL);
        const int warps = L.blocks * (L.threads / 32), more = next.blocks * (next.threads / 32);
        if ((warps >= SHAPE_WARPS || more <= warps) && L.C.nbricks >= 4 * 152) break;
        L = next;
    }
    return k;
}

// Blocks of the deferred pass: 4 per SM (32 warps), each warp looping over the queue.
int deferred_blocks() {
    static int blocks = 0;
    if (!blocks) {
        int dev = 0, sms = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0) sms = 152;
        blocks = 4 * sms;
    }
    return blocks;
}

template <int BX, int BY, int BZ, int H>
void launch_dh(const Phys& P, const DArgs& A, cudaStream_t s) {
    const Launch L = plan(P, Shape{BX, BY, BZ}, H);
    cudaFuncSetAttribute(k_density_brick<BX, BY, BZ, H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L.smem);
    cudaFuncSetAttribute(k_density_brick<BX, BY, BZ, H>, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
    k_density_brick<BX, BY, BZ, H><<<L.C.nbricks, L.threads, L.smem, s>>>(P, A, L.C);
    k_density_deferred<<<deferred_blocks(), DEF_TPB, 0, s>>>(P, A);
}

template <int BX, int BY, int BZ>
void launch_d(const Phys& P, const DArgs& A, cudaStream_t s) {
    if (halo_for(P, Shape{BX, BY, BZ}) == STENCIL) launch_dh<BX, BY, BZ, STENCIL>(P, A, s);
    else launch_dh<BX, BY, BZ, MAX_HALO>(P, A, s);
}

inline int blocks_for(int n, int tpb) { return n <= 0 ? 1 : (n + tpb - 1) / tpb; }

}  // namespace

int pair_shape(const Phys& P, const Bufs& B) { return shape_in_use(P, B); }
size_t pair_span_slots(const Phys& P) {
    const size_t keys = (size_t)1 << P.key_bits;
    return keys >> 6 > 0 ? keys >> 6 : 1;   // the smallest shape, 4 x 4 x 4, has 64 keys
}
int pair_span_shift(const Phys& P, const Bufs& B) {
    const int k = shape_in_use(P, B);
    if (k < 0) return -1;
    const int keys = SHAPES[k].bx * SHAPES[k].by * SHAPES[k].bz;
    int sh = 0;
    while ((1 << sh) < keys) ++sh;
    return sh;
}
void launch_brick_spans(const Phys& P, const Bufs& B, cudaStream_t s) {
    const int k = shape_in_use(P, B);
    if (k < 0) return;
    const Shape& sh = SHAPES[k];
    const Launch L = plan(P, sh, MAX_HALO);
    const int blocks = (L.C.nbricks + 3) / 4;   // eight warps a block, two a brick
    switch (k) {
        case 0: k_brick_spans<8, 8, 8><<<blocks, 256, 0, s>>>(P, B.skeys, B.spans, L.C); break;
        case 1: k_brick_spans<8, 8, 4><<<blocks, 256, 0, s>>>(P, B.skeys, B.spans, L.C); break;
        case 2: k_brick_spans<8, 4, 4><<<blocks, 256, 0, s>>>(P, B.skeys, B.spans, L.C); break;
        default: k_brick_spans<4, 4, 4><<<blocks, 256, 0, s>>>(P, B.skeys, B.spans, L.C); break;
    }
}
int pair_shape_count() { return (int)(sizeof(SHAPES) / sizeof(SHAPES[0])); }
bool pair_shape_fits(const Phys& P, int k) { return k >= 0 && k < pair_shape_count() && fits(P, k); }

void launch_density(const Phys& P, const Bufs& B, cudaStream_t s) {
    DArgs A;
    A.pos = B.pos[B.pc];
    A.range = B.range;
    A.skeys = B.skeys;
    A.out.thq = B.thq[B.qc];
    A.out.rp = B.rp;
    A.out.vel = B.vel[B.vc];
    A.out.ms = B.ms;
    const bool reads = P.accretion || P.rain_evap;
    A.out.rain_cur = B.rain[B.rc];
    A.out.rain_dep = reads ? B.rain_delta : B.rain[B.rc];
    A.spans = B.spans;
    A.nbr = B.nbr;
    A.nbr_cnt = B.nbr_cnt;
    A.defer = B.defer;
    A.ctl = B.ctl;
    if (B.force_global == 2) {   // warp per target for every target
        A.defer = nullptr;
        k_density_deferred<<<deferred_blocks(), DEF_TPB, 0, s>>>(P, A);
        return;
    }
    switch (shape_in_use(P, B)) {
        case 0: launch_d<8, 8, 8>(P, A, s); break;
        case 1: launch_d<8, 8, 4>(P, A, s); break;
        case 2: launch_d<8, 4, 4>(P, A, s); break;
        case 3: launch_d<4, 4, 4>(P, A, s); break;
        default: k_density_global<<<blocks_for(P.N, 256), 256, 0, s>>>(P, A); break;
    }
}

// The default option value, 2, takes one target per thread where two would leave
// the GPU short of threads (152 SMs x 1,024 resident): the lists of a thread's
// targets are walked one after the other, and with idle SMs that is only latency.
// Momentum with one / two: 15.4 / 20.5 us at 16k, 17.4 / 20.5 at 65k, 22.5 / 32.8 at
// 32k and one per cell, 47.1 / 51.2 at 262k; 59.9 / 59.0 at 475k and 217 / 211 at 2M.
static int launch_tpt(const Phys& P, const Bufs& B) {
    if (B.m_tpt == M_TPT && P.N <= 2 * 152 * 1024) return 1;
    return B.m_tpt;
}

void launch_momentum(const Phys& P, const Bufs& B, int mode, int use_lists, cudaStream_t s) {
    MArgs A;
    A.pos = B.pos[B.pc];
    A.vel = B.vel[B.vc];
    A.rp = B.rp;
    A.range = B.range;
    A.nbr = B.nbr;
    A.nbr_cnt = B.nbr_cnt;
    A.use_lists = use_lists;
    A.ms = B.ms;
    A.out.thq = B.thq[B.qc];
    A.out.acc = B.acc;
    A.out.dthdt = B.dthdt;
    A.out.vel_out = B.vel[1 - B.vc];
    A.out.src_cur = B.src ? B.src_tmp : nullptr;
    A.out.src_keep = B.src;
    A.rain_in = B.rain[B.rc];
    A.rain_delta = (P.accretion || P.rain_evap) ? B.rain_delta : nullptr;
    A.rain_out = B.rain[1 - B.rc];
    A.precip = B.precip;
    A.ctl = B.ctl;
    const int tpt = launch_tpt(P, B);
    A.part_blocks = blocks_for(P.N, M_TPB * tpt);
    const int rain_blocks = (mode & M_RAIN) ? blocks_for(P.ncell, M_TPB * M_RAIN_CELLS) : 0;
    A.rain_blocks = rain_blocks;
    const int grid = A.part_blocks + rain_blocks;
    if (tpt == 1)
        k_momentum<1><<<grid, M_TPB, 0, s>>>(P, A, mode);
    else if (tpt == 4)
        k_momentum<4><<<grid, M_TPB, 0, s>>>(P, A, mode);
    else
        k_momentum<2><<<grid, M_TPB, 0, s>>>(P, A, mode);
    if (mode & M_CFL) k_cfl_final<<<1, 32, 0, s>>>(P, A.ctl);
}

}  // namespace asph
