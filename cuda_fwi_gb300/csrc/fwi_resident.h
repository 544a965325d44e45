// fwi_resident.h -- what the engine needs of the resident kernels (fwi_resident.cuh).
#pragma once

#include "fwi_kernels.cuh"

namespace fwi {

constexpr int kResThreads = 512;
constexpr int kResTX = 64;        // largest tile width (columns)
constexpr int kResSmem = 232448;  // dynamic shared memory a launch may use

constexpr int kResMore = 1 << 30;

// One entry of the program a launch runs.  ADV: forward steps a..b-1 (flags of
// FL_STORE on sampled steps, FL_WE, FL_RECORD); SAVE / RESTORE: the forward
// state to / from checkpoint slot a (-1: the zero state); ADJ: adjoint steps
// b-1 down to a (FL_GRAD on sampled steps); FINAL: the state of simulation a
// (0 forward, 1 adjoint) to its global arrays.
struct ResOp {
    int kind, a, b, flags;
};
enum { RES_ADV = 0, RES_SAVE = 1, RES_RESTORE = 2, RES_ADJ = 3, RES_FINAL = 4 };

// Simulations a launch keeps in shared memory.
enum { RES_FORWARD = 0, RES_STORED = 1, RES_BOTH = 2 };  // forward; adjoint over a stored wavefield; both

// Tiling of one shot's grid, and what its tiles hold at most.
struct ResTiling {
    int ntx, ntz;  // tiles
    int tzm;       // rows
    int sxp, szr;  // column pairs and rows inside CPML strips
};

struct ResArgs {
    // descriptors of the launch's first shot (forward, adjoint): the geometry is
    // every shot's, its arrays follow at the strides below
    ItemDesc f, a;
    long long state, field, xstrip, zstrip, nf, nft;
    ResTiling t;
    // layout of shared memory (floats): first simulation, size of one, materials,
    // x- and z-strip memories in a simulation
    int fields, sim, mat, xs, zs;
    int iw;                     // inbox words
    int nops;
    const ResOp* ops;
    const int *evo_f, *evo_a;   // per tile, offsets into the event lists (tiles + 1)
    const int2 *ev_f, *ev_a;    // (shared-memory cell, code): injections of a cell before its recordings;
                                // kResMore marks an event whose predecessor has the same cell
    unsigned long long* inbox;  // [tile][simulation][pass][inbox words]
    float* snap;                // checkpoint slots, first shot of the launch
    long long slot_stride;
    unsigned tag0;              // tags of earlier launches are <= tag0
    float one;                  // 1.0f (a multiplier the compiler cannot see)
    int stall;                  // test hook: CTA 0 leaves at once, so its neighbours' polls run out
    int* err;
    unsigned long long wait_ns;
};

// Tile t of n over `total` rows or column pairs: [lo, hi), sizes differing by at most one.
__host__ __device__ inline int res_cut(int total, int n, int t) { return (int)((long long)total * t / n); }

// Column pairs of a grid (from the even column at or below FP) and first grid
// rows / columns of the strips: strip columns are those < res_left and >=
// res_right, strip rows those < res_top and >= res_bottom (index npml of the
// tables is the identity and counts as outside).
__host__ __device__ inline int res_xb(int fp) { return fp & ~1; }
__host__ __device__ inline int res_pairs(int nxt, int fp) { return (nxt - fp - res_xb(fp) + 1) / 2; }
struct ResStrips {
    int left, right, top, bottom;
};
__host__ __device__ inline ResStrips res_strips(int nzt, int nxt, int ppad, int npml, int fsurf) {
    if (npml <= 0) return {0, nxt, 0, nzt};
    return {ppad, nxt - ppad, fsurf ? 0 : ppad, fsurf ? nzt - ppad - 1 : nzt - ppad};
}

// The resident kernels of one half order.
struct ResSet {
    cudaError_t (*prepare)();  // opt in to the dynamic shared memory
    // cooperative launch; fills in the shared-memory layout of `a`
    cudaError_t (*launch)(int mode, int ctas, cudaStream_t s, ResArgs a);
    size_t (*smem)(const ResTiling& t, int tp, int mode);  // dynamic shared memory of a launch
    int (*inbox_words)(int tzm);                           // 8-byte words per tile, simulation and pass
    int pitch;                                             // row pitch of a tile in shared memory
};
ResSet resident_for(int fp);

// First out-of-range access that a resident kernel recorded (bounds-checked
// build; 0: none), cleared by the call.
cudaError_t resident_bounds_record(unsigned long long* v);

}  // namespace fwi
