// Host interface of the on-chip multi-step kernel (lbm_resident.cu).
#pragma once
#include <cuda_runtime.h>

#include "lbm_bc.cuh"
#include "lbm_step.cuh"

namespace lbm {

// How a 2D lattice is cut into one tile per block: gx x gy tiles, `compute`
// threads that update nodes and `comm` threads that exchange tile edges, over
// at most `links` links out of a tile.
struct ResidentPlan {
    int gx = 0, gy = 0, compute = 0, comm = 0, links = 0;
    size_t smem = 0;
    int tiles() const { return gx * gy; }
    size_t messages() const { return (size_t)2 * tiles() * links; }
};
constexpr int RESIDENT_PLANS = 4;

struct ResidentArgs {
    StepParams p, last;       // fin: the state at entry, fout: where it goes; last: with write_macro as asked
    int steps, gx, gy, compute, links;
    int wrap;                 // links leave the lattice by wrapping round
    unsigned tag;             // messages of this launch carry tag + 1 .. tag + steps - 1
    unsigned long long *mail; // [2][tile][links] messages
    unsigned polls;           // of a message after the first, before its wait gives up
    unsigned *err;            // set when a wait gave up
};

constexpr unsigned RESIDENT_POLLS = 1u << 22;  // seconds

// A plan for an nx x ny lattice of `elem`-byte populations, or false where
// the lattice does not fit on chip.
bool resident_plan(int nx, int ny, int elem, int sms, ResidentPlan *out);
// The kernel for a collision model, storage and mode allowed its shared
// memory; null where there is none, or where a block of `plan` does not fit.
const void *resident_prepare(int coll, int st, int phys, const ResidentPlan &plan);
int resident_launch(const void *kern, const ResidentPlan &plan, const ResidentArgs &a, cudaStream_t s);

}  // namespace lbm
