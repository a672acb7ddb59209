// The batched cavities' device structures and launchers, for the host code and
// the units that define them.  The launchers are only declared here: a unit that
// sees their bodies compiles the kernels once more, with its own floating-point
// flags, and which of the copies a process runs is not defined.
#pragma once

#include "batch_plan.h"
#include "kernels.cuh"

namespace mplb {

struct BatchCav {
    long long base;    // element offset of the cavity in a population array
    long long mbase;   // offset of its nodes in the macro arrays
    int n;             // nodes per side
    int pad;
    double omc;        // 1 - omega of this cavity
    double dt;         // MPLB time step (residual normalisation)
    float omcf;
    float ninv;        // 1 / n (row of node k: (k + 1/2) / n rounded down)
    double lidb[9];    // 2 w_i (c_i . u_lid) for populations bounced at the lid
    float lidbf[9];
};

struct BatchDev {
    const BatchCav* cavs;
    // active tiles: (cavity, first node, nodes per side, element offset of
    // the cavity in 128-byte units), so a tile's population addresses wait
    // on the tile's own load alone and the cavity's constants load beside
    // the populations
    const int4* tiles;
    const int* ntiles;      // number of active tiles (device word)
    int tile_nodes;         // nodes per tile
    double* macro[3];       // rho, u, v of every cavity, packed
    double* macro_old[3];
};

struct GridSync {           // bounded grid-wide barrier state
    unsigned* count;
    unsigned* gen;
    int* err;               // set to 1 when a wait gives up
    long long limit;        // polls before giving up
};

#ifndef MPLB_BATCH_GROUP
#define MPLB_BATCH_GROUP 2
#endif

// Nodes per thread of the step kernels (threads per CTA = tile nodes / this):
// MPLB_BATCH_GROUP in the FP32 form, one in FP64.
template <typename T>
__host__ __device__ constexpr int BatchNodesPerThread() {
    return sizeof(T) < 8 ? MPLB_BATCH_GROUP : 1;
}

// Per active tile: sum (q - q_old)^2 and sum q^2 of rho, u, v; q_old <- q.
__global__ void BatchResidualPartialKernel(BatchDev bd,
                                           double* __restrict__ part);

// Per active cavity c (CTA c): sums its tiles' partials in order and writes
// max_q [sum (q - q_old)^2 / sum q^2] / (check_period dt) (the reference's
// CalcResidualError + GetMaximumResidual on one cavity).
__global__ void BatchResidualFinalKernel(BatchDev bd,
                                         const double* __restrict__ part,
                                         const int4* __restrict__ ranges,
                                         int ncav, int check_period,
                                         double* __restrict__ res);

// Instantiated with the FP64 and the FP32 forms, each in the unit with its
// floating-point contraction rules.
template <typename T>
struct BatchLaunch {
    static cudaError_t Step(bool macro, int grid, int threads, cudaStream_t s,
                            const BatchDev& bd, const PhysConst& pc, int nt,
                            const T* src, T* dst);
    static cudaError_t Persistent(int grid, int threads, cudaStream_t s,
                                  const BatchDev& bd, const PhysConst& pc,
                                  T* a, T* b, int nsteps, int macro_last,
                                  const GridSync& gs);
    static cudaError_t MaxCoResident(int threads, int* per_sm);
    static cudaError_t Init(int grid, int threads, cudaStream_t s,
                            const BatchDev& bd, const PhysConst& pc,
                            const int4* alltiles, int ntiles, T* a);
};

template <typename T>
struct BatchResidentLaunch {
    // `halves`: the CTAs' slots fill 1 / 2^halves of an SM.
    static cudaError_t Run(int halves, int ranks, int warps, int nitems,
                           cudaStream_t s, const BatchDev& bd,
                           const PhysConst& pc, const ResidentItem* items,
                           int steps, bool macro, const T* src, T* dst);
    // Whether the device can hold a cluster of `ranks` such CTAs.
    static bool Held(int halves, int ranks);
};

}  // namespace mplb
