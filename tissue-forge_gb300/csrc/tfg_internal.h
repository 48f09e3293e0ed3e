// Host-side engine state and kernel launch entry points shared by the CUDA translation units.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <string>
#include <vector>

#include "tfg.h"
#include "tfg_device.cuh"

namespace tfg {

// Per-particle device state, stored in cell order.  Two copies exist so the counting
// sort can scatter from one into the other.
struct ParticleArrays {
    float4 *pos = nullptr;     // cell-relative x,y,z ; w = type (int bits)
    float4 *vel = nullptr;     // v.x,v.y,v.z ; w = inverse number density
    float4 *aux = nullptr;     // radius, imass, flags (bits), id (bits)
    float4 *fext = nullptr;    // force_i (external) ; w unused
    float4 *pforce = nullptr;  // persistent random force ; w unused
    int32_t *cell = nullptr;   // cell index of each slot
    float *sval = nullptr;     // species values, [s * cap + slot]
    float *sq = nullptr;       // flux increments, [s * cap + slot]
};

// Launch a kernel that begins with step_kernel_begin(): its blocks may be set up while the
// kernel before it still runs (programmatic dependent launch, in graphs too).
template <typename... P, typename... A>
inline void launch_step_kernel(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// A kernel's set-up, made once on each device that it is launched on: function attributes and
// occupancy are a device's.  make() returns a positive number that is kept (resident warps, say),
// or 0 after an error, which the check of the launch reports; it may run twice when two threads
// are first at once.
class PerDevice {
public:
    template <class F> int get(F make) {
        int d = 0;
        if (cudaGetDevice(&d) != cudaSuccess || d < 0 || d >= kDevices) return make();
        int n = kept[d].load(std::memory_order_relaxed);
        if (n == 0) kept[d].store(n = make(), std::memory_order_relaxed);
        return n;
    }

private:
    static constexpr int kDevices = 64;
    std::atomic<int> kept[kDevices] = {};
};

// Reduction slots in the device double array.
enum RedSlot : int {
    RED_EPOT_NONBOND = 0,
    RED_EPOT_BOND,
    RED_EPOT_ANGLE,
    RED_KINETIC,
    RED_VIRIAL,
    RED_VOLUME,
    RED_MIGRATIONS,
    RED_SPECIES0,               // kMaxSpecies entries
    RED_COUNT = RED_SPECIES0 + kMaxSpecies,
};

struct PairKernelArgs {
    const SimParams *sims;      // per-simulation parameters (device)
    const int32_t *cell_sim;    // simulation of each global cell (device)
    const int4 *cell_at;        // grid location of each global cell; w: its simulation
    int nsims;
    int ncells;                 // global cells over all simulations
    int max_type;               // types per simulation (tables are max_type^2 per simulation)
    int nspec;                  // species per particle (all simulations)
    uint32_t flags;             // union of the simulations' TFG_ENGINE_* flags
    int n;
    const float4 *pos;
    const float4 *vel;
    const float4 *aux;
    const float4 *fext;
    const float4 *pforce;
    const int32_t *cell;
    const int32_t *start;       // ncells+1
    const int2 *items;          // work items of the tiled pass: (first cell of a run of up to four along z, first of up
                                // to `homes` home particles | cells - 1 << 30)
    const int *nitems;
    int homes;                  // 8, 16 or 32
    bool runs;                  // items may span several cells
    unsigned long long *stamp;  // where the pass's begin is stamped, or null
    unsigned *counter;          // work counter of the tiled pass and its finished blocks
    const float *sval;
    float *sq;
    int cap;
    float4 *force;              // out: f.xyz, number density
    const PotDev *pots;         // nsims * max_type^2
    const PotPair *potc;        // the same, compact (tiled pass)
    const float *blob;
    cudaTextureObject_t potc_tex, blob_tex;   // potc and blob as textures of 16 bytes a texel, or 0
    PotPair one;                // the entries that all of potc's and fluxes' are equal to
    FluxSet one_flux;
    bool has_one;               // there are such
    int blob_floats;
    const PotDev *wpots;        // nsims * 6 * max_type wall potentials
    bool has_wall_pots;         // any simulation has a wall potential
    const FluxSet *fluxes;      // nsims * max_type^2
    const float4 *rforce;       // nsims * max_type: mean, std, duration, enabled
    float4 *pforce_out;         // persistent force updated in place (same as pforce)
    double *red;                // RED_COUNT per simulation
    uint32_t *err;
    int32_t *sig_count;         // signature mode: interacting neighbours per particle
    uint32_t *sig_hash;         // signature mode: order-independent hash of neighbour ids
    int32_t *pair_out;          // signature mode, optional: (lower id, higher id) of each pair found
    unsigned long long *pair_n; // pairs found (the first pair_cap are written)
    long long pair_cap;
    int flux_sub;               // >= 0: flux-only substep pass number (simulations with
                                // nr_fluxsteps - 1 > flux_sub take part); -1: the full pass
    bool has_dpd;               // any type pair uses a DPD potential
    bool radii;                 // any table is shifted or scaled by the particles' radii
    bool has_flux;              // any type pair has fluxes
};

// Full-stencil kernel: one thread per particle, no atomics.  General path (any number
// of species); force[] must hold the initial force (external + random, density W(0)).
void launch_pair(const PairKernelArgs &a, cudaStream_t s);
// Launch configuration of the nonbonded pass: the work split picked by the autotuner (warps
// per home cell: 1, 2, 7 or 14; the cell's 14 tasks are divided into that many work items;
// TFG_PAIR_HOME_OUTER means 1), the warps per CTA (4 or 8; 0: by the size of the work items),
// and the fewest work items a warp takes from the shared counter at a time.
struct TileTune {
    int split = 1;
    int warps = 0;
    int grab = 1;
};
// Warps per CTA of the tiled pass.  CTAs of four end more evenly where a warp has few items: 76.7 ->
// 74.6 us a step of 100,000 DPD particles, 70.4 -> 69.3 of 80,000 cells; CTAs of eight share more
// in L1: 703 us a step of 1,953,125 Lennard-Jones particles, 709 with four.
inline int cta_warps(const TileTune &t, int homes) { return t.warps ? t.warps : (homes < 32 ? 4 : 8); }
// Tiled half-shell kernel; force[] must hold the initial force, to which both partners'
// contributions are added atomically.
void launch_pair_tile(const PairKernelArgs &a, int sms, bool signature, const TileTune &tune, cudaStream_t s);
void launch_pair_stencil_fluxonly(const PairKernelArgs &a, cudaStream_t s);
// Flux-only substep pass (a.flux_sub >= 0): species flux increments of the pair set, no
// forces, densities or energies (runner_dopair_fluxonly / runner_doself_fluxonly).
void launch_pair_fluxonly(const PairKernelArgs &a, int sms, bool tile, cudaStream_t s);
// Same stencil walk and pair decision as launch_pair, writing only the per-particle
// pair signature (used to prove the pair set bit-exact against the oracle).
void launch_pair_signature(const PairKernelArgs &a, cudaStream_t s);

// Signature mode with an explicit list: append the pair (ida, idb) once.
__device__ __forceinline__ void record_pair(const PairKernelArgs &a, int ida, int idb) {
    if (!a.pair_out) return;
    const unsigned long long p = atomicAdd(a.pair_n, 1ull);
    if ((long long)p < a.pair_cap) {
        a.pair_out[2 * p] = ida < idb ? ida : idb;
        a.pair_out[2 * p + 1] = ida < idb ? idb : ida;
    }
}

// Hash of one neighbour id for the pair signature.
__host__ __device__ inline uint32_t sig_mix(uint32_t id) {
    uint32_t x = id * 2654435761u + 0x9E3779B9u;
    x ^= x >> 15;
    x *= 0x85EBCA6Bu;
    x ^= x >> 13;
    return x;
}

}  // namespace tfg
