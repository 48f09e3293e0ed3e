// Per-particle, per-cell, per-bond and per-angle kernels of the engine (everything but
// the pair pass).  Every kernel serves an arena of one or more simulations: a particle's
// simulation is cell_sim[cell], and its parameters are sims[that index].
//
//   bin      space_shuffle_local re-check (tfSpace.cpp:274-391) + counting sort into
//            cell order (count, scan, place, rank by id, scatter)
//   scatter  also initialises the pair pass's force: force_i + Gaussian persistent force
//            (gaussian_force, tfForce.cpp:211-223) and W(0) (space_prepare, tfSpace.cpp:182-201)
//   bonded   bond_eval / angle_eval (tfBond.cpp:97-345, tfAngle.cpp:90-382)
//   advance  cell_advance_forward_euler + Fluxes_integrate (tf_engine_advance.cpp:140-247,
//            tfFlux.cpp:175-202) with FP64 per-simulation totals
#include "tfg_kernels.h"

namespace tfg {

namespace {

// Simulation of cell c.  With one simulation there is nothing to look up, and its parameters do
// not wait for the particle's cell.
__device__ __forceinline__ int sim_of(int nsims, const int32_t *cell_sim, int c) { return nsims == 1 ? 0 : cell_sim[c]; }

__device__ __forceinline__ int wrap_shift(int s) { return s > 1 ? -1 : (s < -1 ? 1 : s); }

// Add per-thread partials (FP32, or FP64 of several terms) into per-simulation FP64 totals.  When
// the whole block belongs to one simulation: the partials' type over each warp, FP64 across
// warps, one atomic per block.  Otherwise each warp whose lanes share a simulation adds once, and mixed warps
// add lane by lane.  Every thread of the block must call it.
template <class T> __device__ __forceinline__ void keyed_add(double *red, int rb, int slot, T v) {
    __shared__ double part[32];
    const int rb0 = __shfl_sync(0xffffffffu, rb, 0);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __shared__ int block_rb;
    if (threadIdx.x == 0) block_rb = rb;
    __syncthreads();
    const bool uniform = __syncthreads_and(rb == block_rb || rb < 0);
    if (uniform) {
        T s = v;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) part[w] = (double)s;
        __syncthreads();
        if (threadIdx.x == 0 && block_rb >= 0) {
            double t = 0.0;
            for (int k = 0; k < nw; k++) t += part[k];
            if (t != 0.0) atomicAdd(&red[block_rb + slot], t);
        }
        __syncthreads();
        return;
    }
    if (__all_sync(0xffffffffu, rb == rb0 || rb < 0)) {
        T s = v;
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0 && rb0 >= 0 && s != T(0)) atomicAdd(&red[rb0 + slot], (double)s);
    } else if (rb >= 0 && v != T(0)) {
        atomicAdd(&red[rb + slot], (double)v);
    }
}

// keyed_add of three values to three slots of the same simulation, under one set of block
// barriers.
template <class T>
__device__ __forceinline__ void keyed_add3(double *red, int rb, int s0, T v0, int s1, T v1, int s2, T v2) {
    __shared__ double part3[3][32];
    const int rb0 = __shfl_sync(0xffffffffu, rb, 0);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    __shared__ int block_rb3;
    if (threadIdx.x == 0) block_rb3 = rb;
    __syncthreads();
    const bool uniform = __syncthreads_and(rb == block_rb3 || rb < 0);
    T a = v0, b = v1, c = v2;
    if (uniform || __all_sync(0xffffffffu, rb == rb0 || rb < 0)) {
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_down_sync(0xffffffffu, a, o);
            b += __shfl_down_sync(0xffffffffu, b, o);
            c += __shfl_down_sync(0xffffffffu, c, o);
        }
    }
    if (uniform) {
        if (lane == 0) {
            part3[0][w] = (double)a;
            part3[1][w] = (double)b;
            part3[2][w] = (double)c;
        }
        __syncthreads();
        if (threadIdx.x < 3 && block_rb3 >= 0) {
            double t = 0.0;
            for (int k = 0; k < nw; k++) t += part3[threadIdx.x][k];
            const int slot = threadIdx.x == 0 ? s0 : (threadIdx.x == 1 ? s1 : s2);
            if (t != 0.0) atomicAdd(&red[block_rb3 + slot], t);
        }
        __syncthreads();
        return;
    }
    if (__all_sync(0xffffffffu, rb == rb0 || rb < 0)) {
        if (lane == 0 && rb0 >= 0) {
            if (a != T(0)) atomicAdd(&red[rb0 + s0], (double)a);
            if (b != T(0)) atomicAdd(&red[rb0 + s1], (double)b);
            if (c != T(0)) atomicAdd(&red[rb0 + s2], (double)c);
        }
    } else if (rb >= 0) {
        if (v0 != T(0)) atomicAdd(&red[rb + s0], (double)v0);
        if (v1 != T(0)) atomicAdd(&red[rb + s1], (double)v1);
        if (v2 != T(0)) atomicAdd(&red[rb + s2], (double)v2);
    }
}

__global__ void k_stamp(unsigned long long *t, int k) {
    t[k] = global_timer();
}

// One step's start for a simulation: stop it if it has reached its stop time, else advance its
// clock (time += 1, engine_step, tfEngine.cpp:1387) and clear its FP64 totals (a stopped
// simulation keeps the totals of its last step).  In Verlet mode, the rebuild decision of
// engine_verlet_update (tfEngine.cpp:234-290): rebuild when 2 * maxdx > skin, maxdx being the
// largest displacement since the last rebuild, measured after the previous advance.
__device__ __forceinline__ bool stops_now(const SimParams &P) { return P.stop_at >= 0 && P.time >= P.stop_at; }
__device__ __forceinline__ bool rebuilds_now(const SimParams &P) {
    return P.verlet_rebuild == 2 || __fmul_rn(2.0f, __fsqrt_rn(__uint_as_float(P.verlet_maxdx2))) > P.skin;
}
__device__ __forceinline__ void tick(SimParams &P, double *red) {
    if (stops_now(P)) {
        P.stopped = 1;
        if (P.verlet_rebuild == 1) P.verlet_rebuild = 0;
        return;
    }
    P.stopped = 0;
    P.time += 1;
    for (int r = 0; r < RED_COUNT; r++) red[P.red_base + r] = 0.0;
    if (P.flags & TFG_ENGINE_VERLET) {
        const bool rb = rebuilds_now(P);
        P.verlet_maxdx = rb ? 0.f : __fsqrt_rn(__uint_as_float(P.verlet_maxdx2));
        P.verlet_rebuild = rb;
        P.verlet_maxdx2 = 0u;
        if (rb) P.verlet_rebuilds += 1;
    }
}

// Simulation and grid location of every cell of simulation blockIdx.x.
__global__ void k_fill_cells(const SimParams *sims, int32_t *cell_sim, int4 *cell_at, unsigned char *column) {
    const SimParams &P = sims[blockIdx.x];
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < P.ncells; c += gridDim.y * blockDim.x) {
        int i, j, k;
        cell_loc(P, P.cell_off + c, i, j, k);
        cell_sim[P.cell_off + c] = blockIdx.x;
        cell_at[P.cell_off + c] = make_int4(i, j, k, (int)blockIdx.x);
        column[P.cell_off + c] = k == 0;
    }
}

// space_setpartp (tfSpace.cpp:432-475) for one simulation's particles, written to arena
// slots [slot0, slot0+n) with global cell indices and ids.
__global__ void k_setpartp(int n, const float *__restrict__ xg, SimParams P, float3 lo, float3 hi, float3 org,
                           float3 ih, int slot0, int32_t *cell, float4 *pos, float4 *aux,
                           const int32_t *__restrict__ type, uint32_t *err) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float x[3] = {xg[3 * i], xg[3 * i + 1], xg[3 * i + 2]};
    const float l3[3] = {lo.x, lo.y, lo.z}, h3[3] = {hi.x, hi.y, hi.z}, o3[3] = {org.x, org.y, org.z},
                i3[3] = {ih.x, ih.y, ih.z};
    int ind[3];
    for (int k = 0; k < 3; k++) {
        x[k] = fmaxf(l3[k], fminf(h3[k], x[k]));
        ind[k] = (int)__fmul_rn(__fsub_rn(x[k], o3[k]), i3[k]);
        if (ind[k] < 0 || ind[k] >= P.cdim[k]) {
            atomicOr(err, ERR_RANGE);
            atomicOr(err + 1 + P.red_base / RED_COUNT, ERR_RANGE);
            ind[k] = ind[k] < 0 ? 0 : P.cdim[k] - 1;
        }
    }
    const int s = slot0 + i;
    cell[s] = cell_index(P, ind[0], ind[1], ind[2]);
    pos[s] = make_float4(__fsub_rn(x[0], P.corig[0][ind[0]]), __fsub_rn(x[1], P.corig[1][ind[1]]),
                         __fsub_rn(x[2], P.corig[2][ind[2]]), __int_as_float(type ? type[i] : 0));
    float4 a = aux[s];
    a.w = __int_as_float(P.id_off + i);
    aux[s] = a;
}

// Copy one simulation's particle records from one arena layout to another, moving its
// ids and cells by the change of its offsets.
__global__ void k_relocate(int n, int src0, int dst0, int cap_src, int cap_dst, int nspec, int did, int dcell,
                           ParticleArrays src, ParticleArrays dst) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int a = src0 + i, b = dst0 + i;
    dst.pos[b] = src.pos[a];
    dst.vel[b] = src.vel[a];
    float4 ax = src.aux[a];
    ax.w = __int_as_float(__float_as_int(ax.w) + did);
    dst.aux[b] = ax;
    dst.fext[b] = src.fext[a];
    dst.pforce[b] = src.pforce[a];
    dst.cell[b] = src.cell[a] + dcell;
    for (int s = 0; s < nspec; s++) {
        dst.sval[s * cap_dst + b] = src.sval[s * cap_src + a];
        dst.sq[s * cap_dst + b] = src.sq[s * cap_src + a];
    }
}

// Binning, in four launches (one for small arenas, k_bin_small).  It is bound by launches and L2
// latency below about 100,000 particles and by HBM above:
//   k_bin_count    re-check of the cell-relative positions, count per cell
//   k_scan         block-local scan of the counts; the last block to finish scans the block
//                  totals; the simulations' tick
//   k_place        final cell starts, the pair pass's work items, (id, slot) into cell order
//   k_rank_scatter rank by id inside the cell, then the state itself, with the force init

// Re-check of the cell-relative position (space_shuffle_local, tfSpace.cpp:274-391); returns the
// particle's cell.  The simulations' clocks advance in a later part of the binning, so their
// decisions for this step are taken from the state before it.
__device__ __forceinline__ int recheck(int i, int nsims, const SimParams *sims, const int32_t *cell_sim, float4 *pos,
                                       int32_t *cell, int shuffle) {
    int c = cell[i];
    if (!shuffle) return c;
    float4 p = pos[i];
    const SimParams &P = sims[sim_of(nsims, cell_sim, c)];
    // Verlet mode re-bins only on rebuild steps (engine_verlet_update -> engine_shuffle);
    // a stopped simulation stays as it is
    if (stops_now(P) || ((P.flags & TFG_ENGINE_VERLET) && !rebuilds_now(P))) return c;
    const int d0 = (p.x >= P.h[0]) - (p.x < 0.f);
    const int d1 = (p.y >= P.h[1]) - (p.y < 0.f);
    const int d2 = (p.z >= P.h[2]) - (p.z < 0.f);
    if (d0 | d1 | d2) {
        p.x = __fsub_rn(p.x, __fmul_rn((float)d0, P.h[0]));
        p.y = __fsub_rn(p.y, __fmul_rn((float)d1, P.h[1]));
        p.z = __fsub_rn(p.z, __fmul_rn((float)d2, P.h[2]));
        pos[i] = p;
        int a, b, k;
        cell_loc(P, c, a, b, k);
        c = cell_index(P, (a + d0 + P.cdim[0]) % P.cdim[0], (b + d1 + P.cdim[1]) % P.cdim[1],
                       (k + d2 + P.cdim[2]) % P.cdim[2]);
        cell[i] = c;
    }
    return c;
}

__global__ void k_bin_count(int n, int nsims, const SimParams *sims, const int32_t *cell_sim, float4 *pos, int32_t *cell,
                            int32_t *count, int32_t *lidx, int shuffle, unsigned long long *stamp) {
    step_kernel_begin();
    stamp_begin(stamp);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int c = i < n ? recheck(i, nsims, sims, cell_sim, pos, cell, shuffle) : -1;
    // neighbouring particles mostly share a cell: one atomic per warp and cell (25 -> 17 us on
    // 2,000,000 particles at 13 a cell)
    const unsigned same = __match_any_sync(0xffffffffu, c);
    const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
    int first = 0;
    if (lane == leader && c >= 0) first = atomicAdd(&count[c], __popc(same));
    first = __shfl_sync(0xffffffffu, first, leader);
    if (i < n) lidx[i] = first + __popc(same & ((1u << lane) - 1u));
}

constexpr int kScanThreads = 1024, kScanCells = 4 * kScanThreads;   // cells per block

// Exclusive block scan of (particles, items), packed as low and high word.
__device__ __forceinline__ unsigned long long block_scan2(unsigned long long v, unsigned long long *tot) {
    __shared__ unsigned long long ws[32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned long long x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        unsigned long long s = lane < (int)(blockDim.x >> 5) ? ws[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long y = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += y;
        }
        ws[lane] = s;
    }
    __syncthreads();
    const unsigned long long excl = x - v + (w > 0 ? ws[w - 1] : 0);
    *tot = ws[(blockDim.x >> 5) - 1];
    __syncthreads();
    return excl;
}

// Work items of the tiled pair pass from four consecutive cells with m[] particles: runs of
// neighbouring cells along z (column[k]: cell k is the first of a column) while they hold at most
// `homes` particles together, or single cells (runs false); a crowded cell is several items.
// emit(cell, cells, first home particle, item) is called for each; returns their number.
template <class F>
__device__ __forceinline__ int cell_items(const int *m, uchar4 column, int homes, bool runs, F emit) {
    if (!runs) {
        int count = 0;
#pragma unroll
        for (int k = 0; k < 4; k++)
            for (int c0 = 0; c0 < m[k]; c0 += homes, count++) emit(k, 1, c0, count);
        return count;
    }
    const unsigned char col[4] = {column.x, column.y, column.z, column.w};
    int first = -1, last = 0, total = 0, count = 0;
    auto close = [&] {
        if (first >= 0)
            for (int c0 = 0; c0 < total; c0 += homes, count++) emit(first, last - first + 1, c0, count);
        first = -1;
        total = 0;
    };
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (col[k]) close();
        if (m[k] == 0) continue;
        if (total + m[k] > homes) close();
        if (first < 0) first = k;
        last = k;
        total += m[k];
    }
    close();
    return count;
}

// part[c]: particles and items of the block's cells before c (the items of four consecutive
// cells count as the first one's); pre[b]: of the blocks before b, pre[number of blocks]: all.
// The counts are cleared for the next binning.
__global__ void __launch_bounds__(kScanThreads) k_scan(int ncells, int32_t *count, const uchar4 *column,
                                                       unsigned long long *part, unsigned long long *pre,
                                                       unsigned *ticket, int homes, bool runs, int do_tick, int nsims,
                                                       SimParams *sims, double *red) {
    step_kernel_begin();
    if (do_tick)
        for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nsims; k += gridDim.x * blockDim.x) tick(sims[k], red);
    const int c = blockIdx.x * kScanCells + 4 * threadIdx.x;
    int m[4] = {0, 0, 0, 0};
    int n4 = 0, items = 0;
    if (c < ncells) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            m[k] = c + k < ncells ? count[c + k] : 0;
            n4 += m[k];
        }
        if (n4)
            items = cell_items(m, runs ? column[c / 4] : uchar4(), homes, runs, [](int, int, int, int) {});
    }
    unsigned long long tot, ex = block_scan2((unsigned long long)items << 32 | (unsigned)n4, &tot);
#pragma unroll
    for (int k = 0; k < 4; k++)
        if (c + k < ncells) {
            part[c + k] = ex;
            if (m[k]) count[c + k] = 0;
            ex += (unsigned)m[k] + (k == 0 ? (unsigned long long)items << 32 : 0ull);
        }
    __shared__ bool last;
    if (threadIdx.x == 0) {
        pre[blockIdx.x] = tot;
        __threadfence();
        last = atomicInc(ticket, gridDim.x - 1) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the last block to finish turns the block totals into prefixes
    const int nb = gridDim.x, per = (nb + kScanThreads - 1) / kScanThreads, b0 = threadIdx.x * per;
    unsigned long long sum = 0;
    for (int k = 0; k < per; k++)
        if (b0 + k < nb) sum += __ldcg(&pre[b0 + k]);
    unsigned long long all, run = block_scan2(sum, &all);
    for (int k = 0; k < per; k++)
        if (b0 + k < nb) {
            const unsigned long long t = __ldcg(&pre[b0 + k]);
            pre[b0 + k] = run;
            run += t;
        }
    if (threadIdx.x == 0) pre[nb] = all;
}

__global__ void k_place(int n, int ncells, const int32_t *cell, const int32_t *lidx, const uchar4 *column,
                        const unsigned long long *part, const unsigned long long *pre, int nb, const float4 *aux,
                        int32_t *start, int2 *items, int *nitems, int2 *tmp, int homes, bool runs) {
    step_kernel_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    auto before = [&](int c) { return c < ncells ? part[c] + pre[c / kScanCells] : pre[nb]; };
    if (i < ncells) start[i] = (int)(unsigned)before(i);
    if (i < (ncells + 3) / 4) {   // the items of cells 4 i .. 4 i + 3
        const int c = 4 * i;
        const unsigned long long at = before(c);
        int m[4], p0 = (int)(unsigned)at;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int p1 = (int)(unsigned)before(min(c + k + 1, ncells));
            m[k] = p1 - p0;
            p0 = p1;
        }
        int2 *out = items + (at >> 32);
        cell_items(m, runs ? column[c / 4] : uchar4(), homes, runs, [&](int first, int cells, int c0, int q) {
            out[q] = make_int2(c + first, c0 | (cells - 1) << 30);
        });
        if (i == 0) {
            start[ncells] = (int)(unsigned)pre[nb];
            *nitems = (int)(pre[nb] >> 32);
        }
    }
    if (i < n) {
        const int c = cell[i];
        const int p = (int)(unsigned)(part[c] + pre[c / kScanCells]) + lidx[i];
        tmp[p] = make_int2(__float_as_int(aux[i].w), i);
    }
}

// Place t of the cell order holds particle (id, i): its rank by id among the cell's (the
// deterministic order inside a cell) gives the slot its state moves to.  kExt: some simulation
// has external forces; kRand: some type has had a random force (its persistent value moves).
template <bool kExt, bool kRand>
__device__ __forceinline__ void rank_and_move(int id, int i, int c, int s0, int s1, int cap, int nspec, const int2 *tmp,
                                              const ParticleArrays &src, const ParticleArrays &dst,
                                              int32_t *slot_of_id, int nsims, const SimParams *sims,
                                              const int32_t *cell_sim, const float4 *rforce, float4 *force,
                                              float4 *oldx) {
    const float4 ax = src.aux[i], p = src.pos[i], v = src.vel[i];
    const SimParams &P = sims[sim_of(nsims, cell_sim, c)];
    int d = s0;
#pragma unroll 8
    for (int o = s0; o < s1; o++) d += tmp[o].x < id;
    float4 fe = make_float4(0.f, 0.f, 0.f, 0.f);
    if (kExt) {
        fe = src.fext[i];
        dst.fext[d] = fe;
    }
    if (kRand) {
        const float4 rf = rforce[P.type_base + __float_as_int(p.w)];
        const int lid = id - P.id_off;
        float4 pf;
        if (rf.w != 0.f && (P.time + lid) % (int)rf.z == 0) {
            U4 r = philox({(uint32_t)P.time, (uint32_t)lid, 0u, STREAM_FORCE}, (uint32_t)P.seed,
                          (uint32_t)(P.seed >> 32));
            const float theta = 6.283185307179586f * u01(r.x);
            const float phi = acosf(1.f - 2.f * u01(r.y));
            const float g = sqrtf(-2.0f * logf(u01(r.z))) * cosf(6.283185307179586f * u01(r.w));
            const float rr = rf.x + rf.y * g;
            pf = make_float4(rr * sinf(phi) * cosf(theta), rr * sinf(phi) * sinf(theta), rr * cosf(phi), 0.f);
        } else {
            pf = src.pforce[i];
        }
        dst.pforce[d] = pf;
        if (rf.w != 0.f) {
            fe.x += pf.x;
            fe.y += pf.y;
            fe.z += pf.z;
        }
    }
    force[d] = make_float4(fe.x, fe.y, fe.z, P.self_density);
    dst.pos[d] = p;
    // Verlet reference positions, stored after the rebuild's re-binning (tfEngine.cpp:308-335)
    if (oldx && (P.flags & TFG_ENGINE_VERLET) && P.verlet_rebuild) oldx[d] = make_float4(p.x, p.y, p.z, 0.f);
    dst.vel[d] = v;
    dst.aux[d] = ax;
    dst.cell[d] = c;
    for (int s = 0; s < nspec; s++) {
        dst.sval[s * cap + d] = src.sval[s * cap + i];
        dst.sq[s * cap + d] = src.sq[s * cap + i];
    }
    if (slot_of_id) slot_of_id[id] = d;
}

template <bool kExt, bool kRand>
__global__ void k_rank_scatter(int n, int cap, int nspec, const int2 *tmp, const int32_t *start, ParticleArrays src,
                               ParticleArrays dst, int32_t *slot_of_id, int nsims, const SimParams *sims,
                               const int32_t *cell_sim, const float4 *rforce, float4 *force, float4 *oldx) {
    step_kernel_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int2 me = tmp[t];
    const int c = src.cell[me.y];
    rank_and_move<kExt, kRand>(me.x, me.y, c, start[c], start[c + 1], cap, nspec, tmp, src, dst, slot_of_id, nsims,
                               sims, cell_sim, rforce, force, oldx);
}

// The whole binning of a small arena in one launch, by one cluster of eight blocks.  Four
// launches take 9 to 13 us however few particles there are; this takes two cluster barriers
// (7 us for 500 particles, 10 for 8,000; with two particles a thread it was slower than four
// launches, 16 against 14 us for 11,000).  Every block scans all counts itself, so the cell
// starts are in its shared memory.
constexpr int kSmallBlocks = 8, kSmallThreads = 1024;   // one particle each
constexpr int kSmallCells = 16 * kSmallThreads;   // a multiple of 4 per thread

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

template <bool kExt, bool kRand>
__global__ void __cluster_dims__(kSmallBlocks, 1, 1) __launch_bounds__(kSmallThreads, 1) k_bin_small(BinArgs b) {
    extern __shared__ int32_t start_s[];
    step_kernel_begin();
    stamp_begin(b.stamp);
    const int t0 = blockIdx.x * kSmallThreads + threadIdx.x;
    // count
    int c = 0, l = 0, id = 0;
    if (t0 < b.n) {
        id = __float_as_int(b.src.aux[t0].w);
        c = recheck(t0, b.nsims, b.sims, b.cell_sim, b.src.pos, b.src.cell, b.shuffle);
        l = atomicAdd(&b.count[c], 1);
    }
    cluster_barrier();
    // scan: thread t holds cells [per t, per (t + 1)); the blocks share the writing
    const int per = ((b.ncells + kSmallThreads - 1) / kSmallThreads + 3) & ~3, first = per * threadIdx.x;
    // (the count array and start_s go on to a multiple of four)
    unsigned long long sum = 0;
#pragma unroll 1
    for (int k = first; k < min(first + per, b.ncells); k += 4) {
        const int4 m4 = __ldcg(reinterpret_cast<const int4 *>(b.count + k));
        *reinterpret_cast<int4 *>(start_s + k) = m4;
        const int m[4] = {m4.x, m4.y, m4.z, m4.w}, n4 = m[0] + m[1] + m[2] + m[3];
        if (n4)
            sum += (unsigned long long)cell_items(m, b.runs ? b.column[k / 4] : uchar4(), b.homes, b.runs,
                                                  [](int, int, int, int) {}) << 32 | (unsigned)n4;
    }
    unsigned long long all, run = block_scan2(sum, &all);
    const bool mine = (threadIdx.x & (kSmallBlocks - 1)) == blockIdx.x;
#pragma unroll 1
    for (int k = first; k < min(first + per, b.ncells); k += 4) {
        const int4 m4 = *reinterpret_cast<const int4 *>(start_s + k);
        const int m[4] = {m4.x, m4.y, m4.z, m4.w}, n4 = m[0] + m[1] + m[2] + m[3], p = (int)(unsigned)run;
        const int4 s4 = make_int4(p, p + m[0], p + m[0] + m[1], p + m[0] + m[1] + m[2]);
        *reinterpret_cast<int4 *>(start_s + k) = s4;
        if (mine) *reinterpret_cast<int4 *>(b.start + k) = s4;
        if (n4) {
            int2 *out = b.items + (run >> 32);
            run += (unsigned)n4;
            run += (unsigned long long)cell_items(m, b.runs ? b.column[k / 4] : uchar4(), b.homes, b.runs,
                                                  [&](int f, int cells, int c0, int q) {
                                                      if (mine) out[q] = make_int2(k + f, c0 | (cells - 1) << 30);
                                                  }) << 32;
        }
    }
    if (t0 == 0) *b.nitems = (int)(all >> 32);
    if (b.shuffle)
        for (int k = t0; k < b.nsims; k += kSmallBlocks * kSmallThreads) tick(b.sims[k], b.red);
    __syncthreads();
    // place
    if (t0 < b.n) b.tmp[start_s[c] + l] = make_int2(id, t0);
    cluster_barrier();
    // (behind the last group's four starts)
    if (t0 == 0) b.start[b.ncells] = (int)(unsigned)all;
    // the counts return to zero; rank and move
    if (mine)
        for (int k = 0; k < per; k++)
            if (first + k < b.ncells) b.count[first + k] = 0;
    if (t0 < b.n) {
        const int2 me = b.tmp[t0];
        const int cc = b.src.cell[me.y];
        rank_and_move<kExt, kRand>(me.x, me.y, cc, start_s[cc], cc + 1 < b.ncells ? start_s[cc + 1] : b.n, b.cap, b.nspec,
                                   b.tmp, b.src, b.dst, b.slot_of_id, b.nsims, b.sims, b.cell_sim, b.rforce, b.force,
                                   b.oldx);
    }
}

// A thread's sums over its bonds or angles, in FP64, for one simulation at a time.
struct BondSums {
    int rb = -1;
    double epot = 0.0, vir = 0.0;
    __device__ __forceinline__ void add(double *red, int slot, int to, float e, float v) {
        if (to != rb) {
            if (rb >= 0) {
                atomicAdd(&red[rb + slot], epot);
                atomicAdd(&red[rb + RED_VIRIAL], vir);
            }
            rb = to;
            epot = vir = 0.0;
        }
        epot += e;
        vir += v;
    }
};

// bond_eval (tfBond.cpp:97-345) for table potentials.  Bound by the latency of the gathers by id.  A
// block takes `per` bonds in a row, so that all blocks are resident at once and their atomics to
// the simulation's totals, which are serial, are few: with k_angles 93 -> 83 us on 1.9M bonds and
// 1.8M angles (six blocks per SM; 91 with five, 100 with eight, which are not all resident).
__global__ void k_bonds(int nb, int per, const SimParams *sims, const int32_t *cell_sim, const int2 *bonds,
                        const int32_t *bslot, const PotDev *bpots, const float *bblob, const int32_t *slot_of_id,
                        const float4 *pos, const float4 *aux, const int32_t *cell, float4 *force, double *red,
                        unsigned long long *stamp) {
    step_kernel_begin();
    stamp_begin(stamp);
    BondSums sums;
    const int last = min(nb, ((int)blockIdx.x + 1) * per);
#pragma unroll 1
    for (int b = blockIdx.x * per + threadIdx.x; b < last; b += blockDim.x) {
        const int2 bd = bonds[b];
        const PotDev &pot = bpots[bslot[b]];
        const int si = slot_of_id[bd.x], sj = slot_of_id[bd.y];
        const bool there = pot.kind == POT_TABLE && si >= 0 && sj >= 0;
        float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), pj = pi;
        int ci = 0, cj = 0;
        if (there) {
            pi = pos[si];
            pj = pos[sj];
            ci = cell[si];
            cj = cell[sj];
        }
        const SimParams &P = sims[cell_sim[ci]];
        if (there && !P.stopped) {
            float epot = 0.f, vir = 0.f;
            int s0 = 0, s1 = 0, s2 = 0;
            if (ci != cj) {
                int ai, bi, ki, aj, bj, kj;
                cell_loc(P, ci, ai, bi, ki);
                cell_loc(P, cj, aj, bj, kj);
                s0 = wrap_shift(ai - aj);
                s1 = wrap_shift(bi - bj);
                s2 = wrap_shift(ki - kj);
            }
            const float pix = __fadd_rn(pi.x, __fmul_rn(P.h[0], (float)s0));
            const float piy = __fadd_rn(pi.y, __fmul_rn(P.h[1], (float)s1));
            const float piz = __fadd_rn(pi.z, __fmul_rn(P.h[2], (float)s2));
            const float dx = __fsub_rn(pix, pj.x), dy = __fsub_rn(piy, pj.y), dz = __fsub_rn(piz, pj.z);
            const float r2 = __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
            // potential_eval_adjust_distance2
            float r = __fsqrt_rn(r2);
            if (pot.flags & TFG_POTENTIAL_SCALED) r = __fdiv_rn(r, __fadd_rn(aux[si].x, aux[sj].x));
            else if (pot.flags & TFG_POTENTIAL_SHIFTED)
                r = __fadd_rn(__fsub_rn(r, __fadd_rn(aux[si].x, aux[sj].x)), pot.r0_plusone);
            float rr2 = __fmul_rn(r, r);
            if (!(rr2 > __fmul_rn(pot.b, pot.b))) {
                rr2 = fmaxf(rr2, __fmul_rn(pot.a, pot.a));
                // potential_eval (tf_potential_eval.h:74-102)
                const float rb_ = __fsqrt_rn(rr2);
                const float t = __fadd_rn(pot.alpha0, __fmul_rn(rb_, __fadd_rn(pot.alpha1, __fmul_rn(rb_, pot.alpha2))));
                int ind = (int)fmaxf(0.0f, t);
                if (ind > pot.n) ind = pot.n;
                float ee, eff, c1;
                table_row_eval(bblob + pot.offset + ind * kChunk, rb_, ee, eff, c1);
                const float f = eff * c1 / rb_;
                atomicAdd(&force[si], make_float4(-f * dx, -f * dy, -f * dz, 0.f));
                atomicAdd(&force[sj], make_float4(f * dx, f * dy, f * dz, 0.f));
                epot = ee;
                vir = -f * r2;
            }
            sums.add(red, RED_EPOT_BOND, P.red_base, epot, vir);
        }
    }
    keyed_add3(red, sums.rb, RED_EPOT_BOND, sums.epot, RED_VIRIAL, sums.vir, RED_VIRIAL, 0.0);
}

// angle_eval (tfAngle.cpp:90-382), j is the vertex; blocks as those of k_bonds.
__global__ void k_angles(int na, int per, const SimParams *sims, const int32_t *cell_sim, const int4 *angles,
                         const PotDev *bpots, const float *bblob, const int32_t *slot_of_id, const float4 *pos,
                         const int32_t *cell, float4 *force, double *red, unsigned long long *stamp) {
    step_kernel_begin();
    stamp_begin(stamp);
    BondSums sums;
    const int last = min(na, ((int)blockIdx.x + 1) * per);
#pragma unroll 1
    for (int q = blockIdx.x * per + threadIdx.x; q < last; q += blockDim.x) {
        const int4 A = angles[q];
        const PotDev &pot = bpots[A.w];
        const int si = slot_of_id[A.x], sj = slot_of_id[A.y], sk = slot_of_id[A.z];
        const bool there = pot.kind == POT_TABLE && si >= 0 && sj >= 0 && sk >= 0;
        float4 pi = make_float4(0.f, 0.f, 0.f, 0.f), pj = pi, pk = pi;
        int ci = 0, cj = 0, ck = 0;
        if (there) {
            pi = pos[si];
            pj = pos[sj];
            pk = pos[sk];
            ci = cell[si];
            cj = cell[sj];
            ck = cell[sk];
        }
        const SimParams &P = sims[cell_sim[cj]];
        if (there && !P.stopped) {
            float epot = 0.f;
            int li[3], lj[3], lk[3];
            cell_loc(P, ci, li[0], li[1], li[2]);
            cell_loc(P, cj, lj[0], lj[1], lj[2]);
            cell_loc(P, ck, lk[0], lk[1], lk[2]);
            float xi[3] = {pi.x, pi.y, pi.z}, xj[3] = {pj.x, pj.y, pj.z}, xk[3] = {pk.x, pk.y, pk.z};
            float rji[3], rjk[3];
            for (int k = 0; k < 3; k++) {
                xi[k] = __fadd_rn(xi[k], __fmul_rn((float)wrap_shift(li[k] - lj[k]), P.h[k]));
                xk[k] = __fadd_rn(xk[k], __fmul_rn((float)wrap_shift(lk[k] - lj[k]), P.h[k]));
                rji[k] = __fsub_rn(xi[k], xj[k]);
                rjk[k] = __fsub_rn(xk[k], xj[k]);
            }
            const float dprod = __fadd_rn(__fadd_rn(__fmul_rn(rji[0], rjk[0]), __fmul_rn(rji[1], rjk[1])),
                                          __fmul_rn(rji[2], rjk[2]));
            const float nji = __fadd_rn(__fadd_rn(__fmul_rn(rji[0], rji[0]), __fmul_rn(rji[1], rji[1])),
                                        __fmul_rn(rji[2], rji[2]));
            const float njk = __fadd_rn(__fadd_rn(__fmul_rn(rjk[0], rjk[0]), __fmul_rn(rjk[1], rjk[1])),
                                        __fmul_rn(rjk[2], rjk[2]));
            const float inji = __fdiv_rn(1.0f, __fsqrt_rn(nji));
            const float injk = __fdiv_rn(1.0f, __fsqrt_rn(njk));
            const float ctheta = fmaxf(-1.0f, fminf(1.0f, __fmul_rn(__fmul_rn(dprod, inji), injk)));
            float dxi[3], dxk[3];
            if (ctheta == 0.f || ctheta == -1.f) {
                // Random derivative plane: the reference draws from the global mt19937
                // (tfAngle.cpp:210-223); here a Philox stream keyed on (step, angle).
                U4 r = philox({(uint32_t)P.time, (uint32_t)(q - P.angle_off), 0u, STREAM_ANGLE}, (uint32_t)P.seed,
                              (uint32_t)(P.seed >> 32));
                float x[3] = {2.f * u01(r.x) - 1.f, 2.f * u01(r.y) - 1.f, 2.f * u01(r.z) - 1.f};
                const float vik[3] = {xi[0] - xk[0], xi[1] - xk[1], xi[2] - xk[2]};
                const float dd = x[0] * vik[0] + x[1] * vik[1] + x[2] * vik[2];
                for (int k = 0; k < 3; k++) x[k] = x[k] - dd * vik[k];
                const float len = sqrtf(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
                for (int k = 0; k < 3; k++) dxi[k] = dxk[k] = x[k] / len;
            } else {
                for (int k = 0; k < 3; k++) {
                    dxi[k] = (rjk[k] * injk - ctheta * rji[k] * inji) * inji;
                    dxk[k] = (rji[k] * inji - ctheta * rjk[k] * injk) * injk;
                }
            }
            if (!(ctheta > pot.b)) {
                const float rr = fmaxf(ctheta, pot.a);
                const float t = __fadd_rn(pot.alpha0, __fmul_rn(rr, __fadd_rn(pot.alpha1, __fmul_rn(rr, pot.alpha2))));
                const int ind = (int)fmaxf(0.0f, t);
                if (ind <= pot.n) {
                    float ee, eff, c1;
                    table_row_eval(bblob + pot.offset + ind * kChunk, rr, ee, eff, c1);
                    eff = eff * c1;
                    float wi[3], wk[3];
                    for (int k = 0; k < 3; k++) { wi[k] = eff * dxi[k]; wk[k] = eff * dxk[k]; }
                    atomicAdd(&force[si], make_float4(-wi[0], -wi[1], -wi[2], 0.f));
                    atomicAdd(&force[sk], make_float4(-wk[0], -wk[1], -wk[2], 0.f));
                    atomicAdd(&force[sj], make_float4(wi[0] + wk[0], wi[1] + wk[1], wi[2] + wk[2], 0.f));
                    epot = ee;
                }
            }
            sums.add(red, RED_EPOT_ANGLE, P.red_base, epot, 0.f);
        }
    }
    keyed_add(red, sums.rb, RED_EPOT_ANGLE, sums.epot);
}

// Verlet mode: the integrator branch of engine_advance_forward_euler for Verlet lists
// (tf_engine_advance.cpp:367-427), plus the squared displacement from the reference
// position that engine_verlet_update takes the maximum of (tfEngine.cpp:239-252).
__device__ __forceinline__ float advance_verlet(const SimParams &P, bool newtonian, const float4 &f, float imass,
                                                float4 &p, float4 &v, const float4 &ox) {
    const float dt = P.dt;
    const float fv[3] = {f.x, f.y, f.z};
    float x[3] = {p.x, p.y, p.z}, vv[3] = {v.x, v.y, v.z};
    for (int k = 0; k < 3; k++) {
        if (newtonian) vv[k] = __fadd_rn(vv[k], __fmul_rn(__fmul_rn(fv[k], dt), imass));
        else vv[k] = __fmul_rn(fv[k], imass);
        x[k] = __fadd_rn(x[k], __fmul_rn(vv[k], dt));
    }
    p = make_float4(x[0], x[1], x[2], p.w);
    v = make_float4(vv[0], vv[1], vv[2], v.w);
    const float w0 = __fsub_rn(x[0], ox.x), w1 = __fsub_rn(x[1], ox.y), w2 = __fsub_rn(x[2], ox.z);
    return __fadd_rn(__fadd_rn(__fmul_rn(w0, w0), __fmul_rn(w1, w1)), __fmul_rn(w2, w2));
}

// Add per-thread FP32 partials to slots of one simulation's FP64 totals, as keyed_add does for a
// block of one simulation: FP32 over each warp, FP64 across warps, one atomic per block and
// total, under a single barrier.  Total k is value(k); slot(k) its slot.
template <class V, class K>
__device__ __forceinline__ void block_add(double *red, int rb, int totals, V value, K slot) {
    __shared__ double part[3 + kMaxSpecies][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    for (int k = 0; k < totals; k++) {
        float v = value(k);
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane == 0) part[k][w] = (double)v;
    }
    __syncthreads();
    if (threadIdx.x < totals) {
        double t = 0.0;
        for (int k = 0; k < nw; k++) t += part[threadIdx.x][k];
        if (t != 0.0) atomicAdd(&red[rb + slot(threadIdx.x)], t);
    }
}

// Blocks of 128 end more evenly than of 256 or 512: 46.1, 42.7 and 58.0 us on 2,000,000 particles
// (256, 128, 512), 81, 76 and 107 on 256 tissues.
constexpr int kAdvanceThreads = 128;
constexpr unsigned kStampBlocks = 4096;   // more than two waves of resident blocks

// cell_advance_forward_euler + Fluxes_integrate; one thread per particle.
__global__ void k_advance(int n, int cap, int nspec, int nsims, SimParams *sims, const int32_t *cell_sim, float4 *pos,
                          float4 *vel, const float4 *aux, const float4 *force, int32_t *cell, float *sval, float *sq,
                          const float *type_mass, const int32_t *type_dyn, const uint32_t *species_flags,
                          const float4 *oldx, double *red, uint32_t *err, unsigned long long *stamps, int stamp_mask) {
    step_kernel_begin();
    for (int k = 2; k < 4; k++)
        if (stamp_mask & (1 << k)) stamp_begin(stamps + k);
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    float ke = 0.f, vol = 0.f, mig = 0.f;
    int rb = -1;
    int vsim = -1;          // Verlet simulation of this particle
    uint32_t dx2 = 0u;      // its squared displacement (float bits)
    // particles are in cell order: the block's belong to one simulation if its first and last do (a
    // cell that its particle has already left for another is one of the same simulation)
    const int sim0 = nsims == 1 ? 0 : cell_sim[cell[blockIdx.x * blockDim.x]];
    const bool one_sim = nsims == 1 || sim0 == cell_sim[cell[min((int)((blockIdx.x + 1) * blockDim.x), n) - 1]];
    const int block_rb = sims[sim0].red_base;
    // every particle's state is loaded at once, before it is known whether its simulation runs
    int c0 = 0;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f), v = p, ax = p, f = p;
    if (i < n) {
        c0 = cell[i];
        p = pos[i];
        v = vel[i];
        ax = aux[i];
        f = force[i];
    }
    const int sim = one_sim || i >= n ? sim0 : cell_sim[c0];
    if (i < n && !sims[sim].stopped) {
        const SimParams &P = sims[sim];
        rb = P.red_base;
        const int type = __float_as_int(p.w);
        const uint32_t flags = (uint32_t)__float_as_int(ax.z);
        const float imass = ax.y;
        ke = 0.5f * type_mass[P.type_base + type] * (v.x * v.x + v.y * v.y + v.z * v.z);
        bool migrated = false;
        if (P.flags & TFG_ENGINE_VERLET) {
            const float d2 = advance_verlet(P, type_dyn[P.type_base + type] == TFG_NEWTONIAN, f, imass, p, v, oldx[i]);
            if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) {
                atomicOr(err, ERR_NAN);
                atomicOr(err + 1 + rb / RED_COUNT, ERR_NAN);
            }
            pos[i] = p;
            vel[i] = v;
            vsim = sim;
            dx2 = __float_as_uint(d2);
            goto reduce;
        }
        const bool frozen_all = (flags & TFG_PARTICLE_FROZEN_X) && (flags & TFG_PARTICLE_FROZEN_Y) &&
                                (flags & TFG_PARTICLE_FROZEN_Z);
        if (!frozen_all) {
            const float mask[3] = {(flags & TFG_PARTICLE_FROZEN_X) ? 0.0f : 1.0f,
                                   (flags & TFG_PARTICLE_FROZEN_Y) ? 0.0f : 1.0f,
                                   (flags & TFG_PARTICLE_FROZEN_Z) ? 0.0f : 1.0f};
            float x[3] = {p.x, p.y, p.z}, vv[3] = {v.x, v.y, v.z};
            const float fv[3] = {f.x, f.y, f.z};
            int delta[3];
            const float dt = P.dt;
            if (type_dyn[P.type_base + type] == TFG_NEWTONIAN) {
                for (int k = 0; k < 3; k++) {
                    const float a = __fmul_rn(__fmul_rn(dt, fv[k]), imass);
                    const float nv = __fmul_rn(mask[k], __fadd_rn(vv[k], a));
                    vv[k] = __fmul_rn(nv, nv) <= P.maxv2[k] ? nv : __fmul_rn(__fdiv_rn(nv, fabsf(nv)), P.maxv[k]);
                    x[k] = __fadd_rn(x[k], __fmul_rn(dt, vv[k]));
                    delta[k] = (x[k] >= P.h[k]) - (x[k] < 0.0f);
                }
            } else {
                for (int k = 0; k < 3; k++) {
                    float dx = __fmul_rn(mask[k], __fmul_rn(__fmul_rn(dt, fv[k]), imass));
                    dx = __fmul_rn(dx, dx) <= P.maxx2[k] ? dx : __fmul_rn(__fdiv_rn(dx, fabsf(dx)), P.maxx[k]);
                    vv[k] = __fdiv_rn(dx, dt);
                    x[k] = __fadd_rn(x[k], dx);
                    delta[k] = (x[k] >= P.h[k]) - (x[k] < 0.0f);
                }
            }
            const float nd = f.w;
            const float inv_nd = nd > 0.f ? __fdiv_rn(1.f, nd) : 0.f;
            vol = inv_nd;
            if ((delta[0] | delta[1] | delta[2]) && P.walls_reflect) {
                // reflection at FREESLIP / VELOCITY walls (apply_update_pos_vel,
                // tf_boundary_eval.h:46-134), walls in the reference's order
                int la, lb, lc;
                cell_loc(P, c0, la, lb, lc);
                bool enforced = false;
                for (int w = 0; w < 6; w++) {
                    if (!(P.walls_reflect & (1u << w)) || !on_wall(P, w, la, lb, lc)) continue;
                    const int ax = w >> 1;
                    const bool high = (w & 1) != 0;
                    if (high ? !(x[ax] >= P.h[ax]) : !(x[ax] <= 0.f)) continue;
                    const bool slip = (P.wall_kind[w] & TFG_BOUNDARY_FREESLIP) != 0;
                    const float rest = slip ? 1.0f : P.wall_vel[w].w;
                    if (high)
                        x[ax] = __fsub_rn(P.h[ax], fmaxf(__fmul_rn(__fsub_rn(x[ax], P.h[ax]), rest), 1.1920928955078125e-7f));
                    else
                        x[ax] = fmaxf(__fmul_rn(-x[ax], rest), 0.0f);
                    if (slip) {
                        vv[ax] = -vv[ax];
                    } else {
                        const float U[3] = {P.wall_vel[w].x, P.wall_vel[w].y, P.wall_vel[w].z};
                        for (int k = 0; k < 3; k++) vv[k] = __fsub_rn(U[k], __fmul_rn(__fsub_rn(vv[k], U[k]), rest));
                    }
                    enforced = true;
                }
                if (enforced)
                    for (int k = 0; k < 3; k++) delta[k] = (x[k] >= P.h[k]) - (x[k] < 0.0f);
            }
            if (delta[0] | delta[1] | delta[2]) {
                for (int k = 0; k < 3; k++) {
                    if (x[k] >= P.h2[k] || x[k] <= -P.h[k]) {
                        atomicOr(err, ERR_TOOFAST);
                        atomicOr(err + 1 + rb / RED_COUNT, ERR_TOOFAST);
                        break;
                    }
                    x[k] = __fadd_rn(x[k], -__fmul_rn((float)delta[k], P.h[k]));
                }
                int a, b, c;
                cell_loc(P, c0, a, b, c);
                cell[i] = cell_index(P, (a + delta[0] + P.cdim[0]) % P.cdim[0], (b + delta[1] + P.cdim[1]) % P.cdim[1],
                                     (c + delta[2] + P.cdim[2]) % P.cdim[2]);
                migrated = true;
                mig = 1.f;
                if (nspec > 0) {
                    const int loc[3] = {a, b, c};
                    if (crosses_resetting_wall(P, loc, delta))
                        for (int s = 0; s < nspec; s++) sval[s * cap + i] = P.species_reset[s];
                }
            }
            if (!(isfinite(x[0]) && isfinite(x[1]) && isfinite(x[2]))) {
                atomicOr(err, ERR_NAN);
                atomicOr(err + 1 + rb / RED_COUNT, ERR_NAN);
            }
            pos[i] = make_float4(x[0], x[1], x[2], p.w);
            vel[i] = make_float4(vv[0], vv[1], vv[2], inv_nd);
        }
        // Fluxes_integrate runs over the particles still in their cell: migrants keep their
        // flux increment for the next step (they sit in the destination's incoming list).
        for (int s = 0; s < nspec; s++) {
            float sv = sval[s * cap + i];
            if (!migrated) {
                const float konst = (species_flags[P.spec_base + s] & 1u) ? 0.f : 1.f;
                const float q = sq[s * cap + i];
                sv = fmaxf(0.0f, __fadd_rn(sv, __fmul_rn(__fmul_rn(P.dt_flux, q), konst)));
                sval[s * cap + i] = sv;
                sq[s * cap + i] = 0.f;
            }
        }
    }
reduce:
    {
        // largest displacement per Verlet simulation: one atomic per warp when the warp's
        // particles share a simulation
        const int first = __shfl_sync(0xffffffffu, vsim, 0);
        if (__all_sync(0xffffffffu, vsim == first)) {
            const uint32_t m = __reduce_max_sync(0xffffffffu, dx2);
            if (first >= 0 && (threadIdx.x & 31) == 0) atomicMax(&sims[first].verlet_maxdx2, m);
        } else if (vsim >= 0) {
            atomicMax(&sims[vsim].verlet_maxdx2, dx2);
        }
    }
    auto species = [&](int s) { return rb >= 0 ? sval[s * cap + i] : 0.f; };
    if (one_sim) {
        block_add(red, block_rb, 3 + nspec,
                  [&](int k) { return k == 0 ? ke : (k == 1 ? vol : (k == 2 ? mig : species(k - 3))); },
                  [](int k) { return k == 0 ? RED_KINETIC : (k == 1 ? RED_VOLUME : (k == 2 ? RED_MIGRATIONS : RED_SPECIES0 + k - 3)); });
    } else {
        keyed_add3(red, rb, RED_KINETIC, ke, RED_VOLUME, vol, RED_MIGRATIONS, mig);
        for (int s = 0; s < nspec; s++) keyed_add(red, rb, RED_SPECIES0 + s, species(s));
    }
    // the end of the step: the latest of the blocks that can end last
    if (stamp_mask && threadIdx.x == 0 && blockIdx.x + kStampBlocks >= gridDim.x) atomicMax(stamps + 4, global_timer());
}

__global__ void k_flux_integrate(int n, int cap, int nspec, int sub, const SimParams *sims, const int32_t *cell_sim,
                                 const int32_t *cell, float *sval, float *sq, const uint32_t *species_flags) {
    step_kernel_begin();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const SimParams &P = sims[cell_sim[cell[i]]];
    if (P.stopped || sub >= P.nr_fluxsteps - 1) return;
    for (int s = 0; s < nspec; s++) {
        const float konst = (species_flags[P.spec_base + s] & 1u) ? 0.f : 1.f;
        const float q = sq[s * cap + i];
        sval[s * cap + i] = fmaxf(0.0f, __fadd_rn(sval[s * cap + i], __fmul_rn(__fmul_rn(P.dt_flux, q), konst)));
        sq[s * cap + i] = 0.f;
    }
}

// Per-particle state of slots [slot0, slot0+n) gathered by local id (id - id_off).
__global__ void k_gather(int n, int slot0, int cap, int nspec, SimParams P, ParticleArrays A, const float4 *force,
                         float *x, float *xrel, int32_t *cellout, float *v, float *f, float *dens, float *species,
                         float *q) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = slot0 + k;
    const float4 p = A.pos[i];
    const int id = __float_as_int(A.aux[i].w) - P.id_off;
    if (id < 0 || id >= n) return;
    const int c = A.cell[i];
    int l0, l1, l2;
    cell_loc(P, c, l0, l1, l2);
    if (x) {
        x[3 * id] = __fadd_rn(P.corig[0][l0], p.x);
        x[3 * id + 1] = __fadd_rn(P.corig[1][l1], p.y);
        x[3 * id + 2] = __fadd_rn(P.corig[2][l2], p.z);
    }
    if (xrel) { xrel[3 * id] = p.x; xrel[3 * id + 1] = p.y; xrel[3 * id + 2] = p.z; }
    if (cellout) cellout[id] = c - P.cell_off;
    if (v) { const float4 w = A.vel[i]; v[3 * id] = w.x; v[3 * id + 1] = w.y; v[3 * id + 2] = w.z; }
    if (f || dens) {
        const float4 w = force[i];
        if (f) { f[3 * id] = w.x; f[3 * id + 1] = w.y; f[3 * id + 2] = w.z; }
        if (dens) dens[id] = w.w;
    }
    for (int s = 0; s < nspec; s++) {
        if (species) species[id * nspec + s] = A.sval[s * cap + i];
        if (q) q[id * nspec + s] = A.sq[s * cap + i];
    }
}

// Forces, densities and flux increments of every particle, kept by its id over binnings that move
// it to another slot, and put back.
__global__ void k_keep(int n, int cap, int nspec, bool restore, const float4 *aux, float4 *force, float *sq,
                       float4 *kept_force, float *kept_sq) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int id = __float_as_int(aux[i].w);
    if (restore) force[i] = kept_force[id];
    else kept_force[id] = force[i];
    for (int s = 0; s < nspec; s++) {
        const size_t a = (size_t)s * cap + i, b = (size_t)s * n + id;
        if (restore) sq[a] = kept_sq[b];
        else kept_sq[b] = sq[a];
    }
}

inline int nblk(long long n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

void launch_stamp(unsigned long long *t, int k, cudaStream_t s) { k_stamp<<<1, 1, 0, s>>>(t, k); }

void launch_fill_cells(int nsims, const SimParams *sims, int32_t *cell_sim, int4 *cell_at, unsigned char *column,
                       cudaStream_t s) {
    if (nsims > 0) k_fill_cells<<<dim3(nsims, 32), kThreads, 0, s>>>(sims, cell_sim, cell_at, column);
}

void launch_setpartp(int n, const float *xg, const SimParams &P, float3 lo, float3 hi, float3 org, float3 ih,
                     int slot0, int32_t *cell, float4 *pos, float4 *aux, const int32_t *type, uint32_t *err,
                     cudaStream_t s) {
    if (n > 0)
        k_setpartp<<<nblk(n, kThreads), kThreads, 0, s>>>(n, xg, P, lo, hi, org, ih, slot0, cell, pos, aux, type, err);
}

void launch_relocate(int n, int src0, int dst0, int cap_src, int cap_dst, int nspec, int did, int dcell,
                     const ParticleArrays &src, const ParticleArrays &dst, cudaStream_t s) {
    if (n > 0)
        k_relocate<<<nblk(n, kThreads), kThreads, 0, s>>>(n, src0, dst0, cap_src, cap_dst, nspec, did, dcell, src,
                                                          dst);
}

void launch_keep(int n, int cap, int nspec, bool restore, const ParticleArrays &A, float4 *force, float4 *kept_force,
                 float *kept_sq, cudaStream_t s) {
    if (n > 0)
        k_keep<<<nblk(n, kThreads), kThreads, 0, s>>>(n, cap, nspec, restore, A.aux, force, A.sq, kept_force, kept_sq);
}

int scan_blocks(int ncells) { return nblk(ncells, kScanCells); }

template <bool kExt, bool kRand> void launch_bin_variant(const BinArgs &b, cudaStream_t s) {
    if (b.n <= kSmallBlocks * kSmallThreads && b.ncells <= kSmallCells) {
        static PerDevice ready;
        ready.get([] {
            return cudaFuncSetAttribute(k_bin_small<kExt, kRand>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        kSmallCells * (int)sizeof(int32_t)) == cudaSuccess;
        });
        launch_step_kernel(k_bin_small<kExt, kRand>, kSmallBlocks, kSmallThreads, sizeof(int32_t) * kSmallCells, s, b);
        return;
    }
    if (b.n > 0)
        launch_step_kernel(k_bin_count, nblk(b.n, kThreads), kThreads, 0, s, b.n, b.nsims, b.sims, b.cell_sim, b.src.pos,
                           b.src.cell, b.count, b.lidx, b.shuffle, b.stamp);
    const int nb = scan_blocks(b.ncells);
    launch_step_kernel(k_scan, nb, kScanThreads, 0, s, b.ncells, b.count, b.column, b.part, b.pre, b.ticket, b.homes,
                       b.runs, b.shuffle, b.nsims, b.sims, b.red);
    launch_step_kernel(k_place, nblk(b.n > b.ncells ? b.n : b.ncells, kThreads), kThreads, 0, s, b.n, b.ncells,
                       b.src.cell, b.lidx, b.column, b.part, b.pre, nb, b.src.aux, b.start, b.items, b.nitems, b.tmp,
                       b.homes, b.runs);
    if (b.n > 0)
        launch_step_kernel(k_rank_scatter<kExt, kRand>, nblk(b.n, kThreads), kThreads, 0, s, b.n, b.cap, b.nspec, b.tmp,
                           b.start, b.src, b.dst, b.slot_of_id, b.nsims, b.sims, b.cell_sim, b.rforce, b.force,
                           b.oldx);
}

void launch_bin(const BinArgs &b, cudaStream_t s) {
    if (b.has_ext && b.has_rand) launch_bin_variant<true, true>(b, s);
    else if (b.has_ext) launch_bin_variant<true, false>(b, s);
    else if (b.has_rand) launch_bin_variant<false, true>(b, s);
    else launch_bin_variant<false, false>(b, s);
}

// Bonds or angles of a block: a multiple of its threads, for at most six blocks per SM.
static int per_block(int n, int sms) { return nblk(nblk(n, 6 * sms), kThreads) * kThreads; }

void launch_bonds(int nb, int sms, const SimParams *sims, const int32_t *cell_sim, const int2 *bonds, const int32_t *bslot,
                  const PotDev *bpots, const float *bblob, const int32_t *slot_of_id, const float4 *pos,
                  const float4 *aux, const int32_t *cell, float4 *force, double *red, unsigned long long *stamp,
                  cudaStream_t s) {
    if (nb > 0)
        launch_step_kernel(k_bonds, nblk(nb, per_block(nb, sms)), kThreads, 0, s, nb, per_block(nb, sms), sims, cell_sim, bonds, bslot, bpots, bblob,
                           slot_of_id, pos, aux, cell, force, red, stamp);
}

void launch_angles(int na, int sms, const SimParams *sims, const int32_t *cell_sim, const int4 *angles, const PotDev *bpots,
                   const float *bblob, const int32_t *slot_of_id, const float4 *pos, const int32_t *cell,
                   float4 *force, double *red, unsigned long long *stamp, cudaStream_t s) {
    if (na > 0)
        launch_step_kernel(k_angles, nblk(na, per_block(na, sms)), kThreads, 0, s, na, per_block(na, sms), sims, cell_sim, angles, bpots, bblob,
                           slot_of_id, pos, cell, force, red, stamp);
}

void launch_advance(int n, int cap, int nspec, int nsims, SimParams *sims, const int32_t *cell_sim,
                    const ParticleArrays &A, const float4 *force, const float *type_mass, const int32_t *type_dyn,
                    const uint32_t *species_flags, const float4 *oldx, double *red, uint32_t *err,
                    unsigned long long *stamps, int stamp_mask, cudaStream_t s) {
    if (n > 0)
        launch_step_kernel(k_advance, nblk(n, kAdvanceThreads), kAdvanceThreads, 0, s, n, cap, nspec, nsims, sims, cell_sim, A.pos, A.vel,
                           A.aux, force, A.cell, A.sval, A.sq, type_mass, type_dyn, species_flags, oldx, red, err,
                           stamps, stamp_mask);
}

void launch_flux_integrate(int n, int cap, int nspec, int sub, const SimParams *sims, const int32_t *cell_sim,
                           const int32_t *cell, float *sval, float *sq, const uint32_t *species_flags,
                           cudaStream_t s) {
    if (n > 0 && nspec > 0)
        launch_step_kernel(k_flux_integrate, nblk(n, kThreads), kThreads, 0, s, n, cap, nspec, sub, sims, cell_sim,
                           cell, sval, sq, species_flags);
}

void launch_gather(int n, int slot0, int cap, int nspec, const SimParams &P, const ParticleArrays &A,
                   const float4 *force, float *x, float *xrel, int32_t *cell, float *v, float *f, float *dens,
                   float *species, float *q, cudaStream_t s) {
    if (n > 0)
        k_gather<<<nblk(n, kThreads), kThreads, 0, s>>>(n, slot0, cap, nspec, P, A, force, x, xrel, cell, v, f, dens,
                                                       species, q);
}

}  // namespace tfg
