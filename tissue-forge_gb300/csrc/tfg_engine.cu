// Engine internals: simulation set-up, arena layout, the per-step pipeline and the
// reductions.  One step over the arena (engine_step, tfEngine.cpp:1378-1429):
//   tick     every simulation's time += 1 (on the device)
//   bin      space_shuffle_local re-check + counting sort into cell order
//   pair     fused nonbonded pass (tfg_pair_tile.cu, or tfg_pair.cu in deterministic mode)
//   bonded   bond_eval / angle_eval
//   advance  forward Euler + Fluxes_integrate + FP64 per-simulation totals
#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "tfg_engine_impl.h"

namespace tfg {

int fail(tfg_engine *e, int code, const std::string &msg) {
    if (e) e->last_error = msg;
    return code;
}

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t _e = (call);                                                              \
        if (_e != cudaSuccess)                                                                \
            return fail(eng, TFG_E_CUDA, std::string(#call ": ") + cudaGetErrorString(_e));   \
    } while (0)

namespace {

inline float bits_to_float(int32_t v) {
    float f;
    std::memcpy(&f, &v, sizeof(f));
    return f;
}

int alloc_particles(tfg_engine *eng, ParticleArrays &A, int cap) {
    int rc;
    const size_t ns = std::max(1, eng->nspec);
    if ((rc = dalloc(eng, &A.pos, cap)) || (rc = dalloc(eng, &A.vel, cap)) || (rc = dalloc(eng, &A.aux, cap)) ||
        (rc = dalloc(eng, &A.fext, cap)) || (rc = dalloc(eng, &A.pforce, cap)) || (rc = dalloc(eng, &A.cell, cap)) ||
        (rc = dalloc(eng, &A.sval, (size_t)cap * ns)) || (rc = dalloc(eng, &A.sq, (size_t)cap * ns)))
        return rc;
    // both copies start at zero: they are not moved while no simulation has such a force
    CK(cudaMemsetAsync(A.fext, 0, sizeof(float4) * cap, eng->stream));
    CK(cudaMemsetAsync(A.pforce, 0, sizeof(float4) * cap, eng->stream));
    return TFG_OK;
}

void free_particles(ParticleArrays &A) {
    cudaFree(A.pos); cudaFree(A.vel); cudaFree(A.aux); cudaFree(A.fext); cudaFree(A.pforce);
    cudaFree(A.cell); cudaFree(A.sval); cudaFree(A.sq);
    A = ParticleArrays();
}

// Upload one simulation's pending particle data into arena slots [slot0, slot0+n) of D.
int upload_pending(tfg_engine *eng, SimHost &S, ParticleArrays &D, int cap) {
    const int n = S.n;
    if (n == 0) return TFG_OK;
    cudaStream_t s = eng->stream;
    const int slot0 = S.P.id_off;
    std::vector<float4> vel(n), aux(n), fext(n), pf(n, make_float4(0, 0, 0, 0));
    for (int i = 0; i < n; i++) {
        vel[i] = make_float4(S.v.empty() ? 0.f : S.v[3 * i], S.v.empty() ? 0.f : S.v[3 * i + 1],
                             S.v.empty() ? 0.f : S.v[3 * i + 2], 0.f);
        aux[i] = make_float4(S.radius.empty() ? 1.0f : S.radius[i], S.imass.empty() ? 1.0f : S.imass[i],
                             bits_to_float((int32_t)(S.flags.empty() ? 0u : S.flags[i])), bits_to_float(S.P.id_off + i));
        fext[i] = make_float4(S.force_i.empty() ? 0.f : S.force_i[3 * i], S.force_i.empty() ? 0.f : S.force_i[3 * i + 1],
                              S.force_i.empty() ? 0.f : S.force_i[3 * i + 2], 0.f);
    }
    CK(cudaMemcpyAsync(D.vel + slot0, vel.data(), sizeof(float4) * n, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(D.aux + slot0, aux.data(), sizeof(float4) * n, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(D.fext + slot0, fext.data(), sizeof(float4) * n, cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(D.pforce + slot0, pf.data(), sizeof(float4) * n, cudaMemcpyHostToDevice, s));
    for (int k = 0; k < eng->nspec; k++) {
        std::vector<float> col(n, 0.f);
        if (!S.species.empty())
            for (int i = 0; i < n; i++) col[i] = S.species[(size_t)i * eng->nspec + k];
        CK(cudaMemcpyAsync(D.sval + (size_t)k * cap + slot0, col.data(), sizeof(float) * n, cudaMemcpyHostToDevice, s));
        if (S.q_pending.size() == (size_t)n * eng->nspec) {
            // a resumed simulation keeps the increments its migrants carry to the next step
            std::vector<float> qc(n);
            for (int i = 0; i < n; i++) qc[i] = S.q_pending[(size_t)i * eng->nspec + k];
            CK(cudaMemcpyAsync(D.sq + (size_t)k * cap + slot0, qc.data(), sizeof(float) * n, cudaMemcpyHostToDevice,
                               s));
        } else {
            CK(cudaMemsetAsync(D.sq + (size_t)k * cap + slot0, 0, sizeof(float) * n, s));
        }
    }
    CK(cudaStreamSynchronize(s));
    S.q_pending.clear();
    if (!S.pending_binned) {
        float *dx = nullptr;
        int32_t *dtype = nullptr;
        int rc;
        if ((rc = dalloc(eng, &dx, (size_t)3 * n)) || (rc = dalloc(eng, &dtype, n))) return rc;
        CK(cudaMemcpyAsync(dx, S.x.data(), sizeof(float) * 3 * n, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(dtype, S.type.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, s));
        float3 lo, hi, org, ih;
        float *plo = &lo.x, *phi = &hi.x, *porg = &org.x, *pih = &ih.x;
        for (int k = 0; k < 3; k++) {
            const float o = S.desc.origin[k], dm = S.desc.dim[k];
            plo[k] = (float)(o * (1.0 + FLT_EPSILON));
            phi[k] = (float)((dm + o) * (1.0 - FLT_EPSILON));
            porg[k] = o;
            pih[k] = (float)(1.0 / S.P.h[k]);
        }
        launch_setpartp(n, dx, S.P, lo, hi, org, ih, slot0, D.cell, D.pos, D.aux, dtype, eng->err, s);
        cudaError_t e = cudaStreamSynchronize(s);
        cudaFree(dx);
        cudaFree(dtype);
        if (e != cudaSuccess) return fail(eng, TFG_E_CUDA, cudaGetErrorString(e));
    } else {
        std::vector<float4> pos(n);
        std::vector<int32_t> cg(n);
        for (int i = 0; i < n; i++) {
            pos[i] = make_float4(S.xrel[3 * i], S.xrel[3 * i + 1], S.xrel[3 * i + 2], bits_to_float(S.type[i]));
            cg[i] = S.cell[i] + S.P.cell_off;
        }
        CK(cudaMemcpyAsync(D.pos + slot0, pos.data(), sizeof(float4) * n, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(D.cell + slot0, cg.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, s));
        CK(cudaStreamSynchronize(s));
    }
    return TFG_OK;
}

template <typename T> int ensure(tfg_engine *eng, T **p, size_t &cap, size_t need) {
    if (need <= cap && *p) return TFG_OK;
    int rc = dalloc(eng, p, std::max<size_t>(need, 1));
    if (rc) return rc;
    cap = std::max<size_t>(need, 1);
    return TFG_OK;
}

// Lay the arena out again: offsets of every live simulation, relocation of particles
// already on the device, upload of pending particles, per-cell simulation index,
// per-simulation parameters, bonds and angles; then a non-shuffling sort into cell order.
int relayout(tfg_engine *eng) {
    cudaStream_t s = eng->stream;
    const int T = eng->max_type;
    // errors raised under the old layout belong to the simulations of the old order
    if (int rc0 = collect_errors(eng)) return rc0;
    std::vector<int> order;
    for (int k = 0; k < (int)eng->sims.size(); k++)
        if (eng->sims[k].live && eng->sims[k].loaded) order.push_back(k);
    // Verlet state kept on the device (rebuild count, last displacement) survives the
    // re-upload of the parameters; every Verlet simulation rebuilds at the next step.
    bool any_verlet = false;
    for (int k : order) any_verlet |= (eng->sims[k].P.flags & TFG_ENGINE_VERLET) != 0;
    if (any_verlet && eng->sims_dev && !eng->order.empty()) {
        std::vector<SimParams> dev(eng->order.size());
        CK(cudaMemcpyAsync(dev.data(), eng->sims_dev, sizeof(SimParams) * dev.size(), cudaMemcpyDeviceToHost, s));
        CK(cudaStreamSynchronize(s));
        for (size_t q = 0; q < eng->order.size(); q++) {
            SimHost &S = eng->sims[eng->order[q]];
            if (!S.live || S.pending) continue;
            S.P.verlet_rebuilds = dev[q].verlet_rebuilds;
            S.P.verlet_maxdx = dev[q].verlet_maxdx;
        }
    }
    for (int k : order) {
        eng->sims[k].P.verlet_rebuild = 2;
        eng->sims[k].P.verlet_maxdx2 = 0u;
    }
    int N = 0, C = 0, NA = 0, NB = 0;
    std::vector<int> old_slot(order.size()), old_cell(order.size());
    std::vector<bool> was_in(order.size());
    for (size_t q = 0; q < order.size(); q++) {
        SimHost &S = eng->sims[order[q]];
        was_in[q] = S.in_arena && !S.pending;
        old_slot[q] = S.arena_slot0;
        old_cell[q] = S.arena_cell_off;
        S.P.cell_off = C;
        S.P.id_off = N;
        S.P.angle_off = NA;
        S.P.pot_base = (int)q * T * T;
        S.P.type_base = (int)q * T;
        S.P.red_base = (int)q * RED_COUNT;
        S.P.spec_base = (int)q * kMaxSpecies;
        S.P.wpot_base = (int)q * 6 * T;
        resolve_boundaries(S);
        S.P.time = S.time;
        N += S.n;
        C += S.P.ncells;
        NA += (int)S.angles.size();
        NB += (int)S.bonds.size();
    }
    // particle buffers: relocate into the spare buffer, or into new ones when they grow
    const int old_cap = eng->cap;
    ParticleArrays src = eng->A[eng->cur];
    ParticleArrays dst;
    int new_cap = old_cap;
    bool fresh = false;
    if (N > old_cap || !src.pos) {
        new_cap = std::max(std::max(N, eng->capacity_hint), 1);
        int rc = alloc_particles(eng, dst, new_cap);
        if (rc) return rc;
        fresh = true;
    } else {
        dst = eng->A[eng->cur ^ 1];
    }
    for (size_t q = 0; q < order.size(); q++) {
        SimHost &S = eng->sims[order[q]];
        if (was_in[q])
            launch_relocate(S.n, old_slot[q], S.P.id_off, old_cap, new_cap, eng->nspec, S.P.id_off - old_slot[q],
                            S.P.cell_off - old_cell[q], src, dst, s);
    }
    CK(cudaStreamSynchronize(s));
    if (fresh) {
        free_particles(eng->A[0]);
        free_particles(eng->A[1]);
        eng->A[0] = dst;
        int rc = alloc_particles(eng, eng->A[1], new_cap);
        if (rc) return rc;
        eng->cur = 0;
        int r2;
        if ((r2 = dalloc(eng, &eng->force, new_cap)) || (r2 = dalloc(eng, &eng->lidx, new_cap)) ||
            (r2 = dalloc(eng, &eng->bin_tmp, new_cap)) || (r2 = dalloc(eng, &eng->slot_of_id, new_cap)))
            return r2;
        eng->cap = new_cap;
    } else {
        eng->cur ^= 1;
    }
    if (any_verlet && eng->oldx_cap < eng->cap) {
        int r2 = dalloc(eng, &eng->oldx, eng->cap);
        if (r2) return r2;
        eng->oldx_cap = eng->cap;
    }
    // per-simulation parameters with device pointers to the concatenated cell origins
    size_t norig = 0;
    for (int k : order) norig += eng->sims[k].orig.size();
    int rc = ensure(eng, &eng->corig, eng->corig_cap, norig);
    if (rc) return rc;
    std::vector<float> orig_all;
    orig_all.reserve(norig);
    std::vector<SimParams> P_all;
    for (size_t q = 0; q < order.size(); q++) {
        SimHost &S = eng->sims[order[q]];
        const size_t base = orig_all.size();
        orig_all.insert(orig_all.end(), S.orig.begin(), S.orig.end());
        for (int k = 0; k < 3; k++) S.P.corig[k] = eng->corig + base + (size_t)k * S.maxc;
        P_all.push_back(S.P);
    }
    if (norig) CK(cudaMemcpyAsync(eng->corig, orig_all.data(), sizeof(float) * norig, cudaMemcpyHostToDevice, s));
    if ((int)order.size() > eng->sims_cap) {
        if ((rc = dalloc(eng, &eng->sims_dev, order.size()))) return rc;
        eng->sims_cap = (int)order.size();
    }
    if (!P_all.empty())
        CK(cudaMemcpyAsync(eng->sims_dev, P_all.data(), sizeof(SimParams) * P_all.size(), cudaMemcpyHostToDevice, s));
    if (C + 1 > eng->cells_cap) {
        const int cc = (C + 4) & ~3;   // the binning takes cells four at a time
        if ((rc = dalloc(eng, &eng->count, cc)) || (rc = dalloc(eng, &eng->start, cc + 4)) ||
            (rc = dalloc(eng, &eng->column, cc)) ||
            (rc = dalloc(eng, &eng->scan_part, cc)) || (rc = dalloc(eng, &eng->scan_pre, scan_blocks(cc) + 1)) ||
            (rc = dalloc(eng, &eng->cell_sim, cc)) || (rc = dalloc(eng, &eng->cell_at, cc)))
            return rc;
        CK(cudaMemsetAsync(eng->count, 0, sizeof(int32_t) * cc, s));
        eng->cells_cap = cc;
    }
    if ((rc = ensure(eng, &eng->items, eng->items_cap, (size_t)C + N / 8 + 1))) return rc;
    launch_fill_cells((int)order.size(), eng->sims_dev, eng->cell_sim, eng->cell_at, eng->column, s);
    if ((int)order.size() > eng->err_slots) {
        const int slots = std::max((int)order.size(), 2 * eng->err_slots);
        if ((rc = dalloc(eng, &eng->err, 1 + (size_t)slots))) return rc;
        eng->err_slots = slots;
    }
    CK(cudaMemsetAsync(eng->err, 0, sizeof(uint32_t) * (1 + (size_t)eng->err_slots), s));
    size_t rneed = std::max<size_t>(order.size(), 1) * RED_COUNT;
    if ((rc = ensure(eng, &eng->red, eng->red_cap, rneed))) return rc;
    CK(cudaMemsetAsync(eng->red, 0, sizeof(double) * rneed, s));
    // pending particles (need the new offsets and origin pointers)
    for (size_t q = 0; q < order.size(); q++) {
        SimHost &S = eng->sims[order[q]];
        if (!was_in[q] && (rc = upload_pending(eng, S, eng->A[eng->cur], eng->cap))) return rc;
    }
    // bonds and angles with global ids
    std::vector<int2> b;
    std::vector<int32_t> bs;
    std::vector<int4> a;
    for (int k : order) {
        SimHost &S = eng->sims[k];
        for (size_t q = 0; q < S.bonds.size(); q++) {
            b.push_back(make_int2(S.bonds[q].x + S.P.id_off, S.bonds[q].y + S.P.id_off));
            bs.push_back(S.bond_slot[q]);
        }
        for (const int4 &g : S.angles)
            a.push_back(make_int4(g.x + S.P.id_off, g.y + S.P.id_off, g.z + S.P.id_off, g.w));
    }
    if (NB > eng->bcap) {
        if ((rc = dalloc(eng, &eng->bonds, NB)) || (rc = dalloc(eng, &eng->bond_slot, NB))) return rc;
        eng->bcap = NB;
    }
    if (NA > eng->acap) {
        if ((rc = dalloc(eng, &eng->angles, NA))) return rc;
        eng->acap = NA;
    }
    if (NB) {
        CK(cudaMemcpyAsync(eng->bonds, b.data(), sizeof(int2) * NB, cudaMemcpyHostToDevice, s));
        CK(cudaMemcpyAsync(eng->bond_slot, bs.data(), sizeof(int32_t) * NB, cudaMemcpyHostToDevice, s));
    }
    if (NA) CK(cudaMemcpyAsync(eng->angles, a.data(), sizeof(int4) * NA, cudaMemcpyHostToDevice, s));
    eng->nb = NB;
    eng->na = NA;
    eng->n = N;
    eng->ncells = C;
    eng->order = order;
    CK(cudaStreamSynchronize(s));
    rc = read_err(eng);
    if (rc) return rc;
    for (size_t q = 0; q < order.size(); q++) {
        SimHost &S = eng->sims[order[q]];
        S.in_arena = true;
        S.arena_slot0 = S.P.id_off;
        S.arena_cell_off = S.P.cell_off;
        S.pending = false;
        S.x.clear(); S.xrel.clear(); S.cell.clear(); S.v.clear(); S.radius.clear(); S.imass.clear();
        S.species.clear(); S.force_i.clear(); S.type.clear(); S.flags.clear();
    }
    for (auto &S : eng->sims)
        if (!S.live) S.in_arena = false;
    eng->tables_dirty = true;
    eng->layout_dirty = false;
    return TFG_OK;
}

// A potential in the tiled pair pass's compact form.
PotPair to_pair(const PotDev &p) {
    PotPair c;
    std::memset(&c, 0, sizeof(c));
    if (p.kind == POT_NONE) return c;
    const bool table = p.kind == POT_TABLE;
    c.p0 = table ? p.alpha0 : p.dpd_alpha;
    c.p1 = table ? p.alpha1 : p.dpd_gamma;
    c.p2 = table ? p.alpha2 : p.dpd_sigma;
    c.b = p.b;
    c.a = p.a;
    c.c = table ? p.r0_plusone : 1.0f / p.b;
    c.nk = table ? (uint32_t)p.n | POTC_TABLE : (uint32_t)POTC_DPD;
    if (p.flags & TFG_POTENTIAL_SHIFTED) c.nk |= POTC_SHIFTED;
    if (table && (p.flags & TFG_POTENTIAL_SCALED)) c.nk |= POTC_SCALED;
    c.offset = p.offset;
    return c;
}

// A table buffer for `need` elements and, when `fetched`, a texture of 16-byte texels over all of
// it, by which the pair pass on tables reads it; tex stays 0 where the buffer has more texels than
// a texture can have.
template <typename T>
int ensure_fetched(tfg_engine *eng, T **p, size_t &cap, size_t need, bool fetched, cudaTextureObject_t &tex) {
    const bool kept = need <= cap && *p;
    const int rc = ensure(eng, p, cap, need);   // (cudaFree waits for the kernels that read the old one)
    if (!kept && tex) {
        cudaDestroyTextureObject(tex);
        tex = 0;
    }
    if (rc || !fetched || tex) return rc;
    cudaResourceDesc res;
    std::memset(&res, 0, sizeof(res));
    res.resType = cudaResourceTypeLinear;
    res.res.linear.devPtr = *p;
    res.res.linear.desc = cudaCreateChannelDesc<uint4>();
    res.res.linear.sizeInBytes = cap * sizeof(T);
    size_t most = 0;
    CK(cudaDeviceGetTexture1DLinearMaxWidth(&most, &res.res.linear.desc, eng->device));
    if (cap * sizeof(T) / sizeof(uint4) > most) return TFG_OK;
    cudaTextureDesc how;
    std::memset(&how, 0, sizeof(how));
    how.readMode = cudaReadModeElementType;
    CK(cudaCreateTextureObject(&tex, &res, &how, nullptr));
    return TFG_OK;
}

// Upload the interaction tables of every live simulation (potentials with their table
// blob, fluxes, per-type arrays, species flags) and the bonded potentials.
int upload_tables(tfg_engine *eng) {
    cudaStream_t s = eng->stream;
    const int T = eng->max_type;
    const size_t nsim = std::max<size_t>(eng->order.size(), 1);
    std::vector<PotDev> pots(nsim * T * T);
    std::vector<PotDev> wp(nsim * 6 * T);
    for (auto &p : wp) std::memset(&p, 0, sizeof(p));
    eng->has_wall_pots = false;
    std::vector<FluxSet> fl(nsim * T * T);
    std::vector<float4> rf(nsim * T, make_float4(0, 0, 1, 0));
    std::vector<float> mass(nsim * T, 1.0f);
    std::vector<int32_t> dyn(nsim * T, TFG_NEWTONIAN);
    std::vector<uint32_t> spf(nsim * kMaxSpecies, 0u);
    std::vector<float> blob;
    for (auto &p : pots) std::memset(&p, 0, sizeof(p));
    for (auto &f : fl) std::memset(&f, 0, sizeof(f));
    eng->has_dpd = false;
    eng->has_flux = false;
    eng->radii = false;
    eng->max_fluxsteps = 1;
    uint32_t nodens = TFG_ENGINE_NO_DENSITY;
    for (size_t q = 0; q < eng->order.size(); q++) {
        SimHost &S = eng->sims[eng->order[q]];
        nodens &= S.desc.flags;
        for (int k = 0; k < T * T; k++) {
            PotDev d = S.pots[k];
            if (d.kind == POT_TABLE) {
                // a table equal to an earlier one of the same simulation (the (j,i) copy of
                // (i,j), or a shared potential) is stored once
                int found = -1;
                for (int k2 = 0; k2 < k && found < 0; k2++)
                    if (S.pots[k2].kind == POT_TABLE && S.tables[k2] == S.tables[k]) found = pots[q * T * T + k2].offset;
                if (found >= 0) {
                    d.offset = found;
                } else {
                    d.offset = (int)blob.size();
                    blob.insert(blob.end(), S.tables[k].begin(), S.tables[k].end());
                }
            }
            if (d.kind == POT_DPD) eng->has_dpd = true;
            if (d.kind == POT_TABLE && (d.flags & (TFG_POTENTIAL_SHIFTED | TFG_POTENTIAL_SCALED))) eng->radii = true;
            if (S.fluxes[k].count > 0) {
                eng->has_flux = true;
                eng->max_fluxsteps = std::max(eng->max_fluxsteps, S.P.nr_fluxsteps);
            }
            pots[q * T * T + k] = d;
            fl[q * T * T + k] = S.fluxes[k];
        }
        for (int t = 0; t < T; t++) {
            rf[q * T + t] = S.rforce[t];
            eng->has_rand |= rf[q * T + t].w != 0.f;
            mass[q * T + t] = S.mass[t];
            dyn[q * T + t] = S.dyn[t];
        }
        for (int k = 0; k < kMaxSpecies; k++) spf[q * kMaxSpecies + k] = S.species_flags[k];
        for (int k = 0; k < 6 * T; k++) {
            PotDev d = S.wpots[k];
            if (d.kind == POT_NONE) continue;
            eng->has_wall_pots = true;
            if (d.kind == POT_TABLE) {
                d.offset = (int)blob.size();
                blob.insert(blob.end(), S.wtables[k].begin(), S.wtables[k].end());
            }
            if (d.kind == POT_DPD) eng->has_dpd = true;
            wp[q * 6 * T + k] = d;
        }
    }
    eng->flags_all = nodens;
    if (blob.empty()) blob.assign(kChunk, 0.f);   // row 0 of no table is readable
    int rc;
    const bool tables = !eng->has_dpd && !(eng->has_flux && eng->nspec > 0);   // as launch_pair_tile has it
    if ((rc = ensure_fetched(eng, &eng->blob, eng->blob_cap, blob.size(), tables, eng->blob_tex)) ||
        (rc = ensure(eng, &eng->pots, eng->pots_cap, pots.size())) ||
        (rc = ensure(eng, &eng->fluxes, eng->fluxes_cap, fl.size())) ||
        (rc = ensure(eng, &eng->species_flags, eng->spec_cap, spf.size())) ||
        (rc = ensure(eng, &eng->wpots, eng->wpots_cap, wp.size())))
        return rc;
    std::vector<PotPair> pc(pots.size());
    for (size_t k = 0; k < pots.size(); k++) pc[k] = to_pair(pots[k]);
    if ((rc = ensure_fetched(eng, &eng->potc, eng->potc_cap, pc.size(), tables, eng->potc_tex))) return rc;
    eng->one = pc[0];
    eng->one_flux = fl[0];
    eng->has_one = std::all_of(pc.begin(), pc.end(), [&](const PotPair &c) { return !std::memcmp(&c, &pc[0], sizeof(c)); }) &&
                   std::all_of(fl.begin(), fl.end(), [&](const FluxSet &f) { return !std::memcmp(&f, &fl[0], sizeof(f)); });
    CK(cudaMemcpyAsync(eng->potc, pc.data(), sizeof(PotPair) * pc.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(eng->wpots, wp.data(), sizeof(PotDev) * wp.size(), cudaMemcpyHostToDevice, s));
    if (rf.size() > eng->types_cap) {
        if ((rc = dalloc(eng, &eng->rforce, rf.size())) || (rc = dalloc(eng, &eng->type_mass, rf.size())) ||
            (rc = dalloc(eng, &eng->type_dyn, rf.size())))
            return rc;
        eng->types_cap = rf.size();
    }
    eng->blob_floats = (int)blob.size();
    CK(cudaMemcpyAsync(eng->blob, blob.data(), sizeof(float) * blob.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(eng->pots, pots.data(), sizeof(PotDev) * pots.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(eng->fluxes, fl.data(), sizeof(FluxSet) * fl.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(eng->rforce, rf.data(), sizeof(float4) * rf.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(eng->type_mass, mass.data(), sizeof(float) * mass.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(eng->type_dyn, dyn.data(), sizeof(int32_t) * dyn.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(eng->species_flags, spf.data(), sizeof(uint32_t) * spf.size(), cudaMemcpyHostToDevice, s));
    // bonded potentials (engine-wide slots)
    std::vector<float> bblob;
    std::vector<PotDev> bp = eng->h_bpots;
    for (int k = 0; k < kMaxBondSlots; k++)
        if (bp[k].kind == POT_TABLE) {
            bp[k].offset = (int)bblob.size();
            bblob.insert(bblob.end(), eng->h_btables[k].begin(), eng->h_btables[k].end());
        }
    if (bblob.empty()) bblob.push_back(0.f);
    if ((rc = ensure(eng, &eng->bblob, eng->bblob_cap, bblob.size()))) return rc;
    CK(cudaMemcpyAsync(eng->bblob, bblob.data(), sizeof(float) * bblob.size(), cudaMemcpyHostToDevice, s));
    CK(cudaMemcpyAsync(eng->bpots, bp.data(), sizeof(PotDev) * kMaxBondSlots, cudaMemcpyHostToDevice, s));
    CK(cudaStreamSynchronize(s));
    eng->tables_dirty = false;
    return TFG_OK;
}

}  // namespace

int check_launch(tfg_engine *eng) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return fail(eng, TFG_E_CUDA, std::string("kernel launch: ") + cudaGetErrorString(e));
    return TFG_OK;
}

static int err_code(uint32_t flags) {
    if (flags & ERR_NAN) return TFG_E_NAN;
    if (flags & ERR_RANGE) return TFG_E_RANGE;
    if (flags & ERR_TOOFAST) return TFG_E_TOOFAST;
    if (flags & ERR_OVERFLOW) return TFG_E_OVERFLOW;
    return TFG_OK;
}

// Copy the device error words to the host, in stream order (collect_errors reads them).
static int fetch_errors(tfg_engine *eng) {
    const size_t words = 1 + (size_t)std::min((int)eng->order.size(), eng->err_slots);
    if (words > eng->err_host_cap) {
        if (eng->err_host) cudaFreeHost(eng->err_host);
        eng->err_host = nullptr;
        eng->err_host_cap = 0;
        CK(cudaMallocHost((void **)&eng->err_host, sizeof(uint32_t) * words));
        eng->err_host_cap = words;
    }
    CK(cudaMemcpyAsync(eng->err_host, eng->err, sizeof(uint32_t) * words, cudaMemcpyDeviceToHost, eng->stream));
    return TFG_OK;
}

// Read and clear the device error words.  A simulation's word goes to its sticky status
// (the reference flags the offending particle, toofast_error, tf_engine_advance.cpp:72-85,
// 204-206; here the simulation is the unit that fails), the engine's word to pending_err.
// `fetched`: fetch_errors was called and the stream has been waited for since.
int collect_errors(tfg_engine *eng, bool fetched) {
    if (!fetched) {
        int rc = fetch_errors(eng);
        if (rc) return rc;
        CK(cudaStreamSynchronize(eng->stream));
    }
    const int ns = std::min((int)eng->order.size(), eng->err_slots);
    const uint32_t *w = eng->err_host;
    bool any = false;
    for (int k = 0; k <= ns; k++) any |= w[k] != 0u;
    if (!any) return TFG_OK;
    CK(cudaMemsetAsync(eng->err, 0, sizeof(uint32_t) * (1 + ns), eng->stream));
    CK(cudaStreamSynchronize(eng->stream));
    eng->pending_err |= w[0];
    for (int q = 0; q < ns; q++) {
        SimHost &S = eng->sims[eng->order[q]];
        if (w[1 + q] && S.status == TFG_OK) S.status = err_code(w[1 + q]);
    }
    return TFG_OK;
}

int read_err(tfg_engine *eng, bool fetched) {
    int rc = collect_errors(eng, fetched);
    if (rc) return rc;
    const uint32_t flags = eng->pending_err;
    eng->pending_err = 0u;
    if (flags) {
        std::string which;
        for (int k : eng->order)
            if (eng->sims[k].status != TFG_OK) which += (which.empty() ? " (simulation " : ", ") + std::to_string(k);
        if (!which.empty()) which += ")";
        if (flags & ERR_NAN) return fail(eng, TFG_E_NAN, "non-finite particle position" + which);
        if (flags & ERR_RANGE) return fail(eng, TFG_E_RANGE, "particle outside the space" + which);
        if (flags & ERR_TOOFAST)
            return fail(eng, TFG_E_TOOFAST, "particle moved more than one cell in a step" + which);
        if (flags & ERR_OVERFLOW) return fail(eng, TFG_E_OVERFLOW, "capacity exceeded");
    }
    return TFG_OK;
}

int sim_status(tfg_engine *eng, int sim, int *status) {
    int rc = sim_check(eng, sim);
    if (rc) return rc;
    if (!status) return TFG_E_INVAL;
    if ((rc = collect_errors(eng))) return rc;
    *status = eng->sims[sim].status;
    return TFG_OK;
}

int sim_check(tfg_engine *eng, int sim) {
    if (!eng) return TFG_E_INVAL;
    if (sim < 0 || sim >= (int)eng->sims.size() || !eng->sims[sim].live)
        return fail(eng, TFG_E_INVAL, "no such simulation");
    return TFG_OK;
}

PotDev to_dev(const tfg_potential *p) {
    PotDev d;
    std::memset(&d, 0, sizeof(d));
    d.kind = p->kind == TFG_POTENTIAL_KIND_DPD ? POT_DPD : POT_TABLE;
    d.flags = p->flags;
    d.alpha0 = p->alpha[0];
    d.alpha1 = p->alpha[1];
    d.alpha2 = p->alpha[2];
    d.r0_plusone = p->r0_plusone;
    d.a = p->a;
    d.b = p->b;
    d.n = p->n;
    d.dpd_alpha = p->dpd_alpha;
    d.dpd_gamma = p->dpd_gamma;
    d.dpd_sigma = p->dpd_sigma;
    return d;
}

// Periodicity and wall flags of a simulation from its six walls as set (BoundaryConditions,
// tfBoundaryConditions.cpp:192-216 and space_init's cell flags, tfSpace.cpp:780-835): a
// periodic wall facing a non-periodic one makes both periodic.  Walls are set one at a
// time, so the rule is applied to the current settings, which stay as set.
void resolve_boundaries(SimHost &S) {
    SimParams &P = S.P;
    P.periodic = 0;
    P.walls_active = 0;
    P.walls_reflect = 0;
    uint32_t kind[6];
    for (int w = 0; w < 6; w++) kind[w] = S.walls[w].kind;
    for (int ax = 0; ax < 3; ax++) {
        const bool lo = kind[2 * ax] & TFG_BOUNDARY_PERIODIC, hi = kind[2 * ax + 1] & TFG_BOUNDARY_PERIODIC;
        if (lo != hi) kind[2 * ax] = kind[2 * ax + 1] = TFG_BOUNDARY_PERIODIC;
        if (lo || hi) P.periodic |= 1u << ax;
    }
    const uint32_t active = TFG_BOUNDARY_FREESLIP | TFG_BOUNDARY_VELOCITY | TFG_BOUNDARY_POTENTIAL;
    for (int w = 0; w < 6; w++) {
        const tfg_boundary &b = S.walls[w];
        P.wall_kind[w] = kind[w];
        P.wall_vel[w] = make_float4(b.velocity[0], b.velocity[1], b.velocity[2], b.restore);
        P.wall_radius[w] = b.radius;
        if (kind[w] & active) P.walls_active |= 1u << w;
        if (kind[w] & (TFG_BOUNDARY_FREESLIP | TFG_BOUNDARY_VELOCITY)) P.walls_reflect |= 1u << w;
    }
}

int set_boundary_sim(tfg_engine *eng, int sim, int wall, const tfg_boundary *bc) {
    int rc = sim_check(eng, sim);
    if (rc) return rc;
    if (wall < 0 || wall > 5 || !bc) return fail(eng, TFG_E_INVAL, "wall must be 0..5");
    tfg_boundary b = *bc;
    if (b.kind & TFG_BOUNDARY_NO_SLIP) {
        b.kind = (b.kind & ~TFG_BOUNDARY_NO_SLIP) | TFG_BOUNDARY_VELOCITY;
        b.velocity[0] = b.velocity[1] = b.velocity[2] = 0.f;
    }
    SimHost &S = eng->sims[sim];
    S.walls[wall] = b;
    resolve_boundaries(S);
    eng->layout_dirty = true;   // parameters are uploaded with the layout
    return TFG_OK;
}

int set_boundary_potential_sim(tfg_engine *eng, int sim, int wall, int type, const tfg_potential *p) {
    int rc = sim_check(eng, sim);
    if (rc) return rc;
    const int T = eng->max_type;
    if (wall < -1 || wall > 5 || type < 0 || type >= T) return fail(eng, TFG_E_INVAL, "bad wall or type");
    SimHost &S = eng->sims[sim];
    for (int w = (wall < 0 ? 0 : wall); w <= (wall < 0 ? 5 : wall); w++) {
        const int k = w * T + type;
        if (!p) {
            std::memset(&S.wpots[k], 0, sizeof(PotDev));
            S.wtables[k].clear();
            continue;
        }
        if (p->kind == TFG_POTENTIAL_KIND_POTENTIAL) {
            if (!p->c || p->n < 1 || p->n > TFG_POTENTIAL_IVALSMAX) return fail(eng, TFG_E_INVAL, "bad table");
            S.wtables[k].assign(p->c, p->c + (size_t)(p->n + 1) * kChunk);
        } else if (p->kind != TFG_POTENTIAL_KIND_DPD) {
            return fail(eng, TFG_E_INVAL, "unsupported potential kind");
        }
        S.wpots[k] = to_dev(p);
    }
    eng->tables_dirty = true;
    return TFG_OK;
}

// A new simulation: space geometry (space_init, tfSpace.cpp:737-777) and integrator
// limits (tf_engine_advance.cpp:337-350).
int add_sim(tfg_engine *eng, const tfg_engine_desc *d, int *out) {
    if (!d) return TFG_E_INVAL;
    if (d->max_type != eng->max_type || d->nr_species != eng->nspec)
        return fail(eng, TFG_E_INVAL, "simulation types/species differ from the engine's");
    if (!(d->cutoff > 0) || !(d->dt > 0)) return fail(eng, TFG_E_INVAL, "cutoff and dt must be positive");
    for (int k = 0; k < 3; k++) {
        if (d->cells[k] < 3 || !(d->dim[k] > 0)) return fail(eng, TFG_E_INVAL, "need at least 3 cells per axis");
        const float h = d->dim[k] / d->cells[k];
        const float ih = 1.0 / h;
        if ((int)std::ceil(d->cutoff * ih) != 1)
            return fail(eng, TFG_E_INVAL, "cell edge must be at least the cutoff (27-cell stencil)");
    }
    SimHost S;
    S.desc = *d;
    SimParams &P = S.P;
    std::memset(&P, 0, sizeof(P));
    for (int k = 0; k < 3; k++) {
        P.dim[k] = d->dim[k];
        P.cdim[k] = d->cells[k];
        P.h[k] = P.dim[k] / P.cdim[k];
    }
    P.ncells = P.cdim[0] * P.cdim[1] * P.cdim[2];
    P.cutoff = d->cutoff;
    P.cutoff2 = d->cutoff * d->cutoff;
    P.cut_hi = P.cutoff2 * (1.f + 2e-6f + 1.2e-5f * (std::max(P.h[0], std::max(P.h[1], P.h[2])) / P.cutoff));
    P.dt = d->dt;
    const float frac = d->particle_max_dist_fraction > 0 ? d->particle_max_dist_fraction : 0.05f;
    for (int k = 0; k < 3; k++) {
        P.h2[k] = 2. * P.h[k];
        P.maxx[k] = P.h[k] * frac;
        P.maxx2[k] = P.maxx[k] * P.maxx[k];
        P.maxv[k] = P.maxx[k] / P.dt;
        P.maxv2[k] = P.maxv[k] * P.maxv[k];
    }
    P.inv_cutoff = 1.0f / P.cutoff;
    P.self_density = (float)(1.0 / (3.14159265358979323846 * (double)P.cutoff * P.cutoff * P.cutoff));
    P.dpd_delta = 1.f / std::sqrt(P.dt);
    P.max_type = d->max_type;
    P.nspec = d->nr_species;
    P.nr_fluxsteps = d->nr_fluxsteps > 0 ? d->nr_fluxsteps : 1;
    P.dt_flux = P.dt / (float)P.nr_fluxsteps;   // tfSimulator.cpp:653
    P.flags = d->flags;
    P.seed = d->seed;
    // engine_verlet_update (tfEngine.cpp:231): skin = min(h) - cutoff, in FP32
    P.skin = std::fmin(P.h[0], std::fmin(P.h[1], P.h[2])) - P.cutoff;
    P.verlet_rebuild = 2;
    P.stop_at = -1;
    S.maxc = std::max(P.cdim[0], std::max(P.cdim[1], P.cdim[2]));
    S.orig.assign((size_t)3 * S.maxc, 0.f);
    for (int k = 0; k < 3; k++)
        for (int l = 0; l < P.cdim[k]; l++) S.orig[(size_t)k * S.maxc + l] = d->origin[k] + l * P.h[k];
    const int T = eng->max_type;
    S.pots.resize(T * T);
    for (auto &p : S.pots) std::memset(&p, 0, sizeof(p));
    S.tables.assign(T * T, std::vector<float>());
    FluxSet empty;
    std::memset(&empty, 0, sizeof(empty));
    S.fluxes.assign(T * T, empty);
    S.rforce.assign(T, make_float4(0, 0, 1, 0));
    S.mass.assign(T, 1.0f);
    S.dyn.assign(T, TFG_NEWTONIAN);
    S.species_flags.assign(kMaxSpecies, 0u);
    for (int w = 0; w < 6; w++) {
        std::memset(&S.walls[w], 0, sizeof(tfg_boundary));
        S.walls[w].kind = TFG_BOUNDARY_PERIODIC;
        S.walls[w].restore = 1.f;
    }
    S.wpots.resize(6 * T);
    for (auto &p : S.wpots) std::memset(&p, 0, sizeof(p));
    S.wtables.assign(6 * T, std::vector<float>());
    resolve_boundaries(S);
    eng->sims.push_back(std::move(S));
    if (out) *out = (int)eng->sims.size() - 1;
    return TFG_OK;
}

int load_sim(tfg_engine *eng, int sim, int n, const float *xg, const int32_t *cellv, const float *xrel,
             const float *v, const int32_t *type, const float *radius, const float *imass, const uint32_t *flags,
             const float *species, const float *force_i) {
    int rc = sim_check(eng, sim);
    if (rc) return rc;
    if (n < 0 || (n > 0 && !xg && !(cellv && xrel))) return fail(eng, TFG_E_INVAL, "positions missing");
    SimHost &S = eng->sims[sim];
    const int T = eng->max_type, ns = eng->nspec;
    if (type)
        for (int i = 0; i < n; i++)
            if (type[i] < 0 || type[i] >= T) return fail(eng, TFG_E_INVAL, "particle type out of range");
    if (cellv)
        for (int i = 0; i < n; i++)
            if (cellv[i] < 0 || cellv[i] >= S.P.ncells) return fail(eng, TFG_E_RANGE, "cell out of range");
    auto cp = [](std::vector<float> &dst, const float *src, size_t cnt) {
        if (src) dst.assign(src, src + cnt);
        else dst.clear();
    };
    S.pending_binned = !xg;
    cp(S.x, xg, (size_t)3 * n);
    cp(S.xrel, xrel, xg ? 0 : (size_t)3 * n);
    if (!xg) S.cell.assign(cellv, cellv + n);
    else S.cell.clear();
    cp(S.v, v, (size_t)3 * n);
    cp(S.radius, radius, n);
    cp(S.imass, imass, n);
    cp(S.species, species, (size_t)n * ns);
    cp(S.force_i, force_i, (size_t)3 * n);
    if (force_i && !eng->has_ext) {
        eng->has_ext = true;
        eng->gen++;
    }
    S.type.assign(n, 0);
    if (type) std::memcpy(S.type.data(), type, sizeof(int32_t) * n);
    if (flags) S.flags.assign(flags, flags + n);
    else S.flags.clear();
    S.n = n;
    S.loaded = true;
    S.pending = true;
    S.time = 0;
    S.q_pending.clear();
    S.P.verlet_rebuilds = 0;
    S.P.verlet_maxdx = 0.f;
    eng->layout_dirty = true;
    return TFG_OK;
}

// Work items of the tiled pass: the most home particles of one, and whether one may span several
// cells.  A small arena leaves warps without an item, and its time is that of the longest one,
// a crowded cell's; larger items share more.  Particles stand for the items a warp gets: of that,
// kinds of systems differ, so that each line lies among the sizes where the two sides meet.
// Microseconds a step, each side with the work split that is best for it:
//   8 or 16 homes, 24,000       cells 20,000 40.3 43.8, 24,000 46.6 46.2, 32,000 50.6 47.9; LJ fluids
//                               20,000 38.0 35.7, 33,000 48.3 43.8; DPD 10,000 35.7 35.8, 24,000
//                               44.1 39.7, 28,000 44.7 46.4, 50,000 53.8 54.1, 80,000 69.4 63.3
//   16 or 32, tables, 110,000   LJ 80,000 61.2 62.4, 110,592 72.4 72.2, 148,877 84.2 81.1; cells 80,000
//                               67.0 75.2, 110,000 78.0 82.1, 130,000 86.6 86.7, 150,000 94.5 93.2,
//                               200,000 109.7 107.2, 300,000 142.0 132.0
//   16 or 32, DPD, never        100,000 particles 77 81, 200,000 109.3 107.7, 300,000 146.5 149.8,
//                               400,000 198.5 193.6, 2,000,000 967 1007: pairs cost more each and
//                               droplets spread out, so that balance counts at every size
//   32 without or with runs     cells 300,000 132.0 136.6, 400,000 164.0 167.2, 450,000 186.8 181.7,
//   of cells, tables, 400,000   600,000 232.3 232.1, 2,000,000 696.6 681.4; LJ 300,763 129.6 127.8,
//                               405,224 165.1 160.5, 1,000,000 365.1 349.5; 80 and 256 tissues of 0.7
//                               and 3.0 million cells 281.9 282.7, 1,115.6 1,092.1
// Runs share set-up and targets, most where cells hold few particles (DPD droplets that have spread
// out: 77 -> 38 us a pass), but leave fewer items.
static void plan_items(tfg_engine *eng) {
    const bool pairs_cost = eng->has_dpd || (eng->has_flux && eng->nspec > 0);
    eng->homes = eng->n < 24000 ? 8 : (pairs_cost || eng->n < 110000 ? 16 : 32);
    eng->runs = pairs_cost || eng->n >= 400000;
}

int bin(tfg_engine *eng, int shuffle, bool timed) {
    BinArgs b;
    b.stamp = timed ? eng->stamps : nullptr;
    b.n = eng->n;
    b.cap = eng->cap;
    b.ncells = eng->ncells;
    b.nspec = eng->nspec;
    b.shuffle = shuffle;
    b.sims = eng->sims_dev;
    b.cell_sim = eng->cell_sim;
    b.src = eng->A[eng->cur];
    b.dst = eng->A[eng->cur ^ 1];
    b.count = eng->count;
    b.start = eng->start;
    b.lidx = eng->lidx;
    b.slot_of_id = eng->nb + eng->na > 0 ? eng->slot_of_id : nullptr;
    b.tmp = eng->bin_tmp;
    b.part = eng->scan_part;
    b.pre = eng->scan_pre;
    b.ticket = eng->counters;
    b.items = eng->items;
    plan_items(eng);
    b.column = reinterpret_cast<const uchar4 *>(eng->column);
    b.homes = eng->homes;
    b.runs = eng->runs;
    b.nitems = reinterpret_cast<int *>(eng->counters + 1);
    b.nsims = (int)eng->order.size();
    b.red = eng->red;
    b.has_ext = eng->has_ext;
    b.has_rand = eng->has_rand;
    b.rforce = eng->rforce;
    b.force = eng->force;
    // (only a step takes reference positions: after the advance, verlet_rebuild still names the
    // step that is over)
    b.oldx = shuffle ? eng->oldx : nullptr;
    if (b.ncells == 0) return TFG_OK;
    launch_bin(b, eng->stream);
    eng->cur ^= 1;
    return TFG_OK;
}

int commit(tfg_engine *eng) {
    int rc;
    const bool relaid = eng->layout_dirty;
    if (eng->layout_dirty || eng->tables_dirty) eng->gen++;
    if (eng->layout_dirty && (rc = relayout(eng))) return rc;
    if (eng->tables_dirty && (rc = upload_tables(eng))) return rc;
    if (relaid) {
        if ((rc = bin(eng, 0))) return rc;
        CK(cudaStreamSynchronize(eng->stream));
        if ((rc = check_launch(eng))) return rc;
    }
    return TFG_OK;
}

PairKernelArgs pair_args(tfg_engine *eng) {
    ParticleArrays &A = eng->A[eng->cur];
    PairKernelArgs a;
    std::memset(&a, 0, sizeof(a));
    a.sims = eng->sims_dev;
    a.cell_sim = eng->cell_sim;
    a.cell_at = eng->cell_at;
    a.nsims = (int)eng->order.size();
    a.ncells = eng->ncells;
    a.max_type = eng->max_type;
    a.nspec = eng->nspec;
    a.flags = eng->flags_all;
    a.n = eng->n;
    a.pos = A.pos;
    a.vel = A.vel;
    a.aux = A.aux;
    a.fext = A.fext;
    a.pforce = A.pforce;
    a.cell = A.cell;
    a.start = eng->start;
    a.items = eng->items;
    a.homes = eng->homes;   // as the items were listed
    a.runs = eng->runs;
    a.nitems = reinterpret_cast<const int *>(eng->counters + 1);
    a.counter = eng->counters + 2;
    a.sval = A.sval;
    a.sq = A.sq;
    a.cap = eng->cap;
    a.force = eng->force;
    a.pots = eng->pots;
    a.potc = eng->potc;
    a.blob = eng->blob;
    a.blob_floats = eng->blob_floats;
    a.potc_tex = eng->potc_tex;
    a.blob_tex = eng->blob_tex;
    a.one = eng->one;
    a.one_flux = eng->one_flux;
    a.has_one = eng->has_one;
    a.fluxes = eng->fluxes;
    a.wpots = eng->wpots;
    a.has_wall_pots = eng->has_wall_pots;
    a.rforce = eng->rforce;
    a.pforce_out = A.pforce;
    a.red = eng->red;
    a.err = eng->err;
    a.has_dpd = eng->has_dpd;
    a.radii = eng->radii;
    a.flux_sub = -1;
    a.has_flux = eng->has_flux;
    return a;
}

// Deterministic mode runs the stencil kernel instead of the tiled one.
bool use_tile(const tfg_engine *eng) { return !eng->deterministic; }

int force_pass(tfg_engine *eng, bool bonded, bool timed) {
    cudaStream_t s = eng->stream;
    ParticleArrays &A = eng->A[eng->cur];
    PairKernelArgs a = pair_args(eng);
    if (timed && eng->max_fluxsteps <= 1) a.stamp = eng->stamps + 1;   // else stamped before the substeps
    if (eng->n > 0) {
        if (use_tile(eng)) {
            launch_pair_tile(a, eng->sms, false, tune_of(eng), s);
        } else {
            if (a.stamp) launch_stamp(a.stamp, 0, s);
            launch_pair(a, s);
        }
    }
    if (bonded) {
        launch_bonds(eng->nb, eng->sms, eng->sims_dev, eng->cell_sim, eng->bonds, eng->bond_slot, eng->bpots, eng->bblob,
                     eng->slot_of_id, A.pos, A.aux, A.cell, eng->force, eng->red, timed ? eng->stamps + 2 : nullptr, s);
        launch_angles(eng->na, eng->sms, eng->sims_dev, eng->cell_sim, eng->angles, eng->bpots, eng->bblob, eng->slot_of_id,
                      A.pos, A.cell, eng->force, eng->red, timed && eng->nb == 0 ? eng->stamps + 2 : nullptr, s);
    }
    return check_launch(eng);
}

// Flux substeps (tf_engine_advance.cpp:314-323): before the step's force pass, each
// simulation with nr_fluxsteps > 1 runs nr_fluxsteps - 1 flux-only passes over its pair set,
// each followed by Fluxes_integrate over all its particles with dt_flux.
int flux_substeps(tfg_engine *eng) {
    if (!eng->has_flux || eng->nspec == 0 || eng->max_fluxsteps <= 1 || eng->n == 0) return TFG_OK;
    cudaStream_t s = eng->stream;
    for (int sub = 0; sub < eng->max_fluxsteps - 1; sub++) {
        PairKernelArgs a = pair_args(eng);
        a.flux_sub = sub;
        launch_pair_fluxonly(a, eng->sms, use_tile(eng), s);
        ParticleArrays &A = eng->A[eng->cur];
        launch_flux_integrate(eng->n, eng->cap, eng->nspec, sub, eng->sims_dev, eng->cell_sim, A.cell, A.sval, A.sq,
                              eng->species_flags, s);
    }
    return check_launch(eng);
}

int enqueue_step(tfg_engine *eng, bool advance, bool timed) {
    cudaStream_t s = eng->stream;
    // the step's kernels stamp the phase boundaries themselves; without particles they do not run
    if (eng->n == 0 && timed)
        for (int k = 0; k < 5; k++) launch_stamp(eng->stamps, k, s);
    int rc = bin(eng, 1, timed);
    if (rc) return rc;
    if (timed && eng->max_fluxsteps > 1) launch_stamp(eng->stamps, 1, s);
    if ((rc = flux_substeps(eng))) return rc;
    rc = force_pass(eng, true, timed);
    if (rc) return rc;
    if (advance)
        launch_advance(eng->n, eng->cap, eng->nspec, (int)eng->order.size(), eng->sims_dev, eng->cell_sim, eng->A[eng->cur], eng->force,
                       eng->type_mass, eng->type_dyn, eng->species_flags, eng->oldx, eng->red, eng->err, eng->stamps,
                       timed ? 1 << 3 | (eng->nb + eng->na == 0) << 2 : 0, s);
    return check_launch(eng);
}

void advance_clocks(tfg_engine *eng) {
    for (int k : eng->order) {
        SimHost &S = eng->sims[k];
        if (S.P.stop_at < 0 || S.time < S.P.stop_at) S.time += 1;
    }
}

int one_step(tfg_engine *eng, bool advance, bool timed) {
    advance_clocks(eng);
    return enqueue_step(eng, advance, timed);
}

// Stop simulation `sim` once its clock reaches `step` (-1: run on).  A simulation in the
// arena gets the new value in its device parameters at once, in stream order; one not yet
// laid out takes it with the next re-layout.
int set_stop_sim(tfg_engine *eng, int sim, int64_t step) {
    int rc = sim_check(eng, sim);
    if (rc) return rc;
    if (step < -1) return fail(eng, TFG_E_INVAL, "stop step must be -1 or at least 0");
    SimHost &S = eng->sims[sim];
    S.P.stop_at = step;
    if (S.in_arena && !S.pending && eng->sims_dev) {
        const size_t q = (size_t)S.P.red_base / RED_COUNT;
        CK(cudaMemcpyAsync(reinterpret_cast<char *>(eng->sims_dev + q) + offsetof(SimParams, stop_at), &S.P.stop_at,
                           sizeof(int64_t), cudaMemcpyHostToDevice, eng->stream));
    }
    return TFG_OK;
}

void drop_graphs(tfg_engine *eng) {
    for (StepGraph &g : eng->graphs) {
        if (g.exec) cudaGraphExecDestroy(g.exec);
        g = StepGraph();
    }
}

// `steps` steps (1 or kGraphSteps) replayed from the graph captured for the current buffer.
int graph_steps(tfg_engine *eng, int steps) {
    const int p = eng->cur;
    StepGraph &G = eng->graphs[2 * p + (steps > 1)];
    if (!G.exec || G.gen != eng->gen) {
        if (G.exec) cudaGraphExecDestroy(G.exec);
        G = StepGraph();
        cudaGraph_t g = nullptr;
        CK(cudaStreamBeginCapture(eng->stream, cudaStreamCaptureModeThreadLocal));
        int rc = TFG_OK;
        for (int k = 0; k < steps && !rc; k++) rc = enqueue_step(eng, true, eng->phase_timing);
        cudaError_t e = cudaStreamEndCapture(eng->stream, &g);
        // the capture swapped the host's buffer index; the replay does the swap for real
        G.next = eng->cur;
        eng->cur = p;
        if (rc || e != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            return rc ? rc : fail(eng, TFG_E_CUDA, std::string("step capture: ") + cudaGetErrorString(e));
        }
        e = cudaGraphInstantiate(&G.exec, g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            G.exec = nullptr;
            return fail(eng, TFG_E_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
        }
        G.gen = eng->gen;
    }
    CK(cudaGraphLaunch(G.exec, eng->stream));
    eng->cur = G.next;
    for (int k = 0; k < steps; k++) advance_clocks(eng);
    return TFG_OK;
}

int run_steps(tfg_engine *eng, int nsteps) {
    // After any change of the captured launch arguments one step runs eagerly (it also sets
    // every kernel's launch attributes up); the others replay the captured step of the
    // current buffer parity.  With phase timing on, every step writes its phase stamps.
    // Between two graph launches the GPU idles about 5 us, a fifth of a small arena's step:
    // once a generation has replayed kGraphAfter steps, so that capturing more pays, they are
    // launched kGraphSteps at a time.
    for (int k = 0; k < nsteps;) {
        int rc, steps = 1;
        if (eng->use_graphs && eng->eager_gen == eng->gen) {
            if (eng->replayed >= kGraphAfter && nsteps - k >= kGraphSteps) steps = kGraphSteps;
            else eng->replayed++;
            rc = graph_steps(eng, steps);
        } else {
            rc = one_step(eng, true, eng->phase_timing);
            eng->eager_gen = eng->gen;
            eng->replayed = 0;
        }
        if (rc) return rc;
        k += steps;
    }
    return TFG_OK;
}

int tune_if_needed(tfg_engine *eng) {
    if (eng->split == 0) return autotune(eng);
    // A batch whose population changed by more than 4x since the autotuner ran (a served
    // batch that filled up or drained) re-times the work split, the knob that follows size.
    if (eng->tune_auto && (eng->n > 4 * eng->tuned_n || 4 * eng->n < eng->tuned_n)) return autotune(eng);
    return TFG_OK;
}

// Pick the tiled pair kernel's work split (warps per home cell) by timing each choice on
// the current state.  Every trial re-initialises the forces with a non-shuffling re-bin.  What the
// trials change is kept and put back, by particle id: after a step the first re-bin moves the
// particles that have left their cell to other slots.  So the engine state is unchanged.
int autotune(tfg_engine *eng) {
    // Arenas on tables whose simulations are all in Verlet mode take split 1 from 12,000 particles
    // on.  Trials double the time from the load to the first step there (2.5 ms without, 5.6 with
    // them on 262,144 particles, 6.4 and 12.7 on 1,000,000) and find nothing better: a step with
    // splits 1 and 2 takes 28.5 and 27.6 us on 8,000 particles, 39.5 and 41.3 on 15,625, 44.2 and
    // 47.4 on 32,768, 62.1 and 64.8 on 64,000 (skin 0.2 cutoffs; with 0.5, 79.6 and 76.7 on 64,000).
    bool verlet = !eng->has_dpd && !(eng->has_flux && eng->nspec > 0) && eng->n >= 12000;
    for (int k : eng->order) verlet &= (eng->sims[k].P.flags & TFG_ENGINE_VERLET) != 0;
    if (!use_tile(eng) || eng->n == 0 || verlet) {
        eng->split = 1;
        eng->tune_auto = true;
        eng->tuned_n = eng->n;
        return TFG_OK;
    }
    cudaStream_t s = eng->stream;
    const size_t nred = eng->order.size() * RED_COUNT;
    struct Kept {
        float4 *force = nullptr;
        float *sq = nullptr;
        double *red = nullptr;
        ~Kept() { cudaFree(force); cudaFree(sq); cudaFree(red); }
    } kept;
    int rc;
    if ((rc = dalloc(eng, &kept.force, eng->n)) || (rc = dalloc(eng, &kept.sq, (size_t)eng->n * eng->nspec)) ||
        (rc = dalloc(eng, &kept.red, nred)))
        return rc;
    launch_keep(eng->n, eng->cap, eng->nspec, false, eng->A[eng->cur], eng->force, kept.force, kept.sq, s);
    CK(cudaMemcpyAsync(kept.red, eng->red, sizeof(double) * nred, cudaMemcpyDeviceToDevice, s));
    // candidates: every work split of the tiled kernel (it sizes its grabs itself)
    std::vector<TileTune> cand;
    for (int split : {1, 2, 7, 14}) {
        TileTune t;
        t.split = split;
        cand.push_back(t);
    }
    // one timed launch of a candidate on freshly initialised forces (ms, or < 0 on error)
    auto trial = [&](const TileTune &tc) -> float {
        rc = bin(eng, 0);
        if (rc) return -1.f;
        PairKernelArgs a = pair_args(eng);
        cudaEventRecord(eng->ev[0], s);
        launch_pair_tile(a, eng->sms, false, tc, s);
        cudaEventRecord(eng->ev[1], s);
        const cudaError_t e = cudaEventSynchronize(eng->ev[1]);
        if (e != cudaSuccess) {
            rc = fail(eng, TFG_E_CUDA, std::string("cudaEventSynchronize: ") + cudaGetErrorString(e));
            return -1.f;
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, eng->ev[0], eng->ev[1]);
        return ms;
    };
    // every candidate is timed once (three times when a launch takes under 0.5 ms, where one
    // launch is too noisy to rank and three cost little); the three fastest are then timed
    // twice more and the best of their times decides
    std::vector<float> once(cand.size());
    for (size_t c = 0; c < cand.size(); c++) {
        if ((once[c] = trial(cand[c])) < 0.f) return rc;
        for (int rep = 0; rep < 2 && once[c] < 0.5f; rep++) {
            const float ms = trial(cand[c]);
            if (ms < 0.f) return rc;
            once[c] = std::min(once[c], ms);
        }
    }
    std::vector<size_t> order(cand.size());
    for (size_t c = 0; c < cand.size(); c++) order[c] = c;
    const size_t top = std::min<size_t>(3, cand.size());
    std::partial_sort(order.begin(), order.begin() + top, order.end(),
                      [&](size_t x, size_t y) { return once[x] < once[y]; });
    float best = 1e30f;
    TileTune best_t = cand[order[0]];
    for (size_t k = 0; k < top; k++) {
        float tmin = once[order[k]];
        for (int rep = 0; rep < 2; rep++) {
            const float ms = trial(cand[order[k]]);
            if (ms < 0.f) return rc;
            tmin = std::min(tmin, ms);
        }
        if (tmin < best) { best = tmin; best_t = cand[order[k]]; }
    }
    if ((rc = bin(eng, 0))) return rc;
    launch_keep(eng->n, eng->cap, eng->nspec, true, eng->A[eng->cur], eng->force, kept.force, kept.sq, s);
    CK(cudaMemcpyAsync(eng->red, kept.red, sizeof(double) * nred, cudaMemcpyDeviceToDevice, s));
    CK(cudaStreamSynchronize(s));
    eng->split = best_t.split;
    eng->tune_warps = best_t.warps;
    eng->tune_grab = best_t.grab;
    eng->tune_auto = true;
    eng->tuned_n = eng->n;
    eng->gen++;
    return check_launch(eng);
}

int download_sim(tfg_engine *eng, int sim, float *x, float *xrel, int32_t *cell, float *v, float *f, float *dens,
                 float *species, float *q) {
    int rc = sim_check(eng, sim);
    if (rc) return rc;
    // A simulation already in the arena is read where it lies, without re-laying the arena
    // out for other simulations' pending changes.
    if ((!eng->sims[sim].in_arena || eng->sims[sim].pending) && (rc = commit(eng))) return rc;
    SimHost &S = eng->sims[sim];
    const int n = S.n, ns = eng->nspec;
    if (n == 0) return TFG_OK;
    cudaStream_t s = eng->stream;
    // the wanted arrays are gathered into a buffer that the engine keeps (it grows to the
    // largest download), then copied
    struct { float *host, *dev; size_t count; } out[8] = {
        {x, nullptr, (size_t)3 * n},  {xrel, nullptr, (size_t)3 * n}, {v, nullptr, (size_t)3 * n},
        {f, nullptr, (size_t)3 * n},  {dens, nullptr, (size_t)n},     {ns ? species : nullptr, nullptr, (size_t)n * ns},
        {ns ? q : nullptr, nullptr, (size_t)n * ns}, {reinterpret_cast<float *>(cell), nullptr, (size_t)n}};
    size_t need = 0;
    for (auto &o : out) need += o.host ? o.count : 0;
    if ((rc = ensure(eng, &eng->stage, eng->stage_cap, need))) return rc;
    size_t at = 0;
    for (auto &o : out)
        if (o.host) {
            o.dev = eng->stage + at;
            at += o.count;
        }
    launch_gather(n, S.P.id_off, eng->cap, ns, S.P, eng->A[eng->cur], eng->force, out[0].dev, out[1].dev,
                  reinterpret_cast<int32_t *>(out[7].dev), out[2].dev, out[3].dev, out[4].dev, out[5].dev, out[6].dev, s);
    for (const auto &o : out)
        if (o.host) CK(cudaMemcpyAsync(o.host, o.dev, sizeof(float) * o.count, cudaMemcpyDeviceToHost, s));
    if ((rc = fetch_errors(eng))) return rc;
    CK(cudaStreamSynchronize(s));
    return read_err(eng, true);
}

int reductions_sim(tfg_engine *eng, int sim, tfg_reductions *out) {
    int rc = sim_check(eng, sim);
    if (rc) return rc;
    if (!out) return TFG_E_INVAL;
    std::memset(out, 0, sizeof(*out));
    SimHost &S = eng->sims[sim];
    out->steps = S.time;
    if (!S.in_arena) return TFG_OK;
    double r[RED_COUNT];
    CK(cudaMemcpyAsync(r, eng->red + S.P.red_base, sizeof(r), cudaMemcpyDeviceToHost, eng->stream));
    if ((rc = fetch_errors(eng))) return rc;
    CK(cudaStreamSynchronize(eng->stream));
    out->epot_nonbond = r[RED_EPOT_NONBOND];
    out->epot_bond = r[RED_EPOT_BOND];
    out->epot_angle = r[RED_EPOT_ANGLE];
    out->epot = out->epot_nonbond + out->epot_bond + out->epot_angle;
    out->kinetic = r[RED_KINETIC];
    out->virial = r[RED_VIRIAL];
    out->computed_volume = r[RED_VOLUME];
    for (int k = 0; k < kMaxSpecies; k++) out->species_total[k] = r[RED_SPECIES0 + k];
    out->migrations = (int64_t)r[RED_MIGRATIONS];
    return read_err(eng, true);
}

int verlet_sim(tfg_engine *eng, int sim, int64_t *rebuilds, float *maxdx) {
    int rc = sim_check(eng, sim);
    if (rc) return rc;
    SimHost &S = eng->sims[sim];
    SimParams P = S.P;
    if (S.in_arena && eng->sims_dev) {
        const auto it = std::find(eng->order.begin(), eng->order.end(), sim);
        if (it != eng->order.end()) {
            CK(cudaMemcpyAsync(&P, eng->sims_dev + (it - eng->order.begin()), sizeof(SimParams),
                               cudaMemcpyDeviceToHost, eng->stream));
            CK(cudaStreamSynchronize(eng->stream));
        }
    }
    if (rebuilds) *rebuilds = P.verlet_rebuilds;
    if (maxdx) *maxdx = P.verlet_maxdx;
    return read_err(eng);
}

void destroy(tfg_engine *eng) {
    if (eng->stream) cudaStreamSynchronize(eng->stream);
    drop_graphs(eng);
    for (int b = 0; b < 2; b++) free_particles(eng->A[b]);
    void *bufs[] = {eng->wpots, eng->stamps, eng->force, eng->count, eng->start, eng->lidx, eng->bin_tmp, eng->items,
                    eng->slot_of_id, eng->scan_part, eng->scan_pre, eng->counters, eng->cell_sim, eng->cell_at, eng->column,
                    eng->sims_dev, eng->corig, eng->pots, eng->potc, eng->blob, eng->fluxes, eng->rforce, eng->type_mass,
                    eng->type_dyn, eng->species_flags, eng->bonds, eng->bond_slot, eng->angles, eng->bpots,
                    eng->bblob, eng->red, eng->err, eng->oldx, eng->stage};
    for (cudaTextureObject_t t : {eng->potc_tex, eng->blob_tex})
        if (t) cudaDestroyTextureObject(t);
    for (void *p : bufs) cudaFree(p);
    for (int k = 0; k < 5; k++)
        if (eng->ev[k]) cudaEventDestroy(eng->ev[k]);
    if (eng->err_host) cudaFreeHost(eng->err_host);
    if (eng->own_stream && eng->stream) cudaStreamDestroy(eng->stream);
    delete eng;
}

}  // namespace tfg
