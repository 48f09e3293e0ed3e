"""Performance cases of the per-step particle path, run through the public entry points.

A case is a dict of plain values.  Its "kind" names the model, its "call" what a program does
in one pass:
  step    tfg_step(steps), then a download of the particle state the program works on next
          (a frame of an interactive run, a sample of a trajectory);
  force   tfg_force_only, then a download of forces, densities and flux increments (the
          reference's offload hooks engine_force_prep + engine_nonbond_cuda);
  job     a whole request: a new batch, its simulations loaded from host arrays, all steps,
          every simulation downloaded.
Downloads go to page-locked buffers that the program keeps, with only the wanted arrays asked
for, as a host program in C++ does; `job` uses the Python download call.

Multi-step passes return velocities and forces of every particle, not positions and number
densities: a particle within rounding of a box face is reported on either side of the box, and
the number density jumps as a pair crosses the cutoff, so neither can be compared between two
runs whose sums were taken in another order.  For the same reason starts have no overlaps
(jittered lattices) except where the potential is soft (DPD).
"""
import ctypes as C
import dataclasses
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tissue-forge_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from tfg import abi, configs  # noqa: E402
from tfg.engine import Batch, Engine, TfgError, setup_model  # noqa: E402

F_P, I_P = abi.F_P, abi.I_P


def listed():
    return [
        # One step of a very small tissue, read back at once: an interactive program that
        # steps and draws.  Latency and launches are all there is.
        dict(name="cells_500_one_step", kind="cells", call="step", n=500, steps=1),
        # The reference's cell-sorting demo size: twenty steps between two frames.
        dict(name="cells_4000", kind="cells", call="step", n=4000, steps=20),
        # One member of a large served stream: a tissue of 150,001 cells (an odd count).
        dict(name="cells_150001", kind="cells", call="step", n=150_001, steps=20),
        # Two DPD droplets with one diffusing species, the full-size single simulation.
        dict(name="dpd_100000", kind="dpd", call="step", n=100_000, steps=20),
        # The DPD droplets with three species: one force pass through the offload hook.
        dict(name="dpd3_force_60000", kind="dpd3", call="force", n=60_000, steps=1),
        # A mid-size tissue through the offload hook.
        dict(name="cells_force_30000", kind="cells", call="force", n=30_000, steps=1),
        # Lennard-Jones fluid with cell lists, 125^3 particles.
        dict(name="lj_1953125", kind="lj", call="step", n=125 ** 3, steps=10),
        # The same physics in Verlet mode (skin 0.2 cutoffs, device pair lists).
        dict(name="lj_verlet_262144", kind="lj_verlet", call="step", n=64 ** 3, steps=20),
        # Chains of 16 with bonds and angles in a Lennard-Jones fluid, the largest single simulation.
        dict(name="bonded_2000000", kind="bonded", call="step", n=2_000_000, steps=10),
        # The parameter sweep: 256 independent tissues of 500 to 50,000 cells in one batch,
        # thirty steps between two samples of the trajectories.
        dict(name="ensemble_256", kind="ensemble", call="step", sims=256, nmin=500, nmax=50_000, steps=30),
        # A served batch of DPD requests of 1,000 to 50,000 particles.
        dict(name="dpd_batch_24", kind="dpd_batch", call="step", sims=24, nmin=1000, nmax=50_000, steps=20),
        # A small request from arrival to result: set-up, upload, 50 steps, download.
        dict(name="dpd_job_4", kind="dpd_batch", call="job", sims=4, nmin=1000, nmax=8000, steps=50),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cells", "cells", "cells_force", "dpd", "dpd3_force", "lj", "lj_verlet", "bonded", "ensemble",
                       "dpd_batch", "dpd_job"])
    if kind == "cells":
        n = _log(rng, 500, 300_000)
        return dict(kind="cells", call="step", n=n, steps=rng.choice([1, 5, 20]) if n < 20_000 else 20)
    if kind == "cells_force":
        return dict(kind="cells", call="force", n=_log(rng, 500, 60_000), steps=1)
    if kind == "dpd":
        return dict(kind="dpd", call="step", n=_log(rng, 1000, 200_000), steps=20)
    if kind == "dpd3_force":
        return dict(kind="dpd3", call="force", n=_log(rng, 1000, 80_000), steps=1)
    if kind in ("lj", "lj_verlet"):
        return dict(kind=kind, call="step", n=_log(rng, 16, 100) ** 3, steps=10)
    if kind == "bonded":
        return dict(kind="bonded", call="step", n=16 * _log(rng, 200, 50_000), steps=10)
    if kind == "ensemble":
        return dict(kind="ensemble", call="step", sims=_log(rng, 4, 128), nmin=500, nmax=_log(rng, 2000, 50_000), steps=30)
    if kind == "dpd_batch":
        return dict(kind="dpd_batch", call="step", sims=_log(rng, 4, 32), nmin=1000, nmax=_log(rng, 4000, 50_000), steps=20)
    return dict(kind="dpd_batch", call="job", sims=_log(rng, 2, 8), nmin=1000, nmax=_log(rng, 2000, 10_000), steps=50)


# ---------------------------------------------------------------- workloads

def _lattice(n, side, rng, jitter, snake=False):
    """n sites of the smallest cubic lattice that holds them, jittered by a fraction of its
    spacing; chosen at random, or with `snake` the first n along a path of neighbours."""
    m = 1
    while m ** 3 < n:
        m += 1
    a = side / m
    if snake:
        s = np.arange(n, dtype=np.int64)
        i, r = s // (m * m), s % (m * m)
        j, k = r // m, r % m
        line = i * m + j
        k = np.where(line % 2 == 1, m - 1 - k, k)
        j = np.where(i % 2 == 1, m - 1 - j, j)
    else:
        s = rng.permutation(m ** 3)[:n] if n < m ** 3 else np.arange(n)
        i, j, k = s // (m * m), (s // m) % m, s % m
    x = (np.stack([i, j, k], axis=1) + 0.5) * a
    return configs.in_box(x + rng.uniform(-jitter * a, jitter * a, size=x.shape), side)


def _cells(n, seed, depth_ab=0.5, random_force=None):
    side = float((n / 0.5) ** (1.0 / 3.0))
    w = configs.cell_sorting(n=n, side=side, depth_ab=depth_ab, seed=seed, random_force=random_force)
    # a time step that resolves the steep wells: trajectories of two runs stay comparable
    return dataclasses.replace(w, x=_lattice(n, side, np.random.default_rng([seed, 11]), 0.15), dt=0.001)


def _sizes(case, rng):
    return np.exp(rng.uniform(math.log(case["nmin"]), math.log(case["nmax"]), size=case["sims"])).astype(np.int64)


def _workloads(case, seed):
    """The simulations of a case: one, or a batch's members (their sizes are the case's own)."""
    kind = case["kind"]
    seed = int(seed) % (1 << 30)
    if kind == "cells":
        return [_cells(case["n"], seed)]
    if kind in ("dpd", "dpd3"):
        n = case["n"]
        scale = (n / 100_000) ** (1.0 / 3.0)
        make = configs.dpd_droplets if kind == "dpd" else configs.dpd_droplets_species
        return [make(n=n, side=max(40.0 * scale, 8.0), radius=12.0 * scale, seed=seed)]
    if kind in ("lj", "lj_verlet"):
        w = configs.lj_fluid(n=case["n"], seed=seed)
        return [configs.verlet(w) if kind == "lj_verlet" else w]
    if kind == "bonded":
        w = configs.bonded_fluid(n=case["n"], seed=seed)
        rng = np.random.default_rng([seed, 13])
        x = _lattice(w.n, w.dim[0], rng, 0.05, snake=True)
        v = rng.normal(0.0, math.sqrt(0.5), size=(w.n, 3)).astype(np.float32)
        return [dataclasses.replace(w, x=x, v=v)]
    rng = np.random.default_rng([case["sims"], case["nmax"], 17])
    ns = _sizes(case, rng)
    depth = rng.uniform(0.1, 2.0, size=case["sims"])
    if kind == "ensemble":
        return [_cells(int(n), seed + 7919 * i, float(d), (0.0, 0.1, 1)) for i, (n, d) in enumerate(zip(ns, depth))]
    ws = []
    for i, n in enumerate(ns):
        scale = (int(n) / 100_000) ** (1.0 / 3.0)
        ws.append(configs.dpd_droplets(n=int(n), side=max(40.0 * scale, 8.0), radius=12.0 * scale, seed=seed + 7919 * i))
    return ws


# ---------------------------------------------------------------- passes

class _Out:
    """Page-locked result arrays of one simulation."""

    def __init__(self, n, nspec, want):
        size = dict(x=3, v=3, f=3, density=1, species=nspec, q=nspec)
        self.t = {k: torch.zeros((n, size[k]) if size[k] != 1 or k in ("species", "q") else (n,), dtype=torch.float32).pin_memory()
                  for k in want if size[k] > 0}
        p = {k: C.cast(t.data_ptr(), F_P) for k, t in self.t.items()}
        self.args = (p.get("x"), None, None, p.get("v"), p.get("f"), p.get("density"), p.get("species"), p.get("q"))


class _State:
    pass


def _ok(rc, what):
    if rc != 0:
        raise TfgError(rc, what)


def prepare(case, seed):
    s = _State()
    s.case = case
    s.ws = _workloads(case, seed)
    if case["call"] == "job":
        return s
    nspec = s.ws[0].nr_species
    want = ["v", "f"] + (["species"] if nspec else [])
    if case["call"] == "force":
        want = ["f", "density"] + (["q"] if nspec else [])
    elif case["steps"] == 1:
        want = ["x", "v", "f", "density"]
    if case["kind"] in ("ensemble", "dpd_batch"):
        s.eng = Batch(s.ws[0].max_type, nspec)
        cache = {}
        s.sims = []
        for w in s.ws:
            sim = s.eng.add_sim(w.desc())
            s.eng._keep += setup_model(sim, w, pot_cache=cache)
            s.sims.append(sim)
    else:
        w = s.ws[0]
        s.eng = Engine(w.desc())
        s.eng._keep = setup_model(s.eng, w)
        s.sims = None
    s.out = [_Out(w.n, nspec, want) for w in s.ws]
    s.ws = None
    s.eng.autotune()
    s.eng.sync()
    return s


def run(s):
    case = s.case
    if case["call"] == "job":
        ws = s.ws
        b = Batch(ws[0].max_type, ws[0].nr_species)
        cache, sims = {}, []
        for w in ws:
            sim = b.add_sim(w.desc())
            b._keep += setup_model(sim, w, pot_cache=cache)
            sims.append(sim)
        b.step(case["steps"], sync=False)
        got = [sim.download() for sim in sims]
        b.close()
        return [{k: d[k] for k in ("v", "f", "species")} for d in got]
    e = s.eng
    L = e.L
    if case["call"] == "force":
        _ok(L.tfg_force_only(e.h, 1), "tfg_force_only")
    else:
        _ok(L.tfg_step(e.h, case["steps"]), "tfg_step")
    if s.sims is None:
        _ok(L.tfg_download(e.h, *s.out[0].args), "tfg_download")
    else:
        for sim, o in zip(s.sims, s.out):
            _ok(L.tfg_batch_download(e.h, sim.sid, *o.args), "tfg_batch_download")
    if len(s.out) <= 8:
        return [o.t for o in s.out]
    # one array over all members (the values are every member's own)
    return {k: torch.cat([o.t[k] for o in s.out]) for k in s.out[0].t}


def work(case):
    """Particle state read and written once per step (position and velocity 48 B, species and
    increment 8 B each; a force pass reads positions, types and radii and writes force and
    density), and the flops of every interacting pair, bond, angle and particle update."""
    kind = case["kind"]
    if "sims" in case:
        rng = np.random.default_rng([case["sims"], case["nmax"], 17])
        n = int(_sizes(case, rng).sum())
    else:
        n = case["n"]
    steps = case["steps"]
    if kind in ("cells", "ensemble"):
        pairs, per = n * 0.5 * 0.5 * 4.0 / 3.0 * math.pi * 27.0, 62
    elif kind in ("dpd", "dpd3", "dpd_batch"):
        pairs, per = 11.4 * n, 93 if kind == "dpd3" else 69
    else:
        pairs, per = n * 0.5 * 0.85 * 4.0 / 3.0 * math.pi * 2.5 ** 3, 62
    flops = pairs * per + 30.0 * n
    if kind == "bonded":
        flops += n * 15.0 / 16.0 * 45.0 + n * 14.0 / 16.0 * 75.0
    nspec = {"dpd": 1, "dpd_batch": 1, "dpd3": 3}.get(kind, 0)
    if case["call"] == "force":
        nbytes = n * (20.0 + 16.0 + (12.0 if kind == "dpd3" else 0.0) + 8.0 * nspec)
    else:
        nbytes = steps * n * (48.0 + 8.0 * nspec)
    return dict(bytes=nbytes, flops=flops * steps)


# ---------------------------------------------------------------- 64-bit values of the force cases

def _pairs(x, side, cutoff):
    """(i, j, dx, r) of every pair within the cutoff, i < j, minimum image, by brute force."""
    n = x.shape[0]
    ii, jj = [], []
    step = max(1, 40_000_000 // n)
    c2 = cutoff * cutoff
    for b in range(0, n, step):
        r2 = torch.zeros((min(step, n - b), n), dtype=x.dtype, device=x.device)
        for k in range(3):
            d = x[b:b + step, k, None] - x[None, :, k]
            d -= side * torch.round(d / side)
            r2 += d * d
        i, j = torch.nonzero(r2 <= c2, as_tuple=True)
        i = i + b
        keep = i < j
        ii.append(i[keep])
        jj.append(j[keep])
    i, j = torch.cat(ii), torch.cat(jj)
    dx = x[i] - x[j]
    dx -= side * torch.round(dx / side)
    return i, j, dx, dx.square().sum(1).sqrt()


def _gauss(seed, step, lo, hi):
    """The engine's normal deviate of a pair: Philox4x32-10 (Salmon et al., SC'11), Box-Muller."""
    m = 0xFFFFFFFF
    c = [torch.full_like(lo, step & m), lo.clone(), hi.clone(), torch.full_like(lo, 0xD0D0)]
    k0, k1 = seed & m, (seed >> 32) & m
    for _ in range(10):
        p0, p1 = 0xD2511F53 * c[0], 0xCD9E8D57 * c[2]
        c = [((p1 >> 32) & m) ^ c[1] ^ k0, p1 & m, ((p0 >> 32) & m) ^ c[3] ^ k1, p0 & m]
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    u = [((v >> 8).double() + 0.5) / 16777216.0 for v in c[:2]]
    return torch.sqrt(-2.0 * torch.log(u[0])) * torch.cos(2.0 * math.pi * u[1])


def exact(case, seed):
    """Forces, number densities and flux increments of a force pass in 64 bits: Morse (held
    constant below its table's start) or DPD with Fick fluxes; None for stepped cases, whose
    trajectories amplify rounding."""
    if case["call"] != "force":
        return None
    w = _workloads(case, seed)[0]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.from_numpy(w.x).to(dev).double()
    rc = float(w.cutoff)
    i, j, dx, r = _pairs(x, float(np.float32(w.dim[0])), rc)
    n = x.shape[0]
    if w.species is None:
        t = torch.from_numpy(w.type).to(dev)
        depth = torch.where(t[i] == t[j], 3.0, 0.5).double()
        y = torch.clamp(r, min=float(np.float32(1.01))) - 1.0
        mag = depth * 10.0 * (torch.exp(-10.0 * y) - torch.exp(-5.0 * y))   # -dV/dr
        q = None
    else:
        v = torch.from_numpy(w.v).to(dev).double()
        e = dx / r[:, None]
        om = 1.0 - r / rc
        xi = _gauss(int(w.seed), 1, torch.minimum(i, j), torch.maximum(i, j))
        mag = 10.0 * om - 4.5 * om * om * (e * (v[i] - v[j])).sum(1) + 3.0 * om * xi / math.sqrt(float(np.float32(w.dt)))
        s = torch.from_numpy(w.species).to(dev).double()
        q = torch.zeros_like(s)
        for (_, _, F) in w.fluxes:
            a = F.index_a
            term = om * om
            si, sj = s[i, a], s[j, a]
            fl = term * F.coef * (si - sj)
            q[:, a].index_add_(0, i, -fl - 0.5 * F.decay * si)
            q[:, a].index_add_(0, j, fl - 0.5 * F.decay * sj)
    pf = dx * (mag / r)[:, None]
    f = torch.zeros((n, 3), dtype=torch.float64, device=dev).index_add_(0, i, pf).index_add_(0, j, -pf)
    norm = 1.0 / (math.pi * rc ** 3)
    h = r / rc
    wd = (1.0 - 1.5 * h * h + 0.75 * h * h * h) * norm
    den = torch.full((n,), norm, dtype=torch.float64, device=dev).index_add_(0, i, wd).index_add_(0, j, wd)
    out = dict(f=f, density=den)
    if q is not None:
        out["q"] = q
    return [out]
