"""The binning and the tiled pair pass at the sizes where their launches change: arenas of one
cluster launch or four (8,192 particles and 16,384 cells), 8, 16 or 32 home particles per work
item (24,000 and 110,000 particles), runs of cells (400,000 particles), partly filled groups,
windows and tiles, cells of several items; one potential or several; and the graphs of several
steps. Cells and pair sets bit-exact against the oracle, forces and densities at its bar."""
import dataclasses

import numpy as np
import pytest

from helpers import FORCE_RTOL, force_error, make_gpu, make_oracle
from tfg import abi, configs
from tfg.engine import _potential

pytestmark = pytest.mark.gpu


def _cells(n, side=None):
    side = max(float((n / 0.5) ** (1.0 / 3.0)), 9.5) if side is None else side
    return configs.cell_sorting(n=n, side=side, seed=600 + n % 97)


def _dpd(n, ref=True):
    scale = (n / 100_000) ** (1.0 / 3.0)
    w = configs.dpd_droplets(n=n, side=max(40.0 * scale, 8.0), radius=max(12.0 * scale, 1.0), seed=3)
    return dataclasses.replace(w, flags=w.flags | abi.ENGINE_DPD_REFERENCE_RANDOM) if ref else w


def _clumps(n):
    """Every particle in a few clumps of up to 150: cells of several work items beside empty ones."""
    w = _cells(n, side=24.0)
    rng = np.random.default_rng(n)
    centre = rng.uniform(2.0, 22.0, size=(max(n // 150, 1), 3))
    x = centre[np.arange(n) % len(centre)] + rng.normal(0.0, 0.4, size=(n, 3))
    return dataclasses.replace(w, x=configs.in_box(x, 24.0))


def _sparse(cells):
    """400 particles in a box of the given grid."""
    w = _cells(400, side=9.5)
    dim = tuple(3.0 * c for c in cells)
    x = np.random.default_rng(5).uniform(0.0, 1.0, size=(400, 3)) * np.array([6.0, 7.0, dim[2]])
    return dataclasses.replace(w, x=x.astype(np.float32), dim=dim, cells=cells)


CASES = {"cells_%d" % n: (lambda n=n: _cells(n)) for n in
         (1, 2, 31, 33, 97, 1000, 8192, 8193, 16385, 23999, 24000, 109_999, 110_001, 399_999,
          400_001)}
CASES.update({"dpd_%d" % n: (lambda n=n: _dpd(n)) for n in (1, 64, 129, 3001, 8192, 16385, 24001, 250_001)})
CASES.update({"clumps_%d" % n: (lambda n=n: _clumps(n)) for n in (150, 1203, 6000, 26_001)})
# runs of one to four cells along z per work item: few particles a cell, columns of 3 to 9 cells
CASES.update({"thin_%d" % k: (lambda k=k: _thin(k)) for k in (3, 4, 5, 6, 7, 9)})
# one bond or angle to a thread and several
CASES.update({"bonded_%d" % n: (lambda n=n: configs.bonded_fluid(n=n, seed=9)) for n in (16 * 99, 16 * 17_000)})
CASES.update({"grid_%dx%dx%d" % c: (lambda c=c: _sparse(c)) for c in ((3, 3, 1820), (3, 3, 1821))})


def _thin(k):
    """1,000 particles, one or two per cell, in a box of k cells along z."""
    w = configs.lj_fluid(n=1000, seed=k)
    dim = (2.5 * 18, 2.5 * 1300 // (18 * k) * 1.0 + 10.0, 2.5 * k)
    rng = np.random.default_rng(k)
    x = rng.uniform(0.0, 1.0, size=(w.n, 3)) * np.array(dim)
    cells = tuple(max(3, int(d // 2.5)) for d in dim)
    return dataclasses.replace(w, x=np.minimum(x, np.array(dim) * (1 - 1e-6)).astype(np.float32), dim=dim, cells=cells)


@pytest.mark.parametrize("name", list(CASES))
def test_force_pass_at_the_edges(name):
    w = CASES[name]()
    g, o = make_gpu(w), make_oracle(w, threads=8)
    g.force_only()
    o.force_only()
    a, r = g.download(), o.download()
    assert np.array_equal(a["cell"], r["cell"]) and np.array_equal(a["xrel"], r["xrel"])
    gc, gh = g.pair_signature()
    oc, oh = o.signature()
    assert np.array_equal(gc, oc) and np.array_equal(gh, oh)
    assert force_error(a["f"], r["f"], o.fmag()) < FORCE_RTOL
    assert np.abs(a["density"] - r["density"]).max() <= 1e-5 * np.abs(r["density"]).max()


def test_potentials_replaced():
    """Tables, DPD, one table for all types, tables again on one engine: the pair pass reads each
    set another way, and the table buffers grow under it."""
    w = _cells(3000)
    g, o = make_gpu(w), make_oracle(w)
    spec = list(w.pots.values())
    dpd = _dpd(8).pots
    sets = [[next(iter(dpd.values()))] * len(spec), [spec[0]] * len(spec), spec]
    keep = []
    for specs in [None] + sets:
        for e in (g, o):
            for (ti, tj), q in zip(w.pots, specs or []):
                keep.append(_potential(q, None, getattr(e, "potential_from_spec", None)))
                e.set_potential(ti, tj, keep[-1].ptr)
            e.force_only()
        a, r = g.download(), o.download()
        if specs is None or specs[0] not in dpd.values():   # (DPD draws differ)
            assert force_error(a["f"], r["f"], o.fmag()) < FORCE_RTOL
        assert np.array_equal(g.pair_signature()[1], o.signature()[1])


@pytest.mark.parametrize("name", ["dpd", "cells"])
def test_signature_after_a_step(name):
    """The pair set of a state that was advanced but not binned again: cells as binned before the
    step, positions after it, also for particles that have left their cell."""
    w = _dpd(3001, ref=False) if name == "dpd" else _cells(3001)
    g = make_gpu(w)
    g.step(30)
    c0 = g.download()["cell"].astype(np.int64)
    g.step(1)
    d = g.download()
    assert (d["cell"] != c0).any()
    dims = np.array(w.cells)
    loc = np.stack([c0 // (dims[1] * dims[2]), c0 // dims[2] % dims[1], c0 % dims[2]], axis=1)
    h = np.array(w.dim, np.float64) / dims
    count, _ = g.pair_signature()
    x = d["xrel"].astype(np.float64)
    low, high = np.zeros(w.n, int), np.zeros(w.n, int)
    for i in range(w.n):
        off = loc - loc[i]
        off -= dims * np.rint(off / dims).astype(np.int64)
        r = np.sqrt((((x - x[i]) + off * h) ** 2).sum(axis=1))
        near = (np.abs(off) <= 1).all(axis=1)
        near[i] = False
        low[i], high[i] = (near & (r < w.cutoff * (1 - 1e-5))).sum(), (near & (r < w.cutoff * (1 + 1e-5))).sum()
    assert (low <= count).all() and (count <= high).all()


@pytest.mark.parametrize("n", [500, 16385])
def test_steps_in_graphs_of_several(n):
    """One call of 45 steps (single and several-step graphs) and 45 calls give the same bits in
    deterministic mode."""
    w = _cells(n)
    a, b = make_gpu(w), make_gpu(w)
    for e in (a, b):
        e.set_deterministic(True)
    a.step(45)
    for _ in range(45):
        b.step(1)
    x, y = a.download(), b.download()
    for k in ("cell", "xrel", "v", "f", "density"):
        assert np.array_equal(x[k], y[k]), k
    assert a.reductions().steps == b.reductions().steps == 45


def test_download_of_some_arrays():
    w = _dpd(1500, ref=False)
    g = make_gpu(w)
    g.step(3)
    full = g.download()
    f = np.zeros((w.n, 3), np.float32)
    s = np.zeros((w.n, 1), np.float32)
    cell = np.zeros(w.n, np.int32)
    fp = lambda a: a.ctypes.data_as(abi.F_P)
    assert g.L.tfg_download(g.h, None, None, cell.ctypes.data_as(abi.I_P), None, fp(f), None, fp(s), None) == 0
    assert np.array_equal(f, full["f"]) and np.array_equal(s, full["species"]) and np.array_equal(cell, full["cell"])
    assert g.L.tfg_download(g.h, *([None] * 8)) == 0
