"""The binning and the tiled pair pass at the sizes where their launches change: arenas of one
cluster launch or four (16,384 particles and 16,384 cells), 8, 16 or 32 home particles per
work item (24,000 and 100,000 particles), partly filled groups, windows and tiles, cells of
several items; and the graphs of several steps.  Cells and pair sets bit-exact against the
oracle, forces and densities at its bar."""
import dataclasses

import numpy as np
import pytest

from helpers import FORCE_RTOL, force_error, make_gpu, make_oracle
from tfg import abi, configs

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
         (1, 2, 31, 33, 97, 1000, 8191, 8193, 16384, 16385, 23999, 24000, 99_999, 100_001)}
CASES.update({"dpd_%d" % n: (lambda n=n: _dpd(n)) for n in (1, 64, 129, 3001, 16385, 24001)})
CASES.update({"clumps_%d" % n: (lambda n=n: _clumps(n)) for n in (150, 1203, 6000, 26_001)})
CASES.update({"grid_%dx%dx%d" % c: (lambda c=c: _sparse(c)) for c in ((3, 3, 1820), (3, 3, 1821))})


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
