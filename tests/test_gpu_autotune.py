"""The autotuner on an engine that has stepped: it leaves the state as it was, also where
particles have moved to cells that the arena is not sorted by yet.  The reported launch shape."""
import numpy as np
import pytest

from helpers import make_gpu
from tfg import configs
from tfg.engine import Batch, setup_model

pytestmark = pytest.mark.gpu

CASES = {
    "dpd": lambda: configs.dpd_droplets(n=4000, side=12.0, radius=3.5, seed=7),
    "dpd_three_species": lambda: configs.dpd_droplets_species(n=4000, side=12.0, radius=3.5, seed=7),
    "cells": lambda: configs.cell_sorting(n=3000, side=18.0, seed=31, random_force=(0.0, 0.1, 1)),
    "bonded": lambda: configs.bonded_fluid(n=16 * 100, seed=9),
}


def _same(before, after):
    assert [k for k in before if not np.array_equal(before[k], after[k])] == []


@pytest.mark.parametrize("name", sorted(CASES))
def test_autotune_leaves_a_running_engine_unchanged(name):
    g = make_gpu(CASES[name]())
    g.step(10)
    c0 = g.download()["cell"]
    g.step(1)
    before, totals = g.download(), g.reductions()
    assert (before["cell"] != c0).any()          # migrants: the arena is not in cell order
    if name == "dpd_three_species":
        assert (before["q"] != 0).any()          # they keep their increments for the next step
    g.autotune()
    _same(before, g.download())
    after = g.reductions()
    for k in ("epot", "kinetic", "virial", "computed_volume", "migrations"):
        assert getattr(after, k) == getattr(totals, k), k


def test_autotune_leaves_the_members_of_a_batch_unchanged():
    ws = [configs.dpd_droplets(n=n, side=max(8.0, (n / 2.0) ** (1 / 3)), radius=3.0, seed=n) for n in (1500, 700, 4001)]
    b = Batch(ws[0].max_type, ws[0].nr_species)
    sims = []
    for w in ws:
        s = b.add_sim(w.desc())
        b._keep.extend(setup_model(s, w))
        sims.append(s)
    b.step(11)
    before = [s.download() for s in sims]
    assert any((d["q"] != 0).any() for d in before)
    b.autotune()
    for s, d in zip(sims, before):
        _same(d, s.download())


def test_autotune_keeps_the_verlet_reference_positions():
    """After a step that rebuilt, the displacements go on being measured from the rebuild."""
    w = configs.verlet(configs.lj_fluid(n=4000, density=0.8), skin=0.3)
    g, h = make_gpu(w), make_gpu(w)
    for e in (g, h):
        e.step(1)
    assert g.verlet()[0] == 1
    g.autotune()
    for e in (g, h):
        e.step(2)
    (rg, mg), (rh, mh) = g.verlet(), h.verlet()
    assert rg == rh == 1
    # positions of the two runs differ by the rounding of force sums taken in another order
    assert abs(mg - mh) <= 1e-3 * mh


@pytest.mark.parametrize("name,n,warps", [("cells", 3000, 4), ("cells", 120_000, 8), ("dpd", 120_000, 4)])
def test_tuning_reports_the_warps_of_a_block(name, n, warps):
    """Blocks have four warps where work items are small (up to 16 home particles), else eight, and
    what the caller fixes."""
    w = configs.cell_sorting(n=n, side=float((2 * n) ** (1 / 3)), seed=3) if name == "cells" else \
        configs.dpd_droplets(n=n, side=42.5, radius=12.75, seed=3)
    g = make_gpu(w)
    g.autotune()
    assert g.tuning()[1] == warps
    g.set_tuning(1, 12 - warps, 1)
    g.force_only()
    assert g.tuning() == (1, 12 - warps, 1)
    f = g.download()["density"]
    g = make_gpu(w)
    g.force_only()
    assert np.abs(f - g.download()["density"]).max() <= 1e-5 * f.max()
