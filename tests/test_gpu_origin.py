"""Boxes whose origin is not zero: the cell origins are then rounded, and shifts across a periodic
face are differences of the size of the box.  Pair sets bit-exact against the oracle for pairs laid
within 2e-5 of the cutoff across the z faces of long boxes, where work items span several cells."""
import dataclasses

import numpy as np
import pytest

from helpers import make_gpu, make_oracle
from tfg import abi, configs

pytestmark = pytest.mark.gpu

# cells along z, cell edge, origin
BOXES = [(512, 1.0028567, 0.49892256699), (500, 514.09 / 500, 0.0066), (250, 257.51 / 250, 8.71),
         (128, 1.02058, -0.8615), (300, 1.01, -151.3), (3, 1.01, 77.7), (512, 1.0028567, 0.0)]
COLUMNS = 12


def _seam(cells, edge, origin):
    """A DPD box of 12 x 12 columns.  Each has three pairs across its upper z face, three across the
    face to a neighbouring column (whose partner in the walk sits at the lower face), all of them at
    0 to 2e-5 below or above the cutoff, and a particle two cells from either face, so that the
    items at the faces span several cells."""
    f32 = np.float32
    dim = (1.1 * COLUMNS, 1.1 * COLUMNS, edge * cells)
    w = configs.dpd_droplets(n=8, side=8.0, radius=2.0, seed=1)
    w = dataclasses.replace(w, origin=(0.3, -7.7, origin), dim=dim, cells=(COLUMNS, COLUMNS, cells),
                            flags=w.flags | abi.ENGINE_DPD_REFERENCE_RANDOM)
    h = [f32(f32(d) / f32(c)) for d, c in zip(dim, w.cells)]
    corig = [f32(o) + np.arange(c, dtype=f32) * k for o, c, k in zip(w.origin, w.cells, h)]

    def shift(k, a, b):
        s = float(f32(corig[k][b] - corig[k][a]))
        return s - float(f32(dim[k])) if 2 * s > dim[k] else (s + float(f32(dim[k])) if 2 * s < -dim[k] else s)

    rng = np.random.default_rng(cells)
    at, x = [], []
    top, wide = cells - 1, float(h[0])
    for i in range(COLUMNS):
        for j in range(COLUMNS):
            for lk in {min(1, top), max(top - 2, 0)}:
                at.append((i, j, lk))
                x.append((0.9 * wide, 0.1 * wide, 0.02))
            for k in range(6):
                r = 1.0 + rng.uniform(-2e-5, 2e-5)
                up = k < 3                      # from the top cell over the face, or from cell 0 below it
                e = np.array([rng.uniform(-0.2, 0.2), rng.uniform(-0.2, 0.2) if up else rng.uniform(0.4, 0.6), 0.0])
                e[2] = np.sqrt(1.0 - e @ e) * (1 if up else -1)
                d = r * e
                a = (i, j, top if up else 0)
                b = (i, j if up else (j + 1) % COLUMNS, 0 if up else top)
                z0 = float(h[2]) - d[2] if up else 0.0    # z of the first such that the second is in its cell
                p = np.array([rng.uniform(0.3, 0.7) * wide, rng.uniform(0.3, 0.7) * wide if up else wide - 0.2,
                              rng.uniform(z0 + 0.02, float(h[2]) - 0.02) if up else rng.uniform(0.02, -d[2] - 0.02)])
                p = p.astype(f32).astype(np.float64)
                at += [a, b]
                x += [tuple(p), tuple(p + d - [shift(q, a[q], b[q]) for q in range(3)])]
    at, x = np.array(at), np.array(x, np.float32)
    assert (x >= 0).all() and (x < np.array(h)).all()
    n = len(x)
    cell = (at[:, 0] * COLUMNS + at[:, 1]) * cells + at[:, 2]
    ones = np.ones(n, np.float32)
    w = dataclasses.replace(w, x=np.zeros((n, 3), np.float32), v=np.zeros((n, 3), np.float32), type=np.zeros(n, np.int32),
                            radius=ones, imass=ones, species=np.zeros((n, 1), np.float32))
    return w, cell.astype(np.int32), x


@pytest.mark.parametrize("box", BOXES, ids=lambda b: "%d_%g" % (b[0], b[2]))
@pytest.mark.parametrize("split", [1, 7])
def test_pairs_at_the_cutoff_across_a_face(box, split):
    w, cell, xrel = _seam(*box)
    w = dataclasses.replace(w, x=np.tile(np.float32([1.0, -7.0, box[2] + 1.0]), (len(cell), 1)))   # replaced below
    g, o = make_gpu(w), make_oracle(w, threads=8)
    for e in (g, o):
        e.load_binned(cell, xrel, type=w.type, species=w.species)
    g.set_split(split)
    g.force_only()
    o.force_only()
    gc, gh = g.pair_signature()
    oc, oh = o.signature()
    assert np.array_equal(gc, oc), "%d of %d particles' pairs differ" % (int((gc != oc).sum()), len(oc))
    assert np.array_equal(gh, oh)
