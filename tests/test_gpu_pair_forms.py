"""The tiled pair pass against another walk of the same state (the stencil kernel of deterministic
mode) at full size in Verlet mode, and the work splits that the other pair-list tests leave out."""
import numpy as np
import pytest

from helpers import make_gpu, make_oracle, small_bonded, small_dpd
from tfg import configs

pytestmark = pytest.mark.gpu


def test_full_size_verlet_pairs_equal_the_stencil_walk():
    """2.0M-particle LJ fluid in Verlet mode, on a step that did not rebuild: particles sit up to
    half a skin outside their cells."""
    w = configs.verlet(configs.lj_fluid(n=2_000_000), skin=0.2)
    g = make_gpu(w)
    g.step(12)
    rebuilds, moved = g.verlet()
    assert rebuilds < 12 and moved > 0.0
    tc, th = g.pair_signature()
    g.set_deterministic(True)
    sc, sh = g.pair_signature()
    assert np.array_equal(tc, sc) and np.array_equal(th, sh)
    assert int(tc.sum()) // 2 > 50_000_000


CASES = {
    "cell_sorting": lambda: configs.cell_sorting(),
    "bonded": lambda: small_bonded(),
    "dpd": lambda: small_dpd(),
    "crowded": lambda: configs.cell_sorting(n=10_000, side=12.6, seed=22),
}


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("split", [2, 14])
def test_pair_list_of_every_split_equals_oracle(name, split):
    w = CASES[name]()
    g, o = make_gpu(w), make_oracle(w)
    g.set_split(split)
    o.record_pairs(True)
    g.force_only()
    o.force_only()
    p = np.sort(o.pairs().astype(np.int32), axis=1)
    assert np.array_equal(g.pair_list(), p[np.lexsort((p[:, 1], p[:, 0]))])
