"""The FP64 prune where clusters are long: nothing but pairs a little inside
the cutoff, far apart along z, so that the eight atoms of a cluster spread over
up to 10,000 A.  The pairs counted are those of a direct count, pruned or not,
and pruned forces equal unpruned ones to the fixed-point rounding."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

from md_b200 import abi, engine
from tests import helpers as H

pytestmark = pytest.mark.gpu
PHYS, FP64 = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64


def _dimers(n, lx, spacing, seed=4):
    """n pairs of opposite unit charges 9.9 to 9.999 A apart, one per `spacing` along z."""
    rng = np.random.default_rng(seed)
    box = np.array([lx, lx, n * spacing])
    o = np.stack([rng.uniform(0, lx, n), rng.uniform(0, lx, n), (np.arange(n) + rng.uniform(0.3, 0.7, n)) * spacing], 1)
    d = rng.normal(0.0, 1.0, (n, 3))
    d *= rng.uniform(9.9, 9.999, (n, 1)) / np.linalg.norm(d, axis=1, keepdims=True)
    x = np.stack([o, o + d], 1).reshape(-1, 3)
    return x, np.tile([1.0, -1.0], n), box


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("n,lx,spacing", [(48, 26.0, 12.0), (48, 26.0, 40.0), (48, 26.0, 300.0), (48, 26.0, 1500.0),
                                          (48, 26.0, 9000.0), (8500, 600.0, 15.0)])
def test_fp64_prune_keeps_every_pair_of_long_clusters(n, lx, spacing, layout):
    x, q, box = _dimers(n, lx, spacing)
    w = x - box * np.floor(x / box)
    want = len(cKDTree(np.minimum(w, np.nextafter(box, 0)), boxsize=box).query_pairs(10.0))
    assert want >= n
    flat = H.simple_flat(q)
    # alpha 0.13: a pair at the cutoff still pulls with about 0.3 kcal/mol/A
    common = dict(semantics=PHYS, precision=FP64, ewald_tol=0.1, grid=(24, 24, 64))
    res = []
    for every in (1, 0):
        eng = engine.Engine(flat, box, prune_every=every, pair_layout=layout if every else 0, **common)
        eng.set_positions(x)
        res.append(eng.compute()[1])
        assert eng.pairlist_info()["pairs_in_cutoff"] == want, every
        eng.close()
    # at most 2 additions per entry, of fewer than 64 entries, each rounded to 2^-32
    assert np.abs(res[0] - res[1]).max() <= 128 * 2.0 ** -33
