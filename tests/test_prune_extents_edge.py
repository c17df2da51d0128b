"""The prune around the cluster extent (256 A) where it leaves the FP32 expansion:
pairs at 9.9 to 9.999 A in clusters of 50 to 600 A, pruned counts equal to a
direct count (FP64) and to unpruned ones (mixed)."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

from md_b200 import abi, engine
from tests import helpers as H
from tests.test_prune_extents import _dimers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("spacing", [2.0, 4.0, 6.0, 7.0, 8.0, 9.0, 11.0, 16.0])
def test_counts_on_both_sides(spacing, layout):
    x, q, box = _dimers(400, 26.0, spacing, seed=int(10 * spacing))
    w = x - box * np.floor(x / box)
    want = len(cKDTree(np.minimum(w, np.nextafter(box, 0)), boxsize=box).query_pairs(10.0))
    flat, n = H.simple_flat(q), {}
    for prec in (abi.MDF_PREC_FP64, abi.MDF_PREC_MIXED):
        for every in (0, 1):
            eng = engine.Engine(flat, box, precision=prec, ewald_tol=0.1, grid=(24, 24, 64), prune_every=every,
                                pair_layout=layout if every else 0)
            eng.set_positions(x)
            eng.compute()
            n[prec, every] = eng.pairlist_info()["pairs_in_cutoff"]
            eng.close()
    assert n[abi.MDF_PREC_FP64, 0] == n[abi.MDF_PREC_FP64, 1] == want
    assert n[abi.MDF_PREC_MIXED, 0] == n[abi.MDF_PREC_MIXED, 1]
