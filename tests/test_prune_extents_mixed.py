"""The mixed prune where clusters are long (the systems of test_prune_extents.py):
pruned evaluations count the pairs that unpruned ones do, and where both run the
same pair kernel give their forces to the order of the FP32 sums.  (The half
layout adds the frame offset to the other atom, and FP32 rounds coordinates of
thousands of A to 1e-3 A.)"""
import numpy as np
import pytest

from md_b200 import abi, engine
from tests import helpers as H
from tests.test_prune_extents import _dimers

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("n,lx,spacing", [(48, 26.0, 12.0), (48, 26.0, 300.0), (48, 26.0, 1500.0), (48, 26.0, 9000.0),
                                          (8500, 600.0, 15.0)])
def test_mixed_prune_keeps_every_pair_of_long_clusters(n, lx, spacing, layout):
    x, q, box = _dimers(n, lx, spacing)
    flat, res = H.simple_flat(q), []
    for every in (1, 0):
        eng = engine.Engine(flat, box, precision=abi.MDF_PREC_MIXED, ewald_tol=0.1, grid=(24, 24, 64),
                            prune_every=every, pair_layout=layout if every else 0)
        eng.set_positions(x)
        res.append((eng.compute()[1], eng.pairlist_info()["pairs_in_cutoff"]))
        eng.close()
    assert res[0][1] == res[1][1] >= n - 2      # FP32 places a pair at 9.999 A to 1e-3 A in the longest boxes
    if layout == 0:
        assert H.frel(res[0][0], res[1][0]) < 1e-6
