"""The pair lists' shares (mdf_params has no switch for them: they follow from
the system's size) and the prune's two forms, on both sides of the sizes where
the rules change, in both layouts and schedules: mixed forces within the mixed
bound of the FP64 path and bit for bit the same in either schedule and block
size, pruned or not to the order of the sums."""
import numpy as np
import pytest

from md_b200 import abi, engine, synth, topology
from tests import helpers as H

pytestmark = pytest.mark.gpu
PHYS, FP64, MIXED = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64, abi.MDF_PREC_MIXED
# edge (A), waters: about 110, 950, 1,800 and 2,400 clusters (2,048 is the line)
SIZES = [(22.0, 300), (42.0, 2470), (52.0, 4690), (58.0, 6300)]
_CACHE = {}


def _system(edge, nw):
    if edge not in _CACHE:
        s = synth.make_system("split", edge, nw, 6, 31)
        _CACHE[edge] = (s, topology.flatten(s, PHYS, engine.cmap_coefficients))
    return _CACHE[edge]


def _compute(s, flat, prec, energy=True, **shape):
    g = synth.smooth_grid_size(s.box[0], 1.0)
    eng = engine.Engine(flat, s.box, semantics=PHYS, precision=prec, ewald_tol=1e-5, grid=(g, g, g), **shape)
    eng.set_positions(s.coords)
    eng.compute()                       # the first evaluation counts pairs: another kernel
    E, F = eng.compute(energy=energy)
    n = eng.pairlist_info()["clusters"]
    eng.close()
    return E, F, n


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("edge,nw", SIZES)
def test_shares_change_no_bit_and_hold_the_mixed_bound(edge, nw, layout):
    s, flat = _system(edge, nw)
    E, F, n = _compute(s, flat, MIXED, pair_layout=layout)
    for shape in (dict(pair_schedule=1), dict(pair_warps=2), dict(pair_warps=4, pair_schedule=1)):
        E1, F1, _ = _compute(s, flat, MIXED, pair_layout=layout, **shape)
        assert np.array_equal(F1, F) and E1["vdw"] == E["vdw"] and E1["ee_direct"] == E["ee_direct"], shape
    _, Ff, _ = _compute(s, flat, MIXED, energy=False, pair_layout=layout)
    assert H.frel(Ff, F) < 1e-6         # the forces-only kernel
    E64, F64, _ = _compute(s, flat, FP64, pair_layout=layout)
    assert H.frel(F, F64) <= 1e-5
    assert abs(E["total"] - E64["total"]) <= 1e-6 * sum(abs(E64[k]) for k in abi.E_NAMES)
    E0, F0, _ = _compute(s, flat, MIXED, prune_every=0)
    assert H.frel(F0, F) < 1e-6


def test_sizes_lie_on_both_sides_of_the_line():
    n = [_compute(*_system(e, w), MIXED)[2] for e, w in SIZES]
    assert n[2] < 2048 <= n[3], n
