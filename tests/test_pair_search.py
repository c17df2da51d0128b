"""The pair search where its buffers and rules change: lists longer than a
warp's buffer (512 entries: 16 + 5 A at liquid density), a box whose columns
wrap onto themselves, atoms outside the box, and exclusions across periodic
boundaries; FP64 against the oracle, unpruned and pruned."""
import numpy as np
import pytest

from md_b200 import abi, engine, synth
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu
PHYS, FP64 = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64


@pytest.mark.parametrize("edge,cutoff,skin,longer", [((44.0, 45.0, 43.0), 16.0, 5.0, True),
                                                     ((44.0, 45.0, 43.0), 10.0, 2.0, False),
                                                     ((22.0, 24.0, 31.0), 10.5, 0.4, False)])
def test_lists_match_the_oracle(edge, cutoff, skin, longer):
    nw = int(0.095 * np.prod(edge) / 3)
    s = synth.make_system("search", edge, nw, 6, 91)
    flat = H.flat(s, PHYS, engine.cmap_coefficients)
    x = s.coords + np.array([0.3, -7.7, 100.1])          # molecules across every face, some boxes away
    grid = tuple(synth.smooth_grid_size(v, 1.0) for v in edge)
    p = O.make_params(PHYS, s.box, grid, H.alpha_for(1e-5, cutoff), H.KC, cutoff=cutoff, switch=cutoff - 1.0)
    e2, f2, _, _, n2 = O.evaluate(flat, p, x)
    for every in (0, 1):
        eng = engine.Engine(flat, s.box, semantics=PHYS, precision=FP64, ewald_tol=1e-5, grid=grid, cutoff=cutoff,
                            skin=skin, switch_radius=cutoff - 1.0, prune_every=every)
        eng.set_positions(x)
        eng.build_pairlist()
        E, F = eng.compute()
        info = eng.pairlist_info()
        eng.close()
        # half lists: the first clusters hold nearly all their neighbours, twice the mean
        assert (info["cluster_pairs"] > 300 * info["clusters"]) == longer
        assert info["pairs_in_cutoff"] == n2
        assert H.frel(F, f2) < 1e-9
        for k in ("vdw", "ee_direct", "ee_excl"):
            assert abs(E[k] - e2[abi.E_INDEX[k]]) <= 1e-9 * max(1.0, abs(e2[abi.E_INDEX[k]])), k
