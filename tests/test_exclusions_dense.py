"""Excluded pairs of atoms with many partners, which the list build clears after
the search, beside those with few: a rigid body with all its pairs excluded, rows
at the line between the two (32 partners) and above it, rows above it for every
atom (which stay in the search), and bonded pairs, some across the box edge; pair
counts against a direct count, forces against the oracle."""
import numpy as np
import pytest
from scipy.spatial import cKDTree

from md_b200 import abi, engine
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu
PHYS, FP64 = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64


@pytest.mark.parametrize("body,hub", [(0, 32), (0, 33), (60, 32), (250, 40), (1500, 0)])
@pytest.mark.parametrize("shift", [0.0, 14.3])
def test_counts_and_forces(body, hub, shift):
    L, n = 30.0, 2700
    rng = np.random.default_rng(6)
    g = int(np.ceil(n ** (1 / 3)))
    p = (np.stack(np.meshgrid(*[np.arange(g)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n] + 0.5) * (L / g)
    p += rng.uniform(-0.2, 0.2, p.shape)
    x = p[np.argsort(((p - L / 2) ** 2).sum(1))] + shift     # the first atoms: a ball
    q = np.where(rng.random(n) < 0.5, 0.3, -0.3)
    ex = {tuple(v) for v in np.stack(np.triu_indices(body, 1), 1).tolist()}
    ex |= {(body, body + 1 + k) for k in range(hub)}         # an atom with `hub` partners
    ex |= {(a, a + 1) for a in range(1700, n - 1, 2)}        # pairs
    ex = np.array(sorted(ex), np.int32)
    flat = H.simple_flat(q, lj_a=[1.0e5], lj_b=[200.0], excl_pairs=ex)
    d = np.abs((x[:, None] - x[None]) - L * np.round((x[:, None] - x[None]) / L))
    near = (d ** 2).sum(-1) <= 100.0
    near[ex[:, 0], ex[:, 1]] = near[ex[:, 1], ex[:, 0]] = False
    want = int(np.triu(near, 1).sum())
    eng = engine.Engine(flat, [L] * 3, precision=FP64, ewald_tol=1e-5, grid=(30, 30, 30))
    eng.set_positions(x)
    E, F = eng.compute()
    assert eng.pairlist_info()["pairs_in_cutoff"] == want
    eng.close()
    prm = O.make_params(PHYS, np.array([L] * 3), (30, 30, 30), H.alpha_for(1e-5), H.KC)
    e2, f2, _, _, _ = O.evaluate(flat, prm, x)
    assert H.frel(F, f2) < 1e-9
    for k in ("vdw", "ee_direct", "ee_excl"):
        assert abs(E[k] - e2[abi.E_INDEX[k]]) <= 1e-9 * max(1.0, abs(e2[abi.E_INDEX[k]])), k


@pytest.mark.parametrize("n", [5000, 6000])      # 2,600 pairs per partner: 5,200 atoms
def test_long_rows_for_every_atom(n):
    L, K = 44.0, 40
    rng = np.random.default_rng(7)
    x = rng.uniform(0, L, (n, 3))
    i = np.arange(n)
    ex = np.concatenate([np.stack([i, (i + k) % n], 1) for k in range(1, K // 2 + 1)])
    ex.sort(axis=1)
    near = cKDTree(x, boxsize=L).query_pairs(10.0, output_type="ndarray")
    want = len(near) - len(np.intersect1d(near[:, 0] * n + near[:, 1], ex[:, 0].astype(np.int64) * n + ex[:, 1]))
    eng = engine.Engine(H.simple_flat(np.tile([0.1, -0.1], n // 2), excl_pairs=ex), [L] * 3, precision=FP64,
                        grid=(44, 44, 44))
    eng.set_positions(x)
    eng.compute()
    assert eng.pairlist_info()["pairs_in_cutoff"] == want
    eng.close()
