"""The FFT passes over lengths of every form: two and three register radices,
single radices, and lengths with a factor 7 or 11 (table-driven passes), mixed
in one grid, with lines per block set and left to the rule.  The gathered
potential equals N irfftn(c rfftn(Q)) of torch.fft on the engine's own charge
grid, and energies, virial and forces equal the oracle's."""
import numpy as np
import pytest

from md_b200 import abi, engine
from oracle import oracle as O
from tests import helpers as H

pytestmark = pytest.mark.gpu
PHYS, FP64, MIXED = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64, abi.MDF_PREC_MIXED
GRIDS = [(24, 27, 25), (28, 30, 33), (30, 28, 36), (33, 35, 32), (45, 64, 81), (22, 100, 54), (48, 49, 50),
         (125, 40, 30), (30, 144, 45), (36, 25, 216), (160, 27, 31), (25, 162, 128)]


def _bmod(n):
    a = 2 * np.pi * np.arange(n) / n
    return 1.0 / np.abs((1 + 4 * np.exp(1j * a) + np.exp(2j * a)) / 6) ** 2


@pytest.mark.parametrize("prec,tol", [(FP64, 1e-12), (MIXED, 1e-5)])
@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("lines", [0, 4])
def test_potential_matches_torch_fft(grid, prec, tol, lines):
    s = H.system("tiny")
    flat = H.flat(s, PHYS, engine.cmap_coefficients)
    eng = engine.Engine(flat, s.box, semantics=PHYS, precision=prec, ewald_tol=1e-5, grid=grid, fft_lines=lines)
    eng.set_positions(s.coords)
    E, F = eng.compute()
    Q, P = eng.pme_grids()
    _, Ff = eng.compute(energy=False)
    assert np.array_equal(F, Ff) if prec == FP64 else H.frel(Ff, F) < 1e-6
    eng.close()
    L, al = s.box, H.alpha_for(1e-5)
    m = [np.fft.fftfreq(grid[d], 1.0 / grid[d]) / L[d] for d in range(2)] + [np.arange(grid[2] // 2 + 1) / L[2]]
    m2 = m[0][:, None, None] ** 2 + m[1][None, :, None] ** 2 + m[2][None, None] ** 2
    m2[0, 0, 0] = 1.0
    c = H.KC / (np.pi * np.prod(L)) * np.exp(-np.pi ** 2 * m2 / al ** 2) / m2
    c = c * _bmod(grid[0])[:, None, None] * _bmod(grid[1])[None, :, None] * _bmod(grid[2])[None, None, :len(m[2])]
    c[0, 0, 0] = 0.0
    ref = np.fft.irfftn(np.fft.rfftn(Q) * c, s=grid, axes=(0, 1, 2)) * np.prod(grid)
    assert np.linalg.norm(P - ref) <= tol * np.linalg.norm(ref)
    if prec == FP64 and lines == 0:
        p = O.make_params(PHYS, s.box, grid, al, H.KC)
        e2, f2, vir2, _, _ = O.evaluate(flat, p, s.coords)
        assert H.frel(F, f2) < 1e-9
        assert abs(E["ee_recip"] - e2[abi.E_INDEX["ee_recip"]]) <= 1e-9 * abs(e2[abi.E_INDEX["ee_recip"]])
        assert np.allclose(E["virial"].ravel(), vir2, rtol=1e-9, atol=1e-7)
