"""mdf_backward over the forms its kernels take: FFT lengths with register
radices, without, and both in one grid (the charge and the dipole chain share
each pass's launch), odd numbers of lines, no Ewald polynomials, and many LJ
types.  Gradients of tests/adjoint_ref.py with the bounds of test_adjoint.py;
dL/dA and dL/dB entry by entry where they are sums of positive terms."""
import numpy as np
import pytest

from md_b200 import abi, engine
from tests import helpers as H

pytestmark = pytest.mark.gpu
PHYS, FP64, MIXED = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64, abi.MDF_PREC_MIXED
BOUND = {FP64: 1e-8, MIXED: 1e-5}


def _setup(flat, s, prec, grid=(24, 24, 24), tol=1e-5, **kw):
    eng = engine.Engine(flat, s.box, semantics=PHYS, precision=prec, ewald_tol=tol, grid=grid, **kw)
    eng.set_positions(s.coords)
    return eng


def _ref(flat, s, grid=(24, 24, 24), tol=1e-5):
    from tests.adjoint_ref import NonbondedRef
    return NonbondedRef(flat, s.box, grid, H.alpha_for(tol), H.KC)


def _check(prec, got, want):
    for name, g, w in zip(("q", "A", "B"), got, want):
        assert np.linalg.norm(g - w) <= BOUND[prec] * np.linalg.norm(w), name


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("grid", [(28, 30, 33), (22, 27, 25), (33, 35, 32), (25, 27, 45), (21, 25, 28), (27, 26, 24)])
def test_gradients_at_grid_lengths_of_every_form(grid, prec):
    s = H.system("tiny")
    flat = H.flat(s, PHYS, engine.cmap_coefficients)
    v = np.random.default_rng(8).normal(0.0, 1.0, (s.natoms, 3))
    eng = _setup(flat, s, prec, grid)
    got = eng.backward(v, 0.4)
    eng.close()
    _check(prec, got, _ref(flat, s, grid).vjp(flat.charge, flat.lj_a, flat.lj_b, s.coords, v, 0.4))


def test_gradients_without_the_ewald_polynomials():
    s = H.system("tiny")
    flat = H.flat(s, PHYS, engine.cmap_coefficients)
    v = np.random.default_rng(9).normal(0.0, 1.0, (s.natoms, 3))
    eng = _setup(flat, s, FP64, tol=1e-9)
    got = eng.backward(v, 0.4)
    eng.close()
    _check(FP64, got, _ref(flat, s, tol=1e-9).vjp(flat.charge, flat.lj_a, flat.lj_b, s.coords, v, 0.4))


@pytest.mark.parametrize("prec", [FP64, MIXED])
@pytest.mark.parametrize("ntypes", [60, 150])   # block sums in shared memory; too many entries for them
def test_every_entry_of_many_types(ntypes, prec):
    s = H.system("tiny")
    flat = H.many_types(H.flat(s, PHYS, engine.cmap_coefficients), ntypes)
    ref = _ref(flat, s)
    v = np.random.default_rng(10).normal(0.0, 1.0, (s.natoms, 3))
    eng = _setup(flat, s, prec)
    got = eng.backward(v, 0.4)
    _, dA, dB = eng.backward(None, 1.0)
    eng.close()
    _check(prec, got, ref.vjp(flat.charge, flat.lj_a, flat.lj_b, s.coords, v, 0.4))
    _, rA, rB = ref.vjp(flat.charge, flat.lj_a, flat.lj_b, s.coords, np.zeros((s.natoms, 3)), 1.0)
    # dE/dA = sum S/r^12 and -dE/dB = sum S/r^6: no cancellation.  FP32 frames
    # place an atom to about 5e-7 A, 12 times that relative in r^-12 at 2 A and
    # 1e-6 in the switch, whose terms start at 9 A; FP64 likewise with 2^-53
    rtol, atol = (1e-9, 1e-10) if prec == FP64 else (1e-4, 1e-4)
    for g, w, p in ((dA, rA, 12), (dB, rB, 6)):
        assert np.all(np.abs(g - w) <= rtol * np.abs(w) + atol * 9.0 ** -p), np.abs((g - w) / np.where(w == 0, 1, w)).max()
