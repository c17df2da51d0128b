"""mdf_backward over the LJ bookkeeping of its pair kernel: systems whose atom
types are nearly all outside the two most frequent (60 types, tables in global
memory), types that share one LJ entry, and force-shifted LJ, where the energy
is linear in A and B so its difference quotient is exact to rounding."""
import numpy as np
import pytest

from md_b200 import abi, engine
from tests import helpers as H

pytestmark = pytest.mark.gpu
PHYS, FP64, MIXED = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64, abi.MDF_PREC_MIXED


def _engine(flat, s, prec, **kw):
    eng = engine.Engine(flat, s.box, semantics=PHYS, precision=prec, ewald_tol=1e-5, grid=(24, 24, 24), **kw)
    eng.set_positions(s.coords)
    return eng


@pytest.mark.parametrize("prec,tol", [(FP64, 1e-9), (MIXED, 1e-5)])
@pytest.mark.parametrize("switch", [9.0, 0.0])
def test_gradients_do_not_depend_on_how_types_are_numbered(prec, tol, switch):
    s = H.system("tiny")
    flat = H.flat(s, PHYS, engine.cmap_coefficients)
    v = np.random.default_rng(2).normal(0.0, 1.0, (s.natoms, 3))
    res = []
    for f in (flat, H.many_types(flat)):
        eng = _engine(f, s, prec, switch_radius=switch)
        res.append(eng.backward(v, 0.3))
        eng.close()
    (q0, A0, B0), (q1, A1, B1) = res
    assert H.frel(q1, q0) < tol
    # the many-type table holds copies of the same pairs: their sums agree
    assert abs(A1.sum() - A0.sum()) <= tol * np.abs(A0).sum()
    assert abs(B1.sum() - B0.sum()) <= tol * np.abs(B0).sum()


@pytest.mark.parametrize("prec,tol", [(FP64, 1e-7), (MIXED, 1e-4)])
def test_force_shifted_energy_gradient_is_its_difference_quotient(prec, tol):
    s = H.system("tiny")
    flat = H.flat(s, PHYS, engine.cmap_coefficients)
    eng = _engine(flat, s, FP64, switch_radius=0.0)
    g = _engine(flat, s, prec, switch_radius=0.0)
    _, dA, dB = g.backward(None, 1.0)
    g.close()
    used = np.argsort(-np.abs(dA))[:4]
    for k in used:
        for which, d in ((0, dA), (1, dB)):
            p = [flat.lj_a.copy(), flat.lj_b.copy()]
            E = []
            for h in (1.0, -1.0):
                q = [a.copy() for a in p]
                q[which][k] += h * max(1.0, abs(p[which][k]))
                eng.set_parameters(None, *q)
                E.append(eng.compute()[0]["vdw"])
            fd = (E[0] - E[1]) / (2.0 * max(1.0, abs(p[which][k])))
            assert abs(fd - d[k]) <= tol * max(abs(fd), np.abs(d).max()), (k, which, fd, d[k])
    eng.close()
