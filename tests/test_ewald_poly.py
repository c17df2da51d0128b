"""The polynomials of the FP64 real-space Ewald terms (md_b200/csrc/ewald_poly.hpp)
against long double on the CPU (tests/ewald_poly.cpp), and the FP64 kernels
around the range they serve: ewald_tol on both sides of it against the oracle,
and a batch whose systems differ in cutoff and alpha (a launch per run of equal
tables) bit for bit against single systems."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from md_b200 import abi, engine, synth
from oracle import oracle as O
from tests import helpers as H

HERE = os.path.dirname(os.path.abspath(__file__))
PHYS, FP64 = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("poly") / "ewald_poly")
    subprocess.run(["g++", "-O2", "-std=c++17", "-I" + os.path.join(os.path.dirname(HERE), "md_b200", "csrc"),
                    os.path.join(HERE, "ewald_poly.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("alpha,rc", [(1e-12, 10.0), (0.05, 12.0), (0.329, 10.0), (0.3654, 9.0), (0.3622, 10.0),
                                      (0.3646, 10.0), (0.3647, 10.0), (1.0, 10.0)])
def test_polynomials_reach_double_rounding(harness, alpha, rc):
    out = subprocess.run([harness, repr(alpha), repr(rc), "4000"], check=True, capture_output=True, text=True).stdout
    if (alpha * rc) ** 2 > 13.3:
        assert out.strip() == "none"
        return
    a = np.array([l.split() for l in out.splitlines()], dtype=np.longdouble)
    # Horner over coefficients that sum to about 1.3 times the largest value:
    # a few units of 2^-53 of it
    for k in (0, 2):
        assert np.abs(a[:, k] - a[:, k + 1]).max() <= 6e-16 * a[:, k + 1].max()


@pytest.mark.gpu
@pytest.mark.parametrize("tol", [1e-3, 1e-6, 9e-7, 1e-9])
@pytest.mark.parametrize("layout", [0, 1])
def test_fp64_matches_oracle_around_the_polynomials_range(tol, layout):
    s = H.system("tiny")
    flat = H.flat(s, PHYS, engine.cmap_coefficients)
    eng = engine.Engine(flat, s.box, semantics=PHYS, precision=FP64, ewald_tol=tol, grid=(24, 24, 24),
                        pair_layout=layout)
    eng.set_positions(s.coords)
    E, F = eng.compute()
    _, Ff = eng.compute(energy=False)
    p = O.make_params(PHYS, s.box, (24, 24, 24), H.alpha_for(tol), H.KC)
    e2, f2, _, _, _ = O.evaluate(flat, p, s.coords)
    assert H.frel(F, f2) < 1e-9 and H.frel(Ff, f2) < 1e-9
    for k in ("vdw", "ee_direct", "ee_recip"):
        assert abs(E[k] - e2[abi.E_INDEX[k]]) <= 1e-9 * max(1.0, abs(e2[abi.E_INDEX[k]])), k
    eng.close()


@pytest.mark.gpu
def test_fp64_batch_of_different_cutoffs_equals_single_systems():
    ss = synth.make_batch(n_systems=4, seed=77)
    flats = [H.flat(s, PHYS, engine.cmap_coefficients) for s in ss]
    cut, tol = [9.0, 9.0, 8.5, 9.0], [1e-5, 1e-5, 1e-5, 1e-9]
    ref = []
    params = (abi.mdf_params * 4)()
    for k, s in enumerate(ss):
        eng = engine.Engine(flats[k], s.box, semantics=PHYS, precision=FP64, grid=s.meta["grid"], cutoff=cut[k],
                            switch_radius=8.0, ewald_tol=tol[k])
        params[k] = eng.params
        eng.set_positions(s.coords)
        ref.append(eng.compute()[1])
        eng.close()
    lib, h = engine.library(), C.c_void_p()
    tops = (C.POINTER(abi.mdf_topology) * 4)(*[C.pointer(f.struct()) for f in flats])
    assert lib.mdf_batch_create(4, tops, params, C.byref(h)) == 0
    x = np.ascontiguousarray(np.concatenate([s.coords for s in ss]))
    F, E = np.zeros_like(x), (abi.mdf_energies * 4)()
    dp = C.POINTER(C.c_double)
    assert lib.mdf_batch_set_positions(h, x.ctypes.data_as(dp)) == 0
    assert lib.mdf_batch_compute(h, 3, F.ctypes.data_as(dp), E) == 0
    lib.mdf_batch_destroy(h)
    assert np.array_equal(F, np.concatenate(ref))
