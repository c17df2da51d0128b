"""The bonded terms, excluded pairs and 1-4 pairs in one launch beside the PME
chain against the same lists launched one after the other (per-kernel timing
puts every launch on one stream): the sums are fixed point, so forces and
energies are the same bit for bit, with lists that are empty, shorter and longer
than a block."""
import numpy as np
import pytest

from md_b200 import abi, engine, synth, topology

pytestmark = pytest.mark.gpu
FP64, MIXED = abi.MDF_PREC_FP64, abi.MDF_PREC_MIXED


@pytest.mark.parametrize("semantics,precision", [(abi.MDF_SEM_PHYSICAL, MIXED), (abi.MDF_SEM_PHYSICAL, FP64),
                                                 (abi.MDF_SEM_REFERENCE, FP64)])
@pytest.mark.parametrize("waters,residues", [(3, 0), (90, 0), (40, 3), (300, 12)])
def test_one_launch_equals_separate_ones(waters, residues, semantics, precision):
    s = synth.make_system("terms", 30.0, waters, residues, 41)
    flat = topology.flatten(s, semantics, engine.cmap_coefficients)
    eng = engine.Engine(flat, s.box, semantics=semantics, precision=precision, ewald_tol=1e-5, grid=(30, 30, 30))
    eng.set_positions(s.coords)
    flags = dict(pme_reference=True) if semantics == abi.MDF_SEM_REFERENCE else {}
    eng.compute(**flags)                # the first evaluation counts pairs: another kernel
    E, F = eng.compute(**flags)
    _, F0 = eng.compute(energy=False, **flags)
    eng.enable_timing(True)
    E1, F1 = eng.compute(**flags)
    _, F2 = eng.compute(energy=False, **flags)
    eng.close()
    assert np.array_equal(F, F1) and np.array_equal(F0, F2)
    assert all(E[k] == E1[k] for k in abi.E_NAMES)
