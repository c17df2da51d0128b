"""mdf_backward walks the whole-entry list that it prunes itself, whatever layout
the forward kernels use: mixed gradients of both layouts are the same bits (an
unpruned list groups the FP32 sums otherwise), and a forward evaluation after
the gradient is the one before it."""
import numpy as np
import pytest

from md_b200 import abi, engine
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("every", [1, -1])
@pytest.mark.parametrize("prec", [abi.MDF_PREC_FP64, abi.MDF_PREC_MIXED])
def test_layouts_give_the_same_gradients(prec, every):
    s = H.system("tiny")
    flat = H.flat(s, abi.MDF_SEM_PHYSICAL, engine.cmap_coefficients)
    v = np.random.default_rng(12).normal(0.0, 1.0, (s.natoms, 3))
    got = []
    for layout in (0, 1):
        eng = engine.Engine(flat, s.box, precision=prec, grid=(24, 24, 24), pair_layout=layout, prune_every=every,
                            prune_margin=0.2 if every < 0 else 0.0)
        eng.set_positions(s.coords)
        eng.compute()
        F = eng.compute()[1]
        got.append(eng.backward(v, 0.3))
        assert np.array_equal(eng.compute()[1], F)
        eng.close()
    (q0, A0, B0), (q1, A1, B1) = got
    assert np.array_equal(q1, q0)
    tol = 1e-12 if prec == abi.MDF_PREC_FP64 else 1e-6   # order of the atomic additions
    assert np.linalg.norm(A1 - A0) <= tol * np.linalg.norm(A0) and np.linalg.norm(B1 - B0) <= tol * np.linalg.norm(B0)
