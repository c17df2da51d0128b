"""The device memory a context's first gradient takes: one set of grids for the
dipole chain (8 bytes a point and half a complex grid) beside the context's own,
and buffers of the size of the system."""
import numpy as np
import pytest

from md_b200 import abi, engine
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,half_complex", [(abi.MDF_PREC_MIXED, 4), (abi.MDF_PREC_FP64, 8)])
def test_first_gradient_takes_one_set_of_grids(prec, half_complex):
    import torch
    s = H.system("tiny")
    flat = H.flat(s, abi.MDF_SEM_PHYSICAL, engine.cmap_coefficients)
    K = 200
    eng = engine.Engine(flat, s.box, precision=prec, grid=(K, K, K))
    eng.set_positions(s.coords)
    eng.compute()
    free = torch.cuda.mem_get_info()[0]
    eng.backward(np.ones((s.natoms, 3)), 1.0)
    took = free - torch.cuda.mem_get_info()[0]
    eng.close()
    # 2 % more points in the half-complex grid, and 8 MiB for what is not a grid and the driver's blocks
    assert took <= K ** 3 * (8 + 1.02 * half_complex) + (8 << 20), took
