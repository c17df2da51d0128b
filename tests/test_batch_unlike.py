"""A batch of systems that need different launches (LJ switched in some, force-
shifted in others) runs every system's own chain in the graph, on the contexts'
streams, which a batch's contexts make when they need them."""
import ctypes as C

import numpy as np
import pytest

from md_b200 import abi, engine, synth
from tests import helpers as H

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [abi.MDF_PREC_MIXED, abi.MDF_PREC_FP64])
def test_unlike_systems_equal_single_ones(prec):
    n, switch = 4, [8.0, 0.0, 8.0, 0.0]
    ss = synth.make_batch(n_systems=n, seed=80)
    flats = [H.flat(s, abi.MDF_SEM_PHYSICAL, engine.cmap_coefficients) for s in ss]
    params, ref = (abi.mdf_params * n)(), []
    for k, s in enumerate(ss):
        eng = engine.Engine(flats[k], s.box, precision=prec, grid=s.meta["grid"], cutoff=9.0, switch_radius=switch[k])
        params[k] = eng.params
        eng.set_positions(s.coords)
        eng.compute()                       # the first evaluation counts pairs: another kernel
        ref.append(eng.compute()[1])
        eng.close()
    lib, h = engine.library(), C.c_void_p()
    tops = (C.POINTER(abi.mdf_topology) * n)(*[C.pointer(f.struct()) for f in flats])
    assert lib.mdf_batch_create(n, tops, params, C.byref(h)) == 0
    x = np.ascontiguousarray(np.concatenate([s.coords for s in ss]))
    F, E = np.zeros_like(x), (abi.mdf_energies * n)()
    dp = C.POINTER(C.c_double)
    assert lib.mdf_batch_set_positions(h, x.ctypes.data_as(dp)) == 0
    for _ in range(2):                      # the capture, and a replay
        assert lib.mdf_batch_compute(h, 3, F.ctypes.data_as(dp), E) == 0
        assert np.array_equal(F, np.concatenate(ref))
    lib.mdf_batch_destroy(h)
