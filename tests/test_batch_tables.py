"""FP64 batches of systems with different Ewald polynomials (cutoff and alpha):
one pair launch per table whatever the order of the systems, and forces bit for
bit those of single systems, through the plain and the pipelined entry points."""
import ctypes as C

import numpy as np
import pytest

from md_b200 import abi, engine, synth
from tests import helpers as H

pytestmark = pytest.mark.gpu
N = 8


def _batch(cut, tol):
    ss = synth.make_batch(n_systems=N, seed=78)
    flats = [H.flat(s, abi.MDF_SEM_PHYSICAL, engine.cmap_coefficients) for s in ss]
    params = (abi.mdf_params * N)()
    ref = []
    for k, s in enumerate(ss):
        eng = engine.Engine(flats[k], s.box, precision=abi.MDF_PREC_FP64, grid=s.meta["grid"], cutoff=cut[k],
                            switch_radius=8.0, ewald_tol=tol[k])
        params[k] = eng.params
        eng.set_positions(s.coords)
        ref.append(eng.compute()[1])
        eng.close()
    lib, h = engine.library(), C.c_void_p()
    tops = (C.POINTER(abi.mdf_topology) * N)(*[C.pointer(f.struct()) for f in flats])
    assert lib.mdf_batch_create(N, tops, params, C.byref(h)) == 0
    x = np.ascontiguousarray(np.concatenate([s.coords for s in ss]))
    F, F2, E = np.zeros_like(x), np.zeros_like(x), (abi.mdf_energies * N)()
    dp = C.POINTER(C.c_double)
    assert lib.mdf_batch_set_positions(h, x.ctypes.data_as(dp)) == 0
    assert lib.mdf_batch_compute(h, 3, F.ctypes.data_as(dp), E) == 0
    kernels = C.c_int64()
    assert lib.mdf_batch_info(h, None, None, C.byref(kernels)) == 0
    assert lib.mdf_batch_submit(h, 3, x.ctypes.data_as(dp), F2.ctypes.data_as(dp)) == 0
    assert lib.mdf_batch_collect(h, E) == 0
    lib.mdf_batch_destroy(h)
    ref = np.concatenate(ref)
    assert np.array_equal(F, ref) and np.array_equal(F2, ref)
    return kernels.value


def test_one_pair_launch_per_table():
    one = _batch([9.0] * N, [1e-5] * N)
    assert _batch([9.0, 8.5] * (N // 2), [1e-5] * N) == one + 1
    assert _batch([9.0] * N, [1e-5, 1e-4, 1e-9, 1e-5] * (N // 4)) == one + 2
    assert _batch([9.0 - 0.05 * k for k in range(N)], [1e-5] * N) == one + N - 1
