"""Batches whose systems take different forms of one kernel: FFT lengths with
register radices and without (two launches per pass), and systems on both sides
of the size below which pair lists are cut into parts (2,048 clusters), or all
above it.  Forces bit for bit those of single systems, plain and pipelined."""
import numpy as np
import pytest

from md_b200 import abi, engine, synth
from tests import helpers as H

pytestmark = pytest.mark.gpu
PHYS, FP64, MIXED = abi.MDF_SEM_PHYSICAL, abi.MDF_PREC_FP64, abi.MDF_PREC_MIXED
KW = dict(cutoff=9.0, skin=2.0, switch_radius=8.0, ewald_tol=1e-5)
_BIG = {}


def _compare(ss, grids, prec, layout, clusters=None):
    flats = [H.flat(s, PHYS, engine.cmap_coefficients) for s in ss]
    ref, ncl = [], []
    for s, f, g in zip(ss, flats, grids):
        eng = engine.Engine(f, s.box, precision=prec, grid=g, pair_layout=layout, **KW)
        eng.set_positions(s.coords)
        eng.compute()                       # the first evaluation counts pairs: another kernel
        ref.append(eng.compute())
        ncl.append(eng.pairlist_info()["clusters"])
        eng.close()
    if clusters:
        assert [n >= 2048 for n in ncl] == clusters, ncl
    b = engine.Batch(flats, [s.box for s in ss], grids, precision=prec, pair_layout=layout, **KW)
    b.set_positions([s.coords for s in ss])
    res = b.compute()
    x = np.ascontiguousarray(np.concatenate([s.coords for s in ss]))
    f = np.zeros_like(x)
    b.submit(x.ctypes.data, f.ctypes.data)
    e = b.collect()
    b.close()
    assert np.array_equal(f, np.concatenate([r[1] for r in ref]))
    for (E, F), (E1, F1), E2 in zip(res, ref, e):
        assert np.array_equal(F, F1)
        for t in abi.E_NAMES:               # per-block FP64 sums, then 2^-32 fixed point
            assert abs(E[t] - E1[t]) <= 1e-12 * abs(E1[t]) + 1e-8, t
            assert abs(E2[t] - E1[t]) <= 1e-12 * abs(E1[t]) + 1e-8, t


@pytest.mark.parametrize("prec", [MIXED, FP64])
@pytest.mark.parametrize("grids", [[(28, 30, 33), (33, 28, 30), (30, 33, 32), (27, 32, 30)],
                                   [(28, 33, 35), (33, 35, 28), (35, 28, 33), (28, 28, 28)]])
def test_grid_lengths_of_every_form(grids, prec):
    _compare(synth.make_batch(n_systems=4, seed=79), grids, prec, 0)


def _system(edge, nw):
    if edge not in _BIG:
        _BIG[edge] = synth.make_system("forms", edge, nw, 4, 32)
    return _BIG[edge]


@pytest.mark.parametrize("layout", [0, 1])
@pytest.mark.parametrize("sizes,above", [([(24.0, 400), (58.0, 6300), (30.0, 800)], [False, True, False]),
                                         ([(58.0, 6300), (60.0, 7000)], [True, True])])
def test_mixed_batches_around_the_size_of_cut_lists(sizes, above, layout):
    ss = [_system(*v) for v in sizes]
    _compare(ss, [(synth.smooth_grid_size(s.box[0], 1.0),) * 3 for s in ss], MIXED, layout, above)
