"""Split evaluations at FFT lengths without register radices and with both forms
in one grid: slab-distributed reciprocal space and halo exchange, forces bit for
bit those of one context (two gloo ranks on one GPU; no kernel waits on another
rank)."""
import numpy as np
import pytest

from md_b200 import abi
from tests import helpers as H
from tests.test_distributed import _init, _run

pytestmark = pytest.mark.gpu


def _engine(grid, prec, **kw):
    from md_b200 import engine
    s = H.system("tiny")
    flat = H.flat(s, abi.MDF_SEM_PHYSICAL, engine.cmap_coefficients)
    return s, engine.Engine(flat, s.box, precision=prec, ewald_tol=1e-5, grid=grid, **kw)


def _worker(rank, world, port, q, grid, prec, halo):
    from md_b200 import distributed
    dist = _init(rank, world, port)
    s, eng = _engine(grid, prec, rank=rank, nranks=world)
    eng.set_allreduce(distributed.torch_allreduce())
    eng.set_collectives(*distributed.torch_collectives())
    if halo:
        eng.set_halo_exchange(distributed.torch_alltoallv())
    eng.set_positions(s.coords)
    eng.build_pairlist()
    q.put((rank, [eng.compute() for _ in range(2)]))
    eng.close()
    dist.destroy_process_group()


@pytest.mark.parametrize("halo", [False, True])
@pytest.mark.parametrize("prec", [abi.MDF_PREC_MIXED, abi.MDF_PREC_FP64])
@pytest.mark.parametrize("grid", [(28, 33, 26), (26, 24, 35), (27, 28, 30)])
def test_slab_passes_at_every_form(grid, prec, halo):
    res = _run(_worker, 2, grid, prec, halo)
    s, eng = _engine(grid, prec)
    eng.set_positions(s.coords)
    eng.build_pairlist()
    ref = [eng.compute() for _ in range(2)]
    eng.close()
    for out in res:
        for (E, F), (E1, F1) in zip(out, ref):
            assert np.array_equal(F, F1)
            assert abs(E["total"] - E1["total"]) <= 1e-12 * abs(E1["total"]) + 1e-8
