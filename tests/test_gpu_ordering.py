"""Calls enqueued back to back, with no wait on the host between them, give the
bits of calls that are waited for one by one: the kernels of a call, and those
of neighbouring calls, may overlap only where nothing they read is still being
written."""
import numpy as np
import pytest

from lb3d_b200.config import Params
from lb3d_b200.ic import uniform_mixture

pytestmark = pytest.mark.gpu

LOOPS = [1, 2, 3, 5, 4, 1, 1, 2] * 25  # an odd number of loops ends on each parity


def _params(dims, nc, precision, **kw):
    base = dict(nx=dims[0], ny=dims[1], nz=dims[2], ncomp=nc, tau_d=1.0, g_br=0.08, g_bs=-0.006, g_ss=-0.0045,
                beta=10.0, d_0=1.0, bdist=2, restore=1, precision=precision)
    base.update(kw)
    return Params(**base).finalize()


def _loops(p, st, wait):
    from lb3d_b200.lib import Lattice
    lat = Lattice(p)
    lat.upload_state(st)
    for n in LOOPS:
        lat.time_loop(n)
        if wait:
            lat.sync()
    out = lat.download()
    lat.close()
    return out


@pytest.mark.parametrize("nc,dims", [(3, (16, 16, 16)), (3, (33, 20, 18)), (2, (40, 17, 12))])
def test_fp32_loops_back_to_back(nc, dims):
    p, st = _params(dims, nc, 1), uniform_mixture(*dims, nc, seed=3)
    a, b = _loops(p, st, True), _loops(p, st, False)
    assert np.array_equal(a["n"], b["n"]) and np.array_equal(a["db"], b["db"])
    assert np.isfinite(a["n"]).all()


def test_ensemble_chunks_back_to_back():
    """Chunks of one to three steps (enqueued pass by pass) and of four and more
    (replayed from a graph)."""
    from lb3d_b200.ensemble import Ensemble
    out = []
    for wait in (True, False):
        ens = Ensemble(3, capacity_sites=20000, max_lattices=4)
        slots = [ens.admit(_params(d, 3, 1), uniform_mixture(*d, 3, seed=4), steps=sum(LOOPS))
                 for d in ((16, 16, 16), (17, 9, 7))]
        for n in LOOPS:
            assert ens.step(n) == n
            if wait:
                ens.sync()
        out.append([ens.retire(s, d) for s, d in zip(slots, ((16, 16, 16), (7, 9, 17)))])
        ens.close()
    for a, b in zip(*out):
        assert np.array_equal(a["n"], b["n"]) and np.array_equal(a["db"], b["db"])
