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


FP64 = {"ternary 16^3": (3, (16, 16, 16), {}, False), "ternary 104x100x98": (3, (104, 100, 98), {}, False),
        "binary": (2, (40, 17, 12), {}, False),
        "binary rock": (2, (21, 18, 16), dict(g_wr=-0.1, rock_colour_r=1.0), True),
        "sheared": (2, (33, 18, 17), dict(boundary_cond=-1, inv_fluid=5, shear_u=0.05), False),
        "sheared rock": (2, (18, 17, 16), dict(boundary_cond=-1, inv_fluid=5, shear_u=0.05, g_wr=-0.1), True)}


@pytest.mark.parametrize("kind", FP64)
def test_fp64_loops_back_to_back(kind):
    """Both ways a step is launched (all components in one stream launch up to
    a million sites, two above): every field of the download, the moments and the
    dipole flux among them."""
    nc, dims, kw, rock = FP64[kind]
    p, st = _params(dims, nc, 0, **kw), uniform_mixture(*dims, nc, seed=3)
    if rock:
        st["rock"] = (np.random.default_rng(8).random(st["n"].shape[2:]) < 0.2).astype(np.float64)
        st["n"] = st["n"] * (1 - st["rock"])
    a, b = _loops(p, st, True), _loops(p, st, False)
    for f in a:
        assert np.array_equal(a[f], b[f]), f
    assert np.isfinite(a["n"]).all()


@pytest.mark.parametrize("nc,dims", [(3, (16, 16, 16)), (2, (33, 20, 18))])
def test_no_alloc_calls_back_to_back(nc, dims):
    """Calls of one to five steps on the caller's buffers, against the handle's
    time loop waited for after every call."""
    import torch

    from .test_zz_no_alloc import _last_error, _noalloc
    p, st = _params(dims, nc, 0), uniform_mixture(*dims, nc, seed=3)
    ref = _loops(p, st, True)
    n = torch.from_numpy(np.ascontiguousarray(st["n"])).cuda()
    db = torch.from_numpy(np.ascontiguousarray(st["db"])).cuda() if nc == 3 else None
    stream = torch.cuda.current_stream().cuda_stream
    for steps in LOOPS:
        rc = _noalloc(p, n.data_ptr(), db.data_ptr() if nc == 3 else None, None, steps, stream)
        assert rc == 0, _last_error()
    torch.cuda.synchronize()
    assert np.array_equal(n.cpu().numpy(), ref["n"])
    if nc == 3:
        assert np.array_equal(db.cpu().numpy(), ref["db"])


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
