"""FP32 strategy 3 (the equilibrium's arguments carried between the steps of a
loop) at the sizes where its tiles, halos and loops can go wrong, against
strategy 2 bit for bit, and the FP32 download's planes formed on the device."""
import numpy as np
import pytest

from lb3d_b200.config import Params
from lb3d_b200.ic import uniform_mixture

pytestmark = pytest.mark.gpu


def _params(dims, nc, **kw):
    base = dict(nx=dims[0], ny=dims[1], nz=dims[2], ncomp=nc, tau_d=1.0, g_br=0.08, g_bs=-0.006, g_ss=-0.0045,
                beta=10.0, d_0=1.0, bdist=2, restore=1, precision=1)
    base.update(kw)
    return Params(**base).finalize()


def _state(dims, nc, rock=False, shear=False):
    st = uniform_mixture(*dims, nc, seed=41)
    if rock:
        st["rock"] = (np.random.default_rng(8).random(st["n"].shape[2:]) < 0.25).astype(np.float64)
    if shear:
        st["shear_sum"] = 0.37
    return st


def _run(p, st, shape, loops):
    from lb3d_b200.lib import Lattice
    lat = Lattice(p, precision=1)
    lat.upload_state(st)
    lat.set_launch_shape(*shape)
    out = []
    for steps in loops:
        lat.time_loop(steps)
        out.append(lat.download())
    lat.close()
    return out


KINDS = {"ternary": (3, {}, False, False), "binary": (2, {}, False, False),
         "rock": (2, dict(g_wr=-0.1, g_wb=0.05, rock_colour_r=1.0, rock_colour_b=0.5, g_accn_x=1e-4), True, False),
         "sheared": (2, dict(boundary_cond=-1, inv_fluid=5, shear_u=-0.3), False, True),
         "sheared rock": (2, dict(boundary_cond=-1, inv_fluid=5, shear_u=0.05, g_wr=-0.1, rock_colour_r=1.0), True, True)}


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("dims", [(16, 8, 1), (17, 9, 2), (31, 7, 3), (32, 16, 4), (33, 17, 5), (2, 2, 37),
                                  (48, 3, 9)])
def test_loops_equal_the_staged_split(kind, dims):
    """Tile edges and remainders in x, y and z, lattices thinner than a halo;
    loops of one step (populations in and out), two (no step between) and more."""
    nc, kw, rock, shear = KINDS[kind]
    p, st = _params(dims, nc, **kw), _state(dims, nc, rock, shear)
    a = _run(p, st, (16, 8, 16, 2), (1, 2, 6))
    b = _run(p, st, (16, 8, 16, 3), (1, 2, 6))
    for x, y in zip(a, b):
        for f in ("n", "db", "rho", "mom"):
            assert np.array_equal(x[f], y[f]), f


@pytest.mark.parametrize("rock", [False, True])
def test_large_sheared_lattice_forks(rock):
    """From 2^20 sites the boundary tiles run beside the others."""
    dims = (128, 96, 96)
    kw = dict(boundary_cond=-1, inv_fluid=5, shear_u=0.2, shear_omega=0.31)
    p, st = _params(dims, 2, **kw), _state(dims, 2, rock, True)
    a, b = (_run(p, st, (16, 8, 16, s), (5,))[0]["n"] for s in (2, 3))
    assert np.array_equal(a, b)


@pytest.mark.parametrize("rock", [False, True])
@pytest.mark.parametrize("dims", [(128, 128, 128), (75, 509, 17), (48, 1024, 16)])
def test_forked_sheared_lattices_equal_the_staged_split(dims, rock):
    """More moments tiles than resident CTAs: the boundary tiles run beside the
    others."""
    kw = dict(boundary_cond=-1, inv_fluid=5, shear_u=0.2, shear_omega=0.31)
    p, st = _params(dims, 2, **kw), _state(dims, 2, rock, True)
    a, b = (_run(p, st, (16, 8, 16, s), (1, 4)) for s in (2, 3))
    for x, y in zip(a, b):
        assert np.array_equal(x["n"], y["n"])


def test_rock_populations_survive_a_change_of_strategy():
    """A loop lays its arguments over the buffer it read first; rock sites hold
    their populations again afterwards, in both buffers."""
    from lb3d_b200.lib import Lattice
    nc, kw, rock, shear = KINDS["sheared rock"]
    dims = (20, 10, 12)
    p, st = _params(dims, nc, **kw), _state(dims, nc, rock, shear)
    out = []
    for plan in ((2, 2, 2, 2), (3, 2, 3, 2), (2, 3, 3, 2)):
        lat = Lattice(p, precision=1)
        lat.upload_state(st)
        for split in plan:
            lat.set_launch_shape(16, 8, 16, split)
            lat.time_loop(3)
        # the counts cover rock sites, whose FP32 deviations are as uploaded
        out.append((lat.download()["n"], lat.sanity()))
        lat.close()
    for n, counts in out[1:]:
        assert np.array_equal(out[0][0], n) and out[0][1] == counts


@pytest.mark.parametrize("dims,nc,per_step,first", [((32, 16, 12), 2, 4, 4), ((192, 64, 64), 2, 4, 4),
                                                    ((80, 512, 16), 2, 5, 5), ((32, 512, 80), 2, 4, 4),
                                                    ((20, 18, 16), 3, 4, 3)])
def test_kernel_stats_count_every_launch(dims, nc, per_step, first):
    """Sheared: two halo kernels, moments (in two parts where the tiles fill more
    than one round of the resident CTAs and some lie off the sheared boundary)
    and collide pass.  Ternary: moments,
    after a loop's first step in two launches, dipole and collide pass.  One
    parity flip a loop."""
    from lb3d_b200.lib import Lattice
    kw = dict(boundary_cond=-1, inv_fluid=5, shear_u=0.05) if nc == 2 else {}
    lat = Lattice(_params(dims, nc, **kw), precision=1)
    lat.upload_state(_state(dims, nc, shear=nc == 2))
    assert lat.launch_shape[3] == 3
    lat.set_profiling(True)
    lat.time_loop(1)
    lat.time_loop(5)
    assert lat.kernel_stats()[2] == 2 * first + 4 * per_step + 2
    lat.close()


@pytest.mark.parametrize("kind", ["rock", "sheared rock"])
def test_rock_populations_after_loops_of_one_step_and_more(kind):
    """A loop of one step lays no arguments over the rock sites' populations, a
    longer one over the first planes of the buffer it read: whichever buffer is
    current afterwards holds them as uploaded."""
    from lb3d_b200.lib import Lattice
    nc, kw, rock, shear = KINDS[kind]
    dims = (35, 9, 11)
    p, st = _params(dims, nc, **kw), _state(dims, nc, rock, shear)
    out = []
    for split in (2, 3):
        lat = Lattice(p, precision=1)
        lat.upload_state(st)
        lat.set_launch_shape(16, 8, 16, split)
        got = []
        for steps in (1, 3, 1, 1, 2, 1, 4, 2):
            lat.time_loop(steps)
            got.append((lat.download()["n"], lat.sanity()))
        out.append(got)
        lat.close()
    for a, b in zip(*out):
        assert np.array_equal(a[0], b[0]) and a[1] == b[1]


def test_ensemble_members_on_strategy_3():
    """Odd sizes, one member alone in a chunk of one step, and a member that
    does not relax fully joining (all run strategy 2 then)."""
    from lb3d_b200.ensemble import Ensemble
    sizes = [((17, 9, 5), 1), ((16, 33, 12), 8), ((7, 8, 31), 8)]
    ens = Ensemble(3, capacity_sites=20000, max_lattices=8)
    slots = [ens.admit(_params(d, 3), _state(d, 3), steps=n) for d, n in sizes]
    late = (9, 9, 9)
    for k in range(100):
        if not ens.stats()["active"]:
            break
        ens.step(3)
        if k == 1:
            slots.append(ens.admit(_params(late, 3, tau_s=1.2), _state(late, 3), steps=4))
    for slot, (d, n), tau in zip(slots, sizes + [(late, 4)], (1.0, 1.0, 1.0, 1.2)):
        got = ens.retire(slot, d[::-1])
        ref = _run(_params(d, 3, tau_s=tau), _state(d, 3), (16, 8, 16, 2), (n,))[0]
        assert np.array_equal(got["n"], ref["n"]) and np.array_equal(got["db"], ref["db"])


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("kw", [{}, dict(g_accn=2e-4, g_accn_x=-1e-4)], ids=["free", "body force"])
def test_ensemble_strategy_is_the_one_asked_for(nc, kw):
    """Binary and ternary members, without and with a body force, in chunks of
    1 to 3 steps and in chunks replayed from a graph: strategy 3 by default while
    all of them relax fully, 2 (or 0) where the caller says so, the same bits
    either way; a member that does not relax fully takes all to strategy 2."""
    from lb3d_b200.ensemble import Ensemble
    members = [(17, 9, 5), (16, 33, 12), (7, 8, 31)]
    got = {}
    for shape in (None, (32, 4, 8, 3), (16, 8, 4, 2), (32, 4, 8, 0)):
        ens = Ensemble(nc, capacity_sites=20000, max_lattices=8, **({} if shape is None else dict(shape=shape)))
        want = 3 if shape is None else shape[3]
        assert ens.launch_shape == (shape or (32, 4, 8))[:3] + (want,)
        slots = [ens.admit(_params(d, nc, **kw), _state(d, nc), steps=21) for d in members]
        for chunk in (1, 3, 5, 5, 5, 2):
            assert ens.launch_shape[3] == want and ens.step(chunk) == chunk
        got[shape] = [ens.retire(s, d[::-1]) for s, d in zip(slots, members)]
        ens.admit(_params((9, 9, 9), nc, tau_r=1.2), _state((9, 9, 9), nc), steps=1)
        assert ens.launch_shape[3] == (2 if want == 3 else want)
        ens.close()
    for shape, out in got.items():
        for a, b in zip(got[(16, 8, 4, 2)], out):
            assert np.array_equal(a["n"], b["n"]), shape
            assert nc == 2 or np.array_equal(a["db"], b["db"]), shape
    for a, d in zip(got[None], members):
        ref = _run(_params(d, nc, **kw), _state(d, nc), (16, 8, 16, 2), (21,))[0]
        assert np.array_equal(a["n"], ref["n"])


@pytest.mark.parametrize("nc,rock", [(3, False), (2, True)])
def test_download_planes(nc, rock):
    """Densities and momenta of a download are the FP64 sums, in direction order,
    over the populations of the same download; rock sites hold none."""
    dims = (13, 6, 7)
    g = np.array([2.0] * 6 + [1.0] * 13)
    c = np.array([(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (1, -1, 0),
                  (1, 0, 1), (1, 0, -1), (-1, 1, 0), (-1, -1, 0), (-1, 0, 1), (-1, 0, -1), (0, 1, 1), (0, 1, -1),
                  (0, -1, 1), (0, -1, -1), (0, 0, 0)], dtype=np.float64)
    st = _state(dims, nc, rock)
    out = _run(_params(dims, nc), st, (16, 8, 16, 3), (4,))[0]
    rho, mom = np.zeros_like(out["rho"]), np.zeros_like(out["mom"])
    for q in range(19):
        ng = out["n"][:, q] * g[q]
        rho += ng
        for k in range(3):
            mom[:, k] += ng * c[q, k]
    assert np.array_equal(out["rho"], rho) and np.array_equal(out["mom"], mom)
    if rock:
        assert not out["n"][:, :, st["rock"] != 0].any()
