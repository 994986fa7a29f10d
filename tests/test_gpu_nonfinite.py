"""Infinite and overflowing values on the FP64 path spread as in the oracle, NaN
for NaN and infinity for infinity: the stencil sums leave out the terms of zero
direction components, and those are not zero for a factor that is not finite."""
import numpy as np
import pytest

from lb3d_b200.config import Params
from lb3d_b200.ic import uniform_mixture
from tests._oracle import Oracle, set_math

pytestmark = pytest.mark.gpu

INF = np.inf
# field, index within the field's leading axes, value
PLANTS = {"dipole inf": ("db", (1,), INF), "dipole -inf": ("db", (2,), -INF), "dipole nan": ("db", (0,), np.nan),
          "dipole overflow": ("db", (0,), 1.7e308), "population inf": ("n", (0, 3), INF),
          "rest population inf": ("n", (-1, 18), INF),
          # psi = 1 - exp(-rho) overflows to -inf at a density of -1000
          "psi -inf": ("n", (0, 18), -1000.0), "psi -inf, last component": ("n", (-1, 18), -1000.0),
          "population overflow": ("n", (1, 6), 1.2e308)}
KINDS = {"ternary": (3, {}, False), "ternary, no surfactant coupling": (3, dict(g_bs=0.0, g_ss=0.0), False),
         "binary": (2, {}, False),
         "binary rock": (2, dict(g_wr=-0.1, g_wb=0.05, rock_colour_r=1.0), True),
         "sheared rock": (2, dict(boundary_cond=-1, inv_fluid=5, shear_u=0.05, g_wr=-0.1), True)}


@pytest.fixture(autouse=True, scope="module")
def _detmath():
    set_math(1)
    yield
    set_math(0)


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("plant", PLANTS)
def test_spread_as_in_the_oracle(kind, plant):
    from lb3d_b200.lib import Lattice
    nc, kw, rock = KINDS[kind]
    field, index, value = PLANTS[plant]
    if field == "db" and nc == 2:
        pytest.skip("binary lattices hold no dipoles")
    dims = (9, 10, 11)
    base = dict(nx=dims[0], ny=dims[1], nz=dims[2], ncomp=nc, tau_d=1.0, g_br=0.08, g_bs=-0.006, g_ss=-0.0045,
                beta=10.0, d_0=1.0, bdist=2, restore=1)
    base.update(kw)
    p, st = Params(**base).finalize(), uniform_mixture(*dims, nc, seed=6)
    if rock:
        st["rock"] = (np.random.default_rng(4).random(dims[::-1]) < 0.1).astype(np.float64)
        st["rock"][5, 4, 3] = 0
        st["n"] = st["n"] * (1 - st["rock"])
    st[field] = np.ascontiguousarray(st[field])
    st[field][index + (5, 4, 3)] = value
    lat, o = Lattice(p, precision=0), Oracle(p, st)
    lat.upload_state(st)
    for _ in range(2):
        lat.time_loop(1)
        o.run(1)
        a, b = lat.download(), o.get()
        for f in ("n", "rho", "mom") + (("db", "da") if nc == 3 else ()):
            np.testing.assert_array_equal(a[f], b[f], err_msg=f)
    lat.close()
