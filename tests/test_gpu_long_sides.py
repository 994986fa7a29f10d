"""FP32 lattices with a side beyond 32767 sites: a state that repeats along the
long side stays the repeated short lattice's state, bit for bit."""
import numpy as np
import pytest

from lb3d_b200.config import Params
from lb3d_b200.ic import uniform_mixture

pytestmark = pytest.mark.gpu

PERIOD, TIMES = 16, 2100  # 33600 sites


def _params(dims, nc):
    return Params(nx=dims[0], ny=dims[1], nz=dims[2], ncomp=nc, tau_d=1.0, g_br=0.08, g_bs=-0.006, g_ss=-0.0045,
                  beta=10.0, d_0=1.0, bdist=2, restore=1, precision=1).finalize()


def _repeat(a, axis, times):
    """a, whose last axes are [nz][ny][nx], `times` times along x, y or z."""
    return np.concatenate([a] * times, axis=a.ndim - 1 - axis)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("nc,split", [(3, 2), (3, 3), (2, 2), (2, 3)])
def test_long_side(axis, nc, split):
    from lb3d_b200.lib import Lattice
    short = [2, 3, 4]
    short[axis] = PERIOD
    st = uniform_mixture(*short, nc, seed=9)
    out = []
    for times in (1, TIMES):
        dims = list(short)
        dims[axis] *= times
        lat = Lattice(_params(dims, nc))
        lat.upload(_repeat(st["n"], axis, times), _repeat(st["db"], axis, times) if nc == 3 else None)
        lat.set_launch_shape(16, 8, 16, split)
        lat.time_loop(3)
        got = lat.download()
        lat.close()
        out.append([_repeat(got[f], axis, TIMES // times) for f in ("n", "db")])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
