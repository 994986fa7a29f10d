"""Work on a device that has almost no memory left: what strategy 3 takes beyond
strategy 2 makes way for what a call cannot do without."""
import contextlib

import numpy as np
import pytest

from lb3d_b200.config import Params
from lb3d_b200.ic import uniform_mixture

pytestmark = pytest.mark.gpu
MB = 1 << 20


@contextlib.contextmanager
def _only(left):
    """Leaves about `left` bytes of device memory free."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = []
    while True:
        free = torch.cuda.mem_get_info()[0]
        size = (free - left) // (2 * MB) * (2 * MB)
        if size < 12 * MB or len(held) == 8:
            break
        held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
    assert abs(torch.cuda.mem_get_info()[0] - left) < 16 * MB
    try:
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def _params(dims, nc=3, **kw):
    return Params(nx=dims[0], ny=dims[1], nz=dims[2], ncomp=nc, tau_d=1.0, g_br=0.08, g_bs=-0.006, g_ss=-0.0045,
                  beta=10.0, d_0=1.0, bdist=2, restore=1, precision=1, **kw).finalize()


@pytest.mark.parametrize("first", ["admit", "retire", "retire_async"])
def test_ensemble_gives_the_strategy_3_fields_back(first):
    """A 72^3 member's staging takes 170 MB (179 MB with its dipoles); 100 MB are
    left beside the fields of strategy 3 (216 MB)."""
    from lb3d_b200.ensemble import Ensemble
    from lb3d_b200.lib import lib
    dims, small = (72, 72, 72), (16, 16, 16)
    p, st = _params(dims), uniform_mixture(*dims, 3, seed=5)
    out = []
    for full in (False, True):
        ens = Ensemble(3, capacity_sites=2_000_000, max_lattices=4)
        before = lib().lb3dc_ensemble_bytes(ens.h)
        seeded = first != "admit"
        with contextlib.ExitStack() as stack:
            if full:
                stack.enter_context(_only(100 * MB))
            slot = ens.admit(p, None if seeded else st, steps=6, seed=11)
            assert slot is not None
            ens.step(3), ens.step(3), ens.sync()
            if first == "retire_async":
                ens.retire_async(slot, dims)
                while not ens.poll(slot):
                    pass
                got = ens.collect(slot)
            else:
                got = ens.retire(slot, dims)
            assert ens.launch_shape[3] == (2 if full else 3)
            assert lib().lb3dc_ensemble_bytes(ens.h) == before - (108 * 2_000_000 if full else 0)
            # and it goes on
            slot = ens.admit(_params(small), seed=3, steps=2)
            ens.step(2)
            more = ens.retire(slot, small)
        out.append((got, more))
        ens.close()
    for a, b in zip(*out):
        assert np.array_equal(a["n"], b["n"]) and np.array_equal(a["db"], b["db"])



def test_failed_admission_leaves_no_member():
    """Strategy 3's fields (28 MB) do not make enough room for the staging
    (114 MB): the request stays with the caller, and neither a slot
    nor its sites are taken."""
    from lb3d_b200.ensemble import Ensemble
    dims = (64, 64, 64)
    st = uniform_mixture(*dims, 3, seed=5)
    ens = Ensemble(3, capacity_sites=270_000, max_lattices=2)
    before = ens.stats()
    with _only(40 * MB):
        assert ens.admit(_params(dims), st, steps=2) is None
        assert ens.stats() == before
    slot = ens.admit(_params(dims), st, steps=2)
    assert slot == 0 and ens.step(2) == 2
    assert np.isfinite(ens.retire(slot, dims)["n"]).all()
    ens.close()


@contextlib.contextmanager
def _nothing():
    """Leaves no device memory free."""
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held, size = [], torch.cuda.mem_get_info()[0] // (2 * MB) * (2 * MB)
    while size >= 2 * MB:
        try:
            held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        except torch.OutOfMemoryError:
            size = size // (4 * MB) * (2 * MB)
    try:
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("split", [2, 3])
def test_a_launch_shape_without_room_leaves_the_present_one(split):
    """Chunks of one plane make a tile list of 6 MB on this lattice; nothing can
    make way for it (strategy 2: a lattice that strategy 3 does not apply to)."""
    from lb3d_b200.lib import LB3DC_ENOMEM, Lattice, Lb3dError
    dims = (2, 2, 300_000)
    p, st = _params(dims, 2, tau_r=1.2 if split == 2 else 1.0), uniform_mixture(*dims, 2, seed=5)
    out = []
    for full in (False, True):
        lat = Lattice(p)
        lat.upload_state(st)
        lat.set_launch_shape(32, 4, 64, split)
        lat.time_loop(2)
        lat.sync()
        with _nothing() if full else contextlib.nullcontext():
            if full:
                with pytest.raises(Lb3dError) as err:
                    lat.set_launch_shape(16, 8, 1, split)
                assert err.value.code == LB3DC_ENOMEM and lat.launch_shape == (32, 4, 64, split)
            lat.time_loop(3)
            lat.sync()
        out.append(lat.download()["n"])
        lat.close()
    assert np.array_equal(*out)


@pytest.mark.parametrize("what,per_site", [("dump", 586), ("autotune", 218), ("split 1", 26)])
def test_lattice_gives_the_strategy_3_fields_back(what, per_site):
    """A ternary lattice holds 44 bytes a site for strategy 3.  What is left lies
    22 bytes a site below what the call needs (a dump 608, the tuner's copy of
    the state 240, the own-moment field of strategy 1 48)."""
    from lb3d_b200.lib import Lattice
    dims = (128, 128, 128)
    n = 128 ** 3
    p, st = _params(dims), uniform_mixture(*dims, 3, seed=5)
    out = []
    for full in (False, True):
        lat = Lattice(p)
        lat.upload_state(st)
        lat.time_loop(2)
        lat.sync()
        held = lat.device_bytes
        assert lat.launch_shape[3] == 3
        got = []
        with _only(per_site * n) if full else contextlib.nullcontext():
            if what == "dump":
                got.append(lat.dump("od"))
                held += 8 * n  # the dump's output
            elif what == "autotune":
                lat.autotune()
            else:
                lat.set_launch_shape(16, 8, 16, 1)
                held += (48 - (44 if full else 0)) * n
            if full or what != "autotune":
                assert lat.launch_shape[3] == (1 if what == "split 1" else 3)
                assert lat.device_bytes == held
            lat.time_loop(3)
            lat.sync()
        state = lat.download()
        out.append(got + [state["n"], state["db"]])
        lat.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_sheared_fp64_lattice_without_room_for_its_boundary_planes():
    """A thin sheared lattice whose post-stream boundary planes (152 MiB) do not
    fit beside the rest (513 MiB): it steps all the same, to the same bits."""
    from lb3d_b200.lib import Lattice
    dims = (2, 512, 512)
    p = _params(dims, 2, boundary_cond=-1, inv_fluid=5, shear_u=0.05)
    st = uniform_mixture(*dims, 2, seed=5)
    out = []
    for full in (False, True):
        with _only(590 * MB) if full else contextlib.nullcontext():
            lat = Lattice(p, precision=0)
        lat.upload_state(st)
        lat.time_loop(3)
        out.append((lat.download(), lat.device_bytes))
        lat.close()
    for f in out[0][0]:
        assert np.array_equal(out[0][0][f], out[1][0][f]), f
    assert out[0][1] - out[1][1] == 2 * 2 * 19 * 512 * 512 * 8
