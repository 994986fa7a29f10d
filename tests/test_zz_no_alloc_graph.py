"""The no-allocation FP64 step inside a captured CUDA graph: its kernels follow
each other with programmatic dependent launch, which becomes edges of the graph.
A replay between other work of the graph gives the allocating entry point's bits,
for an odd and an even number of steps.
"""
import numpy as np
import pytest

from lb3d_b200.config import Params
from lb3d_b200.ic import uniform_mixture

from .test_zz_no_alloc import _last_error, _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc,dims,steps", [(3, (16, 16, 16), 3), (3, (33, 31, 17), 4), (2, (40, 30, 29), 5)])
def test_captured_steps_match(nc, dims, steps):
    import torch
    from lb3d_b200.lib import Lattice

    p = Params(nx=dims[0], ny=dims[1], nz=dims[2], ncomp=nc, tau_d=1.0, g_br=0.08, g_bs=-0.006, g_ss=-0.0045,
               beta=10.0, d_0=1.0, bdist=2, restore=1).finalize()
    st = uniform_mixture(*dims, nc, seed=5)
    lat = Lattice(p, precision=0)
    lat.upload_state(st)
    lat.time_loop(2 * steps)
    ref = lat.download()
    lat.close()

    n0 = torch.from_numpy(np.ascontiguousarray(st["n"])).cuda()
    d0 = torch.from_numpy(np.ascontiguousarray(st["db"])).cuda() if nc == 3 else None
    f, db = torch.empty_like(n0), torch.empty_like(d0) if nc == 3 else None

    def enqueue():
        stream = torch.cuda.current_stream().cuda_stream
        f.copy_(n0)
        if nc == 3:
            db.copy_(d0)
        for _ in range(2):
            rc = _noalloc(p, f.data_ptr(), db.data_ptr() if nc == 3 else None, None, steps, stream)
            assert rc == 0, _last_error()

    enqueue()  # the first call looks the scratch address up, which a capture may not
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        enqueue()
    for _ in range(2):
        f.zero_()
        g.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(f.cpu().numpy(), ref["n"])
        if nc == 3:
            np.testing.assert_array_equal(db.cpu().numpy(), ref["db"])
