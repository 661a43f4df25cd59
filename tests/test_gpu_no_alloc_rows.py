"""The allocation-free term has no wait that can give up.

The z pass of a handle stages long rows by bulk copies behind bounded waits and
reports a wait that gave up on the handle.  The allocation-free entry point has
no handle: its z pass reads every row where it is used.  At every z extent, on
grids whose lines no CTA divides: the launches of a call (as a captured graph
shows them) hold no staged form, and the result is the oracle's to 1e-12 (the
tolerance of the other parity tests).
"""
import ctypes
import re

import numpy as np
import pytest

from tests.test_zz_no_alloc import TOL, _field, _noalloc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxy", [(8, 8), (24, 8)])
@pytest.mark.parametrize("nz", [8, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512])
def test_rows_are_read_in_place(nz, nxy, tmp_path):
    import torch

    from ns3dperiodic_b200 import _lib
    from oracle import ns3d_oracle as O

    lib = _lib.lib()
    g = O.Grid(*nxy, nz)
    grid = (*nxy, nz, 2 * np.pi, 2 * np.pi, 2 * np.pi)
    Uh = _field(g.shape_c, nz)
    U = [torch.from_numpy(u).cuda() for u in Uh]
    Q = [torch.full(g.shape_c, complex(np.nan, np.nan), dtype=torch.complex128, device="cuda")
         for _ in range(3)]
    torch.cuda.synchronize()
    assert _noalloc(lib, grid, U, Q) == 0
    torch.cuda.synchronize()
    assert O.rel_l2([q.cpu().numpy() for q in Q], O.convolution(g, Uh)) <= TOL
    st = torch.cuda.Stream()
    drv = ctypes.CDLL("libcuda.so.1")
    graph, path = ctypes.c_void_p(), str(tmp_path / "g.dot")
    assert drv.cuStreamBeginCapture_v2(ctypes.c_void_p(st.cuda_stream), 1) == 0  # thread-local
    rc = _noalloc(lib, grid, U, Q, stream=st.cuda_stream)
    assert drv.cuStreamEndCapture(ctypes.c_void_p(st.cuda_stream), ctypes.byref(graph)) == 0
    assert rc == 0
    assert drv.cuGraphDebugDotPrint(graph, path.encode(), 1) == 0  # 1: verbose
    assert drv.cuGraphDestroy(graph) == 0
    text = open(path).read()
    names = set(re.findall(r"z_kernelI\w+", text))
    assert names, "no z pass in the captured call"
    staged = [n for n in names if nz > 64 and "Lb0E" not in n]  # STAGED = false
    assert not staged, staged
