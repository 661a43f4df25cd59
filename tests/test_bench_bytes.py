"""The bench's byte and launch counts follow the passes.

pass_bytes against a count of the mask's modes, lines and planes on the oracle's
own mask; a factorisation's reads of the basis, three a column here and four in
the reference; and the launches of a tangent step against the nodes of a captured
call (GPU).
"""
import ctypes

import numpy as np
import pytest

import bench


@pytest.mark.parametrize("fp32", [False, True])
@pytest.mark.parametrize("N", [16, 24, 32])
def test_pass_bytes_count_what_the_mask_leaves(N, fp32):
    from oracle import ns3d_oracle as O

    keep = np.asarray(O.Grid(N, N, N).mask, bool).copy()
    keep[0, 0, 0] = True  # the mean is cut apart from the cut-offs
    el = 8 if fp32 else 16  # a scratch element; the state's have 16
    modes, lines = int(keep.sum()), int(keep.any(axis=0).sum()) * N
    kz = int(keep.any(axis=(0, 1)).sum()) * N * N
    full = N * N * (N // 2 + 1)
    inv_x = 3 * 16 * modes + 6 * el * lines
    inv_y = 6 * el * lines + 9 * el * kz
    z = 9 * el * kz + 3 * el * full
    fwd_y, fwd_x = 6 * el * full, (3 * el + 6 * 16) * full
    b = bench.pass_bytes(N, fp32)
    want = {"inv_x": inv_x, "inv_y": inv_y, "z": z, "fwd_y": fwd_y, "fwd_x": fwd_x}
    assert b["rhs"].keys() == want.keys()
    for name, v in want.items():
        assert b["rhs"][name] == pytest.approx(v, rel=1e-12), name
    nl = inv_x + inv_y + z + fwd_y + fwd_x
    uv = 2 * (inv_x + inv_y) + z + 9 * el * kz + fwd_y + fwd_x
    partner = 3 * 16 * full  # u^n of a combining update
    assert b["rk3"] == pytest.approx(3 * nl + 2 * partner, rel=1e-12)
    assert b["linearised"] == pytest.approx(uv, rel=1e-12)
    step = uv + (3 * nl + 2 * partner - inv_x - inv_y) + uv + partner
    assert b["jvp"] == pytest.approx(step, rel=1e-12)
    assert b["jvp_held"] == pytest.approx(step - inv_x - inv_y, rel=1e-12)


def test_basis_reads():
    n = 1000
    assert bench.arnoldi_bytes(n, 4) == 3 * (2 + 3 + 4) * n * 8
    assert bench.arnoldi_bytes(n, 4, fused=False) == 4 * (2 + 3 + 4) * n * 8
    assert bench.arnoldi_bytes(n, 50, first=47) == (3 * 48 + 4 * 49 + 4 * 50) * n * 8


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [1, 3])
def test_launches_of_a_tangent_step(steps):
    import torch

    from ns3dperiodic_b200 import Solver

    st = torch.cuda.Stream()
    drv = ctypes.CDLL("libcuda.so.1")
    raw, graph, count = ctypes.c_void_p(st.cuda_stream), ctypes.c_void_p(), ctypes.c_size_t()
    with Solver(16, 16, 16) as s:
        s.set_stream(st)
        U, V = s.zeros(), s.zeros()
        s.rk3_ssp_uv(U, V, 1e-3, 30.0, 1)  # the tangent scratch
        s.synchronize()
        s.set_stream(st)
        assert drv.cuStreamBeginCapture_v2(raw, 1) == 0
        s.rk3_ssp_uv(U, V, 1e-3, 30.0, steps)
        assert drv.cuStreamEndCapture(raw, ctypes.byref(graph)) == 0
        assert drv.cuGraphGetNodes(graph, None, ctypes.byref(count)) == 0
        assert drv.cuGraphDestroy(graph) == 0
    assert count.value == steps * bench.JVP_LAUNCHES
