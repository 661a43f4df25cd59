"""A tangent call that fails leaves no graph under another call's arguments.

ns3d_jvp_steps keeps two captured steps (a call's first, its later ones) under
the arguments they were captured for.  Arguments change, one of the two captures
fails, and the call before comes again: it has to give what a fresh handle gives,
and must not touch the failed call's fields.  Tolerance: none, the same kernels.
"""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [0, 1])
def test_a_failed_capture_keeps_no_graph_of_its_call(graph):
    import torch

    from ns3dperiodic_b200 import Solver
    from ns3dperiodic_b200._lib import lib
    from oracle import ns3d_oracle as O

    dims = (16, 24, 32)
    g = O.Grid(*dims)
    U0, V0 = O.random_perturbation(g, 1), O.random_perturbation(g, 2)
    stream = torch.cuda.Stream()

    def fields(s):
        return s.to_device([1e3 * u for u in U0]), s.to_device(V0)

    def step(s, U, V, dt):
        s.rk3_ssp_uv(U, V, dt, 30.0, 3)
        s.synchronize()

    with Solver(*dims) as s, torch.cuda.stream(stream):
        s.set_stream(stream)
        U, V = fields(s)
        step(s, U, V, 1e-3)
        step(s, U, V, 1e-3)
        want = [x.clone() for x in U + V]
    with Solver(*dims) as s, torch.cuda.stream(stream):
        s.set_stream(stream)
        U, V = fields(s)
        other = fields(s)
        kept = [x.clone() for x in other[0] + other[1]]
        step(s, U, V, 1e-3)
        assert lib().ns3d_selftest_fail_capture(s._h, graph) == 0
        with pytest.raises(RuntimeError):
            step(s, *other, 2e-3)
        step(s, U, V, 1e-3)
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(U + V, want))
        assert all(torch.equal(a, b) for a, b in zip(other[0] + other[1], kept))
