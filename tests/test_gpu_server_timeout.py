"""Requests whose steps met a wait that gave up are reported so.

One bounded wait runs out on the grid's stream before the first step.  Both
requests in the grid's slots then ran beside it and end with the timeout,
however finite their fields; the one admitted after them is served as ever.
"""
import pytest

pytestmark = pytest.mark.gpu

TIMEOUT = 6  # NS3D_ERR_TIMEOUT


def test_the_active_requests_time_out_and_later_ones_do_not():
    from ns3dperiodic_b200 import Server
    from ns3dperiodic_b200._lib import lib

    N, T = 16, 0.05
    reqs = [(N, 100.0, T, seed, 0.0, 1) for seed in (1, 2, 3)]
    with Server([N], capacity=[2]) as srv:
        srv.submit(reqs)
        assert srv.run() == 3
        assert [r["status"] for r in srv.results()] == [0, 0, 0]
        want = srv.result_field(2, N)
    with Server([N], capacity=[2]) as srv:
        srv.submit(reqs)
        assert lib().ns3d_selftest_expire_server_wait(srv._h, N) == 0
        assert srv.run() == 3
        assert [r["status"] for r in srv.results()] == [TIMEOUT, TIMEOUT, 0]
        assert all((a == b).all() for a, b in zip(srv.result_field(2, N), want))
