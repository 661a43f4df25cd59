"""A multi-step tangent call keeps u's transforms between its evaluations.

Steps after the first of one ns3d_jvp_steps call start from the transforms the
step before left; calls of one step each make them anew.  Both have to agree (to
1e-12, FP32 mode 1e-5: the same sums, possibly rounded by differently compiled
kernels), also where u and v are the same arrays, which rules the reuse out.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 1e-5)])
@pytest.mark.parametrize("dims", [(8, 8, 8), (16, 24, 32), (64, 16, 48), (128, 32, 64)])
def test_steps_of_one_call_match_single_steps(dims, precision, tol):
    from ns3dperiodic_b200 import Solver
    from oracle import ns3d_oracle as O

    g = O.Grid(*dims)
    U0, V0 = O.random_perturbation(g, 1), O.random_perturbation(g, 2)
    vol = float(np.prod(dims))
    U0 = [vol * u for u in U0]
    with Solver(*dims) as s:
        s.precision = precision
        s.set_forcing(s.to_device(O.kolmogorov_forcing(g)))
        for same in (False, True):
            U, V = s.to_device(U0), s.to_device(V0)
            one = (U, U) if same else (U, V)
            U2, V2 = s.to_device(U0), s.to_device(V0)
            many = (U2, U2) if same else (U2, V2)
            for _ in range(4):
                s.rk3_ssp_uv(*one, 1e-3, 30.0, 1)
            s.rk3_ssp_uv(*many, 1e-3, 30.0, 4)
            s.synchronize()
            for A, B in zip(one, many):
                a, b = (np.stack([x.cpu().numpy() for x in F]) for F in (A, B))
                assert np.isfinite(a).all()
                assert np.linalg.norm(a - b) <= tol * np.linalg.norm(a)
