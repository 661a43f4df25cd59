"""fwd_x on few and on many groups of lines gives the same bits.

Lines of 128 and 512 points run fwd_x_kernel up to 98 groups of lines (FP32
lines: 148) and the ring beyond, whose update spells out fwd_x_kernel's
multiply-adds.  A batch just below and just above that line takes the two
kernels through the plain and the combining update; every instance has to equal
its single run bit for bit, which takes fwd_x_kernel.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# groups of an instance: Ny Mz / (16 lines of 128 points, 4 of 512)
@pytest.mark.parametrize("precision,limit", [("fp64", 98), ("fp32", 148)])
@pytest.mark.parametrize("dims,groups", [((128, 16, 16), 9), ((512, 8, 8), 10)])
def test_instances_equal_their_single_runs(dims, groups, precision, limit):
    import torch

    from ns3dperiodic_b200 import Ensemble, Solver
    from oracle import ns3d_oracle as O

    g = O.Grid(*dims)
    vol = float(np.prod(dims))
    base = [vol * u for u in O.random_perturbation(g, 3)]
    F = O.kolmogorov_forcing(g)
    most = limit // groups
    for batch in (most, most + 1):
        dt = [1e-3 * (1.0 + 0.1 * b / batch) for b in range(batch)]
        re = [20.0 + b for b in range(batch)]
        U0 = [np.stack([u * (1.0 + 0.01 * b) for b in range(batch)]) for u in base]
        with Ensemble(batch, *dims) as e:
            e.set_precision(precision)
            e.set_forcing([torch.as_tensor(f, device="cuda") for f in F])
            e.set_params(dt, re)
            U = e.rk3_steps(e.to_device(U0), 2)
            torch.cuda.synchronize()
            got = [u.cpu().numpy() for u in U]
        with Solver(*dims) as s:
            s.precision = precision
            s.set_forcing(s.to_device(F))
            for b in (0, batch - 1):
                V = s.rk3_ssp(s.to_device([u[b] for u in U0]), dt[b], re[b], 2)
                s.synchronize()
                assert all(np.isfinite(v.cpu().numpy()).all() for v in V)
                assert all(np.array_equal(a[b], v.cpu().numpy()) for a, v in zip(got, V))
