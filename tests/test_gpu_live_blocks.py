"""inv_x's blocks of live lines on rows that 8 does not divide.

Rows of 4, 6 and 12 kept modes (Nz = 8, 16, 24 and 32) take blocks of 8 lines that
run past a row on small grids, and blocks of 4 or 2 from 32 CTAs a field on.
Grids just below and above that line, x extents of every thread count, both
precisions, against the oracle: FP64 to 1e-12, FP32 to 2e-5 (as the other parity
tests on white spectra); and a batch whose instances together cross the line,
bit for bit against single runs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(64, 64, 32), (128, 64, 32), (256, 16, 32), (128, 128, 16), (32, 128, 24),
         (96, 128, 24), (384, 48, 8), (256, 64, 8), (512, 24, 16)]


@pytest.mark.parametrize("dims", GRIDS)
def test_blocks_match_the_oracle(dims):
    from ns3dperiodic_b200 import Solver
    from oracle import ns3d_oracle as O

    g = O.Grid(*dims)
    rng = np.random.default_rng(sum(dims))
    U = [O.r2c(g, rng.standard_normal(dims)) for _ in range(3)]
    want = np.stack(O.convolution(g, U))
    with Solver(*dims) as s:
        for precision, tol in (("fp64", 1e-12), ("fp32", 2e-5)):
            s.precision = precision
            got = s.calculate_convolution_2p3(s.to_device(U))
            s.synchronize()
            out = np.stack([c.cpu().numpy() for c in got])
            assert np.linalg.norm(out - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("dims,batch", [((32, 32, 32), 9), ((16, 16, 16), 24)])
def test_a_batch_across_the_line_equals_its_single_runs(dims, batch):
    from ns3dperiodic_b200 import Ensemble, Solver
    from oracle import ns3d_oracle as O

    g = O.Grid(*dims)
    base = [float(np.prod(dims)) * u for u in O.random_perturbation(g, 5)]
    U0 = [np.stack([u * (1.0 + 0.01 * b) for b in range(batch)]) for u in base]
    with Ensemble(batch, *dims) as e:
        e.set_params([1e-3] * batch, [20.0] * batch)
        got = [u.cpu().numpy() for u in e.rk3_steps(e.to_device(U0), 2)]
    with Solver(*dims) as s:
        for b in (0, batch - 1):
            V = s.rk3_ssp(s.to_device([u[b] for u in U0]), 1e-3, 20.0, 2)
            s.synchronize()
            assert all(np.array_equal(a[b], v.cpu().numpy()) for a, v in zip(got, V))
