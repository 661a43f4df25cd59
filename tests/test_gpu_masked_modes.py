"""The passes skip what the 2/3 mask removes: no stale scratch may reach a result.

The x and y passes neither write nor read the masked lines of their scratch, so
whatever an earlier call left there must not show.  A first call on a state of
NaNs fills every scratch element the passes touch with NaN; the next call has to
equal the oracle's and, bit for bit, a fresh handle's.  Grids: the smallest
extents, rows that cannot be padded to whole blocks of 8 modes (Nz = 8, 24), a
mode exactly on the mask's border (Nz = 16), lines of every thread count, and
extents that differ per direction.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(8, 8, 8), (16, 24, 16), (24, 8, 24), (48, 16, 32), (32, 96, 48), (8, 64, 128),
         (128, 8, 64), (16, 256, 96), (64, 24, 192), (16, 8, 512)]


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-12), ("fp32", 2e-5)])
@pytest.mark.parametrize("dims", GRIDS)
def test_no_stale_scratch(dims, precision, tol):
    import torch

    from ns3dperiodic_b200 import Solver
    from oracle import ns3d_oracle as O

    g = O.Grid(*dims)
    rng = np.random.default_rng(sum(dims))
    U, V = ([O.r2c(g, rng.standard_normal(dims)) for _ in range(3)] for _ in range(2))
    want, want_uv = O.convolution(g, U), O.convolution_uv(g, U, V)

    def both(s):
        s.precision = precision
        Ud, Vd = s.to_device(U), s.to_device(V)
        return (s.calculate_convolution_2p3(Ud), s.calculate_convolution_2p3_uv(Ud, Vd))

    with Solver(*dims) as s:
        fresh = both(s)
    with Solver(*dims) as s:
        s.precision = precision
        bad = [torch.full(s.shape, complex(float("nan"), float("nan")), dtype=torch.complex128,
                          device=s.device) for _ in range(3)]
        s.calculate_convolution_2p3(bad)
        s.calculate_convolution_2p3_uv(bad, bad)
        after = both(s)
    for got, again, ref in zip(fresh, after, (want, want_uv)):
        ref = np.stack(ref)
        assert all(torch.equal(a, b) for a, b in zip(got, again))
        out = np.stack([a.cpu().numpy() for a in again])
        assert np.linalg.norm(out - ref) <= tol * np.linalg.norm(ref)
