"""The z pass's staged rows, at every z extent and a line count no CTA divides.

A CTA of the z pass takes 4 to 128 lines and copies whole groups of them; with
8 x 8 lines (and 24 x 8, whose last group is cut short) the groups of the short
extents are partly or wholly past the end.  Both forms of the product, both
precisions, against the oracle: FP64 to 1e-12, FP32 to 2e-5 (a white spectrum:
some 50 roundings of 6e-8 over the transforms' length, random in sign).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nxy", [(8, 8), (24, 8)])
@pytest.mark.parametrize("nz", [8, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512])
def test_products_at_every_z_extent(nz, nxy):
    from ns3dperiodic_b200 import Solver
    from oracle import ns3d_oracle as O

    dims = nxy + (nz,)
    g = O.Grid(*dims)
    rng = np.random.default_rng(nz)
    U, V = ([O.r2c(g, rng.standard_normal(dims)) for _ in range(3)] for _ in range(2))
    want = np.stack(O.convolution(g, U)), np.stack(O.convolution_uv(g, U, V))
    with Solver(*dims) as s:
        Ud, Vd = s.to_device(U), s.to_device(V)
        for precision, tol in (("fp64", 1e-12), ("fp32", 2e-5)):
            s.precision = precision
            got = s.calculate_convolution_2p3(Ud), s.calculate_convolution_2p3_uv(Ud, Vd)
            s.synchronize()
            for a, ref in zip(got, want):
                out = np.stack([c.cpu().numpy() for c in a])
                assert np.linalg.norm(out - ref) <= tol * np.linalg.norm(ref)
