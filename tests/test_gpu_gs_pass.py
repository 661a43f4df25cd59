"""The Gram-Schmidt passes at the edges of their column tiles and row blocks.

Factorisations over the 1-D Laplacian whose columns run through every register
tile (8, 16, ... 48 columns) and past the last one, at row counts below, at and
just above a block, a full grid of blocks and odd ones, against the oracle's
driver; and a continuation from the middle.  Tolerance 1e-11 of each result's
norm (as the factorisation tests have it: the basis' rounding, accumulated over
the columns, amplified by ||A|| / beta).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,m", [(100, 9), (128, 17), (129, 25), (1001, 50), (56832, 33),
                                 (56833, 8), (70001, 49)])
def test_factorisation_matches_the_oracle(n, m):
    import torch

    from ns3dperiodic_b200 import Krylov
    from oracle import krylov_oracle as K

    f0 = np.random.default_rng(n + m).standard_normal(n)
    V, H, f = np.zeros((m, n)), np.zeros((m, m)), f0.copy()
    K.arnoldi_driver(K.laplace1d, V, H, f, 0, m)
    kr = Krylov(n, m)
    A = kr.laplace_map()
    for k in (0, m // 2):
        Vd = torch.zeros((m, n), dtype=torch.float64, device="cuda")
        Hd = np.zeros((m, m))
        fd = torch.as_tensor(f0, device="cuda").clone()
        if k:
            kr.arnoldi(A, Vd, Hd, fd, 0, k)
        kr.arnoldi(A, Vd, Hd, fd, max(k - 1, 0), m)
        for got, ref in ((Vd.cpu().numpy(), V), (Hd, H), (fd.cpu().numpy(), f)):
            assert np.linalg.norm(got - ref) <= 1e-11 * np.linalg.norm(ref)
    kr.close()
