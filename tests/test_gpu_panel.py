"""The FP32 factorisation's one-launch panel steps at the sizes where their
parts meet: less than a block, blocks and panels just filled and just
exceeded, rows that fill and exceed a CTA, and the height at which tall panels
go to the separate kernels; row strides that are not the width."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n, pad', [(1, 0), (2, 3), (63, 0), (64, 1), (65, 0), (128, 0), (191, 2), (192, 0), (193, 0),
                                    (255, 0), (256, 0), (257, 3), (319, 0), (320, 0), (321, 0), (513, 0), (769, 1),
                                    (3711, 0), (3713, 0), (4097, 3)])
def test_lu_factors(cuda, n, pad):
    import torch
    g = torch.Generator('cuda').manual_seed(n)
    A = torch.rand((n, n), generator=g, device='cuda', dtype=torch.float64) - 0.5
    A += torch.diag(torch.full((n,), 0.5 * n ** 0.5 + 1.0, dtype=torch.float64, device='cuda'))
    full = torch.full((n, n + pad), 7.0, dtype=torch.float32, device='cuda')
    LU = full[:, :n]
    LU.copy_(A)
    cuda.dev_lu_nopiv_tc(LU)
    f = LU.double()
    L, U = torch.tril(f, -1) + torch.eye(n, device='cuda', dtype=torch.float64), torch.triu(f)
    # FP32 elimination of n steps: n u sum |l||u| at worst, sqrt(n) of it in the mean; growth is bounded by the
    # diagonal's dominance in the mean
    scale = (L.abs() @ U.abs()).max()
    assert float((L @ U - A).abs().max()) <= 2.0 ** -24 * 4 * (n ** 0.5 + 2) * float(scale)
    assert bool((full[:, n:] == 7.0).all())


@pytest.mark.parametrize('n', [1, 5, 64, 101, 257, 2501])
def test_mixed_solve_odd_sizes(cuda, n):
    """The whole mixed solve at widths that are not multiples of four (its factors have a padded row stride)."""
    import torch
    g = torch.Generator('cuda').manual_seed(n)
    A = torch.rand((n, n), generator=g, device='cuda', dtype=torch.float64) - 0.5
    A += torch.diag(torch.full((n,), 0.5 * n ** 0.5 + 1.0, dtype=torch.float64, device='cuda'))
    F = torch.rand((3, n), generator=g, device='cuda', dtype=torch.float64)
    X, it, rel = cuda.dev_solve_mixed(A, F)
    want = torch.linalg.solve(A, F.T).T
    assert float((X - want).abs().max()) <= 1e-10 * float(want.abs().max())
