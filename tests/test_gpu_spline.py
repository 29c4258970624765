"""The axial cubic splines at the sizes where the kernel's parts meet (the
longest grid solved by elimination alone, the shortest by sums, the edges of
a block and of the rows eliminated at either end) against SciPy."""
import numpy as np
import pytest

from test_gpu_parity import assert_same_polynomials

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nz', [5, 135, 136, 137, 138, 160, 161, 162, 163, 256, 257, 258, 288, 289, 290, 291, 385, 386,
                                1025, 4601, 12288])
def test_axial_cubic_sizes(cuda, nz):
    import torch
    from oracle.oracle import axial_coefficients
    z = np.linspace(-1e-3, 2e-3, nz)
    d = np.random.default_rng(nz).normal(size=(nz, 9)) * 10.0 ** np.arange(9)
    c = cuda.dev_axial_coefficients(cuda.to_dev(d, torch.float64), z[1] - z[0]).cpu().numpy()
    c_or = axial_coefficients(z, d)
    # SciPy takes each interval's own rounded width: nz 1e-16 of it, the tolerance of the other spline test
    assert_same_polynomials(c[:, 7:], c_or[:, 7:], z[1] - z[0], 1e-11)


def test_axial_cubic_range(cuda):
    import torch
    d = torch.zeros((12289, 9), dtype=torch.float64, device='cuda')
    with pytest.raises(cuda.BackendError):
        cuda.dev_axial_coefficients(d, 1e-6)
