"""Field sums at points that are on the axis or not a number, on every path
that a call can take: a cluster or a warp per point, and the ring tree."""
import numpy as np
import pytest

from test_gpu_tree import _lens, _sources

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('n, M', [(40, 1), (40, 200), (40, 3000), (1000, 64), (1000, 300), (1000, 3000)])
def test_points_on_the_axis_and_without_a_number(cuda, n, M):
    import torch
    v = _lens(n)
    src = _sources(cuda, v, np.random.default_rng(1).uniform(0.5, 2, n))
    assert (cuda.backend_lib.tb_field_points_workspace(M, src.shape[1]) > 0) == (n == 1000 and M > 250)
    nan, h = np.nan, 2e-3
    special = np.array([(0.0, 0.0, h), (-0.0, 5e-11, h), (-5e-11, -5e-11, -h), (nan, 1e-3, h), (1e-4, nan, h),
                        (nan, nan, 0.0), (1e-4, 2e-4, nan), (0.0, 0.0, nan), (1e-4, -2e-4, h)])
    for k in range(len(special)):
        p = np.tile(special[-1], (M, 1))
        p[M // 2] = special[k]
        pot, f = cuda.dev_field_points(cuda.to_dev(p, torch.float64), src)
        f, pot = f[M // 2].cpu().numpy(), float(pot[M // 2])
        r = np.hypot(p[M // 2, 0], p[M // 2, 1])
        if not r >= 1e-10:
            assert f[0] == 0.0 and f[1] == 0.0 and not np.signbit(f[:2]).any()
        assert np.isnan(f[2]) == np.isnan(pot) == np.isnan(special[k]).any()
