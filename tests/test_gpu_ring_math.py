"""Device math of the ring field sums (tb_fastmath.cuh): the one-step
reciprocal square root and the table logarithm against the CUDA library
functions, over the arguments the sums produce (rho^2 squared times D, and t
in (0, 1]) and at the edges of the table's intervals."""
import numpy as np
import pytest

from test_gpu_kernels import _probe, _ulps

pytestmark = pytest.mark.gpu


def test_rsqrt_one_step(cuda):
    x = 10.0 ** np.random.default_rng(0).uniform(-90, 30, 200000)
    # the step's own roundings: half an ulp each of x*y's error in e (halved) and of the result, and the library's
    assert np.max(_ulps(_probe(cuda, x, 3), _probe(cuda, x, 11))) <= 2


def test_neglog_table(cuda):
    rng = np.random.default_rng(1)
    edge = np.array([0x3fe6a09e + 0x2000 * i for i in range(129)], dtype=np.uint64) << np.uint64(32)
    edge = edge.view(np.float64)
    x = np.concatenate([10.0 ** rng.uniform(-300, 0, 100000), 1 - 10.0 ** rng.uniform(-16, -1, 50000),
                        edge, np.nextafter(edge, 0), edge / 2, [1.0, 0.5, 2.0 ** -600]])
    mine, lib = _probe(cuda, x, 4), -_probe(cuda, x, 12)
    # table entry (half an ulp of at most 0.35), r's rounding (2^-53 2^-8), and the two final additions
    assert np.max(np.abs(mine - lib) / (1.0 + np.abs(lib))) <= 4e-16
    assert mine[x == 1.0] == 0.0
