"""Axial table rows read 32 bytes at a time and quotients by a launch's constants
(tb_internal.cuh, tb_fastmath.cuh) against the plain reads and divisions: the
same bits, for tables that start at every multiple of 8 bytes and on both sides
of the grid's points."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_kernels import _probe

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('mine,lib', [(5, 13), (6, 14)])
def test_quotient_by_constant(cuda, mine, lib):
    rng = np.random.default_rng(2)
    x = np.concatenate([rng.uniform(-1, 1, 200000) * 10.0 ** rng.uniform(-80, 80, 200000), np.arange(5000) * 9.0,
                        np.arange(5000) * 0.00075, [0.0]])
    assert np.array_equal(_probe(cuda, x, mine), _probe(cuda, x, lib))


@pytest.mark.parametrize('Nz', [2, 3, 4, 101])
@pytest.mark.parametrize('offset', [0, 1, 2, 3])
def test_axial_rows(cuda, Nz, offset):
    import torch
    from conftest import load_probe
    lib = load_probe()
    zi = torch.linspace(-0.013, 0.017, Nz, dtype=torch.float64, device='cuda')
    table = torch.randn(offset + (Nz - 1) * 54, dtype=torch.float64, device='cuda')[offset:]
    z = torch.cat([zi, torch.nextafter(zi, zi - 1), torch.nextafter(zi, zi + 1),
                   -0.014 + 0.032 * torch.rand(1000, dtype=torch.float64, device='cuda')])
    out = torch.empty(2, len(z), 8, dtype=torch.float64, device='cuda')
    for wide in (0, 1):
        assert lib.tb_probe_axial(C.c_void_p(z.data_ptr()), C.c_int64(len(z)), C.c_void_p(zi.data_ptr()),
                                  C.c_void_p(table.data_ptr()), C.c_int64(Nz), wide, C.c_void_p(out[wide].data_ptr()),
                                  C.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    plain, rows = out.view(torch.int64).cpu()
    assert torch.equal(plain, rows)
