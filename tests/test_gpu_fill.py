"""The matrix fill's shorter quadrature rules against the 16-point sums in
NumPy (scipy's elliptic integrals), over the sizes and elements where the
choice of the rule can go wrong: tile edges, row ranges, elements that are
sloped, curved, unevenly parametrised or given with other rings than their
own, potential and flux rows."""
import numpy as np
import pytest
from scipy.special import ellipe, ellipkm1

from test_gpu_tree import _arc, _lens, _polyline

pytestmark = pytest.mark.gpu

MM = 1e-3


def _stretched(v, a):
    """The elements with their inner points moved along them by the fraction a of their length."""
    v = v.copy()
    v[:, 2:] += a * (v[:, 1:2] - v[:, :1])
    return v


MESHES = {
    'one': lambda: _lens(9)[4:5],
    'tile - 1': lambda: _lens(63),
    'tile': lambda: _lens(64),
    'tile + 1': lambda: _lens(65),
    'ragged': lambda: _lens(517),
    'cone': lambda: _polyline([(0.5, -2.0), (1.5, -1.0), (1.5, 2.0)], [70, 131]),
    'graded': lambda: _polyline([(1.0, -2.0), (1.0, 2.0)], [400]) * np.array([1.0, 1.0, 1e-3]),
    'arc': lambda: np.concatenate([_arc(60), _polyline([(1.0, -3.0), (1.0, 3.0)], [77])]),
    'uneven': lambda: np.concatenate([_stretched(_lens(60), a) for a in (1e-9, 1e-6, 1e-4, 1e-2)]),
    'disc': lambda: _polyline([(0.0, 0.0), (3.0, 0.0)], [90]),
}


def _inputs(cuda, v, seed):
    import torch
    rng = np.random.default_rng(seed)
    types = rng.choice([1, 2, 3, 5, 6], len(v)).astype(np.uint8)
    values = rng.uniform(0.5, 5.0, len(v))
    vt = cuda.to_dev(v, torch.float64)
    jac, pos = cuda.dev_jacobian_buffer(vt)
    return vt, cuda.to_dev(types, torch.uint8), cuda.to_dev(values, torch.float64), jac, pos, types, values


def _reference(cuda, vt, types, values, jac, pos):
    """The 16-point sums and the sums of their absolute terms."""
    tgt, nrm = (a.cpu().numpy() for a in cuda.dev_element_targets(vt))
    r, z = pos[None, ..., 0], pos[None, ..., 1]
    r0, z0 = tgt[:, 0, None, None], tgt[:, 1, None, None]
    with np.errstate(divide='ignore', invalid='ignore'):
        dr, dz = r - r0, z - z0
        rho2 = dr * dr + dz * dz
        D = dz * dz + (r + r0) ** 2
        t = rho2 / D
        K, E = ellipkm1(t), ellipe(1 - t)
        q = jac[None] * r / (np.pi * np.sqrt(D))
        pot = q * K
        er = np.where(r0 < 1e-10, 0.0, q * (rho2 * K + (dr * dr - 2 * dr * r - dz * dz) * E) / (2 * r0 * rho2))
        era = np.where(r0 < 1e-10, 0.0, q * (rho2 * K + abs(dr * dr - 2 * dr * r - dz * dz) * E) / (2 * r0 * rho2))
        ez = -q * dz * E / rho2
    f = 2 * (values - 1) / (1 + values)
    flux = np.isin(types, [3, 6])[:, None]
    n = nrm * f[:, None]
    A = np.where(flux, n[:, :1] * er.sum(2) + n[:, 1:] * ez.sum(2), pot.sum(2))
    S = np.where(flux, abs(n[:, :1]) * era.sum(2) + abs(n[:, 1:]) * abs(ez).sum(2), pot.sum(2))
    return A, S


@pytest.mark.parametrize('name', list(MESHES))
def test_fill_rules_equal_sixteen_points(cuda, name):
    import torch
    v = MESHES[name]()
    N = len(v)
    vt, t, val, jac, pos, types, values = _inputs(cuda, v, list(MESHES).index(name))
    A = torch.full((N, N), 7.0, dtype=torch.float64, device=vt.device)
    cuda.dev_fill_matrix(A, vt, t, val, jac, pos)
    ref, scale = _reference(cuda, vt, types, values, jac.cpu().numpy(), pos.cpu().numpy())
    got = A.cpu().numpy()
    off = ~np.eye(N, dtype=bool)
    assert np.array_equal(got[~off], np.full(N, 7.0))
    # the degree-7 forms of K and E: 1.6e-13; the rules 1e-16 (5e-16 for uneven elements); rounding 1e-15
    assert np.all(np.abs(got - ref)[off] <= 5e-13 * scale[off])
    # a range of rows, added to what is there, with the diagonal's 16-point value
    r0, r1 = N // 3, N - N // 4
    B = torch.full((N, N), 3.0, dtype=torch.float64, device=vt.device)
    cuda.dev_fill_matrix(B, vt, t, val, jac, pos, r0, r1, accumulate=True, gauss_diagonal=True)
    b = B.cpu().numpy()
    assert np.array_equal(np.delete(b, np.s_[r0:r1], 0), np.full((N - (r1 - r0), N), 3.0))
    # 3 + a in one rounding
    assert np.all(np.abs(b - 3.0 - got)[r0:r1][off[r0:r1]] <= 4e-16 * (3.0 + np.abs(got)[r0:r1][off[r0:r1]]))


def test_fill_takes_the_rings_it_is_given(cuda):
    """Rings that are not the vertices' own (here: moved along z, with other weights) are summed as given."""
    import torch
    v = _lens(70)
    vt, t, val, jac, pos, types, values = _inputs(cuda, v, 3)
    pos[5, :, 1] += 2e-5
    jac[9] *= 1.5
    pos[64, 3, 0] *= 1 + 1e-10
    A = torch.empty((70, 70), dtype=torch.float64, device=vt.device)
    cuda.dev_fill_matrix(A, vt, t, val, jac, pos)
    ref, scale = _reference(cuda, vt, types, values, jac.cpu().numpy(), pos.cpu().numpy())
    off = ~np.eye(70, dtype=bool)
    assert np.all(np.abs(A.cpu().numpy() - ref)[off] <= 5e-13 * scale[off])


def test_fill_unknown_type(cuda):
    import torch
    v = _lens(66)
    vt, t, val, jac, pos, _, _ = _inputs(cuda, v, 4)
    t[65] = 4
    A = torch.zeros((66, 66), dtype=torch.float64, device=vt.device)
    cuda.dev_fill_matrix(A, vt, t, val, jac, pos)
    a = A.cpu().numpy()
    assert np.isnan(a[65, :65]).all() and np.isfinite(a[:65]).all()
