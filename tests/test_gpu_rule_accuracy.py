"""The fill's shorter quadrature rules and the ring tree's proxies against the
same kernels without them, so that what the two have in common (the degree of
K, E and G) does not hide a rule that is taken too near; and what the calls do
without their scratch."""
import numpy as np
import pytest
from scipy.special import ellipe, ellipkm1

from test_gpu_fill import MESHES, _inputs, _reference
from test_gpu_tree import _direct, _lens, _polyline, _sources

pytestmark = pytest.mark.gpu


def _field_scale(cuda, vt, types, values, jac, pos):
    """Per entry the sum of the absolute potential terms, or the factor times that of the field's (as a vector: where
    the normal is at right angles to it, the flux is only rounding), and the size of the coordinates over the distance
    between point and element."""
    t = cuda.dev_element_targets(vt)[0].cpu().numpy()
    r, z = pos[None, ..., 0], pos[None, ..., 1]
    r0, z0 = t[:, 0, None, None], t[:, 1, None, None]
    with np.errstate(divide='ignore', invalid='ignore'):
        dr, dz = r - r0, z - z0
        rho2, D = dr * dr + dz * dz, dz * dz + (r + r0) ** 2
        K, E = ellipkm1(rho2 / D), ellipe(1 - rho2 / D)
        c = jac[None] * r / (np.pi * np.sqrt(D))
        er = np.where(r0 < 1e-10, 0.0, c * (rho2 * K + abs(dr * dr - 2 * dr * r - dz * dz) * E) / (2 * r0 * rho2))
        field = np.hypot(er.sum(2), (c * abs(dz) * E / rho2).sum(2)) * abs(2 * (values - 1) / (1 + values))[:, None]
        size = (abs(t).sum(1)[:, None] + abs(t).sum(1)[None]) / np.sqrt(rho2.min(2))
    return np.where(np.isin(types, [3, 6])[:, None], field, (c * K).sum(2)), size


@pytest.mark.parametrize('name', list(MESHES))
def test_short_rules_against_sixteen_points_of_the_same_kernels(cuda, name):
    """Rings with doubled weights are not the map's own, so all 16 are summed; halved, they are the same sums."""
    import torch
    v = MESHES[name]()
    N = len(v)
    vt, t, val, jac, pos, types, values = _inputs(cuda, v, 200 + list(MESHES).index(name))
    A, B = (torch.zeros((N, N), dtype=torch.float64, device=vt.device) for _ in range(2))
    cuda.dev_fill_matrix(A, vt, t, val, jac, pos)
    cuda.dev_fill_matrix(B, vt, t, val, 2 * jac, pos)
    scale, size = _field_scale(cuda, vt, types, values, jac.cpu().numpy(), pos.cpu().numpy())
    # a term: 1 / sqrt (2 ulp), the logarithm (4e-16), two polynomials and five products, some 2e-15 at worst, and so
    # for each of the two sums; their additions 16 x 1.1e-16; the rules 1e-16 (uneven elements 5e-16).  The nodes'
    # coordinates: three roundings of 1.1e-16 each, which the field's 1 / distance^2 doubles, in both sums: 1.3e-15 of
    # the coordinates' size over the distance.  (Four points from 20 half-lengths on instead of 50 leave 1e-13.)
    off = ~np.eye(N, dtype=bool)
    assert np.all((A - 0.5 * B).abs().cpu().numpy()[off] <= ((6e-15 + 1.3e-15 * size) * scale)[off])


@pytest.mark.parametrize('name', ['ragged', 'arc', 'uneven'])
def test_gauss_diagonal(cuda, name):
    """gauss_diagonal: the 16-point sum of an element at its own middle."""
    import torch
    v = MESHES[name]()
    N = len(v)
    vt, t, val, jac, pos, types, values = _inputs(cuda, v, 7)
    A = torch.zeros((N, N), dtype=torch.float64, device=vt.device)
    cuda.dev_fill_matrix(A, vt, t, val, jac, pos, 0, N, accumulate=False, gauss_diagonal=True)
    ref, scale = _reference(cuda, vt, types, values, jac.cpu().numpy(), pos.cpu().numpy())
    # the degree-7 forms of K and E: 1.6e-13
    assert np.all(np.abs(A.cpu().numpy() - ref).diagonal() <= 5e-13 * scale.diagonal())


STRETCHES = {  # 2 mm long: half-length, middle and constant coordinate (mm)
    'tube': ([(1.5, -1.0), (1.5, 1.0)], 0.0, 1.5),
    'disc': ([(0.5, 0.25), (2.5, 0.25)], 1.5, 0.25),
}


@pytest.mark.parametrize('kind', list(STRETCHES))
@pytest.mark.parametrize('n', [32, 64])  # a root from its rings, and one from its children's proxies
def test_proxies_at_the_distance_where_they_are_first_taken(cuda, kind, n):
    """One charged element at the end of a stretch, seen from where the sum of the distances to the stretch's ends is
    10.2 to 10.4 half-lengths.  In extended precision the interpolation then leaves up to 8e-16 of the field; from
    8.2 half-lengths on (the ellipse of 8) it would leave 2e-15 to 1e-14."""
    import torch
    line, mid, across = STRETCHES[kind]
    v = _polyline(line, [n])
    q = np.zeros(n)
    q[-1] = 1.0
    src = _sources(cuda, v, q)
    M = 8192
    rng = np.random.default_rng(n)
    a = 0.5 * rng.uniform(10.2 * (1 + 1e-6), 10.4, M)  # the ellipse's half-axes for foci at +-1
    th = rng.uniform(0, 2 * np.pi, M)
    u, w = mid + a * np.cos(th), across + np.sqrt(a * a - 1) * np.sin(th)
    r, z = (w, u) if kind == 'tube' else (u, w)
    keep = r > 0.05
    p = 1e-3 * np.stack([r[keep], 0 * r[keep], z[keep]], 1)
    p = np.concatenate([p, p])[:M]
    assert len(p) * src.shape[1] >= 2e6
    p = np.tile(p, (2 if len(p) * src.shape[1] < 4e6 else 1, 1))
    pts = cuda.to_dev(p, torch.float64)
    assert cuda.backend_lib.tb_field_points_workspace(len(p), src.shape[1]) > 0
    _, f = cuda.dev_field_points(pts, src)
    _, g = _direct(cuda, pts, src)
    e = np.linalg.norm(f.cpu().numpy() - g, axis=1) / np.linalg.norm(g, axis=1)
    # rounding: a term some 4e-16 (root mean square), twice, times the root of the squared weights' sum (1.5 for 16
    # nodes), with the interpolation below 1.5e-15
    assert np.sqrt(np.mean(e * e)) <= 1.5e-15


def test_points_and_traces_without_scratch(cuda, monkeypatch):
    """With no memory for the tree the sums run ring by ring, bit for bit as the entries without it."""
    import torch
    from traceon_b200 import geometry as G
    from traceon_b200.field import EffectivePointCharges, FieldRadialBEM
    v = _lens(600)
    jac, pos = (a.cpu().numpy() for a in cuda.dev_jacobian_buffer(cuda.to_dev(v, torch.float64)))
    f = FieldRadialBEM(EffectivePointCharges(np.linspace(0.9e5, 1.1e5, 600), jac, pos))
    src = f.electrostatic_point_charges.device_sources()
    rng = np.random.default_rng(4)
    p = np.stack([rng.uniform(0, 2e-3, 900), np.zeros(900), rng.uniform(-4e-3, 4e-3, 900)], 1)
    pts = cuda.to_dev(p, torch.float64)
    x, u = G.surrogate_beam(40, 4)
    tr = f.get_tracer(G.LENS_BOUNDS)
    start, qm = tr._start(x, u, 9.1093837015e-31, -1.602176634e-19)
    tree = tr.trace_device(start, qm, plane_z=G.LENS_EXIT_Z)
    assert cuda.backend_lib.tb_field_points_workspace(900, src.shape[1]) > 0
    monkeypatch.setattr(cuda, 'dev_scratch', lambda *a: None)
    pot, field = cuda.dev_field_points(pts, src)
    pot2, field2 = _direct(cuda, pts, src)
    assert np.array_equal(pot.cpu().numpy(), pot2) and np.array_equal(field.cpu().numpy(), field2)
    rings = tr.trace_device(start, qm, plane_z=G.LENS_EXIT_Z)
    assert torch.equal(tree.status, rings.status) and torch.equal(tree.counters, rings.counters)
    # on the exit plane, as the trace through the tree and without
    assert float((tree.plane[:, 1:3] - rings.plane[:, 1:3]).abs().max()) < 1e-12
