"""Field sums through the ring tree (tb_field_radial_points_ws) against the
direct sums (tb_field_radial_points): element orders, orientations and charges
that the tree takes and those that it has to leave to the rings, at points from
the axis to within a micrometre of an electrode."""
import numpy as np
import pytest
from scipy.special import ellipe, ellipkm1

pytestmark = pytest.mark.gpu

MM = 1e-3


def _lens(n, seed=1):
    from traceon_b200.geometry import einzel_lens
    return einzel_lens(n).vertices


def _polyline(pts, counts):
    from traceon_b200.geometry import polyline_elements
    return polyline_elements(np.array(pts) * MM, counts)


def _arc(n):
    """A half circle of radius 0.5 mm around (2, 0) mm."""
    a = np.linspace(np.pi / 2, 3 * np.pi / 2, 3 * n + 1)
    p = np.stack([2 + 0.5 * np.cos(a), 0 * a, 0.5 * np.sin(a)], 1) * MM
    return np.stack([p[0:-1:3], p[3::3], p[1::3], p[2::3]], 1)


GEOMETRIES = {
    'one': lambda: _lens(9)[:1],
    'few': lambda: _lens(33),
    'lens': lambda: _lens(1000),
    'fine': lambda: _lens(8001),
    'reversed': lambda: _lens(700)[::-1],
    'shuffled': lambda: _lens(700)[np.random.default_rng(0).permutation(700)],
    'twice': lambda: np.concatenate([_lens(300), _lens(300)]),
    'disc': lambda: _polyline([(0.0, 0.0), (3.0, 0.0)], [400]),
    'cone': lambda: _polyline([(0.5, -2.0), (1.5, -1.0), (1.5, 2.0), (3.0, 2.5)], [130, 257, 64]),
    'arc': lambda: np.concatenate([_arc(150), _polyline([(1.0, -3.0), (1.0, 3.0)], [333])]),
}


def _sources(cuda, vertices, charges):
    import torch
    v = cuda.to_dev(vertices, torch.float64)
    jac, pos = cuda.dev_jacobian_buffer(v)
    return cuda.dev_pack_sources(cuda.to_dev(charges, torch.float64), jac, pos)


def _points(rng, vertices, n=600):
    r, z = rng.uniform(0, 3.5 * MM, n), rng.uniform(-6 * MM, 6 * MM, n)
    r[:40] = 10.0 ** rng.uniform(-9, -4, 40)      # near the axis
    r[40:44] = 0.0
    k = rng.integers(0, len(vertices), 200)       # near an electrode
    near = vertices[k, 2] + rng.choice([-1, 1], (200, 3)) * 10.0 ** rng.uniform(-6, -3.5, (200, 1))
    r[100:300], z[100:300] = np.abs(near[:, 0]), near[:, 2]
    a = rng.uniform(0, 2 * np.pi, n)
    return np.stack([r * np.cos(a), r * np.sin(a), z], 1)


def _scale(p, src):
    """Per point, the sums of the absolute terms of (E_r, E_z, potential)."""
    rs, zs, w = src[:, None]
    r0, z0 = np.hypot(p[:, 0], p[:, 1])[:, None], p[:, 2:]
    out = np.empty((3, len(p)))
    for i in range(len(p)):
        dr, dz = rs - r0[i], zs - z0[i]
        rho2 = dr * dr + dz * dz
        D = dz * dz + (rs + r0[i]) ** 2
        t = rho2 / D
        K, E = ellipkm1(t), ellipe(1 - t)
        c = np.abs(w) * rs / (np.pi * np.sqrt(D))
        er = c * (rho2 * K + np.abs(dr * dr - 2 * dr * rs - dz * dz) * E) / rho2
        out[:, i] = er.sum() / max(2 * r0[i, 0], 1e-10), (c * np.abs(dz) * E / rho2).sum(), (c * K).sum()
    return out


def _direct(cuda, pts, src):
    import torch
    M = pts.shape[0]
    pot = torch.empty(M, dtype=torch.float64, device=pts.device)
    f = torch.empty((M, 3), dtype=torch.float64, device=pts.device)
    cuda._call('tb_field_radial_points', pts.data_ptr(), M, src.data_ptr(), src.shape[1], pot.data_ptr(), f.data_ptr(),
               cuda._stream())
    return pot.cpu().numpy(), f.cpu().numpy()


def _tree(cuda, pts, src):
    """The tree's sums whatever the size: the points repeated up to its rule."""
    import torch
    M, Nq = pts.shape[0], src.shape[1]
    k = 1
    while cuda.backend_lib.tb_field_points_workspace(k * M, Nq) == 0:
        k *= 2
    pot, f = cuda.dev_field_points(pts.repeat(k, 1).contiguous(), src)
    assert torch.equal(f[:M], f[-M:])
    return pot[:M].cpu().numpy(), f[:M].cpu().numpy()


@pytest.mark.parametrize('name', list(GEOMETRIES))
def test_tree_equals_direct_sums(cuda, name):
    import torch
    rng = np.random.default_rng(list(GEOMETRIES).index(name))
    v = GEOMETRIES[name]()
    q = rng.standard_normal(len(v)) if len(v) % 2 else rng.uniform(0.5, 2, len(v))
    src = _sources(cuda, v, q)
    p = _points(rng, v)
    pts = cuda.to_dev(p, torch.float64)
    (pot, f), (pot2, f2) = _direct(cuda, pts, src), _tree(cuda, pts, src)
    # the nodes' interpolation: 2 8^-16 times the Lebesgue constant of 16 nodes (2.7) = 2e-14 of the sum of the
    # absolute terms; the two sums' roundings (some 1e-15 a term, 16 N terms in 32 to 256 parts); and where a
    # stretch's constant coordinate varies by rounding, at most 1e-14 (TREE_JITTER)
    tol = 5e-14 * _scale(p, src.cpu().numpy())
    d = np.abs(f2 - f)
    assert np.all(np.hypot(d[:, 0], d[:, 1]) <= 1.5 * tol[0])
    assert np.all(d[:, 2] <= tol[1])
    assert np.all(np.abs(pot2 - pot) <= tol[2])


def test_tree_charges_without_a_number(cuda):
    """No charge at all, and charges that are not finite: the direct sums' values."""
    import torch
    v = _lens(600)
    pts = cuda.to_dev(_points(np.random.default_rng(5), v), torch.float64)
    q = np.zeros(len(v))
    pot, f = _tree(cuda, pts, _sources(cuda, v, q))
    assert not pot.any() and not f.any()
    for bad in (np.nan, np.inf):
        q[:] = 1.0
        q[123] = bad
        src = _sources(cuda, v, q)
        (pot, f), (pot2, f2) = _direct(cuda, pts, src), _tree(cuda, pts, src)
        assert np.array_equal(np.isnan(pot), np.isnan(pot2)) and np.array_equal(np.isnan(f), np.isnan(f2))
        assert np.array_equal(np.isinf(pot), np.isinf(pot2))


@pytest.mark.parametrize('tw', [1, 2, 4, 8])
def test_trace_through_the_tree_and_without(cuda, tw):
    """Exit-plane crossings and step counts of a beam through the tree against the direct sums (the C entry
    without scratch)."""
    import ctypes as C
    import torch
    from traceon_b200 import geometry as G
    from traceon_b200.field import EffectivePointCharges, FieldRadialBEM
    geo = G.einzel_lens(301)
    jac, pos = (a.cpu().numpy() for a in cuda.dev_jacobian_buffer(cuda.to_dev(geo.vertices, torch.float64)))
    q = geo.voltages_to_values([1e5, 1.5e6, -2e5]) * np.random.default_rng(2).uniform(0.9, 1.1, len(geo))
    f = FieldRadialBEM(EffectivePointCharges(q, jac, pos))
    x, u = G.surrogate_beam(150, 4)
    tr = f.get_tracer(G.LENS_BOUNDS)
    start, qm = tr._start(x, u, 9.1093837015e-31, -1.602176634e-19)
    res = tr.trace_device(start, qm, atol=1e-9, plane_z=G.LENS_EXIT_Z, team_warps=tw)
    field, keep = f._trace_field()
    assert cuda.backend_lib.tb_trace_workspace(C.byref(field), 150, 0) > 0
    o = cuda.TbTraceOpts()
    for i, b in enumerate(G.LENS_BOUNDS.reshape(-1)):
        o.bounds[i] = float(b)
    o.atol, o.max_attempts, o.team_warps = 1e-9, 100_000, tw
    o.plane_z, o.record_plane = G.LENS_EXIT_Z, 1
    st, pl, cnt = torch.empty_like(res.status), torch.empty_like(res.plane), torch.empty_like(res.counters)
    work = torch.empty(1, dtype=torch.int32, device=pl.device)
    cuda._call('tb_trace_rk45', start.data_ptr(), None, qm.data_ptr(), 150, C.byref(field), C.byref(o), None, None,
               st.data_ptr(), None, pl.data_ptr(), cnt.data_ptr(), work.data_ptr(), cuda._stream())
    assert torch.equal(st, res.status) and torch.equal(cnt, res.counters)
    # On the exit plane (the last step's own length follows the rounding of its error estimate): some 100
    # accepted steps, each amplifying a field difference of 5e-14 by the beam's own divergence.
    ok = torch.isfinite(pl[:, 0])
    assert torch.equal(ok, torch.isfinite(res.plane[:, 0]))
    assert float((pl[ok, 1:3] - res.plane[ok, 1:3]).abs().max()) < 1e-12
