"""How the ring tree deals its chunks out: meshes whose neighbouring elements
are not on one line must not be slower through the tree than ring by ring."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_tree import _arc, _lens, _points, _polyline, _scale, _sources

pytestmark = pytest.mark.gpu


def _time(fn, reps=5):
    """Median device time of fn(), us."""
    import torch
    fn()
    out = []
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        out.append(1e3 * a.elapsed_time(b))
    return sorted(out)[reps // 2]


class _Trace:
    """n particles (at most 60 attempts each) in the field of a mesh, through the tree or ring by ring."""

    def __init__(self, cuda, v, n, tw):
        import torch
        from traceon_b200 import geometry as G
        from traceon_b200.field import EffectivePointCharges, FieldRadialBEM
        jac, pos = (a.cpu().numpy() for a in cuda.dev_jacobian_buffer(cuda.to_dev(v, torch.float64)))
        f = FieldRadialBEM(EffectivePointCharges(np.random.default_rng(3).uniform(0.9e5, 1.1e5, len(v)), jac, pos))
        x, u = G.surrogate_beam(n, 4)
        self.B, self.n, self.keep = cuda, n, f
        self.start, self.qm = f.get_tracer(G.LENS_BOUNDS)._start(x, u, 9.1093837015e-31, -1.602176634e-19)
        self.field, self.arrays = f._trace_field()
        o = self.o = cuda.TbTraceOpts()
        for i, b in enumerate(G.LENS_BOUNDS.reshape(-1)):
            o.bounds[i] = float(b)
        o.atol, o.max_attempts, o.team_warps, o.plane_z, o.record_plane = 1e-8, 60, tw, G.LENS_EXIT_Z, 1
        self.status = torch.empty(n, dtype=torch.int32, device='cuda')
        self.final = torch.empty((n, 7), dtype=torch.float64, device='cuda')
        self.plane = torch.empty_like(self.final)
        self.count = torch.empty((n, 2), dtype=torch.int64, device='cuda')
        self.work = torch.empty(1, dtype=torch.int32, device='cuda')
        self.nbytes = cuda.backend_lib.tb_trace_workspace(C.byref(self.field), n, 0)
        assert self.nbytes > 0
        self.scratch = cuda.dev_scratch(self.nbytes, self.status.device)

    def run(self, tree):
        self.B._call('tb_trace_rk45_ws', self.start.data_ptr(), None, self.qm.data_ptr(), None, self.n,
                     C.byref(self.field), None, 0, None, C.byref(self.o), None, None, self.status.data_ptr(),
                     self.final.data_ptr(), self.plane.data_ptr(), self.count.data_ptr(), self.work.data_ptr(),
                     self.scratch.data_ptr() if tree else None, self.nbytes, self.B._stream())


def _some_single():
    """500 of 1,600 elements in an order that puts no two neighbours on one line."""
    v = _lens(1600)
    odd = v[np.random.default_rng(0).permutation(1600)[:500]]
    return np.concatenate([odd, v[:1100]])


@pytest.mark.parametrize('n, tw', [(1, 8), (150, 8), (600, 4)])
def test_single_element_runs_are_shared_by_the_team(cuda, n, tw):
    t = _Trace(cuda, _some_single(), n, tw)
    assert _time(lambda: t.run(True)) <= 1.5 * _time(lambda: t.run(False))


def _mesh(kind, n):
    if kind == 'lens':
        return _lens(n)
    if kind == 'cone':
        return _polyline([(0.5, -2.0), (1.5, -1.0), (2.5, 2.0)], [n // 2, n - n // 2])
    if kind == 'shuffled':
        return _lens(n)[np.random.default_rng(0).permutation(n)]
    if kind == 'mixed':
        return np.concatenate([_arc(n // 4), _lens(n - n // 4)])
    return _arc(n)


MESHES = ['lens', 'arc', 'cone', 'shuffled', 'mixed']


def _both(cuda, pts, src, pot=None):
    """The field by both entries: what to call, and where it goes."""
    import torch
    M, Nq = pts.shape[0], src.shape[1]
    nbytes = cuda.backend_lib.tb_field_points_workspace(M, Nq)
    assert nbytes > 0
    work = cuda.dev_scratch(nbytes, pts.device)
    f = torch.empty((2, M, 3), dtype=torch.float64, device=pts.device)
    p = torch.empty((2, M), dtype=torch.float64, device=pts.device)
    ptr = (lambda i: p[i].data_ptr()) if pot else (lambda i: None)
    args = pts.data_ptr(), M, src.data_ptr(), Nq
    return (lambda: cuda._call('tb_field_radial_points_ws', *args, ptr(0), f[0].data_ptr(), work.data_ptr(), nbytes,
                               cuda._stream()),
            lambda: cuda._call('tb_field_radial_points', *args, ptr(1), f[1].data_ptr(), cuda._stream()), f, p)


@pytest.mark.parametrize('kind', MESHES)
@pytest.mark.parametrize('M', [64, 512, 4096])
def test_points_are_not_slower_than_the_direct_sums(cuda, kind, M):
    import torch
    rng = np.random.default_rng(M)
    src = _sources(cuda, _mesh(kind, 4096), rng.uniform(0.5, 2, 4096))
    pts = cuda.to_dev(np.stack([rng.uniform(0, 2e-3, M), np.zeros(M), rng.uniform(-5e-3, 5e-3, M)], 1), torch.float64)
    tree, direct, _, _ = _both(cuda, pts, src)
    # on 64 points the build takes a third of the direct sums' time
    assert _time(tree) <= 1.5 * _time(direct)


@pytest.mark.parametrize('kind', MESHES)
@pytest.mark.parametrize('M', [64, 74, 75, 148, 149, 296, 297, 592, 593, 1184, 1185])  # 32, 16, 8, 4, 2 and 1 warps a point
def test_points_with_several_warps(cuda, kind, M):
    import torch
    v = _mesh(kind, 4096)
    rng = np.random.default_rng(M)
    q = rng.standard_normal(len(v))
    src = _sources(cuda, v, q)
    p = _points(rng, v, max(M, 300))[:M]
    pts = cuda.to_dev(p, torch.float64)
    tree, direct, f, pot = _both(cuda, pts, src, pot=True)
    tree()
    direct()
    # both sums' terms carry the same error of K, E and G; the proxies 2 10^-16 x 2.7 (the Lebesgue constant of 16
    # nodes) = 6e-16 of them and the stretches' variation 1e-14 (TREE_JITTER) at most; roundings, 65,536 terms in
    # parts: some 1e-15.  The radial sum's terms are the larger ones of the form that _scale has.
    tol = 2e-14 * _scale(p, src.cpu().numpy())
    d = (f[0] - f[1]).abs().cpu().numpy()
    assert np.all(np.hypot(d[:, 0], d[:, 1]) <= 1.5 * tol[0]) and np.all(d[:, 2] <= tol[1])
    assert np.all((pot[0] - pot[1]).abs().cpu().numpy() <= tol[2])


@pytest.mark.parametrize('kind', ['arc', 'cone', 'shuffled'])
@pytest.mark.parametrize('n, tw', [(1, 8), (1024, 4), (4096, 1)])
def test_traces_are_not_slower_than_the_direct_sums(cuda, kind, n, tw):
    import torch
    t = _Trace(cuda, _mesh(kind, 800), n, tw)
    assert _time(lambda: t.run(True)) <= 1.25 * _time(lambda: t.run(False))
    t.run(True)
    plane, count = t.plane.clone(), t.count.clone()
    t.run(False)
    assert torch.equal(torch.isfinite(plane), torch.isfinite(t.plane)) and torch.equal(count, t.count)


@pytest.mark.parametrize('kind', MESHES)
@pytest.mark.parametrize('n, tw', [(3, 8), (70, 1)])
def test_traces_are_ring_by_ring_where_the_tree_is_of_no_use(cuda, kind, n, tw):
    """... bit for bit, and through the tree otherwise."""
    import torch
    t = _Trace(cuda, _mesh(kind, 400), n, tw)
    t.run(True)
    final, count = t.final.clone(), t.count.clone()
    t.run(False)
    same = torch.equal(final, t.final)
    assert torch.equal(count, t.count) and same == (kind in ('arc', 'cone', 'shuffled'))


@pytest.mark.parametrize('cut', [16 * 150, 16 * 150 + 8, 16 * 150 + 1])
def test_geometries_that_do_not_start_at_an_element(cuda, cut):
    """Source offsets that are not multiples of 16 rings: the rings that tb_trace_rk45_geometries sums."""
    import torch
    n = 24
    t = _Trace(cuda, _lens(400), n, 4)
    geom = torch.arange(n, dtype=torch.int32, device='cuda') % 2
    off = torch.tensor([0, cut, 16 * 400], dtype=torch.int64, device='cuda')
    nbytes = cuda.backend_lib.tb_trace_workspace(C.byref(t.field), n, 2)
    assert nbytes > 0
    work = cuda.dev_scratch(nbytes, off.device)
    args = (t.start.data_ptr(), None, t.qm.data_ptr(), geom.data_ptr(), n, C.byref(t.field), off.data_ptr(), 2, None,
            C.byref(t.o), None, None, t.status.data_ptr(), t.final.data_ptr(), t.plane.data_ptr(), t.count.data_ptr(),
            t.work.data_ptr())
    cuda._call('tb_trace_rk45_geometries', *args, cuda._stream())
    want, count = t.final.clone(), t.count.clone()
    t.final.zero_()
    cuda._call('tb_trace_rk45_ws', *args, work.data_ptr(), nbytes, cuda._stream())
    assert torch.equal(count, t.count)
    if cut % 16:
        assert torch.equal(want, t.final)
    else:  # through the tree; the field differs by some 1e-14, a trace of up to 60 steps by some 1e-12
        assert bool(((want - t.final).abs() <= 1e-10 * want.abs().amax(0)).all())
