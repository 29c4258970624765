"""How the ring tree deals its chunks out: meshes whose neighbouring elements
are not on one line must not be slower through the tree than ring by ring."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_tree import _lens

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
