"""The batch solve's tile tasks at the edges of their range: one element, one
tile with and without padding, two tiles, and a geometry alone with many block
steps (every tile's products taken as they become final)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('sizes', [(1,), (63, 64, 65), (127, 128, 129, 2), (1400,)])
def test_tiles(cuda, port, sizes):
    from traceon_b200 import geometry as G
    from traceon_b200.batch import BatchSolve
    from traceon_b200.excitation import Excitation, Mesh
    geo = G.mirror_lens(1, n_range=(1500, 1500)).geometry
    mesh = []
    for n in sizes:
        pick = np.linspace(0, len(geo.vertices) - 1, n).astype(int) if n > 1 else np.array([len(geo.vertices) // 2])
        groups = {'a': np.arange(0, n, 2), 'b': np.arange(1, n, 2)}
        e = Excitation(Mesh(geo.vertices[pick].reshape(-1, 3), np.arange(4 * n).reshape(n, 4),
                            {k: g for k, g in groups.items() if len(g)}))
        e.add_voltage(**{k: u for k, u in (('a', 1.0), ('b', -2.0)) if len(groups[k])})
        mesh.append(e)
    bs = BatchSolve(mesh)
    got = bs.solve()
    assert (bs.status.cpu().numpy() == 0).all()
    for x, solver in zip(got, bs.solvers):
        vals = solver.device()[2].cpu().numpy()
        A = port.matrix(solver.vertices, np.ones(len(vals), np.uint8), vals, threads=8)
        y = np.linalg.solve(A, vals)
        # the bound of the ragged batch test: rounding of an LU with growth 1 and the fill's 1e-11
        assert np.max(np.abs(x - y)) <= 1e-10 * np.max(np.abs(y))
