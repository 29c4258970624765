"""The tracer's scratch for the ring tree: whose memory it is, and how long."""
import numpy as np
import pytest

from test_gpu_tree import _lens

pytestmark = pytest.mark.gpu


def test_scratch_is_not_memory_in_use_on_another_stream(cuda):
    """A block that was dropped here while this stream still works with it is not handed to another stream."""
    import torch
    n = 24 << 20
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    side = torch.cuda.Stream()
    a = torch.empty(n, dtype=torch.uint8, device='cuda')
    torch.cuda._sleep(20_000_000)  # some 10 ms of work before a's last use
    a.zero_()
    p = a.data_ptr()
    del a
    t = cuda.dev_scratch(n, torch.device('cuda', 0), side.cuda_stream)
    assert t is not None and t.data_ptr() != p
    torch.cuda.synchronize()


def _tracer(cuda, n):
    import torch
    from traceon_b200 import geometry as G
    from traceon_b200.field import EffectivePointCharges, FieldRadialBEM
    v = _lens(n)
    jac, pos = (a.cpu().numpy() for a in cuda.dev_jacobian_buffer(cuda.to_dev(v, torch.float64)))
    f = FieldRadialBEM(EffectivePointCharges(np.full(n, 1e5), jac, pos))
    tr = f.get_tracer(G.LENS_BOUNDS)
    x, u = G.surrogate_beam(64, 4)
    return tr, tr._start(x, u, 9.1093837015e-31, -1.602176634e-19), G.LENS_EXIT_Z


def test_results_do_not_hold_the_scratch(cuda):
    import torch
    tr, (start, qm), z = _tracer(cuda, 2000)
    tr.trace_device(start, qm, plane_z=z)  # the sources are on the device from here on
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    res = [tr.trace_device(start, qm, plane_z=z) for _ in range(4)]
    assert torch.cuda.memory_allocated() - before < 4 * 200_000  # one scratch: 2,000 elements, 1.7 MB
    assert all(torch.equal(r.final, res[0].final) for r in res)


def test_trace_on_a_given_stream_and_in_a_graph(cuda):
    """The same end states from the current stream, a given one, and replays of a capture whose result is held."""
    import torch
    tr, (start, qm), z = _tracer(cuda, 600)
    want = tr.trace_device(start, qm, plane_z=z).final
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    got = tr.trace_device(start, qm, plane_z=z, stream=side.cuda_stream)
    side.synchronize()
    assert torch.equal(want, got.final)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        res = tr.trace_device(start, qm, plane_z=z)
    junk = [torch.full((1 << 20,), 7.0, device='cuda') for _ in range(8)]
    for _ in range(2):
        res.final.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(want, res.final)
    del junk
