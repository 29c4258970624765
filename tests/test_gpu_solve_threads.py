"""The mixed solve's factorisation enqueued by several host threads at once,
each on its own stream: the same factors, bit for bit, as one after another."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _factor(cuda, S):
    import torch
    n = S.shape[0]
    nbytes = cuda.backend_lib.tb_lu_nopiv_f32_tc_workspace(n)
    work = torch.empty(nbytes, dtype=torch.uint8, device=S.device)
    err = torch.zeros(1, dtype=torch.int32, device=S.device)
    LU = S.clone()
    cuda._call('tb_lu_nopiv_f32_tc', LU.data_ptr(), n, n, work.data_ptr(), nbytes, err.data_ptr(), cuda._stream())
    return LU, err, work


@pytest.mark.parametrize('threads', [2, 10])  # ten: more than there are side streams
def test_factors_from_several_threads(cuda, threads):
    import torch
    sizes = [900 + 332 * (k % 5) for k in range(threads)]
    rng = np.random.default_rng(7)
    mats, want = [], []
    for n in sizes:
        a = rng.uniform(-1, 1, (n, n)).astype(np.float32)
        a[np.arange(n), np.arange(n)] += np.float32(n)
        mats.append(torch.as_tensor(a, device='cuda'))
        want.append(_factor(cuda, mats[-1])[0])
    torch.cuda.synchronize()
    gate, bad = threading.Barrier(threads), []

    def run(k):
        try:
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                gate.wait(60)
                out = [_factor(cuda, mats[k]) for _ in range(12)]
            stream.synchronize()
            if any(int(e) for _, e, _ in out) or not all(torch.equal(LU, want[k]) for LU, _, _ in out):
                bad.append(k)
        except BaseException as e:  # noqa: BLE001 (reported by the main thread)
            bad.append((k, repr(e)))

    ts = [threading.Thread(target=run, args=(k,)) for k in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(300)
    assert not bad


def test_two_solves_in_one_capture_beside_another_solve(cuda):
    """A capture keeps its side stream until it ends: a solve outside it in the meantime takes another."""
    import torch
    n = 1300
    rng = np.random.default_rng(8)
    a = rng.uniform(-1, 1, (n, n)).astype(np.float32)
    a[np.arange(n), np.arange(n)] += np.float32(n)
    S = torch.as_tensor(a, device='cuda')
    want = _factor(cuda, S)[0]
    torch.cuda.synchronize()
    g, other = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    beside = []

    def outside():
        with torch.cuda.stream(other):
            beside.append(_factor(cuda, S))
        other.synchronize()

    with torch.cuda.stream(other):  # its memory, before the capture
        del_me = _factor(cuda, S)
    torch.cuda.synchronize()
    del del_me
    with torch.cuda.graph(g, capture_error_mode='thread_local'):
        first = _factor(cuda, S)
        t = threading.Thread(target=outside)
        t.start()
        t.join(120)
        second = _factor(cuda, S)
    g.replay()
    torch.cuda.synchronize()
    for LU, err, _ in (first, second, beside[0]):
        assert int(err) == 0 and torch.equal(LU, want)
