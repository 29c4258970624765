"""Host logic of the autotuner's table (no GPU)."""
from traceon_b200 import autotune


def test_size_buckets():
    assert [autotune._bucket(x) for x in (0, 1, 2, 3, 1000, 1024, 1025)] == [0, 1, 2, 4, 1024, 1024, 2048]


def test_table_is_copied_and_cleared():
    autotune.clear()
    with autotune._lock:
        autotune._table[('k',)] = 4
    t = autotune.table()
    t[('k',)] = 8
    assert autotune.table() == {('k',): 4}
    autotune.clear()
    assert autotune.table() == {}


def test_lookahead_tuner_picks_the_fastest_width(monkeypatch):
    """tune_solve_lookahead with a fake backend: every candidate width is
    timed once, the fastest is left set, the setting in force before the
    tuning is restored around it, and a second call of the same size bucket
    reuses the table entry without timing again."""
    import types
    from traceon_b200 import backend as B
    state = {'reserve': 29, 'calls': []}

    def set_la(r):
        prev = state['reserve']
        state['reserve'] = 29 if r < 0 else r
        state['calls'].append(r)
        return prev

    cost = {0: 48.0, 15: 44.0, 30: 39.5, 44: 40.8}
    timed = []

    def fake_time(fn, reps=2):
        timed.append(state['reserve'])
        return cost[state['reserve']]

    class FakeCuda:
        @staticmethod
        def get_device_name(dev):
            return 'fake B200'

    monkeypatch.setattr(B, 'num_sms', lambda: 148)
    monkeypatch.setattr(B, 'set_solve_lookahead', set_la)
    monkeypatch.setattr(B, 'dev_solve_mixed', lambda A, F: None)
    monkeypatch.setattr(B, '_torch', lambda: types.SimpleNamespace(cuda=FakeCuda))
    monkeypatch.setattr(autotune, '_time_ms', fake_time)
    A = types.SimpleNamespace(shape=(16384, 16384), device='cuda:0')
    autotune.clear()
    try:
        hit = autotune.tune_solve_lookahead(A, None)
        assert sorted(timed) == [0, 15, 30, 44]
        assert hit == {'reserve_sms': 30, 'times_ms': cost}
        assert state['reserve'] == 30
        assert state['calls'][0] == -1 and state['calls'][-2:] == [29, 30]  # restored, then the choice set
        n = len(timed)
        state['reserve'] = 29
        assert autotune.tune_solve_lookahead(A, None)['reserve_sms'] == 30
        assert len(timed) == n and state['reserve'] == 30
    finally:
        autotune.clear()


def test_team_sizes_are_kept_apart_by_what_is_summed(monkeypatch):
    """Tracer.trace_device(team_warps='tune') on fields with the same number of rings: through the tree, with a
    magnetic part, with coils -- each is timed, and none takes another's choice."""
    import types
    from traceon_b200 import backend as B
    from traceon_b200.tracing import Tracer

    chosen = []

    class Lib:
        def __getattr__(self, name):
            return getattr(real, name)

        @staticmethod
        def tb_trace_workspace(field, n, geoms):
            f = field._obj
            return 0 if f.n_mag or f.n_cur or f.n_elec < 512 else 1000

        @staticmethod
        def tb_trace_rk45_ws(*args):
            chosen.append(args[9]._obj.team_warps)
            return B.TB_OK

    class Array:
        device, shape = 'cuda:0', (64, 6)

        def data_ptr(self):
            return 0

    def fake(n_elec, n_mag, n_cur):
        f = types.SimpleNamespace(_trace_field=lambda: (B.TbField(None, n_elec, None, n_mag, None, n_cur, None, None,
                                                                  None, None, 0), None))
        return Tracer(f, [[-1, 1]] * 3)

    real = B.backend_lib
    best = {}
    timed = []

    def fake_time(fn, reps=2):
        fn()
        timed.append(chosen[-1])
        return 1.0 if chosen[-1] == best['now'] else 2.0

    torch = types.SimpleNamespace(cuda=types.SimpleNamespace(get_device_name=lambda d: 'fake B200'),
                                  empty=lambda *a, **k: Array(), int32=0, int64=0, float64=0)
    monkeypatch.setattr(B, '_torch', lambda: torch)
    monkeypatch.setattr(B, '_stream', lambda: 0)
    monkeypatch.setattr(B, 'dev_scratch', lambda *a: None)
    monkeypatch.setattr(B, 'backend_lib', Lib())
    monkeypatch.setattr(autotune, '_time_ms', fake_time)
    autotune.clear()
    try:
        for now, rings in ((2, (16000, 0, 0)), (8, (8000, 8000, 0)), (4, (8000, 8000, 100_000)), (1, (16000, 0, 12))):
            best['now'] = now
            tr = fake(*rings)
            for again in (False, True):
                timed.clear()
                tr.trace_device(Array(), Array(), team_warps='tune')
                assert chosen[-1] == now
                assert timed == ([] if again else list(autotune.TEAM_CANDIDATES))
    finally:
        autotune.clear()
