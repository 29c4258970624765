"""What the bench line says about rates that are not measured (CPU)."""
import json
import types

import bench


def test_units_that_are_not_computed_have_no_rate():
    r = bench.fp64_roofline(1e12, bench.FLOP_FIELD_PAIR, 10.0, 36.0, 'k', 'pairs of the direct sums', direct=False)
    assert r['achieved'] is None and r['frac'] is None and r['units'] == 1e12
    assert r['counts'] == 'direct-sum units'


def test_reference_arm_runs_the_reference_or_nothing(monkeypatch, capsys):
    from oracle import oracle
    monkeypatch.setattr(oracle, 'available', lambda kind: kind == 'port')
    monkeypatch.setattr(bench, 'cpu_reference_rate', lambda *a, **k: 1 / 0)
    bench.run_reference(types.SimpleNamespace(beam='wide', warmup=1, steps=1, ref_seconds=1.0))
    line = json.loads(capsys.readouterr().out)
    assert line['impl'] == 'reference' and 'not built' in line['unavailable'] and 'value' not in line


def test_cpu_baseline_names_what_ran():
    assert set(bench.CPU_TRACERS) == {'ref', 'port'}
    assert 'restatement' in bench.CPU_TRACERS['port'] and 'restatement' not in bench.CPU_TRACERS['ref']
