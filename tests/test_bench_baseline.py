"""bench.py's CPU baselines where the reference package is not staged: the
line says so instead of not being printed."""

import pytest

from oracle import ref_baseline


@pytest.mark.parametrize("call", [lambda b: b.cpu_baseline_full({})[0], lambda b: b.cpu_sweep_sample([], [])])
def test_missing_reference_is_reported(call, monkeypatch):
    import bench

    def missing():
        raise ImportError("reference package not staged")

    monkeypatch.setattr(ref_baseline, "import_reference", missing)
    monkeypatch.setattr(ref_baseline, "pin_threads", lambda n=None: 1)
    assert call(bench) == {"unavailable": "reference package not staged"}
