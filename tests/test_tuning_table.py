"""The autotuner's table and its cases: every knob has a value that was timed, as fast as any within the 2 % that its
timings repeat to, and the CRT's cases are of the size that reads the knob (more than one and at most two tiles of 128
entries per SM)."""
import json

import pytest

SMS = 148


def test_table_covers_the_knobs():
    from sdpvibe_b200 import autotune
    with open(autotune.TABLE) as f:
        table = json.load(f)
    assert set(table["knobs"]) == set(table["ms"]) == set(autotune.KNOBS)
    for name, (_, values) in autotune.KNOBS.items():
        assert table["knobs"][name] in values
        assert set(table["ms"][name]) == {str(v) for v in values}
        assert table["ms"][name][str(table["knobs"][name])] <= 1.02 * min(table["ms"][name].values())


@pytest.mark.gpu
def test_crt_cases_reach_the_knob(monkeypatch):
    from sdpvibe_b200 import autotune, rns
    tiles = []
    monkeypatch.setattr(rns.RNS, "crt_block", lambda self, acc, N, j0, w, rows: tiles.append((rows * w + 127) // 128))
    monkeypatch.setattr(rns.RNS, "crt_norm", lambda self, acc, N, j0, w, rows, *a: tiles.append((rows * w + 127) // 128))
    monkeypatch.setattr(autotune, "KNOBS", {"crt_ctas": autotune.KNOBS["crt_ctas"]})
    monkeypatch.setattr(autotune, "_time", lambda fn, reps: fn() or 1.0)
    monkeypatch.setattr(autotune, "_gram_case", lambda *a: None)
    autotune.tune(1)
    assert tiles and all(SMS < t <= 2 * SMS for t in tiles)
