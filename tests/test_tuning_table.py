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


@pytest.mark.gpu
@pytest.mark.parametrize("L,count", [(8, 37888), (26, 19000), (26, 30001)])
def test_one_and_two_ctas_per_sm_agree(L, count):
    """calls of one to two tiles per SM: with one CTA per SM each takes several tiles on its resident table"""
    import numpy as np
    import torch
    from sdpvibe_b200 import autotune
    from sdpvibe_b200.mpmat import lib_ctx
    R = lib_ctx(L)
    m = torch.tensor(R.mods, dtype=torch.int64, device="cuda")[:, None, None]
    acc = (torch.randint(0, 1 << 30, (R.n, 1, count), device="cuda") % m).to(torch.int16)
    rexp, cexp = torch.tensor([3], device="cuda"), torch.arange(count, device="cuda")
    saved, out = autotune.get_knob("crt_ctas"), []
    try:
        for ctas in (1, 2):
            autotune.set_knob("crt_ctas", ctas)
            out.append([t.cpu().numpy() for t in (*R.crt_block(acc, count, 0, count, 1)[:2],
                                                   *R.crt_norm(acc, count, 0, count, 1, rexp, cexp, L))])
    finally:
        autotune.set_knob("crt_ctas", saved)
    assert all(np.array_equal(a, b) for a, b in zip(*out))
