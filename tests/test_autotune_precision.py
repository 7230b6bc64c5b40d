"""What the autotuner leaves out (CPU, a fake timing model in place of the device): shapes that would interpolate
in FP32 where the library does not, knobs that nothing reads on a grid, and tunings cached for other kernels."""
import json

import pytest

from cfd_b200 import autotune
from test_autotune_logic import fake_model


@pytest.mark.parametrize("ng1,ng2,marches", [(384, 192, True), (256, 18, False), (384, 54, False), (54, 384, False)])
def test_march_is_searched_at_named_lengths(monkeypatch, ng1, ng2, marches):
    calls = []
    monkeypatch.setattr(autotune, "time_step", fake_model(calls))
    autotune.autotune(grid(ng1, ng2, 33), "mixed")
    assert any(json.loads(c)["xline_path"] == 6 for c in calls) == marches


def searched(monkeypatch, setup, precision, start, knob):
    """Values of a knob that the search times, from a library default of `start`."""
    calls = []

    def time_step(setup, precision, device, tuning, steps=5, warmup=2):
        eff = dict(start, **(tuning or {}))
        calls.append(eff[knob])
        return 1e-3, eff

    monkeypatch.setattr(autotune, "time_step", time_step)
    best, _ = autotune.autotune(setup, precision)
    assert best == start  # (no candidate is faster: the default stays)
    return set(calls)


def grid(ng1, ng2, planes):
    class S:
        class cfg:
            ngal1, ngal2 = ng1, ng2

        class grid:
            nyu = planes

        class ibu:
            n = 0
    return S


START = {"xline_path": 1, "xline_rows": 4, "zlines": 8, "solve_kind": 1, "solve_cols": 64, "rhs_chunk": 4, "xsplit": 1, "zsplit": 1}


def test_knobs_that_nothing_reads_are_not_timed(monkeypatch):
    assert searched(monkeypatch, grid(64, 96, 33), "fp64", START, "solve_cols") == {64}
    assert searched(monkeypatch, grid(64, 96, 736), "fp64", START, "solve_cols") == {64}
    assert searched(monkeypatch, grid(64, 96, 737), "fp64", START, "solve_cols") == {64, 128, 256}
    # 384 points march in FP64, by two rows
    assert searched(monkeypatch, grid(384, 384, 33), "fp64", dict(START, xline_rows=2), "xline_rows") == {2}
    assert searched(monkeypatch, grid(64, 96, 33), "fp64", START, "xline_rows") == {2, 4, 8}


def test_tunings_of_other_kernels_are_not_used(monkeypatch, tmp_path):
    torch = pytest.importorskip("torch")
    monkeypatch.setattr(autotune, "time_step", lambda *a, **k: (1e-3, dict(START, **(a[3] or {}))))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda device=None: "FAKE B200")
    path = tmp_path / "tune.json"
    monkeypatch.setenv("CFD_TUNE_CACHE", str(path))
    s = grid(384, 384, 348)
    path.write_text(json.dumps({"v9|FAKE B200|384x348x384|fp64|ibFalse": {"tuning": dict(START, xsplit=2), "ms_per_step": 1.0}}))
    assert autotune.tuned(s, "fp64")["xsplit"] == 1
    assert len(json.loads(path.read_text())) == 2
