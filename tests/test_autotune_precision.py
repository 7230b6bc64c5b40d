"""The autotuner leaves out the shapes that would interpolate in FP32 where the library does not (CPU, a fake
timing model in place of the device)."""
import json

import pytest

from cfd_b200 import autotune
from test_autotune_logic import fake_model


@pytest.mark.parametrize("ng1,ng2,marches", [(384, 192, True), (256, 18, False), (384, 54, False), (54, 384, False)])
def test_march_is_searched_at_named_lengths(monkeypatch, ng1, ng2, marches):
    class S:
        class cfg:
            ngal1, ngal2 = ng1, ng2

    calls = []
    monkeypatch.setattr(autotune, "time_step", fake_model(calls))
    autotune.autotune(S, "mixed")
    assert any(json.loads(c)["xline_path"] == 6 for c in calls) == marches
