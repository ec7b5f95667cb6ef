"""The autotuner's file: a choice is taken from it only for the library build that it was timed with (no GPU: the timing is
replaced by a count)."""
import json

import numpy as np
import pytest

from cubokit_b200 import autotune


@pytest.fixture
def timed(tmp_path, monkeypatch):
    monkeypatch.setenv("CUBOKIT_B200_CACHE", str(tmp_path))
    monkeypatch.setattr(autotune, "device_name", lambda device=0: "GPU")
    calls = []

    def time(*args):
        calls.append(args)
        return 2, {"16x16": 1.0}

    monkeypatch.setattr(autotune, "_time", time)
    return calls


def _tune():
    return autotune.tune(None, [0] * 9, np.ones((80, 90)), np.ones((64, 64)))


def test_one_timing_per_library(timed, monkeypatch):
    assert _tune() == _tune() == (2, {"16x16": 1.0}) and len(timed) == 1
    monkeypatch.setattr(autotune, "library_id", lambda: "another build")
    assert _tune()[0] == 2 and len(timed) == 2
    assert _tune()[0] == 2 and len(timed) == 2


def test_choices_of_unknown_builds_are_timed_again(timed, tmp_path):
    k = "gather|" + autotune.key((64, 64), (80, 90), 9, "fp32", "GPU")
    (tmp_path / "autotune.json").write_text(json.dumps({k: {"choice": 3, "ms": {}}}))
    assert _tune()[0] == 2 and len(timed) == 1
    assert json.loads((tmp_path / "autotune.json").read_text())[k]["library"] == autotune.library_id()
