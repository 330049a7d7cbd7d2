"""The split autotuner times contraction launches at every size, or says that there are none."""
from __future__ import annotations

import os

import pytest

from myplacement_b200 import tune


def _engine(launches_of):
    """A stand-in for the profiled session: split 2 is the faster one where anything is launched."""

    def run(design, bins, warmup, iterations):
        launches = launches_of(bins, os.environ.get("MPGP_FIELD_SOLVE"))
        return (100.0 / tune.get_splits()[bins] if launches else 0.0), launches

    return run


@pytest.mark.parametrize("chosen", [None, "banded"])
def test_sizes_of_the_one_launch_solve_are_timed_staged(monkeypatch, chosen):
    if chosen is None:
        monkeypatch.delenv("MPGP_FIELD_SOLVE", raising=False)
    else:
        monkeypatch.setenv("MPGP_FIELD_SOLVE", chosen)
    monkeypatch.setattr(tune, "contraction_us_per_iteration",
                        _engine(lambda bins, solve: 40 if bins > 128 or solve == "staged" else 0))
    before = tune.get_splits()
    report = tune.tune([128, 256], 1, 1, 2)
    assert {bins: r["split"] for bins, r in report.items()} == {128: 2, 256: 2}
    assert report[128]["us_per_iteration"] == {1: 100.0, 2: 50.0}
    assert os.environ.get("MPGP_FIELD_SOLVE") == chosen and tune.get_splits() == before


def test_a_size_without_launches_is_refused(monkeypatch):
    monkeypatch.delenv("MPGP_FIELD_SOLVE", raising=False)
    monkeypatch.setattr(tune, "contraction_us_per_iteration", _engine(lambda bins, solve: 0))
    before = tune.get_splits()
    with pytest.raises(RuntimeError, match="no contraction launches"):
        tune.tune([128], 1, 1, 1)
    assert tune.get_splits() == before


@pytest.mark.gpu
def test_the_default_sizes_have_launches(gpu):
    report = tune.tune([128, 256], 1, 2, 1)
    assert all(us > 0.0 for r in report.values() for us in r["us_per_iteration"].values())
