"""bench.py names the kernel that ran behind a timed family and counts that kernel's FLOPs (CPU only)."""
from __future__ import annotations

import sys
from pathlib import Path
from types import SimpleNamespace

import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1]))

import bench  # noqa: E402

DESIGN = SimpleNamespace(pin_count=1000, net_count=300)


@pytest.mark.parametrize("bins_x,bins_y,solve,kernel", [
    (64, 64, None, "fieldSmallKernel"), (128, 96, "", "fieldSmallKernel"), (64, 64, "banded", "fieldKernel"),
    (512, 512, None, "fieldKernel"), (100, 300, None, "fieldKernel"),
])
def test_field_families(monkeypatch, bins_x, bins_y, solve, kernel):
    if solve is None:
        monkeypatch.delenv("MPGP_FIELD_SOLVE", raising=False)
    else:
        monkeypatch.setenv("MPGP_FIELD_SOLVE", solve)
    for family in ("field_forward", "field_gradient", "field_inverse"):
        assert bench.kernel_of_family(family, bins_x, bins_y) == kernel
    assert bench.kernel_of_family("dct_inverse", bins_x, bins_y) == "tcGemmKernel"
    units = {k: v[1] for k, v in bench.algorithmic_units(DESIGN, 400, bins_x, bins_y).items()}
    along_x, along_y = 2.0 * bins_x * bins_y * bins_x, 2.0 * bins_x * bins_y * bins_y
    # Forward: one along each axis.  Inverse: two along y, and in one launch two along x as well.
    assert units["field_forward"] == along_x + along_y
    inverse = 2 * along_y + (2 * along_x if kernel == "fieldSmallKernel" else 0.0)
    assert units["field_inverse"] == inverse
    assert units["field_gradient"] == units["field_forward"] + inverse
