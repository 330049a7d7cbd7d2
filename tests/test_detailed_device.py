"""Detailed placement with its passes on the device against the host's lists (needs a GPU).

A memory budget that the host's lists fit but the device's passes do not takes the same design
down the host's path, so the two run on the same inputs: counters, HPWLs, centres and
orientations are equal bit for bit.  Designs with everything the device's kernels distinguish:
gaps, rows in any order, cells between rows, segment ends of two and three cells, nets of one
pin, above the degree limit and repeated in a window, modules without pins, and cells at the
same x of a row (whose order is the host sort's: the host's path runs).
"""
from __future__ import annotations

import numpy as np
import pytest

import myplacement_b200 as mp
from myplacement_b200.design import packed_placement

pytestmark = pytest.mark.gpu


def _case(seed: int, cells: int, gaps: float, spacing: float = 1.0) -> tuple[mp.Design, np.ndarray]:
    rng = np.random.default_rng(seed)
    design = mp.synthetic_design(cells=cells, nets=int(cells * 1.04), terminals=max(8, cells // 50),
                                 macros=max(1, cells // 2000), seed=seed, name=f"passes{seed}")
    if spacing != 1.0:
        design.module_width[:cells] = np.round(rng.uniform(0.6, 6.5, cells), 3)
        design.row_site_spacing[:] = spacing
        design.row_site_count[:] = np.ceil(design.row_site_count / spacing).astype(np.int64)
    design.pin_offset_x[:] = rng.uniform(-0.5, 0.5, design.pin_count) * design.module_width[design.pin_module]
    design.pin_offset_y[:] = rng.uniform(-0.5, 0.5, design.pin_count) * design.module_height[design.pin_module]
    design.net_weight[:] = rng.choice([1.0, 0.5, 2.0, 1.25, 0.0], design.net_count)
    placed = packed_placement(design, seed + 1, gap_probability=gaps)
    placed.module_orientation = rng.integers(0, 9, design.module_count).astype(np.int32)
    off_row = rng.random(design.module_count) < 0.01
    placed.module_y[off_row] += 0.25
    return placed, rng.integers(0, 9, design.row_bottom.shape[0]).astype(np.int32)


def _host_bytes(d: mp.Design) -> int:
    m, p, n = d.module_count, d.pin_count, d.net_count
    w, t = m // 4 + 1, m // 2 + 1
    return 54 * m + 40 * p + 4 * (n + 1) + 8 * n + w * 62 + 4 * (w + 1) + t * 46 + 4 * (t + 1)


def _compare(design, rows, **overrides):
    options = mp.default_detailed_options(**overrides)
    placed, result = mp.DetailedPlacer().run(design, options, row_orientation=rows)
    tight = mp.default_detailed_options(**overrides, maximum_cuda_memory_bytes=_host_bytes(design))
    expected, theirs = mp.DetailedPlacer().run(design, tight, row_orientation=rows)
    for key in ("hpwl_before", "hpwl_after", "evaluated_windows", "evaluated_permutations", "accepted_operations",
                "completed_passes"):
        assert result[key] == theirs[key], (key, result[key], theirs[key])
    assert np.array_equal(placed.module_x, expected.module_x) and np.array_equal(placed.module_y, expected.module_y)
    assert np.array_equal(placed.module_orientation, expected.module_orientation)
    return result, theirs


@pytest.mark.parametrize("cells,gaps,spacing", [(4, 0.0, 1.0), (5, 0.0, 1.0), (90, 0.5, 1.0), (3000, 0.08, 1.0),
                                                (3000, 0.08, 0.19), (20_000, 0.0, 1.0), (20_000, 0.35, 0.5)])
@pytest.mark.parametrize("passes,degree", [(1, 64), (3, 4)])
def test_device_equals_host(gpu, cells, gaps, spacing, passes, degree):
    design, rows = _case(cells + 7, cells, gaps, spacing)
    result, theirs = _compare(design, rows, passes=passes, maximum_net_degree=degree)
    assert result["cuda_reserved_memory_bytes"] > theirs["cuda_reserved_memory_bytes"]  # two paths


def test_long_dependency_chains(gpu):
    """One row of abutting cells whose neighbours are all connected: a decision of one window
    changes the next one's, so the rounds have a long chain to follow."""
    rng = np.random.default_rng(4)
    n = 4000
    design = mp.Design(module_width=rng.integers(1, 6, n).astype(float), module_height=np.full(n, 10.0),
                       module_x=np.zeros(n), module_y=np.full(n, 5.0), module_flags=np.zeros(n, np.int32),
                       net_weight=rng.uniform(0.5, 2.0, n), net_pin_start=np.arange(0, 3 * n + 1, 3),
                       pin_module=np.clip(np.arange(n)[:, None] + rng.integers(-6, 7, (n, 3)), 0, n - 1).ravel(),
                       pin_offset_x=rng.uniform(-1, 1, 3 * n), pin_offset_y=rng.uniform(-4, 4, 3 * n),
                       row_bottom=np.zeros(1), row_height=np.full(1, 10.0), row_site_width=np.ones(1),
                       row_site_spacing=np.ones(1), row_x_start=np.zeros(1), row_site_count=np.array([30_000]))
    left = np.concatenate([[0.0], np.cumsum(design.module_width)[:-1]])
    design.module_x[:] = left + design.module_width / 2
    result, _ = _compare(design, None, passes=4)
    assert result["accepted_operations"] > 0


def test_cells_at_the_same_x(gpu):
    design, rows = _case(11, 2000, 0.1)
    design.module_x[100:140] = design.module_x[100] + (design.module_width[100:140] - design.module_width[100]) / 2
    design.module_y[100:140] = design.module_y[100]
    result, theirs = _compare(design, rows, passes=2)
    assert result["cuda_reserved_memory_bytes"] == theirs["cuda_reserved_memory_bytes"]  # the host's path, both


def test_budget_limits(gpu):
    design, rows = _case(12, 500, 0.1)
    with pytest.raises(mp.EngineError):
        mp.DetailedPlacer().run(design, mp.default_detailed_options(maximum_cuda_memory_bytes=_host_bytes(design) - 1), row_orientation=rows)
