"""A session set up on the device equals one set up on the host, bit for bit (needs a GPU).

Designs above the size from which the device sets a session up, with everything its kernels
distinguish: module orientations, fixed modules between movable ones, movable macros, modules
outside the core and without area, ragged and partial rows, nets of no, one and many pins, no
nets at all.  A memory budget that the host path fits but the device path's scratch does not
sends the same design down the host path.
"""
from __future__ import annotations

import numpy as np
import pytest

import myplacement_b200 as mp
from myplacement_b200 import _abi
from myplacement_b200.design import Design

pytestmark = pytest.mark.gpu


def _design(seed: int, modules: int, pins: int, fixed_share: float = 0.03) -> Design:
    rng = np.random.default_rng(seed)
    rows = 300
    flags = np.where(rng.random(modules) < fixed_share,
                     np.where(rng.random(modules) < 0.5, _abi.MODULE_FIXED, _abi.MODULE_TERMINAL), 0)
    width = rng.integers(1, 9, modules).astype(float)
    height = np.where(rng.random(modules) < 0.02, 24.0, 12.0)
    width[rng.random(modules) < 0.01] = 0.0
    side = 3600.0
    x = rng.uniform(-40.0, side + 40.0, modules)
    y = rng.uniform(-40.0, rows * 12.0 + 40.0, modules)
    degree = rng.integers(0, 9, max(1, pins // 4))
    degree[::97] = 70
    start = np.concatenate([[0], np.cumsum(degree)])
    start = start[: np.searchsorted(start, pins) + 1] if pins else np.zeros(1, np.int64)
    count = int(start[-1])
    order = rng.permutation(rows)
    return Design(
        module_width=width, module_height=height, module_x=x, module_y=y, module_flags=flags,
        net_weight=rng.uniform(0.5, 2.0, len(start) - 1), net_pin_start=start,
        pin_module=rng.integers(0, modules, count), pin_offset_x=rng.uniform(-4, 4, count),
        pin_offset_y=rng.uniform(-6, 6, count), row_bottom=order * 12.0, row_height=np.full(rows, 12.0),
        row_site_width=np.ones(rows), row_site_spacing=np.ones(rows),
        row_x_start=np.where(rng.random(rows) < 0.2, 100.0, 0.0),
        row_site_count=np.where(rng.random(rows) < 0.2, 3300, 3500),
        module_orientation=rng.integers(0, 9, modules), name=f"device_setup_{seed}")


def _run(design: Design, bins: tuple[int, int], **overrides):
    options = mp.default_options(bins_x=bins[0], bins_y=bins[1], target_density=0.9, iterations=4, **overrides)
    session = mp.Session(design, options)
    setup = mp.host_setup(design, options)
    start = session.positions(int(setup["particle_count"]))
    session.step(4)
    placed = session.finish()
    session.close()
    return setup, start, placed


@pytest.mark.parametrize("seed,modules,pins,bins", [
    (1, 40_000, 120_000, (64, 64)), (2, 9_000, 200_000, (100, 57)), (3, 140_000, 0, (130, 96)),
    (4, 70_000, 61_500, (33, 260)), (6, 12_000, 20_800, (64, 32)),
])
def test_device_and_host_set_ups_agree(gpu, seed, modules, pins, bins):
    design = _design(seed, modules, pins)
    setup, start, placed = _run(design, bins)
    movable = design.movable_mask
    count = int(setup["movable_count"])
    assert np.array_equal(start[:count, 0], design.module_x[movable])
    assert np.array_equal(start[:count, 1], design.module_y[movable])
    assert np.array_equal(start[count:], np.stack([setup["x"], setup["y"]], 1)[count:])
    options = mp.default_options(bins_x=bins[0], bins_y=bins[1], target_density=0.9, iterations=4)
    budget = mp.estimate_bytes(design, options)
    _, host_start, host_placed = _run(design, bins, maximum_cuda_memory_bytes=budget)
    assert np.array_equal(start, host_start)
    assert np.array_equal(placed.module_x, host_placed.module_x)
    assert np.array_equal(placed.module_y, host_placed.module_y)
    assert placed.history == host_placed.history
    different = ("elapsed_seconds", "cuda_reserved_memory_bytes")
    assert {k: v for k, v in placed.result.items() if k not in different} == {
        k: v for k, v in host_placed.result.items() if k not in different}


def test_overlapping_rows_are_refused(gpu):
    design = _design(5, 60_000, 120_000)
    design.row_bottom[1] = design.row_bottom[0]
    options = mp.default_options(bins_x=64, bins_y=64, target_density=0.9, iterations=2)
    with pytest.raises(mp.EngineError, match="Overlapping SiteRows"):
        mp.Session(design, options)
