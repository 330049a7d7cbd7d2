"""Which path sets a session up: nothing that the host's set-up takes is refused (needs a GPU).

The device's set-up needs scratch beside the session's arrays: the design as it is, and per bin
row a list of the SiteRows and fixed modules that span it.  A design whose scratch does not fit
its memory budget is set up on the host.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

import myplacement_b200 as mp
from myplacement_b200 import _abi

pytestmark = pytest.mark.gpu


def _with_blocks(blocks: int, height: float, seed: int = 3, cells: int = 12_000) -> mp.Design:
    """A design with fixed blocks of `height` (a share of the core) that are a small part of a bin wide."""
    design = mp.synthetic_design(cells=cells, nets=cells, terminals=16, seed=seed)
    design = design.copy_with_positions(*mp.random_placement(design, seed))
    rng = np.random.default_rng(seed)
    llx, lly, urx, ury = design.core
    fields = {k: getattr(design, k) for k in design.__dataclass_fields__ if not k.startswith("_")}
    fields["module_width"] = np.concatenate([design.module_width, np.full(blocks, 1e-4 * (urx - llx))])
    fields["module_height"] = np.concatenate([design.module_height, np.full(blocks, height * (ury - lly))])
    fields["module_x"] = np.concatenate([design.module_x, rng.uniform(llx, urx, blocks)])
    fields["module_y"] = np.concatenate([design.module_y, rng.uniform(lly, ury, blocks)])
    fields["module_flags"] = np.concatenate([design.module_flags, np.full(blocks, _abi.MODULE_FIXED)])
    return mp.Design(**fields)


def _place(design: mp.Design, **overrides):
    options = mp.default_options(bins_x=256, bins_y=256, target_density=0.9, iterations=2, **overrides)
    return mp.GlobalPlacer().run(design, options)


@pytest.mark.parametrize("blocks,height", [(20_000, 1.0), (60_000, 0.3)])
def test_lists_beyond_the_budget(gpu, blocks, height):
    design = _with_blocks(blocks, height)
    # Every block is listed in each of the bin rows it spans, 40 bytes a time: about 200 MB, far more
    # than the rest of the set-up.
    options = mp.default_options(bins_x=256, bins_y=256, target_density=0.9, iterations=2)
    budget = mp.estimate_bytes(design, options) + (100 << 20)
    tight = _place(design, maximum_cuda_memory_bytes=budget)
    free = _place(design)
    assert tight.result["cuda_reserved_memory_bytes"] <= budget
    assert np.array_equal(tight.module_x, free.module_x) and np.array_equal(tight.module_y, free.module_y)
    assert tight.history == free.history


@pytest.mark.parametrize("bins", [(64, 64), (257, 320), (130, 96)])
def test_budgets_between_the_paths(gpu, bins):
    """From the budget that the host's set-up needs to one that the device's fits: no budget is
    refused, and the path makes no difference."""
    design = _with_blocks(500, 0.2, seed=5, cells=20_000)
    overrides = {"bins_x": bins[0], "bins_y": bins[1], "target_density": 0.9, "iterations": 2}
    need = mp.estimate_bytes(design, mp.default_options(**overrides))
    runs = [mp.GlobalPlacer().run(design, mp.default_options(maximum_cuda_memory_bytes=need + (extra << 20), **overrides))
            for extra in range(0, 56, 4)]
    for run in runs[1:]:
        assert np.array_equal(run.module_x, runs[0].module_x) and np.array_equal(run.module_y, runs[0].module_y)
        assert run.history == runs[0].history


@pytest.mark.parametrize("room", [0, 8 << 20, 1 << 30])
def test_served_set_ups_stay_within_the_budget(gpu, room):
    """A served job is admitted by its estimate; what a set-up on the device holds beyond that is
    taken out of the server's budget too, or the host sets the job up."""
    design = _with_blocks(100, 0.1, seed=6)  # short lists: the device takes it where memory allows
    options = mp.default_options(bins_x=256, bins_y=256, target_density=0.9, iterations=3)
    estimate = mp.estimate_bytes(design, options)
    with mp.PlacementServer(device=0, workers=1, memory_budget=estimate + room, batched=False) as server:
        job = server.submit(design, options)
        assert server.wait(job, 120.0)
        placed, stats = server.take(job)
        peak = server.stats()["peak_reserved"]
    assert stats["estimated_bytes"] == estimate and peak <= estimate + room
    assert (peak > estimate) == (room == 1 << 30)  # 32 MB of slack alone is more than 8 MB
    alone = mp.GlobalPlacer().run(design, options)
    assert np.array_equal(placed.module_x, alone.module_x) and np.array_equal(placed.module_y, alone.module_y)


def test_more_sessions_at_once_than_device_set_ups(gpu):
    """Sessions beyond the set-ups that run on the device at once are set up on the host: each
    placement is the one it is alone."""
    options = mp.default_options(bins_x=64, bins_y=64, target_density=0.9, iterations=3)
    designs = [_with_blocks(50, 0.1, seed=20 + k % 3) for k in range(14)]
    alone = [mp.GlobalPlacer().run(design, options) for design in designs[:3]]
    placed = [None] * len(designs)

    def work(k: int) -> None:
        for _ in range(3):
            placed[k] = mp.GlobalPlacer().run(designs[k], options)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(designs))]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    for k, run in enumerate(placed):
        assert np.array_equal(run.module_x, alone[k % 3].module_x)
        assert np.array_equal(run.module_y, alone[k % 3].module_y)
        assert run.history == alone[k % 3].history
