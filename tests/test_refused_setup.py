"""A session that is refused in the middle of its set-up on the device (needs a GPU).

A design without rows has no core, which the static layers refuse after the area sort has been
launched on the set-up's second stream.  The set-up's memory goes back to a pool that the other
sessions of the process allocate from, so it may only be given back once that sort is done: a
neighbour that sets up and runs at the same time gets the placement it gets alone.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

import myplacement_b200 as mp

pytestmark = pytest.mark.gpu


def _placed(cells: int, seed: int) -> mp.Design:
    design = mp.synthetic_design(cells=cells, nets=int(cells * 1.05), terminals=64, macros=8, seed=seed)
    return design.copy_with_positions(*mp.random_placement(design, seed))


def _without_rows(design: mp.Design) -> mp.Design:
    fields = {k: getattr(design, k) for k in design.__dataclass_fields__ if not k.startswith("_")}
    for name in fields:
        if name.startswith("row_"):
            fields[name] = fields[name][:0]
    return mp.Design(**fields)


def test_neighbour_of_refused_set_ups(gpu):
    options = mp.default_options(bins_x=64, bins_y=64, target_density=0.9, iterations=4)
    neighbour = _placed(20_000, 3)
    refused = _without_rows(_placed(60_000, 4))
    alone = mp.GlobalPlacer().run(neighbour, options)
    results, stop = [], threading.Event()

    def place():
        while not stop.is_set() or not results:
            results.append(mp.GlobalPlacer().run(neighbour, options))

    thread = threading.Thread(target=place)
    thread.start()
    try:
        for _ in range(12):
            with pytest.raises(mp.EngineError, match="valid region"):
                mp.Session(refused, options)
    finally:
        stop.set()
        thread.join()
    for placed in results:
        assert np.array_equal(placed.module_x, alone.module_x)
        assert np.array_equal(placed.module_y, alone.module_y)
        assert placed.history == alone.history
