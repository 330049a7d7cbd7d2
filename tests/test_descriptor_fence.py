"""Tensor maps in device memory: the thread that issues the loads acquires their bytes.

The batched field kernels read their tensor maps from device memory that an earlier engine's
maps may have used, so they execute a tensor-map acquire fence before the first load through
them.  The fence orders the loads of the thread that executes it: it stands on the issuing
thread.  That is read from the sources; on a GPU, batches of changing grids, whose maps take
turns in the same memory, equal the plain runs.
"""
from __future__ import annotations

import re
from pathlib import Path

import numpy as np
import pytest

import myplacement_b200 as mp

CSRC = Path(mp.__file__).resolve().parent / "csrc"


def _guard_before(source: str, marker: str) -> str:
    """The thread of the innermost guard before the first `marker`."""
    guards = re.findall(r"threadIdx\.x == (\w+)\)|(warp == 0 && lane == 0)\)", source[:source.index(marker)])
    thread, first_lane = guards[-1]
    return "0" if first_lane else thread


@pytest.mark.parametrize("name,first_load", [("dct_tc.cu", "tmaLoad3d(smemAddress(stage), &t.map_a"),
                                             ("field_tc.cu", "tmaLoad3d(stage"),
                                             ("field_small.cu", "fetchA(forward")])
def test_fence_is_on_the_issuing_thread(name, first_load):
    source = (CSRC / name).read_text()
    assert _guard_before(source, "fence.proxy.tensormap") == _guard_before(source, first_load)


@pytest.mark.gpu
def test_batches_of_changing_grids(gpu):
    design = mp.synthetic_design(cells=700, nets=750, terminals=16, utilization=0.7, seed=5)
    design = design.copy_with_positions(*mp.random_placement(design, 5))
    for grids in ((64, 48, 32), (128, 100, 72), (40, 128, 64), (96, 33, 17), (64, 128, 65)):
        options = [mp.default_options(bins_x=b, bins_y=b, target_density=0.9, iterations=6) for b in grids]
        placed, _, _ = mp.batch_place([design] * len(grids), options, workers=len(grids))
        for result, o in zip(placed, options):
            plain = mp.GlobalPlacer().run(design, o)
            assert np.array_equal(result.module_x, plain.module_x)
            assert np.array_equal(result.module_y, plain.module_y)
