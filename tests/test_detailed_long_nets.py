"""Detailed placement with nets on many cells (needs a GPU): a block walks what eight lanes do.

Nets at and beyond the length from which a block walks them (512 pins), with the degree limit
below them (their windows are not evaluated, as with a clock net) and above (their extremes
are asked for).  The host's lists, which a tight memory budget chooses, give the same bits.
"""
from __future__ import annotations

import numpy as np
import pytest

import myplacement_b200 as mp
from myplacement_b200.design import packed_placement

pytestmark = pytest.mark.gpu


def _design(cells: int, degrees: list[int], seed: int) -> mp.Design:
    rng = np.random.default_rng(seed)
    base = packed_placement(mp.synthetic_design(cells=cells, nets=cells, terminals=16, macros=1, seed=seed), seed)
    movable = np.nonzero(base.movable_mask)[0]
    pins = sum(degrees)
    fields = {k: getattr(base, k) for k in base.__dataclass_fields__ if not k.startswith("_")}
    order = rng.permutation(base.net_count + len(degrees))  # long nets between the others
    lengths = np.concatenate([np.diff(base.net_pin_start), degrees])[order]
    starts = np.concatenate([base.net_pin_start[:-1], base.net_pin_start[-1] + np.cumsum([0] + degrees[:-1])])[order]
    take = np.concatenate([np.arange(s, s + n) for s, n in zip(starts, lengths)])
    fields["pin_module"] = np.concatenate([base.pin_module, rng.choice(movable, pins)])[take]
    fields["pin_offset_x"] = np.concatenate([base.pin_offset_x, rng.uniform(-2, 2, pins)])[take]
    fields["pin_offset_y"] = np.concatenate([base.pin_offset_y, rng.uniform(-4, 4, pins)])[take]
    fields["net_pin_start"] = np.concatenate([[0], np.cumsum(lengths)])
    fields["net_weight"] = rng.choice([1.0, 0.5, 2.0, 0.0], len(lengths))
    return mp.Design(**fields)


def _host_bytes(d: mp.Design) -> int:
    m, p, n = d.module_count, d.pin_count, d.net_count
    w, t = m // 4 + 1, m // 2 + 1
    return 54 * m + 40 * p + 4 * (n + 1) + 8 * n + w * 62 + 4 * (w + 1) + t * 46 + 4 * (t + 1)


@pytest.mark.parametrize("cells,degrees", [(900, [511, 512, 513]), (2500, [513, 1024, 1025, 5000]), (4000, [40_000, 600])])
@pytest.mark.parametrize("limit", [64, 512, 1_000_000])
def test_device_equals_host(gpu, cells, degrees, limit):
    design = _design(cells, degrees, cells + len(degrees))
    results = []
    for budget in ({}, {"maximum_cuda_memory_bytes": _host_bytes(design)}):
        options = mp.default_detailed_options(passes=2, maximum_net_degree=limit, **budget)
        results.append(mp.DetailedPlacer().run(design, options))
    (placed, result), (expected, theirs) = results
    assert result["cuda_reserved_memory_bytes"] > theirs["cuda_reserved_memory_bytes"]  # two paths
    for key in ("hpwl_before", "hpwl_after", "evaluated_windows", "evaluated_permutations", "accepted_operations"):
        assert result[key] == theirs[key], key
    assert np.array_equal(placed.module_x, expected.module_x) and np.array_equal(placed.module_y, expected.module_y)
    assert np.array_equal(placed.module_orientation, expected.module_orientation)
