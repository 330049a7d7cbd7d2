"""The one-launch field solve of small grids against the staged contractions (needs a GPU).

Grids of at most 128 x 128 run the whole field solve in one cluster: a single CTA up to
64 x 64, two or four CTAs of 32 columns beyond.  MPGP_FIELD_SOLVE=staged runs the same
contractions as four launches, with the same exponents and the same FP64 sums, so the two
agree to the rounding of single values: an FP32 intermediate may differ by one unit in the
last place where the one-launch solve rounds once instead of twice.  Three intermediates
and the result give at most 4 * 2^-23 = 4.8e-7 of the largest value; the tolerance is 1e-6
of it.
"""
from __future__ import annotations

import numpy as np
import pytest

import myplacement_b200 as mp

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _near(a, b):
    a, b = np.asarray(a, float), np.asarray(b, float)
    assert np.isfinite(a).all() and np.abs(a - b).max() <= TOL * max(np.abs(b).max(), 1e-300)


def _design():
    return mp.synthetic_design(cells=900, nets=1000, terminals=32, utilization=0.7, seed=9)


def _backend(design, bins_x: int, bins_y: int):
    options = mp.default_options(bins_x=bins_x, bins_y=bins_y, target_density=0.9)
    setup = mp.host_setup(design, options)
    count = int(setup["particle_count"])
    layout = mp.build_layout(design, setup["width"], setup["height"], setup["layer"], np.zeros(count, np.int32),
                             int(setup["movable_count"]), bins_x, bins_y, 0.9, setup["static_fixed"],
                             setup["static_dark"])
    backend, reason = mp.try_create_backend(layout, 0)
    assert backend is not None, reason
    return backend, count


# One K-block exactly, one past it, ragged and odd widths, each combination of one and two
# K-blocks per axis, the smallest and the largest; then one past it (staged either way).
@pytest.mark.parametrize("bins_x,bins_y", [(8, 8), (24, 24), (33, 17), (63, 64), (64, 64), (65, 64), (64, 65),
                                           (50, 128), (128, 50), (97, 111), (128, 128), (129, 128)])
def test_one_launch_equals_staged(gpu, monkeypatch, bins_x, bins_y):
    rng = np.random.default_rng(bins_x * 1000 + bins_y)
    design = _design()
    monkeypatch.delenv("MPGP_FIELD_SOLVE", raising=False)
    small, count = _backend(design, bins_x, bins_y)
    monkeypatch.setenv("MPGP_FIELD_SOLVE", "staged")
    staged, _ = _backend(design, bins_x, bins_y)
    monkeypatch.delenv("MPGP_FIELD_SOLVE")
    llx, lly, urx, ury = design.core
    for source in (rng.standard_normal((bins_y, bins_x)) + 3.0, 1e-30 * np.abs(rng.standard_normal((bins_y, bins_x))) ** 3,
                   np.zeros((bins_y, bins_x)), np.full((bins_y, bins_x), 2.5)):
        for a, b in zip(small.field_solve(source), staged.field_solve(source)):
            _near(a, b)
    for seed in range(2):
        positions = np.random.default_rng(seed).uniform((llx, lly), (urx, ury), (count, 2))
        for gradient in (False, True, False):
            a = small.evaluate(positions, 2.0, gradient)
            b = staged.evaluate(positions, 2.0, gradient)
            assert a.keys() == b.keys()
            for key, value in b.items():
                if value is not None and not isinstance(value, (str, dict)):
                    _near(a[key], value)
    small.close()
    staged.close()


@pytest.mark.parametrize("bins", [48, 64, 100, 128])
def test_placements_and_batches(gpu, monkeypatch, bins):
    """Placements reuse the kept coefficients (an evaluation without the forward transform);
    a batch of mixed grids runs its small ones in shared launches, as the plain runs."""
    design = _design()
    x, y = mp.random_placement(design, 5)
    design = design.copy_with_positions(x, y)
    options = [mp.default_options(bins_x=b, bins_y=b, target_density=0.9, iterations=12) for b in (bins, 32, 96, 160, 320)]
    monkeypatch.delenv("MPGP_FIELD_SOLVE", raising=False)
    plain = [mp.GlobalPlacer().run(design, o) for o in options]
    placed, _, _ = mp.batch_place([design] * len(options), options, workers=len(options))
    for a, b in zip(placed, plain):
        np.testing.assert_array_equal(a.module_x, b.module_x)
        np.testing.assert_array_equal(a.module_y, b.module_y)
        assert a.hpwl_after == b.hpwl_after
    monkeypatch.setenv("MPGP_FIELD_SOLVE", "staged")
    staged = mp.GlobalPlacer().run(design, options[0])
    side = max(design.core[2] - design.core[0], design.core[3] - design.core[1])
    # Few iterations, so that a rounding of one value stays below 1e-4 of a bin.
    assert np.abs(staged.module_x - plain[0].module_x).max() <= 1e-4 * side / bins
    assert np.abs(staged.module_y - plain[0].module_y).max() <= 1e-4 * side / bins
