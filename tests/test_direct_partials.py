"""Scalars reduced from few blocks' partials directly and from folded ones (needs a GPU).

Particle and row counts on both sides of the 128 blocks up to which the reduction reads every
block's partials.  The metrics are recomputed from the fixed-point layers in float64; sums of at
most 20,000 positive terms in another order differ by 20,000 * 2^-53 = 2.3e-12 of their value, the
tolerance is 1e-11.  Maxima are equal.
"""
from __future__ import annotations

import numpy as np
import pytest

import myplacement_b200 as mp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("particles,bins_x,bins_y", [(200, 8, 8), (32_768, 60, 127), (32_769, 60, 128),
                                                     (33_500, 150, 129), (70_000, 128, 130)])
def test_metrics(gpu, particles, bins_x, bins_y):
    rng = np.random.default_rng(particles)
    side = 1000.0
    movable = particles * 3 // 4
    target = 0.8
    width = rng.uniform(1.0, 6.0, particles)
    height = rng.uniform(1.0, 6.0, particles)
    layer = np.where(np.arange(particles) < movable, rng.integers(0, 2, particles), 2).astype(np.uint8)
    fixed = rng.uniform(0.0, 1.0, bins_x * bins_y)
    start = np.arange(0, 2 * movable + 1, 2, dtype=np.int64)
    pin_particle = rng.integers(0, movable, 2 * movable).astype(np.int32)
    layout = mp.BackendLayout(width, height, layer, np.bincount(pin_particle, minlength=particles).astype(np.int32),
                              movable, np.ones(movable), start, pin_particle, np.zeros(2 * movable),
                              np.zeros(2 * movable), bins_x, bins_y, (0.0, 0.0, side, side), target, fixed,
                              np.zeros(bins_x * bins_y))
    backend, reason = mp.try_create_backend(layout, 0)
    assert backend is not None, reason
    positions = rng.uniform(10.0, side - 10.0, (particles, 2))
    result = backend.evaluate(positions, 5.0, True)
    standard, macro, filler = (np.asarray(q, float) for q in backend.density_layers(bins_x, bins_y))
    area = (side / bins_x) * (side / bins_y)
    unit = result["design_density"]["normalization_area"] / (standard.sum() + target * macro.sum())
    placed = (standard + target * macro) * unit
    for name, charge in (("design_density", placed + target * fixed.reshape(bins_y, bins_x)),
                         ("optimizer_density", placed + target * fixed.reshape(bins_y, bins_x) + target * filler * unit)):
        m = result[name]
        assert abs(m["total_overflow_area"] - np.maximum(0.0, charge - target * area).sum()) <= 1e-11 * charge.sum()
        assert abs(m["total_charge_area"] - charge.sum()) <= 1e-11 * charge.sum()
        assert abs(m["maximum_density"] - charge.max() / area) <= 1e-11 * charge.max() / area
    again = backend.evaluate(positions, 5.0, False)
    assert again["design_density"] == result["design_density"]
    backend.close()
