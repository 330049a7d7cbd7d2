"""The net layout built on the device, through the gradients it leads to (needs a GPU).

Nets of every degree class and around its edges, nets of no and one pin, static pins anywhere in
a net, blocks of nets with a remainder, particles with no, few, many and more than a thousand
pins (whose slots take the sorted path), no nets at all.  The wirelength gradient of the layout
is checked against the float64 restatement of test_noalloc_classes, whose tolerance it shares:
FP32 offsets and exponents of coordinate differences, 1e-5 of a pin's largest contribution (the
largest weight) for each pin of the particle.
"""
from __future__ import annotations

import numpy as np
import pytest

import myplacement_b200 as mp
from test_noalloc_classes import _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nets,degrees,crowded", [
    (0, (0,), 0), (1, (1,), 0), (1, (2,), 0), (255, (0, 1, 2, 3), 0), (256, (2,), 40), (257, (2, 4, 5, 8, 9), 33),
    (3000, (1, 2, 3, 16, 17, 32, 33, 70), 200), (3000, (2, 3, 5), 1024), (3000, (2, 3, 5), 1500), (40_000, (2, 2, 3), 50),
])
def test_layout(gpu, nets, degrees, crowded):
    rng = np.random.default_rng(nets + crowded)
    degree = rng.choice(degrees, nets)
    start = np.concatenate([[0], np.cumsum(degree)]).astype(np.int64)
    pins, particles = int(start[-1]), max(8, nets // 2)
    particle = rng.integers(-1, particles - 1, pins).astype(np.int32)  # the last particle has no pin
    particle[rng.permutation(pins)[:crowded]] = particles // 2
    xy = rng.normal(0.0, 2.0, (pins, 2))
    xy[particle < 0] = rng.uniform(0.0, 30.0, (int((particle < 0).sum()), 2))
    positions = rng.uniform(1.0, 29.0, (particles, 2))
    weight = rng.uniform(0.5, 2.0, nets)
    bins = 16
    layout = mp.BackendLayout(
        np.ones(particles), np.ones(particles), np.zeros(particles, np.uint8), np.zeros(particles, np.int32), particles,
        weight, start, particle, np.ascontiguousarray(xy[:, 0]), np.ascontiguousarray(xy[:, 1]), bins, bins,
        (0.0, 0.0, 30.0, 30.0), 0.9, np.zeros(bins * bins), np.zeros(bins * bins))
    backend, reason = mp.try_create_backend(layout, 0)
    assert backend is not None, reason
    result = backend.evaluate(positions, 1.5, True)
    expected, smooth, hpwl = _reference(positions, start, particle, xy, weight, 1.5, particles)
    gradient = np.asarray(result["wire_gradient"]).reshape(-1, 2)
    count = np.bincount(particle[particle >= 0], minlength=particles)
    assert (np.abs(gradient - expected).max(axis=1) <= 2e-5 * np.maximum(count, 0.0)).all()
    assert abs(result["smooth_wirelength"] - smooth) <= 1e-5 * max(smooth, 1.0)
    assert abs(result["hpwl"] - hpwl) <= 1e-5 * max(hpwl, 1.0)
    backend.close()
