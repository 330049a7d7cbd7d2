"""Particles with long pin lists side by side, as macros are (needs a GPU).

Lists around the lengths a thread and a warp rank (32) and the sort takes over (256), on
neighbouring particles, in few particles and in many.  Gradients against the float64
restatement, with the tolerance of test_net_layout.
"""
from __future__ import annotations

import numpy as np
import pytest

import myplacement_b200 as mp
from test_noalloc_classes import _reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("particles", [7, 300, 9000])
@pytest.mark.parametrize("lists", [(31, 32, 33), (255, 256), (255, 256, 257), (40,) * 70, (200,) * 33])
def test_neighbouring_lists(gpu, particles, lists):
    rng = np.random.default_rng(particles + sum(lists))
    crowded = np.repeat(np.arange(len(lists)) % particles, lists)
    others = rng.integers(-1, particles, len(crowded))
    particle = np.stack([crowded, others], 1)[rng.permutation(len(crowded))].ravel().astype(np.int32)
    pins = len(particle)
    start = np.arange(0, pins + 1, 2).astype(np.int64)
    xy = rng.normal(0.0, 2.0, (pins, 2))
    xy[particle < 0] = rng.uniform(0.0, 30.0, (int((particle < 0).sum()), 2))
    positions = rng.uniform(1.0, 29.0, (particles, 2))
    weight = rng.uniform(0.5, 2.0, len(start) - 1)
    layout = mp.BackendLayout(
        np.ones(particles), np.ones(particles), np.zeros(particles, np.uint8), np.zeros(particles, np.int32), particles,
        weight, start, particle, np.ascontiguousarray(xy[:, 0]), np.ascontiguousarray(xy[:, 1]), 16, 16,
        (0.0, 0.0, 30.0, 30.0), 0.9, np.zeros(256), np.zeros(256))
    backend, reason = mp.try_create_backend(layout, 0)
    assert backend is not None, reason
    result = backend.evaluate(positions, 1.5, True)
    backend.close()
    expected, smooth, hpwl = _reference(positions, start, particle, xy, weight, 1.5, particles)
    count = np.bincount(particle[particle >= 0], minlength=particles)
    assert (np.abs(result["wire_gradient"] - expected).max(axis=1) <= 2e-5 * np.maximum(count, 0.0)).all()
    assert abs(result["smooth_wirelength"] - smooth) <= 1e-5 * smooth
    assert abs(result["hpwl"] - hpwl) <= 1e-5 * hpwl
