"""Allocation-free wirelength of netlists with large nets side by side (needs a GPU).

Large nets behind many small ones, as in a netlist sorted by degree, nets of more than 32 pins on
average (a warp per net) and just below that, and malformed ranges between them.  Checked
against the float64 restatement with the tolerances of test_noalloc_classes.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import myplacement_b200 as mp
from myplacement_b200 import _abi
from test_noalloc_classes import _reference

pytestmark = pytest.mark.gpu


def _call(positions, start, particle, xy, weight, gamma, particles):
    torch = pytest.importorskip("torch")
    movable = np.nonzero(particle >= 0)[0]
    order = movable[np.argsort(particle[movable], kind="stable")].astype(np.int32)
    pin_start = np.concatenate([[0], np.cumsum(np.bincount(particle[movable], minlength=particles))]).astype(np.int32)
    held = [torch.tensor(a, device="cuda") for a in (positions, start, particle, xy, weight, pin_start, order)]
    wire = torch.full((particles, 2), np.nan, dtype=torch.float64, device="cuda")
    totals = torch.full((2,), np.nan, dtype=torch.float64, device="cuda")
    lib = mp.load_library()
    out = []
    for _ in range(2):
        status = lib.mpgp_wirelength_noalloc(
            held[0].data_ptr(), held[1].data_ptr(), held[2].data_ptr(), held[3].data_ptr(), held[4].data_ptr(),
            len(weight), len(particle), held[5].data_ptr(), held[6].data_ptr(), particles, gamma, wire.data_ptr(),
            totals.data_ptr(), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert status == _abi.MPGP_OK, lib.mpgp_last_error()
        out.append((wire.cpu().numpy(), totals.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    return *out[0], np.diff(pin_start).max()


@pytest.mark.parametrize("degrees", [
    [2] * 6000 + [300] * 40, [40] * 70 + [2] * 9000, [33] * 8, [33] * 9, [33] * 300, [32] * 300, [5000], [2, 500, 2, 2],
    [2] * 1300 + [33] * 1300, [1] * 50 + [64] * 3000,
])
def test_large_nets(gpu, degrees):
    rng = np.random.default_rng(len(degrees) + degrees[-1])
    start = np.concatenate([[0], np.cumsum(degrees)]).astype(np.int32)
    pins, particles = int(start[-1]), max(8, int(start[-1]) // 3)
    particle = rng.integers(-1, particles, pins).astype(np.int32)
    xy = rng.normal(0.0, 2.0, (pins, 2))
    positions = rng.uniform(0.0, 30.0, (particles, 2))
    weight = rng.uniform(0.5, 2.0, len(degrees))
    wire, totals, most = _call(positions, start, particle, xy, weight, 1.5, particles)
    gradient, smooth, hpwl = _reference(positions, start, particle, xy, weight, 1.5, particles)
    assert np.abs(wire - gradient).max() <= 1e-5 * most * weight.max()
    assert totals[0] == pytest.approx(smooth, rel=1e-5) and totals[1] == pytest.approx(hpwl, rel=1e-5)


@pytest.mark.parametrize("degree", [3, 40])
def test_malformed_ranges_add_nothing(gpu, degree):
    """A range that ends before it begins, begins below zero or ends past the pins is left out."""
    rng = np.random.default_rng(degree)
    nets = 60
    start = np.arange(0, degree * (nets + 1), degree).astype(np.int32)
    pins, particles = int(start[-1]), 50
    particle = rng.integers(0, particles, pins).astype(np.int32)
    xy = rng.normal(0.0, 2.0, (pins, 2))
    positions = rng.uniform(0.0, 30.0, (particles, 2))
    weight = rng.uniform(0.5, 2.0, nets)
    broken = start.copy()
    broken[10], broken[30] = -5, pins + 7  # nets 9, 10, 29 and 30 lose their range
    wire, totals, most = _call(positions, broken, particle, xy, weight, 1.5, particles)
    weight[[9, 10, 29, 30]] = 0.0
    gradient, smooth, hpwl = _reference(positions, start, particle, xy, weight, 1.5, particles)
    assert np.abs(wire - gradient).max() <= 1e-5 * most * weight.max()
    assert totals[0] == pytest.approx(smooth, rel=1e-5) and totals[1] == pytest.approx(hpwl, rel=1e-5)
