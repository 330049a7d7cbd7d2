"""The allocation-free net pass at the edges of its degree classes and block chunks (needs a GPU).

Every case is checked against a float64 restatement of the log-sum-exp wirelength
(AdaptiveGlobalPlacer.cpp:29-82).  The engine forms exponents of FP32 coordinate differences d:
each is off by at most 2^-24 |d| / gamma, which is at most 40 * 2^-24 = 2.4e-6 where an exponential
is not negligible (|d| / gamma < 40), and a few FP32 roundings of 6e-8 follow; so gradients agree
within 1e-5 of the largest component times the pins of a particle, and the totals within 1e-5.
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

import myplacement_b200 as mp
from myplacement_b200 import _abi

pytestmark = pytest.mark.gpu


def _reference(positions, start, particle, xy, weight, gamma, particles):
    gradient = np.zeros((particles, 2))
    smooth = hpwl = 0.0
    for n in range(len(start) - 1):
        b, e = int(start[n]), int(start[n + 1])
        if e - b < 2:
            continue
        p = particle[b:e]
        points = xy[b:e] + np.where(p[:, None] >= 0, positions[np.maximum(p, 0)], 0.0)
        for axis in range(2):
            v = points[:, axis]
            up, down = np.exp((v - v.max()) / gamma), np.exp((v.min() - v) / gamma)
            smooth += weight[n] * (np.ptp(v) + gamma * (np.log(up.sum()) + np.log(down.sum())))
            hpwl += weight[n] * np.ptp(v)
            np.add.at(gradient[:, axis], p[p >= 0], (weight[n] * (up / up.sum() - down / down.sum()))[p >= 0])
    return gradient, smooth, hpwl


@pytest.mark.parametrize("nets,degrees", [
    (1, (2,)), (31, (2,)), (33, (1, 2)), (70, (2, 3, 4, 5)), (257, (1, 2, 4, 5, 8, 9, 16, 17, 32, 33)),
    (300, (32, 33, 64, 100)), (9_000, (2, 2, 2, 3, 8, 17)), (80_000, (1, 2, 2, 3, 4)),
])
@pytest.mark.parametrize("captured", [False, True])
def test_classes_and_chunks(gpu, nets, degrees, captured):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(nets)
    degree = rng.choice(degrees, nets)
    start = np.concatenate([[0], np.cumsum(degree)]).astype(np.int32)
    pins, particles = int(start[-1]), max(8, nets // 2)
    particle = rng.integers(-1, particles, pins).astype(np.int32)
    xy = rng.normal(0.0, 2.0, (pins, 2))
    positions = rng.uniform(0.0, 30.0, (particles, 2))
    positions[::7] = positions[0]  # coincident pins
    weight = rng.uniform(0.5, 2.0, nets)
    gamma = 1.5
    movable = np.nonzero(particle >= 0)[0]
    order = movable[np.argsort(particle[movable], kind="stable")].astype(np.int32)
    pin_start = np.concatenate([[0], np.cumsum(np.bincount(particle[movable], minlength=particles))]).astype(np.int32)
    t = lambda a: torch.tensor(a, device="cuda")
    held = [t(positions), t(start), t(particle), t(xy), t(weight), t(pin_start), t(order)]
    wire = torch.empty((particles, 2), dtype=torch.float64, device="cuda")
    totals = torch.empty(2, dtype=torch.float64, device="cuda")
    lib = mp.load_library()

    def call():
        stream = torch.cuda.current_stream().cuda_stream
        status = lib.mpgp_wirelength_noalloc(
            held[0].data_ptr(), held[1].data_ptr(), held[2].data_ptr(), held[3].data_ptr(), held[4].data_ptr(), nets,
            pins, held[5].data_ptr(), held[6].data_ptr(), particles, gamma, wire.data_ptr(), totals.data_ptr(),
            ctypes.c_void_p(stream))
        assert status == _abi.MPGP_OK, lib.mpgp_last_error()

    call()
    torch.cuda.synchronize()
    if captured:
        first = (wire.clone(), totals.clone())
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            call()
        wire.zero_()
        totals.zero_()
        graph.replay()
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(wire, first[0]) and torch.equal(totals, first[1])
    gradient, smooth, hpwl = _reference(positions, start, particle, xy, weight, gamma, particles)
    most = np.diff(pin_start).max()
    assert np.abs(wire.cpu().numpy() - gradient).max() <= 1e-5 * most * np.abs(weight).max()
    got = totals.cpu().numpy()
    assert got[0] == pytest.approx(smooth, rel=1e-5, abs=1e-12) and got[1] == pytest.approx(hpwl, rel=1e-5, abs=1e-12)
