"""The RUDY deposit's two paths and the gradient's lane groups against a float64 restatement (needs a GPU).

Designs on both sides of the rule that sends the deposit through shared memory (nets against map
cells), grids at and past the shared memory's size, nets of every degree class.  The restatement is
evaluateRudy (Rudy.cpp:227-456) with the demand maps as matrix products and the derivative of the
hinge penalty by automatic differentiation; at generic positions the subgradient is the gradient.
Pin offsets are FP32 in the engine: a relative 6e-8 of an offset (at most half a cell, under a
tenth of a bin), and the maps are quantized to 2^-32 of a bin's width: 1e-7 of the largest
component bounds both.
"""
from __future__ import annotations

import math

import numpy as np
import pytest

import myplacement_b200 as mp

pytestmark = pytest.mark.gpu


def _reference(torch, layout, positions, columns, rows, span, capacity):
    llx, lly, urx, ury = layout.region
    pos = torch.tensor(positions, dtype=torch.float64, requires_grad=True)
    start = torch.tensor(layout.net_pin_start)
    net = torch.repeat_interleave(torch.arange(len(start) - 1), start[1:] - start[:-1])
    particle = torch.tensor(layout.pin_particle).long()
    points = torch.tensor(np.stack([layout.pin_x, layout.pin_y], 1)) + torch.where(
        (particle >= 0)[:, None], pos[particle.clamp(min=0)], 0.0)
    weight = torch.tensor(layout.net_weight)
    counted = (torch.bincount(net, minlength=weight.numel()) >= 2) & (weight > 0)

    def axis(v, minimum, origin, length, count):
        low = torch.full_like(weight, math.inf).scatter_reduce(0, net, v, "amin")[counted]
        high = torch.full_like(weight, -math.inf).scatter_reduce(0, net, v, "amax")[counted]
        center, thin = 0.5 * (low + high), high - low < minimum
        low = torch.where(thin, center - 0.5 * minimum, low)
        high = torch.where(thin, center + 0.5 * minimum, high)
        edge = origin + length * torch.arange(count, dtype=torch.float64)
        over = (torch.minimum(high[:, None], edge + length) - torch.maximum(low[:, None], edge)).clamp(min=0.0)
        return over, high - low

    bin_w, bin_h = (urx - llx) / columns, (ury - lly) / rows
    ox, wide = axis(points[:, 0], span * bin_w, llx, bin_w, columns)
    oy, high = axis(points[:, 1], span * bin_h, lly, bin_h, rows)
    w = weight[counted]
    horizontal, vertical = (oy * (w / high)[:, None]).T @ ox, (oy * (w / wide)[:, None]).T @ ox
    over = [(m / c - 1.0).clamp(min=0.0) for m, c in zip((horizontal, vertical), capacity(horizontal, vertical))]
    energy = sum(0.5 * (o ** 2).sum() for o in over) / (columns * rows)
    energy.backward()
    return (float(horizontal.detach().sum()), float(vertical.detach().sum()), float(energy.detach()),
            pos.grad.numpy())


@pytest.mark.parametrize("cells,columns,rows,pins_per_net", [
    (300, 5, 3, 4.6),          # a few nets of every lane group, wider than the grid's cells
    (14_500, 24, 31, 4.6),     # either side of the rule on a small grid
    (16_000, 24, 31, 4.6),
    (24_000, 64, 64, 3.85),    # the default grid through shared memory
    (40_000, 111, 111, 3.0),   # the largest square grid of the shared copy, and past it
    (40_000, 160, 80, 3.0),
])
def test_deposit_and_gradient(gpu, cells, columns, rows, pins_per_net):
    torch = pytest.importorskip("torch")
    design = mp.synthetic_design(cells=cells, nets=int(cells * 1.05), terminals=40, utilization=0.6,
                                 pins_per_net=pins_per_net, locality_window=200, seed=cells)
    x, y = mp.random_placement(design, 3)
    design = design.copy_with_positions(x, y)
    options = mp.default_options(bins_x=32, bins_y=32, target_density=0.9, rudy_columns=columns, rudy_rows=rows,
                                 rudy_penalty_model=1)
    setup = mp.host_setup(design, options)
    count, movable = int(setup["particle_count"]), int(setup["movable_count"])
    layout = mp.build_layout(design, setup["width"], setup["height"], setup["layer"], np.zeros(count, np.int32),
                             movable, 32, 32, 0.9, setup["static_fixed"], setup["static_dark"])
    positions = np.stack([setup["x"], setup["y"]], 1)
    positions[:movable, 0], positions[:movable, 1] = x[design.movable_mask], y[design.movable_mask]
    backend, reason = mp.try_create_backend(layout, 0)
    assert backend is not None, reason
    raw = backend.rudy(positions, options)
    capacity = (0.9 * raw["horizontal_mean"], 0.9 * raw["vertical_mean"])
    results = [backend.rudy(positions, options, capacity, gradient=True) for _ in range(2)]
    backend.close()
    horizontal, vertical, energy, gradient = _reference(torch, layout, positions, columns, rows, 0.25,
                                                        lambda h, v: capacity)
    for mine in results:
        assert mine["horizontal_total"] == pytest.approx(horizontal, rel=1e-7)
        assert mine["vertical_total"] == pytest.approx(vertical, rel=1e-7)
        assert mine["energy"] == pytest.approx(energy, rel=1e-6)
        assert mine["evaluation_energy"] == mine["energy"]
        assert np.abs(mine["gradient"] - gradient).max() <= 1e-7 * np.abs(gradient).max()
    assert np.array_equal(results[0]["gradient"], results[1]["gradient"])
