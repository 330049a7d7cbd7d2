"""Performance cases: the calls that programs built on this package make.

Six kinds of call, each through the public entry point that a program uses:

  evaluate    CudaPlacementBackend.evaluate: one evaluation of the placement objective at host
              positions, with the wire and density gradients or without (a controller of the
              caller's own; a candidate needs no gradient)
  rudy        CudaPlacementBackend.rudy: the routing-demand proxy with its subgradient
  wirelength  mpgp_wirelength_noalloc: wirelength and wire gradient of device arrays, for callers
              that own all device memory
  place       GlobalPlacer.run: a whole call with a small iteration budget (a warm start or an
              incremental placement): set-up, controller iterations, final metrics
  batch       batch_place: many small designs at once
  detail      DetailedPlacer.run: window reordering of a legal placement

Designs follow the law of the named workloads (design.py): 5k cells on 64 x 64 bins, 210k cells on
512 x 512, 1.3M cells on 1024 x 1024.  Positions are of a placement's two ends: "random" (the
initial placement, cells uniform in the core, so nets span it) or "spread" (late in a run: the
cells of a net lie near each other and cover the core evenly).
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import myplacement_b200 as mp
from myplacement_b200.design import packed_placement

TARGET_DENSITY = 0.9


def listed() -> list[dict]:
    return [
        # The smallest evaluation: launches, latency and host work are all of it.
        {"name": "evaluate_5k", "kind": "evaluate", "cells": 5_000, "macros": 0, "bins_x": 64, "bins_y": 64,
         "positions": "spread", "gradient": True},
        # A grid and counts that are no powers of two, with macros.
        {"name": "evaluate_odd_37k", "kind": "evaluate", "cells": 37_411, "macros": 61, "bins_x": 250, "bins_y": 187,
         "positions": "random", "gradient": True},
        # The mid design late in a run, as a controller evaluates its current point ...
        {"name": "evaluate_210k", "kind": "evaluate", "cells": 210_000, "macros": 400, "bins_x": 512, "bins_y": 512,
         "positions": "spread", "gradient": True},
        # ... and a candidate step from the random start, which needs no gradient.
        {"name": "candidate_210k", "kind": "evaluate", "cells": 210_000, "macros": 400, "bins_x": 512, "bins_y": 512,
         "positions": "random", "gradient": False},
        # The largest design of the workloads.
        {"name": "evaluate_1m3", "kind": "evaluate", "cells": 1_300_000, "macros": 2_000, "bins_x": 1024,
         "bins_y": 1024, "positions": "spread", "gradient": True},
        # The routability term of the mid design on the default 64 x 64 map.
        {"name": "rudy_210k", "kind": "rudy", "cells": 210_000, "macros": 400, "grid": 64, "positions": "spread"},
        # Allocation-free wirelength: a small netlist in a latency-critical loop, and one near the
        # entry point's limit of 2^20 pins.
        {"name": "wirelength_5k", "kind": "wirelength", "cells": 5_000, "positions": "spread"},
        {"name": "wirelength_210k", "kind": "wirelength", "cells": 210_000, "positions": "random"},
        # Whole calls with a small budget, the second one the headline design.  (A longer run is
        # chaotic: a last-bit difference of one sum grows past the results' own precision.)
        {"name": "place_5k", "kind": "place", "cells": 5_000, "macros": 0, "bins_x": 64, "bins_y": 64,
         "iterations": 16, "rudy": False},
        {"name": "place_210k", "kind": "place", "cells": 210_000, "macros": 400, "bins_x": 512, "bins_y": 512,
         "iterations": 16, "rudy": False},
        # Many small designs of mixed sizes at once.
        {"name": "batch_24", "kind": "batch", "count": 24, "cells": 3_000, "iterations": 16},
        # Window reordering of the mid design, packed legally.
        {"name": "detail_210k", "kind": "detail", "cells": 210_000, "passes": 2},
    ]


def draw(rng) -> dict:
    def log_uniform(low, high):
        return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))

    kind = rng.choice(["evaluate", "evaluate", "rudy", "wirelength", "place", "batch", "detail"])
    positions = rng.choice(["random", "spread"])
    if kind == "evaluate":
        cells = log_uniform(3_000, 700_000)
        side = math.sqrt(cells) * rng.uniform(0.8, 1.25)
        return {"kind": kind, "cells": cells, "macros": rng.choice([0, cells // 600]),
                "bins_x": min(1024, max(24, int(side * rng.uniform(0.7, 1.4)))), "bins_y": min(1024, max(24, int(side))),
                "positions": positions, "gradient": rng.random() < 0.7}
    if kind == "rudy":
        return {"kind": kind, "cells": log_uniform(5_000, 300_000), "macros": rng.choice([0, 50]),
                "grid": rng.randint(32, 128), "positions": positions}
    if kind == "wirelength":
        return {"kind": kind, "cells": log_uniform(2_000, 220_000), "positions": positions}
    if kind == "place":
        cells = log_uniform(3_000, 300_000)
        bins = int(min(512, max(32, 2 ** round(math.log2(math.sqrt(cells))))))
        return {"kind": kind, "cells": cells, "macros": rng.choice([0, cells // 600]), "bins_x": bins, "bins_y": bins,
                "iterations": rng.randint(8, 16), "rudy": rng.random() < 0.25}
    if kind == "batch":
        return {"kind": kind, "count": rng.randint(8, 24), "cells": log_uniform(1_000, 3_000),
                "iterations": rng.randint(8, 16)}
    return {"kind": kind, "cells": log_uniform(5_000, 210_000), "passes": rng.randint(1, 2)}


# ---- inputs ----------------------------------------------------------------------------


def _design(cells: int, macros: int, seed: int):
    """A design of the named workloads' law (3.85 pins a net with macros, 70 % utilisation)."""
    return mp.synthetic_design(cells=cells, nets=int(cells * 1.0476), terminals=max(16, min(1_200, cells // 40)),
                               macros=macros, utilization=0.70, pins_per_net=3.85, seed=seed)


def _fillers(cells: int) -> int:
    """Filler limit: the default 50,000, and fewer for a small design (so that their number is given)."""
    return min(50_000, cells // 4)


def _spread(design, seed: int):
    """Module centres late in a run: blocks of 256 consecutive cells (a net's cells are within 1,024
    consecutive ones) each over a tile of the core, tiles in boustrophedon order."""
    rng = np.random.Generator(np.random.PCG64([seed, 1]))
    llx, lly, urx, ury = design.core
    x, y = design.module_x.copy(), design.module_y.copy()
    movable = np.nonzero(design.movable_mask)[0]
    block = np.arange(movable.shape[0]) // 256
    side = int(math.ceil(math.sqrt(block[-1] + 1)))
    row = block // side
    column = np.where(row % 2 == 0, block % side, side - 1 - block % side)
    rows = row[-1] + 1
    jitter = rng.normal(0.5, 0.5, size=(2, movable.shape[0]))
    half_w, half_h = 0.5 * design.module_width[movable], 0.5 * design.module_height[movable]
    x[movable] = np.clip(llx + (column + jitter[0]) * (urx - llx) / side, llx + half_w, urx - half_w)
    y[movable] = np.clip(lly + (row + jitter[1]) * (ury - lly) / rows, lly + half_h, ury - half_h)
    return x, y


def _placed(case: dict, seed: int):
    design = _design(case["cells"], case.get("macros", 0), seed)
    if case.get("positions", "random") == "random":
        x, y = mp.random_placement(design, seed)
    else:
        x, y = _spread(design, seed)
    return design.copy_with_positions(x, y)


def _layout(design, bins_x: int, bins_y: int):
    """The backend's flattened layout and the particle positions (movable modules, then fillers)."""
    options = mp.default_options(bins_x=bins_x, bins_y=bins_y, target_density=TARGET_DENSITY,
                                 maximum_fillers=_fillers(int(design.movable_mask.sum())))
    setup = mp.host_setup(design, options)
    count, movable = int(setup["particle_count"]), int(setup["movable_count"])
    pin_count = np.zeros(count, np.int32)
    pin_count[:movable] = np.bincount(design.pin_module, minlength=design.module_count)[design.movable_mask]
    layout = mp.build_layout(design, setup["width"], setup["height"], setup["layer"], pin_count, movable, bins_x,
                             bins_y, TARGET_DENSITY, setup["static_fixed"], setup["static_dark"])
    positions = np.stack([setup["x"], setup["y"]], 1)
    positions[:movable, 0] = design.module_x[design.movable_mask]
    positions[:movable, 1] = design.module_y[design.movable_mask]
    return layout, positions


def _smoothing(case: dict, layout) -> float:
    """The LSE smoothing a run has at this stage (0.75 bins at its start, about 0.3 late)."""
    llx, lly, urx, ury = layout.region
    bin_size = max((urx - llx) / layout.bins_x, (ury - lly) / layout.bins_y)
    return (0.75 if case["positions"] == "random" else 0.3) * bin_size


def _backend(layout):
    backend, reason = mp.try_create_backend(layout, 0)
    if backend is None:
        raise RuntimeError(reason)
    return backend


def _rudy_options(case: dict):
    return mp.default_options(rudy_columns=case["grid"], rudy_rows=case["grid"], rudy_penalty_model=1)


def _rudy_capacity(design) -> tuple[float, float]:
    """Capacities a program has from an earlier placement: here from the netlist and the core alone,
    near the mean demand of a spread placement, so that part of the map overflows."""
    llx, lly, urx, ury = design.core
    demand = design.net_count * 0.02 * (urx - llx)
    return demand / (ury - lly), demand / (urx - llx)


def _small_designs(case: dict, seed: int):
    designs, options = [], []
    for k in range(case["count"]):
        cells = int(case["cells"] * 4.0 ** ((k + 0.5) / case["count"] - 0.5))  # half to twice the median
        design = _design(cells, 0, seed + 1 + k)
        x, y = mp.random_placement(design, seed + k)
        designs.append(design.copy_with_positions(x, y))
        bins = int(2 ** round(math.log2(math.sqrt(cells))))
        options.append(mp.default_options(bins_x=bins, bins_y=bins, target_density=TARGET_DENSITY,
                                          iterations=case["iterations"]))
    return designs, options


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    state = {"kind": kind}
    if kind == "evaluate":
        layout, positions = _layout(_placed(case, seed), case["bins_x"], case["bins_y"])
        state |= {"backend": _backend(layout), "positions": positions, "smoothing": _smoothing(case, layout),
                  "gradient": case["gradient"]}
    elif kind == "rudy":
        design = _placed(case, seed)
        layout, positions = _layout(design, 128, 128)
        state |= {"backend": _backend(layout), "positions": positions, "options": _rudy_options(case),
                  "capacity": _rudy_capacity(design)}
    elif kind == "wirelength":
        design = _placed(case, seed)
        state |= _device_netlist(case, design)
    elif kind == "place":
        design = _placed(case, seed)
        rudy = {"rudy_penalty_model": 1, "rudy_capacity_factor": 1.2, "routability_start_overflow": 2.0}
        options = mp.default_options(bins_x=case["bins_x"], bins_y=case["bins_y"], target_density=TARGET_DENSITY,
                                     iterations=case["iterations"], **(rudy if case["rudy"] else {}))
        state |= {"design": design, "options": options}
    elif kind == "batch":
        state["designs"], state["options"] = _small_designs(case, seed)
    else:
        design = _design(case["cells"], case["cells"] // 600, seed)
        state |= {"design": packed_placement(design, seed),
                  "options": mp.default_detailed_options(passes=case["passes"])}
    return state


def _device_netlist(case: dict, design) -> dict:
    device = torch.device("cuda", 0)
    movable = np.nonzero(design.movable_mask)[0]
    particle = np.full(design.module_count, -1, np.int32)
    particle[movable] = np.arange(movable.shape[0], dtype=np.int32)
    pin_particle = particle[design.pin_module]
    static = pin_particle < 0
    pin_xy = np.stack([design.pin_offset_x, design.pin_offset_y], 1)
    pin_xy[static, 0] += design.module_x[design.pin_module[static]]
    pin_xy[static, 1] += design.module_y[design.pin_module[static]]
    pins = np.nonzero(~static)[0]
    order = pins[np.argsort(pin_particle[pins], kind="stable")]
    start = np.concatenate([[0], np.cumsum(np.bincount(pin_particle[pins], minlength=movable.shape[0]))])
    side = math.sqrt(design.core[2] * design.core[3])
    gamma = (0.75 if case["positions"] == "random" else 0.3) * side / max(32.0, math.sqrt(movable.shape[0]))

    def put(a, dtype):
        return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=device)

    xy = np.stack([design.module_x[movable], design.module_y[movable]], 1)
    return {"positions": put(xy, torch.float64), "net_pin_start": put(design.net_pin_start, torch.int32),
            "pin_particle": put(pin_particle, torch.int32), "pin_xy": put(pin_xy, torch.float64),
            "net_weight": put(design.net_weight, torch.float64), "net_count": design.net_count,
            "pin_count": design.pin_count, "particle_pin_start": put(start, torch.int32),
            "particle_pins": put(order, torch.int32), "particle_count": int(movable.shape[0]), "smoothing": gamma,
            "wire_gradient": torch.empty((movable.shape[0], 2), dtype=torch.float64, device=device),
            "totals": torch.empty(2, dtype=torch.float64, device=device)}


# ---- one pass ----------------------------------------------------------------------------

# What a run reports that is not computed from its inputs.
_NOT_RESULTS = ("elapsed_seconds", "cuda_reserved_memory_bytes")


def _placement(placed) -> dict:
    rows = placed.history
    history = {name: np.array([row[name] for row in rows]) for name in (rows[0] if rows else ())}
    scalars = np.array([float(v) for k, v in placed.result.items() if k not in _NOT_RESULTS])
    return {"x": placed.module_x, "y": placed.module_y, "scalars": scalars, "history": history}


def run(state: dict):
    kind = state["kind"]
    if kind == "evaluate":
        return state["backend"].evaluate(state["positions"], state["smoothing"], state["gradient"])
    if kind == "rudy":
        return state["backend"].rudy(state["positions"], state["options"], state["capacity"], gradient=True)
    if kind == "wirelength":
        s = state
        library = mp.load_library()
        stream = torch.cuda.current_stream(s["positions"].device).cuda_stream
        status = library.mpgp_wirelength_noalloc(
            s["positions"].data_ptr(), s["net_pin_start"].data_ptr(), s["pin_particle"].data_ptr(),
            s["pin_xy"].data_ptr(), s["net_weight"].data_ptr(), s["net_count"], s["pin_count"],
            s["particle_pin_start"].data_ptr(), s["particle_pins"].data_ptr(), s["particle_count"], s["smoothing"],
            s["wire_gradient"].data_ptr(), s["totals"].data_ptr(), ctypes.c_void_p(stream))
        if status != 0:
            raise RuntimeError(library.mpgp_last_error())
        return {"wire_gradient": s["wire_gradient"], "totals": s["totals"]}
    if kind == "place":
        return _placement(mp.GlobalPlacer().run(state["design"], state["options"]))
    if kind == "batch":
        placed, _, _ = mp.batch_place(state["designs"], state["options"], workers=16)
        return {"x": np.concatenate([p.module_x for p in placed]), "y": np.concatenate([p.module_y for p in placed]),
                "hpwl": np.array([p.hpwl_after for p in placed]),
                "overflow": np.array([p.overflow_after for p in placed]),
                "evaluations": np.array([p.evaluations for p in placed])}
    placed, result = mp.DetailedPlacer().run(state["design"], state["options"])
    return {"x": placed.module_x, "y": placed.module_y, "orientation": placed.module_orientation,
            **{k: v for k, v in result.items() if k not in _NOT_RESULTS}}


# ---- what a pass cannot do without ---------------------------------------------------------


def work(case: dict) -> dict:
    """Compulsory bytes (each input read once, each output written once) and FLOPs of one pass.

    An evaluation reads 20 bytes a pin (particle, offset, slot), 8 a net, 16 (position) + 33
    (static) a particle and the static density, and writes 32 a particle for the two gradients;
    its field transforms, done as fast transforms, take about 2.5 n log2 n each (a forward pair,
    and two inverse pairs with a gradient).
    """
    kind = case["kind"]
    if kind == "batch":
        one = work({"kind": "place", "cells": case["cells"], "bins_x": 55, "bins_y": 55,
                    "iterations": case["iterations"], "macros": 0, "rudy": False})
        return {k: v * case["count"] for k, v in one.items()}
    cells = case["cells"]
    nets = int(cells * 1.0476)
    pins = int(3.85 * nets)
    if kind == "wirelength":
        return {"bytes": 24.0 * pins + 12.0 * nets + 36.0 * cells + 4.0 * pins, "flops": 40.0 * pins}
    if kind == "rudy":
        bins = case["grid"] ** 2
        return {"bytes": 20.0 * pins + 12.0 * nets + 32.0 * cells + 16.0 * bins, "flops": 100.0 * nets}
    if kind == "detail":
        return {"bytes": case["passes"] * (28.0 * pins + 48.0 * cells), "flops": case["passes"] * 25.0 * 8.0 * pins}
    particles = cells + _fillers(cells)
    bins = case["bins_x"] * case["bins_y"]

    def evaluation(gradient):
        transforms = 3 if gradient else 1
        return ((20.0 * pins + 8.0 * nets + 49.0 * particles + 8.0 * bins + (32.0 * particles if gradient else 0.0)),
                40.0 * pins + 60.0 * particles + transforms * 2.5 * bins * math.log2(max(2, bins)))

    if kind == "evaluate":
        moved, flops = evaluation(case["gradient"])
        return {"bytes": moved, "flops": flops}
    # A controller iteration: the current point and the lookahead with a gradient, a candidate without.
    with_gradient, without = evaluation(True), evaluation(False)
    n = case["iterations"]
    return {"bytes": n * (2 * with_gradient[0] + without[0]), "flops": n * (2 * with_gradient[1] + without[1])}


# ---- the same in 64 bits -------------------------------------------------------------------


def _device(a, dtype=torch.float64):
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device="cuda")


def _pins(net_pin_start, pin_particle, pin_x, pin_y, positions):
    """(net of each pin, particle index, movable mask, x, y) in 64 bits on the GPU."""
    start = _device(net_pin_start, torch.int64)
    net = torch.repeat_interleave(torch.arange(start.numel() - 1, device="cuda"), start[1:] - start[:-1])
    particle = _device(pin_particle, torch.int64)
    movable = particle >= 0
    index = particle.clamp(min=0)
    x = _device(pin_x) + torch.where(movable, positions[index, 0], 0.0)
    y = _device(pin_y) + torch.where(movable, positions[index, 1], 0.0)
    return net, index, movable, x, y


def _exact_wirelength(net, index, movable, x, y, weight, particles: int, gamma: float):
    """Weighted log-sum-exp wirelength, HPWL and the gradient by particle."""
    nets = weight.numel()
    counted = (torch.bincount(net, minlength=nets) >= 2).double() * weight
    smooth = torch.zeros((), dtype=torch.float64, device="cuda")
    hpwl = torch.zeros_like(smooth)
    gradient = torch.zeros((particles, 2), dtype=torch.float64, device="cuda")
    for axis, v in enumerate((x, y)):
        top = torch.full((nets,), -math.inf, dtype=torch.float64, device="cuda").scatter_reduce_(0, net, v, "amax")
        low = torch.full((nets,), math.inf, dtype=torch.float64, device="cuda").scatter_reduce_(0, net, v, "amin")
        ep, en = torch.exp((v - top[net]) / gamma), torch.exp((low[net] - v) / gamma)
        sp = torch.zeros(nets, dtype=torch.float64, device="cuda").index_add_(0, net, ep)
        sn = torch.zeros(nets, dtype=torch.float64, device="cuda").index_add_(0, net, en)
        span = torch.where(counted > 0, top - low, 0.0)
        soft = torch.where(counted > 0, torch.log(sp) + torch.log(sn), 0.0)
        hpwl += (counted * span).sum()
        smooth += (counted * (span + gamma * soft)).sum()
        pin = counted[net] * (ep / sp[net] - en / sn[net])
        gradient[:, axis].index_add_(0, index[movable], pin[movable])
    return smooth, hpwl, gradient


def _exact_density(layout, positions):
    """Area of each layer in each bin (bins_y, bins_x): standard cells, macros, fillers."""
    llx, lly, urx, ury = layout.region
    nx, ny = layout.bins_x, layout.bins_y
    bw, bh = (urx - llx) / nx, (ury - lly) / ny
    half_w, half_h = 0.5 * _device(layout.particle_width), 0.5 * _device(layout.particle_height)
    layer = _device(layout.particle_layer, torch.int64)
    left, right = (positions[:, 0] - half_w).clamp(min=llx), (positions[:, 0] + half_w).clamp(max=urx)
    bottom, top = (positions[:, 1] - half_h).clamp(min=lly), (positions[:, 1] + half_h).clamp(max=ury)
    c0 = ((left - llx) / bw).floor().clamp(0, nx - 1).long()
    r0 = ((bottom - lly) / bh).floor().clamp(0, ny - 1).long()
    wide = int((((right - llx) / bw).ceil().long() - c0).max())
    high = int((((top - lly) / bh).ceil().long() - r0).max())
    area = torch.zeros(3 * nx * ny, dtype=torch.float64, device="cuda")
    for i in range(high):
        row = r0 + i
        y0 = lly + row.double() * bh
        oy = (torch.minimum(top, y0 + bh) - torch.maximum(bottom, y0)).clamp(min=0.0)
        for j in range(wide):
            column = c0 + j
            x0 = llx + column.double() * bw
            ox = (torch.minimum(right, x0 + bw) - torch.maximum(left, x0)).clamp(min=0.0)
            inside = (row < ny) & (column < nx)
            at = (layer * ny + row.clamp(max=ny - 1)) * nx + column.clamp(max=nx - 1)
            area.index_add_(0, at, torch.where(inside, ox * oy, 0.0))
    return area.reshape(3, ny, nx)


def _density_metrics(charge, movable, t: float, bin_area: float, dark):
    overflow = (charge - t * bin_area).clamp(min=0.0).sum()
    normalization = movable.sum()
    density = charge / bin_area
    return {"total_overflow_area": overflow, "normalized_overflow": overflow / normalization,
            "maximum_density": density.max(), "average_density": density.mean(), "total_charge_area": charge.sum(),
            "normalization_area": normalization, "placeable_area": (bin_area - dark).sum(), "dark_area": dark.sum()}


def _exact_field(source, width: float, height: float):
    """(energy sum, Ex, Ey) of the Neumann problem with the transforms as matrices."""
    ny, nx = source.shape

    def angles(n):
        k = torch.arange(n, dtype=torch.float64, device="cuda")
        return math.pi * k[:, None] * (2 * k[None, :] + 1) / (2 * n)

    ax, ay = angles(nx), angles(ny)
    kx = math.pi * torch.arange(nx, dtype=torch.float64, device="cuda") / width
    ky = math.pi * torch.arange(ny, dtype=torch.float64, device="cuda") / height
    rho = (2 * torch.cos(ay)) @ source @ (2 * torch.cos(ax)).T
    square = ky[:, None] ** 2 + kx[None, :] ** 2
    square[0, 0] = 1.0
    phi = rho / (4.0 * nx * ny * square)
    phi[0, 0] = 0.0
    weight_y = torch.ones(ny, dtype=torch.float64, device="cuda")
    weight_x = torch.ones(nx, dtype=torch.float64, device="cuda")
    weight_y[0] = weight_x[0] = 0.5
    energy = (phi * rho * weight_y[:, None] * weight_x[None, :]).sum()
    cy, cx = 2 * torch.cos(ay), 2 * torch.cos(ax)
    cy[0], cx[0] = 1.0, 1.0
    ex = cy.T @ phi @ (2 * torch.sin(ax) * kx[:, None])
    ey = (2 * torch.sin(ay) * ky[:, None]).T @ phi @ cx
    return energy, ex, ey


def _sample(field, gx, gy, odd_in_x: bool):
    """Bilinear sample at bin coordinates, mirrored past the edges (odd in x or in y)."""
    ny, nx = field.shape
    fx, fy = gx.floor(), gy.floor()
    tx, ty = gx - fx, gy - fy
    total = torch.zeros_like(gx)
    for j in (0, 1):
        for i in (0, 1):
            column, row = fx.long() + i, fy.long() + j
            out_x, out_y = (column < 0) | (column >= nx), (row < 0) | (row >= ny)
            column = torch.where(column < 0, -column - 1, torch.where(column >= nx, 2 * nx - column - 1, column))
            row = torch.where(row < 0, -row - 1, torch.where(row >= ny, 2 * ny - row - 1, row))
            sign = torch.where(out_x if odd_in_x else out_y, -1.0, 1.0)
            total += sign * field[row, column] * (tx if i else 1 - tx) * (ty if j else 1 - ty)
    return total


def _exact_evaluate(case: dict, seed: int) -> dict:
    layout, host_positions = _layout(_placed(case, seed), case["bins_x"], case["bins_y"])
    positions = _device(host_positions)
    smooth, hpwl, wire = _exact_wirelength(
        *_pins(layout.net_pin_start, layout.pin_particle, layout.pin_x, layout.pin_y, positions),
        _device(layout.net_weight), positions.shape[0], _smoothing(case, layout))
    llx, lly, urx, ury = layout.region
    nx, ny, t = layout.bins_x, layout.bins_y, layout.target_density
    bin_w, bin_h = (urx - llx) / nx, (ury - lly) / ny
    bin_area = bin_w * bin_h
    cells, macros, fillers = _exact_density(layout, positions)
    dark = _device(layout.static_dark).reshape(ny, nx)
    design_charge = cells + t * (macros + _device(layout.static_fixed).reshape(ny, nx) + dark)
    charge = design_charge + t * fillers
    source = charge / bin_area - t
    energy, ex, ey = _exact_field(source - source.mean(), urx - llx, ury - lly)
    out = {"hpwl": hpwl, "smooth_wirelength": smooth, "electrostatic_energy": 0.5 * bin_area * energy,
           "optimizer_density": _density_metrics(charge, cells + t * macros, t, bin_area, dark),
           "design_density": _density_metrics(design_charge, cells + t * macros, t, bin_area, dark)}
    if case["gradient"]:
        area = _device(layout.particle_width) * _device(layout.particle_height)
        area = torch.where(_device(layout.particle_layer, torch.int64) == 0, area, t * area)
        gx = (positions[:, 0].clamp(llx, urx) - llx) / bin_w - 0.5
        gy = (positions[:, 1].clamp(lly, ury) - lly) / bin_h - 0.5
        out["wire_gradient"] = wire
        out["density_gradient"] = -area[:, None] * torch.stack([_sample(ex, gx, gy, True),
                                                                _sample(ey, gx, gy, False)], 1)
    return out


def _exact_rudy(case: dict, seed: int) -> dict:
    """Demand maps as matrix products of the nets' bin overlaps along x and y; gradient by autograd
    (positions are generic: no edge on a grid line, no two pins on one edge)."""
    design = _placed(case, seed)
    layout, host_positions = _layout(design, 128, 128)
    n = case["grid"]
    llx, lly, urx, ury = layout.region
    bin_w, bin_h = (urx - llx) / n, (ury - lly) / n
    span = 0.25
    positions = _device(host_positions).requires_grad_(True)
    net, _, _, x, y = _pins(layout.net_pin_start, layout.pin_particle, layout.pin_x, layout.pin_y, positions)
    weight = _device(layout.net_weight)
    counted = torch.bincount(net, minlength=weight.numel()) >= 2

    def box(v, minimum):
        low = torch.full_like(weight, math.inf).scatter_reduce(0, net, v, "amin")[counted]
        high = torch.full_like(weight, -math.inf).scatter_reduce(0, net, v, "amax")[counted]
        center = 0.5 * (low + high)
        thin = high - low < minimum
        return (torch.where(thin, center - 0.5 * minimum, low), torch.where(thin, center + 0.5 * minimum, high))

    def overlaps(low, high, origin, length):
        edge = origin + length * torch.arange(n, dtype=torch.float64, device="cuda")
        return (torch.minimum(high[:, None], edge + length) - torch.maximum(low[:, None], edge)).clamp(min=0.0)

    left, right = box(x, span * bin_w)
    bottom, top = box(y, span * bin_h)
    ox, oy = overlaps(left, right, llx, bin_w), overlaps(bottom, top, lly, bin_h)
    w = weight[counted]
    horizontal = (oy * (w / (top - bottom))[:, None]).T @ ox
    vertical = (oy * (w / (right - left))[:, None]).T @ ox
    capacity = _rudy_capacity(design)
    uh, uv = horizontal / capacity[0], vertical / capacity[1]
    over_h, over_v = (uh - 1.0).clamp(min=0.0), (uv - 1.0).clamp(min=0.0)
    energy = (0.5 * over_h ** 2 + 0.5 * over_v ** 2).sum() / (n * n)
    energy.backward()
    utilization = torch.maximum(uh, uv).detach().reshape(-1)
    p95 = utilization.sort().values[int(math.floor(0.95 * (n * n - 1)))]
    e = energy.detach()
    return {"horizontal_total": horizontal.sum().detach(), "vertical_total": vertical.sum().detach(),
            "horizontal_mean": horizontal.mean().detach(), "vertical_mean": vertical.mean().detach(),
            "horizontal_capacity": capacity[0], "vertical_capacity": capacity[1],
            "proxy_overflow": (over_h + over_v).sum().detach() / (n * n), "maximum_utilization": utilization.max(),
            "p95_utilization": p95, "energy": e, "gradient": positions.grad, "evaluation_energy": e}


def exact(case: dict, seed: int):
    """What run() returns, in 64 bits without the engine; None where no such value exists (a
    controller's trajectory, a choice of orders)."""
    if case["kind"] == "evaluate":
        return _exact_evaluate(case, seed)
    if case["kind"] == "rudy":
        return _exact_rudy(case, seed)
    if case["kind"] == "wirelength":
        s = prepare(case, seed)
        net, index, movable, x, y = _pins(s["net_pin_start"].cpu(), s["pin_particle"].cpu(), s["pin_xy"][:, 0].cpu(),
                                          s["pin_xy"][:, 1].cpu(), s["positions"])
        smooth, hpwl, gradient = _exact_wirelength(net, index, movable, x, y, s["net_weight"], s["particle_count"],
                                                   s["smoothing"])
        return {"wire_gradient": gradient, "totals": torch.stack([smooth, hpwl])}
    return None
