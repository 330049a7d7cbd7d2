"""Evaluations' host transfers at the sizes where their path changes (needs a GPU).

Particle counts below and above the size that helper threads copy, and past the ring of pinned
slots: positions with a non-finite value anywhere are refused and leave the last evaluation's
state, repeated and interleaved evaluations equal a fresh backend's bit for bit, and the layers
equal the fixed-point oracle's.
"""
from __future__ import annotations

import numpy as np
import pytest

import myplacement_b200 as mp
from myplacement_b200 import _abi
from oracle.ref import fixed_deposit

pytestmark = pytest.mark.gpu


def _layout(cells: int, bins: int):
    design = mp.synthetic_design(cells=cells, nets=cells, terminals=32, utilization=0.7, seed=cells)
    options = mp.default_options(bins_x=bins, bins_y=bins, target_density=0.9)
    setup = mp.host_setup(design, options)
    count = int(setup["particle_count"])
    layout = mp.build_layout(design, setup["width"], setup["height"], setup["layer"], np.zeros(count, np.int32),
                             int(setup["movable_count"]), bins, bins, 0.9, setup["static_fixed"],
                             setup["static_dark"])
    return design, setup, layout, count


def _positions(design, count: int, seed: int) -> np.ndarray:
    llx, lly, urx, ury = design.core
    return np.random.default_rng(seed).uniform((llx, lly), (urx, ury), (count, 2))


def _same(a: dict, b: dict) -> None:
    assert a.keys() == b.keys()
    for key, value in a.items():
        assert np.array_equal(value, b[key]) if isinstance(value, np.ndarray) else value == b[key], key


@pytest.mark.parametrize("cells,bins", [(700, 16), (24_000, 64), (27_500, 96), (270_000, 128)])
def test_transfers(gpu, cells, bins):
    design, setup, layout, count = _layout(cells, bins)
    places = [_positions(design, count, seed) for seed in range(3)]
    expected = []
    for place in places:
        backend, reason = mp.try_create_backend(layout, 0)
        assert backend is not None, reason
        expected.append(backend.evaluate(place, 3.0, True))
        backend.close()
    backend, reason = mp.try_create_backend(layout, 0)
    assert backend is not None, reason
    options = mp.default_options(rudy_columns=16, rudy_rows=16, rudy_penalty_model=1)
    _same(backend.evaluate(places[0], 3.0, True), expected[0])
    for index, bad in ((0, np.nan), (count // 2, np.inf), (count - 1, -np.inf)):
        broken = places[1].copy()
        broken[index, index % 2] = bad
        with pytest.raises(mp.EngineError) as error:
            backend.evaluate(broken, 3.0, True)
        assert error.value.status == _abi.MPGP_ERR_NON_FINITE
    # The refused positions left the last evaluation's in place.
    layers = backend.density_layers(bins, bins)
    wanted = fixed_deposit(places[0][:, 0], places[0][:, 1], setup["width"], setup["height"], setup["layer"],
                           design.core, bins, bins)
    for mine, theirs in zip(layers, wanted):
        assert np.array_equal(mine, theirs)
    for k in (1, 2, 0, 2):
        _same({key: value for key, value in backend.evaluate(places[k], 3.0, False).items()},
              {key: value for key, value in expected[k].items() if not key.endswith("gradient")})
        backend.rudy(places[1], options)
        _same(backend.evaluate(places[k], 3.0, True), expected[k])
    backend.close()


def test_two_threads_share_the_ring(gpu):
    """Two backends on two host threads: one at a time has the shared ring and helpers, the other
    copies through slots of its own; both return what they return alone."""
    import threading

    made = [_layout(cells, 64) for cells in (30_000, 45_000)]
    backends, expected, places = [], [], []
    for design, _, layout, count in made:
        backend, reason = mp.try_create_backend(layout, 0)
        assert backend is not None, reason
        place = _positions(design, count, 5)
        backends.append(backend)
        places.append(place)
        expected.append(backend.evaluate(place, 3.0, True))
    failures = []

    def work(k: int) -> None:
        try:
            for _ in range(40):
                _same(backends[k].evaluate(places[k], 3.0, True), expected[k])
        except BaseException as error:  # noqa: BLE001 -- reported below
            failures.append(error)

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    for backend in backends:
        backend.close()
    assert not failures, failures[0]
