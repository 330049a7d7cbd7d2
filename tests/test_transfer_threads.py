"""Backend evaluations of several threads at once: the hub's copies and the driver's (needs a GPU).

One call at a time has the ring and the helpers; the others' arrays are copied by the driver.
Every thread evaluates, with and without a gradient, has positions refused that are not finite,
and evaluates the routing demand; all results are those the backend returns alone.
"""
from __future__ import annotations

import threading

import numpy as np
import pytest

import myplacement_b200 as mp
from myplacement_b200 import _abi

pytestmark = pytest.mark.gpu


def _backend(cells: int):
    design = mp.synthetic_design(cells=cells, nets=cells, terminals=32, utilization=0.7, seed=cells)
    options = mp.default_options(bins_x=64, bins_y=64, target_density=0.9)
    setup = mp.host_setup(design, options)
    count = int(setup["particle_count"])
    layout = mp.build_layout(design, setup["width"], setup["height"], setup["layer"], np.zeros(count, np.int32),
                             int(setup["movable_count"]), 64, 64, 0.9, setup["static_fixed"], setup["static_dark"])
    backend, reason = mp.try_create_backend(layout, 0)
    assert backend is not None, reason
    llx, lly, urx, ury = design.core
    return backend, np.random.default_rng(cells).uniform((llx, lly), (urx, ury), (count, 2))


def _same(a: dict, b: dict) -> None:
    assert a.keys() == b.keys()
    for key, value in a.items():
        assert np.array_equal(value, b[key]) if isinstance(value, np.ndarray) else value == b[key], key


def test_threads_get_what_they_get_alone(gpu):
    options = mp.default_options(rudy_columns=24, rudy_rows=24, rudy_penalty_model=1)
    made = [_backend(cells) for cells in (26_000, 30_000, 45_000, 90_000)]
    alone = [(b.evaluate(p, 3.0, True), b.evaluate(p, 3.0, False), b.rudy(p, options, (5.0, 5.0), gradient=True))
             for b, p in made]
    failures = []

    def work(k: int) -> None:
        backend, place = made[k]
        broken = place.copy()
        broken[len(place) // 2, 1] = np.nan
        try:
            for _ in range(15):
                _same(backend.evaluate(place, 3.0, True), alone[k][0])
                with pytest.raises(mp.EngineError) as error:
                    backend.evaluate(broken, 3.0, True)
                assert error.value.status == _abi.MPGP_ERR_NON_FINITE
                _same(backend.evaluate(place, 3.0, False), alone[k][1])
                _same(backend.rudy(place, options, (5.0, 5.0), gradient=True), alone[k][2])
        except BaseException as error:  # noqa: BLE001 -- reported below
            failures.append(error)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(made))]
    for thread in threads:
        thread.start()
    for thread in threads:
        thread.join()
    for backend, _ in made:
        backend.close()
    assert not failures, failures[0]
