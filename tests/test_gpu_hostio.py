"""Field transfers through page-locked staging: what goes up comes back, for
fields below the staging threshold, of one piece, of several pieces with an odd
last one, and from several threads with engines of their own."""
import threading

import numpy as np
import pytest

from comcot_b200 import synth
from comcot_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _round_trip(nx, ny, seed):
    rng = np.random.default_rng(seed)
    H = np.full((ny, nx), 1000.0, np.float32)
    x, y = synth.pc.axes(140.0, 10.0, nx, ny, 0.5)
    L = synth.spherical_layer(1, x, y, H, rng.standard_normal((ny, nx)).astype(np.float32), 0.2, 0.5)
    case = synth.Case("io", [L], 4)
    with Engine(budget=4 << 30) as eng:
        mid = eng.add(case)
        now = eng.read(mid, fields=("z", "m", "zmax", "arrival"))
        pend = eng.read_async(mid, fields=("z", "zmax"))
        later = pend.take()
    for got in (now, later):
        assert np.array_equal(got["z"], L.Z0) and np.array_equal(got["zmax"], L.Z0)
    assert not now["m"].any() and set(np.unique(now["arrival"])) <= {-1, 0}


@pytest.mark.parametrize("nx,ny", [(33, 17), (256, 256), (257, 255), (1025, 2047), (2048, 1024), (2401, 2001)])
def test_round_trip(nx, ny):
    _round_trip(nx, ny, nx + ny)


def test_round_trips_from_threads():
    errors = []

    def work(k):
        try:
            for q in range(3):
                _round_trip(700 + 13 * k, 500 + 7 * q, 10 * k + q)
        except Exception as exc:   # noqa: BLE001 - reported below
            errors.append(exc)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
