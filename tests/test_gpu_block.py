"""The register-tile kernel (kernels_block.cu: several steps per launch)
against the FP32 oracle, bit for bit, where its windows can go wrong: widths
and heights at and around one window (128 columns; 16 to 64 rows) and around
the stride of the next, last windows that hold a single row or column of their
own, runs whose length leaves every remainder of the steps per launch, still
water beside moving water, and cells at rest that differ from +0."""
import numpy as np
import pytest

from comcot_b200 import _lib, synth
from comcot_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _forms():
    lib = _lib.load()
    n = lib.gc_engine_num_candidates()
    return list(range(n - 8, n))   # the last candidates


def _case(nx, ny, steps, land=True):
    case = synth.single_layer_case("b", nx, ny, 2.0, 2.0, steps, seed=nx + 7 * ny, n_seamounts=2,
                                   shelf_cols=max(2, nx // 10) if land else 0, land_cols=max(1, nx // 30) if land else 0,
                                   source="hump", amp=2.0)
    # moving water in one corner only, some of it on the boundary
    z = np.zeros((ny, nx), np.float32)
    k = min(nx, ny, 9)
    z[:k, :k] = np.linspace(0.5, -0.4, k * k, dtype=np.float32).reshape(k, k)
    z[case.root.H <= 0] = 0.0
    z[ny // 2, nx // 2] = -0.0
    case.root.Z0 = z
    if nx > 4 and ny > 4:
        case.gauges = [(1, 2, 2, 0.25, 0.75), (1, nx - 2, ny - 2, 0.5, 0.5)]
    return case


def _check(case, got, oracle_mod, what):
    o = oracle_mod.OracleRun(case)
    ts = o.run(case.nsteps)
    ref = o.layer(0)
    for k in ("z", "m", "n", "zmax"):
        assert np.array_equal(got[k].view(np.uint32), ref[k].view(np.uint32)), (what, k)
    assert np.array_equal(got["arrival"], ref["arrival"]), what
    if case.gauges:
        assert np.array_equal(got["ts"].view(np.uint32), ts.view(np.uint32)), what


@pytest.mark.parametrize("nx,ny", [(3, 3), (127, 16), (128, 17), (129, 32), (132, 33), (240, 49), (241, 65), (249, 25),
                                   (250, 113)])
@pytest.mark.parametrize("land", [True, False])
def test_window_edges(oracle_mod, nx, ny, land):
    case = _case(nx, ny, 21, land)
    for v in _forms():
        with Engine(budget=1 << 30) as eng:
            eng.config(variant=v, use_graphs=0, chunk=8)
            mid = eng.add(case)
            eng.step(case.nsteps + 1)
            eng.sync()
            _check(case, eng.read(mid), oracle_mod, (v, nx, ny, land))


@pytest.mark.parametrize("steps", [1, 2, 3, 4, 5, 6, 7, 8, 9, 11, 16, 17])
def test_every_remainder(oracle_mod, steps):
    case = _case(150, 70, steps)
    for v in _forms():
        with Engine(budget=1 << 30) as eng:
            eng.config(variant=v, use_graphs=0, chunk=8)
            mid = eng.add(case)
            eng.step(steps + 1)
            eng.sync()
            _check(case, eng.read(mid), oracle_mod, (v, steps))
