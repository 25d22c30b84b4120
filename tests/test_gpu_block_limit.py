"""Grids whose fields the register-tile kernel's 32-bit offsets cannot reach (4 GB
and more) take two steps a launch: engine members of one grid, of one class and
of a work list, and gcomcot_drive, against the oracle, with the limit lowered so
that small grids are beyond it; and the autotuner leaves the forms out that do
not fit."""
import numpy as np
import pytest

from comcot_b200 import _lib, synth
from comcot_b200.abi import ReferenceSession
from comcot_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.fixture
def low_limit():
    lib = _lib.load()
    lib.gcomcot_set_block_limit(16 << 10)
    yield lib
    lib.gcomcot_set_block_limit(0)


def _case(nx, ny, nsteps):
    return synth.single_layer_case("l", nx, ny, 2.0, 2.0, nsteps, seed=nx + ny, n_seamounts=2, shelf_cols=nx // 10,
                                   land_cols=nx // 30, source="hump", amp=2.0, ngauges=3)


def _same(got, ref, ts):
    for k in ("z", "m", "n", "zmax"):
        assert np.array_equal(got[k].view(np.uint32), ref[k].view(np.uint32)), k
    assert np.array_equal(got["arrival"], ref["arrival"]) and np.array_equal(got["ts"].view(np.uint32), ts.view(np.uint32))


@pytest.mark.parametrize("sizes", [[(150, 70)], [(150, 70)] * 3, [(150, 70), (129, 81)]])
def test_members_beyond_the_limit_take_two_steps_a_launch(oracle_mod, low_limit, sizes):
    steps = 31
    cases = {s: _case(*s, steps) for s in sizes}
    with Engine(budget=1 << 30) as eng:
        eng.config(use_graphs=0)
        ids = [eng.add(cases[s]) for s in sizes]
        eng.step(steps + 1)
        eng.sync()
        # 15 pairs, the 31st step, the launch that samples its gauges
        assert eng.launches() == 17
        for mid, s in zip(ids, sizes):
            o = oracle_mod.OracleRun(cases[s])
            ts = o.run(steps)
            _same(eng.read(mid), o.layer(0), ts)


@pytest.mark.parametrize("steps", [1, 2, 31, 1029])
def test_drive_beyond_the_limit_takes_two_steps_a_launch(oracle_mod, low_limit, steps):
    case = _case(150, 70, steps)
    o = oracle_mod.OracleRun(case)
    ts = o.run(steps)
    s = ReferenceSession(case)
    try:
        before = low_limit.gcomcot_launch_count()
        raw = s.drive(steps)
        launches = low_limit.gcomcot_launch_count() - before
        m, n = s.getmn()
        got = {"z": s.getz(), "m": m, "n": n, "zmax": s.getzmax()}
    finally:
        s.close()
    ref = o.layer(0)
    for k in got:
        assert np.array_equal(got[k].view(np.uint32), ref[k].view(np.uint32)), k
    f = np.float32
    for q, (_, _, _, cx, cy) in enumerate(case.gauges):
        l1, l2, l3, l4 = (raw[:, q, c] for c in range(4))
        cx, cy, one = f(cx), f(cy), f(1.0)
        v = l1 * (one - cx) * (one - cy) + l2 * cx * (one - cy) + l3 * (one - cx) * cy + l4 * cx * cy
        assert np.array_equal(v.view(np.uint32), ts[:, q].view(np.uint32)), q
    # a pair a launch; a last odd step alone, with its gauges; the gauges of each 1024-step chunk's last pair
    pairs = steps // 2
    assert launches == pairs + 2 * (steps % 2) + (-(-2 * pairs // 1024) if pairs else 0)


def test_autotuner_leaves_out_what_does_not_fit(low_limit):
    ncand, case = low_limit.gc_engine_num_candidates(), _case(150, 70, 600)
    with Engine(budget=1 << 30) as eng:
        eng.config(use_graphs=0)
        eng.add(case)
        best = eng.autotune(1)
        eng.step(1)
        assert 0 <= best < ncand - low_limit.gc_engine_num_block_forms() and eng.variant() == best


def test_a_long_work_list_keeps_its_steps_a_launch(oracle_mod):
    """13500 grids: the windows of one times the square of their number, the bound of a class launch (at most 64
    members), is beyond 32 bits"""
    lib, n, steps = _lib.load(), 13500, 8
    case = synth.single_layer_case("w", 3, 200, 2.0, 2.0, steps, seed=4, n_seamounts=0, shelf_cols=1, land_cols=0,
                                   source="hump", amp=2.0)
    with Engine(budget=8 << 30) as eng:
        eng.config(variant=lib.gc_engine_num_candidates() - lib.gc_engine_num_block_forms(), use_graphs=0)   # 16 rows a window, 4 steps a launch
        cls = eng.add_class(case.root)
        ids = [eng.add(case, cls=cls) for _ in range(n)]
        eng.step(steps + 1)
        eng.sync()
        assert eng.launches() == 3
        got = [eng.read(i) for i in (ids[0], ids[n // 2], ids[-1])]
    o = oracle_mod.OracleRun(case)
    o.run(steps)
    ref = o.layer(0)
    for g in got:
        for k in ("z", "m", "n", "zmax"):
            assert np.array_equal(g[k].view(np.uint32), ref[k].view(np.uint32)), k
