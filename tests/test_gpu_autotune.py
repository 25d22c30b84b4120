"""The autotuner on a fresh engine: every candidate's steps go out in launches
of that candidate's own number of steps (so what is timed is the candidate),
the winner is what runs afterwards, and the steps it took are ordinary steps of
the forecast."""
import numpy as np
import pytest

from comcot_b200 import _lib, synth
from comcot_b200.engine import Engine

pytestmark = pytest.mark.gpu


# an untuned engine takes four steps a launch on the first grid and eight on the others
@pytest.mark.parametrize("nx,ny,members", [(600, 480, 1), (150, 70, 1), (150, 70, 3)])
def test_candidates_are_timed_as_themselves(oracle_mod, nx, ny, members):
    reps = 1
    case = synth.single_layer_case("t", nx, ny, 2.0, 2.0, 600, seed=2, n_seamounts=2, shelf_cols=15, land_cols=5,
                                   source="hump", amp=2.0, ngauges=2)
    ncand = _lib.load().gc_engine_num_candidates()
    with Engine(budget=1 << 30) as eng:
        eng.config(use_graphs=0)
        ids = [eng.add(case) for _ in range(members)]
        best = eng.autotune(reps)
        assert 0 <= best < ncand and eng.lib.gc_engine_variant(eng.h) == best
        # one warm launch and `reps` timed ones each, then three finalists with three times the steps
        assert eng.launches() == ncand * (1 + reps) + 3 * (1 + 3 * reps)
        eng.step(case.nsteps + 1)
        eng.sync()
        got = [eng.read(i) for i in ids]
    o = oracle_mod.OracleRun(case)
    ts = o.run(case.nsteps)
    ref = o.layer(0)
    for g in got:
        for k in ("z", "m", "n", "zmax"):
            assert np.array_equal(g[k].view(np.uint32), ref[k].view(np.uint32)), k
        assert np.array_equal(g["arrival"], ref["arrival"]) and np.array_equal(g["ts"].view(np.uint32), ts.view(np.uint32))
