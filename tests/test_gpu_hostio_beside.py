"""A read of one engine returns while another engine, whose read came first and
is waiting in another thread, still has work queued."""
import threading
import time

import numpy as np
import pytest
import torch

from comcot_b200 import synth
from comcot_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _case(nx, ny):
    return synth.single_layer_case("r", nx, ny, 2.0, 2.0, 4, seed=nx, n_seamounts=1, shelf_cols=20, land_cols=6,
                                   source="hump")


def test_reads_of_two_engines_are_independent():
    ca, cb = _case(900, 700), _case(700, 500)   # both above the staging threshold
    with Engine(budget=1 << 30) as a, Engine(budget=1 << 30) as b:
        ia, ib = a.add(ca), b.add(cb)
        a.read(ia), b.read(ib)                  # the buffers are there
        with torch.cuda.stream(torch.cuda.ExternalStream(int(a.lib.gc_engine_stream(a.h)))):
            torch.cuda._sleep(1_500_000_000)    # most of a second of work ahead of the read
        got = {}
        t = threading.Thread(target=lambda: got.update(a.read(ia)))
        t.start()
        time.sleep(0.1)
        mine = b.read(ib)
        still_running = a.lib.gc_engine_query(a.h) == 0
        t.join()
        assert still_running
        assert np.array_equal(mine["z"], cb.root.Z0) and np.array_equal(got["z"], ca.root.Z0)
