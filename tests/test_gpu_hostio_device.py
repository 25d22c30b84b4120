"""Surfaces that a caller holds on the device go into and out of the engine as
host arrays do, at every size."""
import ctypes as C

import numpy as np
import pytest
import torch

from comcot_b200 import _lib, synth
from comcot_b200.engine import Engine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(100, 80), (400, 300)])   # below and above the staging threshold
def test_device_pointers(nx, ny):
    case = synth.single_layer_case("d", nx, ny, 2.0, 2.0, 4, seed=3, n_seamounts=1, shelf_cols=20, land_cols=6,
                                   source="hump")
    z = torch.from_numpy(case.root.Z0.copy()).cuda()
    back = torch.zeros_like(z)
    torch.cuda.synchronize()
    with Engine(budget=1 << 30) as eng:
        cls = eng.add_class(case.root)
        mid = eng.lib.gc_engine_add_member(eng.h, cls, C.cast(z.data_ptr(), _lib.P_F), case.nsteps, 0, None, None, -1.0)
        assert mid >= 0
        assert eng.lib.gc_engine_read(eng.h, mid, C.cast(back.data_ptr(), _lib.P_F), None, None, None, None, None) == 0
    assert np.array_equal(back.cpu().numpy(), case.root.Z0)
