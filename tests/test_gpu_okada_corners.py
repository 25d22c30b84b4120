"""The fault source where its corner sums can go wrong: cells level with a
fault end (y1 = 0, the arc tangent's branch), cells on the fault's trace, a
vertical dip, pure strike-slip and pure dip-slip, more faults than one launch
takes, blocks that end inside the layer.  Against the oracle's double
restatement, with the tolerance of the double evaluation rounded to float."""
import ctypes as C

import numpy as np
import pytest

from comcot_b200 import _lib

pytestmark = pytest.mark.gpu


def _apply(faults, laycord, nx, ny, x, y, dx, dy):
    import torch

    dev = torch.device("cuda", 0)
    pitch = (nx + 31) // 32 * 32
    z = torch.zeros((ny, pitch), dtype=torch.float32, device=dev)
    h = torch.full((ny, pitch), 1000.0, dtype=torch.float32, device=dev)
    xd, yd = torch.from_numpy(x).to(dev), torch.from_numpy(y).to(dev)
    arr = _lib.faults_array(faults)
    torch.cuda.synchronize()
    rc = _lib.load().gc_okada_apply(C.cast(arr, C.c_void_p), len(faults), laycord, nx, ny, pitch, xd.data_ptr(),
                                    yd.data_ptr(), dx, dy, z.data_ptr(), h.data_ptr(), None)
    assert rc == 0
    torch.cuda.synchronize()
    return z[:, :nx].cpu().numpy()


FAULT = dict(hh=6000.0, l=40000.0, w=20000.0, d=2.0, th=0.0, dl=30.0, rd=75.0, x0=142.0, y0=38.0, sw=0)
FORMS = [dict(), dict(dl=89.9), dict(dl=45.0, rd=0.0), dict(rd=90.0), dict(rd=180.0, th=90.0), dict(th=37.0, sw=9),
         dict(hh=1.0e-3, dl=60.0)]


@pytest.mark.parametrize("laycord", [0, 1])
@pytest.mark.parametrize("form", range(len(FORMS)))
def test_corner_sums(oracle_mod, laycord, form):
    nx, ny = 131, 83
    x = (np.float32(141.0) + np.arange(nx, dtype=np.float32) * np.float32(2.0 / nx)).astype(np.float32)
    y = (np.float32(37.0) + np.arange(ny, dtype=np.float32) * np.float32(2.0 / ny)).astype(np.float32)
    # Cartesian: the origin is the epicentre moved by whole cells, so rows lie exactly level with the fault's ends
    f = dict(FAULT, **FORMS[form], xo=142.0, yo=38.0)
    dx = dy = 1000.0
    z = _apply([f], laycord, nx, ny, x, y, dx, dy)
    z64, _ = oracle_mod.okada_apply([f], laycord, nx, ny, x.astype(np.float64), y.astype(np.float64), dx, dy,
                                    np.zeros((ny, nx), np.float32), np.full((ny, nx), 1000.0, np.float32),
                                    dtype=np.float64)
    scale = float(np.abs(z64).max())
    assert scale > 1e-3
    # 1e-6: a displacement at the 1e-5 m threshold may fall on either side of it
    assert np.all(np.abs(z - z64) <= 1e-6 * scale + 1.1e-5)
    assert (np.abs(z - z64) > 1e-6 * scale + 1e-6).mean() < 1e-3


def test_more_faults_than_one_launch(oracle_mod):
    nx, ny = 130, 9
    x = (np.float32(141.0) + np.arange(nx, dtype=np.float32) * np.float32(0.01)).astype(np.float32)
    y = (np.float32(37.5) + np.arange(ny, dtype=np.float32) * np.float32(0.1)).astype(np.float32)
    faults = [dict(FAULT, th=15.0 * k, d=0.5 + 0.1 * k) for k in range(14)]
    z = _apply(faults, 0, nx, ny, x, y, 0.0, 0.0)
    z64, _ = oracle_mod.okada_apply(faults, 0, nx, ny, x.astype(np.float64), y.astype(np.float64), 0.0, 0.0,
                                    np.zeros((ny, nx), np.float32), np.full((ny, nx), 1000.0, np.float32),
                                    dtype=np.float64)
    scale = float(np.abs(z64).max())
    assert np.all(np.abs(z - z64) <= 14 * 2.0 ** -23 * scale + 14 * 1.1e-5)
    assert (np.abs(z - z64) > 1e-6 * scale + 1e-6).mean() < 1e-2
