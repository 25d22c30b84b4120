"""The reference ABI's field setters read the caller's array before they return,
ordinary or page-locked, also behind work that is still queued."""
import ctypes as C

import numpy as np
import pytest
import torch

from comcot_b200 import _lib, synth
from comcot_b200.abi import ReferenceSession, _i

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(200, 200), (300, 300)])   # below and above the staging threshold
@pytest.mark.parametrize("locked", [False, True])
def test_setters_read_before_they_return(nx, ny, locked):
    lib = _lib.load()
    case = synth.single_layer_case("s", nx, ny, 2.0, 2.0, 4, seed=3, n_seamounts=1, shelf_cols=20, land_cols=6,
                                   source="hump")
    rng = np.random.default_rng(5)
    want = [rng.standard_normal((ny, nx)).astype(np.float32) for _ in range(3)]
    ptrs, arrays = [], []
    for _ in want:
        if locked:
            ptrs.append(lib.gc_host_alloc(4 * nx * ny))
            arrays.append(np.ctypeslib.as_array(C.cast(ptrs[-1], C.POINTER(C.c_float)), (ny, nx)))
        else:
            arrays.append(np.empty((ny, nx), np.float32))
    s = ReferenceSession(case)
    try:
        for a, w in zip(arrays, want):
            a[:] = w
        with torch.cuda.stream(torch.cuda.ExternalStream(s.stream())):
            torch.cuda._sleep(100_000_000)   # about 50 ms of work ahead of the copies
        lib.cuda_setz1_(_lib.fptr(arrays[0]), _i(1))
        arrays[0][:] = -7.0
        lib.cuda_setmn1_(_lib.fptr(arrays[1]), _lib.fptr(arrays[2]), _i(1))
        arrays[1][:] = -8.0
        arrays[2][:] = -9.0
        got = [np.empty((ny, nx), np.float32) for _ in range(3)]
        lib.cuda_getz1_(_lib.fptr(got[0]), _i(1))
        lib.cuda_getmn1_(_lib.fptr(got[1]), _lib.fptr(got[2]), _i(1))
        for g, w in zip(got, want):
            assert np.array_equal(g.view(np.uint32), w.view(np.uint32))
    finally:
        s.close()
        for p in ptrs:
            lib.gc_host_free(p)


@pytest.mark.parametrize("nx,ny", [(200, 200), (300, 300)])
def test_setter_follows_work_on_the_librarys_stream(nx, ny):
    """page-locked memory that queued work on the library's stream fills"""
    lib = _lib.load()
    case = synth.single_layer_case("o", nx, ny, 2.0, 2.0, 4, seed=3, n_seamounts=1, shelf_cols=20, land_cols=6,
                                   source="hump")
    want = torch.arange(nx * ny, dtype=torch.float32, device="cuda").reshape(ny, nx)
    # the library's own page-locked block: torch's would note the session's stream and ask it after the session's end
    p = lib.gc_host_alloc(4 * nx * ny)
    a = np.ctypeslib.as_array(C.cast(p, C.POINTER(C.c_float)), (ny, nx))
    a[:] = 0.0
    torch.cuda.synchronize()
    s = ReferenceSession(case)
    try:
        with torch.cuda.stream(torch.cuda.ExternalStream(s.stream())):
            torch.cuda._sleep(100_000_000)
            torch.from_numpy(a).copy_(want, non_blocking=True)
        lib.cuda_setz1_(_lib.fptr(a), _i(1))
        got = np.empty((ny, nx), np.float32)
        lib.cuda_getz1_(_lib.fptr(got), _i(1))
        assert np.array_equal(got, want.cpu().numpy())
    finally:
        s.close()
        lib.gc_host_free(p)
