"""The one-step kernel (kernels_step.cu) through the allocation-free step and
the reference ABI, against the FP32 oracle bit for bit, at the edges of its
120-column windows and of its rows per CTA, alone, in short and in long lists
of grids, with and without the maximum."""
import ctypes as C

import numpy as np
import pytest

from comcot_b200 import _lib, synth

pytestmark = pytest.mark.gpu


class StepIO(C.Structure):
    _fields_ = ([("nx", C.c_int), ("ny", C.c_int), ("pitch", C.c_int)]
                + [(n, C.c_void_p) for n in ("z1", "m1", "n1", "z2", "m2", "n2", "h", "rows", "zmax")])


def _case(nx, ny, land):
    c = synth.single_layer_case("s", nx, ny, 2.0, 2.0, 2, seed=nx * 31 + ny, n_seamounts=2,
                                shelf_cols=max(2, nx // 10) if land else 0, land_cols=max(1, nx // 30) if land else 0,
                                source="dipole", amp=2.0)
    rng = np.random.default_rng(nx + ny)
    c.root.Z0 = np.where(c.root.H > 0, rng.uniform(-0.5, 0.5, size=(ny, nx)), 0.0).astype(np.float32)
    return c


def _steps(cases, use_max):
    import torch

    def pitched(a):
        pitch = (a.shape[1] + 31) // 32 * 32
        t = torch.full((a.shape[0], pitch), float("nan"), dtype=torch.float32, device="cuda")  # padding is the caller's
        t[:, :a.shape[1]] = torch.from_numpy(np.ascontiguousarray(a, np.float32)).cuda()
        return t

    lib, bufs = _lib.load(), []
    for c in cases:
        L = c.root
        rec = np.zeros((L.ny, 8), np.float32)
        rec[:, :7] = L.coefs.rows().T
        zero = np.zeros((L.ny, L.nx), np.float32)
        bufs.append({"L": L, "f": [[pitched(L.Z0), pitched(zero), pitched(zero)] for _ in range(2)], "h": pitched(L.H),
                     "rows": torch.from_numpy(rec).cuda(), "x": pitched(L.Z0)})
    for k in range(2):
        arr = (StepIO * len(bufs))()
        for q, b in zip(arr, bufs):
            q.nx, q.ny, q.pitch = b["L"].nx, b["L"].ny, b["h"].shape[1]
            q.z1, q.m1, q.n1 = (t.data_ptr() for t in b["f"][k])
            q.z2, q.m2, q.n2 = (t.data_ptr() for t in b["f"][1 - k])
            q.h, q.rows = b["h"].data_ptr(), b["rows"].data_ptr()
            q.zmax = b["x"].data_ptr() if use_max else None
        rc = lib.gcomcot_fused_step_noalloc(len(bufs), C.cast(arr, C.c_void_p),
                                            C.c_void_p(torch.cuda.current_stream().cuda_stream))
        assert rc == 0
    torch.cuda.synchronize()
    return [dict(zip(("z", "m", "n", "zmax"), (t[:, :b["L"].nx].cpu().numpy() for t in (*b["f"][0], b["x"]))))
            for b in bufs]


SIZES = [(3, 3), (127, 4), (128, 5), (129, 7), (132, 8), (244, 9), (248, 17), (249, 3), (367, 33), (1500, 1400)]


@pytest.mark.parametrize("land", [True, False])
@pytest.mark.parametrize("use_max", [True, False])
def test_sizes(oracle_mod, land, use_max):
    cases = [_case(nx, ny, land) for nx, ny in SIZES]
    got = [g for c in cases for g in _steps([c], use_max)]
    got_list = _steps(cases, use_max)
    for c, a, b in zip(cases, got, got_list):
        o = oracle_mod.OracleRun(c)
        o.run(2)
        ref = o.layer(0)
        for k in ("z", "m", "n") + (("zmax",) if use_max else ()):
            assert np.array_equal(a[k].view(np.uint32), ref[k].view(np.uint32)), (c.root.nx, c.root.ny, k)
            assert np.array_equal(b[k].view(np.uint32), ref[k].view(np.uint32)), (c.root.nx, c.root.ny, k)
