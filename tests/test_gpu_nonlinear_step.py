"""The one-launch step of a nonlinear layer (k_nonlinear_step) against the FP32
oracle bit for bit: children whose last block is one column or row, exactly one
block, one cell more, and grids on both sides of the line where a cell's two
faces go to two threads; one to four sub-steps, Cartesian and spherical, with
and without the modified-scheme term; root layers with and without the
maximum.  A steep surface in shallow water makes waves break and cells dry."""
import numpy as np
import pytest

from comcot_b200 import synth
from comcot_b200.abi import ReferenceSession

pytestmark = pytest.mark.gpu


def _steep(L, seed, amp):
    rng = np.random.default_rng(seed)
    jj, ii = np.mgrid[0:L.ny, 0:L.nx]
    z = amp * np.sin(ii * 0.7 + 0.3) * np.cos(jj * 0.5) + 0.2 * amp * rng.uniform(-1, 1, size=(L.ny, L.nx))
    z[:, : L.nx // 4] = 0.0  # and still water
    z[0] = 0.0  # a child's first row and column hold no wave before its first step
    L.Z0 = np.where(L.H > 0.0, z, 0.0).astype(np.float32)


def _same(a, b, what):
    assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), what


# child size = cells * ratio + 1
CHILD = [(2, 2, 3), (10, 2, 3), (9, 5, 7), (21, 13, 3), (13, 3, 5), (33, 9, 7), (80, 29, 7), (84, 33, 7), (110, 37, 7), (117, 38, 7)]


@pytest.mark.parametrize("cw,ch,r", CHILD)
@pytest.mark.parametrize("rel_time,laycord,modscm", [(1, 1, 1), (2, 1, 0), (3, 0, 1), (4, 1, 1)])
def test_child(oracle_mod, cw, ch, r, rel_time, laycord, modscm):
    is_, js = 70, 12
    case = synth.nested_case("c", 90 + cw, 24 + ch, 2.0, 2.0, [is_, is_ + cw - 1, js, js + ch - 1], r, 0,
                             seed=cw + ch, rel_time=rel_time, child_laycord=laycord, child_laygov=1)
    P, C = case.layers
    assert (C.nx, C.ny) == (cw * r + 1, ch * r + 1)
    C.modscm = modscm
    _steep(P, 3, 0.5)
    _steep(C, 4, 2.0)
    steps = 3
    s = ReferenceSession(case, fusion=True)
    try:
        for _ in range(steps):
            s.step(maxamp=True)
        got = [(s.getz(L.id), *s.getmn(L.id)) for L in case.layers]
    finally:
        s.close()
    o = oracle_mod.OracleRun(case)
    o.run(steps)
    for k in range(2):
        ref = o.layer(k)
        for a, f in zip(got[k], ("z", "m", "n")):
            _same(a, ref[f], (k, f))


@pytest.mark.parametrize("nx,ny", [(3, 3), (32, 8), (33, 9), (31, 17), (64, 24), (65, 25), (353, 211), (700, 130)])
@pytest.mark.parametrize("maxamp", [True, False])
def test_root(oracle_mod, nx, ny, maxamp):
    case = synth.single_layer_case("r", nx, ny, 2.0, 2.0, 0, seed=nx + ny, n_seamounts=2,
                                   shelf_cols=min(10, nx // 4), land_cols=min(4, nx // 8), ngauges=0, laygov=1)
    L = case.root
    L.H = np.where(L.H > 0.0, np.minimum(L.H, 40.0), L.H).astype(np.float32)  # shallow: friction and breaking count
    L.hp, L.hq = synth.pc.pq_depth(L.H)
    _steep(L, 5, 3.0)
    s = ReferenceSession(case, fusion=True)
    try:
        for _ in range(4):
            s.step(maxamp=maxamp)
        got = {"z": s.getz(1), "m": s.getmn(1)[0], "n": s.getmn(1)[1], "zmax": s.getzmax(1)}
    finally:
        s.close()
    o = oracle_mod.OracleRun(case)
    o.run(4)
    ref = o.layer(0)
    for f in ("z", "m", "n") + (("zmax",) if maxamp else ()):
        _same(got[f], ref[f], f)


@pytest.mark.parametrize("seed", [1, 2, 3])
@pytest.mark.parametrize("fric", [0.025, 0.0, 1.0e-4])
def test_friction_lines(oracle_mod, seed, fric):
    """depths and surfaces spread over many decades put friction on both sides
    of the sizes below which it is left out, at every face"""
    nx, ny = 131, 75
    case = synth.single_layer_case("f", nx, ny, 2.0, 2.0, 0, seed=seed, n_seamounts=0, shelf_cols=0, land_cols=0,
                                   ngauges=0, laygov=1, fric=fric)
    L = case.root
    rng = np.random.default_rng(seed)
    jj, ii = np.mgrid[0:ny, 0:nx]
    L.H = (10.0 ** (0.85 + 2.85 * np.sin(ii * 0.11 + seed) * np.cos(jj * 0.13))
           * rng.uniform(0.7, 1.4, size=(ny, nx))).astype(np.float32)
    L.hp, L.hq = synth.pc.pq_depth(L.H)
    L.Z0 = (np.minimum(L.H, 3.0) * 0.5 * 10.0 ** rng.uniform(-7, 0, size=(ny, nx))
            * np.where(rng.uniform(size=(ny, nx)) < 0.5, -1, 1)).astype(np.float32)
    s = ReferenceSession(case, fusion=True)
    try:
        for _ in range(6):
            s.step(maxamp=True)
        got = {"z": s.getz(1), "m": s.getmn(1)[0], "n": s.getmn(1)[1]}
    finally:
        s.close()
    o = oracle_mod.OracleRun(case)
    o.run(6)
    ref = o.layer(0)
    assert np.isfinite(ref["m"]).all()
    for f in ("z", "m", "n"):
        _same(got[f], ref[f], f)


@pytest.mark.parametrize("rel_time", [3, 4, 5])
@pytest.mark.parametrize("laygov", [0, 1])
@pytest.mark.parametrize("graphs", [0, 1])
def test_outer_window_beside_later_sub_steps(oracle_mod, rel_time, laygov, graphs):
    """sub-steps after the feedback run beside the outer window's momentum and
    outputs; gauges on the child are sampled after the last one"""
    from comcot_b200.engine import Engine
    case = synth.nested_case("w", 97, 81, 2.0, 2.0, [60, 79, 30, 49], 3, 30, seed=9, rel_time=rel_time,
                             child_laygov=laygov, ngauges=2)
    P, C = case.layers
    _steep(C, 6, 0.5)
    case.gauges += [(C.id, 12, 20, 0.4, 0.7), (C.id, 40, 33, 0.1, 0.2), (P.id, 64, 35, 0.3, 0.6)]
    with Engine(budget=2 << 30) as eng:
        eng.config(variant=-1, use_graphs=graphs, chunk=8)
        mid = eng.add(case)
        eng.step(32)
        got = eng.read(mid)
    o = oracle_mod.OracleRun(case)
    ts = o.run(case.nsteps)
    ref, rc = o.layer(0), o.layer(1)
    for f in ("z", "m", "n"):
        _same(got[f], ref[f], f)
        _same(got["child_" + f], rc[f], "child " + f)
    _same(got["zmax"], ref["zmax"], "zmax")
    _same(got["ts"], ts, "gauges")
    assert np.array_equal(got["arrival"], ref["arrival"])
