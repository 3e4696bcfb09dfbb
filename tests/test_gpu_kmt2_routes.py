"""KMT2 by each of its routes (every cell in a lane to its end, every cell in a warp, lanes with the last cells handed
over): state, fixed species, outputs and counters bit for bit, with cells whose set-up fails, and the
lanes' against the oracle."""
import ctypes as C

import numpy as np
import pytest

from cmaq_gb300.synthetic import make_cloud_cells, make_cloud_columns

pytestmark = pytest.mark.gpu
LANES, COOP, HAND_OVER = 0, 1, 2


def up(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a.T)).cuda()


def workspace(n, lanes):
    import torch
    from cmaq_gb300 import _lib
    lanes = min(n, lanes or _lib.lib().cmaqchem_kmt2_default_lanes(0))
    return torch.empty(_lib.lib().cmaqchem_kmt2_workspace_doubles(lanes), dtype=torch.float64, device="cuda")


def kinetics(route, p, v, lanes=None):
    import torch
    from cmaq_gb300 import _lib
    n, p, v, ws = len(p), up(p), up(v), workspace(len(p), lanes)
    var, fix = (torch.empty((r, n), dtype=torch.float64, device="cuda") for r in (161, 4))
    st = torch.zeros((10, n), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _lib.check(_lib.lib().cmaqchem_diag_kmt2_solve(route, n, *(C.c_void_p(t.data_ptr()) for t in (p, v, var, fix, st, ws)),
                                                   ws.numel(), None))
    return [t.cpu().numpy() for t in (var, fix, st)]


def whole(route, p, g, a, index, factors, lanes=None):
    import torch
    from cmaq_gb300 import _lib
    n, p, g, a, ws = len(p), up(p), up(g), up(a), workspace(len(p), lanes)
    gw, aw = torch.empty_like(g), torch.empty_like(a)
    out = torch.empty((10, n), dtype=torch.float64, device="cuda")
    st = torch.zeros((10, n), dtype=torch.int32, device="cuda")
    idx, fac = np.ascontiguousarray(index, np.int32), np.ascontiguousarray(factors, np.float64)
    torch.cuda.synchronize()
    ptr = lambda t: C.c_void_p(t.data_ptr())
    _lib.check(_lib.lib().cmaqchem_diag_aqchem(route, n, ptr(p), ptr(g), ptr(a), a.shape[0] // 3,
                                               C.c_void_p(idx.ctypes.data), C.c_void_p(fac.ctypes.data),
                                               *(ptr(t) for t in (gw, aw, out, st, ws)), ws.numel(), None))
    return [t.cpu().numpy() for t in (g, a, gw, aw, out, st)]


def same(a, b):
    assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


@pytest.mark.parametrize("n,lanes,ispc8,mtpyrac", [(1, None, 0, 0), (37, 32, 1, 0), (1217, 96, 0, 1), (20000, None, 1, 1)])
def test_kinetics(n, lanes, ispc8, mtpyrac):
    p, v = make_cloud_cells(n, seed=45, ispc8=ispc8, mtpyrac=mtpyrac)
    if n > 30:
        p[5, 0], p[n - 1, 6] = -1.0, 0.0       # MET DATA ERROR
    a = kinetics(LANES, p, v, lanes)
    assert (a[2][8] < 0).sum() == (2 if n > 30 else 0)
    for route in (COOP, HAND_OVER, -1):
        same(kinetics(route, p, v, lanes), a)


@pytest.mark.parametrize("n,lanes,ispc8", [(1, None, 0), (333, 64, 1), (20000, None, 0)])
def test_aqchem(n, lanes, ispc8):
    p, g, a, index, factors = make_cloud_columns(n, seed=46, ispc8=ispc8, mtpyrac=1)
    if n > 30:
        p[7, 1] = 0.0
    want = whole(LANES, p, g, a, index, factors, lanes)
    for route in (COOP, HAND_OVER, -1):
        same(whole(route, p, g, a, index, factors, lanes), want)


def test_lanes_equal_the_oracle():
    from kmt2 import KMT2Oracle
    o = KMT2Oracle()
    p, v = o.synthetic_cells(64, seed=47)
    var, _, st = kinetics(LANES, p, v)
    want, _, counts, failed = o.cells(p, v)
    assert failed == 0 and np.array_equal(var.T, want) and np.array_equal(st.T, counts)


def test_unknown_routes_are_refused():
    from cmaq_gb300 import _lib
    p, v = make_cloud_cells(3, seed=48)
    for route in (-2, 3):
        with pytest.raises(_lib.ChemError):
            kinetics(route, p, v)
