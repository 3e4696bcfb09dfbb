"""The cooperative KMT2 kernels (csrc/kmt2_coop.cuh) against the one-cell-per-lane kernels: the
same operations in the same order, so state, fixed species, outputs and counters must agree
bit for bit, at one cell, around the device's cells, with cells whose set-up fails and for
the ISPC8 / MTPYRAC switches.  A call above the size that the cooperative kernels take is
made of copies of the same cells."""
import numpy as np
import pytest

from cmaq_gb300.synthetic import make_cloud_cells, make_cloud_columns

pytestmark = pytest.mark.gpu
MANY = 40000         # above the cooperative kernels' range


def up(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


@pytest.mark.parametrize("n,ispc8,mtpyrac", [(1, 0, 0), (37, 1, 0), (1217, 0, 1)])
def test_kinetics_same_bits_as_one_cell_per_lane(n, ispc8, mtpyrac):
    from cmaq_gb300.aqchem import aqchem_kinetics
    p, v = make_cloud_cells(n, seed=41, ispc8=ispc8, mtpyrac=mtpyrac)
    if n > 30:
        p[5, 0] = -1.0                      # MET DATA ERROR
        p[n - 1, 6] = 0.0
    var, fix, st = (x.cpu().numpy() for x in aqchem_kinetics(up(p.T), up(v.T), with_fix=True))
    idx = np.arange(MANY) % n
    var2, fix2, st2 = (x.cpu().numpy()[:, :n] for x in aqchem_kinetics(up(p[idx].T), up(v[idx].T), with_fix=True))
    assert np.array_equal(var, var2, equal_nan=True) and np.array_equal(fix, fix2, equal_nan=True)
    assert np.array_equal(st, st2)
    assert (st[8] < 0).sum() == (2 if n > 30 else 0)


@pytest.mark.parametrize("n,ispc8", [(1, 0), (333, 1)])
def test_aqchem_same_bits_as_one_cell_per_lane(n, ispc8):
    from cmaq_gb300.aqchem import aqchem
    p, g, a, index, fac = make_cloud_columns(n, seed=42, ispc8=ispc8, mtpyrac=1)
    if n > 30:
        p[7, 1] = 0.0
    out = []
    for idx in (np.arange(n), np.arange(MANY) % n):
        gas, aer = up(g[idx].T), up(a[idx].T)
        rest = aqchem(up(p[idx].T), gas, aer, index, fac)
        out.append([x.cpu().numpy()[:, :n] for x in (gas, aer, *rest)])
    for x, y in zip(*out):
        assert np.array_equal(x, y, equal_nan=True)


@pytest.mark.parametrize("copies", [40000, 90001])
def test_cells_that_the_queue_kernel_leaves(copies):
    """The last cells of a call that does not take the cooperative kernels go on there: every copy ends alike."""
    from cmaq_gb300.aqchem import aqchem
    n = 1217
    p, g, a, index, fac = make_cloud_columns(n, seed=43, mtpyrac=1)
    p[11, 1] = 0.0                          # a failed set-up
    out = []
    for idx in (np.arange(n), np.arange(copies) % n):
        gas, aer = up(g[idx].T), up(a[idx].T)
        rest = aqchem(up(p[idx].T), gas, aer, index, fac)
        out.append([x.cpu().numpy() for x in (gas, aer, *rest)])
    for x, y in zip(*out):
        assert np.array_equal(x[:, np.arange(copies) % n], y, equal_nan=True)
