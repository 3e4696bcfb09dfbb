"""The cooperative ROS3 kernel (csrc/coop.cuh) against the one-cell-per-lane kernels: the same
operations in the same order, so every concentration, counter and DDM-3D sensitivity must
agree bit for bit, at one cell, around a block's and the device's cells, for both mechanisms,
with failed cells, and from a captured graph."""
import numpy as np
import pytest

from cmaq_gb300.synthetic import make_grid

pytestmark = pytest.mark.gpu
FIELDS = ("conc", "ta", "qv", "dens", "pres", "seaice", "ocean_szone", "rj", "khetero")


def setup(mech, dims, seed, schedule="queue", **kw):
    import torch
    from cmaq_gb300.chem import ChemSolver
    g = make_grid(mech, *dims, seed=seed, het=True, plume_fraction=0.2)
    t = [torch.from_numpy(np.ascontiguousarray(getattr(g, k))).cuda() for k in FIELDS]
    s = ChemSolver(mech, ncols=g.ncols, nrows=g.nrows, nlays=g.nlays, nspcsd=g.nspcsd, cgrid_index=g.cgrid_index,
                   rtol=1e-3, atol=1e-9, schedule=schedule, **kw)
    return g, t, s


def run(s, t, mode, calls=2):
    s.set_tuning(ros3_coop=mode, queue_history=0)
    conc = t[0].clone()
    st = [s.step(conc, *t[1:]) for _ in range(calls)]
    status, attempts = s.cell_stats()
    for q in st:
        q.pop("device_ms", None)
    return conc.cpu().numpy(), st, status, attempts


def same(a, b):
    assert np.array_equal(a[0], b[0], equal_nan=True)
    assert a[1] == b[1] and np.array_equal(a[2], b[2]) and np.array_equal(a[3], b[3])


@pytest.mark.parametrize("mech,dims", [("cb6r5_ae7_aq", (1, 1, 1)), ("cb6r5_ae7_aq", (11, 7, 2)),
                                       ("cb6r5_ae7_aq", (153, 1, 1)), ("cb6r5_ae7_aq", (19, 32, 2)),
                                       ("cb6r5_ae7_aq", (1217, 1, 1)), ("cracmm2", (1, 1, 1)),
                                       ("cracmm2", (13, 59, 1))])
def test_same_bits_as_one_cell_per_lane(mech, dims):
    _, t, s = setup(mech, dims, seed=31)
    same(run(s, t, 1), run(s, t, 0))


def test_static_schedule_and_the_rule_by_size():
    _, t, s = setup("cb6r5_ae7_aq", (23, 5, 3), seed=32, schedule="static")
    a = run(s, t, 0)
    same(run(s, t, -1), a)      # by size: the cooperative kernel
    same(run(s, t, 1), a)


def test_cells_that_reach_the_attempt_cap():
    _, t, s = setup("cb6r5_ae7_aq", (17, 5, 2), seed=33, max_iter=40)
    a, b = run(s, t, 1, 1), run(s, t, 0, 1)
    assert 0 < a[1][0]["failed_cells"] < 170
    same(a, b)


def test_graph_replay_and_ddm():
    import torch
    g, t, s = setup("cb6r5_ae7_aq", (14, 9, 2), seed=34)
    out = []
    for mode in (1, 0):
        s.set_tuning(ros3_coop=mode, queue_history=0)
        conc = t[0].clone()
        s.steps(3, conc, *t[1:])
        sen = torch.zeros((g.nspcsd, 2, *g.ta.shape), dtype=torch.float32, device="cuda")
        sen[int(g.cgrid_index[0]) - 1, 0] = conc[int(g.cgrid_index[0]) - 1]
        mask = torch.zeros((2, s.info.nrxns), dtype=torch.uint8, device="cuda")
        mask[1, 5] = 1
        s.step_ddm(sen, conc, *t[1:], rate_mask=mask)
        out.append((conc.cpu().numpy(), sen.cpu().numpy()))
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("mech,dims", [("cb6r5_ae7_aq", (1, 1, 1)), ("cb6r5_ae7_aq", (153, 4, 1)),
                                       ("cracmm2", (7, 5, 1))])
def test_ebi_same_bits_as_one_cell_per_lane(mech, dims):
    _, t, s = setup(mech, dims, seed=35, solver="ebi")
    s.set_tuning(ebi_warp=1, ebi_defer=0)
    a = run(s, t, -1)
    s.set_tuning(ebi_warp=0)
    same(run(s, t, -1), a)


def test_ebi_cells_that_reach_the_iteration_cap():
    _, t, s = setup("cb6r5_ae7_aq", (13, 5, 2), seed=36, solver="ebi", max_iter=60)
    s.set_tuning(ebi_warp=1, ebi_defer=0)
    a = run(s, t, -1, 1)
    s.set_tuning(ebi_warp=0)
    assert 0 < a[1][0]["failed_cells"] < 130
    same(run(s, t, -1, 1), a)


@pytest.mark.parametrize("mech,dims", [("cb6r5_ae7_aq", (1, 1, 1)), ("cb6r5_ae7_aq", (13, 4, 2)),
                                       ("cracmm2", (5, 4, 1))])
def test_gear_same_bits_as_one_cell_per_lane(mech, dims):
    _, t, s = setup(mech, dims, seed=37, solver="gear")
    s.set_tuning(gear_warp=1)
    a = run(s, t, -1)
    s.set_tuning(gear_warp=0)
    same(run(s, t, -1), a)


def test_gear_cells_that_reach_the_evaluation_cap():
    _, t, s = setup("cb6r5_ae7_aq", (9, 5, 2), seed=38, solver="gear", max_iter=150)
    s.set_tuning(gear_warp=1)
    a = run(s, t, -1, 1)
    s.set_tuning(gear_warp=0)
    assert 0 < a[1][0]["failed_cells"] < 90
    same(run(s, t, -1, 1), a)


@pytest.mark.parametrize("mech,dims", [("cb6r5_ae7_aq", (1, 1, 1)), ("cb6r5_ae7_aq", (37, 29, 3)), ("cracmm2", (31, 17, 2))])
@pytest.mark.parametrize("most", [1, 64, 255])
def test_cells_handed_over_by_the_work_queue(mech, dims, most):
    _, t, s = setup(mech, dims, seed=34)
    s.set_tuning(ros3_hand_over=0)
    a = run(s, t, 0)
    s.set_tuning(ros3_hand_over=most)
    same(run(s, t, 0), a)


def gradients(s, t, nsync, mode, tape_bytes=None):
    import torch
    from cmaq_gb300.adjoint import Ros3Window
    s.set_tuning(adjoint_coop=mode)
    w = Ros3Window(s, t["rki"], t["night"], nsync, 5.0, tape_bytes=tape_bytes)
    x = [t[k].clone().requires_grad_(True) for k in ("y0", "log_k", "emis")]
    y = w(*x)
    g = torch.autograd.grad(y, x, t["cost"])
    return [v.detach().cpu().numpy() for v in (y, g[0], g[2], g[1])]


@pytest.mark.parametrize("mech,cells,tape,tape_mb", [("cb6r5_ae7_aq", 1, None, 0), ("cb6r5_ae7_aq", 913, None, 0),
                                                     ("cb6r5_ae7_aq", 150, 0, 0), ("cb6r5_ae7_aq", 150, 0, 1),
                                                     ("cracmm2", 457, None, 0)])
def test_adjoint_as_one_cell_per_lane(mech, cells, tape, tape_mb):
    """States and the gradients of a cell bit for bit, with the tape recorded by the forward pass, re-run whole,
    and in batches; the rate gradients, sums over the cells in another order, within 100 roundings of the
    sum of the terms' magnitudes, which the largest gradient stands for up to their cancellation (1e-10)."""
    import torch
    from helpers import gather_cells
    from oracle import Oracle
    from cmaq_gb300.chem import ChemSolver
    g = make_grid(mech=mech, ncols=cells, nrows=1, nlays=1, seed=51, het=True)
    y0, rki, night = gather_cells(g, Oracle(mech))
    rng = np.random.default_rng(7)
    t = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in dict(
        y0=y0, rki=rki, night=night, log_k=0.05 * rng.standard_normal(rki.shape[0]), emis=1e-6 * rng.random(y0.shape),
        cost=rng.standard_normal(y0.shape) / np.maximum(y0, 1e-12)).items()}
    s = ChemSolver(mech, ncols=cells, nrows=1, nlays=1, nspcsd=g.nspcsd, rtol=1e-3, atol=1e-9)
    s.set_tuning(adjoint_tape_mb=tape_mb)
    a, b = gradients(s, t, 2, 1, tape), gradients(s, t, 2, 0, tape)
    for u, v in zip(a[:3], b[:3]):
        assert np.array_equal(u, v)
    assert np.max(np.abs(a[3] - b[3])) <= 1e-10 * np.max(np.abs(b[3]))
