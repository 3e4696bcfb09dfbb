"""The one-cell-per-lane ROS3 kernels (work queue and static schedule) by themselves: the cooperative kernel
takes small calls and the last cells of larger ones by default, so both are switched off here
(ros3_coop = 0, ros3_hand_over = 0), and the lane kernels are compared with the oracle, over their
launch shapes, on chunked host arrays and from a graph.  The cooperative kernel and the hand-over
are then compared with them."""
import numpy as np
import pytest

from cmaq_gb300.synthetic import make_grid
from helpers import rel_err

pytestmark = pytest.mark.gpu
FIELDS = ("conc", "ta", "qv", "dens", "pres", "seaice", "ocean_szone", "rj", "khetero")
CB6, CRACMM = "cb6r5_ae7_aq", "cracmm2"
LANES = dict(ros3_coop=0, ros3_hand_over=0)
RTOL, ATOL = float(np.float32(1e-3)), float(np.float32(1e-9))


def solver(g, schedule="queue", **kw):
    from cmaq_gb300.chem import ChemSolver
    return ChemSolver(g.mech, ncols=g.ncols, nrows=g.nrows, nlays=g.nlays, nspcsd=g.nspcsd, cgrid_index=g.cgrid_index,
                      rtol=1e-3, atol=1e-9, schedule=schedule, **kw)


def run(g, knobs, schedule="queue", calls=2, host=False, ddm=False, replayed=0, **kw):
    """Concentrations, sensitivities, per-cell status and attempts and the calls' totals."""
    import torch
    t = [np.ascontiguousarray(getattr(g, k)).copy() for k in FIELDS]
    if not host:
        t = [torch.from_numpy(a).cuda() for a in t]
    with solver(g, schedule, **kw) as s:
        s.set_tuning(**knobs)
        st = [s.steps(replayed, *t)] if replayed else [s.step(*t) for _ in range(calls)]
        sen = None
        if ddm:
            sen = torch.zeros((g.nspcsd, 2, *g.ta.shape), dtype=torch.float32, device="cuda")
            row = int(g.cgrid_index[0]) - 1
            sen[row, 0] = t[0][row]
            mask = torch.zeros((2, s.info.nrxns), dtype=torch.uint8, device="cuda")
            mask[1, 5] = 1
            st.append(s.step_ddm(sen, *t, rate_mask=mask))
            sen = sen.cpu().numpy()
        status, attempts = s.cell_stats()
    for q in st:
        q.pop("device_ms", None)
    return t[0] if host else t[0].cpu().numpy(), sen, status, attempts, st


def same(a, b):
    assert all(np.array_equal(x, y) for x, y in zip(a[:4], b[:4])) and a[4] == b[4]


@pytest.mark.parametrize("schedule", ["queue", "static"])
@pytest.mark.parametrize("mech,dims,dark", [(CB6, (12, 10, 5), False), (CB6, (33, 1, 1), False), (CB6, (8, 4, 2), True),
                                            (CRACMM, (9, 7, 2), False)])
def test_lane_kernels_match_the_oracle(mech, dims, dark, schedule):
    from oracle import Oracle
    g = make_grid(mech, *dims, seed=91, het=True, seawater_fraction=0.3, sza_range=(95.0, 100.0) if dark else (0.0, 100.0))
    conc, _, status, _, st = run(g, LANES, schedule, calls=1)
    ref, tot = Oracle(mech).chem(g, blksize=1, rtol=RTOL, atol=ATOL, threads=4)
    assert tot["rc"] == 0 and not status.any()
    assert (st[0]["accepted_steps"], st[0]["rejected_steps"]) == (tot["nsteps"], tot["nfails"])
    assert rel_err(conc, ref) < 1e-5
    if not dark:
        same(run(g, LANES, schedule, calls=1), run(g, LANES, "static" if schedule == "queue" else "queue", calls=1))


SHAPES = [(8, 0), (8, 1), (8, 2), (4, 1), (4, 2), (2, 1), (2, 2)]


@pytest.mark.parametrize("mech,dims", [(CB6, (37, 29, 2)), (CRACMM, (31, 17, 1))])
def test_launch_shapes_and_the_hand_over(mech, dims):
    """Every launch shape, without and with the hand-over, by calls, with sensitivities and with cells that
    reach the cap on their attempts."""
    g = make_grid(mech, *dims, seed=92, het=True, plume_fraction=0.2)
    for kw in (dict(ddm=True), dict(calls=1, max_iter=40)):
        a = run(g, LANES, **kw)
        assert kw.get("max_iter") is None or 0 < a[4][0]["failed_cells"] < g.ncell
        for warps, lockstep in SHAPES:
            shape = dict(block_warps=warps, lockstep=lockstep)
            same(run(g, {**LANES, **shape}, **kw), a)
            for most in (-1, 1) if lockstep else ():
                same(run(g, {**LANES, **shape, "ros3_hand_over": most}, **kw), a)


@pytest.mark.parametrize("mech,dims", [(CB6, (1, 1, 1)), (CB6, (153, 1, 1)), (CB6, (1217, 1, 1)), (CRACMM, (1, 1, 1)),
                                       (CRACMM, (13, 59, 1))])
def test_cooperative_kernel(mech, dims):
    g = make_grid(mech, *dims, seed=93, het=True, plume_fraction=0.2)
    for kw in (dict(ddm=True), dict(calls=1, max_iter=40), dict(replayed=3, ddm=True)):
        same(run(g, dict(ros3_coop=1), **kw), run(g, LANES, **kw))


@pytest.mark.parametrize("chunks", [1, 3, 16])
def test_host_arrays_and_graphs(chunks):
    g = make_grid(CB6, 12, 10, 5, seed=94, het=True)
    a = run(g, LANES)
    b = run(g, {**LANES, "host_chunks": chunks}, host=True)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[3], b[3])
    assert [x["accepted_steps"] for x in a[4]] == [x["accepted_steps"] for x in b[4]]
    c = run(g, LANES, replayed=2)
    assert np.array_equal(a[0], c[0]) and np.array_equal(a[3], c[3])


def test_a_call_above_the_cooperative_limit():
    """By size: the work queue with its hand-over, against each kernel by itself and a host call in chunks."""
    g = make_grid(CB6, 60, 60, 15, seed=95, het=True, plume_fraction=0.1)
    a = run(g, LANES)
    same(run(g, {}), a)
    same(run(g, dict(ros3_coop=1)), a)
    b = run(g, {}, host=True)
    assert np.array_equal(a[0], b[0]) and np.array_equal(a[3], b[3])
