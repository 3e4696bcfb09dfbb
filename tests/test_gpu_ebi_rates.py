"""EBI and SMVGEAR calls whose rate constants are not formed in a pass over the call's cells (the arrays did
not fit at set-up, or rconst_pass = 0): the cells that iterate long still go to warps, and
concentrations, counters and sensitivities have the same bits by every route."""
import numpy as np
import pytest

from cmaq_gb300.synthetic import make_grid

pytestmark = pytest.mark.gpu
FIELDS = ("conc", "ta", "qv", "dens", "pres", "seaice", "ocean_szone", "rj", "khetero")


def calls(mech, dims, solver, knobs):
    import torch
    from cmaq_gb300.chem import ChemSolver
    g = make_grid(mech, *dims, seed=81, het=True, plume_fraction=0.2)
    out = []
    for kw in knobs:
        t = [torch.from_numpy(np.ascontiguousarray(getattr(g, k))).cuda() for k in FIELDS]
        with ChemSolver(mech, ncols=g.ncols, nrows=g.nrows, nlays=g.nlays, nspcsd=g.nspcsd, cgrid_index=g.cgrid_index,
                        rtol=1e-3, atol=1e-9, solver=solver) as s:
            s.set_tuning(**kw)
            st = s.step(*t)
            sen = torch.zeros((g.nspcsd, 1, *g.ta.shape), dtype=torch.float32, device="cuda")
            row = int(g.cgrid_index[0]) - 1
            sen[row, 0] = t[0][row]
            st2 = s.step_ddm(sen, *t)
            status, steps = s.cell_stats()
        for q in (st, st2):
            q.pop("device_ms", None)
        out.append((t[0].cpu().numpy(), sen.cpu().numpy(), status, steps, st, st2))
    return out


def same(out):
    for other in out[1:]:
        assert all(np.array_equal(a, b) for a, b in zip(out[0][:4], other[:4])) and out[0][4:] == other[4:]


@pytest.mark.parametrize("mech,dims", [("cb6r5_ae7_aq", (1, 1, 1)), ("cb6r5_ae7_aq", (13, 31, 3)), ("cracmm2", (7, 11, 3))])
def test_ebi_without_the_pass(mech, dims):
    same(calls(mech, dims, "ebi", [dict(rconst_pass=0, ebi_warp=0), dict(rconst_pass=0), dict(rconst_pass=0, ebi_defer=0),
                                   dict(rconst_pass=0, ebi_defer=1), dict(rconst_pass=1)]))


@pytest.mark.parametrize("mech,dims", [("cb6r5_ae7_aq", (5, 4, 3)), ("cracmm2", (5, 4, 1))])
def test_gear_without_the_pass(mech, dims):
    same(calls(mech, dims, "gear", [dict(rconst_pass=0, gear_warp=0), dict(rconst_pass=0), dict(rconst_pass=1)]))
