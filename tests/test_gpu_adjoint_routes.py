"""The adjoint's sweeps by different routes: a tape that the cooperative kernels recorded is reversed one cell
per lane and the other way round (the forward and the reverse sweep have limits of their own), with
the same states and gradients of every cell bit for bit."""
import numpy as np
import pytest

from cmaq_gb300.synthetic import make_grid, solver_inputs

pytestmark = pytest.mark.gpu


def window(mech, cells, forward, reverse, tape_bytes):
    import torch
    from cmaq_gb300.adjoint import Ros3Window
    from cmaq_gb300.chem import ChemSolver
    g = make_grid(mech, cells, 1, 1, seed=83, het=True)
    with ChemSolver(mech, ncols=cells, nrows=1, nlays=1, nspcsd=g.nspcsd, cgrid_index=g.cgrid_index, rtol=1e-3,
                    atol=1e-9) as s:
        y0, rki, night = solver_inputs(g, s)
        w = Ros3Window(s, rki, night, 2, 5.0, tape_bytes=tape_bytes)
        x = [y0.clone().requires_grad_(True),
             torch.zeros(rki.shape[0], dtype=torch.float64, device="cuda", requires_grad=True),
             torch.full_like(y0, 1e-7).requires_grad_(True)]
        s.set_tuning(adjoint_coop=forward)
        y = w(*x)
        s.set_tuning(adjoint_coop=reverse)
        gy, gk, ge = torch.autograd.grad(y.sum(), x)
        return [v.detach().cpu().numpy() for v in (y, gy, ge, gk)]


@pytest.mark.parametrize("tape_bytes", [None, 0])
@pytest.mark.parametrize("mech,cells", [("cb6r5_ae7_aq", 157), ("cracmm2", 35)])
def test_one_route_forward_the_other_back(mech, cells, tape_bytes):
    lanes = window(mech, cells, 0, 0, tape_bytes)
    for forward, reverse in ((1, 0), (0, 1)):
        got = window(mech, cells, forward, reverse, tape_bytes)
        for a, b in zip(got[:3], lanes[:3]):
            assert np.array_equal(a, b)
        # sums over the cells, in another order: the largest gradient stands for the sum of magnitudes
        assert np.max(np.abs(got[3] - lanes[3])) <= 1e-10 * np.max(np.abs(lanes[3]))


def test_backward_when_the_tape_fills_the_memory():
    """A backward call that takes the one-cell-per-lane kernels on a handle that has not taken them before, with so
    much memory free that its tape fits alone but not beside their workspaces (1.8 GB): the tape gives way."""
    import torch
    from cmaq_gb300.adjoint import Ros3Window
    from cmaq_gb300.chem import ChemSolver
    mech, cells = "cb6r5_ae7_aq", 70000
    window(mech, 33, 0, 0, 0)                  # the kernels' own memory
    g = make_grid(mech, cells, 1, 1, seed=84)
    got = []
    for room in (None, 900 << 20):
        with ChemSolver(mech, ncols=cells, nrows=1, nlays=1, nspcsd=g.nspcsd, cgrid_index=g.cgrid_index, rtol=1e-3,
                        atol=1e-9) as s:
            y0, rki, night = solver_inputs(g, s)
            w = Ros3Window(s, rki, night, 1, 5.0, tape_bytes=0)
            x = y0.clone().requires_grad_(True)
            s.set_tuning(adjoint_coop=1)
            y = w(x)
            s.set_tuning(adjoint_coop=0)
            held = None
            if room is not None:
                tape = int(y.grad_fn.saved_tensors[1].sum()) * (s.info.ischan + 1) * 8
                assert tape > 1800 << 20       # so that half of it and the workspaces fit
                torch.cuda.empty_cache()
                held = torch.empty(torch.cuda.mem_get_info()[0] - tape - room, dtype=torch.uint8, device="cuda")
            try:
                got.append(torch.autograd.grad(y.sum(), x)[0].cpu().numpy())
            finally:
                del held
                torch.cuda.empty_cache()       # for the tests that follow
    assert np.array_equal(got[0], got[1])
