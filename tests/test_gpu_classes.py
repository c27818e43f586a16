"""Kernels compiled for a range of matrix sizes m = species + 1 (to 32, 33 .. 64,
65 .. 128, any) at the edges of the ranges, on a B200: solves that mix mechanisms
of every range in one launch, the Jacobian, and the gradient, whose transposed
solves have two, four or ten rows per lane. Oracle and tolerances are those of the
tests of the same quantities (tests/parity.py, tests/test_adjoint.py)."""
import numpy as np
import pytest

from gpufoam_b200 import adjoint as AD
from gpufoam_b200 import evaluator as E
from gpufoam_b200 import mechanism as M
from oracle.complex_step import ComplexStepMap
from oracle.oracle import Oracle, ode_inputs
from tests.parity import (assert_jacobian_close, assert_rates_close, assert_states_close, jacobian_scale, rate_scale,
                          step_count_agreement)
from tests.test_adjoint import Case
from tests.test_gpu_edges import filled

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    from gpufoam_b200 import build
    build.build()
    assert torch.cuda.is_available()
    return torch


def mechanism(n_species):
    """A mechanism of n_species with about two reactions per species, of every reversible rate type."""
    n = min(n_species, 14) if n_species < 20 else 2 * n_species
    return M.make_mechanism(n_species, n, max(2, n // 8), max(2, n // 10), seed=n_species)


@pytest.mark.parametrize("sizes", [(15, 31, 32, 63), (64, 100, 127), (128, 12, 40)])
@pytest.mark.parametrize("threads", [32, 64, 256])
def test_mixed_sizes(torch, sizes, threads):
    raws = [mechanism(s) for s in sizes]
    nS = max(r.n_species for r in raws)
    per, ld = 9, nS + 2
    Y = np.zeros((per * len(raws), ld))
    mid = np.zeros(per * len(raws), dtype=np.int32)
    for k, raw in enumerate(raws):
        Y[k * per:(k + 1) * per, :raw.n_eqns] = M.make_cells(raw, per, seed=30 + k)
        mid[k * per:(k + 1) * per] = k
    order = np.random.default_rng(31).permutation(len(Y))
    s = E.Solver([E.Mechanism(r) for r in raws], E.OdeInputs("Rosenbrock34", absTol=1e-8, relTol=1e-4))
    s.set_launch(kind=1, threads_per_cell=threads, scratch_in_shared=1)
    dtc = torch.full((len(Y),), 1e-7, dtype=torch.float64, device="cuda")
    out = s.solve(torch.as_tensor(Y[order], device="cuda"), 1e-6, dtc,
                  mech_id=torch.as_tensor(mid[order], device="cuda"))
    got = {k: np.empty_like(out[k].cpu().numpy()) for k in ("Ynew", "status", "counters")}
    for k in got:
        got[k][order] = out[k].cpu().numpy()
    for k, raw in enumerate(raws):
        rows = slice(k * per, (k + 1) * per)
        ref = Oracle(raw, "port").cells(ode_inputs(34), np.ascontiguousarray(Y[rows, :raw.n_eqns]), 1e-6, 1e-7)
        assert np.array_equal(got["status"][rows], ref[3]), raw.n_species
        ok = ref[3] == 0
        assert_states_close(got["Ynew"][rows, :raw.n_eqns][ok], ref[0][ok], raw.n_species, 1e-4, f"{raw.n_species} species")
        assert step_count_agreement(got["counters"][rows], ref[2]) >= 0.99, raw.n_species


@pytest.mark.parametrize("sizes", [(12,), (15, 31), (32,), (40, 63), (64,), (100, 127), (128,)])
def test_one_range(torch, sizes):
    """Launches whose mechanisms are all of one range, with the forms that have a kernel for it; more cells
    than are resident, so that a warp per cell takes the kernel with fewer registers."""
    raws = [mechanism(s) for s in sizes]
    nS = max(r.n_species for r in raws)
    n, few, ld = (20000 if nS <= 31 else 300), 24, nS + 2
    solver = E.Solver([E.Mechanism(r) for r in raws], E.OdeInputs("Rosenbrock23", absTol=1e-8, relTol=1e-4))
    Y, mid = np.zeros((n, ld)), (np.arange(n) % len(raws)).astype(np.int32)
    ref = []
    for k, raw in enumerate(raws):
        cells = M.make_cells(raw, few, seed=33 + k)
        Y[mid == k, :raw.n_eqns] = cells[np.arange((mid == k).sum()) % few]
        ref.append(Oracle(raw, "port").cells(ode_inputs(23), cells, 1e-6, 1e-7))
    for form in (dict(threads_per_cell=32), dict(threads_per_cell=32, cells_per_block=1, lu_panel=4),
                 dict(threads_per_cell=64), dict(threads_per_cell=128), dict(threads_per_cell=256)):
        solver.set_launch(kind=1, scratch_in_shared=1, **form)
        dtc = torch.full((n,), 1e-7, dtype=torch.float64, device="cuda")
        out = {k: v.cpu().numpy() for k, v in solver.solve(torch.as_tensor(Y, device="cuda"), 1e-6, dtc,
               mech_id=torch.as_tensor(mid, device="cuda")).items() if k in ("Ynew", "status", "counters")}
        for k, raw in enumerate(raws):
            at = np.arange((mid == k).sum()) % few
            got = {name: v[mid == k] for name, v in out.items()}
            assert np.array_equal(got["status"], ref[k][3][at]), form
            ok = got["status"] == 0
            assert_states_close(got["Ynew"][ok, :raw.n_eqns], ref[k][0][at][ok], raw.n_species, 1e-4, str(form))
            assert step_count_agreement(got["counters"], ref[k][2][at]) >= 0.99, form


@pytest.mark.parametrize("n_species", [12, 31, 32, 63, 64, 127, 128])
def test_jacobian_sizes(torch, n_species):
    raw = mechanism(n_species)
    y = M.make_cells(raw, 3, seed=32)
    dfdx, J = E.jacobian(E.Mechanism(raw), y)
    ref_f, ref_J = Oracle(raw, "port").jacobian(y)
    assert_rates_close(dfdx.cpu().numpy(), ref_f, rate_scale(raw, y))
    assert_jacobian_close(J.cpu().numpy(), ref_J, jacobian_scale(raw, y))


@pytest.mark.parametrize("n_species, solver", [(15, 34), (31, 23), (32, 34), (63, 34), (64, 23), (100, 34), (127, 12),
                                               (128, 34), (135, 23)])
def test_gradient_sizes(torch, n_species, solver):
    """The gradient along a random direction of all states and one of all rate parameters against the
    tangent-linear map in complex arithmetic, and the recorded integration against the oracle's replay."""
    raw = mechanism(n_species)
    case = Case(raw, 2, 2e-7 if solver == 12 else 1e-6, solver, seed=40 + n_species)
    for c in range(case.n):
        np.testing.assert_allclose(case.orc.replay(case.inp, case.cells[c], case.steps[c]), case.Y1[c], rtol=1e-10,
                                   atol=1e-14)
    d = case.rng.standard_normal(case.cells.shape) * (np.abs(case.cells) + 1e-6)
    d[:, raw.n_species + 1] = 0.0
    cs, th0 = ComplexStepMap(raw, solver), AD.parameters_of(raw)
    tl = sum(float(np.dot(case.w[c], cs.directional(case.cells[c], case.steps[c], th0, dy=d[c]))) for c in range(2))
    ad = float(np.sum(case.Y0bar * d))
    assert abs(ad - tl) <= 1e-5 * abs(tl), ("states", ad, tl)
    dth = case.rng.standard_normal(th0.shape) * np.maximum(np.abs(th0), 1.0)
    tl = sum(float(np.dot(case.w[c], cs.directional(case.cells[c], case.steps[c], th0, dtheta=dth))) for c in range(2))
    ad = float(np.sum(case.thb * dth))
    assert abs(ad - tl) <= 1e-5 * abs(tl), ("parameters", ad, tl)


@pytest.mark.parametrize("n_species, n_reactions", [(15, 18), (25, 1300), (40, 98), (40, 1300)])
def test_recorded_forms(torch, n_species, n_reactions):
    """The recorded solve with a warp, 64 threads and, for long lists of reactions, 128 threads per cell."""
    raw = mechanism(n_species)
    raw.reactions = [raw.reactions[k % raw.n_reactions] for k in range(n_reactions)]
    adj = AD.AdjointSolver(raw, E.OdeInputs("Rosenbrock34", absTol=1e-8, relTol=1e-4), traj_cap=256)
    few, n = 12, 2400   # more cells than are resident
    cells = M.make_cells(raw, few, seed=61)
    ref = Oracle(raw, "port").cells(ode_inputs(34), cells, 1e-7, 1e-8)
    at = np.arange(n) % few
    Y1, status, _ = adj.forward(torch.as_tensor(cells[at], device="cuda"), 1e-7,
                                torch.full((n,), 1e-8, dtype=torch.float64, device="cuda"))
    assert np.array_equal(status.cpu().numpy(), ref[3][at])
    ok = status.cpu().numpy() == 0
    assert ok.any()
    assert_states_close(Y1.cpu().numpy()[ok], ref[0][at][ok], n_species, 1e-4)


@pytest.mark.parametrize("n_species, n_reactions, threads, shared", [
    (31, 75, 32, 1), (31, 500, 64, 1), (25, 1300, 128, 1), (40, 98, 64, 1), (64, 156, 64, 1), (80, 194, 128, 1),
    (100, 245, 128, 1), (127, 310, 256, 1), (135, 329, 256, 1), (160, 390, 64, 0)])
def test_default_form(torch, n_species, n_reactions, threads, shared):
    """The default launch form by the number of workspaces that an SM's shared memory holds: eight, four, two, one,
    none."""
    raw = mechanism(n_species)
    raw.reactions = [raw.reactions[k % raw.n_reactions] for k in range(n_reactions)]
    s = E.Solver([E.Mechanism(raw)], E.OdeInputs("Rosenbrock34", absTol=1e-8, relTol=1e-4))
    cfg = s.get_launch()
    assert (cfg["threads_per_cell"], cfg["scratch_in_shared"], cfg["specialize"]) == (threads, shared, 0)
    n = 6
    cells = M.make_cells(raw, n, seed=60)
    ref = Oracle(raw, "port").cells(ode_inputs(34), cells, 1e-7, 1e-8)
    dtc = torch.full((n,), 1e-8, dtype=torch.float64, device="cuda")
    out = s.solve(torch.as_tensor(cells, device="cuda"), 1e-7, dtc)
    assert np.array_equal(out["status"].cpu().numpy(), ref[3])
    ok = ref[3] == 0
    assert_states_close(out["Ynew"].cpu().numpy()[ok], ref[0][ok], n_species, 1e-4)
    assert step_count_agreement(out["counters"].cpu().numpy(), ref[2]) >= 0.99


def filled_workspace(factory, doubles):
    """A mechanism whose solve workspace is `doubles` long (and the mechanism's own check of that)."""
    raw = factory(0)
    nS, m = raw.n_species, raw.n_species + 1
    raw = filled(raw, doubles - (m * (m | 1) + 11 * m + nS + 1 + nS + 1) + 2 * nS)
    mech = E.Mechanism(raw)
    solver = E.Solver([mech], E.OdeInputs("Rosenbrock34", absTol=1e-8, relTol=1e-4))
    assert solver.workspace_doubles() == doubles
    return raw, mech, solver


def test_workspaces_that_just_fit(torch):
    """Workspaces that fill a block's 227 KB but for the 64 bytes that a group's reductions take at
    least: every number of threads takes them, as do the recorded solve and the Jacobian."""
    raw, mech, solver = filled_workspace(M.gri_size, (227 * 1024 - 64) // 8 - 6)
    n, dT = 3, 1e-8
    cells = M.make_cells(raw, n, seed=50)
    ref = Oracle(raw, "port").cells(ode_inputs(34), cells, dT, 1e-9)
    assert (ref[3] == 0).all()
    forms = [None] + [dict(threads_per_cell=G, register_budget=r) for G in (32, 64, 96, 128, 256) for r in (0, 1)]
    for f in forms:
        if f is not None:
            solver.set_launch(kind=1, scratch_in_shared=1, **f)
        dtc = torch.full((n,), 1e-9, dtype=torch.float64, device="cuda")
        out = solver.solve(torch.as_tensor(cells, device="cuda"), dT, dtc)
        assert np.array_equal(out["status"].cpu().numpy(), ref[3]), f
        assert_states_close(out["Ynew"].cpu().numpy(), ref[0], raw.n_species, 1e-4, str(f))
    adj = AD.AdjointSolver(raw, E.OdeInputs("Rosenbrock34", absTol=1e-8, relTol=1e-4), traj_cap=64)
    Y1, status, _ = adj.forward(torch.as_tensor(cells, device="cuda"), dT,
                                torch.full((n,), 1e-9, dtype=torch.float64, device="cuda"))
    assert (status.cpu().numpy() == 0).all()
    assert_states_close(Y1.cpu().numpy(), ref[0], raw.n_species, 1e-4, "recorded")
    # the Jacobian needs no reductions beside the workspace: one warp takes eight doubles more
    raw, mech, _ = filled_workspace(M.gri_size, 227 * 1024 // 8 - 6)
    dfdx, J = E.jacobian(mech, cells)
    ref_f, ref_J = Oracle(raw, "port").jacobian(cells)
    assert_rates_close(dfdx.cpu().numpy(), ref_f, rate_scale(raw, cells))
    assert_jacobian_close(J.cpu().numpy(), ref_J, jacobian_scale(raw, cells))
