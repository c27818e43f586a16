"""The kernels at the sizes where their paths change, on a B200.

* the factorisation by register panels and matrix tiles (32 or more threads,
  m <= 128) and the blocked solves, at the edges of panels, tiles, lanes and of
  the range, against the one-thread blocked form (itself pinned to the reference's
  factors by test_gpu_lu_forms.py): bit for bit, ties and a zero column included;
* calculate() / tc() with a lane per cell (8,192 cells and more) against the
  oracle and against the warp-per-cell form, ragged last tiles included;
* reactions that the compact record does not hold (non-integer exponents,
  exponent 3, four species on a side, a third-body row past 4,094);
* rates clipped by the reaction temperature limits, which the Jacobian does not clip;
* the default launch form of every range of its rule;
* Qdot on ragged cell counts and padded rows.

Tolerances are those of the tests of the same quantities (tests/parity.py).
"""
import copy
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from gpufoam_b200 import evaluator as E
from gpufoam_b200 import mechanism as M
from oracle.oracle import Oracle, ode_inputs
from tests.parity import (assert_jacobian_close, assert_rates_close, assert_states_close, jacobian_scale, rate_scale,
                          step_count_agreement)
from tests.test_gpu_fields import species_scale
from tests.test_oracle import fixture_mech, load

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    import torch
    from gpufoam_b200 import build
    build.build()
    assert torch.cuda.is_available()
    return torch


def lu_cases(m):
    rng = np.random.default_rng(m)
    A = rng.standard_normal((4, m, m))
    A[1] *= 10.0 ** rng.uniform(-8, 8, (m, 1))                 # rows of very different size
    A[2] = rng.integers(-2, 3, (m, m)) + 3.0 * np.eye(m)       # exact ties of the pivot rule
    A[3, :, m // 2] = 0.0                                      # the zero pivot's replacement
    return A, rng.standard_normal((4, 2, m))


@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 15, 16, 17, 24, 31, 32, 33, 40, 48, 56, 63, 64, 65, 72, 96, 127, 128, 129, 160])
@pytest.mark.parametrize("exact", [True, False])
def test_lu_edges(torch, m, exact):
    A, b = lu_cases(m)
    LU1, piv1, x1 = (t.cpu().numpy() for t in E.lu_factor_solve(A, b, 1, exact))
    for G in (32, 64, 96, 128, 256):
        LU, piv, x = (t.cpu().numpy() for t in E.lu_factor_solve(A, b, G, exact))
        assert np.array_equal(piv, piv1), (m, G)
        assert np.array_equal(LU, LU1), (m, G)
        ok = [0, 2] if m > 1 else [0]
        scale = np.abs(x1[ok]).max(axis=2, keepdims=True)
        cond = np.array([np.linalg.cond(A[k]) for k in ok])[:, None, None]
        assert (np.abs(x - x1)[ok] <= 1e-14 * m * np.maximum(cond, 1.0) * scale).all(), (m, G)


LANE_MECHS = {
    "gri": lambda: fixture_mech(load("grisize")),
    "coverage": lambda: fixture_mech(load("coverage")),   # fractional exponents, irreversible, Lindemann
    "yao": lambda: fixture_mech(load("foam_yao")),        # exponent 3, four species on a side
}


@pytest.mark.parametrize("name", list(LANE_MECHS))
@pytest.mark.parametrize("n", [8192, 8192 + 37])
def test_lane_per_cell_rates(torch, name, n):
    raw = LANE_MECHS[name]()
    mech = E.Mechanism(raw)
    y = M.make_cells(raw, n, seed=5)
    rho = np.random.default_rng(6).uniform(0.05, 2.0, n)
    RR, tc = (t.cpu().numpy() for t in E.cell_rates(mech, rho, y))
    pick = np.r_[0:40, n - 70:n]
    o = Oracle(raw, "port")
    ref_RR, ref_tc = o.cell_fields(rho[pick], y[pick])
    sc = species_scale(raw, o.rate_parts(rho[pick], y[pick]))
    assert (np.abs(RR[pick] - ref_RR) <= 1e-12 * sc + 1e-300).all()
    assert np.allclose(tc[pick], ref_tc, rtol=1e-12, atol=0)
    RRw, tcw = (t.cpu().numpy() for t in E.cell_rates(mech, rho[pick], y[pick]))   # a warp per cell
    assert (np.abs(RR[pick] - RRw) <= 2e-12 * sc + 1e-300).all()
    assert np.allclose(tc[pick], tcw, rtol=2e-12, atol=0)


def test_third_body_rows_past_the_record(torch):
    """4,200 third-body reactions: the rows past 4,094 are not in the compact record."""
    raw = M.coverage(0)
    tb = [r for r in raw.reactions if r.rate_type == M.RATE_THIRD_BODY]
    raw = copy.deepcopy(raw)
    raw.reactions = raw.reactions + [copy.deepcopy(tb[i % len(tb)]) for i in range(4200)]
    rng = np.random.default_rng(7)
    for r in raw.reactions[-200:]:
        r.efficiencies = rng.uniform(0.5, 12.0, raw.n_species)
    mech = E.Mechanism(raw)
    n = 8192
    y = M.make_cells(raw, n, seed=8)
    rho = rng.uniform(0.05, 2.0, n)
    RR, tc = (t.cpu().numpy() for t in E.cell_rates(mech, rho, y))
    o = Oracle(raw, "port")
    ref_RR, ref_tc = o.cell_fields(rho[-8:], y[-8:])
    sc = species_scale(raw, o.rate_parts(rho[-8:], y[-8:]))
    assert (np.abs(RR[-8:] - ref_RR) <= 1e-12 * sc + 1e-300).all()
    assert np.allclose(tc[-8:], ref_tc, rtol=1e-12, atol=0)


@pytest.mark.parametrize("limits", [(0.0, 1500.0), (1600.0, 3000.0)])
def test_clipped_rates(torch, limits):
    raw = M.make_mechanism(12, 14, 3, 2, seed=0, n_lindemann=2, n_irreversible=3, n_fractional=2, rxn_Tlow=limits[0],
                           rxn_Thigh=limits[1])
    mech = E.Mechanism(raw)
    y = M.make_cells(raw, 24, seed=9, T_range=(1200.0, 2200.0))
    o = Oracle(raw, "port")
    assert_rates_close(E.rates(mech, y).cpu().numpy(), o.derivatives(y), rate_scale(raw, y))
    dfdx, J = E.jacobian(mech, y)
    ref_f, ref_J = o.jacobian(y)
    assert_rates_close(dfdx.cpu().numpy(), ref_f, rate_scale(raw, y))
    assert_jacobian_close(J.cpu().numpy(), ref_J, jacobian_scale(raw, y))
    ref = o.cells(ode_inputs(34), y, 1e-6, 1e-7)
    s = E.Solver([mech], E.OdeInputs("Rosenbrock34", absTol=1e-8, relTol=1e-4))
    dtc = torch.full((24,), 1e-7, dtype=torch.float64, device="cuda")
    out = s.solve(torch.as_tensor(y, device="cuda"), 1e-6, dtc)
    assert np.array_equal(out["status"].cpu().numpy(), ref[3])
    assert_states_close(out["Ynew"].cpu().numpy(), ref[0], raw.n_species, 1e-4)
    assert step_count_agreement(out["counters"].cpu().numpy(), ref[2]) >= 0.99


DEFAULTS = [(M.h2_size, 32, 1), (M.coverage, 32, 0), (M.gri_size, 128, 1), (M.large, 256, 0)]


@pytest.mark.parametrize("factory, threads, specialize", DEFAULTS)
def test_default_launch(torch, factory, threads, specialize):
    raw = factory(0)
    s = E.Solver([E.Mechanism(raw)], E.OdeInputs("Rosenbrock34", absTol=1e-8, relTol=1e-4))
    cfg = s.get_launch()
    assert cfg["kind"] == 1 and cfg["threads_per_cell"] == threads and cfg["specialize"] == specialize
    n = 37
    cells = M.make_cells(raw, n, seed=10)
    dT = 1e-5 if raw.n_species <= 12 else 1e-6
    ref = Oracle(raw, "port").cells(ode_inputs(34), cells, dT, 1e-7)
    dtc = torch.full((n,), 1e-7, dtype=torch.float64, device="cuda")
    out = s.solve(torch.as_tensor(cells, device="cuda"), dT, dtc)
    st = out["status"].cpu().numpy()
    assert np.array_equal(st, ref[3])
    ok = st == 0
    assert_states_close(out["Ynew"].cpu().numpy()[ok], ref[0][ok], raw.n_species, 1e-4)
    assert step_count_agreement(out["counters"].cpu().numpy(), ref[2]) >= 0.99


def test_jacobian_of_100_species(torch):
    raw = M.large(0)
    y = M.make_cells(raw, 2, seed=11)
    dfdx, J = E.jacobian(E.Mechanism(raw), y)
    ref_f, ref_J = Oracle(raw, "port").jacobian(y)
    assert_rates_close(dfdx.cpu().numpy(), ref_f, rate_scale(raw, y))
    assert_jacobian_close(J.cpu().numpy(), ref_J, jacobian_scale(raw, y))


@pytest.mark.parametrize("n, pad", [(1, 0), (31, 3), (32, 0), (33, 1), (129, 0), (4099, 2)])
@pytest.mark.parametrize("factory", [M.h2_size, M.gri_size, M.large])
def test_qdot_ragged(torch, factory, n, pad):
    raw = factory(0)
    mech = E.Mechanism(raw)
    RR = np.random.default_rng(n).standard_normal((n, raw.n_species + pad))
    q = np.zeros(n)
    hf = -E.qdot(mech, np.eye(raw.n_species)).cpu().numpy()   # one species at a time: 0 - hf_i
    for i in range(raw.n_species):
        q = q - hf[i] * RR[:, i]
    assert np.array_equal(E.qdot(mech, RR).cpu().numpy(), q)


@pytest.mark.parametrize("solver", [12, 23, 34])
def test_one_species(torch, solver):
    """One species, A -> 1.05 A (no net zero to hide behind): a group of 64 or more threads
    splits the Jacobian row's single column into an empty part and the rest."""
    a = np.array([[3.5, 1e-3, -2e-7, 1e-11, 0.0, -3e4, 4.0]])
    raw = M.RawMechanism("one-species", ["A"], np.array([1.0]), np.array([200.0]), np.array([5000.0]),
                         np.array([1000.0]), a, a, [M.RawReaction(M.RATE_ARRHENIUS, True, [(0, 1.0, 1.0)],
                                                                  [(0, 1.05, 1.0)], 1e6, 0.5, 9e3)])
    n = 16
    cells = M.make_cells(raw, n, seed=12, T_range=(1200.0, 2200.0))
    ref = Oracle(raw, "port").cells(ode_inputs(solver), cells, 1e-6, 1e-8)
    s = E.Solver([E.Mechanism(raw)], E.OdeInputs(f"Rosenbrock{solver}", absTol=1e-8, relTol=1e-4))
    for G in (8, 32, 64, 96, 128, 256):
        s.set_launch(kind=1, threads_per_cell=G, scratch_in_shared=1)
        dtc = torch.full((n,), 1e-8, dtype=torch.float64, device="cuda")
        out = s.solve(torch.as_tensor(cells, device="cuda"), 1e-6, dtc)
        assert np.array_equal(out["status"].cpu().numpy(), ref[3]), G
        assert np.array_equal(out["counters"].cpu().numpy(), ref[2]), G
        # the same steps: rounding only, amplified at most by the steps' number and a stiffness of order one
        assert np.allclose(out["Ynew"].cpu().numpy(), ref[0], rtol=1e-10, atol=0), G


HAMMER = r"""
#include <atomic>
#include <thread>
#include "gpufoam_b200.h"
// two host threads, each launching for its own number of species; the number of refused launches
extern "C" int hammer(const double* const* fields, double* const* out, const double* T, double* y, int n, int loops,
                      const int* sizes, const gf_mech* const* mechs, double* q) {
    std::atomic<int> refused{0};
    auto work = [&](int k) {
        for (int i = 0; i < loops; ++i) {
            refused += gf_gather_states(n, sizes[k], fields, T, T, y, sizes[k] + 2, nullptr) != GF_OK;
            refused += gf_scatter_rates(n, sizes[k], y, sizes[k], out, nullptr) != GF_OK;
            refused += gf_qdot(mechs[k], n, y, 100, q, nullptr) != GF_OK;
        }
    };
    std::thread a(work, 0), b(work, 1);
    a.join();
    b.join();
    return refused;
}
"""


def test_host_threads_with_different_sizes(torch, tmp_path):
    """The shared memory that one host thread's launches ask for is not taken away by those of
    another with fewer species (64 cells a launch: the threads meet between setting and launching)."""
    from gpufoam_b200 import _native as N
    src, lib = tmp_path / "hammer.cpp", tmp_path / "libhammer.so"
    src.write_text(HAMMER)
    pkg = os.path.dirname(N.LIB_PATH)
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-pthread", "-I",
                    os.path.join(os.path.dirname(pkg), "include"), "-o", str(lib), str(src), "-L", pkg,
                    "-lgpufoam_b200", f"-Wl,-rpath,{pkg}"], check=True, capture_output=True)
    n, sizes = 64, (300, 200)
    cols = torch.zeros((300, n), dtype=torch.float64, device="cuda")
    out = torch.zeros((300, n), dtype=torch.float64, device="cuda")
    y = torch.zeros((n, 302), dtype=torch.float64, device="cuda")
    q = torch.zeros(n, dtype=torch.float64, device="cuda")
    mechs = [E.Mechanism(M.large(0)), E.Mechanism(M.gri_size(0))]
    ptrs = lambda t: (C.c_void_p * 300)(*[t[i].data_ptr() for i in range(300)])  # noqa: E731
    torch.cuda.synchronize()
    refused = C.CDLL(str(lib)).hammer(ptrs(cols), ptrs(out), C.c_void_p(cols.data_ptr()), C.c_void_p(y.data_ptr()),
                                      n, 4000, (C.c_int * 2)(*sizes), (C.c_void_p * 2)(*[m.handle.value for m in mechs]),
                                      C.c_void_p(q.data_ptr()))
    torch.cuda.synchronize()
    assert refused == 0


def filled(raw, doubles):
    """raw with its reactions repeated until a cell of calculate() takes `doubles` of shared memory:
    the staging slots, twice the species, the third-body sums."""
    raw = copy.deepcopy(raw)
    cost = lambda r: (2 + len(r.lhs) + len(r.rhs) + (r.rate_type == M.RATE_THIRD_BODY)  # noqa: E731
                      + (r.rate_type != M.RATE_ARRHENIUS))
    base = list(raw.reactions)
    left = doubles - 2 * raw.n_species - sum(cost(r) for r in base)
    small, large = (next(r for r in base if cost(r) == k) for k in (5, 6))
    k = 0
    while left > 60:
        raw.reactions.append(copy.deepcopy(base[k % len(base)]))
        left -= cost(base[k % len(base)])
        k += 1
    n6 = left % 5
    for r in [large] * n6 + [small] * ((left - 6 * n6) // 5):
        raw.reactions.append(copy.deepcopy(r))
    assert 2 * raw.n_species + sum(cost(r) for r in raw.reactions) == doubles
    return raw


@pytest.mark.parametrize("factory", [M.h2_size, M.coverage, M.gri_size])
@pytest.mark.parametrize("less", [0, 1, 2])
def test_rates_that_just_fit(torch, factory, less):
    """As many reactions as a block's 227 KB of shared memory hold: a warp per cell takes them, and the
    places that a cell uses twice do not meet. Also every single-reaction rate of a few reactions."""
    raw = filled(factory(0), 227 * 1024 // 8 - less)
    mech = E.Mechanism(raw)
    n = 5
    y = M.make_cells(raw, n, seed=14)
    rho = np.random.default_rng(15).uniform(0.05, 2.0, n)
    o = Oracle(raw, "port")
    ref_RR, ref_tc = o.cell_fields(rho, y)
    parts = o.rate_parts(rho, y)
    RR, tc = (t.cpu().numpy() for t in E.cell_rates(mech, rho, y))
    assert (np.abs(RR - ref_RR) <= 1e-12 * species_scale(raw, parts) + 1e-300).all()
    assert np.allclose(tc, ref_tc, rtol=1e-12, atol=0)
    for r in (0, 7, raw.n_reactions - 1):
        om, RR1 = (t.cpu().numpy() for t in E.reaction_rates(mech, r, rho, y))
        ref_om, ref_RR1 = o.reaction_fields(r, rho, y)
        gross = np.abs(parts[:, r]).sum(axis=1)
        assert (np.abs(om - ref_om) <= 1e-12 * gross + 1e-300).all(), r
        sc = np.zeros((n, raw.n_species))
        for i, st, _ in raw.reactions[r].lhs + raw.reactions[r].rhs:
            sc[:, i] += abs(st) * gross * raw.W[i]
        assert (np.abs(RR1 - ref_RR1) <= 1e-12 * sc + 1e-300).all(), r


@pytest.mark.parametrize("name", list(LANE_MECHS))
def test_single_reaction_rates(torch, name):
    """reactionRR / specieReactionRR of every reaction against the port, general reactions included."""
    raw = LANE_MECHS[name]()
    mech = E.Mechanism(raw)
    n = 9
    y = M.make_cells(raw, n, seed=16)
    rho = np.random.default_rng(17).uniform(0.05, 2.0, n)
    o = Oracle(raw, "port")
    parts = o.rate_parts(rho, y)
    for r, rx in enumerate(raw.reactions):
        om, RR = (t.cpu().numpy() for t in E.reaction_rates(mech, r, rho, y))
        ref_om, ref_RR = o.reaction_fields(r, rho, y)
        gross = np.abs(parts[:, r]).sum(axis=1)
        assert (np.abs(om - ref_om) <= 1e-12 * gross + 1e-300).all(), r
        sc = np.zeros((n, raw.n_species))
        for i, st, _ in rx.lhs + rx.rhs:
            sc[:, i] += abs(st) * gross * raw.W[i]
        assert (np.abs(RR - ref_RR) <= 1e-12 * sc + 1e-300).all(), r


def widened(raw, n_species):
    """raw with copies of its species (before the last, inert one); every other reaction takes the copies."""
    raw = copy.deepcopy(raw)
    b, k = raw.n_species, n_species - raw.n_species
    assert 0 <= k < b
    ix = np.r_[0:b - 1, np.arange(k), b - 1]
    raw.species = [raw.species[i] + ("" if j < b - 1 or j == n_species - 1 else "_copy") for j, i in enumerate(ix)]
    for f in ("W", "Tlow", "Thigh", "Tcommon", "high_raw", "low_raw"):
        setattr(raw, f, getattr(raw, f)[ix])
    for j, r in enumerate(raw.reactions):
        if r.efficiencies is not None:
            r.efficiencies = r.efficiencies[ix]
        move = lambda i: n_species - 1 if i == b - 1 else (b - 1 + i if j % 2 and i < k else i)  # noqa: E731
        r.lhs = [(move(i), st, e) for i, st, e in r.lhs]
        r.rhs = [(move(i), st, e) for i, st, e in r.rhs]
    return raw


@pytest.mark.parametrize("n_species", [144, 145, 300])
def test_rates_of_many_species(torch, n_species):
    """calculate() and tc() on 8,192 + 5 cells where the lane-per-cell form has two warps (144 species)
    and where a warp per cell takes over, to the largest number of species."""
    raw = widened(M.make_mechanism(min(n_species, 151), 300, 60, 40, seed=1), n_species)
    mech = E.Mechanism(raw)
    n = 8192 + 5
    y = M.make_cells(raw, n, seed=18)
    rho = np.random.default_rng(19).uniform(0.05, 2.0, n)
    RR, tc = (t.cpu().numpy() for t in E.cell_rates(mech, rho, y))
    pick = np.r_[0:33, n - 9:n]
    o = Oracle(raw, "port")
    ref_RR, ref_tc = o.cell_fields(rho[pick], y[pick])
    sc = species_scale(raw, o.rate_parts(rho[pick], y[pick]))
    assert (np.abs(RR[pick] - ref_RR) <= 1e-12 * sc + 1e-300).all()
    assert np.allclose(tc[pick], ref_tc, rtol=1e-12, atol=0)
