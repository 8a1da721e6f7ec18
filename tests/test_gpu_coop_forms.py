"""Which form of the FP64 solve runs (pm_coop.cu), and what follows when an
exchange between its CTAs does not complete."""
import ctypes

import numpy as np
import pytest

import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu

TOL = 1e-11
PHASES, WARP_PER_NODE, NODE_PAIRS = 0, 1, 2


def _mesh(kind, n):
    if kind == "column":
        pb = meshgen.column_problem(nx=1, ny=1, nz=n, lz=float(n))
    else:
        pb = meshgen.tetra_problem(n=n) if kind == "tetra" else meshgen.cube_problem(n=n)
    m = pg.from_problem(pb)
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    return m, np.random.default_rng(n).standard_normal(m.neq)


def _form(m):
    t = np.zeros(9)
    assert m.lib.pm_get_timers(m.h, ctypes.c_void_p(t.ctypes.data), 9) == 0
    return int(t[8])


def _solve(m, b, solver):
    return m.solve(b, solver=solver, precond=2, tol=TOL, maxit=20000)[0]


# nodes with a free dof, and per SM of 152: 20, 69, 4,741 (31.2: the last cube with a warp
# per node), 4,705 (31.0), 6,216 (40.9: the first cube with pairs), 8,941 (58.8, odd: the
# last pair has one node), 15,136 (58 k panel values per SM), 18,241 (70 k: the kernels
# per phase)
@pytest.mark.parametrize("solver", [1, 11])
@pytest.mark.parametrize("kind,n,form", [
    ("column", 1, WARP_PER_NODE), ("cube", 2, WARP_PER_NODE), ("cube", 10, WARP_PER_NODE),
    ("tetra", 8, WARP_PER_NODE), ("cube", 11, NODE_PAIRS), ("tetra", 10, NODE_PAIRS),
    ("cube", 15, NODE_PAIRS), ("cube", 16, PHASES)])
def test_form_and_solution(kind, n, form, solver, monkeypatch):
    """The form the size asks for ran, and its solution is the phase kernels' within
    1e4 tol, the bar of the solver parity tests."""
    m, b = _mesh(kind, n)
    x = _solve(m, b, solver)
    assert _form(m) == form
    monkeypatch.setenv("PM_POLLED_GRAPHS", "1")
    xp = _solve(m, b, solver)
    assert _form(m) == PHASES
    assert np.abs(x - xp).max() <= 1e4 * TOL * np.abs(xp).max()


def test_form_of_other_solves():
    m, b = _mesh("cube", 3)
    _solve(m, b, 1)
    assert _form(m) == WARP_PER_NODE
    m.solve(b, solver=7, precond=5, tol=1e-8, maxit=20000)
    assert _form(m) == PHASES
    m.set_precision(pg.capi.PM_FP32C_REFINE)
    _solve(m, b, 1)
    assert _form(m) == PHASES


# no poll at all: every CTA leaves at its first exchange; one: those that find all sums
# there go on until they miss one
@pytest.mark.parametrize("polls", ["0", "1"])
@pytest.mark.parametrize("solver", [1, 11])
@pytest.mark.parametrize("n", [3, 11])
def test_an_exchange_that_does_not_complete(n, solver, polls, monkeypatch):
    """The host solves again from the start with the phase kernels: their solution to
    the bit, at once and in later solves of the handle, and a new handle is not
    affected."""
    m, b = _mesh("cube", n)
    with monkeypatch.context() as mp:
        mp.setenv("PM_POLLED_GRAPHS", "1")
        ref = _solve(m, b, solver)
    m, b = _mesh("cube", n)
    with monkeypatch.context() as mp:
        mp.setenv("PM_COOP_POLLS", polls)
        x = _solve(m, b, solver)
    assert _form(m) == PHASES
    assert np.array_equal(x, ref)
    assert np.array_equal(_solve(m, b, solver), ref) and _form(m) == PHASES
    m2, _ = _mesh("cube", n)
    x2 = _solve(m2, b, solver)
    assert _form(m2) != PHASES
    assert np.abs(x2 - ref).max() <= 1e4 * TOL * np.abs(ref).max()
