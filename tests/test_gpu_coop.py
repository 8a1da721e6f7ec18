"""The cooperative FP64 PCG / rpsqmr solve (pm_coop.cu) at the edges of its
forms: fewer nodes than schedulers, the last mesh with a warp per node and the
first with two nodes per warp, and the last and first side of the limit above
which the phase kernels solve."""
import threading

import numpy as np
import pytest

import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _mesh(kind, n):
    if kind == "column":
        pb = meshgen.column_problem(nx=1, ny=1, nz=n, lz=float(n))
    else:
        pb = meshgen.tetra_problem(n=n) if kind == "tetra" else meshgen.cube_problem(n=n)
    m = pg.from_problem(pb)
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    return pb, m


def _product(m):
    import scipy.sparse as sp
    ia, ja, ad, al = m.get_csrd()
    L = sp.csr_matrix((al, ja - 1, ia - 1), shape=(m.neq, m.neq))
    return ad, lambda x: ad * x + L @ x + L.T @ x


# nodes: 20, 81, 3,700 (23 active ones per SM), 4,961 (31), 18,785 (120); panel values
# 10.6 M (16^3) and 12.7 M (17^3), above the 152 x 65,000 of the cooperative solve
@pytest.mark.parametrize("solver", [1, 11])
@pytest.mark.parametrize("kind,n", [("column", 1), ("cube", 2), ("cube", 9), ("cube", 10),
                                    ("tetra", 4), ("cube", 16), ("cube", 17)])
def test_solve_meets_its_own_test(kind, n, solver):
    """The solver's stopping test re-evaluated on the CPU with the exported
    matrix: within 1.1 tol (the recursive residual may drift from the true
    one), and the phase kernels' solution within 1e4 tol, the bar of the solver
    parity tests."""
    pb, m = _mesh(kind, n)
    b = np.random.default_rng(n).standard_normal(m.neq)
    x, info = m.solve(b, solver=solver, precond=2, tol=TOL, maxit=20000)
    ad, mul = _product(m)
    r = b - mul(x)
    w = np.ones_like(ad) if solver == 11 else 1.0 / ad
    assert np.sqrt(abs(np.sum(r * r * w))) <= 1.1 * TOL * np.sqrt(abs(np.sum(b * b * w)))
    assert info.iters == m.timers()[6]
    x2, info2 = m.solve(b, solver=solver, precond=2, tol=TOL, maxit=20000)
    assert np.array_equal(x, x2) and info2.iters == info.iters


@pytest.mark.parametrize("solver", [1, 11])
@pytest.mark.parametrize("kind,n", [("cube", 3), ("tetra", 6), ("cube", 11)])
def test_matches_the_phase_kernels(kind, n, solver, monkeypatch):
    pb, m = _mesh(kind, n)
    b = np.random.default_rng(7).standard_normal(m.neq)
    x, info = m.solve(b, solver=solver, precond=2, tol=TOL, maxit=20000)
    monkeypatch.setenv("PM_POLLED_GRAPHS", "1")
    xp, ip = m.solve(b, solver=solver, precond=2, tol=TOL, maxit=20000)
    assert np.abs(x - xp).max() <= 1e4 * TOL * np.abs(xp).max()
    if solver == 1:  # rpsqmr's count moves by 8 % with a relative change of 1e-15 in b
        assert abs(info.iters - ip.iters) <= 0.03 * ip.iters + 2


@pytest.mark.parametrize("n", [4, 11])
def test_limits_and_breakdown(n):
    """maxit reached and a non-finite right-hand side give the solver's
    status, and the handle solves again."""
    pb, m = _mesh("cube", n)
    b = np.random.default_rng(3).standard_normal(m.neq)
    with pytest.raises(pg.PMError) as e:
        m.solve(b, solver=1, precond=2, tol=TOL, maxit=7)
    assert e.value.status == 4 and "7 iterations" in str(e.value)
    bad = b.copy()
    bad[m.neq // 2] = np.nan
    for solver in (1, 11):
        with pytest.raises(pg.PMError) as e:
            m.solve(bad, solver=solver, precond=2, tol=TOL, maxit=500)
        assert e.value.status == 4
    x, info = m.solve(b, solver=1, precond=2, tol=TOL, maxit=20000)
    ad, mul = _product(m)
    r = b - mul(x)
    assert np.sqrt(abs(np.sum(r * r / ad))) <= 1.1 * TOL * np.sqrt(abs(np.sum(b * b / ad)))


def test_two_handles_in_two_threads():
    """Two host threads solve on their own handles at the same time: each gets
    the solution it gets alone."""
    pairs = [_mesh("cube", 5), _mesh("cube", 9)]
    rhs = [np.random.default_rng(k).standard_normal(m.neq) for k, (_, m) in enumerate(pairs)]
    alone = [m.solve(b, solver=1, precond=2, tol=TOL, maxit=20000)[0]
             for (_, m), b in zip(pairs, rhs)]
    got = [[], []]

    def work(k):
        for _ in range(10):
            got[k].append(pairs[k][1].solve(rhs[k], solver=1, precond=2, tol=TOL, maxit=20000)[0])

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for k in range(2):
        assert len(got[k]) == 10 and all(np.array_equal(x, alone[k]) for x in got[k])
