"""The cooperative FP64 solve (pm_coop.cu) on right-hand sides whose inner
products are at the lower end of the doubles."""
import numpy as np
import pytest

import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _assembled(n):
    m = pg.from_problem(meshgen.cube_problem(n=n))
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    return m


# the fused form and the one with two nodes per warp
@pytest.mark.parametrize("solver", [1, 11])
@pytest.mark.parametrize("n", [3, 11])
def test_inner_products_below_the_normal_range(n, solver):
    """b scaled by a power of two until its larger inner product is 1e-300, solved
    to 1e-5: the products end near 1e-310, where the reciprocal of a product is no
    longer a double but the quotient of two is. The stopping test holds for the
    scaled-back solution with the margin of the other solver tests."""
    m = _assembled(n)
    ia, ja, ad, al = m.get_csrd()
    b = np.random.default_rng(n).standard_normal(m.neq)
    s = 2.0 ** np.round(0.5 * np.log2(1e-300 / max(b @ b, abs(np.sum(b * b / ad)))))
    tol = 1e-5
    x, info = m.solve(b * s, solver=solver, precond=2, tol=tol, maxit=20000)
    r = b - m.matvec(x / s)
    w = np.ones_like(ad) if solver == 11 else 1.0 / ad
    assert info.iters > 1
    assert np.sqrt(abs(np.sum(r * r * w))) <= 1.1 * tol * np.sqrt(abs(np.sum(b * b * w)))


def test_tolerance_whose_square_is_no_double():
    """b = A v for an eigenvector v of D^-1 A (D the diagonal of A): PCG's first step
    is exact. Scaled so that (r, z) starts near 1e-318, five digits of a double, it
    ends at 0 and the target, 1e-4 of its root, squares to 0: converged after one
    iteration. A product is some 2e5 units of the smallest double and each of its terms
    is rounded by half of one, so x is within 2 neq / 2 / 2e5 < 2e-3 of v."""
    import scipy.linalg
    m = _assembled(2)
    ia, ja, ad, al = m.get_csrd()
    A = np.diag(ad)
    rows = np.repeat(np.arange(m.neq), np.diff(ia))
    A[rows, ja - 1] = al
    A[ja - 1, rows] = al
    lam, V = scipy.linalg.eig(A / ad[:, None])
    real = np.abs(lam.imag) <= 1e-12 * np.abs(lam)
    V, lam = V.real[:, real], lam.real[real]
    # the eigenvector with the largest (b, D^-1 b) for its entries: no cancellation
    b = A @ V
    k = np.argmax(np.abs(np.sum(b * b / ad[:, None], 0)) / np.sum(b * b / np.abs(ad[:, None]), 0))
    v, b = V[:, k], b[:, k]
    s = 2.0 ** np.round(0.5 * np.log2(1e-318 / abs(np.sum(b * b / ad))))
    x, info = m.solve(b * s, solver=1, precond=2, tol=1e-4, maxit=50)
    assert info.iters == 1
    assert m.neq <= 400
    assert np.abs(x / s - v).max() <= 2e-3 * np.abs(v).max()
