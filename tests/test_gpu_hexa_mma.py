"""The hexa20 element matrices summed on the FP16 tensor pipe (pm_hexa_mma.h):
distorted, flat and widely scaled elements, one element and many, against the
oracle, and values that are not finite."""
import numpy as np
import pytest

import oracle
import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _problem(n, jitter, scale, seed):
    """A cube mesh with moved vertices (the geometry is the vertices'), stretched
    per axis, and materials over several decades."""
    pb = meshgen.cube_problem(n=max(n, 2)) if n > 1 else meshgen.column_problem(1, 1, 1, lz=1.0)
    rng = np.random.default_rng(seed)
    pb["x"] = (pb["x"] + jitter / max(n, 1) * rng.uniform(-1, 1, pb["x"].shape)) * np.asarray(scale)
    e = np.atleast_2d(np.array(pb["e"], float))
    e[:, 0] *= 10.0 ** rng.uniform(-3, 3, len(e))
    e[:, 2] *= 10.0 ** rng.uniform(-4, 4, len(e))
    pb["e"] = e
    return pb


@pytest.mark.parametrize("n,jitter,scale", [
    (1, 0.0, (1, 1, 1)), (1, 0.2, (1, 1, 1)), (2, 0.15, (1, 1, 1)), (3, 0.1, (1, 1, 0.01)),
    (3, 0.1, (300.0, 1, 0.02)), (4, 0.2, (1e3, 1e3, 1e3)), (5, 0.1, (1e-3, 2e-3, 1e-3))])
def test_element_matrices_against_the_oracle(n, jitter, scale):
    """K, scaled by its diagonal, within 2e-14 of the oracle's (its 64-term sums
    round at about 64 x 2^-53 = 7e-15 of the diagonal), and the product of the
    same launch within the matching bound."""
    pb = _problem(n, jitter, scale, 11 + n)
    m, o = pg.from_problem(pb), oracle.from_fixture(pb)
    u = np.random.default_rng(5).standard_normal((m.nnode, 4))
    b = m.pform(2, True, True, u, np.zeros(m.neq))
    bo = np.zeros(o.neq)
    o.pform(2, True, True, u, bo)
    ia, ja, ad, al = m.get_csrd()
    _, _, ado, alo = o.get_csrd()
    rows = np.repeat(np.arange(m.neq), np.diff(ia))
    d = np.sqrt(np.abs(ado))
    assert np.all(np.abs(ad - ado) <= 2e-14 * np.abs(ado))
    assert np.all(np.abs(al - alo) <= 2e-14 * d[rows] * d[ja - 1] +
                  2e-14 * np.abs(alo))
    # |K| |u| bounds the product's rounding; u also holds restrained dofs, whose
    # columns are outside K, so the element-wise scale is the larger of the two
    scale_b = np.abs(bo).max()
    assert np.abs(b - bo).max() <= 1e-12 * scale_b


def test_not_finite_and_inverted():
    """An inverted element is refused, a displacement that is not a number
    reaches the product, and the panels repeat bit for bit."""
    pb = meshgen.cube_problem(n=2)
    bad = dict(pb)
    bad["x"] = pb["x"].copy()
    bad["x"][:, 2] *= -1.0
    m = pg.from_problem(bad)
    with pytest.raises(pg.PMError) as e:
        m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    assert e.value.status == 2
    m = pg.from_problem(pb)
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    _, _, ad, _ = m.get_csrd()
    assert np.all(np.isfinite(ad)) and np.all(ad != 0)
    u = np.zeros((m.nnode, 4))
    u[3, 0] = np.nan
    b = m.pform(2, True, True, u, np.zeros(m.neq))
    assert np.isnan(b).any()
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    assert np.array_equal(m.get_csrd()[2], ad)
