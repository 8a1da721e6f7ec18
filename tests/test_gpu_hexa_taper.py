"""The hexa20 element matrix of strongly tapered elements: the digit sums of
pm_hexa_mma.h hold each derivative at the scale of its own row, so an element whose
thickness changes by orders of magnitude is as accurate as with FP64 sums."""
import numpy as np
import pytest

import poromec_gb300 as pg
from hexa_blocks import matrix
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu

def _gpu_matrix(pb):
    m = pg.from_problem(pb)
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    ia, ja, ad, al = m.get_csrd()
    A = np.diag(ad)
    rows = np.repeat(np.arange(m.neq), np.diff(ia))
    A[rows, ja - 1] = al
    A[ja - 1, rows] = al
    # equations node by node, all free, the pressure on vertex nodes
    has = np.ones((m.nnode, 4), bool)
    has[:, 3] = np.asarray(pb["fnno"]) == 1
    eq = np.where(has, np.cumsum(has.ravel()).reshape(-1, 4) - 1, -1)
    nd = np.asarray(pb["ix"])[0, :20] - 1
    at = np.concatenate([eq[nd, :3].ravel(), eq[nd[:8], 3]])
    assert m.neq == 68 and np.all(at >= 0)
    return A[np.ix_(at, at)]


def _element(taper, tilt):
    """One element of thickness 1 at one corner and taper at the opposite one."""
    pb = meshgen.column_problem(1, 1, 1, lz=1.0)
    pb["id"] = np.zeros_like(pb["id"])
    x = np.asarray(pb["x"], float).copy()
    r = (x - x.min(0)) / (x.max(0) - x.min(0))
    x = r.copy()
    x[:, 2] = r[:, 2] * taper ** (0.5 * (r[:, 0] + r[:, 1])) + tilt * r[:, 0]
    pb["x"] = x
    return pb


@pytest.mark.parametrize("taper", [0.5, 1e-1, 1e-2, 1e-4, 1e-6])
@pytest.mark.parametrize("tilt", [0.0, 0.3])
def test_as_accurate_as_fp64_sums(taper, tilt):
    """Error against extended precision, each entry by the root of its two diagonal
    ones, no larger than that of plain FP64 sums over the points: both round the
    geometry alike (a quarter for the order of its operations), and the digits' own
    error, 2^-54 of a row's largest value, is below one rounding of an entry."""
    pb = _element(taper, tilt)
    nd = np.asarray(pb["ix"])[0, :8] - 1
    args = (np.asarray(pb["x"])[nd], np.atleast_2d(pb["e"])[0], np.asarray(pb["gravity"], float),
            float(pb["dt"]))
    exact = matrix(*args, np.longdouble)
    d = np.sqrt(np.abs(np.diag(exact)))
    err = [np.asarray((K - exact) / np.outer(d, d), float) for K in
           (_gpu_matrix(pb), matrix(*args, np.float64))]
    rms = [np.sqrt(np.mean(e * e)) for e in err]
    big = [np.abs(e).max() for e in err]
    print("taper %g tilt %g: rms %.2e (FP64 sums %.2e), largest %.2e (%.2e)"
          % (taper, tilt, rms[0], rms[1], big[0], big[1]))
    assert rms[0] <= 1.25 * rms[1] + 2.0 ** -54
    assert big[0] <= 1.25 * big[1] + 2.0 ** -52


def test_values_out_of_range():
    """Edges of 1e105: the determinant overflows, the weights with it. All entries are
    NaN, as sums of infinities by zeros, and the next mesh is not affected."""
    pb = _element(0.5, 0.0)
    good = _gpu_matrix(pb)
    far = dict(pb)
    far["x"] = pb["x"] * 1e105
    assert np.all(np.isnan(_gpu_matrix(far)))
    assert np.array_equal(_gpu_matrix(pb), good)
