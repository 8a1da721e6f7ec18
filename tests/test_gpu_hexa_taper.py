"""The hexa20 element matrix of strongly tapered elements: the digit sums of
pm_hexa_mma.h hold each derivative at the scale of its own row, so an element whose
thickness changes by orders of magnitude is as accurate as with FP64 sums."""
import numpy as np
import pytest

import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu

# quadrature digits as the reference types them (Elmlib.f:3780-3962)
_X4 = (-.861136311594053, -.339981043584856, .339981043584856, .861136311594053)
_W4 = (.347854845137454, .652145154862546, .652145154862546, .347854845137454)
_NODE = np.array([(1, 1, 1), (-1, 1, 1), (-1, -1, 1), (1, -1, 1), (1, 1, -1), (-1, 1, -1),
                  (-1, -1, -1), (1, -1, -1), (0, 1, 1), (-1, 0, 1), (0, -1, 1), (1, 0, 1),
                  (0, 1, -1), (-1, 0, -1), (0, -1, -1), (1, 0, -1), (1, 1, 0), (-1, 1, 0),
                  (-1, -1, 0), (1, -1, 0)])


def _matrix(X, e, grav, dt, T):
    """K_e (60 displacements node by node, 8 pressures) in arithmetic T."""
    x, w = np.array(_X4, T), np.array(_W4, T)
    pts = np.array([(x[i], x[j], x[k]) for k in range(4) for j in range(4) for i in range(4)], T)
    W = np.array([w[i] * w[j] * w[k] for k in range(4) for j in range(4) for i in range(4)], T)
    hp, dl, dq = np.zeros((64, 8), T), np.zeros((64, 8, 3), T), np.zeros((64, 20, 3), T)
    for k, c in enumerate(_NODE.astype(T)):
        f, q = 1 + pts * c, 1 - pts * pts
        for d in range(3):
            a, b = (d + 1) % 3, (d + 2) % 3
            if k < 8:
                hp[:, k] = f[:, 0] * f[:, 1] * f[:, 2] / 8
                dl[:, k, d] = c[d] * f[:, a] * f[:, b] / 8
                dq[:, k, d] = c[d] * f[:, a] * f[:, b] * (
                    pts[:, 0] * c[0] + pts[:, 1] * c[1] + pts[:, 2] * c[2] - 1 +
                    pts[:, d] * c[d]) / 8
            else:
                g = np.where(c == 0, q, f)
                dq[:, k, d] = (-2 * pts[:, d] if c[d] == 0 else c[d]) * g[:, a] * g[:, b] / 4
    J = np.einsum("gki,kj->gij", dl, X.astype(T))
    co = np.zeros_like(J)  # cofactors: co[a][j] of dx_j / dr_a
    for a in range(3):
        for j in range(3):
            p, q, s, t = (a + 1) % 3, (a + 2) % 3, (j + 1) % 3, (j + 2) % 3
            co[:, a, j] = J[:, p, s] * J[:, q, t] - J[:, p, t] * J[:, q, s]
    det = (J[:, 0] * co[:, 0]).sum(1)
    inv = co / det[:, None, None]
    W = W * det
    gp, gq = np.einsum("gaj,gka->gkj", inv, dl), np.einsum("gaj,gka->gkj", inv, dq)
    E, nu = T(e[0]), T(e[1])
    a, b = E * (1 - nu) / ((1 + nu) * (1 - 2 * nu)), nu / (1 - nu)
    c = T(0.5) * (1 - 2 * nu) / (1 - nu)
    fd = T(e[6]) * T(1e-6)
    perm = T(e[2]) / (fd * np.sqrt((grav.astype(T) ** 2).sum()))
    P = np.einsum("gik,gjl->ikjl", W[:, None, None] * gq, gq)
    tr = np.einsum("ikjk->ij", P)
    K = np.zeros((68, 68), T)
    Kuu = np.zeros((20, 3, 20, 3), T)
    for k in range(3):
        for m in range(3):
            Kuu[:, k, :, m] = (a * (P[:, k, :, k] + c * (tr - P[:, k, :, k])) if k == m else
                               a * (b * P[:, k, :, m] + c * P[:, m, :, k]))
    Kpu = -T(e[4]) * np.einsum("gl,gjk->ljk", W[:, None] * hp, gq).reshape(8, 60)
    K[:60, :60], K[60:, :60], K[:60, 60:] = Kuu.reshape(60, 60), Kpu, Kpu.T
    K[60:, 60:] = -(np.einsum("gl,gm->lm", W[:, None] * hp, hp) / T(e[3]) +
                    T(dt) * perm * np.einsum("glk,gmk->lm", W[:, None, None] * gp, gp))
    return K


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
    exact = _matrix(*args, np.longdouble)
    d = np.sqrt(np.abs(np.diag(exact)))
    err = [np.asarray((K - exact) / np.outer(d, d), float) for K in
           (_gpu_matrix(pb), _matrix(*args, np.float64))]
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
