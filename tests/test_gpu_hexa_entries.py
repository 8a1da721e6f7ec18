"""The rewritten hexa20 passes entry by entry: the adjoint's gradients of every element
and the assembly's product row by row, each with the bound of its own terms, on meshes
whose elements differ by decades in stiffness and permeability."""
import numpy as np
import pytest

import poromec_gb300 as pg
from hexa_blocks import blocks
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

MESHES = [(1, 0.0, (1, 1, 1)), (2, 0.15, (1, 1, 1)), (3, 0.1, (1, 1, 0.05)),
          (3, 0.1, (50.0, 1, 0.1)), (3, 0.2, (1e3, 1e3, 1e3))]


def _problem(n, jitter, scale):
    pb = meshgen.cube_problem(n=n) if n > 1 else meshgen.column_problem(1, 1, 1, lz=1.0)
    rng = np.random.default_rng(41 + n)
    pb["x"] = (pb["x"] + jitter / n * rng.uniform(-1, 1, pb["x"].shape)) * np.asarray(scale)
    e = np.atleast_2d(np.array(pb["e"], float))
    e[:, 0] *= 10.0 ** rng.uniform(-2, 2, len(e))
    e[:, 2] *= 10.0 ** rng.uniform(-3, 3, len(e))
    pb["e"] = e
    free = np.asarray(pb["id"]).reshape(-1, 4) == 0
    free[:, 3] &= np.asarray(pb["fnno"]) == 1
    eq = np.where(free, np.cumsum(free.ravel()).reshape(-1, 4) - 1, -1)
    return pb, eq


def _elements(pb):
    ix, e, x = np.asarray(pb["ix"]), np.atleast_2d(pb["e"]), np.asarray(pb["x"])
    for k, row in enumerate(ix):
        yield k, row[:20] - 1, blocks(x[row[:8] - 1], e[row[20] - 1],
                                      np.asarray(pb["gravity"], float), float(pb["dt"]),
                                      np.longdouble)


def _scale(A, B, C):
    """sqrt(A_ii C_jj) + |B_ij|: what a product's terms may reach through cancellation."""
    d = np.sqrt(np.outer(np.abs(np.diag(A)), np.abs(np.diag(C))))
    return np.asarray(d + np.abs(B), float)


# 64 x 20 terms an entry, each rounded at 2^-53 = 1.1e-16 of itself, over a hundred
# operations deep at most: 1e-13 of the scales above
TOL = 1e-13


@pytest.mark.parametrize("n,jitter,scale", MESHES)
def test_gradients_of_every_element(n, jitter, scale):
    pb, eq = _problem(n, jitter, scale)
    m = pg.from_problem(pb)
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    rng = np.random.default_rng(3)
    lam = rng.standard_normal(m.neq)
    un, dun = rng.standard_normal((m.nnode, 4)), rng.standard_normal((m.nnode, 4))
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a)).cuda()  # noqa: E731
    tl, tu, td, tg = dev(lam), dev(un), dev(dun), dev(np.zeros((m.numel, 3)))
    torch.cuda.synchronize()
    m.adjoint_grad_dev(tl.data_ptr(), tu.data_ptr(), td.data_ptr(), tg.data_ptr())
    torch.cuda.synchronize()
    got = tg.cpu().numpy()
    lf = np.where(eq >= 0, lam[eq], 0.0)
    for k, nd, (Kuu, Kpu, Kperm, Kstor, Gk, Gabs) in _elements(pb):
        lu, lp = lf[nd, :3].ravel(), lf[nd[:8], 3]
        uu, up, dp = un[nd, :3].ravel(), un[nd[:8], 3], dun[nd[:8], 3]
        ref = [-lu @ Kuu @ uu, -lp @ (Kperm @ up + Gk), lp @ Kstor @ dp]
        top = [np.abs(lu) @ _scale(Kuu, Kuu, Kuu) @ np.abs(uu),
               np.abs(lp) @ (_scale(Kperm, Kperm, Kperm) @ np.abs(up) + Gabs),
               np.abs(lp) @ _scale(Kstor, Kstor, Kstor) @ np.abs(dp)]
        for j in range(3):
            assert abs(got[k, j] - ref[j]) <= TOL * top[j], (k, j)


@pytest.mark.parametrize("n,jitter,scale", MESHES)
def test_product_of_the_assembly_row_by_row(n, jitter, scale):
    """b -= K u of the launch that assembles, restrained columns included."""
    pb, eq = _problem(n, jitter, scale)
    m = pg.from_problem(pb)
    u = np.random.default_rng(5).standard_normal((m.nnode, 4))
    b = m.pform(2, True, True, u, np.zeros(m.neq))
    ref, top = np.zeros(m.neq, np.longdouble), np.zeros(m.neq)
    for _, nd, (Kuu, Kpu, Kperm, Kstor, _, _) in _elements(pb):
        Kpp = Kperm + Kstor
        K = np.block([[Kuu, Kpu.T], [Kpu, Kpp]])
        x = np.concatenate([u[nd, :3].ravel(), u[nd[:8], 3]])
        at = np.concatenate([eq[nd, :3].ravel(), eq[nd[:8], 3]])
        on = at >= 0
        ref[at[on]] -= (K @ x)[on]
        top[at[on]] += (_scale(K, K, K) @ np.abs(x))[on]
    assert np.all(np.abs(b - ref) <= TOL * top)
