"""The hexa20 element passes by sum factorisation (pm_hexa_sum.h) against the
assembled matrix: isw 2's and isw 4's internal forces, the adjoint's product
and its gradients, on distorted, flat and widely scaled elements."""
import numpy as np
import pytest

import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _problem(n, jitter, scale):
    pb = meshgen.cube_problem(n=n) if n > 1 else meshgen.column_problem(1, 1, 1, lz=1.0)
    rng = np.random.default_rng(17 + n)
    pb["x"] = (pb["x"] + jitter / n * rng.uniform(-1, 1, pb["x"].shape)) * np.asarray(scale)
    e = np.atleast_2d(np.array(pb["e"], float))
    e[:, 0] *= 10.0 ** rng.uniform(-2, 2, len(e))
    e[:, 2] *= 10.0 ** rng.uniform(-3, 3, len(e))
    pb["e"] = e
    return pb


def _dense(m):
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    ia, ja, ad, al = m.get_csrd()
    K = np.diag(ad)
    rows = np.repeat(np.arange(m.neq), np.diff(ia))
    K[rows, ja - 1] = al
    K[ja - 1, rows] = al
    return K


def _dev(a):
    return torch.as_tensor(np.ascontiguousarray(a, np.float64)).cuda()


@pytest.mark.parametrize("n,jitter,scale", [
    (1, 0.0, (1, 1, 1)), (1, 0.2, (1, 1, 1)), (2, 0.15, (1, 1, 1)), (3, 0.1, (1, 1, 0.05)),
    (3, 0.1, (50.0, 1, 0.1)), (4, 0.2, (1e3, 1e3, 1e3)), (5, 0.1, (1e-3, 2e-3, 1e-3))])
def test_against_the_assembled_matrix(n, jitter, scale):
    """Both sides sum some 64 x 20 terms a row, each rounded at 2^-53 = 1.1e-16 of
    itself, over a hundred operations deep at most: 1e-13 of
    sum_j (sqrt(K_ii K_jj) + |K_ij|) |u_j|."""
    pb = _problem(n, jitter, scale)
    m = pg.from_problem(pb)
    pb3 = dict(pb)
    pb3["dt"] = 3.0 * float(pb["dt"])
    m3 = pg.from_problem(pb3)
    K, K3 = _dense(m), _dense(m3)
    m3.close()
    # equations node by node, the pressure on vertex nodes only
    free = np.asarray(pb["id"]).reshape(-1, 4) == 0
    free[:, 3] &= np.asarray(pb["fnno"]) == 1
    eqn = np.cumsum(free.ravel()).reshape(-1, 4) - 1
    rng = np.random.default_rng(3)
    u = rng.standard_normal((m.nnode, 4)) * free
    w = rng.standard_normal((m.nnode, 4)) * free
    dp = rng.standard_normal(m.nnode) * free[:, 3]
    vec = lambda f: np.bincount(eqn[free], f[free], m.neq)  # noqa: E731
    isp = np.zeros(m.neq, bool)
    isp[eqn[:, 3][free[:, 3]]] = True
    d = np.sqrt(np.abs(np.diag(K)))
    G = np.outer(d, d) + np.abs(K)
    Kperm = np.where(np.outer(isp, isp), (K3 - K) / 2, 0.0)

    def check(got, ref, x):
        assert np.all(np.abs(got - ref) <= 1e-13 * (G @ np.abs(x)))

    x = vec(u)
    check(m.pform(2, False, True, u, np.zeros(m.neq)), -K @ x, x)
    # isw 4: the part linear in the state
    z = np.zeros((m.nnode, 4))
    m.set_state(u=z, u0=z, dp=np.zeros(m.nnode))
    b0 = m.pform(4, False, True, z, np.zeros(m.neq))
    m.set_state(u=u, u0=z, dp=dp)
    b4 = m.pform(4, False, True, u, np.zeros(m.neq)) - b0
    f4 = u.copy()
    f4[:, 3] = dp
    xd = vec(f4)
    ref = -np.where(isp, Kperm @ x, K @ xd)
    assert np.all(np.abs(b4 - ref) <= 1e-13 * (G @ (np.abs(x) + np.abs(xd)) + np.abs(b0)))
    # the adjoint's product and gradients
    lam = vec(w)
    mu, nu, gr = _dev(np.zeros(m.neq)), _dev(np.zeros(m.neq)), _dev(np.zeros((m.numel, 3)))
    tl, tu, td = _dev(lam), _dev(u), _dev(f4)
    torch.cuda.synchronize()
    m.adjoint_apply_dev(tl.data_ptr(), mu.data_ptr(), nu.data_ptr())
    m.adjoint_grad_dev(tl.data_ptr(), tu.data_ptr(), td.data_ptr(), gr.data_ptr())
    torch.cuda.synchronize()
    lu = np.where(isp, 0.0, lam)
    check(mu.cpu().numpy(), -np.where(isp, Kperm @ lam, K @ lu), lam)
    check(nu.cpu().numpy(), -np.where(isp, K @ lu, 0.0), lam)
    xu = np.where(isp, 0.0, x)
    bound = 1e-13 * np.abs(lam) @ (G @ np.abs(x))
    gE = gr.cpu().numpy()[:, 0].sum()
    assert abs(gE + lu @ K @ xu) <= bound
    # (K's pp block is perm + storage: the storage is what dt does not scale)
    Kst = np.where(np.outer(isp, isp), K, 0.0) - Kperm
    gM = gr.cpu().numpy()[:, 2].sum()
    assert abs(gM - lam @ Kst @ xd) <= 1e-13 * np.abs(lam) @ (G @ np.abs(xd))
