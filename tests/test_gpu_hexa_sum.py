"""The hexa20 element passes by sum factorisation (pm_hexa_sum.h) against the
assembled matrix: isw 2's and isw 4's internal forces, the adjoint's product
and its gradients, on distorted, flat and widely scaled elements."""
import numpy as np
import pytest

import oracle
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


def _distorted(n, jitter, scale):
    pb = _problem(n, jitter, scale)
    o = oracle.from_fixture(pb)
    rng = np.random.default_rng(23)
    u = 1e-3 * rng.standard_normal((int(pb["nnode"]), 4))
    dp = 1e-3 * rng.standard_normal(int(pb["nnode"]))
    return pb, o, pg.from_problem(pb), u, dp


@pytest.mark.parametrize("n,jitter,scale", [(1, 0.2, (1, 1, 1)), (2, 0.15, (1, 1, 0.1)),
                                            (3, 0.1, (1, 1, 1))])
def test_vertices_against_the_oracle(n, jitter, scale):
    """Nodal stresses and fluxes. A stress is some 20 terms,
    each up to 1e2 of the largest result (a derivative against its differences):
    20 x 100 x 2^-53 = 2e-13 of the largest."""
    pb, o, m, u, dp = _distorted(n, jitter, scale)
    m.set_state(u=u, u0=u, dp=dp)
    o.set_state(u=u, u0=u, dp=dp)
    kh = np.abs(np.asarray(pb["e"]).reshape(-1, oracle.PROP)[:, 2]).max()
    for name, a, b in zip(("stress", "stressB", "stressE", "flux"), m.stress(), o.stress()):
        s = max(np.abs(b).max(), kh if name == "flux" else 0.0)
        assert np.abs(a - b).max() <= 2e-13 * s, name


@pytest.mark.parametrize("n,jitter,kinds", [(1, 0.2, (40, 0)), (1, 0.2, (41, 43)),
                                            (2, 0.15, (40, 43)), (3, 0.1, (41, 0))])
def test_face_loads_against_the_oracle(n, jitter, kinds):
    """Loads on all six faces of every element (a face is left out on every other element):
    some 9 points x 6 faces x 8 elements of products a node, 64 x 20 of the state's
    forces, 2^-53 each and some 10 operations deep: 1e-12 of the largest force."""
    pb = _problem(n, jitter, (1, 1, 1))
    numel, nf = int(pb["numel"]), np.asarray(pb["fload"]).shape[1]
    load = np.array([[kinds[0], 0, 2], [kinds[1], 0, 2]], np.int32)
    fload = np.zeros((2, nf, 2))
    fload[:, 0] = [0.0, 5.0]
    fload[:, 1] = [[1.0, 2.0], [3.0, 1.0]]
    fload[:, 2] = [[-0.5, 0.3], [0.0, 0.0]]
    fload[:, 3] = [[0.7, -2.0], [0.0, 0.0]]
    eload = np.zeros((numel, 7), np.int32)
    eload[:, :6] = 1
    eload[::2, 3] = 0
    eloadp = np.zeros((numel, 7), np.int32)
    if kinds[1]:
        eloadp[:, :6] = 2
        eloadp[::2, 1] = 0
    pb.update(load=load, fload=fload, eload=eload, eloadp=eloadp)
    rng = np.random.default_rng(29)
    u = 1e-3 * rng.standard_normal((int(pb["nnode"]), 4))
    dp = 1e-3 * rng.standard_normal(int(pb["nnode"]))
    m, o = pg.from_problem(pb), oracle.from_fixture(pb)
    o.set_loads(eload=eload, eloadp=eloadp, load=load, fload=fload)
    for t in (m, o):
        t.set_env(pb["gravity"], float(pb["dt"]), 2.0)
        t.set_state(u=u, u0=u, dp=dp)
    b, bo = m.pform(4, False, True, u, np.zeros(m.neq)), np.zeros(o.neq)
    o.pform(4, False, True, u, bo)
    z = m.pform(4, False, True, u, np.zeros(m.neq))
    assert np.array_equal(b, z)
    assert np.abs(b - bo).max() <= 1e-12 * np.abs(bo).max()
