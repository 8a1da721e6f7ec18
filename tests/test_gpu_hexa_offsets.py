"""The hexa20 passes by sum factorisation (pm_hexa_sum.h) take derivatives of
differences: what a field or the coordinates have in common over an element leaves no
rounding, in any of the three directions."""
import numpy as np
import pytest

import poromec_gb300 as pg
from poromec_gb300 import meshgen

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _problem(shift=0.0):
    """A 3^3 cube with all dofs free, stretched and jittered, its coordinates multiples
    of 2^-10: exact also when shifted by a power of two."""
    pb = meshgen.cube_problem(n=3)
    pb["id"] = np.zeros_like(pb["id"])
    x = np.asarray(pb["x"], float)
    x = np.round(6.0 * x / x.max(0)) / np.array([4.0, 2.0, 8.0])
    pb["x"] = x + np.random.default_rng(7).integers(-32, 33, x.shape) / 1024.0 + shift
    return pb


def _mesh(pb):
    m = pg.from_problem(pb)
    m.pform(2, True, False, np.zeros((m.nnode, 4)), None)
    return m


def _eq(pb):
    has = np.ones((int(pb["nnode"]), 4), bool)
    has[:, 3] = np.asarray(pb["fnno"]) == 1
    return np.where(has, np.cumsum(has.ravel()).reshape(-1, 4) - 1, -1)


def _apply(m, lam):
    t = torch.as_tensor(lam).cuda()
    mu, nu = torch.zeros_like(t), torch.zeros_like(t)
    torch.cuda.synchronize()
    m.adjoint_apply_dev(t.data_ptr(), mu.data_ptr(), nu.data_ptr())
    torch.cuda.synchronize()
    return mu.cpu().numpy(), nu.cpu().numpy()


def test_pressure_with_a_large_mean():
    """Flow of 1 + 2^-30 f is 2^-30 times that of f for whole nodal numbers f: their
    differences are exact, and a power of two changes no rounding (1e-13 of the largest
    for the order of nothing). Interpolated values, whose difference is taken after they
    are rounded, leave some 2^-53 / 2^-30 / 8 = 1e-8 of it."""
    pb = _problem()
    m = _mesh(pb)
    eq = _eq(pb)
    p = eq[:, 3] >= 0
    f = np.random.default_rng(3).integers(0, 16, m.nnode).astype(float)
    lam, one = np.zeros(m.neq), np.zeros(m.neq)
    lam[eq[p, 3]] = f[p]
    one[eq[p, 3]] = 1.0 + 2.0 ** -30 * f[p]
    ref = _apply(m, lam)[0][eq[p, 3]]
    got = _apply(m, one)[0][eq[p, 3]] * 2.0 ** 30
    assert np.abs(ref).max() > 0
    assert np.abs(got - ref).max() <= 1e-13 * np.abs(ref).max()


def test_mesh_far_from_the_origin():
    """The mesh moved by 2^16 in all directions, exactly: forces of the residual, the
    adjoint's product and its gradients to 1e-13 of the largest (the element's vertices
    and edges are differences of the same numbers). Differences of interpolated
    coordinates lose 2^-53 2^16 / (1/4) = 3e-11."""
    out = []
    for shift in (0.0, 2.0 ** 16):
        pb = _problem(shift)
        m = _mesh(pb)
        rng = np.random.default_rng(5)
        u = rng.standard_normal((m.nnode, 4))
        lam = rng.standard_normal(m.neq)
        tl, tu = torch.as_tensor(lam).cuda(), torch.as_tensor(u).cuda()
        gr = torch.zeros(m.numel, 3, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        m.adjoint_grad_dev(tl.data_ptr(), tu.data_ptr(), tu.data_ptr(), gr.data_ptr())
        torch.cuda.synchronize()
        g = gr.cpu().numpy()
        out.append([m.pform(2, False, True, u, np.zeros(m.neq)), *_apply(m, lam), g[:, 0], g[:, 1],
                    g[:, 2]])
    for a, b in zip(*out):
        assert np.abs(a - b).max() <= 1e-13 * np.abs(a).max()
