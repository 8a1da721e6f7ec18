"""Element blocks of the hexa20 Biot element in plain numpy, in the arithmetic T
(float64 or longdouble): the formulas of lku_m (Elmlib03.f) over the 4 x 4 x 4 rule."""
import numpy as np

# quadrature digits as the reference types them (Elmlib.f:3780-3962)
X4 = (-.861136311594053, -.339981043584856, .339981043584856, .861136311594053)
W4 = (.347854845137454, .652145154862546, .652145154862546, .347854845137454)
NODE = np.array([(1, 1, 1), (-1, 1, 1), (-1, -1, 1), (1, -1, 1), (1, 1, -1), (-1, 1, -1),
                  (-1, -1, -1), (1, -1, -1), (0, 1, 1), (-1, 0, 1), (0, -1, 1), (1, 0, 1),
                  (0, 1, -1), (-1, 0, -1), (0, -1, -1), (1, 0, -1), (1, 1, 0), (-1, 1, 0),
                  (-1, -1, 0), (1, -1, 0)])


def blocks(X, e, grav, dt, T):
    """Kuu (60, 60), Kpu (8, 60), Kperm and Kstor (8, 8), G_k (8) and the sum of its
    terms' magnitudes, of vertices X (8, 3) and material row e."""
    x, w = np.array(X4, T), np.array(W4, T)
    pts = np.array([(x[i], x[j], x[k]) for k in range(4) for j in range(4) for i in range(4)], T)
    W = np.array([w[i] * w[j] * w[k] for k in range(4) for j in range(4) for i in range(4)], T)
    hp, dl, dq = np.zeros((64, 8), T), np.zeros((64, 8, 3), T), np.zeros((64, 20, 3), T)
    for k, c in enumerate(NODE.astype(T)):
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
    Kuu = np.zeros((20, 3, 20, 3), T)
    for k in range(3):
        for m in range(3):
            Kuu[:, k, :, m] = (a * (P[:, k, :, k] + c * (tr - P[:, k, :, k])) if k == m else
                               a * (b * P[:, k, :, m] + c * P[:, m, :, k]))
    Kpu = -T(e[4]) * np.einsum("gl,gjk->ljk", W[:, None] * hp, gq).reshape(8, 60)
    Kstor = -np.einsum("gl,gm->lm", W[:, None] * hp, hp) / T(e[3])
    Kperm = -T(dt) * perm * np.einsum("glk,gmk->lm", W[:, None, None] * gp, gp)
    Gk = T(dt) * perm * fd * W[:, None] * np.einsum("glk,k->gl", gp, grav.astype(T))
    return Kuu.reshape(60, 60), Kpu, Kperm, Kstor, Gk.sum(0), np.abs(Gk).sum(0)


def matrix(X, e, grav, dt, T):
    """K_e: 60 displacements node by node, 8 pressures."""
    Kuu, Kpu, Kperm, Kstor = blocks(X, e, grav, dt, T)[:4]
    return np.block([[Kuu, Kpu.T], [Kpu, Kstor + Kperm]])
