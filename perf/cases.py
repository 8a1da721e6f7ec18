"""The work that a user of this framework has it do, as cases to be timed and
compared: time steps of Biot problems over meshes from a small column to a
40^3 cube, in FP64 and in the mixed precision, one mesh or a batch of them;
and the step's parts, each through its own entry point (matrix-vector product,
assembly, Krylov solve, the reference-layout product, the adjoint passes).

Meshes and materials are those of :mod:`poromec_gb300.meshgen`, with the
materials (and the tetra meshes' vertex positions) drawn from the seed.
Solves run to 1e-12, the tolerance of the gradient runs, so that the states
that come back do not depend on where the iteration happens to stop.
"""
import math

import numpy as np
import torch

import poromec_gb300 as pg
from poromec_gb300 import meshgen

TOL = 1e-12
# lower-triangle entries and equations per cell of the structured meshes
NNZL = {"cube": 1310.0, "column": 1100.0, "tetra": 1200.0}
NEQ = {"cube": 13.0, "column": 11.0, "tetra": 25.2}


def listed():
    return [
        # the smallest call: one step of the consolidation column, where
        # launches and latency count
        {"name": "step_column_2x2x40", "kind": "step", "mesh": "column", "n": 40, "prec": 0},
        # a step of a small and of the largest heterogeneous cube, FP64
        {"name": "step_cube_8", "kind": "step", "mesh": "cube", "n": 8, "prec": 0},
        {"name": "step_cube_40", "kind": "step", "mesh": "cube", "n": 40, "prec": 0},
        # the same with the mixed-precision operator
        {"name": "step_cube_31_mixed", "kind": "step", "mesh": "cube", "n": 31, "prec": 2},
        # a step of the jittered tetra10 box
        {"name": "step_tetra_20", "kind": "step", "mesh": "tetra", "n": 20, "prec": 0},
        # uneven independent meshes in one handle, mixed precision: a
        # parameter study
        {"name": "step_batch_16", "kind": "batch", "edges": "8,9,10,11,12,13,14,15,16,17,18,19,"
         "20,21,22,24", "prec": 2},
        # the reference's default solver (rpsqmr) on one right-hand side
        {"name": "solve_rpsqmr_tetra_11", "kind": "solve", "mesh": "tetra", "n": 11,
         "solver": 11},
        # one product with the assembled matrix: the largest mesh in FP64, and
        # a tetra mesh with the mixed-precision operator
        {"name": "matvec_cube_56", "kind": "matvec", "mesh": "cube", "n": 56, "prec": 0},
        {"name": "matvec_tetra_30_mixed", "kind": "matvec", "mesh": "tetra", "n": 30, "prec": 2},
        # assembly of K and of the right-hand side, and a first product with it
        {"name": "assemble_cube_28", "kind": "assemble", "mesh": "cube", "n": 28},
        # the product on a caller's own matrix in the reference's layout
        {"name": "csrd_matvec_cube_21", "kind": "csrd", "mesh": "cube", "n": 21},
        # the element passes of a reverse step (gradients)
        {"name": "adjoint_cube_32", "kind": "adjoint", "mesh": "cube", "n": 32},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "batch", "solve", "matvec", "matvec", "assemble",
                       "csrd", "adjoint"])
    if kind == "step":
        mesh = rng.choice(["cube", "cube", "column", "tetra"])
        n = {"cube": (3, 38), "column": (8, 200), "tetra": (3, 24)}[mesh]
        return {"kind": kind, "mesh": mesh, "n": _log_int(rng, *n), "prec": rng.choice([0, 2])}
    if kind == "batch":
        k = rng.randint(2, 20)
        return {"kind": kind, "edges": ",".join(str(_log_int(rng, 3, 24)) for _ in range(k)),
                "prec": rng.choice([0, 2])}
    if kind == "solve":
        mesh = rng.choice(["cube", "tetra"])
        return {"kind": kind, "mesh": mesh, "n": _log_int(rng, 3, 14),
                "solver": rng.choice([1, 11])}
    mesh = rng.choice(["cube", "tetra"])
    n = {"matvec": (3, 56), "assemble": (3, 40), "csrd": (3, 32), "adjoint": (3, 40)}[kind]
    case = {"kind": kind, "mesh": mesh, "n": _log_int(rng, n[0], n[1] if mesh == "cube" else
                                                      n[1] * 2 // 3)}
    if kind == "matvec":
        case["prec"] = rng.choice([0, 2])
    return case


# ---- problems ------------------------------------------------------------------
def _problem(mesh, n, seed):
    """A meshgen problem whose materials (and jitter) come from the seed."""
    rng = np.random.default_rng([seed, 77])
    if mesh == "cube":
        return meshgen.cube_problem(n=n, seed=1000 + 2 * seed)
    if mesh == "tetra":
        pb = meshgen.tetra_problem(n=n, seed=seed)
    else:
        pb = meshgen.column_problem(nz=n, lz=n / 4.0)
    e = np.array(pb["e"], float)
    e[:, 0] *= np.exp(0.3 * rng.standard_normal(len(e)))
    e[:, 2] *= np.exp(0.5 * rng.standard_normal(len(e)))
    pb["e"] = e
    return pb


def _instances(case, seed):
    return [meshgen.batch_instances(ninst=1, nmin=int(n), nmax=int(n), seed=1000 * seed + k)[0]
            for k, n in enumerate(case["edges"].split(","))]


def _eq(pb):
    """Equation numbers (nnode, 4), 0-based, -1 where there is none: node by
    node, the free dofs of each, the pressure on vertex nodes only."""
    free = np.asarray(pb["id"]) == 0
    free[:, 3] &= np.asarray(pb["fnno"]) == 1
    flat = free.ravel()
    return np.where(flat, np.cumsum(flat) - 1, -1).reshape(-1, 4)


def _field(pb, seed, k, amp_u, amp_p, noise=0.1):
    """A nodal field, metres and MPa, zero on restrained dofs: smooth modes
    and a little noise for a state or an increment, much noise for a search
    direction of an iteration."""
    rng = np.random.default_rng([seed, k])
    x = np.asarray(pb["x"])
    f = np.zeros((len(x), 4))
    for j in range(4):
        w = 2.0 * np.pi * rng.uniform(0.3, 2.0, 3)
        s = np.sin(x @ w + rng.uniform(0, 6.28))
        f[:, j] = (amp_u if j < 3 else amp_p) * (s + noise * rng.standard_normal(len(x)))
    f[_eq(pb) < 0] = 0.0
    return f


def _eqvec(pb, f):
    eq = _eq(pb)
    out = np.zeros(int(eq.max()) + 1)
    out[eq[eq >= 0]] = f[eq >= 0]
    return out


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _handle(case, seed):
    if case["kind"] == "batch":
        pb = meshgen.union_problem(_instances(case, seed))
    else:
        pb = _problem(case["mesh"], case["n"], seed)
    m = pg.from_problem(pb)
    if case.get("prec"):
        m.set_precision(case["prec"])
    return pb, m


def prepare(case, seed):
    kind = case["kind"]
    pb, m = _handle(case, seed)
    s = {"kind": kind, "m": m, "pb": pb, "solver": case.get("solver", 1)}
    zero = np.zeros((m.nnode, 4))
    if kind in ("step", "batch"):
        s["u0"], s["dp0"] = np.array(pb["u0"]), np.zeros(m.nnode)
        if case.get("prec"):  # the operator's one-off choice of kernel, as a program's set-up does
            m.pform(2, True, False, zero, None)
            m.tune_spmv()
    elif kind == "assemble":
        s["u"] = _field(pb, seed, 1, 1e-4, 0.1)
        s["b0"] = _eqvec(pb, _field(pb, seed, 2, 1e-3, 1e-6))
        s["x"] = _dev(_eqvec(pb, _field(pb, seed, 3, 1e-3, 1.0, 1.0)))
        s["y"] = torch.zeros_like(s["x"])
    elif kind == "adjoint":
        m.pform(2, True, False, zero, None)
        s["lam"] = _dev(_eqvec(pb, _field(pb, seed, 1, 1e-3, 1.0)))
        s["un"] = _dev(_field(pb, seed, 2, 1e-3, 1.0))
        s["dun"] = _dev(_field(pb, seed, 3, 1e-4, 0.1))
        s["mu"], s["nu"] = (torch.zeros_like(s["lam"]) for _ in range(2))
        s["grad"] = torch.zeros(int(pb["numel"]), 3, dtype=torch.float64, device="cuda")
    else:
        m.pform(2, True, False, zero, None)
        s["x"] = _dev(_eqvec(pb, _field(pb, seed, 1, 1e-3, 1.0, 1.0)))
        s["y"] = torch.zeros_like(s["x"])
        if kind == "solve":
            s["x"] = _dev(_eqvec(pb, _field(pb, seed, 1, 1e-3, 1e-6)))
        if kind == "csrd":
            ia, ja, ad, al = (_dev(a) for a in m.get_csrd())
            s["csrd"] = (ia, ja, ad, al)
        if case.get("prec"):
            m.tune_spmv()
    torch.cuda.synchronize()
    return s


def run(s):
    kind, m, pb = s["kind"], s["m"], s["pb"]
    if kind in ("step", "batch"):
        m.set_env(pb["gravity"], float(pb["dt"]), 0.0, 0)
        m.set_state(u=s["u0"], u0=s["u0"], dp=s["dp0"])
        m.step(maxnlit=500, tol=1e-4, stop_crit=1, solver=1, precond=2, solvtol=TOL,
               maxit=100000)
        u, _, dp = m.get_state()
        return {"u": u[:, :3], "p": u[:, 3], "dp": dp}
    if kind == "assemble":
        b = m.pform(2, True, True, s["u"], s["b0"].copy())
        m.spmv_dev(s["x"].data_ptr(), s["y"].data_ptr())
        return {"b": b, "y": s["y"]}
    if kind == "adjoint":
        st = torch.cuda.current_stream()
        for k in ("mu", "nu", "grad"):
            s[k].zero_()
        st.synchronize()
        m.adjoint_apply_dev(s["lam"].data_ptr(), s["mu"].data_ptr(), s["nu"].data_ptr())
        m.adjoint_grad_dev(s["lam"].data_ptr(), s["un"].data_ptr(), s["dun"].data_ptr(),
                           s["grad"].data_ptr())
        return {"mu": s["mu"], "nu": s["nu"], "grad": s["grad"]}
    if kind == "csrd":
        ia, ja, ad, al = s["csrd"]
        pg.matvec_csrd_dev(ad.numel(), ia.data_ptr(), ja.data_ptr(), ad.data_ptr(),
                           al.data_ptr(), s["x"].data_ptr(), s["y"].data_ptr())
        return s["y"]
    if kind == "solve":
        m.solve_dev(s["x"].data_ptr(), s["y"].data_ptr(), solver=s["solver"], precond=2, tol=TOL,
                    maxit=100000)
        return s["y"]
    m.spmv_dev(s["x"].data_ptr(), s["y"].data_ptr())
    return s["y"]


# ---- the work that cannot be avoided ----------------------------------------------
def _sizes(mesh, n):
    cells = 4.0 * n if mesh == "column" else float(n) ** 3
    return cells, cells * (6 if mesh == "tetra" else 1), NNZL[mesh] * cells, NEQ[mesh] * cells


def _iters(case, mesh, n):
    """Krylov iterations of one solve to 1e-12 on such a mesh (as counted)."""
    if case["kind"] == "batch":
        return 16.0 * n
    return {"cube": 62.0 * n, "tetra": 50.0 * n, "column": 4.0 * n}[mesh]


def _step_work(case, mesh, n, iters):
    _, numel, nnzl, neq = _sizes(mesh, n)
    val = 5.0 if case.get("prec") else 8.0
    per_it = (val + 4) * nnzl + 28 * neq + 88 * neq
    elem = (4.0e6 if mesh != "tetra" else 1.0e5) * numel
    return iters * per_it + 30 * nnzl, iters * (4 * nnzl + 13 * neq) + elem


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [_step_work(case, "cube", int(n), _iters(case, "cube", int(n)))
             for n in case["edges"].split(",")]
        return {"bytes": sum(a for a, _ in w), "flops": sum(b for _, b in w)}
    mesh, n = case["mesh"], case["n"]
    _, numel, nnzl, neq = _sizes(mesh, n)
    if kind in ("step", "solve"):
        b, f = _step_work(case, mesh, n, _iters(case, mesh, n))
        return {"bytes": b, "flops": f}
    val = 5.0 if case.get("prec") else 8.0
    if kind == "assemble":
        el = 2.0e6 if mesh == "cube" else 4.0e4
        return {"bytes": 2 * 8 * nnzl + 40 * neq, "flops": el * numel + 4 * nnzl}
    if kind == "adjoint":
        el = 2.5e5 if mesh == "cube" else 1.5e4
        return {"bytes": 120.0 * neq + 108 * numel, "flops": el * numel}
    return {"bytes": (val + 4) * nnzl + 28 * neq, "flops": 4 * nnzl}


# ---- the same in plain torch, 64 bits ------------------------------------------------
# Quadrature digits as the reference types them (Elmlib.f:3780-3962).
_G4 = [-.861136311594053, -.339981043584856, .339981043584856, .861136311594053]
_W4 = [.347854845137454, .652145154862546, .652145154862546, .347854845137454]
_HEX = np.array([(1, 1, 1), (-1, 1, 1), (-1, -1, 1), (1, -1, 1), (1, 1, -1), (-1, 1, -1),
                 (-1, -1, -1), (1, -1, -1), (0, 1, 1), (-1, 0, 1), (0, -1, 1), (1, 0, 1),
                 (0, 1, -1), (-1, 0, -1), (0, -1, -1), (1, 0, -1), (1, 1, 0), (-1, 1, 0),
                 (-1, -1, 0), (1, -1, 0)], float)
_EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (2, 3), (3, 1)]


def _shapes(hexa):
    """Quadrature weights, linear functions (g, nv) and derivatives
    (g, nv, 3), quadratic derivatives (g, nen, 3)."""
    if hexa:
        pts = np.array([(_G4[i], _G4[j], _G4[k]) for k in range(4) for j in range(4)
                        for i in range(4)])
        w = np.array([_W4[i] * _W4[j] * _W4[k] for k in range(4) for j in range(4)
                      for i in range(4)])
        hp, dp, du = np.zeros((64, 8)), np.zeros((64, 8, 3)), np.zeros((64, 20, 3))
        for k, c in enumerate(_HEX):
            f = 1 + pts * c  # 1 + r r_k per direction; 1 - r^2 where r_k = 0
            q = 1 - pts ** 2
            for d in range(3):
                a, b = (d + 1) % 3, (d + 2) % 3
                if k < 8:
                    hp[:, k] = f.prod(1) / 8
                    dp[:, k, d] = c[d] * f[:, a] * f[:, b] / 8
                    du[:, k, d] = c[d] * f[:, a] * f[:, b] * (pts @ c - 1 + pts[:, d] * c[d]) / 8
                else:
                    g = np.where(c == 0, q, f)
                    dg = -2 * pts[:, d] if c[d] == 0 else np.full(64, c[d])
                    du[:, k, d] = dg * g[:, a] * g[:, b] / 4
        return w, hp, dp, du
    a, b = 0.58541020, 0.13819660
    pts = np.array([(a, b, b), (b, a, b), (b, b, a), (b, b, b)])
    L = np.concatenate([pts, 1 - pts.sum(1, keepdims=True)], 1)
    dL = np.array([(1, 0, 0), (0, 1, 0), (0, 0, 1), (-1, -1, -1)], float)
    du = [(4 * L[:, k, None] - 1) * dL[k] for k in range(4)]
    du += [4 * (L[:, i, None] * dL[j] + L[:, j, None] * dL[i]) for i, j in _EDGES]
    w = np.full(4, 0.25 * 0.166666666666667)
    return w, L, np.repeat(dL[None], 4, 0), np.stack(du, 1)


class _Plain:
    """The element operators of one problem, chunk by chunk, in torch."""

    def __init__(self, pb):
        self.pb, self.hexa = pb, pb["nen"] == 20
        self.nen, self.nv = int(pb["nen"]), int(pb["nenv"])
        self.eq = _dev(_eq(pb))
        self.neq = int(self.eq.max()) + 1
        self.nodes = _dev(np.asarray(pb["ix"])[:, :self.nen].astype(np.int64) - 1)
        self.x = _dev(np.asarray(pb["x"], float))
        e = np.atleast_2d(pb["e"])[np.asarray(pb["ix"])[:, self.nen] - 1]
        g = np.asarray(pb["gravity"], float)
        E, nu = e[:, 0], e[:, 1]
        c = {"a": E * (1 - nu) / ((1 + nu) * (1 - 2 * nu)), "b": nu / (1 - nu),
             "c": 0.5 * (1 - 2 * nu) / (1 - nu), "M": 1 / e[:, 3], "al": e[:, 4],
             "fd": e[:, 6] * 1e-6}
        c["k"] = e[:, 2] / (c["fd"] * np.linalg.norm(g))
        self.c = {k: _dev(v) for k, v in c.items()}
        self.g, self.dt = _dev(g), float(pb["dt"])
        self.sh = [_dev(v) for v in _shapes(self.hexa)]

    def chunks(self):
        n = len(self.nodes)
        step = 1024 if self.hexa else 8192
        for i in range(0, n, step):
            sl = slice(i, min(n, i + step))
            nd = self.nodes[sl]
            w, hp, dl, dq = self.sh
            J = torch.einsum("gki,ekj->egij", dl, self.x[nd[:, :self.nv]])
            Ji = torch.linalg.inv(J)
            W = w * torch.linalg.det(J)
            yield sl, nd, W, hp, torch.einsum("egji,gki->egkj", Ji, dl), torch.einsum(
                "egji,gki->egkj", Ji, dq), {k: v[sl, None] for k, v in self.c.items()}

    @staticmethod
    def stress(c, D):
        e = torch.diagonal(D, dim1=-2, dim2=-1)
        tr = e.sum(-1, keepdim=True)
        s = (c["a"] * c["c"])[..., None, None] * (D + D.transpose(-1, -2))
        n = c["a"][..., None] * (e + c["b"][..., None] * (tr - e))
        return s - torch.diag_embed(torch.diagonal(s, dim1=-2, dim2=-1)) + torch.diag_embed(n)

    def forces(self, ch, u, p, pf, what):
        """(Fu, Fp) of element fields: u (e, nen, 3), p (e, nv) the pressure in
        the total stress, pf (e, nv) the pressure of the flow terms."""
        sl, nd, W, hp, gp, gq, c = ch
        S = self.stress(c, torch.einsum("eki,egkj->egij", u, gq))
        if "p" in what:
            S = S - torch.diag_embed((c["al"] * torch.einsum("gl,el->eg", hp, p))[..., None]
                                     .expand(-1, -1, 3))
        Fu = torch.einsum("eg,egij,egkj->eki", W, S, gq)
        flow = torch.einsum("egkj,ek->egj", gp, pf)
        if "g" in what:
            flow = flow - c["fd"][..., None] * self.g
        Fp = -torch.einsum("eg,egj,eglj->el", W * c["k"] * self.dt, flow, gp)
        if "s" in what:
            tr = torch.einsum("eki,egki->eg", u, gq)
            q = c["al"] * tr + c["M"] * torch.einsum("gl,el->eg", hp, pf)
            Fp = Fp - torch.einsum("eg,gl->el", W * q, hp)
        return Fu, Fp

    def nodal(self, v):
        """Equation vector -> nodal (nnode, 4)."""
        out = torch.zeros(self.eq.shape, dtype=torch.float64, device="cuda")
        out[self.eq >= 0] = v[self.eq[self.eq >= 0]]
        return out

    def scatter(self, out, nd, Fu, Fp):
        if Fu is not None:
            out.index_put_((nd[..., None], torch.arange(3, device="cuda")), Fu, accumulate=True)
        if Fp is not None:
            out.index_put_((nd[:, :self.nv], torch.full_like(nd[:, :self.nv], 3)), Fp,
                           accumulate=True)

    def to_eq(self, f):
        out = torch.zeros(self.neq, dtype=torch.float64, device="cuda")
        out[self.eq[self.eq >= 0]] = f[self.eq >= 0]
        return out

    def apply(self, f):
        """K f of a nodal field f, as an equation vector."""
        out = torch.zeros_like(f)
        for ch in self.chunks():
            nd = ch[1]
            p = f[nd[:, :self.nv], 3]
            self.scatter(out, nd, *self.forces(ch, f[nd, :3], p, p, "ps"))
        return self.to_eq(out)

    def dense(self):
        K = torch.zeros(self.neq + 1, self.neq + 1, dtype=torch.float64, device="cuda")
        for ch in self.chunks():
            nd, nst = ch[1], 3 * self.nen + self.nv
            eq = torch.cat([self.eq[nd, :3].reshape(len(nd), -1), self.eq[nd[:, :self.nv], 3]], 1)
            eq = torch.where(eq < 0, self.neq, eq)
            for k in range(nst):
                I = torch.zeros(len(nd), nst, dtype=torch.float64, device="cuda")
                I[:, k] = 1
                u, p = I[:, :3 * self.nen].reshape(len(nd), -1, 3), I[:, 3 * self.nen:]
                Fu, Fp = self.forces(ch, u, p, p, "ps")
                K.index_put_((eq, eq[:, k:k + 1].expand_as(eq)),
                             torch.cat([Fu.reshape(len(nd), -1), Fp], 1), accumulate=True)
        return K[:-1, :-1]

    def step(self):
        """The first step from rest under the hydrostatic pressure: a linear
        solve, as the elastic elements make it."""
        pb = self.pb
        u0 = _dev(np.asarray(pb["u0"], float))
        out = torch.zeros_like(u0)
        zero = torch.zeros(1, dtype=torch.float64, device="cuda")
        for ch in self.chunks():
            nd = ch[1]
            pf = u0[nd[:, :self.nv], 3]
            Fu, Fp = self.forces(ch, u0[nd, :3], zero, pf, "g")
            self.scatter(out, nd, -Fu, -Fp)
        if "nload" in pb:  # the point source
            at = np.nonzero(np.asarray(pb["nload"])[:, 3])[0]
            out[_dev(at), 3] -= self.dt * float(pb["fload"][0, 0, 0])
        else:  # the traction on the top faces at t = dt
            t, v = pb["fload"][0][0], pb["fload"][0][3]
            tz = float(np.interp(self.dt, t, v)) if len(t) > 1 else float(v[0])
            top = _dev(np.nonzero(np.asarray(pb["eload"])[:, 0])[0])
            nd = self.nodes[top]
            X = self.x[nd]
            A = (X[:, 0, 0] - X[:, 1, 0]).abs() * (X[:, 0, 1] - X[:, 3, 1]).abs()
            for k in list(range(4)) + list(range(8, 12)):
                out[:, 2].index_add_(0, nd[:, k], A * tz * (-1 / 12 if k < 4 else 1 / 3))
        du = self.nodal(torch.linalg.solve(self.dense(), self.to_eq(out)))
        u = u0 + du
        dp = torch.where(_dev(np.asarray(pb["fnno"]) == 1), du[:, 3], 0.0)
        return u, dp


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        if sum(13 * int(n) ** 3 for n in case["edges"].split(",")) > 20000:
            return None
        got = [_Plain(pb).step() for pb in _instances(case, seed)]
        u, dp = torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])
    else:
        pb = _problem(case["mesh"], case["n"], seed)
        P = _Plain(pb)
        if kind == "step":
            if P.neq > 12000:
                return None
            u, dp = P.step()
    if kind in ("step", "batch"):
        u, dp = u.cpu().numpy(), dp.cpu().numpy()
        return {"u": u[:, :3], "p": u[:, 3], "dp": dp}
    if kind in ("matvec", "csrd"):
        return P.apply(_dev(_field(pb, seed, 1, 1e-3, 1.0, 1.0)))
    if kind == "solve":
        if P.neq > 12000:
            return None
        b = _dev(_eqvec(pb, _field(pb, seed, 1, 1e-3, 1e-6)))
        return torch.linalg.solve(P.dense(), b)
    if kind == "assemble":
        b = P.to_eq(_dev(_field(pb, seed, 2, 1e-3, 1e-6))) - P.apply(
            _dev(_field(pb, seed, 1, 1e-4, 0.1)))
        return {"b": b.cpu().numpy(), "y": P.apply(_dev(_field(pb, seed, 3, 1e-3, 1.0, 1.0)))}
    lam, un, dun = (_dev(_field(pb, seed, k, a, b)) for k, a, b in
                    ((1, 1e-3, 1.0), (2, 1e-3, 1.0), (3, 1e-4, 0.1)))
    mu, nu = torch.zeros_like(lam), torch.zeros_like(lam)
    grad = torch.zeros(len(P.nodes), 3, dtype=torch.float64, device="cuda")
    for ch in P.chunks():
        sl, nd, W, hp, gp, gq, c = ch
        lu, lp = lam[nd, :3], lam[nd[:, :P.nv], 3]
        Fu, Fp = P.forces(ch, lu, None, lp, "")
        P.scatter(mu, nd, -Fu, -Fp)
        tr = torch.einsum("eki,egki->eg", lu, gq)
        P.scatter(nu, nd, None, torch.einsum("eg,gl->el", W * c["al"] * tr, hp))
        Gu, Gp = P.forces(ch, un[nd, :3], None, un[nd[:, :P.nv], 3], "g")
        grad[sl, 0] = -(lu * Gu).sum((1, 2))
        grad[sl, 1] = -(lp * Gp).sum(1)
        d = torch.einsum("gl,el->eg", hp, dun[nd[:, :P.nv], 3])
        grad[sl, 2] = -(W * c["M"] * d * torch.einsum("gl,el->eg", hp, lp)).sum(1)
    return {"mu": P.to_eq(mu), "nu": P.to_eq(nu), "grad": grad}
