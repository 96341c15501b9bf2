"""Performance cases of the framework: the work a user's program has it do, through
its public entry points, over the sizes, precisions and options in use.

Kinds (the "kind" of a case):

diffusion   steady scalar diffusion on P2 triangles, -lap u = f with a
            manufactured solution: one linear solve by CG inside Newton, FP64,
            ILU(0) (the plain method, small meshes) or multigrid.
kovasznay   steady Navier-Stokes on Taylor-Hood P2-P1 triangles (Kovasznay
            flow): the whole Newton solve from the boundary values, plain FP64
            or mixed precision.
cavity      the next BDF2 steps of the lid-driven cavity from rest, with the
            extrapolated or the learned Newton guess.
cube        the next BDF2 steps of the unsteady flow in the unit cube on
            tetrahedra (body force, no-slip), the pressure taken relative to
            its mean (it is determined up to a constant).
residual    one residual evaluation at a given state, as a program that drives
            its own nonlinear iteration (the drop-in route) does it: the state
            goes up, the residual comes back.
jacobian    one FP64 Jacobian assembly at a given state, its values brought
            back to the host (a program that uses its own direct solver).
mlp_train   one training step of the network of the learned guess.
mlp_forward the network's prediction for a set of nodes.

The solves stop at the tight tolerances of this repository's parity tests
(relative residuals of 1e-11 to 1e-13), so that a solution is determined by
its problem and not by the path that the iteration takes to it.
"""
import numpy as np
import torch

import feng_gb300 as fe
from feng_gb300 import api, cavity, cube, exact as fields, kovasznay


def listed():
    return [
        # the plain method on its smallest configuration: 64^2, CG + ILU(0)
        {"name": "diffusion_64_cg_ilu0", "kind": "diffusion", "n": 64, "precond": "ilu0"},
        # the same problem at a size where multigrid is the only choice
        {"name": "diffusion_320_cg_amg", "kind": "diffusion", "n": 320, "precond": "amg"},
        # smallest flow solve: latency of a short Newton run in FP64
        {"name": "kovasznay_32_fp64", "kind": "kovasznay", "n": 32, "re": 40.0, "precision": "fp64"},
        # an ordinary odd size in mixed precision
        {"name": "kovasznay_97_mixed", "kind": "kovasznay", "n": 97, "re": 40.0, "precision": "mixed"},
        # the benchmark workload, both precisions
        {"name": "kovasznay_256_mixed", "kind": "kovasznay", "n": 256, "re": 40.0, "precision": "mixed"},
        {"name": "kovasznay_256_fp64", "kind": "kovasznay", "n": 256, "re": 40.0, "precision": "fp64"},
        # time stepping at the transient configuration's size, learned guess on
        {"name": "cavity_384_mixed", "kind": "cavity", "n": 384, "re": 1000.0, "dt": 0.005, "steps": 2,
         "precision": "mixed", "guess": "learned"},
        # time stepping on tetrahedra
        {"name": "cube_32_mixed", "kind": "cube", "n": 32, "re": 100.0, "dt": 0.01, "steps": 2, "precision": "mixed"},
        # single assemblies of a program that keeps its own nonlinear loop
        {"name": "residual_384_mixed", "kind": "residual", "elem": "th2d", "n": 384, "precision": "mixed"},
        {"name": "residual_cube_32_fp64", "kind": "residual", "elem": "th3d", "n": 32, "precision": "fp64"},
        {"name": "jacobian_128_fp64", "kind": "jacobian", "elem": "th2d", "n": 128},
        # the learned guess's network, one batch of the default size
        {"name": "mlp_train_16384", "kind": "mlp_train", "batch": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["diffusion", "kovasznay", "kovasznay", "kovasznay", "cavity", "cavity", "cube", "cube",
                       "residual", "residual", "jacobian", "mlp_train", "mlp_forward"])
    if kind == "diffusion":
        precond = rng.choice(["ilu0", "amg", "amg"])
        return {"kind": kind, "n": _log(rng, 16, 64 if precond == "ilu0" else 320), "precond": precond}
    if kind == "kovasznay":
        return {"kind": kind, "n": _log(rng, 16, 256), "re": rng.choice([20.0, 40.0]),
                "precision": rng.choice(["mixed", "mixed", "fp64"])}
    if kind == "cavity":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        return {"kind": kind, "n": _log(rng, 16, 384 if precision == "mixed" else 128),
                "re": rng.choice([100.0, 400.0, 1000.0]), "dt": rng.choice([0.005, 0.01]), "steps": rng.choice([1, 2]),
                "precision": precision, "guess": rng.choice(["previous", "extrapolate", "learned"])}
    if kind == "cube":
        precision = rng.choice(["mixed", "mixed", "fp64"])
        return {"kind": kind, "n": _log(rng, 4, 32 if precision == "mixed" else 12), "re": rng.choice([50.0, 100.0]),
                "dt": 0.01, "steps": rng.choice([1, 2]), "precision": precision}
    if kind == "residual":
        elem = rng.choice(["th2d", "th2d", "th3d"])
        return {"kind": kind, "elem": elem, "n": _log(rng, 8, 384) if elem == "th2d" else _log(rng, 3, 32),
                "precision": rng.choice(["mixed", "fp64"])}
    if kind == "jacobian":
        elem = rng.choice(["th2d", "th2d", "th3d"])
        return {"kind": kind, "elem": elem, "n": _log(rng, 8, 128) if elem == "th2d" else _log(rng, 3, 8)}
    return {"kind": kind, "batch": _log(rng, 1, 65536)}


# ---- the systems -----------------------------------------------------------


def _diffusion(n, seed, precond):
    mesh = fe.Mesh2DP1.generate_square(n, 0.0, 1.0, 0.0, 1.0, jitter=0.1, seed=seed)
    u = fe.createFiniteElementSpace(mesh, fe.LAGRANGE, 2, "U", "Domaine", 4, fields.zero_scalar)
    ub = fe.createFiniteElementSpace(mesh, fe.LAGRANGE, 2, "U", "Bord", 4, fields.sin_sin)
    num = fe.feMetaNumber(mesh, [ub, u], [ub])
    forms = [fe.createBilinearForm([u], fe.feSysElm_Diffusion(1.0)),
             fe.createBilinearForm([u], fe.feSysElm_Source(api.SRC_SIN_SIN, (-2 * np.pi ** 2,)))]
    return mesh, num, forms


def _assembly_case(elem, n, seed):
    """Mesh, numbering and forms of a transient flow on triangles or tetrahedra."""
    return cavity.build(n, 1000.0, seed=seed) if elem == "th2d" else cube.build(n, 100.0, seed=seed)


def _options(precision, **kw):
    # the parity tests' linear tolerances: FP64 solves to 1e-12, the mixed
    # path's outer iteration controls the accuracy
    tight = {"rel_tol": 1e-12} if precision == "fp64" else {"rel_tol": 1e-8}
    return fe.LinearSolverOptions(precision=precision, max_iter=5000, **{**tight, **kw})


def prepare(case, seed):
    kind, mseed = case["kind"], seed % (1 << 30) + 1
    if kind in ("mlp_train", "mlp_forward"):
        b = case["batch"]
        rng = np.random.default_rng(seed)
        net = fe.MLP(seed=mseed, max_batch=b)
        nin, nout = net.dims[0], net.dims[3]
        return {"case": case, "net": net, "params": net.params(),
                "x": rng.normal(0, 1, (b, nin)).astype(np.float32),
                "t": rng.normal(0, 0.5, (b, nout)).astype(np.float32),
                "mask": (rng.random((b, nout)) > 0.1).astype(np.float32)}
    if kind in ("residual", "jacobian"):
        _, num, forms = _assembly_case(case["elem"], case["n"], mseed)
        precision = case.get("precision", "fp64")
        system = fe.createLinearSystem(fe.CUDA, forms, num, _options(precision, precond="jacobi"))
        u, udot, c0 = _assembly_state(system.nDofs, seed)
        return {"case": case, "system": system, "u": u, "udot": udot, "c0": c0}
    if kind == "diffusion":
        _, num, forms = _diffusion(case["n"], mseed, case["precond"])
        system = fe.createLinearSystem(fe.CUDA, forms, num, _options("fp64", krylov="cg", precond=case["precond"]))
        nl = fe.feNLSolverOptions(tolResidual=0.0, tolCorrection=0.0, maxIter=10, relResidual=1e-11)
    elif kind == "kovasznay":
        _, num, forms = kovasznay.build(case["n"], case["re"], seed=mseed)
        mixed = case["precision"] == "mixed"
        system = fe.createLinearSystem(fe.CUDA, forms, num, _options(case["precision"], precond="amg"))
        nl = fe.feNLSolverOptions(tolResidual=0.0, tolCorrection=0.0, maxIter=30,
                                  relResidual=1e-12 if mixed else 1e-13, linearRtolMin=1e-6 if mixed else 0.0)
    else:
        builder = cavity.build if kind == "cavity" else cube.build
        _, num, forms = builder(case["n"], case["re"], seed=mseed)
        mixed = case["precision"] == "mixed"
        system = fe.createLinearSystem(fe.CUDA, forms, num, _options(case["precision"], precond="amg"))
        nl = fe.feNLSolverOptions(tolResidual=0.0, tolCorrection=0.0, tolDivergence=1e12, maxIter=30,
                                  relResidual=1e-11, linearRtolMin=1e-6 if mixed else 0.0)
    sol = fe.feSolution(system)
    sol.initializeEssentialBC()
    state = {"case": case, "system": system, "sol": sol, "nl": nl, "u0": sol.u.copy()}
    if kind in ("cavity", "cube"):
        learn = {}
        if case.get("guess") == "learned":
            learn = {"trainFrom": 2, "useFrom": 3, "seed": mseed}
        state["stepper"] = fe.createTimeIntegrator(fe.BDF2, nl, system, sol, 0.0, 400 * case["dt"], 400,
                                                   guess=case.get("guess", "extrapolate"), **learn)
        field = system.dofInfo()[2]
        state["pressure"] = np.flatnonzero(field == 1)
    return state


def _assembly_state(n_dofs, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(-1, 1, n_dofs), rng.uniform(-1, 1, n_dofs), 300.0


def run(state):
    kind = state["case"]["kind"]
    if kind == "mlp_forward":
        return state["net"].forward(state["x"])
    if kind == "mlp_train":
        net = state["net"]
        net.set_params(state["params"])
        loss, grad = net.train_step(state["x"], state["t"], state["mask"], 1e-3)
        return {"loss": np.float32(loss), "grad": grad}
    system = state["system"]
    if kind in ("residual", "jacobian"):
        system.setSolution(state["u"], state["udot"])
        system.setTime(0.0, state["c0"])
        if kind == "residual":
            system.setResidualToZero()
            system.assembleResiduals()
            return {"norm": system.getRHSMaxNorm(), "rhs": system.getRHS()}
        system.setMatrixToZero()
        system.assembleMatrices()
        return system.getMatrix()
    sol = state["sol"]
    if kind in ("diffusion", "kovasznay"):
        sol.u = state["u0"]
        fe.solveNewtonRaphson(system, sol, state["nl"])
        return sol.u
    state["stepper"].makeSteps(state["case"]["steps"])
    if kind == "cube":
        p = state["pressure"]
        u = sol.u.copy()
        u[p] -= u[p].mean()
        return u
    return sol.u


# ---- what a pass cannot do without ------------------------------------------


def _counts(case):
    """Elements, unknowns and CSR entries of a case's system (interior mesh)."""
    n, kind = case["n"], case["kind"]
    if kind == "diffusion":
        return 2 * n * n, (2 * n - 1) ** 2, 11.5 * (2 * n - 1) ** 2, 6
    if kind == "cube" or case.get("elem") == "th3d":
        inc = 3 * (2 * n - 1) ** 3 + (n + 1) ** 3
        return 6 * n ** 3, inc, 96.0 * inc, 34
    inc = 2 * (2 * n - 1) ** 2 + (n + 1) ** 2
    return 2 * n * n, inc, 29.0 * inc, 15


def work(case):
    kind = case["kind"]
    if kind in ("mlp_train", "mlp_forward"):
        b, macs = case["batch"], 16 * 64 + 64 * 64 + 64 * 4
        if kind == "mlp_forward":
            return {"bytes": b * 20 * 4.0, "flops": 2.0 * macs * b}
        return {"bytes": b * 24 * 4.0, "flops": 6.0 * macs * b}
    nelm, inc, nnz, nloc = _counts(case)
    # element addressing and vertex coordinates, the solution in and out
    base = nelm * (nloc * 4 + (48 if nloc < 30 else 96)) + inc * 16.0
    if kind == "residual":
        return {"bytes": base + inc * 8.0, "flops": nelm * (2000.0 if nloc < 30 else 20000.0)}
    matrix = nnz * (8.0 if case.get("precision", "fp64") == "fp64" else 4.0)
    if kind == "jacobian":
        return {"bytes": base + matrix, "flops": nelm * 4.0 * nloc * nloc * 10}
    # a solve or a time step: every Jacobian is formed and read at least once
    # with its columns (linear: 1, Newton: 4, a time step: 2)
    systems = {"diffusion": 1, "kovasznay": 4, "cavity": 2 * case.get("steps", 1), "cube": 2 * case.get("steps", 1)}[kind]
    return {"bytes": systems * (base + 2 * matrix + nnz * 4.0), "flops": systems * 2.0 * nnz}


# ---- the same in 64 bits with plain torch / numpy -----------------------------

_EDGES = {2: [(0, 1), (1, 2), (2, 0)], 3: [(0, 2), (2, 1), (1, 0), (1, 3), (3, 0), (3, 2)]}


def _basis(ref, d):
    """P2 values and reference gradients, P1 values, at points (q, d)."""
    lam = np.concatenate([1 - ref.sum(1, keepdims=True), ref], 1)
    dlam = np.concatenate([-np.ones((1, d)), np.eye(d)], 0)
    phi = [lam[:, i] * (2 * lam[:, i] - 1) for i in range(d + 1)]
    dphi = [(4 * lam[:, i:i + 1] - 1) * dlam[i] for i in range(d + 1)]
    for a, b in _EDGES[d]:
        phi.append(4 * lam[:, a] * lam[:, b])
        dphi.append(4 * (lam[:, a:a + 1] * dlam[b] + lam[:, b:b + 1] * dlam[a]))
    return np.stack(phi, 1), np.stack(dphi, 1), lam


class _Elements:
    """Element data of a mesh and numbering as FP64 torch tensors."""

    def __init__(self, mesh, num, d, degree):
        st = num.setup()
        a = mesh.arrays()
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.d, self.n_inc, self.n_dofs = d, st.nInc, st.nDofs
        t = self._t
        cells = a["tri"] if d == 2 else a["tet"]
        coords = np.stack([a["x"], a["y"]] + ([a["z"]] if d == 3 else []), 1)[cells]
        rule = np.stack(api.quadrature_rule(degree) if d == 2 else api.tet_quadrature_rule(degree), 1)
        phi, dphi, psi = _basis(rule[:, :d], d)
        X = t(coords)
        jm = torch.stack([X[:, i + 1] - X[:, 0] for i in range(d)], -1)
        self.phi, self.psi, dphi = t(phi), t(psi), t(dphi)
        self.G = torch.einsum("qkr,erx->eqkx", dphi, torch.linalg.inv(jm))
        self.W = torch.linalg.det(jm)[:, None] * t(rule[:, d])[None, :]
        self.xq = torch.einsum("qv,evx->eqx", self.psi, X)
        self.adr = torch.as_tensor(st.elementDofs(), device=self.dev)
        self.n2 = self.phi.shape[1]

    def _t(self, v):
        return torch.as_tensor(np.ascontiguousarray(v, np.float64), device=self.dev)

    def gather_rhs(self, be):
        out = torch.zeros(self.n_dofs, dtype=torch.float64, device=self.dev)
        out.index_add_(0, self.adr.reshape(-1), be.reshape(-1))
        return out[:self.n_inc]

    def entries(self, ae):
        """(row, column, value) of the coupled unknown pairs of all elements."""
        i = self.adr[:, :, None].expand(ae.shape).reshape(-1)
        j = self.adr[:, None, :].expand(ae.shape).reshape(-1)
        keep = (i < self.n_inc) & (j < self.n_inc)
        return i[keep], j[keep], ae.reshape(-1)[keep]

    def dense(self, ae):
        i, j, v = self.entries(ae)
        m = torch.zeros(self.n_inc * self.n_inc, dtype=torch.float64, device=self.dev)
        m.index_add_(0, i * self.n_inc + j, v)
        return m.reshape(self.n_inc, self.n_inc)


def _flow_residual(E, u, udot, conv, sigma, mu, divu, mass, force=None):
    d, n2 = E.d, E.n2
    ue = u[E.adr]
    U, P = ue[:, :d * n2].reshape(-1, n2, d), ue[:, d * n2:]
    uq = torch.einsum("qk,ekn->eqn", E.phi, U)
    gu = torch.einsum("eqkm,ekn->eqmn", E.G, U)
    pq = torch.einsum("qj,ej->eq", E.psi, P)
    f = -conv * torch.einsum("eqm,eqmn->eqn", uq, gu)
    if mass:
        V = udot[E.adr][:, :d * n2].reshape(-1, n2, d)
        f = f - mass * torch.einsum("qk,ekn->eqn", E.phi, V)
    if force is not None:
        f = f - force
    stress = sigma * mu * (gu + gu.transpose(-1, -2))
    stress = stress - sigma * pq[..., None, None] * torch.eye(d, dtype=u.dtype, device=u.device)
    bu = torch.einsum("eq,qk,eqc->ekc", E.W, E.phi, f) + torch.einsum("eq,eqmc,eqkm->ekc", E.W, stress, E.G)
    bp = -divu * torch.einsum("eq,eqmm,qj->ej", E.W, gu, E.psi)
    return E.gather_rhs(torch.cat([bu.reshape(len(bu), -1), bp], 1))


def _flow_matrix(E, u, conv, sigma, mu, divu, mass, c0):
    d, n2, nv = E.d, E.n2, E.d + 1
    U = u[E.adr][:, :d * n2].reshape(-1, n2, d)
    uq = torch.einsum("qk,ekn->eqn", E.phi, U)
    gu = torch.einsum("eqkm,ekn->eqmn", E.G, U)
    ne, nu = len(E.adr), d * n2
    eye = torch.eye(d, dtype=u.dtype, device=u.device)
    adv = torch.einsum("eqm,eqlm->eql", uq, E.G)
    s = conv * torch.einsum("eq,qk,eql->ekl", E.W, E.phi, adv)
    s = s - sigma * mu * torch.einsum("eq,eqkm,eqlm->ekl", E.W, E.G, E.G)
    s = s + mass * c0 * torch.einsum("eq,qk,ql->ekl", E.W, E.phi, E.phi)
    A = torch.einsum("ekl,ca->ekcla", s, eye)
    A = A + conv * torch.einsum("eq,qk,ql,eqac->ekcla", E.W, E.phi, E.phi, gu)
    A = A - sigma * mu * torch.einsum("eq,eqka,eqlc->ekcla", E.W, E.G, E.G)
    out = torch.zeros(ne, nu + nv, nu + nv, dtype=u.dtype, device=u.device)
    out[:, :nu, :nu] = A.reshape(ne, nu, nu)
    g = torch.einsum("eq,qj,eqkc->ekcj", E.W, E.psi, E.G).reshape(ne, nu, nv)
    out[:, :nu, nu:] = sigma * g
    out[:, nu:, :nu] = divu * g.transpose(1, 2)
    return out


def _exact_mlp(case, seed):
    s = prepare(case, seed)
    p = s["params"].astype(np.float64)
    x, t, mask = (s[k].astype(np.float64) for k in ("x", "t", "mask"))
    nin, h1, h2, nout = s["net"].dims
    cut = np.cumsum([h1 * nin, h1, h2 * h1, h2, nout * h2])
    w1, b1, w2, b2, w3, b3 = np.split(p, cut)
    w1, w2, w3 = w1.reshape(h1, nin), w2.reshape(h2, h1), w3.reshape(nout, h2)
    a1 = np.tanh(x @ w1.T + b1)
    a2 = np.tanh(a1 @ w2.T + b2)
    y = a2 @ w3.T + b3
    if case["kind"] == "mlp_forward":
        return y
    scale = 1.0 / (nout * len(x))
    dy = 2 * scale * mask * (y - t)
    d2 = (dy @ w3) * (1 - a2 * a2)
    d1 = (d2 @ w2) * (1 - a1 * a1)
    grad = [d1.T @ x, d1.sum(0), d2.T @ a1, d2.sum(0), dy.T @ a2, dy.sum(0)]
    return {"loss": float(scale * np.sum(mask * (y - t) ** 2)), "grad": np.concatenate([g.ravel() for g in grad])}


def exact(case, seed):
    kind, mseed = case["kind"], seed % (1 << 30) + 1
    if kind in ("mlp_train", "mlp_forward"):
        return _exact_mlp(case, seed)
    if kind in ("residual", "jacobian"):
        d = 2 if case["elem"] == "th2d" else 3
        mesh, num, _ = _assembly_case(case["elem"], case["n"], mseed)
        E = _Elements(mesh, num, d, 8 if d == 2 else 5)
        u, udot, c0 = _assembly_state(E.n_dofs, seed)
        u, udot = E._t(u), E._t(udot)
        mu = 1.0 / (1000.0 if d == 2 else 100.0)
        if kind == "jacobian":
            i, j, v = E.entries(_flow_matrix(E, u, 1.0, -1.0, mu, 1.0, 1.0, c0))
            ia, ja = num.setup().pattern()
            rows = np.repeat(np.arange(E.n_inc, dtype=np.int64), np.diff(ia))
            keys = torch.as_tensor(rows * E.n_inc + ja.astype(np.int64), device=E.dev)
            key = i * E.n_inc + j
            at = torch.searchsorted(keys, key).clamp(max=len(keys) - 1)
            hit = keys[at] == key  # the pressure rows do not couple to pressure columns
            vals = torch.zeros(len(keys), dtype=torch.float64, device=E.dev)
            vals.index_add_(0, at[hit], v[hit])
            return vals
        force = None
        if d == 3:
            f = -torch.prod(torch.sin(np.pi * E.xq), -1)
            force = torch.stack([f, torch.zeros_like(f), torch.zeros_like(f)], -1)
        r = _flow_residual(E, u, udot, 1.0, -1.0, mu, 1.0, 1.0, force)
        return {"norm": float(r.abs().max()), "rhs": r}
    if kind == "diffusion":
        if case["n"] > 64:
            return None
        mesh, num, _ = _diffusion(case["n"], mseed, case["precond"])
        E = _Elements(mesh, num, 2, 4)
        ke = torch.einsum("eq,eqkm,eqlm->ekl", E.W, E.G, E.G)
        f = 2 * np.pi ** 2 * torch.prod(torch.sin(np.pi * E.xq), -1)
        be = torch.einsum("eq,qk,eq->ek", E.W, E.phi, f)
        u = E._t(_boundary(num, lambda x, y: [np.sin(np.pi * x) * np.sin(np.pi * y)]))
        b = E.gather_rhs(be - torch.einsum("ekl,el->ek", ke, u[E.adr]))
        u[:E.n_inc] = torch.linalg.solve(E.dense(ke), b)
        return u
    if kind == "kovasznay":
        if case["n"] > 32:
            return None
        re = case["re"]
        mesh, num, _ = kovasznay.build(case["n"], re, seed=mseed)
        E = _Elements(mesh, num, 2, 8)
        lam = re / 2 - np.sqrt(re * re / 4 + 4 * np.pi ** 2)
        u = E._t(_boundary(num, lambda x, y: [1 - np.exp(lam * x) * np.cos(2 * np.pi * y),
                                              lam / (2 * np.pi) * np.exp(lam * x) * np.sin(2 * np.pi * y)],
                           lambda x, y: [0.5 * (1 - np.exp(2 * lam * x))]))
        for _ in range(12):
            b = _flow_residual(E, u, None, -1.0, 1.0, 1 / re, 1.0, 0.0)
            m = E.dense(_flow_matrix(E, u, -1.0, 1.0, 1 / re, 1.0, 0.0, 0.0))
            du = torch.linalg.solve(m, b)
            u[:E.n_inc] += du
            if float(du.abs().max()) < 1e-13:
                break
        return u
    return None


def _boundary(num, *fcts):
    """Zero unknowns and the essential values of each field at their nodes."""
    st = num.setup()
    x, y, field, comp, _ = st.dofInfo()
    u = np.zeros(st.nDofs)
    for k, f in enumerate(fcts):
        at = np.flatnonzero((field == k) & (np.arange(st.nDofs) >= st.nInc))
        vals = f(x[at], y[at])
        for c in range(len(vals)):
            u[at[comp[at] == c]] = np.broadcast_to(vals[c], at.shape)[comp[at] == c]
    return u
