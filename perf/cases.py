"""Performance cases of the framework: what a program that uses it has it do, through its public entry points.

Single assembly calls (AssemblyManager), one operator application, one whole Newton solve (SolverManager) and one
batch of local solves (SubgridBatch), from a 32 x 32 mesh, where launches and latency count, to 2 million cells.
``exact`` is a dense-quadrature finite-element assembly in plain torch (64 bits) with its own index arithmetic.
"""
import math

import numpy as np
import torch

import mrhyde_gb300._lib as L
from mrhyde_gb300 import AssemblyManager, Problem, SolverManager
from mrhyde_gb300.subgrid import SubgridBatch

X_FACES = L.MRG_FACE_XLO | L.MRG_FACE_XHI


def _asm(name, dim, order, n, kind, geometry, precision, call, source="const", neumann=False):
    case = {"what": "assemble", "dim": dim, "order": order, "nx": n[0], "ny": n[1], "nz": n[2] if dim == 3 else 1,
            "kind": kind, "geometry": geometry, "precision": precision, "call": call, "source": source,
            "neumann": neumann}
    return {"name": name, **case} if name else case


def listed():
    return [
        # verification-sized 2-D run, one assembly per Newton step: latency and launches
        _asm("quad_q1_32", 2, 1, (32, 32), "thermal", "cube", "fp64", "jacres", source="sinprod"),
        # large steady heat conduction on a cube with a random medium: the headline assembly
        _asm("hex_q1_cube_128", 3, 1, (128, 128, 128), "thermal", "cube", "fp64", "jacres"),
        # box cells that are no cubes, odd counts; the two calls of one mixed-precision Newton step
        _asm("hex_q1_box_97x61x75", 3, 1, (97, 61, 75), "thermal", "box", "mixed", "step"),
        # heat conduction on a mesh fitted to a geometry: every cell its own shape
        _asm("hex_q1_mapped_91x96x101", 3, 1, (91, 96, 101), "thermal", "mapped", "fp64", "jacres"),
        # temperature-dependent conductivity, Q1: a Newton step of the nonlinear serving request
        _asm("hex_q1_nonlinear_95", 3, 1, (95, 95, 95), "diffusion_1pu2", "cube", "fp64", "jacres"),
        # temperature-dependent conductivity, Q2, mixed precision: the large high-order run
        _asm("hex_q2_nonlinear_64", 3, 2, (64, 64, 64), "diffusion_1pu2", "cube", "mixed", "jacres"),
        # high-order conduction through a random medium in full precision
        _asm("hex_q2_thermal_33x30x27", 3, 2, (33, 30, 27), "thermal", "box", "fp64", "jacres"),
        # nonlinear conduction on a fitted mesh
        _asm("hex_q1_nonlinear_mapped_47x45x50", 3, 1, (47, 45, 50), "diffusion_1pu2", "mapped", "fp64", "jacres"),
        # 2-D high-order run with a prescribed heat flux on two sides
        _asm("quad_q2_300x211", 2, 2, (300, 211), "thermal", "box", "fp64", "jacres", source="sinprod", neumann=True),
        # the operator inside a Krylov loop of the caller's own, high-order matrix in single precision
        {"name": "apply_hex_q2_41x38x45", "what": "apply", "dim": 3, "order": 2, "nx": 41, "ny": 38, "nz": 45,
         "precision": "mixed"},
        # a whole solve to a relative residual of 1e-10, as the serving loop runs it for one large request
        {"name": "newton_nonlinear_96", "what": "newton", "edge": 96, "kind": "diffusion_1pu2", "precision": "mixed",
         "preconditioner": "gmg"},
        # the local solves of a multiscale model: a few hundred of its thousands of subgrids
        {"name": "subgrid_700", "what": "subgrid", "problems": 700, "least": 4, "most": 16},
    ]


def _sizes(rng, dim, least, most):
    """Cells per axis: the count log-uniform in [least, most], the axes unlike each other."""
    count = math.exp(rng.uniform(math.log(least), math.log(most)))
    lean = [math.exp(rng.uniform(-0.3, 0.3)) for _ in range(dim)]
    mean = math.prod(lean) ** (1.0 / dim)
    n = [max(2, int(count ** (1.0 / dim) * a / mean)) for a in lean]
    while math.prod(n) > most:
        n[n.index(max(n))] -= 1
    return n


def draw(rng):
    what = rng.choice(["q1", "q1", "q1", "q1_2d", "mapped", "nonlinear", "nonlinear_mapped", "q2", "q2", "q2_2d",
                       "apply", "newton", "subgrid"])
    fp = rng.choice(["fp64", "mixed"])
    call = rng.choice(["jacres", "jacres", "step", "res"])
    if what == "q1":
        if rng.random() < 0.5:
            e = int(math.exp(rng.uniform(math.log(8), math.log(126))))
            return _asm(None, 3, 1, (e, e, e), "thermal", "cube", fp, call)
        return _asm(None, 3, 1, _sizes(rng, 3, 500, 1 << 20), "thermal", "box", fp, call)
    if what == "q1_2d":
        return _asm(None, 2, 1, _sizes(rng, 2, 1000, 1 << 20), rng.choice(["thermal", "diffusion_1pu2"]),
                    rng.choice(["box", "mapped"]), fp, call, source=rng.choice(["const", "sinprod"]))
    if what == "mapped":
        return _asm(None, 3, 1, _sizes(rng, 3, 1000, 900000), "thermal", "mapped", fp, call)
    if what == "nonlinear":
        return _asm(None, 3, 1, _sizes(rng, 3, 1000, 850000), "diffusion_1pu2", "box", fp, call)
    if what == "nonlinear_mapped":
        return _asm(None, 3, 1, _sizes(rng, 3, 1000, 100000), "diffusion_1pu2", "mapped", fp, call)
    if what == "q2":
        kind = rng.choice(["thermal", "diffusion_1pu2"])
        return _asm(None, 3, 2, _sizes(rng, 3, 200, 100000 if fp == "mixed" else 27000), kind, "box", fp, call)
    if what == "q2_2d":
        return _asm(None, 2, 2, _sizes(rng, 2, 300, 100000), rng.choice(["thermal", "diffusion_1pu2"]),
                    rng.choice(["box", "mapped"]), fp, call, source=rng.choice(["const", "sinprod"]))
    if what == "apply":
        order = rng.choice([1, 2])
        n = _sizes(rng, 3, 1000, 70000 if order == 2 else 560000)
        return {"what": "apply", "dim": 3, "order": order, "nx": n[0], "ny": n[1], "nz": n[2], "precision": fp}
    if what == "newton":
        most = 92 if fp == "mixed" else 48
        return {"what": "newton", "edge": int(math.exp(rng.uniform(math.log(12), math.log(most)))),
                "kind": rng.choice(["thermal", "diffusion_1pu2"]), "precision": fp,
                "preconditioner": rng.choice(["gmg", "gmg", "jacobi"]) if most < 60 else "gmg"}
    least = rng.randint(3, 8)
    return {"what": "subgrid", "problems": int(math.exp(rng.uniform(math.log(20), math.log(700)))), "least": least,
            "most": rng.randint(least + 1, 16)}


# ---- inputs -------------------------------------------------------------------------------------
def _extent(case, n):
    if case["geometry"] == "cube":
        return [1.0] * len(n)
    return [1.0, 0.7, 0.45][:len(n)]  # cells unlike along the axes


def _vertices(n, hi, rng):
    """A box's vertices (x fastest), interior ones moved by up to a fifth of a cell."""
    d = len(n)
    idx = np.stack([g.reshape(-1) for g in np.meshgrid(*[np.arange(m + 1) for m in reversed(n)], indexing="ij")][::-1], 1)
    h = np.array(hi) / np.array(n)
    pts = idx * h
    inner = np.all((idx > 0) & (idx < np.array(n)), axis=1)
    pts[inner] += 0.2 * h * rng.uniform(-1.0, 1.0, (int(inner.sum()), d))
    return np.ascontiguousarray(pts)


def _inputs(case, seed):
    rng = np.random.default_rng(seed)
    n = [case["nx"], case["ny"], case["nz"]][:case["dim"]]
    hi = _extent(case, n)
    nodes = math.prod(case["order"] * m + 1 for m in n)
    thermal = case["kind"] == "thermal"
    cfg = {"dim": case["dim"], "order": case["order"], "n": tuple(n), "lo": (0.0,) * len(n), "hi": tuple(hi),
           "kind": case["kind"], "source": ("sinprod", 1.0, math.pi) if case["source"] == "sinprod" else
           ("const", 1.0 if thermal else 10.0, 0.0),
           "kappa": np.exp(0.5 * rng.standard_normal(math.prod(n))) if thermal else 1.0,
           "dirichlet_faces": X_FACES if case["dim"] == 3 or case["neumann"] else L.MRG_FACE_ALL}
    if case["geometry"] == "mapped":
        cfg["vertex_coords"] = _vertices(n, hi, rng)
    u = rng.uniform(0.0, 0.1, nodes) if not thermal else rng.uniform(-1.0, 1.0, nodes)
    flux = None
    if case["neumann"]:
        flux = {f: rng.uniform(-1.0, 1.0, n[0] * (case["order"] + 1)) for f in (2, 3)}
    return cfg, u, flux


def _newton_inputs(case, seed):
    e, thermal = case["edge"], case["kind"] == "thermal"
    rng = np.random.default_rng(seed)
    cfg = {"dim": 3, "order": 1, "n": (e, e, e), "lo": (0.0,) * 3, "hi": (1.0,) * 3, "kind": case["kind"],
           "source": ("const", 1.0 if thermal else 10.0, 0.0),
           "kappa": np.exp(rng.standard_normal(e ** 3)) if thermal else 1.0, "dirichlet_faces": X_FACES}
    # the nonlinear problem's data is its start and its source's strength
    if not thermal:
        cfg["source"] = ("const", float(rng.uniform(8.0, 12.0)), 0.0)
    u0 = np.zeros((e + 1) ** 3) if thermal else rng.uniform(0.0, 0.1, (e + 1) ** 3)
    return cfg, u0


def _subgrid_inputs(case, seed):
    # the meshes belong to the case, coefficients and boundary data to the seed
    meshes = np.random.default_rng([case["problems"], case["least"], case["most"]])
    sizes = meshes.integers(case["least"], case["most"] + 1, size=(case["problems"], 3))
    rng = np.random.default_rng(seed)
    kap = [np.exp(rng.standard_normal(int(np.prod(s)))) for s in sizes]
    dbc = [rng.uniform(-1.0, 1.0, int(np.prod(s + 1))) for s in sizes]
    return sizes, kap, dbc


def _apply_inputs(case, seed, device):
    n, p = (case["nx"], case["ny"], case["nz"]), case["order"]
    nnz, nodes = math.prod(_axis(m, p)[2] for m in n), math.prod(p * m + 1 for m in n)
    g = torch.Generator(device=device).manual_seed(seed)
    dtype = torch.float32 if case["precision"] == "mixed" else torch.float64
    J = torch.randn(nnz, generator=g, device=device, dtype=dtype)
    return J, torch.rand(nodes, generator=g, device=device, dtype=torch.float64)


def prepare(case, seed):
    if case["what"] == "apply":
        P = Problem(dim=3, order=case["order"], n=(case["nx"], case["ny"], case["nz"]), dirichlet_faces=X_FACES)
        J, x = _apply_inputs(case, seed, "cuda")
        return {"case": case, "solver": SolverManager(P), "J": J, "x": x, "y": P.new_vector(), "problem": P}
    if case["what"] == "newton":
        cfg, u0 = _newton_inputs(case, seed)
        P = Problem(**cfg)
        mixed = case["precision"] == "mixed"
        S = SolverManager(P, nonlinear_tol=1e-10, max_nonlinear_iters=30, linear_tol=1e-3 if mixed else 1e-11,
                          linear_maxiter=20000, mixed_precision=mixed, preconditioner=case["preconditioner"])
        u0 = torch.tensor(u0, device="cuda")
        return {"case": case, "solver": S, "u0": u0, "u": torch.empty_like(u0), "problem": P}
    if case["what"] == "subgrid":
        return {"case": case, "batch": SubgridBatch(*_subgrid_inputs(case, seed), source=1.0)}
    cfg, u, flux = _inputs(case, seed)
    P = Problem(**cfg)
    for face, g in (flux or {}).items():
        P.set_face_bc(face, "neumann", g)
    state = {"case": case, "assembly": AssemblyManager(P), "u": torch.tensor(u, device="cuda"), "r": P.new_vector(),
             "problem": P}
    if case["call"] != "res":
        state["J"] = P.new_matrix_values(fp32=case["precision"] == "mixed")
    return state


def run(state):
    case = state["case"]
    if case["what"] == "apply":
        return {"y": state["solver"].apply(state["J"], state["x"], state["y"])}
    if case["what"] == "newton":
        state["u"].copy_(state["u0"])
        state["solver"].nonlinearSolver(state["u"])
        return {"u": state["u"]}
    if case["what"] == "subgrid":
        state["batch"].solve()
        return {"u": state["batch"].u, "J": state["batch"].J}
    A, u, r, fp32 = state["assembly"], state["u"], state["r"], case["precision"] == "mixed"
    if case["call"] == "res":
        A.assembleRes(u, r, overwrite=True)
        return {"r": r}
    J = state["J"]
    if case["call"] == "step":  # the residual for the convergence test, then the Jacobian
        A.assembleRes(u, r, overwrite=True)
        A.assembleJac(u, J, fp32_jacobian=fp32, overwrite=True)
    else:
        A.assembleJacRes(u, r, J, fp32_jacobian=fp32, overwrite=True)
    return {"r": r, "J": J}


def _counts(dim, order, n):
    nodes = math.prod(order * m + 1 for m in n)
    nnz = math.prod(_axis(m, order)[2] for m in n)
    return nodes, math.prod(n), nnz


def _assembly_work(case, n, jac, word):
    """Each input read once, each output written once; element contractions by sum factorisation."""
    p, d = case["order"], len(n)
    nodes, cells, nnz = _counts(d, p, n)
    q, npe = (p + 1) ** d, (p + 1) ** d
    b = 8 * nodes * 2 + (8 * cells if case["kind"] == "thermal" else 0) + (nnz * word if jac else 0)
    if case.get("geometry") == "mapped":
        b += 8 * d * math.prod(m + 1 for m in n)
    f = cells * 2 * 2 * d * d * (p + 1) * q  # the fields at the points and back
    if p == 1 and case["kind"] == "thermal" and case.get("geometry") != "mapped":
        f = 2 * nnz
    elif p == 1 and case["kind"] == "thermal":  # the cells' matrices do not change from call to call
        f = cells * npe * npe * 4
    elif jac:
        f += cells * npe * npe * 2 * (d if p == 1 else 2 * d * (p + 1))
    return b, f


def work(case):
    if case["what"] == "apply":
        nodes, _, nnz = _counts(3, case["order"], (case["nx"], case["ny"], case["nz"]))
        return {"bytes": nnz * (4 if case["precision"] == "mixed" else 8) + 16 * nodes, "flops": 2 * nnz}
    if case["what"] == "newton":
        # five Newton steps, each a residual, a Jacobian and four products with it
        e = case["edge"]
        c, w = {"order": 1, "kind": case["kind"]}, 4 if case["precision"] == "mixed" else 8
        b, f = _assembly_work(c, (e, e, e), True, w)
        _, _, nnz = _counts(3, 1, (e, e, e))
        return {"bytes": 5 * (b + 4 * nnz * w), "flops": 5 * (f + 8 * nnz)}
    if case["what"] == "subgrid":
        m = 0.5 * (case["least"] + case["most"])
        nodes, cells, nnz = _counts(3, 1, (m, m, m))
        # kappa and boundary data in, solution and matrix out; forty operator products a problem
        return {"bytes": case["problems"] * (8 * cells + 16 * nodes + 4 * nnz), "flops": case["problems"] * 40 * 2 * nnz}
    b, f = _assembly_work(case, [case["nx"], case["ny"], case["nz"]][:case["dim"]], case["call"] != "res",
                          4 if case["precision"] == "mixed" else 8)
    return {"bytes": b, "flops": f}


# ---- the same in plain torch, 64 bits -----------------------------------------------------------
def _axis(m, p):
    """First coupled node and number of coupled nodes of each node along an axis of m cells, and their total."""
    if not isinstance(m, int):
        return None, None, (p + 1) * (p + 1) * m - (m - 1)
    i = np.arange(p * m + 1)
    first = np.where(i % p == 0, np.maximum(i // p - 1, 0), i // p)
    last = np.minimum(i // p, m - 1)
    count = p * (last - first) + p + 1
    return p * first, count, int(count.sum())


class _Mesh:
    """Numbering of a structured mesh: x fastest, columns of a row ascending."""

    def __init__(self, n, p, faces, device):
        d = len(n)
        self.n, self.p, self.d = list(n), p, d
        self.axes = [_axis(m, p) for m in n] + [(np.zeros(1, int), np.ones(1, int), 1)] * (3 - d)
        t = lambda a: torch.tensor(a, device=device, dtype=torch.int64)  # noqa: E731
        self.first, self.count = [t(a[0]) for a in self.axes], [t(a[1]) for a in self.axes]
        self.nn = [len(a[0]) for a in self.axes]
        iz, iy, ix = torch.meshgrid(*[torch.arange(m, device=device) for m in reversed(self.nn)], indexing="ij")
        self.at = [v.reshape(-1) for v in (ix, iy, iz)]
        length = self.count[0][self.at[0]] * self.count[1][self.at[1]] * self.count[2][self.at[2]]
        self.row_ptr = torch.zeros(length.numel() + 1, dtype=torch.int64, device=device)
        self.row_ptr[1:] = torch.cumsum(length, 0)
        self.fixed = torch.zeros(length.numel(), dtype=torch.bool, device=device)
        for k in range(d):
            for side, at in ((0, 0), (1, self.nn[k] - 1)):
                if faces >> (2 * k + side) & 1:
                    self.fixed |= self.at[k] == at

    def place(self, row, col):
        """Place of (row, col) in the values of the matrix."""
        at = [(self.at[k][col] - self.first[k][self.at[k][row]]) for k in range(3)]
        c = [self.count[k][self.at[k][row]] for k in range(3)]
        return self.row_ptr[row] + (at[2] * c[1] + at[1]) * c[0] + at[0]

    def columns(self):
        rows = torch.repeat_interleave(torch.arange(self.row_ptr.numel() - 1, device=self.row_ptr.device), self.row_ptr.diff())
        k = torch.arange(rows.numel(), device=rows.device) - self.row_ptr[rows]
        c0, c1 = self.count[0][self.at[0][rows]], self.count[1][self.at[1][rows]]
        x = self.first[0][self.at[0][rows]] + k % c0
        y = self.first[1][self.at[1][rows]] + k // c0 % c1
        z = self.first[2][self.at[2][rows]] + k // (c0 * c1)
        return x + self.nn[0] * (y + self.nn[1] * z)


def _basis(p, d, points):
    """Values and reference derivatives of the equispaced Lagrange basis at the tensor points: [q, i], [q, i, d]."""
    nodes = np.linspace(-1.0, 1.0, p + 1)
    poly = [np.poly1d(np.poly(np.delete(nodes, a)) / np.prod(nodes[a] - np.delete(nodes, a))) for a in range(p + 1)]
    v, dv = np.array([[f(x) for f in poly] for x in points]), np.array([[f.deriv()(x) for f in poly] for x in points])

    def product(tables):
        t = tables[0]
        for s in tables[1:]:  # the later axis is the slower index
            t = np.einsum("ai,bj->baji", t, s).reshape(t.shape[0] * s.shape[0], -1)
        return t

    return product([v] * d), np.stack([product([dv if k == m else v for k in range(d)]) for m in range(d)], -1)


def _fe(cfg, u, jac, mesh, flux=None):
    """Residual and Jacobian values by quadrature over every cell."""
    dev, d, p, n = u.device, cfg["dim"], cfg["order"], cfg["n"]
    t = lambda a: torch.tensor(np.ascontiguousarray(a), device=dev, dtype=torch.float64)  # noqa: E731
    gx, gw = np.polynomial.legendre.leggauss(p + 1)
    w = gw
    for _ in range(d - 1):
        w = np.outer(gw, w).reshape(-1)
    w = t(w)
    phi, dphi = (t(a) for a in _basis(p, d, gx))
    psi, dpsi = (t(a) for a in _basis(1, d, gx))
    cells = math.prod(n)
    r = torch.zeros(u.numel(), dtype=torch.float64, device=dev)
    J = torch.zeros(int(mesh.row_ptr[-1]), dtype=torch.float64, device=dev) if jac else None
    vert = torch.stack([v.reshape(-1) for v in torch.meshgrid(*[torch.arange(m + 1, device=dev) for m in reversed(n)], indexing="ij")][::-1], 1)
    if "vertex_coords" in cfg:
        coords = t(cfg["vertex_coords"])
    else:
        lo, hi = t(cfg["lo"]), t(cfg["hi"])
        coords = lo + (hi - lo) * vert / torch.tensor(n, device=dev)
    kappa = t(cfg["kappa"]).reshape(-1) if not np.isscalar(cfg["kappa"]) else None
    form, amp, freq = cfg["source"]

    def local(q, q1, nn, step):
        at = [step * c[:, None] + (torch.arange(q, device=dev) // q1 ** k % q1)[None, :] for k, c in enumerate(cc)]
        return at[0] + nn[0] * (at[1] + (nn[1] * at[2] if d == 3 else 0))

    npe = phi.shape[1]
    chunk = max(256, int(3e7 / (npe * npe * (3 if jac else 1))))
    for c0 in range(0, cells, chunk):
        c = torch.arange(c0, min(cells, c0 + chunk), device=dev)
        cc = [c % n[0], c // n[0] % n[1], c // (n[0] * n[1])][:d]
        x = coords[local(2 ** d, 2, [m + 1 for m in n], 1)]
        lid = local(npe, p + 1, mesh.nn, p)
        G = torch.einsum("cvk,qvm->cqkm", x, dpsi)
        inv, wq = torch.linalg.inv(G), w * torch.linalg.det(G).abs()
        gp = torch.einsum("qim,cqmk->cqik", dphi, inv)
        ue = u[lid]
        T, dT = ue @ phi.T, torch.einsum("ci,cqik->cqk", ue, gp)
        k = kappa[c][:, None].expand_as(T) if cfg["kind"] == "thermal" else 1.0 + T * T
        f = torch.full_like(T, amp)
        if form == "sinprod":
            f = amp * torch.prod(torch.sin(freq * torch.einsum("cvk,qv->cqk", x, psi)), -1)
        flow = torch.einsum("cqik,cqk->cqi", gp, dT)
        res = torch.einsum("cqi,cq->ci", flow, wq * k) - (wq * f) @ phi
        free = ~mesh.fixed[lid]
        r.index_add_(0, lid.reshape(-1), torch.where(free, -res, 0.0).reshape(-1))
        if jac:
            a = gp.permute(0, 2, 1, 3).reshape(len(c), npe, -1)
            K = torch.bmm(a * (wq * k)[:, None, :, None].expand(-1, npe, -1, d).reshape(len(c), npe, -1), a.transpose(1, 2))
            if cfg["kind"] != "thermal":
                K += torch.matmul((flow * (wq * 2.0 * T)[..., None]).transpose(1, 2), phi)
            rows, cols = lid[:, :, None].expand_as(K), lid[:, None, :].expand_as(K)
            J.index_add_(0, mesh.place(rows, cols)[free].reshape(-1), K[free].reshape(-1))
    for face, g in (flux or {}).items():  # the y faces of a rectangle
        v, _ = _basis(p, 1, gx)
        g = t(g).reshape(n[0], p + 1) * t(gw) * (0.5 * (cfg["hi"][0] - cfg["lo"][0]) / n[0])
        lid = p * torch.arange(n[0], device=dev)[:, None] + torch.arange(p + 1, device=dev) + (face - 2) * mesh.nn[0] * (mesh.nn[1] - 1)
        r.index_add_(0, lid.reshape(-1), torch.where(mesh.fixed[lid], 0.0, g @ t(v)).reshape(-1))
    if jac:
        at = mesh.fixed.nonzero().reshape(-1)
        J[mesh.place(at, at)] = 1.0
    return r, J


def _solve(row_ptr, col, J, diag, b, symmetric):
    """Jacobi-preconditioned CG, or BiCGStab, to the rounding of 64 bits; x = 0 where b is 0 on identity rows."""
    A = torch.sparse_csr_tensor(row_ptr, col, J, size=(b.numel(), b.numel()))
    x, r = torch.zeros_like(b), b.clone()
    stop = 1e-15 * float(b.norm())
    if symmetric:
        z = r / diag
        s, rz = z.clone(), torch.dot(r, z)
        for _ in range(6000):
            q = A @ s
            a = rz / torch.dot(s, q)
            x, r = x + a * s, r - a * q
            if float(r.norm()) <= stop:
                break
            z = r / diag
            rz, old = torch.dot(r, z), rz
            s = z + (rz / old) * s
        return x
    r0, s, v = r.clone(), torch.zeros_like(b), torch.zeros_like(b)
    rho = alpha = omega = torch.ones((), dtype=b.dtype, device=b.device)
    for _ in range(6000):
        rho, old = torch.dot(r0, r), rho
        s = r + (rho / old) * (alpha / omega) * (s - omega * v)
        y = s / diag
        v = A @ y
        alpha = rho / torch.dot(r0, v)
        h = r - alpha * v
        z = h / diag
        w = A @ z
        omega = torch.dot(w, h) / torch.dot(w, w)
        x, r = x + alpha * y + omega * z, h - omega * w
        if not float(r.norm()) > stop:
            break
    return x


def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if case["what"] == "apply":
        J, x = _apply_inputs(case, seed, dev)
        mesh = _Mesh((case["nx"], case["ny"], case["nz"]), case["order"], X_FACES, dev)
        A = torch.sparse_csr_tensor(mesh.row_ptr, mesh.columns(), J.double(), size=(x.numel(), x.numel()))
        return {"y": A @ x}
    if case["what"] == "newton":
        cfg, u0 = _newton_inputs(case, seed)
        u = torch.tensor(u0, device=dev)
        mesh = _Mesh(cfg["n"], 1, cfg["dirichlet_faces"], dev)
        u[mesh.fixed] = 0.0
        col, at = mesh.columns(), torch.arange(u.numel(), device=dev)
        scale = None
        for _ in range(12):
            r, J = _fe(cfg, u, True, mesh)
            size = float(r.abs().max())
            scale = scale or size
            if size <= 1e-14 * scale:
                break
            u = u + _solve(mesh.row_ptr, col, J, J[mesh.place(at, at)], r, case["kind"] == "thermal")
        return {"u": u}
    if case["what"] == "subgrid":
        rows, cols, vals, us, rs, base = [], [], [], [], [], 0
        for s, kap, dbc in zip(*_subgrid_inputs(case, seed)):
            s = [int(v) for v in s]
            cfg = {"dim": 3, "order": 1, "n": s, "lo": (0.0,) * 3, "hi": (1.0,) * 3, "kind": "thermal",
                   "source": ("const", 1.0, 0.0), "kappa": kap}
            mesh = _Mesh(s, 1, L.MRG_FACE_ALL, dev)
            u = torch.where(mesh.fixed, torch.tensor(dbc, device=dev), 0.0)
            r, J = _fe(cfg, u, True, mesh)
            rows.append(mesh.row_ptr.diff())
            cols.append(mesh.columns() + base)
            vals.append(J)
            us.append(u)
            rs.append(r)
            base += u.numel()
        length, col, J, u, b = (torch.cat(v) for v in (rows, cols, vals, us, rs))
        row_ptr = torch.zeros(base + 1, dtype=torch.int64, device=dev)
        row_ptr[1:] = torch.cumsum(length, 0)
        row = torch.repeat_interleave(torch.arange(base, device=dev), length)
        diag = torch.zeros(base, dtype=torch.float64, device=dev)
        diag[row[row == col]] = J[row == col]
        return {"u": u + _solve(row_ptr, col, J, diag, b, True), "J": J}
    cfg, u, flux = _inputs(case, seed)
    mesh = _Mesh(cfg["n"], cfg["order"], cfg["dirichlet_faces"], dev)
    r, J = _fe(cfg, torch.tensor(u, device=dev), case["call"] != "res", mesh, flux)
    return {"r": r} if J is None else {"r": r, "J": J}
