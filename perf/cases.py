"""The work that is measured: what a program using this package has it do, through its public entry points.

Seven kinds of work, each at sizes from a few hundred unknowns to the 3.09M of the largest workload:

* ``spmv``     one FP64 product with an assembled, constrained stiffness matrix (FEMSolver.matvec_device): the
               inner step of a caller's own iteration;
* ``solve``    FEMSolver.solve for a new load vector (``assemble`` False), or the whole analysis of a new stiffness
               field: zeros, assembleStiffness, setRHS, solve (``assemble`` True);
* ``plugin``   linear_solver_crs: the LinearSolver hook, a host CRS system in, x out;
* ``adjoint``  u(E) and dL/dE of every element's modulus (ElasticOperator under torch.autograd);
* ``newmark``  one step of SeismicAnalysis.LinearReyleighNewmark;
* ``eig``      FEMSolver.eig, LOBPCG for the lowest modes;
* ``batch``    FEMSolverBatch.solve: many thin slabs of uneven sizes in one launch.

Meshes are Cube3D boxes with element sizes 1/max(nx, ny, nz); moduli are lognormal per element (sigma 0 is a uniform
material), loads and fields come from the seed.  Tolerances are the workloads' own (1e-10, 1e-8 for the slabs),
or ten times tighter where a solution that just meets them is less sure than its digits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

NU = 0.3
RHO = 1.0e3
DT = 1.0e-3
GAMMA, BETA, RAY_A, RAY_B = 0.5, 0.25, 0.524, 0.00129


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a caller's own iteration on a small part: latency counts
        dict(name="spmv_small", kind="spmv", nx=12, ny=10, nz=9, sigma=0.5),
        # the same on a mesh whose matrix is far larger than any cache
        dict(name="spmv_large", kind="spmv", nx=96, ny=90, nz=84, sigma=0.5),
        # the plain drop-in: 20^3, uniform material, unpreconditioned FP64 BiCGSTAB with the reference's stop rule
        dict(name="analysis_20_bicgstab", kind="solve", nx=20, ny=20, nz=20, sigma=0.0, algorithm="BiCGSTAB",
             precision="fp64", pc="None", storage="full", stop="reference", tol=1e-11, assemble=True),
        # a small organ mesh re-analysed with a new stiffness field, mixed precision
        dict(name="analysis_17_cg_mixed", kind="solve", nx=17, ny=15, nz=13, sigma=0.5, algorithm="CG",
             precision="mixed", pc="BlockJacobi", storage="symmetric", stop="true_relative", tol=1e-10, assemble=True),
        # an ordinary mesh, several load cases, all FP64
        dict(name="solve_50_cg_fp64", kind="solve", nx=52, ny=48, nz=45, sigma=0.5, algorithm="CG",
             precision="fp64", pc="BlockJacobi", storage="full", stop="true_relative", tol=1e-10, assemble=False),
        # the largest workload: 100^3, 3.09M unknowns, mixed CG from the symmetric copy
        dict(name="solve_100_cg_mixed", kind="solve", nx=100, ny=100, nz=100, sigma=0.5, algorithm="CG",
             precision="mixed", pc="BlockJacobi", storage="symmetric", stop="true_relative", tol=1e-10,
             assemble=False),
        # the mixed BiCGSTAB form at an ordinary size
        dict(name="solve_44_bicgstab_mixed", kind="solve", nx=44, ny=43, nz=41, sigma=0.5, algorithm="BiCGSTAB",
             precision="mixed", pc="BlockJacobi", storage="symmetric", stop="true_relative", tol=1e-11,
             assemble=False),
        # the solver hook called by another program with its own (page-locked) CRS arrays
        dict(name="plugin_33", kind="plugin", nx=36, ny=33, nz=31, sigma=0.5, algorithm="CG", precision="mixed",
             pc="BlockJacobi", storage="symmetric", stop="true_relative", tol=1e-10),
        # stiffness identification: 64^3, 262,144 moduli, forward and backward at the operator's default tolerance
        dict(name="adjoint_64_mixed", kind="adjoint", nx=64, ny=64, nz=64, sigma=0.5, precision="mixed", tol=1e-12),
        # time stepping of the 60^3 cantilever, FP64
        dict(name="newmark_60_fp64", kind="newmark", nx=60, ny=60, nz=60, sigma=0.0, precision="fp64",
             storage="full", tol=1e-11),
        # lowest modes of a cantilever beam, FP32 phase and then double-float
        dict(name="eig_40_mixed", kind="eig", nx=40, ny=26, nz=20, sigma=0.2, precision="mixed", nev=8, block=12,
             tol=1e-9),
        # uneven organs in one persistent launch
        dict(name="batch_256_fp64", kind="batch", count=256, mesh_seed=5, lo=8, hi=40, sigma=0.5, precision="fp64",
             tol=1e-8),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _box(rng, lo, hi):
    return dict(nx=_log(rng, lo, hi), ny=_log(rng, lo, hi), nz=_log(rng, lo, hi))


def draw(rng):
    kind = rng.choice(["spmv", "solve", "solve", "solve", "plugin", "adjoint", "newmark", "eig", "batch"])
    sigma = rng.choice([0.0, 0.3, 0.5])
    if kind == "spmv":
        return dict(kind=kind, sigma=sigma, **_box(rng, 6, 96))
    if kind == "solve":
        alg = rng.choice(["CG", "CG", "BiCGSTAB"])
        if rng.random() < 0.45:
            pc = rng.choice(["BlockJacobi", "BlockJacobi", "PointJacobi", "None"])
            stop = "reference" if alg == "BiCGSTAB" and pc == "None" else "true_relative"
            return dict(kind=kind, sigma=sigma, algorithm=alg, precision="fp64", pc=pc, storage="full", stop=stop,
                        tol=1e-10 if alg == "CG" else 1e-11, assemble=rng.random() < 0.5, **_box(rng, 6, 56))
        return dict(kind=kind, sigma=sigma, algorithm=alg, precision="mixed", pc="BlockJacobi",
                    storage=rng.choice(["full", "symmetric", "symmetric"]), stop="true_relative",
                    tol=1e-10 if alg == "CG" else 1e-11, assemble=rng.random() < 0.5, **_box(rng, 6, 72))
    if kind == "plugin":
        return dict(kind=kind, sigma=sigma, algorithm="CG", precision=rng.choice(["mixed", "mixed", "fp64"]),
                    pc="BlockJacobi", storage="symmetric", stop="true_relative", tol=1e-10, **_box(rng, 6, 44))
    if kind == "adjoint":
        return dict(kind=kind, sigma=0.5, precision=rng.choice(["mixed", "fp64"]), tol=1e-12, **_box(rng, 8, 52))
    if kind == "newmark":
        prec = rng.choice(["fp64", "mixed"])
        return dict(kind=kind, sigma=0.0, precision=prec, storage="full" if prec == "fp64" else "symmetric",
                    tol=1e-11, **_box(rng, 8, 60))
    if kind == "eig":
        nz = _log(rng, 6, 18)
        return dict(kind=kind, sigma=0.2, precision="mixed", nev=rng.randint(4, 8), block=12, tol=1e-9,
                    nx=2 * nz + rng.randint(0, 5), ny=nz + rng.randint(2, 6), nz=nz)
    return dict(kind=kind, sigma=0.5, count=_log(rng, 12, 200), mesh_seed=rng.randint(1, 10 ** 6), lo=8,
                hi=rng.choice([20, 30, 40]), precision="fp64", tol=1e-8)


# ------------------------------------------------------------ inputs (the seed's)
def _cell(c):
    return 1.0 / max(c["nx"], c["ny"], c["nz"])


def _ne(c):
    return c["nx"] * c["ny"] * c["nz"]


def _nn(c):
    return (c["nx"] + 1) * (c["ny"] + 1) * (c["nz"] + 1)


def _moduli(c, ne, seed, salt=0):
    rng = np.random.default_rng([seed, salt, 11])
    if c["sigma"] == 0.0:  # one material: its modulus is the seed's
        return np.full(ne, 1.0e4 * rng.uniform(0.5, 2.0))
    return np.exp(rng.normal(math.log(1.0e4), c["sigma"], size=ne))


def _grid(nx, ny, nz):
    """Integer coordinates (x fastest) of the nodes of a Cube3D box."""
    k, j, i = np.meshgrid(np.arange(nz + 1), np.arange(ny + 1), np.arange(nx + 1), indexing="ij")
    return i.ravel(), j.ravel(), k.ravel()


def _top_load(nx, ny, nz, h, t):
    """Consistent nodal loads of a uniform traction t (3 components) on the top face."""
    i, j, k = _grid(nx, ny, nz)
    w = np.where((i == 0) | (i == nx), 0.5, 1.0) * np.where((j == 0) | (j == ny), 0.5, 1.0) * (k == nz) * h * h
    return (w[:, None] * np.asarray(t, dtype=np.float64)[None, :]).reshape(-1)


def _load(c, seed):
    rng = np.random.default_rng([seed, 12])
    return _top_load(c["nx"], c["ny"], c["nz"], _cell(c), [0.2 * rng.normal(), 0.2 * rng.normal(), -1.0])


def _ground(c, seed):
    rng = np.random.default_rng([seed, 14])
    return np.tile([2.0 * rng.normal(), 2.0 * rng.normal(), -9.8 + rng.normal()], _nn(c))


def _slabs(c):
    """(nx, ny, nz, clamped axis) of each slab: one short edge is clamped."""
    rng = np.random.default_rng(c["mesh_seed"])
    nx = rng.integers(c["lo"], c["hi"] + 1, size=c["count"])
    ny = rng.integers(c["lo"], c["hi"] + 1, size=c["count"])
    nz = rng.integers(1, 4, size=c["count"])
    return [(int(a), int(b), int(d), 0 if a <= b else 1) for a, b, d in zip(nx, ny, nz)]


def _clamped(nx, ny, nz, axis):
    """0-based unknowns of the nodes on the box's face x = 0, y = 0 or z = 0."""
    nodes = np.nonzero(_grid(nx, ny, nz)[axis] == 0)[0]
    return (3 * nodes[:, None] + np.arange(3)[None, :]).reshape(-1)


# ------------------------------------------------------- what a program keeps
def _domain(nx, ny, nz, h):
    from plantfem_gb300 import FEMDomain
    return FEMDomain().create("Cube3D", x_num=nx, y_num=ny, z_num=nz, x_len=nx * h, y_len=ny * h, z_len=nz * h)


def _solver(c, seed, axis=2, assembled=True):
    from plantfem_gb300 import FEMSolver
    s = FEMSolver()
    s.setDomain(_domain(c["nx"], c["ny"], c["nz"], _cell(c)))
    s.setCRS(3)
    E = _moduli(c, _ne(c), seed)
    if assembled:
        s.assembleStiffness(E, np.full(E.shape, NU))
    s.fix(1, (_clamped(c["nx"], c["ny"], c["nz"], axis) + 1).astype(np.int32), FixValue=0.0)
    return s, E


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "spmv":
        s, _ = _solver(c, seed)
        s.eliminate()
        g = torch.Generator(device="cpu").manual_seed(seed)
        x = torch.randn(3 * _nn(c), dtype=torch.float64, generator=g).cuda()
        return dict(kind=kind, s=s, x=x, y=torch.empty_like(x))
    if kind == "solve":
        s, E = _solver(c, seed, assembled=not c["assemble"])
        s.relative_er = c["tol"]
        s.er0 = 1e-15  # the reference rule also stops on |r| < er0: here the relative part decides
        kw = dict(algorithm=c["algorithm"], preconditioning=c["pc"], precision=c["precision"], storage=c["storage"],
                  stop_rule=c["stop"])
        return dict(kind=kind, s=s, E=E, nu=np.full(E.shape, NU), rhs=_load(c, seed), kw=kw, assemble=c["assemble"])
    if kind == "plugin":
        s, _ = _solver(c, seed)
        s.setRHS(_load(c, seed))
        s.eliminate()
        pin = [torch.from_numpy(a).pin_memory() for a in (*s.getCRS(), s.CRS_RHS)]
        x = torch.zeros(3 * _nn(c), dtype=torch.float64).pin_memory()
        s.remove()
        kw = dict(algorithm=c["algorithm"], precision=c["precision"], preconditioning=c["pc"], relative_er=c["tol"],
                  stop_rule=c["stop"], storage=c["storage"])
        return dict(kind=kind, pin=pin, xpin=x, args=[t.numpy() for t in pin], x=x.numpy(), kw=kw)
    if kind == "adjoint":
        from plantfem_gb300.adjoint import ElasticOperator
        dom = _domain(c["nx"], c["ny"], c["nz"], _cell(c))
        op = ElasticOperator(dom, NU, _load(c, seed), _clamped(c["nx"], c["ny"], c["nz"], 2) + 1,
                             precision=c["precision"], relative_er=c["tol"])
        # the measured displacements: those of another stiffness field
        target = op.displacement(torch.as_tensor(_moduli(c, _ne(c), seed, 1), device="cuda")).detach()
        return dict(kind=kind, op=op, E=torch.as_tensor(_moduli(c, _ne(c), seed), device="cuda"), target=target)
    if kind == "newmark":
        from plantfem_gb300 import SeismicAnalysis
        dom = _domain(c["nx"], c["ny"], c["nz"], _cell(c))
        ne = _ne(c)
        sa = SeismicAnalysis().init(dom, np.full(ne, RHO), _moduli(c, ne, seed), np.full(ne, NU))
        sa.dt = DT
        nodes = np.nonzero(_grid(c["nx"], c["ny"], c["nz"])[0] == 0)[0] + 1
        for d in "xyz":
            sa.fixDisplacement(nodes, d, 0.0)
        sa.A_ext[:] = 0.0
        sa.LinearReyleighNewmark(TOL=c["tol"], precision=c["precision"], storage=c["storage"])  # set-up, at rest
        sa.A_ext[:] = _ground(c, seed)
        return dict(kind=kind, sa=sa, kw=dict(TOL=c["tol"], precision=c["precision"], storage=c["storage"]))
    if kind == "eig":
        s, E = _solver(c, seed, axis=0, assembled=False)
        s.assembleMass(np.full(E.shape, RHO))
        s.keepThisMatrixAs("B")
        s.zeros()
        s.assembleStiffness(E, np.full(E.shape, NU))
        s.keepThisMatrixAs("A")
        s.fix_eig((_clamped(c["nx"], c["ny"], c["nz"], 0) + 1).astype(np.int32))
        s.use_LOBPCG = True
        s.LOBPCG_TOL = c["tol"]
        s.LOBPCG_MAX_ITR = 3000
        return dict(kind=kind, s=s, nev=c["nev"], kw=dict(block_size=c["block"], precision=c["precision"]),
                    phase=_phase(c))
    if kind == "batch":
        from plantfem_gb300 import FEMSolver, FEMSolverBatch
        solvers = []
        for n, (nx, ny, nz, axis) in enumerate(_slabs(c)):
            h = 1.0 / max(nx, ny)
            s = FEMSolver()
            s.setDomain(_domain(nx, ny, nz, h))
            s.setCRS(3)
            E = _moduli(c, nx * ny * nz, seed, n)
            s.assembleStiffness(E, np.full(E.shape, NU))
            s.setRHS(_top_load(nx, ny, nz, h, [0.0, 0.0, -1.0]))
            s.fix(1, (_clamped(nx, ny, nz, axis) + 1).astype(np.int32), FixValue=0.0)
            solvers.append(s)
        b = FEMSolverBatch(solvers)
        b.config = {"threads": 512, "cluster": 2, "team_fraction": 0.0625}  # what tune() picks on these workloads
        return dict(kind=kind, batch=b, kw=dict(precision=c["precision"], relative_er=c["tol"]))
    raise ValueError(kind)


def _phase(c):
    """Weights that fix the sign of a mode: its weighted sum is made positive."""
    return np.random.default_rng(99).uniform(0.5, 1.5, 3 * _nn(c)) * np.tile([1.0, 1.7, 2.3], _nn(c))


# ------------------------------------------------------------------- one pass
def run(state):
    kind = state["kind"]
    if kind == "spmv":
        return state["s"].matvec_device(state["x"], state["y"])
    if kind == "solve":
        s = state["s"]
        if state["assemble"]:
            s.zeros()
            s.assembleStiffness(state["E"], state["nu"])
        s.setRHS(state["rhs"])
        return s.solve(**state["kw"])
    if kind == "plugin":
        from plantfem_gb300 import linear_solver_crs
        state["x"].fill(0.0)
        linear_solver_crs(*state["args"], state["x"], **state["kw"])
        return state["x"]
    if kind == "adjoint":
        E = state["E"].detach().clone().requires_grad_(True)
        u = state["op"].displacement(E)
        loss = 0.5 * torch.sum((u - state["target"]) ** 2)
        loss.backward()
        return {"u": u.detach(), "loss": loss.detach(), "dE": E.grad}
    if kind == "newmark":
        sa = state["sa"]
        sa.LinearReyleighNewmark(**state["kw"])
        return {"u": sa.U, "v": sa.V, "a": sa.A}
    if kind == "eig":
        lam, X = state["s"].eig(state["nev"], **state["kw"])
        return {"lam": lam, "modes": X * np.sign(state["phase"] @ X)}
    if kind == "batch":
        return np.concatenate(state["batch"].solve(**state["kw"]))
    raise ValueError(kind)


# ------------------------------------------------------ what a pass cannot avoid
def _blocks(nx, ny, nz):
    """3x3 blocks of the node graph: neighbours along each axis multiply."""
    return (3 * nx + 1) * (3 * ny + 1) * (3 * nz + 1)


def work(case):
    """Bytes and operations of one pass.  For the iterative kinds: one read of the matrix and of five vectors per
    iteration, at the iteration counts these workloads take (they grow with the mesh's largest side)."""
    c, kind = case, case["kind"]
    if kind == "batch":
        by = fl = 0.0
        for nx, ny, nz, _ in _slabs(c):
            nb, nn = _blocks(nx, ny, nz), (nx + 1) * (ny + 1) * (nz + 1)
            it = 16.0 * max(nx, ny)
            by += 76.0 * nb + 24.0 * nn * 6  # a system is small enough to stay on chip: its matrix is read once
            fl += it * (18.0 * nb + 42.0 * nn)
        return {"bytes": by, "flops": fl}
    nb, nn, ne = _blocks(c["nx"], c["ny"], c["nz"]), _nn(c), _ne(c)
    n = max(c["nx"], c["ny"], c["nz"])
    if kind == "spmv":
        return {"bytes": 76.0 * nb + 48.0 * nn, "flops": 18.0 * nb}
    if kind == "newmark":
        return {"bytes": 22 * (76.0 * nb + 120.0 * nn) + 4 * 24.0 * nn, "flops": 24 * 18.0 * nb}
    if kind == "eig":
        m, it = c["block"], 8.0 * n
        return {"bytes": it * (2 * 40.0 * nb + 12 * m * 12.0 * nn),
                "flops": it * (2 * 18.0 * nb * m + 3.0 * nn * (2 * 9.0 * m * m + 6 * 3.0 * m * m))}
    half = c["precision"] == "mixed"
    sym = half and c.get("storage", "symmetric") == "symmetric"
    per = (20.0 if sym else 40.0 if half else 76.0) * nb + (60.0 if half else 120.0) * nn
    it = 17.0 * n * (2.6 if c.get("algorithm") == "BiCGSTAB" else 1.0)
    by, fl = it * per, it * 18.0 * nb
    if kind == "adjoint":
        by, fl = 2 * by, 2 * fl
    if kind == "plugin":
        by += 9 * 12.0 * nb + 3 * 24.0 * nn
    if kind == "adjoint" or c.get("assemble"):
        by, fl = by + 72.0 * nb + 8.0 * ne, fl + 9000.0 * ne
    return {"bytes": by, "flops": fl}


# ------------------------------------------------- the same results in 64 bits
_SIGNS = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]],
                  dtype=np.float64)


def _element(h):
    """(stiffness at E = 1, mass at rho = 1) of a cube of side h, 2 x 2 x 2 Gauss points: 24 x 24 each."""
    lam, mu = NU / (1 + NU) / (1 - 2 * NU), 1.0 / 2.0 / (1 + NU)
    D = np.diag([2 * mu] * 3 + [mu] * 3)
    D[:3, :3] += lam
    K, M = np.zeros((24, 24)), np.zeros((24, 24))
    for g in _SIGNS / math.sqrt(3.0):
        one = 1.0 + _SIGNS * g[None, :]
        N = 0.125 * one.prod(axis=1)
        dN = 0.125 * _SIGNS * np.stack([one[:, 1] * one[:, 2], one[:, 0] * one[:, 2], one[:, 0] * one[:, 1]], axis=1)
        dN = dN * (2.0 / h)
        B = np.zeros((6, 24))
        for a in range(8):
            x, y, z = dN[a]
            B[:, 3 * a:3 * a + 3] = [[x, 0, 0], [0, y, 0], [0, 0, z], [y, x, 0], [0, z, y], [z, 0, x]]
        w = (h / 2.0) ** 3
        K += w * B.T @ D @ B
        M += w * np.kron(np.outer(N, N), np.eye(3))
    return K, M


def _conn(nx, ny, nz):
    """Node numbers (0-based) of every element, the order of a Cube3D box."""
    k, j, i = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    b = (i + (nx + 1) * (j + (ny + 1) * k)).ravel()
    q = np.stack([b, b + 1, b + nx + 2, b + nx + 1], axis=1)
    return np.concatenate([q, q + (nx + 1) * (ny + 1)], axis=1)


class _Operator:
    """sum_e scale_e Ke in FP64, element by element, constrained unknowns removed; systems side by side have a
    number of their own in ``part``, so that each has its own iteration."""

    def __init__(self, conn, scale, Ke, nn, fixed, part=None, parts=1):
        dev = "cuda" if torch.cuda.is_available() else "cpu"
        t = lambda a, d=torch.float64: torch.as_tensor(a, dtype=d, device=dev)  # noqa: E731
        self.conn, self.scale, self.Ke, self.nn = t(conn, torch.int64), t(scale), t(Ke), nn
        self.free = torch.ones(3 * nn, dtype=torch.float64, device=dev)
        self.free[t(fixed, torch.int64)] = 0.0
        self.part = torch.zeros(3 * nn, dtype=torch.int64, device=dev) if part is None else t(part, torch.int64)
        self.parts = parts
        d = torch.zeros(nn, 3, dtype=torch.float64, device=dev)
        d.index_add_(0, self.conn.reshape(-1), (self.scale[:, None] * torch.diagonal(self.Ke)).reshape(-1, 3))
        self.dinv = self.free / d.reshape(-1)

    def full(self, x):
        xe = x.reshape(self.nn, 3)[self.conn].reshape(-1, 24)
        y = torch.zeros(self.nn, 3, dtype=torch.float64, device=x.device)
        y.index_add_(0, self.conn.reshape(-1), ((xe @ self.Ke) * self.scale[:, None]).reshape(-1, 3))
        return y.reshape(-1)

    def __call__(self, x):
        return self.full(x) * self.free

    def dot(self, a, b):
        if self.parts == 1:
            return torch.dot(a, b).reshape(1)
        return torch.zeros(self.parts, dtype=torch.float64, device=a.device).index_add_(0, self.part, a * b)

    def solve(self, b, passes=3, most=6000):
        """x with self(x) = b on the free unknowns: Jacobi CG, restarted from the true residual."""
        b = b * self.free
        x = torch.zeros_like(b)
        per = (lambda v: v) if self.parts == 1 else (lambda v: v[self.part])
        for n in range(passes):
            r = b - self(x)
            r0 = self.dot(r, r)
            z = self.dinv * r
            p, rho = z, self.dot(r, z)
            d = torch.zeros_like(b)
            for k in range(most):
                q = self(p)
                pq = self.dot(p, q)
                a = torch.where(pq > 0, rho / pq, torch.zeros_like(pq))
                d = d + per(a) * p
                r = r - per(a) * q
                z = self.dinv * r
                new = self.dot(r, z)
                p = z + per(torch.where(rho > 0, new / rho, torch.zeros_like(rho))) * p
                rho = new
                if k % 50 == 49 and bool((self.dot(r, r) <= (1e-13 if n == 0 else 1e-5) ** 2 * r0).all()):
                    break
            x = x + d
        return x


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "batch":
        return _exact_batch(c, seed)
    if kind == "eig":
        return _exact_eig(c, seed)
    K, M = _element(_cell(c))
    conn, nn = _conn(c["nx"], c["ny"], c["nz"]), _nn(c)
    E = _moduli(c, _ne(c), seed)
    op = _Operator(conn, E, K, nn, _clamped(c["nx"], c["ny"], c["nz"], 0 if kind == "newmark" else 2))
    dev = op.Ke.device
    if kind == "spmv":
        g = torch.Generator(device="cpu").manual_seed(seed)
        x = torch.randn(3 * nn, dtype=torch.float64, generator=g).to(dev)
        return op(x * op.free) + (1.0 - op.free) * x  # unit rows at the constrained unknowns
    if kind in ("solve", "plugin"):
        return op.solve(torch.as_tensor(_load(c, seed), device=dev)).cpu().numpy()
    if kind == "adjoint":
        u = op.solve(torch.as_tensor(_load(c, seed), device=dev))
        other = _Operator(conn, _moduli(c, _ne(c), seed, 1), K, nn, _clamped(c["nx"], c["ny"], c["nz"], 2))
        w = u - other.solve(torch.as_tensor(_load(c, seed), device=dev))
        lam = op.solve(w)
        ue, le = (v.reshape(nn, 3)[op.conn].reshape(-1, 24) for v in (u, lam))
        return {"u": u, "loss": 0.5 * torch.sum(w * w), "dE": -torch.sum(le * (ue @ op.Ke), dim=1)}
    # newmark, from rest: (cM M + cK K) u = M a_ext, E is one value
    cM = 1.0 / (BETA * DT * DT) + GAMMA / (BETA * DT) * RAY_A
    cK = 1.0 + GAMMA / (BETA * DT) * RAY_B
    op = _Operator(conn, np.ones(_ne(c)), cM * RHO * M + cK * E[0] * K, nn, _clamped(c["nx"], c["ny"], c["nz"], 0))
    mass = _Operator(conn, np.ones(_ne(c)), RHO * M, nn, np.zeros(0, dtype=np.int64))
    u = op.solve(mass.full(torch.as_tensor(_ground(c, seed), device=dev)))
    return {k: v.cpu().numpy() for k, v in (("u", u), ("v", GAMMA / (BETA * DT) * u), ("a", u / (BETA * DT * DT)))}


def _exact_batch(c, seed):
    K, _ = _element(1.0)
    conn, scale, fixed, load, part, at = [], [], [], [], [], 0
    for n, (nx, ny, nz, axis) in enumerate(_slabs(c)):
        h = 1.0 / max(nx, ny)
        conn.append(_conn(nx, ny, nz) + at)
        scale.append(_moduli(c, nx * ny * nz, seed, n) * h)  # a cube's stiffness grows with its side
        fixed.append(_clamped(nx, ny, nz, axis) + 3 * at)
        load.append(_top_load(nx, ny, nz, h, [0.0, 0.0, -1.0]))
        nn = (nx + 1) * (ny + 1) * (nz + 1)
        part.append(np.full(3 * nn, n))
        at += nn
    cat = np.concatenate
    op = _Operator(cat(conn), cat(scale), K, at, cat(fixed), cat(part), c["count"])
    return op.solve(torch.as_tensor(cat(load), device=op.Ke.device), most=4000).cpu().numpy()


def _exact_eig(c, seed):
    """Dense, for the meshes where that takes seconds."""
    nn = _nn(c)
    if 3 * nn > 6000:
        return None
    K, M = _element(_cell(c))
    conn = _conn(c["nx"], c["ny"], c["nz"])
    E = _moduli(c, _ne(c), seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    dof = torch.as_tensor((3 * conn[:, :, None] + np.arange(3)).reshape(-1, 24), device=dev)
    at = (dof[:, :, None] * (3 * nn) + dof[:, None, :]).reshape(-1)
    keep = np.setdiff1d(np.arange(3 * nn), _clamped(c["nx"], c["ny"], c["nz"], 0))
    kt = torch.as_tensor(keep, device=dev)

    def dense(Ke, s):
        v = torch.as_tensor(s, device=dev)[:, None, None] * torch.as_tensor(Ke, device=dev)[None]
        A = torch.zeros((3 * nn) ** 2, dtype=torch.float64, device=dev).index_add_(0, at, v.reshape(-1))
        return A.reshape(3 * nn, 3 * nn)[kt][:, kt]

    L = torch.linalg.cholesky(dense(M, np.full(E.shape, RHO)))
    S = torch.linalg.solve_triangular(L, dense(K, E), upper=False)
    S = torch.linalg.solve_triangular(L, S.T.contiguous(), upper=False)
    lam, Q = torch.linalg.eigh(0.5 * (S + S.T))
    X = np.zeros((3 * nn, c["nev"]))
    X[keep] = torch.linalg.solve_triangular(L.T, Q[:, :c["nev"]], upper=True).cpu().numpy()
    return {"lam": lam[:c["nev"]].cpu().numpy(), "modes": X * np.sign(_phase(c) @ X)}
