"""Performance cases: what a user of the GPU solver has it do, through its public entry points.

Every family is one way in which the framework is used:

* ``increment``: one load increment of the Newton driver (``NISTGPU.solveIncrement``: element
  passes, assembly, Krylov solves, convergence checks) from a committed equilibrium state, the way
  ``solveStep`` calls it.  The history before it (one increment from the virgin state) belongs to
  ``prepare``.  Linear and quadratic elements, elastic, J2 and hyperelastic materials, every solver
  (all-FP64 PCG, mixed PCG, FGMRES with the multigrid), with a read-back of stresses where asked for.
* ``tied``: the same for a hex20 | hex8 total-Lagrange box with a tied interface.
* ``batch``: one load increment of a batch of independent J2 cubes (``BatchNISTGPU``).
* ``dropin``: the reference's own assembly per Newton iteration: the element loop, the VIJ -> CSR
  scatter in the reference's layout and the Dirichlet rows, in FP64 on a distorted mesh.
* ``host``: a load increment of a Newton loop that keeps its vectors in host arrays
  (``HostArrayBackend``), as the reference's own driver does.

Materials, loads and meshes come from the seed: J2 rows from the seeded family of the cube batch
(sigma_y ~ U[150, 350], H ~ U[200, 2000], nu ~ U[0.2, 0.4]), loads in proportion to the yield strain:
the timed increment takes a box from the onset of yield into the plastic range, as the benchmark's.  ``exact`` is a small finite element code of
its own in 64 bits (dense solves).  The learned correction is not among the cases: no solver uses it
unless a caller trains it first, and the benchmark's validation drops it.
"""

import math

import numpy as np
import torch

from edelweissfe_gb300 import _lib
from edelweissfe_gb300.batch import BatchNISTGPU, cube_batch_spec
from edelweissfe_gb300.hostbackend import HostArrayBackend
from edelweissfe_gb300.mesh import box_mesh, tied_box_mesh
from edelweissfe_gb300.model import DirichletBC, ElementGroup, Model, NodeForces
from edelweissfe_gb300.solver import LinSolverOptions, NISTGPU, Step, TimeStep

E = 210000.0
H_EL = 0.1  # element edge of the boxes (the benchmark's)
FAMILIES = ("increment", "tied", "batch", "dropin", "host")

SOLVERS = {
    # the solver options by name: the defaults, the all-FP64 mode, the FGMRES of the seeded family
    # and of the tied box, and the benchmark's
    "pcg": (False, dict()),
    "fp64": (True, dict(mixed=False)),
    "fgmres40": (False, dict(method="fgmres", rtol=1e-8, innerRtol=1e-6, restart=40)),
    "fgmres64": (False, dict(method="fgmres", rtol=1e-8, innerRtol=1e-4, restart=64)),
}


def listed():
    inc = dict(family="increment", elType="C3D8", material="vonmises", results=False)
    return [
        # a static analysis: the elastic cantilever under node forces, all in FP64 (latency)
        dict(inc, name="cantilever_fp64", material="linearelastic", nx=20, ny=4, nz=4, solver="fp64"),
        # a small odd-sized J2 box with the default solver options (latency of the Newton loop)
        dict(inc, name="j2_small_pcg", nx=12, ny=5, nz=7, solver="pcg"),
        # the box of the pinned reference history, in FP64 throughout
        dict(inc, name="j2_history_fp64", nx=25, ny=10, nz=10, solver="fp64"),
        # an ordinary box with the default block-Jacobi PCG
        dict(inc, name="j2_box_pcg", nx=50, ny=20, nz=20, solver="pcg"),
        # an ordinary box with FGMRES and the multigrid (the seeded family's box)
        dict(inc, name="j2_box_fgmres", nx=40, ny=16, nz=16, solver="fgmres40"),
        # the benchmark's 160k-element box and solver
        dict(inc, name="j2_headline_fgmres", nx=100, ny=40, nz=40, solver="fgmres64"),
        # quadratic elements (27 Gauss points) with the stresses read back after the increment
        dict(inc, name="j2_quadratic_results", elType="C3D20", nx=21, ny=9, nz=8, solver="fgmres40", results=True),
        # hex20 | hex8 hyperelastic box with a tied interface, half the benchmark's edge counts across
        dict(name="tied_tl_box", family="tied", nxq=15, nxl=15, ny=15, nz=15, solver="fgmres40"),
        # a batch of uneven cubes of the benchmark's sizes
        dict(name="cube_batch", family="batch", nProb=160, nMin=4, nMax=16),
        # the reference's assembly: linear J2 elements and quadratic total-Lagrange elements
        dict(name="dropin_hex8_j2", family="dropin", elType="C3D8", nx=40, ny=16, nz=16),
        dict(name="dropin_hex20_tl", family="dropin", elType="C3D20TL", nx=13, ny=7, nz=6),
        # the reference's Newton loop over host arrays
        dict(name="host_j2_box", family="host", nx=30, ny=12, nz=11, solver="pcg"),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    family = rng.choice(("increment", "increment", "increment", "tied", "batch", "dropin", "dropin", "host"))
    if family == "tied":
        n = log(3, 14)
        return dict(family=family, nxq=log(3, 15), nxl=log(3, 15), ny=n, nz=max(3, n - rng.randint(0, 2)), solver="fgmres40")
    if family == "batch":
        lo = rng.randint(3, 6)
        return dict(family=family, nProb=log(8, 160), nMin=lo, nMax=rng.randint(lo + 2, 14))
    if family == "dropin":
        el = rng.choice(("C3D8", "C3D8R", "C3D8E", "C3D20", "C3D20R", "C3D8TL", "C3D8RTL", "C3D20TL", "C3D20RTL"))
        n = log(3, 6 if "20" in el or el == "C3D8E" else 14)
        return dict(family=family, elType=el, nx=log(4, 12 if "20" in el else 36), ny=n, nz=max(2, n - rng.randint(0, 2)))
    n = log(3, 12)
    if family == "host":
        return dict(family=family, nx=log(6, 30), ny=n, nz=max(3, n - rng.randint(0, 2)), solver="pcg")
    kind = rng.choice(("elastic", "pcg", "fp64", "fgmres40", "fgmres64", "quadratic"))
    case = dict(family=family, elType="C3D8", material="vonmises", results=rng.random() < 0.3, nx=log(6, 30), ny=n,
                nz=max(3, n - rng.randint(0, 2)), solver=kind)  # fmt: skip
    if kind == "elastic":
        case.update(material="linearelastic", solver=rng.choice(("fp64", "pcg")))
    elif kind == "quadratic":
        n = log(2, 8)
        case.update(elType=rng.choice(("C3D20", "C3D20R")), nx=log(4, 18), ny=n, nz=max(2, n - 1), solver="fgmres40")
    elif kind.startswith("fgmres"):
        n = log(6, 36)
        case.update(nx=log(12, 90), ny=n, nz=max(4, n - rng.randint(0, 3)))
    return case


# ---- models ----------------------------------------------------------------------------------


def j2_row(rng):
    return [E, float(rng.uniform(0.2, 0.4)), float(rng.uniform(150.0, 350.0)), float(rng.uniform(200.0, 2000.0)), 0.0, 0.0]


def tl_row(rng):
    return [float(80.0 * rng.uniform(0.9, 1.1)), float(200.0 * rng.uniform(0.9, 1.1))]


def step_times():
    """The increment before and the one that is timed: 55 % of the step, then the benchmark's 5 %."""
    return TimeStep(1, 0.55, 0.55, 0.55, 0.55, 0.55), TimeStep(2, 0.05, 0.60, 0.05, 0.60, 0.60)


def box_problem(case, seed):
    """Mesh, element group, Dirichlet sets and node forces of an ``increment`` or ``host`` case."""
    rng = np.random.default_rng(seed)
    n = case["nx"], case["ny"], case["nz"]
    L = [H_EL * k for k in n]
    el = case.get("elType", "C3D8")
    m = box_mesh(*n, *L, nNodesPerElement=20 if "20" in el else 8)
    left, right = m["nodeSets"]["gen_left"], m["nodeSets"]["gen_right"]
    clamp = {0: 0.0, 1: 0.0, 2: 0.0}
    if case.get("material", "vonmises") == "linearelastic":
        props = [E * float(rng.uniform(0.5, 1.5)), float(rng.uniform(0.2, 0.4))]
        force = np.array([0.0, 0.0, -1.0]) * float(rng.uniform(0.5, 1.5)) * L[1] * L[2] / right.size
        return m, ElementGroup(el, m["elements"], "linearelastic", np.array(props)), [(left, clamp)], [(right, force)]
    props = j2_row(rng)
    ux = float(rng.uniform(1.8, 1.85)) * props[2] / E * L[0]  # 0.6 of the step: 1.1 times the yield strain
    return m, ElementGroup(el, m["elements"], "vonmises", np.array(props)), [(left, clamp), (right, {0: ux})], []


def solver_options(case):
    keFp64, kw = SOLVERS[case["solver"]]
    return dict(keFp64=keFp64, linsolver=LinSolverOptions(**kw))


def tied_problem(case, seed):
    rng = np.random.default_rng(seed)
    h = 1.0 / 30.0
    m = tied_box_mesh(case["nxq"], case["nxl"], case["ny"], case["nz"], case["nxq"] * h, case["nxl"] * h, case["ny"] * h,
                      case["nz"] * h)  # fmt: skip
    p = np.array(tl_row(rng))
    ux = -float(rng.uniform(0.08, 0.1)) * (case["nxq"] + case["nxl"]) * h
    groups = [ElementGroup("C3D20TL", m["elements20"], "neohookewa", p), ElementGroup("C3D8TL", m["elements8"], "neohookewa", p)]
    left, right = m["nodeSets"]["gen_left"], m["nodeSets"]["gen_right"]
    return m, groups, [(left, {0: 0.0, 1: 0.0, 2: 0.0}), (right, {0: ux})]


def dropin_problem(case, seed):
    """A distorted mesh (8-node elements: every node moved; 20-node elements: sheared, which is where
    the reference's hex20 Jacobian is the textbook's), two displacement increments (the first is
    committed in ``prepare``) and the Dirichlet rows."""
    rng = np.random.default_rng(seed)
    el = case["elType"]
    n = case["nx"], case["ny"], case["nz"]
    m = box_mesh(*n, *[H_EL * k for k in n], nNodesPerElement=20 if "20" in el else 8)
    if "20" in el:
        X = m["coords"] @ (np.eye(3) + rng.uniform(-0.1, 0.1, (3, 3)))
    else:
        X = m["coords"] + rng.uniform(-0.04, 0.04, m["coords"].shape) * H_EL
    tl = el.endswith("TL")
    props = tl_row(rng) if tl else j2_row(rng)
    strain = 0.05 if tl else 0.9 * props[2] / E
    ramp = np.stack([X[:, 0], -0.3 * X[:, 1], -0.3 * X[:, 2]], 1) * strain
    d1 = ramp + rng.uniform(-0.1, 0.1, X.shape) * strain * H_EL
    d2 = 0.7 * ramp + rng.uniform(-0.1, 0.1, X.shape) * strain * H_EL
    rows = (3 * m["nodeSets"]["gen_left"][:, None] + np.arange(3)).reshape(-1).astype(np.int64)
    return X, m["elements"], "neohookewa" if tl else "vonmises", props, d1.reshape(-1), d2.reshape(-1), rows


def stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    fam = case["family"]
    if fam in ("increment", "tied"):
        if fam == "increment":
            m, group, dirs, forces = box_problem(case, seed)
            model = Model(m["coords"], [group])
        else:
            m, groups, dirs = tied_problem(case, seed)
            model, forces = Model(m["coords"], groups, ties=m["ties"]), []
        s = NISTGPU(model, [DirichletBC(n, c) for n, c in dirs], [NodeForces(n, f) for n, f in forces], **solver_options(case))
        step = Step(minInc=1e-6, maxIter=25)
        t1, t2 = step_times()
        U, dU, P = (torch.zeros(s.nDof, dtype=torch.float64, device="cuda") for _ in range(3))
        U, dU, P, _ = s.solveIncrement(U, dU, P, t1, None, step)
        _lib.check(s.lib.ef_accept_state(s.ctx), "ef_accept_state")
        col = s.resultCollector(0, None, range(QPS[case["elType"]]), "stress", trial=True) if case.get("results") else None
        if case.get("material") == "linearelastic":
            t1 = None  # without an extrapolation, which would leave nothing to solve
        return dict(family=fam, s=s, step=step, t1=t1, t2=t2, U=U, dU=dU, col=col)
    if fam == "batch":
        sizes = cube_batch_spec(case["nProb"], 0, case["nMin"], case["nMax"])  # of the case; the materials are of the seed
        s = BatchNISTGPU([dict(c, props=j2_row(np.random.default_rng([seed, k]))) for k, c in enumerate(sizes)])
        step = Step(maxInc=0.1, minInc=1e-6, maxIter=25)
        t1, t2 = TimeStep(1, 0.1, 0.1, 0.1, 0.1, 0.1), TimeStep(2, 0.1, 0.2, 0.1, 0.2, 0.2)
        s.solveIncrementBatch(t1, None, step, tune=True)
        s.U_n.add_(s.dU)
        _lib.check(s.lib.ef_accept_state(s.ctx), "ef_accept_state")
        return dict(family=fam, s=s, step=step, t1=t1, t2=t2, dU=s.dU.clone())
    if fam == "dropin":
        X, elements, material, props, d1, d2, rows = dropin_problem(case, seed)
        s = NISTGPU(Model(X, [ElementGroup(case["elType"], elements, material, np.array(props))]), keFp64=True,
                    linsolver=LinSolverOptions(mixed=False), scalarCSR=True)  # fmt: skip
        d1, d2 = torch.as_tensor(d1, device="cuda"), torch.as_tensor(d2, device="cuda")
        t1, t2 = step_times()
        s.computeElements(d1, d1, torch.zeros_like(d1), torch.zeros_like(d1), t1)
        _lib.check(s.lib.ef_accept_state(s.ctx), "ef_accept_state")
        return dict(family=fam, s=s, t2=t2, U=d1 + d2, dU=d2, rows=rows)
    m, group, dirs, _ = box_problem(case, seed)
    model = Model(m["coords"], [group])
    g = dict(elType=group.elType, material=group.material, props=group.props, elDofs=model.element_dofs(group))
    b = HostArrayBackend(model.nDof, model.dof_coordinates(), [g], **solver_options(case))
    bcs = [DirichletBC(n, c) for n, c in dirs]
    t1, t2 = step_times()
    zero = np.zeros(model.nDof)
    U, dU, _, _ = host_increment(b, bcs, zero, zero, t1, None, model.n_accumulated_fluxes())
    b.accept_state()
    return dict(family=fam, b=b, bcs=bcs, U=U, dU=dU, t1=t1, t2=t2, nAcc=model.n_accumulated_fluxes())


def host_increment(b, bcs, U_n, dU, ts, prev, nAcc):
    """The reference's solveIncrement over host arrays (one field, no external loads)."""
    dofs = np.concatenate([bc.dofs for bc in bcs])
    values = np.concatenate([bc.getDelta(ts) for bc in bcs])
    b.begin_increment()
    b.set_dirichlet(dofs)
    if prev is not None:
        dU = dU * (ts.stepProgressIncrement / prev.stepProgressIncrement)
        dU[dofs] = values
    else:
        dU = np.zeros_like(dU)
    ddU, it = None, 0
    while True:
        P, F = b.compute_elements(U_n + dU, dU, [ts.stepTime, ts.totalTime], ts.timeIncrement)
        R = P.copy()
        if it == 0 and prev is None:
            R[dofs] = values
        else:
            R[dofs] = 0.0
            corr = 0.0 if ddU is None else np.max(np.abs(ddU))
            if corr < 1e-8 and np.max(np.abs(R)) <= max(1e-8 * max(1e-10, np.sum(F) / nAcc), 1e-7):
                return U_n + dU, dU, P, it
        if it == 25:
            raise RuntimeError("the increment did not converge")
        b.assemble()
        ddU = b.solve(R)
        dU = dU + ddU
        it += 1


def run(state):
    fam = state["family"]
    if fam in ("increment", "tied"):
        s = state["s"]
        s.krylovIterations.clear()
        P = torch.zeros(s.nDof, dtype=torch.float64, device="cuda")
        U, dU, P, it = s.solveIncrement(state["U"], state["dU"].clone(), P, state["t2"], state["t1"], state["step"])
        out = dict(U=U, dU=dU, P=P, newton=it)
        if state["col"] is not None:
            out["stress"] = state["col"].getCurrentResults()
        return out
    if fam == "batch":
        s = state["s"]
        s.dU.copy_(state["dU"])
        it = s.solveIncrementBatch(state["t2"], state["t1"], state["step"])
        return dict(U=s.U_n + s.dU, dU=s.dU.clone(), P=s.P.clone(), newton=it)
    if fam == "dropin":
        s = state["s"]
        P = torch.empty(s.nDof, dtype=torch.float64, device="cuda")
        F = torch.empty_like(P)
        s.computeElements(state["U"], state["dU"], P, F, state["t2"])
        data = torch.empty(s.info.nnz, dtype=torch.float64, device="cuda")
        _lib.check(s.lib.ef_update_csr(s.ctx, None, data.data_ptr(), stream()), "ef_update_csr")
        rows = state["rows"]
        _lib.check(s.lib.ef_csr_dirichlet_rows(s.ctx, data.data_ptr(), rows.ctypes.data, rows.size, stream()),
                   "ef_csr_dirichlet_rows")  # fmt: skip
        return dict(P=P, F=F, data=data)
    U, dU, P, it = host_increment(state["b"], state["bcs"], state["U"], state["dU"], state["t2"], state["t1"], state["nAcc"])
    return dict(U=U, dU=dU, P=P, newton=it)


# ---- work --------------------------------------------------------------------------------------

QPS = {"C3D8": 8, "C3D8R": 1, "C3D8E": 27, "C3D20": 27, "C3D20R": 8}


def element_counts(elType, nx, ny, nz):
    """(elements, nodes, Gauss points and nodes per element, stored 3x3 blocks about) of a box."""
    quad = "20" in elType
    nEl = nx * ny * nz
    corner = (nx + 1) * (ny + 1) * (nz + 1)
    edges = nx * (ny + 1) * (nz + 1) + (nx + 1) * ny * (nz + 1) + (nx + 1) * (ny + 1) * nz
    nodes = corner + edges if quad else corner
    return nEl, nodes, QPS[elType.replace("TL", "")], 20 if quad else 8, nodes * (60 if quad else 26)


def work(case):
    """One pass's inputs read once and outputs written once: the committed state and the new one, the
    coordinates and vectors and, once, the assembled system, with the arithmetic of one element pass
    and one product with the system (an increment repeats both as often as its tolerances ask for)."""
    fam = case["family"]
    if fam == "tied":
        parts = [("C3D20TL", case["nxq"], case["ny"], case["nz"], 1), ("C3D8TL", case["nxl"], case["ny"], case["nz"], 1)]
    elif fam == "batch":
        mid = (case["nMin"] + case["nMax"]) // 2
        parts = [("C3D8", mid, mid, mid, case["nProb"])]
    else:
        parts = [(case.get("elType", "C3D8"), case["nx"], case["ny"], case["nz"], 1)]
    b = f = 0.0
    for el, nx, ny, nz, times in parts:
        nEl, nodes, nq, nn, blocks = element_counts(el, nx, ny, nz)
        value = 4 if case.get("solver", "fp64") != "fp64" and fam != "batch" else 8
        state = 0 if fam == "increment" and case["material"] == "linearelastic" else 2 * 13
        b += times * (nEl * nq * 8 * state + nEl * nn * 4 + 3 * nodes * 8 * 6 + blocks * 9 * value)
        f += times * (nEl * nq * (nn * (nn + 1) / 2 * 54 + nn * 72) + blocks * 18)
    return {"bytes": b, "flops": f}


# ---- the same in 64 bits, as plain torch ---------------------------------------------------------


def corner_signs(coords, elements):
    """Natural coordinates (-1, 0, 1) of the element nodes, from a box's first element."""
    x = coords[elements[0]]
    lo, hi = x.min(0), x.max(0)
    return np.rint(2 * (x - lo) / (hi - lo) - 1)


def gauss(n):
    x, w = np.polynomial.legendre.leggauss(n)
    q = np.array([(a, b, c) for a in x for b in x for c in x])
    return q, np.array([a * b * c for a in w for b in w for c in w])


def shape_gradients(signs, q):
    """dN_a/dxi at the points q of the 8- or 20-node hexahedron with node positions `signs`."""
    q = torch.tensor(q, requires_grad=True)
    s = torch.tensor(signs)
    prod = 1 + q[:, None, :] * s[None]  # [nq, nn, 3]
    if len(signs) == 8:
        N = prod.prod(2) / 8
    else:
        corner = prod.prod(2) * ((q[:, None, :] * s[None]).sum(2) - 2) / 8
        f = torch.where(s[None] == 0, 1 - q[:, None, :] ** 2, prod)
        N = torch.where((s == 0).any(1)[None], f.prod(2) / 4, corner)
    out = [torch.autograd.grad(N[:, a].sum(), q, retain_graph=True)[0] for a in range(len(signs))]
    return torch.stack(out, 1).detach()  # [nq, nn, 3]


class Exact:
    """Element residuals and stiffnesses of one group in FP64 (material rows as the solver takes them)."""

    def __init__(self, X, elements, signs, nq, material, props, device):
        q, w = gauss(round(nq ** (1 / 3)))
        d = shape_gradients(signs, q).to(device)
        self.el = torch.as_tensor(np.asarray(elements), device=device)
        x = torch.as_tensor(np.asarray(X), device=device)[self.el]  # [e, nn, 3]
        J = torch.einsum("qai,eac->eqic", d, x)
        self.g = torch.einsum("eqci,qai->eqac", torch.linalg.inv(J), d)  # dN/dx
        self.w = torch.linalg.det(J) * torch.as_tensor(w, device=device)
        self.material, self.p = material, props
        self.sig = torch.zeros(*self.w.shape, 3, 3, dtype=torch.float64, device=device)
        self.kap = torch.zeros_like(self.w)

    def pass_(self, U, dU, commit=False, tangent=True):
        """(Pe [e, nn, 3], Ke [e, nn, 3, nn, 3]) from the committed state."""
        eye = torch.eye(3, dtype=torch.float64, device=self.w.device)
        g, w = self.g, self.w
        if self.material == "neohookewa":
            mu, K = self.p[:2]
            u = U.reshape(-1, 3)[self.el]
            F = eye + torch.einsum("eai,eqaj->eqij", u, g)
            Jd = torch.linalg.det(F)
            kk = K - 2.0 / 3.0 * mu
            lb, mb = kk * (Jd * Jd - Jd) - mu, kk * (2 * Jd * Jd - Jd)
            tau = mu * F @ F.transpose(-1, -2) + lb[..., None, None] * eye
            gs = torch.einsum("eqji,eqaj->eqai", torch.linalg.inv(F), g)
            Pe = -torch.einsum("eq,eqij,eqaj->eai", w, tau, gs)
            Ke = None
            if tangent:
                Ke = torch.einsum("eq,eqak,eqbk,ij->eaibj", w * mu, g, g, eye)
                Ke += torch.einsum("eq,eqai,eqbj->eaibj", w * mb, gs, gs)
                Ke -= torch.einsum("eq,eqbi,eqaj->eaibj", w * lb, gs, gs)
            return Pe, Ke
        Em, nu = self.p[:2]
        lam, G = Em * nu / ((1 + nu) * (1 - 2 * nu)), Em / (2 * (1 + nu))
        H = torch.einsum("eai,eqaj->eqij", dU.reshape(-1, 3)[self.el], g)
        de = 0.5 * (H + H.transpose(-1, -2))
        t = self.sig + 2 * G * de + lam * de.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] * eye
        lt, mt = torch.full_like(w, lam), torch.full_like(w, G)
        c1, n, kap = torch.zeros_like(w), torch.zeros_like(t), self.kap
        if self.material == "vonmises":
            fy0, HL = self.p[2], self.p[3]
            dev = t - t.diagonal(dim1=-2, dim2=-1).sum(-1)[..., None, None] / 3 * eye
            dn = dev.flatten(-2).norm(dim=-1)
            f = dn - math.sqrt(2 / 3) * (fy0 + HL * self.kap)
            plastic = f > 0
            dk = torch.where(plastic, f / (math.sqrt(6) * G + math.sqrt(2 / 3) * HL), torch.zeros_like(f))
            dl = math.sqrt(1.5) * dk
            n = torch.where(plastic[..., None, None], dev / torch.where(plastic, dn, torch.ones_like(dn))[..., None, None], n)
            t = t - (2 * G * dl)[..., None, None] * n
            kap = self.kap + dk
            safe = torch.where(plastic, dn, torch.ones_like(dn))
            c2 = 4 * G * G * dl / safe
            c1 = torch.where(plastic, 2 * G * (1 / (1 + HL / (3 * G)) - 2 * G * dl / safe), c1)
            lt, mt = lam + c2 / 3, G - 0.5 * c2
        Pe = -torch.einsum("eq,eqij,eqaj->eai", w, t, g)
        Ke = None
        if tangent:
            Ke = torch.einsum("eq,eqai,eqbj->eaibj", w * lt, g, g)
            Ke += torch.einsum("eq,eqbi,eqaj->eaibj", w * mt, g, g)
            Ke += torch.einsum("eq,eqak,eqbk,ij->eaibj", w * mt, g, g, torch.eye(3, dtype=torch.float64, device=w.device))
            v = torch.einsum("eqij,eqaj->eqai", n, g)
            Ke -= torch.einsum("eq,eqai,eqbj->eaibj", w * c1, v, v)
        if commit:
            self.sig, self.kap = t, kap
        return Pe, Ke

    def dofs(self):
        return (3 * self.el[:, :, None] + torch.arange(3, device=self.el.device)).flatten(1)

    def condense(self, Pe, nDof):
        out = torch.zeros(2, nDof, dtype=torch.float64, device=Pe.device)
        i = self.dofs().flatten()
        out[0].index_add_(0, i, Pe.flatten())
        out[1].index_add_(0, i, Pe.abs().flatten())
        return out[0], out[1]


def exact(case, seed):
    fam = case["family"]
    device = "cuda" if torch.cuda.is_available() else "cpu"
    if fam == "dropin":
        X, elements, material, props, d1, d2, rows = dropin_problem(case, seed)
        m = box_mesh(1, 1, 1, nNodesPerElement=elements.shape[1])
        ex = Exact(X, elements, corner_signs(m["coords"], m["elements"]), QPS[case["elType"].replace("TL", "")], material, props, device)
        d1, d2 = torch.as_tensor(d1, device=device), torch.as_tensor(d2, device=device)
        ex.pass_(d1, d1, commit=True, tangent=False)
        Pe, Ke = ex.pass_(d1 + d2, d2)
        P, F = ex.condense(Pe, d1.numel())
        i = ex.dofs()
        nd = d1.numel()
        key = (i[:, :, None] * nd + i[:, None, :]).flatten()
        slots, inverse = torch.unique(key, return_inverse=True)
        data = torch.zeros(slots.numel(), dtype=torch.float64, device=device).index_add_(0, inverse, Ke.flatten())
        r, c = slots // nd, slots % nd
        fixed = torch.zeros(nd, dtype=torch.bool, device=device)
        fixed[torch.as_tensor(rows, device=device)] = True
        data = torch.where(fixed[r], (r == c).to(torch.float64), data)
        return dict(P=P, F=F, data=data)
    if fam not in ("increment", "host") or 3 * element_counts(case.get("elType", "C3D8"), case["nx"], case["ny"], case["nz"])[1] > 10000:
        return None  # dense solves of more would take too long
    m, group, dirs, forces = box_problem(case, seed)
    ex = Exact(m["coords"], m["elements"], corner_signs(m["coords"], m["elements"]), QPS[group.elType], group.material,
               list(group.props), device)  # fmt: skip
    nd = 3 * m["coords"].shape[0]
    bcs, nfs = [DirichletBC(n, c) for n, c in dirs], [NodeForces(n, f) for n, f in forces]
    fixed = torch.as_tensor(np.concatenate([b.dofs for b in bcs]), device=device)
    i = ex.dofs()
    U = torch.zeros(nd, dtype=torch.float64, device=device)
    for ts in step_times():
        PExt = torch.zeros_like(U)
        for nf in nfs:
            PExt.index_add_(0, torch.as_tensor(nf.dofs, device=device), torch.as_tensor(nf.getCurrentLoad(ts), device=device))
        dU = torch.zeros_like(U)
        values = torch.as_tensor(np.concatenate([b.getDelta(ts) for b in bcs]), device=device)
        for it in range(30):
            Pe, Ke = ex.pass_(U + dU, dU)
            P, F = ex.condense(Pe, nd)
            R = P + PExt
            R[fixed] = values - dU[fixed]
            if it > 0 and float(R.abs().max()) <= 1e-11 * float(F.max()):
                break
            K = torch.zeros(nd, nd, dtype=torch.float64, device=device)
            K.index_put_((i[:, :, None].expand(-1, -1, i.shape[1]).flatten(), i[:, None, :].expand(-1, i.shape[1], -1).flatten()),
                         Ke.flatten(), accumulate=True)  # fmt: skip
            K[fixed] = 0.0
            K[fixed, fixed] = 1.0
            dU = dU + torch.linalg.solve(K, R)
            del K
        ex.pass_(U + dU, dU, commit=True, tangent=False)
        U = U + dU
    if fam == "host":
        return dict(U=U, dU=dU, P=P, newton=None)
    out = dict(U=U, dU=dU, P=P, newton=None)
    if case["results"]:
        out["stress"] = None  # in the solver's own Gauss-point order
    return out
