"""The work this framework is used for, as measurable cases: PISO steps of the P2/P1 Navier-Stokes
solver over the range of meshes, Krylov methods and precisions it offers, the coupled and streaming
loops around them, the discrete adjoint, and the allocation-free divergence.

Physical set-up of all of them: the tube flows of the tests and of the benchmark (density 1060,
viscosity 0.004, dt 0.01, parabolic inlet, no-slip walls, pressure outlet).
"""
from __future__ import annotations

import functools
import math
import random
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "cell-fluid-structure-analysis_b200"))
import cfsa_b200 as cf  # noqa: E402

RHO, NU, DT = 1060.0, 0.004, 0.01
LENGTH, RADIUS = 30.0, 2.0  # straight tube
KRYLOV = {"cg": cf.KRYLOV_CG, "bicgstab": cf.KRYLOV_BICGSTAB, "cg1": cf.KRYLOV_CG1, "cg2l": cf.KRYLOV_CG2L}
PRECISION = {"fp64": cf.PRECISION_FP64, "mixed": cf.PRECISION_MIXED}
NORM = {"reference": cf.NORM_REFERENCE, "jacobi": cf.NORM_JACOBI}


def _case(kind, mesh, momentum="bicgstab", pressure="bicgstab", **more):
    c = dict(kind=kind, momentum=momentum, pressure=pressure, precision="fp64", norm="reference",
             tol=0.0, steps=1, corrections=1, neumann=False, checkpoint=0, objective="", **mesh)
    c.update(more)
    return c


def _tube(rings, layers):  # 18 rings^2 layers tets
    return dict(mesh="tube", n0=rings, n1=layers, n2=0, cell=0.0)


def _channel(nx, ny, nz):  # 6 nx ny nz tets
    return dict(mesh="channel", n0=nx, n1=ny, n2=nz, cell=0.0)


def _bifurcation(cell):
    return dict(mesh="bifurcation", n0=0, n1=0, n2=0, cell=cell)


def listed():
    return [
        # a unit-test or debugging mesh (288 tets), every solver setting at its default: latency
        _case("steps", _tube(2, 4), name="tube_288_default"),
        # the straight tube at the size the CPU reference is run at, its BiCGSTAB for both solves,
        # tight tolerance, a short batch of steps
        _case("steps", _tube(5, 68), tol=1e-10, steps=5, name="tube_30k_bicgstab"),
        # a small odd-sized channel with a Neumann outlet and pressure reference, two correctors,
        # conjugate gradients for both systems
        _case("steps", _channel(37, 13, 11), "cg", "cg", norm="jacobi", tol=1e-8, steps=3, corrections=2,
              neumann=True, name="channel_32k_cg"),
        # a moderate mesh with the out-of-the-box settings (BiCGSTAB, 1e-6 / 1e-8)
        _case("steps", _tube(8, 217), steps=2, name="tube_250k_default"),
        # the same mesh with the solvers the documentation recommends, single-reduction pressure CG
        _case("steps", _tube(8, 217), "cg", "cg1", tol=1e-10, steps=2, name="tube_250k_cg_cg1"),
        # the headline mesh and settings: 1M tets, FP64, momentum CG, two-level pressure CG
        _case("steps", _tube(16, 217), "cg", "cg2l", tol=1e-10, steps=4, name="tube_1m_cg_cg2l"),
        # the same in mixed precision under the Jacobi-scaled criterion
        _case("steps", _tube(16, 217), "cg", "cg2l", precision="mixed", norm="jacobi", tol=1e-10, steps=4,
              name="tube_1m_mixed"),
        # a branching vessel on a lattice mesh (264k tets), mixed-precision BiCGSTAB momentum
        _case("steps", _bifurcation(0.2), "bicgstab", "cg2l", precision="mixed", norm="jacobi", tol=1e-10,
              steps=2, name="bifurcation_264k_mixed"),
        # a pulsatile inlet streamed in and the fields streamed out every step (105k tets)
        _case("stream", _tube(10, 58), "cg", "cg2l", norm="jacobi", tol=1e-8, steps=4, name="stream_104k"),
        # fluid side of a fluid-structure coupling: new vertex positions, a step, the wall forces
        _case("moving", _tube(7, 97), "cg", "cg2l", norm="jacobi", tol=1e-8, name="moving_86k"),
        # gradients for optimisation: recorded steps, then the reverse pass (250k tets)
        _case("adjoint", _tube(8, 217), "cg", "cg2l", norm="jacobi", tol=1e-12, steps=4, checkpoint=2,
              objective="wall_shear", name="adjoint_250k"),
        # divergence of device-resident fields inside another program's loop (1M tets)
        _case("divergence", _tube(16, 217), name="divergence_1m"),
    ]


def _drawn_mesh(rng, lo, hi):
    """A mesh of about exp(U(log lo, log hi)) tets, odd counts among them."""
    nt = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    shape = rng.choice(["tube", "tube", "channel", "bifurcation" if nt > 10000 else "channel"])
    if shape == "tube":
        rings = max(2, round((nt / 18.0 / rng.uniform(8, 16)) ** (1 / 3)))
        return _tube(rings, max(3, int(nt / (18 * rings * rings))))
    if shape == "channel":
        b = max(3, round((nt / 6.0 / rng.uniform(2, 5)) ** (1 / 3)))
        d = max(3, b + rng.randint(-2, 2))
        return _channel(max(4, int(nt / (6 * b * d))), b, d)
    return _bifurcation(round((2112.0 / nt) ** (1 / 3), 4))


def draw(rng: random.Random):
    kind = rng.choice(["steps"] * 6 + ["stream", "stream", "moving", "moving", "adjoint", "adjoint", "divergence"])
    top = {"steps": 990000, "stream": 250000, "moving": 100000, "adjoint": 200000, "divergence": 990000}[kind]
    mesh = _drawn_mesh(rng, 300, top)
    if kind == "divergence":
        return _case(kind, mesh)
    c = _case(kind, mesh, rng.choice(["cg", "bicgstab"]), rng.choice(["cg", "bicgstab", "cg1", "cg2l", "cg2l"]))
    big = mesh["mesh"] == "bifurcation" or mesh["n0"] * mesh["n1"] * max(mesh["n0"], mesh["n2"]) > 15000
    c["tol"] = rng.choice([0.0, 1e-7, 1e-8, 1e-10] if big else [0.0, 1e-6, 1e-8, 1e-10, 1e-12])
    if kind == "adjoint":
        c.update(norm="jacobi", tol=rng.choice([1e-10, 1e-12]), steps=rng.randint(1, 4),
                 checkpoint=rng.randint(0, 3), objective=rng.choice(["wall_shear", "pressure_drop"]))
        return c
    c["precision"] = rng.choice(["fp64", "fp64", "mixed"])
    c["norm"] = "jacobi" if c["precision"] == "mixed" else rng.choice(["reference", "jacobi"])
    c["corrections"] = rng.choice([1, 1, 2])
    c["neumann"] = rng.random() < 0.2
    c["steps"] = 1 if kind == "moving" else rng.randint(1, 3)
    return c


# ------------------------------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=3)
def _mesh(shape, n0, n1, n2, cell):
    if shape == "tube":
        m = cf.Mesh.cylinder(LENGTH, RADIUS, n0, n1)
    elif shape == "channel":
        m = cf.Mesh.structuredRectangularPrism(12.0, 3.0, 2.0, n0, n1, n2)
    else:
        return cf.Mesh.yBifurcation(cell=cell)  # tagged by its generator
    m.setupBoundaryConditions((1.0, 0.0, 0.0), 1.0)
    return m


def _mesh_of(case):
    return _mesh(case["mesh"], case["n0"], case["n1"], case["n2"], case["cell"])


def _radial(case, x):
    """0 on the axis of the inlet section, 1 on its wall."""
    if case["mesh"] == "channel":
        a, b = 2.0 * x[:, 1] / 3.0 - 1.0, 2.0 * x[:, 2] / 2.0 - 1.0
        return 1.0 - (1.0 - a * a) * (1.0 - b * b)
    return (x[:, 1] ** 2 + x[:, 2] ** 2) / RADIUS**2


def _inputs(case, seed):
    """Start-up flow: parabolic inlet profile, a smooth perturbed axial flow that vanishes on the
    walls, a falling pressure; `profiles` one inlet per step of a streamed case, `xyz` the moved
    vertices of a coupled one."""
    rng = np.random.default_rng(seed)
    m = _mesh_of(case)
    x = m.nodePositions()
    p1, p2 = m.fluidBC()
    bc = np.concatenate([p1, p2])
    nv = m.nVertices()
    peak = 0.5 + 0.5 * rng.random()
    inlet = np.zeros_like(x)
    inlet[:, 0] = peak * np.maximum(0.0, 1.0 - _radial(case, x))
    u = np.zeros_like(x)
    u[:, 0] = peak * np.clip(1.0 - _radial(case, x), 0.1, 1.0)
    for _ in range(4):  # smooth perturbations, a few per cent
        k, ph = rng.normal(size=3) * 1.5, rng.uniform(0, 2 * math.pi)
        u += 0.02 * peak * rng.normal(size=3) * np.sin(x @ k + ph)[:, None]
    u[bc == int(cf.FluidBCType.Wall)] = 0.0
    at_inlet = bc == int(cf.FluidBCType.Inlet)
    u[at_inlet] = inlet[at_inlet]
    top = float(x[:, 0].max())
    p = 2.0 * peak * (1.0 - x[:nv, 0] / top) + 0.05 * np.sin(x[:nv] @ rng.normal(size=3))
    d = dict(u=u, p=p, inlet=inlet)
    if case["kind"] == "stream":
        d["profiles"] = [inlet * (1.0 + 0.3 * math.sin(2 * math.pi * (k + rng.random()) / 8)) for k in range(case["steps"])]
    if case["kind"] == "moving":  # the wall bulges by up to 2% of its distance from the axis
        xyz = x[:nv].copy()
        bulge = 1.0 + 0.02 * rng.random() * np.sin(math.pi * xyz[:, 0] / top + rng.uniform(-0.3, 0.3))
        xyz[:, 1:] *= bulge[:, None]
        d["xyz"] = xyz
    return d


def _pinned(shape):
    t = torch.empty(shape, dtype=torch.float64, pin_memory=torch.cuda.is_available())
    return t.numpy()


def _pin(a):
    out = _pinned(a.shape)
    out[...] = a
    return out


# ------------------------------------------------------------------------------------------ the calls
def prepare(case, seed):
    m, d = _mesh_of(case), _inputs(case, seed)
    s = cf.NavierStokesSolver()
    if case["tol"]:
        s.setKrylovTolerances(case["tol"], case["tol"])
        s.setMaxIterations(5000, 50000)
    s.setConvergenceNorm(NORM[case["norm"]])
    s.setMomentumSolver(KRYLOV[case["momentum"]])
    s.setPressureSolver(KRYLOV[case["pressure"]])
    s.setPrecision(PRECISION[case["precision"]])
    s.setNumberOfCorrections(case["corrections"])
    if case["neumann"]:
        s.setOutletType(cf.OutletType.Neumann)
    s.setDt(DT)
    s.initialize(m, cf.Fluid(RHO, NU))
    s.setInletVelocityProfile(d["inlet"])
    state = dict(case=case, solver=s, u0=_pin(d["u"]), p0=_pin(d["p"]))
    if case["kind"] == "divergence":  # another program's device arrays, component-major
        state["u_dev"] = torch.from_numpy(np.ascontiguousarray(d["u"].T)).cuda()
        state["div_dev"] = torch.empty(s.nv, dtype=torch.float64, device="cuda")
        return state
    n = case["steps"] if case["kind"] == "stream" else 1
    state["u"] = [_pinned((s.N2, 3)) for _ in range(n)]
    state["p"] = [_pinned((s.nv,)) for _ in range(n)]
    if case["kind"] == "stream":
        state["profiles"] = [_pin(q) for q in d["profiles"]]
    if case["kind"] == "moving":
        state["xyz"] = _pin(d["xyz"])
    return state


def _objective(case):
    if case["objective"] == "wall_shear":
        return dict(kind=cf.OBJECTIVE_WALL_SHEAR, axis=0, lo=4.0, hi=8.0)
    return dict(kind=cf.OBJECTIVE_PRESSURE_DROP)


def run(state):
    case, s = state["case"], state["solver"]
    if case["kind"] == "divergence":
        s.computeDivergenceNoAlloc(state["u_dev"].data_ptr(), state["div_dev"].data_ptr())
        return state["div_dev"]
    s.setFields(state["u0"], state["p0"])
    if case["kind"] == "adjoint":
        s.adjointForward(case["steps"], case["checkpoint"])
        return s.adjointBackward(**_objective(case))
    if case["kind"] == "stream":
        done = 0
        for k in range(case["steps"]):
            s.setInletVelocityProfile(state["profiles"][k])
            done += int(s.pisoStep())
            s.getVelocityAsync(state["u"][k])
            s.getPressureAsync(state["p"][k])
        s.waitOutputs()
        return dict(done=done, u=state["u"], p=state["p"])
    if case["kind"] == "moving":
        s.updateVertices(state["xyz"])
        done = int(s.pisoStep())
        return dict(done=done, force=s.computeTotalFluidForces(), u=s.getVelocity(state["u"][0]),
                    p=s.getPressure(state["p"][0]))
    done = s.pisoSteps(case["steps"])[1]
    return dict(done=done, u=s.getVelocity(state["u"][0]), p=s.getPressure(state["p"][0]))


def work(case):
    """Each operator read once per step (CSR values and columns of the momentum matrix, M's values on
    the same pattern, G and L), the fields in and out once; one multiply-add per entry and
    right-hand side. Krylov iterations beyond the first product are the method's own."""
    nv, nt, ne, nf, _ = _mesh_of(case).sizes
    n2 = nv + ne
    nnz1 = nv + 2 * ne
    nnz2 = n2 + 2 * (3 * ne + 6 * nf + 3 * nt)  # node pairs that share a tet
    if case["kind"] == "divergence":
        return dict(bytes=nt * (4 * 4 + 13 * 8) + 8 * 4 * nv, flops=30 * nt)
    step = 20 * nnz2 + (12 + 24) * nnz1 + 8 * (6 * n2 + 4 * nv)
    flop = 2 * 3 * 2 * nnz2 + 2 * 7 * nnz1
    steps, fields = case["steps"], 8 * (3 * n2 + nv)
    if case["kind"] == "adjoint":
        return dict(bytes=2 * steps * step + 3 * fields, flops=2 * steps * flop)
    if case["kind"] == "stream":
        return dict(bytes=steps * (step + 2 * fields) + fields, flops=steps * flop)
    if case["kind"] == "moving":  # assembly: geometry in, four operators out
        return dict(bytes=step + 2 * fields + 8 * 6 * nv + 16 * nnz2 + 32 * nnz1, flops=flop + 400 * nt)
    return dict(bytes=steps * step + 2 * fields, flops=steps * flop)


# ------------------------------------------------------------------------------------------ 64-bit values
# The scheme restated with dense element arrays and converged solves, in torch float64.
_EDGES = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]


class _Solve(torch.autograd.Function):
    """x = A^-1 b for a symmetric A given as (product, diagonal); b [n, k], x0 an initial guess."""

    @staticmethod
    def forward(ctx, b, product, diag, x0):
        ctx.system = product, diag
        return _cg(product, diag, b, x0)

    @staticmethod
    def backward(ctx, g):
        product, diag = ctx.system
        return _cg(product, diag, g, torch.zeros_like(g)), None, None, None


def _cg(product, diag, b, x):
    r = b - product(x)
    z = r / diag[:, None]
    p, x = z.clone(), x.clone()
    rz = (r * z).sum(0)
    stop = rz * 1e-28
    for k in range(20000):
        q = product(p)
        pq = (p * q).sum(0)
        a = torch.where(pq > 0, rz / pq, torch.zeros_like(pq))
        x += a * p
        r -= a * q
        z = r / diag[:, None]
        new = (r * z).sum(0)
        if k % 20 == 19 and bool((new <= stop).all()):
            break
        p = z + torch.where(rz > 0, new / rz, torch.zeros_like(rz)) * p
        rz = new
    return x


def _csr(rows, cols, vals, n):
    a = torch.sparse_coo_tensor(torch.stack([rows, cols]), vals, (n, n)).coalesce()
    return a.to_sparse_csr()


class _Flow:
    """Element arrays and operators of one geometry."""

    def __init__(self, case, xyz=None):
        m = _mesh_of(case)
        dev = "cuda" if torch.cuda.is_available() else "cpu"

        def put(a, t=torch.float64):
            return torch.from_numpy(np.ascontiguousarray(a)).to(dev, t)

        self.m, self.put = m, put
        nv, nt, ne, _, _ = m.sizes
        self.nv, self.n = nv, nv + ne
        tets = put(m.tets(), torch.int64)
        self.tets = tets
        self.nodes = torch.cat([tets, nv + put(m.tetEdges(), torch.int64)], 1)
        x = put(m.vertices() if xyz is None else xyz)
        a, b, c, d = (x[tets[:, k]] for k in range(4))
        cross = torch.linalg.cross
        six = (cross(b - a, c - a) * (d - a)).sum(1)
        self.vol = (six / 6).abs()
        inv = (1.0 / six)[:, None]
        self.g = torch.stack([inv * cross(d - b, c - b), inv * cross(c - a, d - a), inv * cross(d - a, b - a),
                              inv * cross(b - a, c - a)], 1)
        self.g10 = torch.cat([self.g] + [(self.g[:, i] + self.g[:, j])[:, None] for i, j in _EDGES], 1)
        mt = torch.full((10, 10), 1 / 30, dtype=torch.float64, device=dev)
        mt[:4, :4], mt[4:, 4:] = 1 / 20, 1 / 60
        mt += torch.diag(torch.tensor([1 / 10 - 1 / 20] * 4 + [1 / 15 - 1 / 60] * 6, dtype=torch.float64, device=dev))
        self.mt = mt
        p1, p2 = m.fluidBC()
        bc = put(np.concatenate([p1, p2]), torch.int64)
        self.inlet, self.wall = bc == int(cf.FluidBCType.Inlet), bc == int(cf.FluidBCType.Wall)
        self.fixed = self.inlet | self.wall
        self.outlet = bc[:nv] == int(cf.FluidBCType.Outlet)
        self.inlet1 = self.inlet[:nv]
        self.wall1 = self.wall[:nv]
        ke = (self.vol / NU)[:, None, None] * (self.g10 @ self.g10.transpose(1, 2))
        me = RHO * self.vol[:, None, None] * mt
        rows = self.nodes[:, :, None].expand(-1, 10, 10).reshape(-1)
        cols = self.nodes[:, None, :].expand(-1, 10, 10).reshape(-1)
        self.A = _csr(rows, cols, (me / DT + ke).reshape(-1), self.n)
        diag = torch.zeros(self.n, dtype=torch.float64, device=dev)
        diag.index_add_(0, self.nodes.reshape(-1), torch.diagonal(me / DT + ke, dim1=1, dim2=2).reshape(-1))
        self.penalty = 1e10 * self.fixed.double()
        self.diag = diag + self.penalty
        lump = torch.zeros(self.n, dtype=torch.float64, device=dev)
        lump.index_add_(0, self.nodes.reshape(-1), (RHO * self.vol[:, None] * mt.sum(1)).reshape(-1))
        self.invm = 1.0 / lump
        le = self.vol[:, None, None] * (self.g @ self.g.transpose(1, 2))
        rows = tets[:, :, None].expand(-1, 4, 4).reshape(-1)
        cols = tets[:, None, :].expand(-1, 4, 4).reshape(-1)
        self.L = _csr(rows, cols, le.reshape(-1), nv)
        ld = torch.zeros(nv, dtype=torch.float64, device=dev)
        ld.index_add_(0, tets.reshape(-1), torch.diagonal(le, dim1=1, dim2=2).reshape(-1))
        self.ref = -1
        if case["neumann"]:
            self.ref = int(np.nonzero(p1 == int(cf.FluidBCType.Internal))[0][0])
            pen = torch.zeros(nv, dtype=torch.float64, device=dev)
            pen[self.ref] = 1e12
        else:
            pen = 1e12 * self.outlet.double()
        self.lpen, self.ldiag = pen, ld + pen
        fv, ft, fg = m.faces()
        b = ft[:, 1] == -1
        self.fv, self.ft = put(fv[b], torch.int64), put(ft[b, 0], torch.int64)
        # outward normals and areas as handed over at initialisation
        self.fn, self.fa = put(fg[b, 0:3]), put(fg[b, 3])

    def add(self, n, index, values):
        out = torch.zeros((n,) + tuple(values.shape[2:]), dtype=torch.float64, device=values.device)
        return out.index_add(0, index.reshape(-1), values.reshape((-1,) + tuple(values.shape[2:])))

    def grad_p(self, p):  # G_a p, [nv, 3]
        c = (self.vol / 4)[:, None] * torch.einsum("tj,tja->ta", p[self.tets], self.g)
        return self.add(self.nv, self.tets, c[:, None, :].expand(-1, 4, 3))

    def divergence(self, u):
        d = torch.einsum("tja,tja->t", u[self.tets], self.g) * self.vol / 4
        return self.add(self.nv, self.tets, d[:, None].expand(-1, 4))

    def step(self, case, u, p, inlet, nu=None):
        dirichlet = torch.where(self.inlet[:, None], inlet, torch.zeros_like(inlet))
        un = u[self.nodes]
        b = self.add(self.n, self.nodes, RHO * self.vol[:, None, None] * torch.einsum("ij,tjc->tic", self.mt, un)) / DT
        uv = un[:, :4]
        gu = torch.einsum("tja,tjb->tab", uv, self.g)
        conv = torch.einsum("tab,tb->ta", gu, uv.mean(1)) * self.vol[:, None]
        w = torch.tensor([1 / 4] * 4 + [1 / 24] * 6, dtype=torch.float64, device=u.device)
        b = b - self.add(self.n, self.nodes, w[None, :, None] * conv[:, None, :])
        b = b + torch.cat([-self.grad_p(p), torch.zeros_like(b[self.nv:])]) + self.penalty[:, None] * dirichlet

        def momentum(x):
            return torch.sparse.mm(self.A, x) + self.penalty[:, None] * x

        us = _Solve.apply(b, momentum, self.diag, dirichlet.detach())
        if nu is not None and nu.requires_grad:  # dA/dnu: K is proportional to 1 / nu
            kx = (self.vol / NU)[:, None, None] * (self.g10 @ (self.g10.transpose(1, 2) @ us.detach()[self.nodes]))
            us = _Solve.apply(b - self.add(self.n, self.nodes, kx) * (NU / nu - 1.0), momentum, self.diag, us.detach())

        def poisson(x):
            return torch.sparse.mm(self.L, x) + self.lpen[:, None] * x

        rhs = -self.divergence(us) / DT
        pc = _Solve.apply(rhs[:, None], poisson, self.ldiag, torch.zeros_like(rhs)[:, None])[:, 0]
        for _ in range(case["corrections"]):
            p = p + pc
            if not case["neumann"]:
                p = torch.where(self.outlet, torch.zeros_like(p), p)
            if self.ref >= 0:
                p = p - p[self.ref]
        new = us + torch.cat([-DT * self.invm[:self.nv, None] * self.grad_p(pc), torch.zeros_like(us[self.nv:])])
        return torch.where(self.fixed[:, None], dirichlet, new), p

    def face_forces(self, u, p, nu, shear, pressure):
        f = torch.zeros_like(self.fn)
        if shear:
            gu = torch.einsum("tjx,tjy->txy", u[self.tets[self.ft]], self.g[self.ft])
            f = f + nu * torch.einsum("txy,ty->tx", gu + gu.transpose(1, 2), self.fn) * self.fa[:, None]
        if pressure:
            f = f - (p[self.fv].mean(1) * self.fa)[:, None] * self.fn
        return self.add(self.nv, self.fv, (f / 3.0)[:, None, :].expand(-1, 3, 3))


def exact(case, seed):
    # the reference's criterion is dominated by the 1e10 penalty rows and leaves the interior loose:
    # iterates stopped by it are no approximation of the converged step
    if case["kind"] != "divergence" and case["norm"] == "reference" and not 0 < case["tol"] <= 1e-11:
        return None
    nt = _mesh_of(case).nTets()
    if nt > (1100000 if case["kind"] == "divergence" else 300000):
        return None
    d = _inputs(case, seed)
    f = _Flow(case, d.get("xyz"))
    u, p, inlet = f.put(d["u"]), f.put(d["p"]), f.put(d["inlet"])
    if case["kind"] == "divergence":
        return f.divergence(u)
    if case["kind"] == "adjoint":
        u0, p0, g = u.clone().requires_grad_(), p.clone().requires_grad_(), inlet.clone().requires_grad_()
        nu = torch.tensor(NU, dtype=torch.float64, device=u.device, requires_grad=True)
        u, p = u0, p0
        for _ in range(case["steps"]):
            u, p = f.step(case, u, p, g, nu)
        if case["objective"] == "wall_shear":
            x = f.put(f.m.vertices())[:, 0]
            patch = f.wall1 & (x >= 4.0) & (x <= 8.0)
            J = f.face_forces(u, p, nu, True, False)[patch].square().sum() / patch.sum()
        else:
            J = p[f.inlet1].mean() - p[f.outlet].mean()
        J.backward()
        return dict(J=float(J), grad_inlet=g.grad.cpu().numpy(), grad_viscosity=float(nu.grad),
                    grad_u0=u0.grad.cpu().numpy(), grad_p0=p0.grad.cpu().numpy())
    us, ps = [], []
    for k in range(case["steps"]):
        if case["kind"] == "stream":
            inlet = f.put(d["profiles"][k])
        u, p = f.step(case, u, p, inlet)
        us.append(u.cpu().numpy())
        ps.append(p.cpu().numpy())
    if case["kind"] == "stream":
        return dict(done=case["steps"], u=us, p=ps)
    out = dict(done=case["steps"], u=us[-1], p=ps[-1])
    if case["kind"] == "moving":
        out["force"] = f.face_forces(u, p, NU, True, True).cpu().numpy()
    return out
