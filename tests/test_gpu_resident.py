"""Resident Krylov solves at the sizes where their partitions can go wrong, bit for bit against the
oracle (same sums in the same order), and the pressure solvers with and without column windows."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RHO, NU = 1060.0, 0.004


def solver(cf, m, momentum, pressure, tol=1e-11):
    s = cf.NavierStokesSolver()
    s.setKrylovTolerances(tol, tol)
    s.setMaxIterations(5000, 20000)
    s.setMomentumSolver(momentum)
    s.setPressureSolver(pressure)
    s.setDt(0.01)
    s.initialize(m, cf.Fluid(RHO, NU))
    s.setMeanInletVelocity([0.5, 0.0, 0.0])
    return s


def mesh(cf, shape):
    m = cf.Mesh.cylinder(30.0, 2.0, *shape) if len(shape) == 2 else cf.Mesh.structuredRectangularPrism(6.0, 2.0, 1.5, *shape)
    m.setupBoundaryConditions((1.0, 0.0, 0.0), 1.0)
    return m


# rows of the momentum operator: below one 256-row block, on both sides of the one-CTA line (768
# rows), few blocks, more blocks than SMs with a ragged last slice
@pytest.mark.parametrize("shape", [(1, 2), (2, 5), (2, 6), (5, 3, 2), (9, 7, 3), (6, 40), (29, 17, 13)],
                         ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("momentum", [0, 1], ids=["cg", "bicgstab"])
def test_resident_solves_match_oracle(cf, po, shape, momentum):
    m = mesh(cf, shape)
    s = solver(cf, m, momentum, cf.KRYLOV_BICGSTAB)
    o = po.Oracle(m.vertices(), m.tets())
    o.set_fluid(RHO, NU)
    o.set_params(dt=0.01, tol_mom=1e-11, tol_p=1e-11, maxit_mom=5000, maxit_p=20000, pressure_solver=0)
    o.set_momentum_solver(1 if momentum == cf.KRYLOV_CG else 0)
    o.initialize()
    inlet = np.zeros((o.N2, 3))
    inlet[:, 0] = 0.5
    o.set_inlet(inlet)
    for _ in range(2):
        assert s.pisoStep() and o.piso_step() == 0
    ref = o.state()
    assert np.array_equal(s.getVelocity(), ref["u"]) and np.array_equal(s.getPressure(), ref["p"])


@pytest.mark.parametrize("shape", [(1, 2), (4, 9), (11, 9, 7), (8, 60)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("pressure", [0, 1, 2, 3], ids=["cg", "bicgstab", "cg1", "cg2l"])
def test_windows_do_not_change_the_bits(cf, monkeypatch, shape, pressure):
    m = mesh(cf, shape)
    got = []
    for off in ("0", "1"):
        monkeypatch.setenv("CFSA_NO_WINDOWS", off)
        s = solver(cf, m, cf.KRYLOV_CG, pressure)
        assert s.pisoSteps(2) == (True, 2)
        got.append((s.getVelocity(), s.getPressure(), s.stats()["pressure_iters"]))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert got[0][2] == got[1][2] > 0


# aggregates: one, a partial panel, several 32-column panels, more than one CTA's worth of columns,
# more boxes asked for than there are vertices
@pytest.mark.parametrize("target", [1, 31, 100, 700])
@pytest.mark.parametrize("shape", [(2, 3), (6, 30)], ids=lambda s: "x".join(map(str, s)))
def test_coarse_space_matches_oracle(cf, po, shape, target):
    m = mesh(cf, shape)
    s = solver(cf, m, cf.KRYLOV_CG, cf.KRYLOV_CG2L)
    s.setCoarseTarget(target)
    o = po.Oracle(m.vertices(), m.tets())
    o.set_fluid(RHO, NU)
    o.set_params(dt=0.01, tol_mom=1e-11, tol_p=1e-11, maxit_mom=5000, maxit_p=20000, pressure_solver=3)
    o.set_momentum_solver(1)
    o.set_coarse_target(target)
    o.initialize()
    inlet = np.zeros((o.N2, 3))
    inlet[:, 0] = 0.5
    o.set_inlet(inlet)
    assert s.pisoStep() and o.piso_step() == 0
    ref = o.state()
    assert np.array_equal(s.getVelocity(), ref["u"]) and np.array_equal(s.getPressure(), ref["p"])
    # a rebuild on moved vertices and back leaves the same coarse space
    x = m.vertices()
    u, p = s.getVelocity().copy(), s.getPressure().copy()
    s.updateVertices(x * [1.0, 1.01, 0.99])
    s.coarseSize()
    s.updateVertices(x)
    s.setFields(u, p)
    assert s.pisoStep() and o.piso_step() == 0
    ref = o.state()
    assert np.array_equal(s.getVelocity(), ref["u"]) and np.array_equal(s.getPressure(), ref["p"])


def test_coarse_space_rebuilt_while_another_handle_solves(cf):
    """The CTAs of one launch of the factorisation are not ordered: with another handle's resident solves
    holding the SMs they start one by one, and the coarse space must still come out the same to the bit."""
    m, busy = mesh(cf, (6, 30)), mesh(cf, (8, 60))
    x = m.vertices()
    s = solver(cf, m, cf.KRYLOV_CG, cf.KRYLOV_CG2L)
    s.setCoarseTarget(700)
    assert s.pisoStep()
    u, p = s.getVelocity().copy(), s.getPressure().copy()
    assert s.pisoStep()
    ref = s.getVelocity().copy(), s.getPressure().copy()
    t = solver(cf, busy, cf.KRYLOV_CG, cf.KRYLOV_CG, 1e-12)
    stop, ok = threading.Event(), []

    def keep_stepping():
        while not stop.is_set():
            ok.append(t.pisoStep())

    worker = threading.Thread(target=keep_stepping)
    worker.start()
    try:
        for _ in range(20):
            s.updateVertices(x * [1.0, 1.01, 0.99])
            s.coarseSize()
            s.updateVertices(x)
            s.setFields(u, p)
            assert s.pisoStep()
            assert np.array_equal(s.getVelocity(), ref[0]) and np.array_equal(s.getPressure(), ref[1])
    finally:
        stop.set()
        worker.join()
    assert ok and all(ok)


# The resident kernels' dynamic shared memory follows the handle's mesh, but the limit set for it belongs
# to the function: a smaller handle made later must not lower it for a larger one.
@pytest.mark.parametrize("pressure", [0, 1, 2, 3], ids=["cg", "bicgstab", "cg1", "cg2l"])
def test_small_handle_leaves_larger_one_its_shared_memory(cf, pressure):
    big, small = mesh(cf, (10, 58)), mesh(cf, (1, 2))
    alone = solver(cf, big, cf.KRYLOV_CG, pressure, 1e-8)
    assert alone.pisoStep() and alone.simpleStep()
    s = solver(cf, big, cf.KRYLOV_CG, pressure, 1e-8)
    t = solver(cf, small, cf.KRYLOV_CG, pressure, 1e-8)
    assert t.pisoStep()
    assert s.pisoStep()  # captured after the small handle was made
    t.updateVertices(small.vertices() * [1.0, 1.01, 0.99])  # rebuilds the small coarse space
    assert t.pisoStep()
    assert s.simpleStep()  # launched without a graph
    assert np.array_equal(s.getVelocity(), alone.getVelocity()) and np.array_equal(s.getPressure(), alone.getPressure())
    rhs = np.ones(s.nv)
    assert np.array_equal(s.solvePressureBiCGSTAB(rhs, None, 1e-8, 50)[0], alone.solvePressureBiCGSTAB(rhs, None, 1e-8, 50)[0])


# A wait that runs out in a momentum solve or in the pressure BiCGSTAB: the first wait gives up on its own,
# the host reads the status word, and the handle steps on. The small mesh's momentum solve is one CTA.
@pytest.mark.parametrize("shape", [(2, 5), (3, 12)], ids=["one_cta", "grid"])
@pytest.mark.parametrize("solve", ["momentum_cg", "momentum_bicgstab", "mixed_cg", "mixed_bicgstab", "pressure_bicgstab"])
@pytest.mark.parametrize("graph", [True, False], ids=["graph", "eager"])
def test_resident_solve_wait_runs_out(cf, shape, solve, graph):
    m = mesh(cf, shape)

    def make():
        s = solver(cf, m, cf.KRYLOV_CG if solve.endswith("_cg") else cf.KRYLOV_BICGSTAB, cf.KRYLOV_BICGSTAB)
        if solve.startswith("mixed"):
            s.setPrecision(cf.PRECISION_MIXED)
        return s

    ref, s = make(), make()
    step = (lambda q: q.pisoStep()) if graph else (lambda q: q.simpleStep())
    assert step(ref)
    u0, p0 = s.getVelocity().copy(), s.getPressure().copy()
    limit = s.setBarrierSpinLimit if solve.startswith("pressure") else s.setMomentumBarrierSpinLimit
    limit(0)
    with pytest.raises(cf.CfsaError, match="grid barrier") as e:
        step(s)
    assert e.value.code == cf.CUDA_ERROR
    assert s.getTime() == 0.0
    assert np.array_equal(s.getVelocity(), u0) and np.array_equal(s.getPressure(), p0)
    half = s.solvePressurePoisson if solve == "pressure_bicgstab" else s.solveMomentumPredictor
    with pytest.raises(cf.CfsaError, match="grid barrier"):
        half()
    if solve == "pressure_bicgstab":
        with pytest.raises(cf.CfsaError, match="grid barrier"):
            s.solvePressureBiCGSTAB(np.ones(s.nv))
    limit(-1)
    s.setFields(u0, p0)
    assert step(s)
    assert np.array_equal(s.getVelocity(), ref.getVelocity()) and np.array_equal(s.getPressure(), ref.getPressure())
    assert s.getTime() == ref.getTime() > 0.0


# A profiled run that was cut short at a grid barrier is an error, not a fast kernel.
@pytest.mark.parametrize("precision", [0, 1], ids=["fp64", "mixed"])
def test_profile_of_a_run_that_gave_up_fails(cf, precision):
    s = solver(cf, mesh(cf, (3, 12)), cf.KRYLOV_CG, cf.KRYLOV_CG1)
    assert s.pisoStep()
    u = s.getVelocity().copy()
    which = cf.KERNEL_MOMENTUM_SPMV_F32 if precision else cf.KERNEL_MOMENTUM_SPMV
    for limit, kernel in ((s.setMomentumBarrierSpinLimit, which), (s.setBarrierSpinLimit, cf.KERNEL_PRESSURE_SOLVE)):
        limit(0)
        with pytest.raises(cf.CfsaError, match="grid barrier"):
            s.profileKernel(kernel, 3)
        s.profileKernel(cf.KERNEL_PRESSURE_SPMV, 3)  # has no barrier
        limit(-1)
        ms, by = s.profileKernel(kernel, 3)
        assert ms > 0.0 and by > 0.0
    assert np.array_equal(s.getVelocity(), u)


# Vertices of no tet (left over in a mesh file): empty rows and columns, which neither the diagonals nor the
# CTAs' shares of the rows may trip over.
# 600: whole 256-row blocks of empty rows end the vertex part.
@pytest.mark.parametrize("extra", [1, 20, 600])
@pytest.mark.parametrize("momentum,pressure", [(0, 0), (1, 1), (0, 2), (0, 3)], ids=["cg", "bicgstab", "cg1", "cg2l"])
def test_vertices_of_no_tet(cf, po, extra, momentum, pressure):
    t = mesh(cf, (3, 12))
    inside = t.vertices().min(0) + np.random.default_rng(7).uniform(0.3, 0.7, (extra, 3)) * np.ptp(t.vertices(), axis=0)
    m = cf.Mesh.fromArrays(np.vstack([t.vertices(), inside]), t.tets())
    m.setupBoundaryConditions((1.0, 0.0, 0.0), 1.0)
    s = solver(cf, m, momentum, pressure)
    o = po.Oracle(m.vertices(), m.tets())
    o.set_fluid(RHO, NU)
    o.set_params(dt=0.01, tol_mom=1e-11, tol_p=1e-11, maxit_mom=5000, maxit_p=20000,
                 pressure_solver={0: 1, 1: 0, 2: 2, 3: 3}[pressure])
    o.set_momentum_solver(1 if momentum == cf.KRYLOV_CG else 0)
    o.initialize()
    inlet = np.zeros((o.N2, 3))
    inlet[:, 0] = 0.5
    o.set_inlet(inlet)
    for _ in range(2):
        assert s.pisoStep() and o.piso_step() == 0
    ref = o.state()
    assert np.array_equal(s.getVelocity(), ref["u"]) and np.array_equal(s.getPressure(), ref["p"])
    assert s.stats()["pressure_iters"] == o.stats()["pressure_iters"] > 0


# The momentum solves' forms (threads per CTA, chunk lengths, order of the vector phases) and the place of
# their chunk sums are chosen by size; here each runs on small odd meshes.
FORMS = [(t, g) for t in ("256", "512", "1024") for g in ("0", "1")]


def formed(cf, monkeypatch, form, m, momentum, pressure, tol):
    monkeypatch.setenv("CFSA_RESIDENT_THREADS", form[0])
    monkeypatch.setenv("CFSA_SUMS_GLOBAL", form[1])
    monkeypatch.setenv("CFSA_NO_WINDOWS", form[1])  # the pressure solve of meshes that large
    return solver(cf, m, momentum, pressure, tol)


# At 1e-30 BiCGSTAB passes its near-breakdown restart several times in both solves (on the oracle's side:
# momentum n = 671, 3175 and 1995 and pressure n = 114, 481 and 320).
@pytest.mark.parametrize("shape", [(2, 5), (3, 12), (9, 7, 3)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("momentum,tol", [(0, 1e-11), (1, 1e-30)], ids=["cg", "bicgstab_restarts"])
@pytest.mark.parametrize("form", FORMS, ids=lambda f: f"{f[0]}{'_global' if f[1] == '1' else ''}")
def test_forms_match_oracle(cf, po, monkeypatch, shape, momentum, tol, form):
    m = mesh(cf, shape)
    s = formed(cf, monkeypatch, form, m, momentum, cf.KRYLOV_BICGSTAB, tol)
    o = po.Oracle(m.vertices(), m.tets())
    o.set_fluid(RHO, NU)
    o.set_params(dt=0.01, tol_mom=tol, tol_p=tol, maxit_mom=5000, maxit_p=20000, pressure_solver=0)
    o.set_momentum_solver(1 if momentum == cf.KRYLOV_CG else 0)
    o.initialize()
    inlet = np.zeros((o.N2, 3))
    inlet[:, 0] = 0.5
    o.set_inlet(inlet)
    for _ in range(2):
        assert s.pisoStep() and o.piso_step() == 0
    ref = o.state()
    assert np.array_equal(s.getVelocity(), ref["u"]) and np.array_equal(s.getPressure(), ref["p"])
    assert s.stats()["momentum_iters"] == o.stats()["momentum_iters"]


@pytest.mark.parametrize("shape", [(2, 5), (9, 7, 3), (8, 31)], ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("momentum", [0, 1], ids=["cg", "bicgstab"])
def test_mixed_forms_agree(cf, monkeypatch, shape, momentum):
    m, got = mesh(cf, shape), []
    for form in FORMS:
        s = formed(cf, monkeypatch, form, m, momentum, cf.KRYLOV_CG2L, 1e-13)
        s.setPrecision(cf.PRECISION_MIXED)
        s.setConvergenceNorm(cf.NORM_JACOBI)
        assert s.pisoSteps(2) == (True, 2)
        got.append((s.getVelocity(), s.getPressure(), s.stats()["momentum_iters"], s.stats()["momentum_outer"]))
    for g in got[1:]:
        assert np.array_equal(g[0], got[0][0]) and np.array_equal(g[1], got[0][1])
        assert g[2:] == got[0][2:] and max(g[3]) > 1
    ref = solver(cf, m, momentum, cf.KRYLOV_CG2L, 1e-14)
    ref.setConvergenceNorm(cf.NORM_JACOBI)
    assert ref.pisoSteps(2) == (True, 2)
    # both solves end at 1e-13 of their right-hand side in the scaled norm: 1e-6 as in the mixed tests
    assert np.linalg.norm(got[0][0] - ref.getVelocity()) <= 1e-6 * np.linalg.norm(ref.getVelocity())


@pytest.mark.parametrize("shape", [(4, 9), (11, 9, 7)], ids=lambda s: "x".join(map(str, s)))
def test_windows_do_not_change_the_bits_of_float_sweeps(cf, monkeypatch, shape):
    m, got = mesh(cf, shape), []
    for off in ("0", "1"):
        monkeypatch.setenv("CFSA_NO_WINDOWS", off)
        s = solver(cf, m, cf.KRYLOV_CG, cf.KRYLOV_CG2L, 1e-10)
        s.setPrecision(cf.PRECISION_MIXED_FULL)
        assert s.pisoSteps(2) == (True, 2)
        got.append((s.getVelocity(), s.getPressure(), s.stats()["pressure_iters"], s.stats()["pressure_outer"]))
    assert np.array_equal(got[0][0], got[1][0]) and np.array_equal(got[0][1], got[1][1])
    assert got[0][2:] == got[1][2:] and got[0][3] > 1
