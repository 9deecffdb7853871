"""CG / GMRES with Jacobi, ILU(0), IC(0) on a jittered-channel SPD system against the oracle."""
import ctypes as C

import numpy as np
import pytest
import torch

import gpupfem2_gb300 as g
from gpupfem2_gb300 import meshgen as mg
from oracle import oracle as O
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


def _system(nx=64, ny=16):
    xy, tri = mg.channel(nx, ny, 4.0, 1.0)
    m = g.Mesh2D.from_arrays(xy, tri)
    A = g.SparseMatrixCSR(m)
    area, invJ = O.mesh_geometry(xy, tri)
    rp, col = O.csr_structure(xy.shape[0], tri)
    val, rhs = O.assemble_poisson(xy, tri, area, invJ, rp, col, 1, 1.0)
    diag = np.array([rp[i] + np.searchsorted(col[rp[i]:rp[i + 1]], i) for i in range(rp.size - 1)])
    val[diag] += 1e-2
    A.upload_values(val)
    return m, A, rp, col, val, rhs


@pytest.mark.parametrize("kind,pc", [("cg", "none"), ("cg", "jacobi"), ("cg", "ilu"), ("cg", "ic"),
                                     ("gmres", "jacobi"), ("gmres", "ilu"), ("gmres", "none")])
def test_solver_matches_oracle(cuda, kind, pc):
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    s = g.LinearSolver(A, kind, pc, tol=1e-8, maxit=1000)
    info = s.solve(A, x, b)
    fn = O.pcg if kind == "cg" else O.gmres
    ox, oinfo = fn(rp, col, val, rhs, tol=1e-8, maxit=1000, precond=pc)
    assert info.converged == 1 and oinfo.converged == 1
    assert abs(info.iterations - oinfo.iterations) <= 2
    # both stop at an absolute 1e-8 criterion; the solutions agree to the solve tolerance
    assert rel_err(x.cpu().numpy(), ox) < 1e-6


@pytest.mark.parametrize("pc", ["ilu", "ic"])
def test_preconditioner_apply_matches_oracle(cuda, pc):
    m, A, rp, col, val, rhs = _system(32, 8)
    s = g.LinearSolver(A, "cg", pc)
    s.setup(A)
    src = torch.tensor(rhs, device="cuda")
    dst = torch.empty_like(src)
    s.apply_preconditioner(dst, src)
    f = O.ilu0(rp, col, val) if pc == "ilu" else O.ic0(rp, col, val)
    ref = np.empty_like(rhs)
    tmp = np.empty_like(rhs)
    src_h = np.ascontiguousarray(rhs)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    O.lib().or_precond_apply.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 7
    O.lib().or_precond_apply(O.PRECOND[pc], rp.size - 1, p(rp), p(col), p(f), None, p(src_h), p(ref), p(tmp))
    assert rel_err(dst.cpu().numpy(), ref) < 1e-12


def test_gmres_restart_converges(cuda):
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    info = g.LinearSolver(A, "gmres", "jacobi", tol=1e-8, maxit=2000, restart=20).solve(A, x, b)
    ox, _ = O.pcg(rp, col, val, rhs, tol=1e-10, maxit=2000, precond="jacobi")
    assert info.converged == 1 and rel_err(x.cpu().numpy(), ox) < 1e-6


def test_spmv(cuda):
    m, A, rp, col, val, rhs = _system()
    x = np.random.default_rng(0).uniform(-1, 1, m.nv)
    y = torch.empty(m.nv, dtype=torch.float64, device="cuda")
    g.spmv(A, torch.tensor(x, device="cuda"), y)
    assert rel_err(y.cpu().numpy(), O.spmv(rp, col, val, x)) < 1e-14


@pytest.mark.parametrize("pc,ordering", [("jacobi", 0), ("ic", 0), ("ilu", 0), ("ic", 1), ("ilu", 1)])
def test_mixed_precision_refinement_reaches_fp64_residual(cuda, pc, ordering):
    """FP32 inner CG (FP32 Jacobi or FP32 ILU(0)/IC(0) factors) inside FP64 iterative
    refinement reaches ||b - A x|| <= 1e-8 ||b||, with the residual checked by the
    oracle's FP64 SpMV.  The multicolour order (ordering 1) runs the whole iteration on
    the permuted system's CSR arrays, the natural order the level-scheduled sweeps."""
    m, A, rp, col, val, rhs = _system(128, 32)
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    s = g.LinearSolver(A, "cg", pc, tol=1e-8, maxit=5000, criterion=g.CRITERION_REL,
                       precision=g.PRECISION_MIXED, ordering=ordering)
    info = s.solve(A, x, b)
    assert info.converged == 1 and info.outer_iterations >= 2
    xs = x.cpu().numpy()
    res = np.linalg.norm(rhs - O.spmv(rp, col, val, xs)) / np.linalg.norm(rhs)
    assert res <= 1e-8
    x64 = torch.zeros_like(b)
    info64 = g.LinearSolver(A, "cg", "jacobi", tol=1e-8, maxit=5000, criterion=g.CRITERION_REL).solve(A, x64, b)
    assert info64.converged == 1
    assert rel_err(xs, x64.cpu().numpy()) < 1e-6


def test_mixed_precision_on_the_permuted_csr_arrays_matches_the_slot_sweeps(cuda, monkeypatch):
    """Mixed-precision IC(0) CG on the multicolour order: the CSR path (whole iteration
    on B's arrays) and the slot sweeps (PF2_CG_SLOTS=1) reach the same solution, and at
    the iteration limit both keep the accumulated update."""
    m, A, rp, col, val, rhs = _system(128, 32)
    b = torch.tensor(rhs, device="cuda")
    out = {}
    for slots in ("0", "1"):
        monkeypatch.setenv("PF2_CG_SLOTS", slots)
        x = torch.zeros_like(b)
        s = g.LinearSolver(A, "cg", "ic", tol=1e-8, maxit=5000, criterion=g.CRITERION_REL,
                           precision=g.PRECISION_MIXED, ordering=1)
        info = s.solve(A, x, b)
        assert info.converged == 1
        y = torch.zeros_like(b)
        s5 = g.LinearSolver(A, "cg", "ic", tol=1e-30, maxit=5, criterion=g.CRITERION_REL,
                            precision=g.PRECISION_MIXED, ordering=1)
        lim = s5.solve(A, y, b, check=False)
        assert lim.converged == 0 and lim.iterations == 5
        ys, xs = y.cpu().numpy(), x.cpu().numpy()
        # CG lowers the A-norm of the error (not necessarily the residual's 2-norm)
        e5 = ys - xs
        assert np.isfinite(ys).all() and e5 @ O.spmv(rp, col, val, e5) < 0.5 * (xs @ O.spmv(rp, col, val, xs))
        # five FP32 iterations follow five FP64 ones up to FP32 rounding
        y64 = torch.zeros_like(b)
        g.LinearSolver(A, "cg", "ic", tol=1e-30, maxit=5, ordering=1).solve(A, y64, b, check=False)
        assert rel_err(ys, y64.cpu().numpy()) < 1e-4
        out[slots] = (xs, info.iterations, ys)
    assert abs(out["0"][1] - out["1"][1]) <= 3
    assert rel_err(out["0"][0], out["1"][0]) < 1e-6
    assert rel_err(out["0"][2], out["1"][2]) < 1e-4  # five FP32 iterations, two sweep orders


def _greedy_colour_perm(rp, col):
    n = rp.size - 1
    colour = -np.ones(n, int)
    for i in range(n):
        used = {colour[j] for j in col[rp[i]:rp[i + 1]] if j < i}
        c = 0
        while c in used:
            c += 1
        colour[i] = c
    return np.argsort(colour, kind="stable"), colour.max() + 1


@pytest.mark.parametrize("pc", ["ilu", "ic"])
def test_multicolour_preconditioner_matches_oracle_on_the_permuted_matrix(cuda, pc):
    m, A, rp, col, val, rhs = _system(32, 8)
    perm, ncol = _greedy_colour_perm(rp, col)
    assert ncol <= 10
    iperm = np.empty_like(perm)
    iperm[perm] = np.arange(perm.size)
    # B = P A P^T as CSR with sorted columns
    rows = []
    for r in range(perm.size):
        o = perm[r]
        ent = sorted((iperm[col[k]], val[k]) for k in range(rp[o], rp[o + 1]))
        rows.append(ent)
    brp = np.zeros(perm.size + 1, np.int32)
    brp[1:] = np.cumsum([len(e) for e in rows])
    bcol = np.array([c for e in rows for c, _ in e], np.int32)
    bval = np.array([v for e in rows for _, v in e])
    f = O.ilu0(brp, bcol, bval) if pc == "ilu" else O.ic0(brp, bcol, bval)
    src_b = np.ascontiguousarray(rhs[perm])
    out_b, tmp = np.empty_like(src_b), np.empty_like(src_b)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    O.lib().or_precond_apply.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 7
    O.lib().or_precond_apply(O.PRECOND[pc], perm.size, p(brp), p(bcol), p(f), None, p(src_b), p(out_b), p(tmp))
    ref = out_b[iperm]
    s = g.LinearSolver(A, "cg", pc, ordering=1)
    s.setup(A)
    src = torch.tensor(rhs, device="cuda")
    dst = torch.empty_like(src)
    s.apply_preconditioner(dst, src)
    assert rel_err(dst.cpu().numpy(), ref) < 1e-12


@pytest.mark.parametrize("pc", ["ilu", "ic"])
def test_multicolour_solve_agrees_with_natural(cuda, pc):
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    xs = []
    for ordering in (0, 1):
        x = torch.zeros_like(b)
        info = g.LinearSolver(A, "cg", pc, tol=1e-10, maxit=2000, criterion=g.CRITERION_REL,
                              ordering=ordering).solve(A, x, b)
        assert info.converged == 1
        xs.append(x.cpu().numpy())
    assert rel_err(xs[1], xs[0]) < 1e-8


@pytest.mark.parametrize("pc,restart", [("jacobi", 0), ("ilu", 0), ("jacobi", 20)])
def test_gmres_classical_gram_schmidt_twice_matches_oracle(cuda, pc, restart):
    """GMRES with classical Gram-Schmidt applied twice (two batched reductions per
    iteration) converges like the reference's modified Gram-Schmidt."""
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    info = g.LinearSolver(A, "gmres", pc, tol=1e-8, maxit=2000, restart=restart,
                          orthogonalization=1).solve(A, x, b)
    assert info.converged == 1
    if restart == 0:
        ox, oinfo = O.gmres(rp, col, val, rhs, tol=1e-8, maxit=2000, precond=pc)
        assert abs(info.iterations - oinfo.iterations) <= 2
    ref, _ = O.pcg(rp, col, val, rhs, tol=1e-12, maxit=5000, precond="jacobi")
    assert rel_err(x.cpu().numpy(), ref) < 1e-6


@pytest.mark.parametrize("pc", ["ilu", "ic"])
@pytest.mark.parametrize("band_rows", [None, "256"])
def test_banded_triangular_solves_match_oracle(cuda, pc, band_rows, monkeypatch):
    """Natural order on the 256 x 64 channel (about 320 levels): the banded solve (ranges
    of rows, one block each) gives the oracle's preconditioner, also with more ranges than
    blocks (256-row ranges), and the CG solve converges as the oracle's."""
    if band_rows:
        monkeypatch.setenv("PF2_BAND_ROWS", band_rows)
    m, A, rp, col, val, rhs = _system(256, 64)
    s = g.LinearSolver(A, "cg", pc, tol=1e-8, maxit=2000)
    s.setup(A)
    src = torch.tensor(rhs, device="cuda")
    dst = torch.empty_like(src)
    s.apply_preconditioner(dst, src)
    f = O.ilu0(rp, col, val) if pc == "ilu" else O.ic0(rp, col, val)
    ref, tmp = np.empty_like(rhs), np.empty_like(rhs)
    src_h = np.ascontiguousarray(rhs)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    O.lib().or_precond_apply.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 7
    O.lib().or_precond_apply(O.PRECOND[pc], rp.size - 1, p(rp), p(col), p(f), None, p(src_h), p(ref), p(tmp))
    assert rel_err(dst.cpu().numpy(), ref) < 1e-12
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    info = s.solve(A, x, b)
    ox, oinfo = O.pcg(rp, col, val, rhs, tol=1e-8, maxit=2000, precond=pc)
    assert info.converged == 1 and abs(info.iterations - oinfo.iterations) <= 2
    assert rel_err(x.cpu().numpy(), ox) < 1e-6


@pytest.mark.parametrize("pc,ordering", [("none", 0), ("jacobi", 0), ("ilu", 0), ("ic", 0), ("ic", 1)])
@pytest.mark.parametrize("criterion", [g.CRITERION_ABS, g.CRITERION_REL])
def test_one_reduction_cg_matches_standard(cuda, pc, ordering, criterion):
    """Chronopoulos-Gear CG (one fused reduction per iteration) reaches the standard
    iteration's solution within the solve tolerance in the same number of iterations, up
    to rounding at the stopping test."""
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    res = {}
    for variant in (g.CG_STANDARD, g.CG_ONE_REDUCTION):
        x = torch.zeros_like(b)
        s = g.LinearSolver(A, "cg", pc, tol=1e-8, maxit=2000, criterion=criterion, ordering=ordering,
                           cg_variant=variant)
        info = s.solve(A, x, b)
        assert info.converged == 1 and info.status == 0
        res[variant] = (x.cpu().numpy(), info.iterations)
    assert abs(res[0][1] - res[1][1]) <= 2
    assert rel_err(res[1][0], res[0][0]) < 1e-6
    ox, _ = O.pcg(rp, col, val, rhs, tol=1e-8, maxit=2000, precond=pc)
    assert rel_err(res[1][0], ox) < 1e-6


@pytest.mark.parametrize("pc", ["ic", "ilu"])
@pytest.mark.parametrize("criterion", [g.CRITERION_ABS, g.CRITERION_REL])
def test_pipelined_cg_matches_standard(cuda, pc, criterion):
    """Pipelined PCG (one grid-wide step per iteration, ILU(0)/IC(0) on the multicolour
    order, B's CSR arrays): the standard iteration's solution within the solve tolerance
    in the same number of iterations up to rounding at the stopping test."""
    m, A, rp, col, val, rhs = _system(128, 32)
    b = torch.tensor(rhs, device="cuda")
    res = {}
    for variant in (g.CG_STANDARD, g.CG_PIPELINED):
        x = torch.zeros_like(b)
        s = g.LinearSolver(A, "cg", pc, tol=1e-8, maxit=3000, criterion=criterion, ordering=1, cg_variant=variant)
        info = s.solve(A, x, b)
        assert info.converged == 1 and info.status == 0
        res[variant] = (x.cpu().numpy(), info.iterations)
    assert abs(res[0][1] - res[2][1]) <= 3
    assert rel_err(res[2][0], res[0][0]) < 1e-6
    if criterion == g.CRITERION_REL:
        r = rhs - O.spmv(rp, col, val, res[2][0])
        assert np.linalg.norm(r) <= 1e-8 * np.linalg.norm(rhs) * 1.01


def test_pipelined_cg_at_the_limit_and_off_the_csr_path(cuda, monkeypatch):
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    # seven iterations of each: the same Krylov iterate up to rounding
    xs = {}
    for variant in (g.CG_STANDARD, g.CG_PIPELINED):
        x = torch.zeros_like(b)
        info = g.LinearSolver(A, "cg", "ic", tol=1e-30, maxit=7, ordering=1, cg_variant=variant).solve(
            A, x, b, check=False)
        assert info.converged == 0 and info.iterations == 7
        xs[variant] = x.cpu().numpy()
    assert rel_err(xs[2], xs[0]) < 1e-9
    # slot sweeps (PF2_CG_SLOTS=1, not B's CSR arrays): the standard iteration runs, bit for bit
    monkeypatch.setenv("PF2_CG_SLOTS", "1")
    out = []
    for variant in (g.CG_STANDARD, g.CG_PIPELINED):
        x = torch.zeros_like(b)
        g.LinearSolver(A, "cg", "ic", tol=1e-8, maxit=2000, ordering=1, cg_variant=variant).solve(A, x, b)
        out.append(x.cpu().numpy())
    assert np.array_equal(out[0], out[1])


def test_one_reduction_cg_stops_at_the_limit(cuda):
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    s = g.LinearSolver(A, "cg", "jacobi", tol=1e-30, maxit=7, cg_variant=g.CG_ONE_REDUCTION)
    info = s.solve(A, x, b, check=False)
    assert info.converged == 0 and info.iterations == 7
    # seven one-reduction iterations equal seven standard ones up to rounding
    y = torch.zeros_like(b)
    g.LinearSolver(A, "cg", "jacobi", tol=1e-30, maxit=7).solve(A, y, b, check=False)
    assert rel_err(x.cpu().numpy(), y.cpu().numpy()) < 1e-10


@pytest.mark.parametrize("pc", ["none", "jacobi"])
@pytest.mark.parametrize("criterion", [g.CRITERION_ABS, g.CRITERION_REL])
def test_bicgstab_matches_oracle(cuda, pc, criterion):
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    info = g.LinearSolver(A, "bicgstab", pc, tol=1e-10, maxit=2000, criterion=criterion).solve(A, x, b)
    assert info.converged == 1 and info.status == 0
    ox, oinfo = O.pcg(rp, col, val, rhs, tol=1e-12, maxit=5000, precond="jacobi")
    assert rel_err(x.cpu().numpy(), ox) < 1e-6
    r = torch.empty_like(b)
    g.spmv(A, x, r)
    if criterion == g.CRITERION_REL:
        assert float(torch.linalg.norm(b - r)) <= 1e-10 * float(torch.linalg.norm(b)) * (1 + 1e-6)


def test_bicgstab_on_the_nonsymmetric_prediction_system(cuda):
    """The velocity-prediction matrix (outlet edge term: not symmetric) of a flow step:
    BiCGStab and GMRES reach the same solution."""
    xy, tri = mg.channel(64, 16, 4.0, 1.0)
    bu, bv, bp = mg.channel_boundary_nodes(xy, 4.0, 1.0)
    m = g.Mesh2D.from_arrays(xy, tri)
    m.set_channel_boundary_ids(4.0, 1.0)
    eng = g.FlowEngine(m, g.default_params(rho=1.0, mu=0.01, dt=0.005, level=2, n_outer=1), bu, bv, bp)
    eng.seed()
    eng.step()
    A, _ = eng.system(0)
    rp_, col_, val_ = A.download()
    dense = np.zeros((rp_.size - 1,) * 2)
    for i in range(rp_.size - 1):
        dense[i, col_[rp_[i]:rp_[i + 1]]] = val_[rp_[i]:rp_[i + 1]]
    assert np.abs(dense - dense.T).max() > 1e-12  # the outlet term breaks the symmetry
    n = A.rows
    b = torch.tensor(mg.uniform_pm1(3, n), device="cuda")
    x1, x2 = torch.zeros_like(b), torch.zeros_like(b)
    i1 = g.LinearSolver(A, "bicgstab", "jacobi", tol=1e-12, maxit=2000).solve(A, x1, b)
    i2 = g.LinearSolver(A, "gmres", "jacobi", tol=1e-12, maxit=2000).solve(A, x2, b)
    assert i1.converged == 1 and i2.converged == 1
    assert rel_err(x1.cpu().numpy(), x2.cpu().numpy()) < 1e-8


def test_bicgstab_stops_at_the_limit_and_rejects_triangular_preconditioners(cuda):
    m, A, rp, col, val, rhs = _system()
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    info = g.LinearSolver(A, "bicgstab", "jacobi", tol=1e-30, maxit=5).solve(A, x, b, check=False)
    assert info.converged == 0 and info.iterations == 5 and np.isfinite(x.cpu().numpy()).all()
    with pytest.raises(g.Pf2Error) as e:
        g.LinearSolver(A, "bicgstab", "ilu")
    assert e.value.status == g.BAD_INPUT


def test_bicgstab_half_step_solution_is_converged(cuda):
    """A diagonal system with power-of-two entries and the Jacobi preconditioner: the
    first half step (alpha = 1) solves it exactly, so s = 0 and t = A M^{-1} s = 0.  That is
    convergence, not a breakdown: x = b / d exactly, reported converged in one iteration."""
    xy, tri = mg.channel(8, 4, 4.0, 1.0)
    m = g.Mesh2D.from_arrays(xy, tri)
    A = g.SparseMatrixCSR(m)
    rp, col, _ = A.download()
    n = rp.size - 1
    d = 2.0 ** np.arange(-3, 5)[np.arange(n) % 8]
    val = np.zeros(col.size)
    for i in range(n):
        val[rp[i] + np.searchsorted(col[rp[i]:rp[i + 1]], i)] = d[i]
    A.upload_values(val)
    rhs = mg.uniform_pm1(7, n)
    for criterion in (g.CRITERION_ABS, g.CRITERION_REL):
        b = torch.tensor(rhs, device="cuda")
        x = torch.zeros_like(b)
        info = g.LinearSolver(A, "bicgstab", "jacobi", tol=1e-10, maxit=50, criterion=criterion).solve(A, x, b)
        assert info.converged == 1 and info.status == 0 and info.iterations == 1
        assert np.array_equal(x.cpu().numpy(), rhs / d)


def test_bicgstab_restarts_an_orthogonal_shadow_residual(cuda):
    """rhat = r0 supported on identity rows that the first iteration zeroes in r: the
    engine restarts the shadow residual as the oracle does and reaches its solution."""
    from tests.helpers import shadow_breakdown_system
    xy, tri, rp, col, val, rhs = shadow_breakdown_system()
    m = g.Mesh2D.from_arrays(xy, tri)
    A = g.SparseMatrixCSR(m)
    A.upload_values(val)
    ox, oinfo = O.bicgstab(rp, col, val, rhs, tol=1e-12, maxit=500, precond="jacobi")
    assert oinfo.converged == 1
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    info = g.LinearSolver(A, "bicgstab", "jacobi", tol=1e-12, maxit=500).solve(A, x, b)
    assert info.converged == 1 and info.iterations > 1
    # the dot products round differently (block sums against chunk sums): a few iterations
    assert abs(info.iterations - oinfo.iterations) <= 5
    assert rel_err(x.cpu().numpy(), ox) < 1e-9


@pytest.mark.parametrize("part", ["1", "0"])
def test_barrier_wait_that_runs_out_returns_timeout(cuda, monkeypatch, part):
    """A grid-barrier wait bounded to one poll (PF2_BARRIER_POLLS, read when the solver
    is created; a test knob) gives up before the other blocks arrive: the solve returns
    PF2_TIMEOUT with the record of the block and barrier that gave up, nothing faults, and
    a solver made afterwards with the normal limit solves on the same context.  Both the
    partitioned kernel (the default) and k_pcg (PF2_CG_PART=0)."""
    m, A, rp, col, val, rhs = _system(128, 32)
    b = torch.tensor(rhs, device="cuda")
    monkeypatch.setenv("PF2_CG_PART", part)
    monkeypatch.setenv("PF2_BARRIER_POLLS", "1")
    s = g.LinearSolver(A, "cg", "jacobi", tol=1e-8, maxit=1000)
    monkeypatch.delenv("PF2_BARRIER_POLLS")
    x = torch.zeros_like(b)
    with pytest.raises(g.Pf2Error) as e:
        s.solve(A, x, b)
    assert e.value.status == g.TIMEOUT
    assert "grid barrier timed out in the solver (block" in str(e.value)
    torch.cuda.synchronize()  # the context is still usable
    x = torch.zeros_like(b)
    info = g.LinearSolver(A, "cg", "jacobi", tol=1e-8, maxit=1000).solve(A, x, b)
    assert info.converged == 1 and info.status == 0
    ox, _ = O.pcg(rp, col, val, rhs, tol=1e-8, maxit=1000, precond="jacobi")
    assert rel_err(x.cpu().numpy(), ox) < 1e-6


def _cylinder_system():
    """The Poisson matrix of the quarter-size cylinder mesh (125,364 nodes) with a small
    shift, the size class of the flow's pressure solves."""
    xy, tri = mg.cylinder_channel(nxh=350, nyh=400, nr=12)
    m = g.Mesh2D.from_arrays(xy, tri)
    A = g.SparseMatrixCSR(m)
    area, invJ = O.mesh_geometry(xy, tri)
    rp, col = O.csr_structure(xy.shape[0], tri)
    val, rhs = O.assemble_poisson(xy, tri, area, invJ, rp, col, 1, 1.0)
    diag = np.array([rp[i] + np.searchsorted(col[rp[i]:rp[i + 1]], i) for i in range(rp.size - 1)])
    val[diag] += 1e-2
    A.upload_values(val)
    return m, A, rp, col, val, rhs


def _solve_both(monkeypatch, A, rhs, pc, ordering, parts="", **kw):
    """The same solve by the partitioned kernel (PF2_CG_PART=2: solver creation fails
    unless it applies) and by the kernels it replaces (PF2_CG_PART=0); keyed "1" and "0"."""
    b = torch.tensor(rhs, device="cuda")
    out = {}
    for part in ("2", "0"):
        monkeypatch.setenv("PF2_CG_PART", part)
        if parts:
            monkeypatch.setenv("PF2_CG_PARTS", parts)
        x = torch.zeros_like(b)
        info = g.LinearSolver(A, "cg", pc, ordering=ordering, **kw).solve(A, x, b, check=False)
        out["1" if part == "2" else part] = (x.cpu().numpy(), info)
    return out


@pytest.mark.parametrize("pc,ordering", [("none", 0), ("jacobi", 0), ("ic", 1), ("ilu", 1)])
@pytest.mark.parametrize("parts", ["", "7"])
def test_partitioned_cg_matches_the_other_kernels(cuda, monkeypatch, pc, ordering, parts):
    """The partitioned CG (one part per block with its vectors in shared memory; 4 parts
    of the 2,193-row system, or 7 with PF2_CG_PARTS) against k_pcg / pcg_csr
    (PF2_CG_PART=0) and the oracle, converged to an absolute 1e-12: each row's arithmetic
    is the same, the reductions' order differs, so the solutions agree to 1e-10 and the
    iteration counts within 2."""
    m, A, rp, col, val, rhs = _system(128, 16)
    out = _solve_both(monkeypatch, A, rhs, pc, ordering, parts, tol=1e-12, maxit=5000)
    (xp, ip), (xo, io) = out["1"], out["0"]
    assert ip.converged == 1 and io.converged == 1 and ip.status == 0
    assert abs(ip.iterations - io.iterations) <= 2
    assert rel_err(xp, xo) < 1e-10
    if pc in ("none", "jacobi"):
        ox, oi = O.pcg(rp, col, val, rhs, tol=1e-12, maxit=5000, precond=pc)
        assert oi.converged == 1 and rel_err(xp, ox) < 1e-10


@pytest.mark.parametrize("pc,ordering", [("jacobi", 0), ("ic", 1)])
def test_partitioned_cg_relative_criterion_and_cap(cuda, monkeypatch, pc, ordering):
    """The relative criterion (r.r reduced every iteration) converges like the other
    kernels; at an iteration cap far from convergence (40 iterations) both paths stop with
    the same count, report the same ||r|| / ||b||, and their iterates agree to 1e-9."""
    m, A, rp, col, val, rhs = _system(128, 16)
    out = _solve_both(monkeypatch, A, rhs, pc, ordering, tol=1e-10, maxit=5000, criterion=g.CRITERION_REL)
    (xp, ip), (xo, io) = out["1"], out["0"]
    assert ip.converged == 1 and io.converged == 1 and abs(ip.iterations - io.iterations) <= 2
    assert ip.residual <= 1e-10 and rel_err(xp, xo) < 1e-8
    res = np.linalg.norm(rhs - O.spmv(rp, col, val, xp)) / np.linalg.norm(rhs)
    assert res <= 2e-10
    out = _solve_both(monkeypatch, A, rhs, pc, ordering, tol=1e-30, maxit=40)
    (xp, ip), (xo, io) = out["1"], out["0"]
    assert ip.converged == 0 and io.converged == 0 and ip.iterations == io.iterations == 40
    assert rel_err(xp, xo) < 1e-9


def test_partitioned_cg_on_the_cylinder_mesh(cuda, monkeypatch):
    """IC(0) on the multicolour order, 152 parts (one per SM) of the 125,364-row cylinder
    system: the partitioned kernel and pcg_csr reach the same converged solution (1e-10)
    in the same number of iterations (within 2)."""
    m, A, rp, col, val, rhs = _cylinder_system()
    out = _solve_both(monkeypatch, A, rhs, "ic", 1, tol=1e-12, maxit=20000)
    (xp, ip), (xo, io) = out["1"], out["0"]
    print("cylinder IC(0): partitioned %d iterations, pcg_csr %d, rel diff %.2e" % (
        ip.iterations, io.iterations, rel_err(xp, xo)))
    assert ip.converged == 1 and io.converged == 1 and abs(ip.iterations - io.iterations) <= 2
    assert rel_err(xp, xo) < 1e-10


@pytest.mark.parametrize("pc", ["ic", "ilu"])
@pytest.mark.parametrize("local", ["1", "0"])
def test_partitioned_mixed_cg_matches_the_csr_kernel(cuda, monkeypatch, pc, local):
    """Mixed-precision CG on the parts (FP32 vectors in shared memory, FP32 sweeps and
    SpMV, FP64 refinement; 8 parts of the 4,257-row system, or 7 forced) against the mixed
    kernel on B's CSR arrays (PF2_CG_PART=0): both reach ||b - A x|| <= 1e-8 ||b||
    (checked with the oracle's FP64 SpMV) and agree with the FP64 solution to 1e-6.  With
    the global factors (the default) the iteration counts agree within 10 %; with the
    partition-local factors (PF2_CG_PART_LOCAL=1: one IC(0) / ILU(0) block per part, no
    wait on another part in the sweeps) the solve takes at most 1.6 times the iterations."""
    monkeypatch.setenv("PF2_CG_PART_LOCAL", local)
    m, A, rp, col, val, rhs = _system(128, 32)
    b = torch.tensor(rhs, device="cuda")
    x64 = torch.zeros_like(b)
    g.LinearSolver(A, "cg", "jacobi", tol=1e-12, maxit=20000, criterion=g.CRITERION_REL).solve(A, x64, b)
    x64 = x64.cpu().numpy()
    for parts in ("", "7"):
        if parts:
            monkeypatch.setenv("PF2_CG_PARTS", parts)
        out = _solve_both(monkeypatch, A, rhs, pc, 1, tol=1e-8, maxit=5000, criterion=g.CRITERION_REL,
                          precision=g.PRECISION_MIXED)
        for key, (x, info) in out.items():
            res = np.linalg.norm(rhs - O.spmv(rp, col, val, x)) / np.linalg.norm(rhs)
            print("mixed %s local %s parts %s path %s: %d iterations, %d refinements, residual %.2e" % (
                pc, local, parts or "default", key, info.iterations, info.outer_iterations, res))
            assert info.converged == 1 and info.outer_iterations >= 2 and res <= 1e-8
            assert rel_err(x, x64) < 1e-6
        ip, io = out["1"][1].iterations, out["0"][1].iterations
        if local == "0":
            assert abs(ip - io) <= 0.1 * io + 2
        else:
            assert ip <= 1.6 * io


def test_partitioned_mixed_cg_on_the_cylinder_mesh(cuda, monkeypatch):
    """Mixed IC(0) on the 152 parts of the 125,364-row cylinder system: 1e-8 relative in
    FP64 and within 1e-6 of the FP64 solve, in about as many iterations as the mixed
    kernel on B's CSR arrays."""
    m, A, rp, col, val, rhs = _cylinder_system()
    out = _solve_both(monkeypatch, A, rhs, "ic", 1, tol=1e-8, maxit=20000, criterion=g.CRITERION_REL,
                      precision=g.PRECISION_MIXED)
    b = torch.tensor(rhs, device="cuda")
    x64 = torch.zeros_like(b)
    g.LinearSolver(A, "cg", "ic", tol=1e-12, maxit=20000, criterion=g.CRITERION_REL, ordering=1).solve(A, x64, b)
    x64 = x64.cpu().numpy()
    for key, (x, info) in out.items():
        res = np.linalg.norm(rhs - O.spmv(rp, col, val, x)) / np.linalg.norm(rhs)
        print("cylinder mixed IC(0) path %s: %d iterations, residual %.2e" % (key, info.iterations, res))
        assert info.converged == 1 and res <= 1e-8 and rel_err(x, x64) < 1e-6
    assert abs(out["1"][1].iterations - out["0"][1].iterations) <= 0.1 * out["0"][1].iterations + 2


@pytest.mark.parametrize("pc,precision", [("none", 0), ("jacobi", 0), ("ic", 0), ("ilu", 0), ("ic", 1), ("ilu", 1)])
@pytest.mark.parametrize("parts,resident", [("1", "1"), ("2", "1"), ("7", "1"), ("23", "1"), ("70", "1"), ("7", "0")])
def test_halo_cg_matches_the_waiting_sweeps(cuda, monkeypatch, pc, precision, parts, resident):
    """The partitioned CG with halo rows (no wait inside a sweep) against the partitioned
    kernel whose sweeps wait for other parts (PF2_CG_PART=3): the rows' arithmetic is the
    same, so both converge in the same number of iterations (within 2; mixed: 10 %) to
    solutions within 1e-10 (FP64, ||r|| <= 1e-12 ||b|| on a system of condition ~1e4) and
    1e-6 (mixed, 1e-8).  One part (no halo), two, seven ragged ones, 23 parts of ~95 rows whose halo
    is as large as the part, 70 parts (a wait that watches the arrival counter); the entries
    resident in shared memory, or read from L2."""
    m, A, rp, col, val, rhs = _system(128, 16)
    b = torch.tensor(rhs, device="cuda")
    monkeypatch.setenv("PF2_CG_PARTS", parts)
    monkeypatch.setenv("PF2_HALO_RESIDENT", resident)
    out = {}
    for part in ("2", "3"):
        monkeypatch.setenv("PF2_CG_PART", part)
        x = torch.zeros_like(b)
        s = g.LinearSolver(A, "cg", pc, ordering=1 if pc in ("ic", "ilu") else 0, precision=precision,
                           tol=1e-8 if precision else 1e-12, maxit=5000, criterion=g.CRITERION_REL)
        out[part] = (s.solve(A, x, b), x)
    (i2, x2), (i3, x3) = out["2"], out["3"]
    assert i2.converged == 1 and i3.converged == 1 and i2.status == 0
    assert abs(i2.iterations - i3.iterations) <= (0.1 * i3.iterations + 2 if precision else 2)
    assert rel_err(x2.cpu().numpy(), x3.cpu().numpy()) < (1e-6 if precision else 1e-10)


def _odd_mesh(kind):
    """channel: ordinary levels; box: up to 13 dependencies a row; wide: few levels, of several units; ring: an
    annulus numbered around, whose last rows depend on ones that have left the sweeps' window of
    solved values; hub / star: a last row of 30 / 20 neighbours, solved one after the other / in the
    two levels before; axis: tetrahedra around an edge, rows of 43 entries."""
    if kind == "channel":
        return mg.channel(64, 16, 4.0, 1.0)
    if kind == "box":
        return mg.box_tets(9, 7, 5)
    if kind == "wide":
        xy, tri = mg.channel(64, 16, 4.0, 1.0)
        order = np.random.default_rng(3).permutation(len(xy))
        return np.asarray(xy)[order], np.argsort(order)[np.asarray(tri)].astype(np.int32)
    if kind == "ring":
        n = 1500
        k = np.arange(n)
        t = 2 * np.pi * k / n
        xy = np.stack([np.stack([r * np.cos(t), r * np.sin(t)], 1) for r in (1.0, 1.01)], 1).reshape(-1, 2)
        a, b = 2 * k, 2 * ((k + 1) % n)
        return xy, np.concatenate([np.stack([a, a + 1, b], 1), np.stack([b, a + 1, b + 1], 1)]).astype(np.int32)
    if kind == "axis":
        n = 40
        t = 2 * np.pi * np.arange(n) / n
        xyz = np.concatenate([np.stack([np.cos(t), np.sin(t), 0 * t], 1), [[0, 0, -1.0], [0, 0, 1.0]]])
        k = np.arange(n)
        return xyz, np.stack([np.full(n, n), k, (k + 1) % n, np.full(n, n + 1)], 1).astype(np.int32)
    n = 30 if kind == "hub" else 20
    t = 2 * np.pi * np.arange(n) / n
    xy = np.concatenate([np.stack([np.cos(t), np.sin(t)], 1), np.zeros((1, 2))])
    # star: every second rim node first, so two levels before the hub's
    name = np.arange(n) if kind == "hub" else np.arange(n) // 2 + np.arange(n) % 2 * (n // 2)
    pts = np.empty_like(xy)
    pts[name], pts[n] = xy[:n], xy[n]
    nxt = np.roll(name, -1)
    return pts, np.stack([name, nxt, np.full(n, n)], 1).astype(np.int32)


@pytest.mark.parametrize("pc", ["ic", "ilu"])
@pytest.mark.parametrize("kind", ["channel", "box", "wide", "ring", "hub", "star", "axis"])
def test_level_sweeps_match_the_other_solves(cuda, monkeypatch, kind, pc):
    """CG in the natural order with one block's level sweeps (PF2_CG_LEVEL=2) against the banded, slot
    or ticket solve (0).  After 6 iterations only rounding differs: off-diagonal sums within 1/1.05
    of the diagonal bound the condition of every factor and of the matrix by 41, so the iterates
    differ by at most some 6 x 20 operations x 41 x 1.1e-16 = 5.4e-13 relative; 1e-11 allowed.  To
    convergence, the iteration counts agree within one."""
    xy, cells = _odd_mesh(kind)
    cells = np.asarray(cells)
    m = (g.Mesh3D if cells.shape[1] == 4 else g.Mesh2D).from_arrays(xy, cells)
    A = g.SparseMatrixCSR(m)
    rp, col, _ = A.download()
    n = rp.size - 1
    row = np.repeat(np.arange(n), np.diff(rp))
    val = np.where(row == col, 0.0, -1.0 - 0.3 * np.cos(row + col.astype(np.float64)))
    sums = np.zeros(n)
    np.add.at(sums, row, -val)
    val[row == col] = 1.05 * sums
    A.upload_values(val)
    b = torch.tensor(np.sin(1.0 + np.arange(n)), device="cuda")
    out = {}
    for level in ("2", "0"):
        monkeypatch.setenv("PF2_CG_LEVEL", level)
        x6, x = torch.zeros_like(b), torch.zeros_like(b)
        g.LinearSolver(A, "cg", pc, tol=0.0, maxit=6, criterion=g.CRITERION_REL).solve(A, x6, b, check=False)
        info = g.LinearSolver(A, "cg", pc, tol=1e-9, maxit=500, criterion=g.CRITERION_REL).solve(A, x, b)
        assert info.converged == 1 and info.status == 0
        out[level] = (info.iterations, x6.cpu().numpy())
    assert abs(out["2"][0] - out["0"][0]) <= 1
    assert rel_err(out["2"][1], out["0"][1]) < 1e-11


@pytest.mark.parametrize("nx,ny,pc,restart", [(12, 4, "none", 0), (48, 12, "jacobi", 0), (64, 24, "none", 0),
                                              (256, 64, "jacobi", 0), (64, 24, "none", 33), (64, 24, "ilu", 7)])
def test_gmres_low_synchronisation_follows_modified_gram_schmidt(cuda, nx, ny, pc, restart):
    """GMRES whose projections share one exchange per iteration (h = (I + L)^{-1} V^T w) against the
    oracle's one-after-another modified Gram-Schmidt: the coefficients are the same up to
    rounding, so the iteration counts agree within 2 and both solutions meet ||r|| <= 1e-10, on
    one block and on many, up to bases of more than 96 vectors (the blocks' own copy of L); with
    restarts the residual alone is checked.  (A system of condition ~1e4: solutions within 1e-6.)"""
    m, A, rp, col, val, rhs = _system(nx, ny)
    b = torch.tensor(rhs, device="cuda")
    x = torch.zeros_like(b)
    info = g.LinearSolver(A, "gmres", pc, tol=1e-10, maxit=1000, restart=restart).solve(A, x, b)
    assert info.converged == 1 and info.status == 0
    xs = x.cpu().numpy()
    if restart == 0:
        ox, oinfo = O.gmres(rp, col, val, rhs, tol=1e-10, maxit=1000, precond=pc)
        assert abs(info.iterations - oinfo.iterations) <= 2
        assert rel_err(xs, ox) < 1e-6
    diag = np.array([val[rp[i] + np.searchsorted(col[rp[i]:rp[i + 1]], i)] for i in range(rp.size - 1)])
    r = rhs - O.spmv(rp, col, val, xs)
    if pc == "none":
        assert np.linalg.norm(r) <= 1.01e-10 + 1e-13 * np.linalg.norm(rhs)
    elif pc == "jacobi":
        assert np.linalg.norm(r / diag) <= 1.01e-10 + 1e-13 * np.linalg.norm(rhs / diag)
    else:
        assert np.linalg.norm(r) <= 1e-7 * np.linalg.norm(rhs)


@pytest.mark.parametrize("pc", ["ic", "ilu"])
@pytest.mark.parametrize("kind", ["channel", "box", "wide", "ring", "hub", "star", "axis"])
def test_factors_of_odd_patterns_match_the_oracle(cuda, kind, pc):
    """ILU(0) / IC(0) of a warp per row (rows of up to 32 entries held by its lanes) against the
    oracle's, through one preconditioner apply: the same sums in the same order up to fused
    multiply-adds.  Factors and solves of a matrix whose off-diagonal sums stay within 1/1.05 of
    the diagonal amplify rounding by at most ~41 (32 operations a row: 41 x 32 x 1.1e-16 =
    1.4e-13); 1e-12 allowed."""
    xy, cells = _odd_mesh(kind)
    cells = np.asarray(cells)
    m = (g.Mesh3D if cells.shape[1] == 4 else g.Mesh2D).from_arrays(xy, cells)
    A = g.SparseMatrixCSR(m)
    rp, col, _ = A.download()
    n = rp.size - 1
    row = np.repeat(np.arange(n), np.diff(rp))
    val = np.where(row == col, 0.0, -1.0 - 0.3 * np.cos(row + col.astype(np.float64)))
    sums = np.zeros(n)
    np.add.at(sums, row, -val)
    val[row == col] = 1.05 * sums
    A.upload_values(val)
    s = g.LinearSolver(A, "cg", pc)
    s.setup(A)
    src = np.sin(1.0 + np.arange(n))
    dst = torch.empty(n, dtype=torch.float64, device="cuda")
    s.apply_preconditioner(dst, torch.tensor(src, device="cuda"))
    f = O.ilu0(rp, col, val) if pc == "ilu" else O.ic0(rp, col, val)
    ref, tmp = np.empty(n), np.empty(n)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    O.lib().or_precond_apply.argtypes = [C.c_int, C.c_int] + [C.c_void_p] * 7
    O.lib().or_precond_apply(O.PRECOND[pc], n, p(rp), p(col), p(f), None, p(src), p(ref), p(tmp))
    assert rel_err(dst.cpu().numpy(), ref) < 1e-12


@pytest.mark.parametrize("pc", ["ic", "ilu"])
@pytest.mark.parametrize("ordering", [0, 1])
def test_factorisations_are_repeatable_bit_for_bit(cuda, pc, ordering):
    """Rows of a factorisation wait for the rows that they depend on and then read them with all lanes of
    a warp: whatever the order in which rows finish, every factorisation gives the same bits
    (compared through one preconditioner apply; 64 of them on 4,257 rows in 160 levels, or in
    a few colours)."""
    m, A, rp, col, val, rhs = _system(128, 32)
    src = torch.tensor(np.sin(1.0 + np.arange(rp.size - 1)), device="cuda")
    s = g.LinearSolver(A, "cg", pc, ordering=ordering)
    first, dst = torch.empty_like(src), torch.empty_like(src)
    for k in range(64):
        s.setup(A)
        s.apply_preconditioner(dst if k else first, src)
        assert k == 0 or torch.equal(dst.view(torch.int64), first.view(torch.int64))


@pytest.mark.parametrize("kind,pc,ordering,precision,gs,level", [
    ("cg", "jacobi", 0, 0, 0, None), ("cg", "none", 0, 0, 0, None), ("cg", "ic", 1, 0, 0, None),
    ("cg", "ilu", 1, 0, 0, None), ("cg", "ic", 1, 1, 0, None), ("cg", "ilu", 1, 1, 0, None),
    ("cg", "ic", 0, 0, 0, None), ("cg", "ic", 0, 0, 0, "0"), ("cg", "ilu", 0, 1, 0, "0"),
    ("gmres", "ilu", 0, 0, 0, None), ("gmres", "ilu", 0, 0, 1, None)])
def test_a_smaller_solver_leaves_a_larger_one_alone(cuda, monkeypatch, kind, pc, ordering, precision, gs, level):
    """Two solvers of the same kernel alive at once, the smaller created last: the larger one still
    solves, to the bits it gave before, and its preconditioner applies.  (How much shared memory a
    kernel may take is a property of the kernel, not of a solver.)"""
    if level is not None:
        monkeypatch.setenv("PF2_CG_LEVEL", level)
    systems = [_system(256, 64), _system(32, 16)]
    mk = lambda A: g.LinearSolver(A, kind, pc, tol=1e-6, maxit=2000, ordering=ordering, precision=precision,  # noqa: E731
                                  orthogonalization=gs, criterion=g.CRITERION_REL if kind == "cg" else 0)

    def solve(s, system):
        A, b = system[1], torch.tensor(system[5], device="cuda")
        x, z = torch.zeros_like(b), torch.empty_like(b)
        assert s.solve(A, x, b).converged == 1
        s.apply_preconditioner(z, b)
        return x, z

    large = mk(systems[0][1])
    before = solve(large, systems[0])
    small = mk(systems[1][1])
    solve(small, systems[1])
    after = solve(large, systems[0])
    for u, v in zip(before, after):
        assert torch.equal(u.view(torch.int64), v.view(torch.int64))


def _numbered(xy, cells, key):
    order = np.argsort(key, kind="stable")
    return np.asarray(xy)[order], np.argsort(order)[np.asarray(cells)].astype(np.int32)


@pytest.mark.parametrize("kind,sweeps", [("own", True), ("shuffled small", True), ("coloured", False),
                                         ("shuffled", False), ("tetrahedra", True), ("shuffled tetrahedra", False)])
def test_wide_levels_keep_the_solve_on_all_sms(cuda, monkeypatch, kind, sweeps):
    """CG with IC(0) in the natural order takes one block's level sweeps where levels are narrow, and the
    kernels that share the triangles among all SMs where they are wide (a mesh numbered by colours, or
    without any order): bit for bit the iterates of the forced kernel, which differ between the two."""
    rng = np.random.default_rng(5)
    if "tetrahedra" in kind:
        xy, cells = mg.box_tets(*((20, 10, 8) if kind == "tetrahedra" else (60, 30, 20)))
    else:
        xy, cells = mg.channel(*{"coloured": (180, 86), "shuffled": (400, 120)}.get(kind, (64, 16)), 4.0, 1.0)
    if "shuffled" in kind:
        xy, cells = _numbered(xy, cells, rng.random(len(xy)))
    M = g.Mesh3D if np.asarray(cells).shape[1] == 4 else g.Mesh2D
    if kind == "coloured":
        rp, col, _ = g.SparseMatrixCSR(M.from_arrays(xy, cells)).download()
        colour = []
        for i in range(rp.size - 1):
            used = {colour[j] for j in col[rp[i]:rp[i + 1]] if j < i}
            colour.append(next(c for c in range(len(used) + 1) if c not in used))
        xy, cells = _numbered(xy, cells, np.array(colour))
    m = M.from_arrays(xy, cells)
    A = g.SparseMatrixCSR(m)
    rp, col, _ = A.download()
    n = rp.size - 1
    row = np.repeat(np.arange(n), np.diff(rp))
    val = np.where(row == col, 0.0, -1.0 - 0.3 * np.cos(row + col.astype(np.float64)))
    sums = np.zeros(n)
    np.add.at(sums, row, -val)
    val[row == col] = 1.05 * sums
    A.upload_values(val)
    b = torch.tensor(np.sin(1.0 + np.arange(n)), device="cuda")
    out = {}
    for level in ("2", "0", None):
        if level is None:
            monkeypatch.delenv("PF2_CG_LEVEL")
        else:
            monkeypatch.setenv("PF2_CG_LEVEL", level)
        x = torch.zeros_like(b)
        g.LinearSolver(A, "cg", "ic", tol=0.0, maxit=6, criterion=g.CRITERION_REL).solve(A, x, b, check=False)
        out[level] = x.view(torch.int64)
    assert not torch.equal(out["2"], out["0"])
    assert torch.equal(out[None], out["2" if sweeps else "0"])


@pytest.mark.parametrize("pc,precision", [("none", 0), ("jacobi", 0), ("ic", 0), ("ilu", 0), ("ic", 1), ("ilu", 1)])
@pytest.mark.parametrize("parts,resident", [("1", "0"), ("2", "1"), ("7", "1"), ("23", "1"), ("70", "1"), ("7", "0")])
def test_the_halo_form_is_the_one_compared(cuda, monkeypatch, pc, precision, parts, resident):
    """The systems and parts of the comparison with the waiting sweeps are solved by the kernel with
    halo rows, with resident entries or (one part of 2,193 rows, or where asked) with entries read from
    L2: creation that requires it (PF2_CG_PART=4) succeeds, and its solve gives the bits of the one
    that requires some partitioned kernel (2)."""
    m, A, rp, col, val, rhs = _system(128, 16)
    b = torch.tensor(rhs, device="cuda")
    monkeypatch.setenv("PF2_CG_PARTS", parts)
    monkeypatch.setenv("PF2_HALO_RESIDENT", resident)
    out = []
    for part in ("4", "2"):
        monkeypatch.setenv("PF2_CG_PART", part)
        x = torch.zeros_like(b)
        s = g.LinearSolver(A, "cg", pc, ordering=1 if pc in ("ic", "ilu") else 0, precision=precision,
                           tol=1e-8 if precision else 1e-12, maxit=5000, criterion=g.CRITERION_REL)
        assert s.solve(A, x, b).converged == 1
        out.append(x.view(torch.int64))
    assert torch.equal(*out)


def test_requiring_the_halo_form_where_it_does_not_apply_is_refused(cuda, monkeypatch):
    """Parts of a dozen rows of a tetrahedral mesh in eight colours, whose halos are many times as large,
    and a solver kind that has no parts."""
    m = g.Mesh3D.from_arrays(*mg.box_tets(12, 10, 8))
    A = g.SparseMatrixCSR(m)
    monkeypatch.setenv("PF2_CG_PART", "4")
    monkeypatch.setenv("PF2_CG_PARTS", "100")
    for kind in ("cg", "gmres"):
        with pytest.raises(g.Pf2Error) as e:
            g.LinearSolver(A, kind, "ic", ordering=1)
        assert e.value.status == g.BAD_INPUT
    monkeypatch.setenv("PF2_CG_PART", "2")
    g.LinearSolver(A, "cg", "ic", ordering=1)


@pytest.mark.parametrize("kind,pc", [("gmres", "jacobi"), ("gmres", "ilu"), ("cg", "ic")])
def test_waits_of_gmres_and_of_the_level_sweeps_that_run_out_return_timeout(cuda, monkeypatch, kind, pc):
    """As above for the exchanges of GMRES with modified Gram-Schmidt and for the blocks that wait for the
    level sweeps: one poll is not enough, the solve returns PF2_TIMEOUT, and the next solver works."""
    m, A, rp, col, val, rhs = _system(128, 32)
    b = torch.tensor(rhs, device="cuda")
    if kind == "cg":
        monkeypatch.setenv("PF2_CG_LEVEL", "2")
    monkeypatch.setenv("PF2_BARRIER_POLLS", "1")
    s = g.LinearSolver(A, kind, pc, tol=1e-8, maxit=1000)
    monkeypatch.delenv("PF2_BARRIER_POLLS")
    with pytest.raises(g.Pf2Error) as e:
        s.solve(A, torch.zeros_like(b), b)
    assert e.value.status == g.TIMEOUT
    torch.cuda.synchronize()  # the context is still usable
    x = torch.zeros_like(b)
    info = g.LinearSolver(A, kind, pc, tol=1e-8, maxit=1000).solve(A, x, b)
    assert info.converged == 1 and info.status == 0
    ox, _ = O.pcg(rp, col, val, rhs, tol=1e-10, maxit=1000, precond="jacobi")
    assert rel_err(x.cpu().numpy(), ox) < 1e-6


@pytest.mark.parametrize("pc,precision", [("ic", 0), ("ilu", 0), ("ic", 1)])
@pytest.mark.parametrize("dims,halo", [((40, 20, 10), True), ((44, 24, 16), False)])
def test_parts_of_a_tetrahedral_mesh(cuda, monkeypatch, dims, halo, pc, precision):
    """Eight colours: parts of at least 512 rows, by the form with halo rows where it applies and by the
    form with waits otherwise; bit for bit the iterates of the form and the parts asked for."""
    xyz, tet = mg.box_tets(*dims)
    m = g.Mesh3D.from_arrays(xyz, tet)
    A = g.SparseMatrixCSR(m)
    rp, col, _ = A.download()
    n = rp.size - 1
    row = np.repeat(np.arange(n), np.diff(rp))
    val = np.where(row == col, 0.0, -1.0 - 0.3 * np.cos(row + col.astype(np.float64)))
    sums = np.zeros(n)
    np.add.at(sums, row, -val)
    val[row == col] = 1.05 * sums
    A.upload_values(val)
    b = torch.tensor(np.sin(1.0 + np.arange(n)), device="cuda")
    out = []
    for part, parts in ((None, None), ("4" if halo else "3", str(n // 512))):
        if part:
            monkeypatch.setenv("PF2_CG_PART", part)
            monkeypatch.setenv("PF2_CG_PARTS", parts)
        x = torch.zeros_like(b)
        g.LinearSolver(A, "cg", pc, ordering=1, precision=precision, tol=0.0, maxit=6,
                       criterion=g.CRITERION_REL).solve(A, x, b, check=False)
        out.append(x.view(torch.int64))
    assert torch.equal(*out)


@pytest.mark.parametrize("restart", [0, 5])
def test_gmres_on_many_rows_per_block(cuda, monkeypatch, restart):
    """More than 4,096 rows a block (rows taken several at a time, all warps in the dot products): 699,281
    rows, 12 iterations, against classical Gram-Schmidt taken twice on the same Krylov space.  The
    basis is short and the matrix diagonally dominant (condition at most 41): both minimise the same
    residual, so iterates differ by rounding, some 12 x 40 operations x 41 x 1.1e-16 = 2.2e-12; 1e-10."""
    xy, tri = mg.channel(1660, 420, 4.0, 1.0)
    m = g.Mesh2D.from_arrays(xy, tri)
    A = g.SparseMatrixCSR(m)
    rp, col, _ = A.download()
    n = rp.size - 1
    assert n > 4096 * torch.cuda.get_device_properties(0).multi_processor_count
    row = np.repeat(np.arange(n), np.diff(rp))
    val = np.where(row == col, 0.0, -1.0 - 0.3 * np.cos(row + col.astype(np.float64)))
    sums = np.zeros(n)
    np.add.at(sums, row, -val)
    val[row == col] = 1.05 * sums
    A.upload_values(val)
    b = torch.tensor(np.sin(1.0 + np.arange(n)), device="cuda")
    out = []
    for gs in (0, 1):
        x = torch.zeros_like(b)
        info = g.LinearSolver(A, "gmres", "jacobi", tol=1e-4, maxit=200, restart=restart,
                              orthogonalization=gs).solve(A, x, b)
        assert info.converged == 1
        out.append((info.iterations, x.cpu().numpy()))
    assert out[0][0] == out[1][0]
    assert rel_err(*[o[1] for o in out]) < 1e-10
