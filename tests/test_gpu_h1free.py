"""Products with H1 formed from the states inside the Krylov solvers against
the stored blocks, and operators of which only the diagonal was assembled.

The mesh sizes put the node count just below, at and above multiples of the
128-node block (27 to 1331 nodes), with one block, partial last blocks and
odd neighbour counts.  Both routes run the same GMRES iterations on the same
preconditioner; in FP64 the products differ by a few 2^-53 per term, so the
iterates agree far below 1e-9; in FP32 by a few 2^-24 through up to eight
iterations: 1e-5."""
import numpy as np
import pytest

from aerof_dev_b200 import workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(64, 1e-9), (32, 1e-5)])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("n,codes,with_dt", [(3, "channel", True), (5, "farfield", True), (6, "channel", False),
                                             (8, "channel", True), (11, "farfield", True)])
def test_products_match_the_stored_blocks(gpu_lib, prec, tol, transpose, n, codes, with_dt):
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes=codes)
    ctx = A.Context.from_mesh(m, W.freestream(0.7))
    U = W.perturbed_state(ctx.N, 0.7, amp=0.05)
    dt = A.SpaceOperator(ctx).computeTimeStep(U, 30.0) if with_dt else None
    mv, pc = A.MatVecProdH1(ctx, prec), A.JacobiPrec(ctx)
    b = np.random.default_rng(n).standard_normal((ctx.N, 5))
    gm = A.GmresSolver(ctx, 8, 8, 0.0)
    mv.evaluate(U, dt)
    blocks = mv.blocks()
    pc.setup()
    free, its, res = gm.solve(b, transpose=transpose)
    mv.set_blocks(blocks)   # an operator given by the caller is read as stored
    pc.setup()
    stored, its2, res2 = gm.solve(b, transpose=transpose)
    assert its == its2 == 8
    assert rel_l2(free, stored) < tol
    assert abs(res - res2) <= tol * np.linalg.norm(b)


@pytest.mark.parametrize("prec", [64, 32])
def test_newton_operator_is_complete_afterwards(gpu_lib, prec):
    # Newton assembles the diagonal blocks only; the operator it leaves
    # behind reads as the one evaluated at its last linearisation point
    A = gpu_lib
    m = W.make_lattice_mesh(7, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.8))
    U = W.perturbed_state(ctx.N, 0.8)
    dt = A.SpaceOperator(ctx).computeTimeStep(U, 10.0)
    A.ImplicitSteadySolver(ctx, precision=prec, max_steps=1).solve(U)
    left = A.MatVecProdH1(ctx, prec)
    p = np.random.default_rng(0).standard_normal((ctx.N, 5))
    y = left.apply(p)
    yt = left.applyTranspose(p)
    fresh = A.MatVecProdH1(A.Context.from_mesh(m, W.freestream(0.8)), prec)
    fresh.evaluate(U, dt)
    assert np.array_equal(left.blocks(), fresh.blocks())
    assert np.array_equal(y, fresh.apply(p)) and np.array_equal(yt, fresh.applyTranspose(p))
    # its preconditioner stays usable, and an ILU(0) can be set up from it
    z = A.JacobiPrec(ctx).apply(p)
    A.JacobiPrec(fresh.ctx).setup()
    assert rel_l2(z, A.JacobiPrec(fresh.ctx).apply(p)) < (1e-12 if prec == 64 else 1e-5)
    ctx.set_preconditioner(A.PC_ILU0)
    A.JacobiPrec(ctx).setup()
    assert A.GmresSolver(ctx, 30, 30, 1e-8).solve(p)[2] <= 1e-6 * np.linalg.norm(p)


@pytest.mark.parametrize("transpose", [False, True])
def test_linearized_solve_leaves_its_operator(gpu_lib, transpose):
    A = gpu_lib
    m = W.make_lattice_mesh(6, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.5))
    U = W.smooth_state(m["X"], 0.5)
    b = np.random.default_rng(2).standard_normal((ctx.N, 5))
    A.Sensitivity(ctx).solve(U, b, transpose=transpose, maxits=20, inner_its=5)
    fresh = A.MatVecProdH1(A.Context.from_mesh(m, W.freestream(0.5)), 32)
    fresh.evaluate(U)
    assert rel_l2(A.MatVecProdH1(ctx, 32).blocks(), fresh.blocks()) < 1e-6


@pytest.mark.parametrize("prec,tol", [(64, 1e-9), (32, 1e-4)])
@pytest.mark.parametrize("nb", ["64", "128", "256"])
def test_node_without_pressure(gpu_lib, monkeypatch, nb, prec, tol):
    # the lanes of a node take its neighbours in whole steps; what fills the
    # last step up must not contribute, also where the node's own speed of
    # sound is zero (its averages with its neighbours are regular)
    A = gpu_lib
    monkeypatch.setenv("AEROF_BLOCK_NODES", nb)
    m = W.make_lattice_mesh(6, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.6), reconstruction=1)
    U = W.perturbed_state(ctx.N, 0.6, amp=0.02)
    for i in (86, 93, 122):   # inner nodes, no neighbours of each other
        U[i, 4] = 0.5 * (U[i, 1:4] ** 2).sum() / U[i, 0]
    sp = A.SpaceOperator(ctx)
    dt = sp.computeTimeStep(U, 10.0)
    b = np.random.default_rng(0).standard_normal((ctx.N, 5))
    mv, pc = A.MatVecProdH1(ctx, prec), A.JacobiPrec(ctx)
    for transpose in (False, True):
        mv.evaluate(U, dt)
        blocks = mv.blocks()
        assert np.isfinite(blocks).all()
        pc.setup()
        free, its, _ = A.GmresSolver(ctx, 8, 8, 0.0).solve(b, transpose=transpose)
        mv.set_blocks(blocks)
        pc.setup()
        stored, its2, _ = A.GmresSolver(ctx, 8, 8, 0.0).solve(b, transpose=transpose)
        assert its == its2 == 8
        assert np.isfinite(free).all() and rel_l2(free, stored) < tol


def _state(N, mach, seed=5):
    rng = np.random.default_rng(seed)
    n = lambda a: a * (1.0 + 0.02 * rng.standard_normal(N))  # noqa: E731
    s = 0.02 * rng.standard_normal((N, 2))
    return W.prim_to_cons(np.column_stack([n(1.0), n(1.0) if mach else np.zeros(N), s * bool(mach),
                                           n(1.0 / (1.4 * (mach or 1.0) ** 2))]))


@pytest.mark.parametrize("mach", [0, 3, 20, 200])
@pytest.mark.parametrize("inner", [0, 5])
def test_diagonal_alone_and_whole_rows_invert_the_same_blocks(gpu_lib, mach, inner):
    # without time steps |A|'s first diagonal entry cancels on supersonic
    # edges; whether the sum over a node is round-off or exactly zero must not
    # decide whether its block is inverted.  At rest it is zero in any
    # arithmetic, and the blocks stay as they are, as in the reference
    A = gpu_lib
    m = W.make_lattice_mesh(9, jitter=0.2, codes="channel")
    Ub = _state(1, mach)[0] if mach else W.freestream(0.5)
    ctx = A.Context.from_mesh(m, Ub, reconstruction=2)
    U = _state(ctx.N, mach)
    S, pc = A.Sensitivity(ctx), A.JacobiPrec(ctx)
    b = A.SpaceOperator(ctx).computeResidual(U)[0]
    x, its, res = S.solve(U, b, krylov=15, maxits=15, eps=1e-9, inner_its=inner)
    lazy = pc.apply(b)
    mv = A.MatVecProdH1(ctx, 32 if inner else 64)
    mv.evaluate(U)
    pc.setup()
    rows = pc.apply(b)
    # blocks of condition below 1e3 here; FP32 ones are formed in FP32
    assert rel_l2(lazy, rows) < (1e-4 if inner else 1e-11)
    if mach and inner:
        # inner solves that invert the blocks cut the residual by far more
        # than the factor 4 that was left where they do not
        assert res <= 1e-2 * np.linalg.norm(b)
