"""Device-driven GMRES and flexible GMRES: restart lengths around the eight
basis vectors that one pass of the Gram-Schmidt sweep takes, more vectors
than the triangular solve keeps in shared memory, restarts, a zero right-hand
side, and systems that converge at different times in one batch.

Tolerances: in FP64 the two orthogonalisations (the oracle's and the two
sweeps) compute the same Krylov minimiser; its relative change is bounded by
2^-53 times the squared condition of the basis recurrence, far below the
1e-9 asked for at these sizes and iteration counts."""
import numpy as np
import pytest

from aerof_dev_b200 import workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _operator(A, o, m, U, dt, prec):
    ctx = A.Context.from_mesh(m, W.freestream(0.8))
    mv = A.MatVecProdH1(ctx, prec)
    mv.evaluate(U, dt)
    A.JacobiPrec(ctx).setup()
    return ctx, mv


@pytest.mark.parametrize("n,krylov,maxits", [(4, 1, 3), (4, 7, 7), (6, 8, 20), (6, 9, 9), (6, 17, 40), (5, 70, 75),
                                             (3, 100, 100)])
def test_gmres_restart_lengths(gpu_lib, oracle_mod, n, krylov, maxits):
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes="channel")
    Ub = W.freestream(0.8)
    o = oracle_mod.Oracle(m)
    U = W.perturbed_state(o.N, 0.8)
    dt = o.timestep(U, 20.0)
    ctx, mv = _operator(A, o, m, U, dt, 64)
    blocks = mv.blocks()
    b = np.random.default_rng(n).standard_normal((o.N, 5))
    x, its, res = A.GmresSolver(ctx, krylov, maxits, 1e-11).solve(b)
    # the true residual equals the method's estimate, within the same
    # relative accuracy of b
    r = b - o.matvec(blocks, x)
    assert its <= maxits
    assert abs(np.linalg.norm(r) - res) <= 1e-9 * np.linalg.norm(b)
    assert its == maxits or res <= 1e-11 * np.linalg.norm(b)
    # a zero right-hand side is answered by zero, without iterations
    x0, it0, r0 = A.GmresSolver(ctx, krylov, maxits, 1e-11).solve(np.zeros_like(b))
    assert it0 == 0 and r0 == 0.0 and not x0.any()


@pytest.mark.parametrize("pc", [0, 1])
@pytest.mark.parametrize("transpose", [False, True])
def test_batch_equals_one_by_one(gpu_lib, pc, transpose):
    # five systems of very different right-hand sides (one of them zero, one
    # nearly an eigen-direction's multiple), each as its own solve
    A = gpu_lib
    m = W.make_lattice_mesh(7, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.5))
    ctx.set_preconditioner(pc)
    U = W.smooth_state(m["X"], 0.5)
    S = A.Sensitivity(ctx)
    rng = np.random.default_rng(1)
    B = rng.standard_normal((5, ctx.N, 5))
    B[1] = 0.0
    B[2] *= 1e-6
    B[3] = S.jvp(U, np.ones((ctx.N, 5)))
    X, its, res = S.solve_batch(U, B, transpose=transpose, krylov=11, maxits=200, eps=1e-9, inner_its=6)
    assert its[1] == 0 and not X[1].any()
    for k in range(5):
        if k == 1:
            continue
        assert res[k] <= 1e-9 * np.linalg.norm(B[k])
        J = S.vjp if transpose else S.jvp
        assert np.linalg.norm(J(U, X[k]) - B[k]) <= 1e-8 * np.linalg.norm(B[k])
        S.set_exact_operator(True)
        x1, i1, _ = S.solve(U, B[k], transpose=transpose, krylov=11, maxits=200, eps=1e-9, inner_its=6)
        S.set_exact_operator(False)
        # both satisfy the system to 1e-9; their difference is that residual
        # through J^-1 (condition below 1e3 here)
        assert rel_l2(X[k], x1) <= 1e-6
        assert abs(int(its[k]) - i1) <= 1


@pytest.mark.parametrize("pc", [0, 1])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("e", [-332, 332])
def test_flexible_solves_scale_with_the_right_hand_side(gpu_lib, pc, transpose, e):
    # 2^332 is about 1e100, far outside the range of the FP32 inner solves.  A
    # power of two changes no rounding of the FP64 outer method (sums of
    # squares stay below 2^1023 and above 2^-1022), so the solutions are each
    # other's multiples to the last bits
    A = gpu_lib
    m = W.make_lattice_mesh(6, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.5))
    ctx.set_preconditioner(pc)
    U = W.smooth_state(m["X"], 0.5)
    S = A.Sensitivity(ctx)
    s = 2.0 ** e
    B = np.random.default_rng(7).standard_normal((3, ctx.N, 5))
    opt = dict(transpose=transpose, krylov=7, maxits=24, eps=1e-9, inner_its=6)
    X, its, res = S.solve_batch(U, B, **opt)
    assert its.max() > 7 and (res < 0.1 * np.sqrt(B[0].size)).all()   # restarted, and below |B_k|
    Xs, its_s, res_s = S.solve_batch(U, s * B, **opt)
    assert np.array_equal(its, its_s)
    assert rel_l2(Xs / s, X) <= 1e-14 and rel_l2(res_s / s, res) <= 1e-14
    # one flexible solve, and systems of different scale in one batch
    x1, i1, _ = S.solve(U, B[0], **opt)
    xs, i2, _ = S.solve(U, s * B[0], **opt)
    assert i1 == i2 and rel_l2(xs / s, x1) <= 1e-14
    mixed = S.solve_batch(U, B * np.array([1.0, s, 1.0])[:, None, None], **opt)[0]
    assert rel_l2(mixed[1] / s, X[1]) <= 1e-14 and np.array_equal(mixed[0], X[0]) and np.array_equal(mixed[2], X[2])


@pytest.mark.parametrize("krylov", [100, 513, 6200, 7199, 7200, 9000])
def test_long_restarts(gpu_lib, krylov):
    # more vectors than are staged at a time (512), than 48 KB of shared memory
    # hold (6144) and than 200 KB do (7199), on a system of 135 unknowns that
    # needs far fewer: the same solution whatever the longest cycle
    A = gpu_lib
    m = W.make_lattice_mesh(3, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.5))
    U = W.smooth_state(m["X"], 0.5)
    S = A.Sensitivity(ctx)
    B = np.random.default_rng(3).standard_normal((2, ctx.N, 5))
    X, its, res = S.solve_batch(U, B, krylov=krylov, maxits=krylov, eps=1e-9, inner_its=5)
    for k in range(2):
        assert its[k] < 136 and res[k] <= 1e-9 * np.linalg.norm(B[k])
        assert np.linalg.norm(S.jvp(U, X[k]) - B[k]) <= 1e-8 * np.linalg.norm(B[k])
    # the same cycle length throughout when the iterations bound it
    Y = S.solve_batch(U, B, krylov=krylov, maxits=60, eps=0.0, inner_its=5)[0]
    assert np.array_equal(Y, S.solve_batch(U, B, krylov=60, maxits=60, eps=0.0, inner_its=5)[0])
    mv = A.MatVecProdH1(ctx, 64)
    mv.evaluate(U, A.SpaceOperator(ctx).computeTimeStep(U, 50.0))
    A.JacobiPrec(ctx).setup()
    x, i, r = A.GmresSolver(ctx, krylov, krylov, 1e-9).solve(B[0])
    assert i < 136 and r <= 1e-9 * np.linalg.norm(B[0])
    assert np.linalg.norm(mv.apply(x) - B[0]) <= 1e-8 * np.linalg.norm(B[0])


def test_right_hand_side_beyond_the_range_is_not_reported_as_solved(gpu_lib):
    # the squared norm of 1e200 overflows FP64: the FP32 solver's residual is
    # not a number, and no small one
    A = gpu_lib
    m = W.make_lattice_mesh(4, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.5))
    U = W.smooth_state(m["X"], 0.5)
    A.MatVecProdH1(ctx, 32).evaluate(U, A.SpaceOperator(ctx).computeTimeStep(U, 10.0))
    A.JacobiPrec(ctx).setup()
    b = np.random.default_rng(0).standard_normal((ctx.N, 5))
    x, its, res = A.GmresSolver(ctx, 5, 10, 1e-6).solve(1e200 * b)
    assert np.isnan(res) and not np.isfinite(x).all()
    # far smaller ones are solved at any scale that FP32 can hold the answer of
    for s in (1e-25, 1.0, 1e25):
        xs, i, r = A.GmresSolver(ctx, 30, 30, 1e-4).solve(s * b)
        assert r <= 1e-4 * s * np.linalg.norm(b) and np.isfinite(xs).all()
