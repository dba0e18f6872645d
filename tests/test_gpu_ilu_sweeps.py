"""Block ILU(0) colour sweeps with several vectors per pass against one vector
at a time: batch sizes around the four vectors of a pass, colours of fewer
rows than a thread block and rows with none, up to and more than the eight
entries that a row's lanes take at once.

The batch and the single systems run the same flexible GMRES to 1e-10; their
solutions differ by that residual through the inverse of the operator, whose
condition is below 1e3 on these meshes: 1e-7."""
import numpy as np
import pytest

from aerof_dev_b200 import workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("n,R", [(2, 3), (3, 4), (5, 2), (6, 6)])
def test_vectors_of_a_batch_match_single_ones(gpu_lib, n, R, transpose):
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.5))
    ctx.set_preconditioner(A.PC_ILU0)
    U = W.smooth_state(m["X"], 0.5)
    S = A.Sensitivity(ctx)
    B = np.random.default_rng(n).standard_normal((R, ctx.N, 5))
    kw = dict(transpose=transpose, krylov=20, maxits=200, eps=1e-10, inner_its=5)
    X, its, res = S.solve_batch(U, B, **kw)
    for k in range(R):
        assert res[k] <= 1e-10 * np.linalg.norm(B[k])
        x1, i1, _ = S.solve_batch(U, B[k:k + 1], **kw)
        assert abs(int(its[k]) - int(i1[0])) <= 1
        assert rel_l2(X[k], x1[0]) < 1e-7


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("n", [2, 3, 4])
def test_small_colours_match_the_oracle(gpu_lib, oracle_mod, n, prec):
    # (larger meshes: test_gpu_ilu.py, with its tolerances)
    m = W.make_lattice_mesh(n, jitter=0.1, codes="farfield")
    o = oracle_mod.Oracle(m)
    U = W.perturbed_state(o.N, 0.8)
    ctx = gpu_lib.Context.from_mesh(m, W.freestream(0.8))
    ctx.set_preconditioner(gpu_lib.PC_ILU0)
    mv = gpu_lib.MatVecProdH1(ctx, prec)
    mv.evaluate(U, o.timestep(U, 10.0))
    pc = gpu_lib.JacobiPrec(ctx)
    pc.setup()
    x = np.random.default_rng(n).standard_normal((o.N, 5))
    for trans in (False, True):
        z = pc.apply(x, transpose=trans)
        zr, bad, _, _ = o.ilu0(mv.blocks(), x, fp32=(prec == 32), transpose=trans)
        assert bad == 0
        assert rel_l2(z, zr) < (1e-12 if prec == 64 else 1e-5)
