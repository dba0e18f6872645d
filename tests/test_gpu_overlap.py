"""Launches that overlap their predecessors, and the kernels' rings and extra
blocks at the sizes where their rules change.

Explicit step: the wave sums are extra blocks of the first edge sweep up to
592 Morton blocks (42^3 nodes: 579 blocks; 43^3: 622, their own launch).  Same
tolerance as one evaluation of the residual, a sum of at most ~26 edge terms
per node with 2^-53 each, magnified below 100 times by their cancellation.

Products with H1 from the states: a lane has four steps of
neighbour data in flight; blocks of 64, 128 and 256 nodes give a node four,
two and one lanes, so four to fourteen steps.  FP64 products differ from the
stored blocks' by a few 2^-53 per term, FP32 ones by a few 2^-24: 1e-9 and
1e-5 after eight iterations."""
import numpy as np
import pytest

from aerof_dev_b200 import workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rec", [1, 2])
@pytest.mark.parametrize("n", [42, 43])
def test_rk2_around_the_wave_blocks_rule(gpu_lib, n, rec):
    import torch
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes="channel")
    Ub = W.freestream(0.6)
    ctx = A.Context.from_mesh(m, Ub, reconstruction=rec)
    edge = A.Context.from_mesh(m, Ub, reconstruction=rec, residual_kernel=A.KERNEL_EDGE)
    U = W.perturbed_state(ctx.N, 0.6, amp=0.02)
    out, bad = A.ExplicitRK2(ctx, 0.8).run(U, 4)
    ref, bad_e = A.ExplicitRK2(edge, 0.8).run(U, 4)
    assert bad == bad_e == 0
    assert rel_l2(out - U, ref - U) < 1e-12
    # run after run on one stream, and a residual between them
    Ud = torch.from_numpy(U).cuda()
    for _ in range(3):
        V, _ = A.ExplicitRK2(ctx, 0.8).run(Ud.clone(), 4)
        A.SpaceOperator(ctx).computeResidual(Ud)
        assert np.array_equal(V.cpu().numpy(), out)


@pytest.mark.parametrize("prec,tol", [(64, 1e-9), (32, 1e-5)])
@pytest.mark.parametrize("transpose", [False, True])
@pytest.mark.parametrize("nb", ["64", "128", "256"])
def test_products_over_lanes_per_node(gpu_lib, monkeypatch, nb, transpose, prec, tol):
    A = gpu_lib
    monkeypatch.setenv("AEROF_BLOCK_NODES", nb)
    m = W.make_lattice_mesh(9, jitter=0.2, codes="channel")
    ctx = A.Context.from_mesh(m, W.freestream(0.7))
    U = W.perturbed_state(ctx.N, 0.7, amp=0.05)
    mv, pc = A.MatVecProdH1(ctx, prec), A.JacobiPrec(ctx)
    b = np.random.default_rng(1).standard_normal((ctx.N, 5))
    gm = A.GmresSolver(ctx, 8, 8, 0.0)
    mv.evaluate(U, A.SpaceOperator(ctx).computeTimeStep(U, 30.0))
    blocks = mv.blocks()
    pc.setup()
    free, its, _ = gm.solve(b, transpose=transpose)
    mv.set_blocks(blocks)
    pc.setup()
    stored, its2, _ = gm.solve(b, transpose=transpose)
    assert its == its2 == 8
    assert rel_l2(free, stored) < tol


@pytest.mark.parametrize("stream", ["default", "own"])
def test_host_array_residuals_of_two_meshes_in_turn(gpu_lib, stream):
    # the blocks of the two meshes stage different amounts; each context's
    # kernels keep their own shared-memory limit whichever ran before
    import torch
    A = gpu_lib
    with torch.cuda.stream(torch.cuda.Stream() if stream == "own" else torch.cuda.default_stream()):
        runs = []
        for jitter in (0.2, 0.05, 0.1):
            m = W.make_lattice_mesh(51, jitter=jitter, codes="channel")
            ctx = A.Context.from_mesh(m, W.freestream(0.6))
            U = W.perturbed_state(ctx.N, 0.6, amp=0.02)
            ref = A.SpaceOperator(ctx).computeResidual(torch.from_numpy(U).cuda())[0].cpu()
            runs.append((ctx, torch.from_numpy(U).pin_memory(), ref))
        for k in (0, 1, 2, 0, 2, 1, 0):
            ctx, Uh, ref = runs[k]
            R = torch.empty_like(Uh).pin_memory()
            A.SpaceOperator(ctx).computeResidual(Uh, R)
            assert torch.equal(R, ref)


def test_contexts_of_different_meshes_in_threads(gpu_lib):
    # every thread has a context of its own; the meshes' blocks stage different
    # amounts, and a kernel's shared-memory limit is shared by all of them
    import threading

    import torch
    A = gpu_lib
    calls = {
        "residual": lambda c, U: A.SpaceOperator(c).computeResidual(U)[0],
        "timestep": lambda c, U: A.SpaceOperator(c).computeTimeStep(U, 1.0),
        "rk2": lambda c, U: A.ExplicitRK2(c, 0.5).run(U.clone(), 1)[0],
        "jvp": lambda c, U: A.Sensitivity(c).jvp(U, U),
        "dRdX": lambda c, U: A.Sensitivity(c).dRdX(U, U[:, :3].contiguous()),
        "vjp": lambda c, U: A.Sensitivity(c).vjp(U, U),
        "newton": lambda c, U: A.ImplicitSteadySolver(c, max_steps=1).solve(U.clone())[0],
    }
    cases = []
    for n, jitter in ((9, 0.0), (9, 0.2), (17, 0.05), (7, 0.1)):
        m = W.make_lattice_mesh(n, jitter=jitter, codes="channel")
        ctx = A.Context.from_mesh(m, W.freestream(0.6))
        U = torch.from_numpy(W.perturbed_state(ctx.N, 0.6, amp=0.02)).cuda()
        cases.append((ctx, U, {k: f(ctx, U) for k, f in calls.items()}))
    torch.cuda.synchronize()
    wrong = []

    def work(ctx, U, ref):
        for k, f in calls.items():
            for _ in range(100 if k != "newton" else 20):
                try:
                    same = torch.equal(f(ctx, U), ref[k])
                except A.AerofError as e:
                    same = e
                if same is not True:
                    wrong.append((ctx.N, k, same))
                    return

    threads = [threading.Thread(target=work, args=c) for c in cases]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
