"""aerof_gpu_gradients with device and host outputs, in the blocked and the
edge organisation, at sizes around the gradient kernel's block of 128 nodes
(one partial block, a remainder, several blocks), against the oracle; and the
unphysical count that the residual's node assembly hands to the host.

Tolerance: each gradient component is a sum of at most ~26 products of
values of one size (2^-53 relative each, in another order than the
oracle's), so relative L2 stays below 26 * 2^-53 ~ 3e-15 times the
cancellation of the sum (below 100 here): 1e-12 with room to spare."""
import ctypes

import numpy as np
import pytest

from aerof_dev_b200 import workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kernel", [0, 1])
@pytest.mark.parametrize("n", [3, 5, 8, 13])
def test_gradients_device_and_host_outputs(gpu_lib, oracle_mod, n, kernel):
    import torch
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes="channel")
    o = oracle_mod.Oracle(m)
    V = o.prim(W.perturbed_state(o.N, 0.8))
    ref = o.gradients(V)
    ctx = A.Context.from_mesh(m, W.freestream(0.8), residual_kernel=kernel)
    sp = A.SpaceOperator(ctx)
    dev = sp.computeGradients(torch.from_numpy(V).cuda())
    host = sp.computeGradients(V)
    for d, h, r in zip(dev, host, ref):
        assert np.array_equal(d.cpu().numpy(), h)
        assert rel_l2(h, r) < 1e-12
    # a residual after the call sees its own state's gradients, not these
    U = torch.from_numpy(W.perturbed_state(o.N, 0.8, seed=7)).cuda()
    R, _ = sp.computeResidual(U)
    sp.computeGradients(torch.from_numpy(V).cuda())
    lam = torch.ones_like(U)
    first = A.Sensitivity(ctx).adjoint_products(U, lam)
    fresh = A.Context.from_mesh(m, W.freestream(0.8), residual_kernel=kernel)
    again = A.Sensitivity(fresh).adjoint_products(U, lam)
    assert all(torch.equal(a, b) for a, b in zip(first, again))


def test_unphysical_counts_of_successive_calls(gpu_lib, oracle_mod):
    # unlimited reconstruction next to a pressure spike: a positive count,
    # the same one twice, none for a good state in between, and the sum over
    # the residuals of an RK2 step whose first stage sees the bad state
    import torch
    A = gpu_lib
    m = W.make_lattice_mesh(7, jitter=0.2, codes="channel")
    o = oracle_mod.Oracle(m)
    Ub = W.freestream(0.8)
    good = W.perturbed_state(o.N, 0.8)
    V = o.prim(good)
    i = 3 * 49 + 3 * 7 + 3
    V[i, 4] *= 40.0
    V[i + 1, 4] *= 0.02
    bad = W.prim_to_cons(V)
    expect = o.residual(bad, Ub, 3)[1]
    assert expect > 0
    sp = A.SpaceOperator(A.Context.from_mesh(m, Ub, reconstruction=3))
    g, b = torch.from_numpy(good).cuda(), torch.from_numpy(bad).cuda()
    assert [sp.computeResidual(x)[1] for x in (b, g, b, b, g)] == [expect, 0, expect, expect, 0]
    sp.computeResidualAsync(b, torch.empty_like(b))
    assert sp.computeResidual(g)[1] == 0
    assert sp.computeResidual(bad)[1] == expect
    assert A.ExplicitRK2(sp.ctx, 1e-9).run(b, 1)[1] >= expect


@pytest.mark.parametrize("first", ["residual", "rk2", "jvp", "newton"])
def test_async_count_after_other_calls(gpu_lib, oracle_mod, first):
    # the status count starts at zero whichever call allocated the counters,
    # also where the allocator hands out memory that was written before
    import torch
    A = gpu_lib
    m = W.make_lattice_mesh(5, jitter=0.2, codes="channel")
    o = oracle_mod.Oracle(m)
    Ub = W.freestream(0.8)
    good = W.perturbed_state(o.N, 0.8)
    V = o.prim(good)
    V[62, 4] *= 40.0
    V[63, 4] *= 0.02
    bad = W.prim_to_cons(V)
    expect = o.residual(bad, Ub, 3)[1]
    assert expect > 0
    g, b = torch.from_numpy(good).cuda(), torch.from_numpy(bad).cuda()
    rt = ctypes.CDLL("libcudart.so.12")
    ptrs = [ctypes.c_void_p() for _ in range(4096)]
    for p in ptrs:
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(32)) == 0
        assert rt.cudaMemset(p, 0x01, ctypes.c_size_t(32)) == 0
    for p in ptrs:
        assert rt.cudaFree(p) == 0
    ctx = A.Context.from_mesh(m, Ub, reconstruction=3)
    sp = A.SpaceOperator(ctx)
    if first == "residual":
        sp.computeResidual(g)
    elif first == "rk2":
        A.ExplicitRK2(ctx, 0.5).run(g.clone(), 1)
    elif first == "jvp":
        A.Sensitivity(ctx).jvp(g, g)
    else:
        A.ImplicitSteadySolver(ctx, max_steps=1).solve(g.clone())
    sp.computeResidualAsync(b, torch.empty_like(b))
    sp.computeResidualAsync(b, torch.empty_like(b))
    assert ctx.status() == 2 * expect
    assert ctx.status() == 0
