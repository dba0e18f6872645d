"""The blocked kernels of the time step, the fused RK2 stages and the forward
products, and the Spalart-Allmaras residual, at sizes around the 128-node
block (27 nodes: less than one; 125: one, partial; 216: two, the last
partial; 512: four full ones), against the oracle and against the edge
organisation.

Tolerances: one evaluation is a sum of at most ~26 edge terms per node with
2^-53 relative each, magnified by the cancellation of the fluxes (below 100
here): 1e-12; the forward products go through one more difference: 1e-11."""
import numpy as np
import pytest

from aerof_dev_b200 import workloads as W
from conftest import rel_l2

pytestmark = pytest.mark.gpu

SIZES = [(3, "channel"), (5, "farfield"), (6, "channel"), (8, "farfield")]


@pytest.mark.parametrize("rec", [1, 2, 3])
@pytest.mark.parametrize("n,codes", SIZES)
def test_time_step_and_rk2(gpu_lib, oracle_mod, n, codes, rec):
    import torch
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes=codes)
    Ub = W.freestream(0.6)
    o = oracle_mod.Oracle(m)
    U = W.perturbed_state(o.N, 0.6, amp=0.02)
    ctx = A.Context.from_mesh(m, Ub, reconstruction=rec)
    edge = A.Context.from_mesh(m, Ub, reconstruction=rec, residual_kernel=A.KERNEL_EDGE)
    assert rel_l2(A.SpaceOperator(ctx).computeTimeStep(U, 0.8), o.timestep(U, 0.8)) < 1e-14
    assert rel_l2(A.SpaceOperator(edge).computeTimeStep(U, 0.8), o.timestep(U, 0.8)) < 1e-14
    ref = o.rk2(U, Ub, rec, 0.8, 3)
    out, bad = A.ExplicitRK2(ctx, 0.8).run(U, 3)
    dev, bad_d = A.ExplicitRK2(ctx, 0.8).run(torch.from_numpy(U).cuda(), 3)
    assert bad == bad_d == 0
    assert rel_l2(out - U, ref - U) < 1e-12 and np.array_equal(dev.cpu().numpy(), out)
    assert rel_l2(out, A.ExplicitRK2(edge, 0.8).run(U, 3)[0]) < 1e-13
    # a run leaves no state behind that a residual of another state would see
    R = A.SpaceOperator(ctx).computeResidual(U)[0]
    assert np.array_equal(R, A.SpaceOperator(A.Context.from_mesh(m, Ub, reconstruction=rec)).computeResidual(U)[0])
    # no steps: the state comes back as it was
    assert np.array_equal(A.ExplicitRK2(ctx, 0.8).run(U, 0)[0], U)


@pytest.mark.parametrize("rec", [1, 2, 3])
@pytest.mark.parametrize("n,codes", SIZES)
def test_forward_products(gpu_lib, oracle_mod, n, codes, rec):
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes=codes)
    Ub = W.freestream(0.6)
    o = oracle_mod.Oracle(m)
    U = W.perturbed_state(o.N, 0.6, amp=0.02)
    rng = np.random.default_rng(n)
    v, xd = rng.standard_normal((o.N, 5)), rng.standard_normal((o.N, 3)) * 0.1 / (n - 1)
    S = A.Sensitivity(A.Context.from_mesh(m, Ub, reconstruction=rec))
    assert rel_l2(S.jvp(U, v), o.jvp(U, Ub, v, rec)) < 1e-11
    assert rel_l2(S.dRdX(U, xd), o.dRdX(U, Ub, xd, rec)[0]) < 1e-11
    # one after the other on one context, in either order
    assert np.array_equal(S.jvp(U, v), S.jvp(U, v))
    # transposes of one another
    w = rng.standard_normal((o.N, 5))
    a, b = float(np.sum(w * S.dRdX(U, xd))), float(np.sum(S.dRdX_T(U, w) * xd))
    assert abs(a - b) <= 1e-10 * np.linalg.norm(w) * np.linalg.norm(S.dRdX(U, xd))


@pytest.mark.parametrize("rec,model", [(1, 0), (2, 1), (2, 2), (3, 2)])
@pytest.mark.parametrize("n,codes", SIZES)
def test_spalart_allmaras(gpu_lib, oracle_mod, n, codes, rec, model):
    import torch
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes=codes)
    Ub6 = np.concatenate([W.freestream(0.6), [1e-3]])
    d2wall = np.abs(m["X"][:, 2]) + 0.02 * m["X"][:, 0]
    o = oracle_mod.Oracle(m)
    U5 = W.perturbed_state(o.N, 0.6, amp=0.02)
    nu = 1e-3 * (1.0 + 3.0 * np.random.default_rng(n).random(o.N))
    U = np.column_stack([U5, U5[:, 0] * nu])
    visc = dict(model=model, reynolds_mu=1500.0, prandtl=0.72, bulk_viscosity=0.1, sutherland_alpha=1.3,
                sutherland_Ts=0.35)
    out = []
    for kernel in (A.KERNEL_BLOCKED, A.KERNEL_EDGE):
        ctx = A.Context.from_mesh(m, Ub6[:5], reconstruction=rec, residual_kernel=kernel)
        ctx.set_viscosity(**visc)
        ctx.set_turbulence(d2wall, Ub6)
        R, bad = A.SpaceOperator(ctx).computeResidualSA(torch.from_numpy(U).cuda())
        assert bad == 0
        out.append(R.cpu().numpy())
    ref, _ = o.residual_sa(U, Ub6, d2wall, order=rec, model=model, reynolds=1500.0, prandtl=0.72, bulk=0.1,
                           alpha=1.3, Ts=0.35)
    for R in out:
        assert rel_l2(R, ref) < 1e-12 and rel_l2(R[:, 5], ref[:, 5]) < 1e-12


@pytest.mark.parametrize("rec", [1, 2])
@pytest.mark.parametrize("n,squash,nodes", [(29, 0.03, 128), (31, 0.04, 128), (33, 0.02, 128), (8, 1.0, 256)])
def test_reverse_sweep_with_fewer_threads(gpu_lib, monkeypatch, n, squash, nodes, rec):
    # stretched cells (or blocks of 256 nodes) stage so many nodes that the
    # reverse sweep's chunk of 512 edges does not fit beside them: it runs
    # blocked all the same, in chunks of 256.  Against blocks of 64 nodes,
    # where 512 fit: the same sums of ~26 terms in another order
    A = gpu_lib
    m = W.make_lattice_mesh(n, jitter=0.2, codes="channel")
    m["X"] = m["X"] * np.array([1.0, 1.0, squash])
    rng = np.random.default_rng(n)
    N = m["X"].shape[0]
    U, lam = W.perturbed_state(N, 0.6), rng.standard_normal((N, 5))
    out = []
    for nb in (nodes, 64):
        monkeypatch.setenv("AEROF_BLOCK_NODES", str(nb))
        S = A.Sensitivity(A.Context.from_mesh(m, W.freestream(0.6), reconstruction=rec))
        A.launch_count()
        w = S.vjp(U, lam)
        launches = A.launch_count()
        out.append((w, *S.adjoint_products(U, lam), launches))
    (w, jt, gx, k), (w64, jt64, gx64, k64) = out
    assert k == k64   # the same organisation
    assert rel_l2(w, w64) < 1e-12 and rel_l2(jt, jt64) < 1e-12 and rel_l2(gx, gx64) < 1e-11
    S = A.Sensitivity(A.Context.from_mesh(m, W.freestream(0.6), reconstruction=rec))
    v = rng.standard_normal((N, 5))
    Jv = S.jvp(U, v)
    assert abs((lam * Jv).sum() - (w * v).sum()) < 1e-12 * np.linalg.norm(lam) * np.linalg.norm(Jv)


@pytest.mark.parametrize("what", ["no pressure", "negative pressure", "infinite density", "infinite energy"])
def test_time_step_at_degenerate_states(gpu_lib, what):
    # the blocked sums take the reciprocals' special values as the divisions
    # and roots of the edge organisation do
    A = gpu_lib
    m = W.make_lattice_mesh(6, jitter=0.2, codes="channel")
    Ub = W.freestream(0.6)
    ctx = A.Context.from_mesh(m, Ub)
    edge = A.Context.from_mesh(m, Ub, residual_kernel=A.KERNEL_EDGE)
    U = W.perturbed_state(ctx.N, 0.6, amp=0.02)
    for i in (86, 87, 122):   # two neighbours, and one alone
        if what == "no pressure":
            U[i] = [1.0, 0.0, 0.0, 0.0, 0.0]
        elif what == "negative pressure":
            U[i, 4] = -3.0
        elif what == "infinite density":
            U[i, 0] = np.inf
        else:
            U[i, 4] = np.inf
    a = A.SpaceOperator(ctx).computeTimeStep(U, 0.8)
    b = A.SpaceOperator(edge).computeTimeStep(U, 0.8)
    ok = np.isfinite(b)
    assert np.array_equal(np.isfinite(a), ok) and ok.sum() > 100
    assert rel_l2(a[ok], b[ok]) < 1e-13
    assert np.array_equal(np.isnan(a), np.isnan(b))
