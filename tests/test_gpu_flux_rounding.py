"""Rounding of the flux arithmetic (refined reciprocals in place of divisions
and roots) against 80-bit references, item by item on random states.

The bounds are on the root mean square over 200,000 items of the error
relative to the item's result.  Every operation contributes at most half a
unit in the last place (2^-53 = 1.1e-16 relative, 0.29 of that on average),
and the same expressions with correctly rounded divisions and roots are the
yardstick: the refined forms may be 2 % above it, five times the scatter of
such a mean between samples."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
L, CL = np.longdouble, np.clongdouble
G = L(1.4)
N = 200000


@pytest.fixture(scope="module")
def probe(gpu_lib, tmp_path_factory):
    so = str(tmp_path_factory.mktemp("probe") / "libflux_probe.so")
    nvcc = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")
    subprocess.check_call([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                           "--expt-relaxed-constexpr", "-Xcompiler", "-fPIC", "-shared",
                           os.path.join(HERE, "probes", "flux_probe.cu"), "-o", so])
    lib = C.CDLL(so)
    lib.flux_probe.argtypes = [C.c_int, C.c_int, C.c_void_p, C.c_void_p]
    lib.flux_probe.restype = C.c_int

    def run(what, x, width):
        x = np.ascontiguousarray(x, dtype=np.float64)
        out = np.empty((x.shape[0], width))
        assert lib.flux_probe(what, x.shape[0], x.ctypes.data, out.ctypes.data) == 0
        return out
    return run


def rms_error(a, ref):
    """Root mean square over the items of |a - ref| / |ref|."""
    e = np.sqrt(((a - ref) ** 2).sum(1) / (ref ** 2).sum(1))
    return float(np.sqrt((e * e).mean()))


def states(rng, n):
    return np.column_stack([rng.uniform(0.2, 3.0, n), rng.uniform(-1.5, 1.5, (n, 3)), rng.uniform(0.2, 3.0, n)])


def normals(rng, n):
    return rng.standard_normal((n, 3)) * 10.0 ** rng.uniform(-5, 0, (n, 1))


def cons(V):
    E = V[:, 4] / (G - 1) + V[:, 0] * (V[:, 1:4] ** 2).sum(1) / 2
    return np.concatenate([V[:, :1], V[:, :1] * V[:, 1:4], E[:, None]], 1)


def apply(f1, fp, fm, n, u, H, c, q):
    """f(A) q for the eigenvalue functions f1, f+, f- along the unit n."""
    un = (u * n).sum(1)
    a = (n * q[:, 1:4]).sum(1) - un * q[:, 0]
    b = (G - 1) * ((u * u).sum(1) * q[:, 0] / 2 - (u * q[:, 1:4]).sum(1) + q[:, 4])
    s1, s2 = (fp + fm) / 2 - f1, (fp - fm) / 2
    k1, k2 = s1 * b / (c * c) + s2 * a / c, s1 * a + s2 * b / c
    one, zero = np.ones_like(un)[:, None], np.zeros_like(un)[:, None]
    r1, r2 = np.concatenate([one, u, H[:, None]], 1), np.concatenate([zero, n, un[:, None]], 1)
    return f1[:, None] * q + k1[:, None] * r1 + k2[:, None] * r2


def pos(x):
    return np.where(x.real > 0, x, 0 * x)


def neg(x):
    return np.where(x.real < 0, x, 0 * x)


def test_far_field_flux(probe):
    rng = np.random.default_rng(1)
    V, n = states(rng, N), normals(rng, N)
    Ub = cons(states(rng, N).astype(L)).astype(np.float64)
    out = probe(0, np.column_stack([V, n, Ub]), 10)
    V, n, Ub = V.astype(L), n.astype(L), Ub.astype(L)
    S = np.sqrt((n * n).sum(1))
    e, u, U = n / S[:, None], V[:, 1:4], cons(V)
    c, H, un = np.sqrt(G * V[:, 4] / V[:, 0]), (U[:, 4] + V[:, 4]) / V[:, 0], (u * e).sum(1)
    lam = (un, un + c, un - c)
    ref = (apply(*map(pos, lam), e, u, H, c, U) + apply(*map(neg, lam), e, u, H, c, Ub)) * S[:, None]
    refined, divided = rms_error(out[:, :5], ref), rms_error(out[:, 5:], ref)
    print(f"far-field flux: refined {refined:.4g}, divisions and roots {divided:.4g}")
    assert divided < 1e-15
    assert refined <= 1.02 * divided


def roe(n, Vi, Vj):
    """The physical flux of the upwind side and the acoustic wave against it."""
    S = np.sqrt((n * n).sum(1))
    e = n / S[:, None]
    wi, wj = np.sqrt(Vi[:, 0]), np.sqrt(Vj[:, 0])
    u = (wi[:, None] * Vi[:, 1:4] + wj[:, None] * Vj[:, 1:4]) / (wi + wj)[:, None]
    Hi, Hj = ((cons(V)[:, 4] + V[:, 4]) / V[:, 0] for V in (Vi, Vj))
    H = (wi * Hi + wj * Hj) / (wi + wj)
    c = np.sqrt((G - 1) * (H - (u * u).sum(1) / 2))
    un = (u * e).sum(1)
    left = un.real > 0
    Vs = np.where(left[:, None], Vi, Vj)
    Us = cons(Vs)
    m = Vs[:, 0] * (Vs[:, 1:4] * e).sum(1)
    f = np.concatenate([m[:, None], m[:, None] * Vs[:, 1:4] + Vs[:, 4:5] * e,
                        (m / Vs[:, 0] * (Us[:, 4] + Vs[:, 4]))[:, None]], 1)
    z, lam = 0 * un, np.where(left, neg(un - c), pos(un + c))
    add = apply(z, np.where(left, z, lam), np.where(left, lam, z), e, u, H, c, cons(Vj) - cons(Vi))
    return (f + np.where(left[:, None], add, -add)) * S[:, None]


def test_adjoint_of_the_roe_flux(probe):
    rng = np.random.default_rng(2)
    Vi = states(rng, N)
    Vj = Vi * (1.0 + 0.2 * rng.uniform(-1, 1, (N, 5)))
    n, w = normals(rng, N), rng.standard_normal((N, 5))
    out = probe(1, np.column_stack([Vi, Vj, n, w]), 13)
    # derivative of w . flux in every direction by a complex step
    x = np.column_stack([Vi, Vj, n]).astype(L)
    ref, h = np.empty((N, 13)), L(1e-40)
    for k in range(13):
        y = x.astype(CL)
        s = np.where(k < 10, L(1.0), np.abs(x[:, 10:]).max(1))   # step relative to the normal's size
        y[:, k] += 1j * h * s
        ref[:, k] = ((roe(y[:, 10:], y[:, :5], y[:, 5:10]) * w).sum(1).imag / (h * s)).astype(np.float64)
    e = [rms_error(out[:, a:b], ref[:, a:b]) for a, b in ((0, 10), (10, 13))]
    print("adjoint of the Roe flux: states %.4g, normal %.4g" % tuple(e))
    # with divisions and roots: 2.850e-16 and 2.647e-16
    assert e[0] <= 1.02 * 2.850e-16
    assert e[1] <= 1.02 * 2.647e-16


def limited(a, b):
    eps, ab = L(1e-16), a * b
    num = np.where(ab > 0, a * (b * b + eps) + b * (a * a + eps), np.where(ab == 0, eps * (a + b) / 2, 0 * a))
    return num / (a * a + b * b + 2 * eps)


def reconstructed(x):
    Vi, di, Vj, dj = x.astype(L).T
    beta = L(1.0 / 3.0)
    d = Vj - Vi
    b2 = (1 - 2 * beta) * d
    return np.column_stack([Vi + limited(b2 + 2 * beta * di, d) / 2, Vj - limited(b2 + 2 * beta * dj, d) / 2])


def test_limiter_rounding_and_range(probe):
    rng = np.random.default_rng(3)
    # the limited increments themselves: V_i = 0 leaves them bare
    d = 10.0 ** rng.uniform(-6, 1, N)
    x = np.column_stack([np.zeros(N), d * rng.uniform(0.2, 2.0, N), d, d * rng.uniform(0.2, 2.0, N)])
    out, ref = probe(2, x, 2), reconstructed(x)
    e = rms_error(out[:, :1], ref[:, :1])
    print(f"limited increment: {e:.4g}")
    # with a reciprocal per side: 1.353e-16
    assert e <= 1.02 * 1.353e-16
    # differences up to 1e100: the numerator's third powers still fit
    big = np.column_stack([np.ones(64), np.ones(64), np.ones(64), np.ones(64)])
    big *= rng.uniform(0.5, 2.0, big.shape) * 10.0 ** rng.uniform(70, 100, (64, 1))
    out, ref = probe(2, big, 2), reconstructed(big)
    assert np.isfinite(out).all() and rms_error(out, ref.astype(np.float64)) < 1e-14


def test_corrected_products(probe):
    # sqrt_ and quot_: half a unit in the last place, and what the correction's
    # own rounding adds (a few 2^-20 of it, from the seed's 23 bits)
    rng = np.random.default_rng(4)
    x = np.column_stack([2.0 ** rng.uniform(-400, 400, N), 2.0 ** rng.uniform(-400, 400, N)])
    out = probe(3, x, 2)
    a, b = x.astype(L).T
    for got, ref in ((out[:, 0], np.sqrt(b)), (out[:, 1], a / b)):
        ulps = np.abs(got - ref) / np.spacing(np.abs(got)).astype(L)
        print(f"{float(ulps.max()):.4f} ulp")
        assert ulps.max() <= 0.51
