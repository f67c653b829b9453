"""Rounding errors of kernels that compute a quantity in another form than the
plain one: against the exact value, and no larger than the plain form's."""
import numpy as np
import pytest

import mesh_gb300 as mg

pytestmark = pytest.mark.gpu


def matrices(g, a, dtype):
    """host objects as complex matrices [..., n, n] of the given complex type"""
    a = a.astype(np.zeros(0, dtype).real.dtype)
    if g != 2:
        n = 1 if g == 1 else 3
        return (a[..., 0::2] + dtype(1j) * a[..., 1::2]).reshape(a.shape[:-1] + (n, n))
    i = dtype(1j)
    m = np.empty(a.shape[:-1] + (2, 2), dtype)
    m[..., 0, 0], m[..., 0, 1] = a[..., 0] - i * a[..., 3], -a[..., 2] - i * a[..., 1]
    m[..., 1, 0], m[..., 1, 1] = a[..., 2] - i * a[..., 1], a[..., 0] + i * a[..., 3]
    return m


def product(a, b):
    return sum(a[..., :, k, None] * b[..., None, k, :] for k in range(a.shape[-1]))


def dagger(a):
    return np.conj(np.swapaxes(a, -1, -2))


def theta_per_link(g, dims, U, G, dtype):
    """theta with A_mu(x) = proj(g(x) U_mu(x) g(x+mu)^+) link by link"""
    nd = len(dims)
    U, G = matrices(g, U, dtype).reshape(nd, *dims, -1), matrices(g, G, dtype)
    n = G.shape[-1]
    G = G.reshape(*dims, n, n)
    D = np.zeros_like(G)
    for mu in range(nd):
        w = product(product(G, U[mu].reshape(G.shape)), dagger(np.roll(G, -1, mu)))
        A = (w - dagger(w)) / 2
        if n > 1:
            A = A - np.trace(A, axis1=-2, axis2=-1)[..., None, None] / n * np.eye(n)
        A = A.astype(dtype)
        D = D + A - np.roll(A, 1, mu)
    return (np.abs(D.astype(np.clongdouble)) ** 2).sum() / (nd * np.prod(dims))


@pytest.mark.parametrize("dims", [[16, 24], [6, 10, 8], [4, 6, 8, 10]], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("g,p", [(1, 1), (2, 1), (3, 1), (1, 2), (2, 2), (3, 2)])
def test_landau_theta_in_the_gauge(ctx, oracle, g, p, dims):
    """theta where it is all rounding: links that are pure gauge, g in Landau gauge.
    What rounding adds to theta, no more than 1.3 times what the link by link form
    adds in the same precision (without fused multiply-adds); the closing sum
    without the shift adds six to nine times as much"""
    grid, rt = mg.Grid(dims), mg.real_dtype(p)
    h = oracle.random_transform(g, 2, dims, 5)
    one, ga = mg.GaugeField(ctx, g, 2, grid).set_unit(), mg.Lattice(ctx, g, 2, grid)
    mg.gauge_transform(one, mg.site_adj(ga, mg.Lattice(ctx, g, 2, grid).import_(h)))
    U, G = one.export().astype(rt), h.astype(rt)
    L = mg.Landau(mg.GaugeField(ctx, g, p, grid).import_(U))
    L.g.import_(G)
    exact = theta_per_link(g, dims, U, G, np.clongdouble)
    if p == 1:
        assert float(exact) == pytest.approx(oracle.landau_condition(g, 2, dims, U.astype(np.float64),
                                                                     G.astype(np.float64)), rel=1e-6)
    plain = theta_per_link(g, dims, U, G, np.complex64 if p == 1 else np.complex128)
    assert abs(L.condition() - exact) <= 1.3 * abs(plain - exact)


@pytest.mark.parametrize("variant", [-1, 58])
@pytest.mark.parametrize("dims", [[6, 10], [64, 64], [6, 4, 10], [16, 24, 20], [2, 6, 4, 10], [6, 10, 14, 18]],
                         ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("g,p", [(1, 1), (2, 1), (1, 2), (2, 2)])
def test_kinetic_energy_of_unchanged_momenta(ctx, g, p, dims, variant):
    """at beta = 0 the momenta stay and H is their norm: both ends of a trajectory sum
    the same link terms in FP64 (some thousand additions: 1e-13)"""
    h = mg.Hmc(ctx, g, p, mg.Grid(dims), seed=3)
    P = mg.Momenta(ctx, g, p, mg.Grid(dims)).random(5)
    try:
        mg.force_variant(variant)
        rec = h.update_supplied(P, 0.0, 0.0, [0.1, 0.2, 0.1])
    finally:
        mg.force_variant(-1)
    assert abs(rec["H_new"] - rec["H_old"]) <= 1e-13 * rec["H_old"]


@pytest.mark.parametrize("variant", [-1, 58])
@pytest.mark.parametrize("dims", [[64, 64], [16, 24, 20], [6, 10, 14, 18], [16, 16, 8, 16]],
                         ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("g", [1, 2])
def test_fused_steps_round_no_more_than_separate_ones(ctx, g, dims, variant):
    """ten leapfrog steps of FP32 links and momenta against the FP64 ones: the rms
    distance of the fused steps at most 1.02 times that of momentum steps and link
    updates apart (the 1.02: the spread of an rms over some thousand reals)"""
    grid, beta, d = mg.Grid(dims), 2.0 * g, mg.make_deltas("2lf", 0.5, 10)

    def fields(p, U=None, P=None):
        u, m = mg.GaugeField(ctx, g, p, grid), mg.Momenta(ctx, g, p, grid)
        return (u.random(3), m.random(5)) if U is None else (u.import_(U), m.import_(P))

    U0, P0 = (f.export() for f in fields(mg.F32))
    exact, fused, apart = fields(mg.F64, U0, P0), fields(mg.F32, U0, P0), fields(mg.F32, U0, P0)
    try:
        mg.force_variant(variant)
        mg.run_hmd(*fused, beta, d)
        mg.force_variant(0)
        mg.run_hmd(*exact, beta, d)
        for i, t in enumerate(d):
            mg.momentum_step(apart[1], apart[0], beta, t) if i % 2 else mg.evolve(*apart, t)
    finally:
        mg.force_variant(-1)
    for x, f, s in zip(exact, fused, apart):
        ef, es = (np.sqrt(np.mean((y.export().astype(np.float64) - x.export()) ** 2)) for y in (f, s))
        assert ef <= 1.02 * es, (ef, es)
