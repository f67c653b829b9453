"""The kernels that work in tiles of sites, at the sizes where a tile can go
wrong: lattices smaller than a tile, volumes that are no multiple of one, the
smallest extents, every number of dimensions. FP64 against the FP64 oracle at
1e-12 (a result is a sum of at most some hundred roundings of O(1) terms), FP32
at 2e-5."""
import numpy as np
import pytest

import mesh_gb300 as mg

pytestmark = pytest.mark.gpu

SHAPES = [[2, 2], [6, 10], [2, 2, 2], [6, 4, 10], [2, 2, 2, 2], [2, 6, 4, 10], [4, 4, 6, 8]]


def rel(a, b):
    a, b = np.asarray(a, dtype=np.float64), np.asarray(b, dtype=np.float64)
    return float(np.max(np.abs(a - b)) / max(1e-300, float(np.max(np.abs(b)))))


def links(oracle, g, dims, seed=4):
    return oracle.random_gauge(g, 2, dims, seed)


@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("g", [1, 2, 3])
def test_landau_closing_sum(ctx, oracle, g, dims):
    """theta, derivative and overrelaxation half sweeps from the closing sum"""
    U64, h64 = links(oracle, g, dims), oracle.random_transform(g, 2, dims, 5)
    L = mg.Landau(mg.GaugeField(ctx, g, 2, mg.Grid(dims)).import_(U64))
    L.g.import_(h64)
    assert L.condition() == pytest.approx(oracle.landau_condition(g, 2, dims, U64, h64), rel=1e-12)
    assert rel(L.deriv().export(), oracle.landau_deriv(g, 2, dims, U64, h64)) < 1e-12
    L.overrelax(1.7, tol=0.0, max_sweeps=2, check_every=2)
    assert rel(L.g.export(), oracle.landau_or_sweeps(g, 2, dims, U64, h64, 1.7, 2)) < 1e-11


@pytest.mark.parametrize("overrelax", [False, True])
@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
def test_fp64_su3_sweeps(ctx, oracle, dims, overrelax):
    """one heat-bath / overrelaxation sweep of FP64 SU(3) links, draw for draw"""
    g = 3
    U64 = links(oracle, g, dims)
    U = mg.GaugeField(ctx, g, 2, mg.Grid(dims)).import_(U64)
    if overrelax:
        mg.overrelax_sweep(U)
    else:
        mg.heatbath_sweep(U, 2.0 * g, 21, 3)
    ref = oracle.gauge_sweep(g, 2, dims, U64, 2.0 * g, 21, 3, overrelax=overrelax)
    assert rel(U.export(), ref) < 1e-11


@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("g,p", [(1, 2), (2, 2), (3, 2), (3, 1)])
def test_plaquette_tiles(ctx, oracle, g, p, dims):
    U64 = links(oracle, g, dims)
    U = mg.GaugeField(ctx, g, p, mg.Grid(dims)).import_(U64.astype(mg.real_dtype(p)))
    assert mg.plaquette(U) == pytest.approx(oracle.plaquette(g, 2, dims, U64), abs=1e-13 if p == 2 else 1e-6)


@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
def test_fp64_su3_md_step_from_products(ctx, oracle, dims):
    """momentum step alone and with the link update, for links that are no
    group elements (the forces are those of the staples for any matrices)"""
    U64 = links(oracle, 3, dims) * 1.01
    P64 = oracle.random_momenta(3, 2, dims, 11, 0)
    U = mg.GaugeField(ctx, 3, 2, mg.Grid(dims)).import_(U64)
    P = mg.Momenta(ctx, 3, 2, mg.Grid(dims)).import_(P64)
    mg.momentum_step(P, U, 5.7, 0.3)
    Po = oracle.momentum_step(3, 2, dims, U64, P64, 5.7, 0.3)
    assert rel(P.export(), Po) < 1e-12
    h = mg.Hmc(ctx, 3, 2, mg.Grid(dims), seed=1)
    h.U.import_(U64)
    h.P.import_(P64)
    h.md_step(5.7, 0.3, 0.25)
    assert rel(h.P.export(), Po) < 1e-12
    assert rel(h.U.export(), oracle.evolve(3, 2, dims, U64, Po, 0.25)) < 1e-12


@pytest.mark.parametrize("dims", [[32, 16, 16, 16], [2, 36, 44, 46], [6, 48, 40, 22]], ids=lambda d: "x".join(map(str, d)))
def test_fp64_su3_md_step_in_slabs(ctx, dims):
    """lattices whose products exceed the scratch (slabs of dimension 0; the
    smallest ring, a ring that does not divide the extent): the same step as the
    thread-per-link kernel, and the kinetic energy of a whole trajectory"""
    grid = mg.Grid(dims)
    out = []
    for variant in (-1, 0):
        h = mg.Hmc(ctx, 3, 2, grid, seed=3)
        h.randomize_gauge_field()
        P = mg.Momenta(ctx, 3, 2, grid).random(5)
        try:
            mg.force_variant(variant)
            rec = h.update_supplied(P, 0.0, 5.7, [0.05, 0.1, 0.05])
        finally:
            mg.force_variant(-1)
        out.append((rec, h.U.export(), h.P.export()))
    (ra, ua, pa), (rb, ub, pb) = out
    assert rel(ua, ub) < 1e-12 and rel(pa, pb) < 1e-12
    assert ra["H_new"] == pytest.approx(rb["H_new"], rel=1e-12)


@pytest.mark.parametrize("dims", SHAPES + [[4, 6, 10, 14]], ids=lambda d: "x".join(map(str, d)))
def test_fp32_su3_step_from_plaquettes(ctx, oracle, dims):
    """one MD step and a trajectory (whose inner steps write rows 0 and 1 of the
    links only) of the autotuned chain against the FP64 oracle; small lattices
    choose the step from stored plaquettes"""
    U64 = oracle.hmc_chain(3, 2, dims, oracle.unit_gauge(3, 2, dims), 5.7, oracle.make_deltas("2lf", 0.5, 8), 3, 0, 2)[0]
    P64 = oracle.random_momenta(3, 2, dims, 11, 0)
    U32, P32 = U64.astype(np.float32), P64.astype(np.float32)
    h = mg.Hmc(ctx, 3, mg.F32, mg.Grid(dims), seed=1)
    h.U.import_(U32)
    h.P.import_(P32)
    h.md_step(5.7, 0.07, 0.05)
    Po = oracle.momentum_step(3, 2, dims, U64, P64, 5.7, 0.07)
    assert rel(h.P.export(), Po) < 2e-5
    assert rel(h.U.export(), oracle.evolve(3, 2, dims, U64, Po, 0.05)) < 2e-5
    h.U.import_(U32)
    d = oracle.make_deltas("2mn", 0.5, 5)
    h.update_supplied(mg.Momenta(ctx, 3, mg.F32, mg.Grid(dims)).import_(P32), 0.0, 5.7, d)
    U_new, _ = oracle.hmc_update(3, 2, dims, U64, P64, 5.7, d, 0.0)
    assert rel(h.U.export(), U_new) < 2e-5


def test_fp32_su3_step_from_plaquettes_in_slabs(ctx):
    """a lattice whose plaquettes exceed the scratch: the trajectory of the
    thread-per-link kernel"""
    dims = [40, 32, 34, 32]
    out = []
    for variant in (-1, 0):
        h = mg.Hmc(ctx, 3, mg.F32, mg.Grid(dims), seed=3)
        h.U.random(9)
        P = mg.Momenta(ctx, 3, mg.F32, mg.Grid(dims)).random(5)
        try:
            mg.force_variant(variant)
            rec = h.update_supplied(P, 0.0, 5.7, [0.05, 0.1, 0.05, 0.1, 0.05])
        finally:
            mg.force_variant(-1)
        out.append((rec, h.U.export(), h.P.export()))
    (ra, ua, pa), (rb, ub, pb) = out
    assert "stored plaquettes" in [ln for ln in mg.tune_report().splitlines() if "md_step/group3/f32/40x32x34x32" in ln][0]
    assert rel(ua, ub) < 2e-5 and rel(pa, pb) < 2e-5
    assert ra["H_new"] == pytest.approx(rb["H_new"], rel=1e-6)


@pytest.mark.parametrize("max_t", [1, 3, 4, 5, 14])
@pytest.mark.parametrize("g,p", [(1, 1), (2, 2), (3, 2), (3, 1)])
def test_wilson_loops_in_chunks(ctx, oracle, g, p, max_t):
    """extents t on both sides of a chunk, tiles with missing sites"""
    dims = [2, 6, 4, 14]
    U64 = links(oracle, g, dims)
    U = mg.GaugeField(ctx, g, p, mg.Grid(dims)).import_(U64.astype(mg.real_dtype(p)))
    W = mg.wilson_loops(U, 2, max_t)
    assert np.max(np.abs(W - oracle.wilson_loops(g, 2, dims, U64, 2, max_t))) < (1e-13 if p == 2 else 2e-6)


@pytest.mark.parametrize("steps", [1, 2])
@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("g,p", [(1, 1), (1, 2), (2, 1), (2, 2), (3, 1), (3, 2)])
def test_run_hmd_fused_steps(ctx, oracle, g, p, dims, steps):
    """momentum steps fused with link updates out of place (an odd and an even
    number of buffer changes) end in U and P"""
    U64, P64 = links(oracle, g, dims), oracle.random_momenta(g, 2, dims, 11, 0)
    dt = mg.real_dtype(p)
    U = mg.GaugeField(ctx, g, p, mg.Grid(dims)).import_(U64.astype(dt))
    P = mg.Momenta(ctx, g, p, mg.Grid(dims)).import_(P64.astype(dt))
    d = oracle.make_deltas("2lf", 0.02, steps)
    mg.run_hmd(U, P, 2.0 * g, d)
    Uo, Po = oracle.run_hmd(g, 2, dims, U64, P64, 2.0 * g, d)
    tol = 1e-12 if p == 2 else 2e-5
    assert rel(U.export(), Uo) < tol and rel(P.export(), Po) < tol


@pytest.mark.parametrize("p", [1, 2])
def test_chains_share_step_scratch(p):
    """graph-replayed chains of a context in turn, the second larger (its scratch
    replaces what later chains share), the third made after the first is gone:
    each as on a context of its own"""
    shapes, d = [[4, 4, 6, 4], [8, 6, 4, 10], [4, 6, 4, 4]], mg.make_deltas("2lf", 0.5, 4)

    def chain(ctx, k):
        h = mg.Hmc(ctx, 3, p, mg.Grid(shapes[k]), seed=5 + k)
        h.cold_start()
        return h

    alone = []
    for k in range(3):
        c = mg.Context(0)
        h = chain(c, k)
        h.run(5.7, d, 3)
        alone.append((h.U.export(), h.history()["plaq_history"]))
        h.close()
        c.close()
    c = mg.Context(0)
    a = chain(c, 0)
    a.run(5.7, d, 1)
    b = chain(c, 1)
    for _ in range(2):
        b.run(5.7, d, 1)
        a.run(5.7, d, 1)
    got = [(a.U.export(), a.history()["plaq_history"])]
    a.close()
    e = chain(c, 2)
    b.run(5.7, d, 1)
    e.run(5.7, d, 3)
    got += [(h.U.export(), h.history()["plaq_history"]) for h in (b, e)]
    for (u, pl), (uo, plo) in zip(got, alone):
        assert rel(u, uo) < (1e-12 if p == 2 else 2e-5)
        assert rel(pl, plo) < (1e-12 if p == 2 else 1e-6)
