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
