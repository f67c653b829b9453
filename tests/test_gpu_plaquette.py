"""The plaquette's two kernels (tiles with a warp per plane, a thread per site) on
both sides of the line between them, and what they cost on large lattices."""
import ctypes as C
import time

import numpy as np
import pytest

import mesh_gb300 as mg

pytestmark = pytest.mark.gpu

SHAPES = [[2, 2], [6, 10], [64, 66], [2, 2, 2], [6, 4, 10], [24, 22, 26], [2, 2, 2, 2], [2, 6, 4, 10], [12, 10, 14, 8]]


def noalloc(U, g, p, dims):
    out = C.c_double()
    d = (C.c_int32 * len(dims))(*dims)
    assert mg.load().mesh_plaquette_noalloc(0, g, p, len(dims), d, U.device_ptr, None, C.byref(out)) == 0
    return out.value


@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("g,p", [(1, 1), (1, 2), (2, 1), (2, 2), (3, 1), (3, 2)])
def test_plaquette_kernels(ctx, oracle, g, p, dims):
    """against the FP64 oracle on the same links: FP64 a mean of terms with roundings of
    some 1e-16; FP32 terms are products of three, up to 24 roundings of 6e-8 each that
    average out: 1e-6 for one site, 1e-6 in all"""
    U64 = oracle.random_gauge(g, 2, dims, 4)
    U = mg.GaugeField(ctx, g, p, mg.Grid(dims)).import_(U64.astype(mg.real_dtype(p)))
    ref = oracle.plaquette(g, 2, dims, U.export().astype(np.float64))
    got = mg.plaquette(U)
    assert got == pytest.approx(ref, abs=1e-13 if p == 2 else 1e-6)
    ctx.synchronize()
    assert noalloc(U, g, p, dims) == got


@pytest.mark.parametrize("dims", [[64, 96, 84], [64, 96, 86]], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("g", [1, 2])
def test_fp64_plaquette_beside_the_line(ctx, oracle, g, dims):
    """516096 sites in tiles, 528384 by sites"""
    U = mg.GaugeField(ctx, g, 2, mg.Grid(dims)).random(7)
    got = mg.plaquette(U)
    assert got == pytest.approx(oracle.plaquette(g, 2, dims, U.export()), abs=1e-13)
    ctx.synchronize()
    assert noalloc(U, g, 2, dims) == got


@pytest.mark.parametrize("g,dims", [(1, [48, 48, 48, 48]), (2, [48, 48, 48, 48]), (2, [128, 128, 128])],
                         ids=lambda v: str(v) if isinstance(v, int) else "x".join(map(str, v)))
def test_fp32_plaquette_of_large_small_group_lattices(ctx, g, dims):
    """a call costs at most three copies of the links (which read and write them; the
    plaquette reads them once from memory and a few times from the caches)"""
    U, W = (mg.GaugeField(ctx, g, mg.F32, mg.Grid(dims)) for _ in range(2))
    U.random(3)

    def seconds(f, n=10):
        best = 1e9
        for _ in range(5):
            ctx.synchronize()
            t = time.perf_counter()
            for _ in range(n):
                f()
            ctx.synchronize()
            best = min(best, (time.perf_counter() - t) / n)
        return best

    assert seconds(lambda: mg.plaquette(U)) < 3 * seconds(lambda: W.copy_from(U))
