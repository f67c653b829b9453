"""Calls whose kernel depends on how they are made."""
import time

import numpy as np
import pytest
import torch

import mesh_gb300 as mg

pytestmark = pytest.mark.gpu


def test_captured_fp64_step_after_a_warm_up():
    """an FP64 SU(3) momentum step captured after a first call (which a captured one does
    not share the scratch of): the momenta of the step without scratch, at no more than
    1.5 times its time"""
    s = torch.cuda.Stream()
    c = mg.Context(0, stream=s.cuda_stream)
    grid = mg.Grid([8, 8, 8, 8])
    U, P = mg.GaugeField(c, 3, 2, grid).random(1), mg.Momenta(c, 3, 2, grid).random(2)
    Q = mg.Momenta(c, 3, 2, grid).copy_from(P)
    mg.momentum_step(P, U, 5.7, 0.0)
    try:
        mg.force_variant(0)
        mg.momentum_step(Q, U, 5.7, 0.0)
    finally:
        mg.force_variant(-1)
    c.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=s):
        mg.momentum_step(P, U, 5.7, 0.1)

    def seconds(f):
        best = 1e9
        for _ in range(5):
            c.synchronize()
            t = time.perf_counter()
            for _ in range(10):
                f()
            c.synchronize()
            best = min(best, (time.perf_counter() - t) / 10)
        return best

    with torch.cuda.stream(s):
        t_graph = seconds(graph.replay)
    try:
        mg.force_variant(0)
        t_plain = seconds(lambda: mg.momentum_step(Q, U, 5.7, 0.1))
    finally:
        mg.force_variant(-1)
    a, b = P.export(), Q.export()
    assert np.max(np.abs(a - b)) <= 1e-12 * np.max(np.abs(b))
    assert t_graph <= 1.5 * t_plain
    c.close()


SCRATCH = 59  # pins the SU(3) steps through scratch


def tuned(prefix):
    return [ln for ln in mg.tune_report().splitlines() if ln.startswith(prefix)]


def rel(a, b):
    return float(np.max(np.abs(a.astype(np.float64) - b)) / np.max(np.abs(b)))


@pytest.mark.parametrize("dims", [[2, 4], [6, 14], [2, 2, 4], [6, 4, 14], [2, 2, 2, 6], [2, 6, 4, 14], [4, 4, 6, 12],
                                  [6, 6, 10, 14]], ids=lambda d: "x".join(map(str, d)))
def test_fp32_step_from_plaquettes_pinned(ctx, oracle, dims):
    """the step from stored plaquettes by name, on lattices that nothing else times:
    one step, and a trajectory whose inner steps write rows 0 and 1 of the links only,
    against the FP64 oracle; nothing was timed for it, so it was the pinned one"""
    d = oracle.make_deltas("2mn", 0.5, 5)
    U64 = oracle.hmc_chain(3, 2, dims, oracle.unit_gauge(3, 2, dims), 5.7, oracle.make_deltas("2lf", 0.5, 8), 3, 0, 2)[0]
    P64 = oracle.random_momenta(3, 2, dims, 11, 0)
    U32, P32 = U64.astype(np.float32), P64.astype(np.float32)
    h = mg.Hmc(ctx, 3, mg.F32, mg.Grid(dims), seed=1)
    h.U.import_(U32)
    h.P.import_(P32)
    try:
        mg.force_variant(SCRATCH)
        h.md_step(5.7, 0.07, 0.05)
        Po = oracle.momentum_step(3, 2, dims, U64, P64, 5.7, 0.07)
        assert rel(h.P.export(), Po) < 2e-5
        assert rel(h.U.export(), oracle.evolve(3, 2, dims, U64, Po, 0.05)) < 2e-5
        h.U.import_(U32)
        h.update_supplied(mg.Momenta(ctx, 3, mg.F32, mg.Grid(dims)).import_(P32), 0.0, 5.7, d)
    finally:
        mg.force_variant(-1)
    assert rel(h.U.export(), oracle.hmc_update(3, 2, dims, U64, P64, 5.7, d, 0.0)[0]) < 2e-5
    assert not tuned("md_step/group3/f32/" + "x".join(map(str, dims)))


@pytest.mark.parametrize("dims", [[44, 32, 30, 32], [6, 88, 92, 90]], ids=lambda d: "x".join(map(str, d)))
def test_fp32_step_from_plaquettes_pinned_in_slabs(ctx, dims):
    """lattices whose plaquettes exceed the scratch (a ring that does not divide the
    extent, two slices): the trajectory of the kernel with a thread per link"""
    out = []
    for variant in (SCRATCH, 0):
        h = mg.Hmc(ctx, 3, mg.F32, mg.Grid(dims), seed=3)
        h.U.random(9)
        P = mg.Momenta(ctx, 3, mg.F32, mg.Grid(dims)).random(5)
        try:
            mg.force_variant(variant)
            rec = h.update_supplied(P, 0.0, 5.7, [0.05, 0.1, 0.05, 0.1, 0.05])
        finally:
            mg.force_variant(-1)
        out.append((rec, h.U.export(), h.P.export()))
        h.close()
    (ra, ua, pa), (rb, ub, pb) = out
    assert not tuned("md_step/group3/f32/" + "x".join(map(str, dims)))
    assert rel(ua, ub) < 2e-5 and rel(pa, pb) < 2e-5
    assert ra["H_new"] == pytest.approx(rb["H_new"], rel=1e-6)


@pytest.mark.parametrize("dims,lines", [([16, 32, 32, 30], 0), ([16, 32, 32, 32], 1)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, list) else "")
def test_chain_without_scratch(dims, lines):
    """a chain made when there is no memory for its scratch runs the kernels without
    (timing the fused ones where tiles divide the extents), and leaves the lattice's
    other chains their choice"""
    mb, V, grid = 1 << 20, int(np.prod(dims)), mg.Grid(dims)
    d = mg.make_deltas("2lf", 0.5, 4)
    c = mg.Context(0)
    small = mg.Hmc(c, 3, mg.F32, mg.Grid([4, 4, 4, 6]), seed=1)
    small.run(5.7, d, 1)
    mg.Momenta(c, 3, mg.F32, mg.Grid([4, 4, 4, 6])).random(5)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    own = V * (3 * 288 + 128)
    hog = torch.empty(torch.cuda.mem_get_info(0)[0] - own - 60 * mb, dtype=torch.uint8, device="cuda")
    out, key = [], "md_step/group3/f32/" + "x".join(map(str, dims))
    for scratch in (False, True):
        h = mg.Hmc(c, 3, mg.F32, grid, seed=3)
        if not scratch:
            del hog
            torch.cuda.empty_cache()
        h.U.random(9)
        P = mg.Momenta(c, 3, mg.F32, grid).random(5)
        h.update_supplied(P, 0.0, 5.7, d)
        out.append(h.U.export())
        assert ["stored plaquettes=" in ln for ln in tuned(key)] == [True] * scratch + [False] * lines
        h.close()
        P.close()
    assert rel(*out) < 2e-5
    small.close()
    c.close()


@pytest.mark.parametrize("eps", [3e3, 4e5, 1.5e6, 1e7])
@pytest.mark.parametrize("dims", [[14, 14, 14, 16], [16, 16, 16, 16]], ids=lambda d: "x".join(map(str, d)))
def test_line_search_trials(ctx, oracle, dims, eps):
    """FP64 SU(3) links of 25 and 38 MB: both trials read together, and one after the
    other; steps that grow and steps that overshoot. The step is a ratio of differences of
    functionals that agree in some digits: 1e-6"""
    U64, g64 = oracle.random_gauge(3, 2, dims, 4), oracle.random_transform(3, 2, dims, 5)
    L = mg.Landau(mg.GaugeField(ctx, 3, 2, mg.Grid(dims)).import_(U64))
    L.g.import_(g64)
    F = L.deriv()
    got = L.line_search(F, eps)
    assert got == pytest.approx(oracle.landau_line_search(3, 2, dims, U64, g64, F.export(), eps), rel=1e-6)


def test_line_search_makes_no_trial_in_vain(ctx):
    """SU(2) FP64 32^4: a search that the longer trial wins, against one on the same
    fields that needs the shorter one too (four trials for three): at most 0.85 of its time"""
    U = mg.GaugeField(ctx, 2, 2, mg.Grid([32] * 4)).random(3)
    L = mg.Landau(U)
    F = L.deriv()

    def search(eps):
        best = 1e9
        for _ in range(5):
            t = time.perf_counter()
            for _ in range(3):
                s = L.line_search(F, eps)
            best = min(best, time.perf_counter() - t)
        return best, s

    (t1, s1), (t2, s2) = search(1.0), search(1e7)
    assert s1 == 1.2 and s2 > 1.3e7  # neither was halved
    assert t1 <= 0.85 * t2
