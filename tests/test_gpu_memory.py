"""Device memory that calls keep: bounded, given back, and not needed."""
import pytest
import torch

import mesh_gb300 as mg

pytestmark = pytest.mark.gpu

MB = 1 << 20


def free_bytes():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info(0)[0]


@pytest.fixture()
def own():
    """a context of the test's own, with the kernels of FP64 SU(3) steps loaded"""
    c = mg.Context(0)
    U, P = mg.GaugeField(c, 3, 2, mg.Grid([4] * 4)), mg.Momenta(c, 3, 2, mg.Grid([4] * 4))
    mg.run_hmd(U.random(1), P.random(2), 5.7, [0.1, 0.2, 0.1])
    mg.momentum_step(P, U, 5.7, 0.1)
    try:
        mg.force_variant(0)
        mg.momentum_step(P, U, 5.7, 0.1)
    finally:
        mg.force_variant(-1)
    U.close()
    P.close()
    c.synchronize()
    yield c
    c.close()


def distance(a, b):
    """|a - b| / |b| of two algebra fields; a is overwritten"""
    n = b.norm2()
    return (mg.axpby(a, 1.0, a, -1.0, b).norm2() / n) ** 0.5


@pytest.mark.parametrize("dims", [[4, 64, 64, 64], [32, 52, 52, 52]], ids=lambda d: "x".join(map(str, d)))
def test_momentum_step_keeps_at_most_the_workspace(own, dims):
    """FP64 SU(3) whose two slices of products exceed the workspace's bound, on a short
    lattice (no scratch) and a long one (the call's own): the same momenta as without
    scratch, and no more than 512 MB kept"""
    grid = mg.Grid(dims)
    U, P, Q = mg.GaugeField(own, 3, 2, grid).random(1), mg.Momenta(own, 3, 2, grid).random(2), mg.Momenta(own, 3, 2, grid)
    Q.copy_from(P)
    before = free_bytes()
    mg.momentum_step(P, U, 5.7, 0.3)
    mg.run_hmd(U, P, 5.7, [0.0, 0.2, 0.0])
    own.synchronize()
    assert before - free_bytes() <= 512 * MB + 32 * MB
    try:
        mg.force_variant(0)
        mg.momentum_step(Q, U, 5.7, 0.3)
        mg.momentum_step(Q, U, 5.7, 0.2)
    finally:
        mg.force_variant(-1)
    assert distance(P, Q) < 1e-12


def test_chain_of_a_short_lattice_takes_no_larger_scratch_than_its_bound(own):
    """4x64^3 in FP64: two slices of products are 1.1 GB for 604 MB of links"""
    grid = mg.Grid([4, 64, 64, 64])
    V = 4 * 64**3
    before = free_bytes()
    h = mg.Hmc(own, 3, 2, grid, seed=1)
    own.synchronize()
    used = before - free_bytes()
    h.close()
    assert used <= V * (3 * 576 + 256) + 512 * MB + 64 * MB


@pytest.mark.parametrize("g,p,dims", [(1, 1, [66, 64, 64, 64]), (3, 2, [32, 32, 30, 32])],
                         ids=lambda v: str(v) if isinstance(v, int) else "x".join(map(str, v)))
def test_run_hmd_without_the_second_buffer(own, g, p, dims):
    """links beyond the workspace: the steps apart give the steps' results"""
    grid = mg.Grid(dims)
    U, P = mg.GaugeField(own, g, p, grid).random(1), mg.Momenta(own, g, p, grid).random(2)
    W, Q = mg.GaugeField(own, g, p, grid).copy_from(U), mg.Momenta(own, g, p, grid).copy_from(P)
    d = [0.05, 0.1, 0.05]
    mg.run_hmd(U, P, 2.0 * g, d)
    mg.evolve(W, Q, d[0])
    mg.momentum_step(Q, W, 2.0 * g, d[1])
    mg.evolve(W, Q, d[2])
    assert distance(P, Q) < (1e-14 if p == 2 else 1e-6)
    assert mg.plaquette(U) == pytest.approx(mg.plaquette(W), abs=1e-13 if p == 2 else 1e-8)


@pytest.mark.parametrize("kept", ["workspace", "chains"])
def test_kept_memory_is_given_back_to_an_allocation(own, kept):
    """with 200 MB free, a field of 302 MB finds the 256 MB or more that the context keeps"""
    grid = mg.Grid([64, 16, 16, 16])
    if kept == "workspace":
        U, P = mg.GaugeField(own, 3, 2, grid).random(1), mg.Momenta(own, 3, 2, grid).random(2)
        mg.momentum_step(P, U, 5.7, 0.1)
        own.synchronize()
        U.close()
        P.close()
    else:
        mg.Hmc(own, 3, 2, grid, seed=1).close()
    torch.cuda.empty_cache()
    hog = torch.empty(free_bytes() - 200 * MB, dtype=torch.uint8, device="cuda")
    try:
        assert free_bytes() < 220 * MB
        f = mg.GaugeField(own, 3, 1, mg.Grid([32] * 4))
        f.set_unit()
        assert mg.plaquette(f) == 1.0
        f.close()
    finally:
        del hog
        torch.cuda.empty_cache()


def test_refused_allocation_leaves_the_context_usable(own):
    """a field larger than the device (1.2e9 sites of FP64 SU(3): 702 GB) is refused, and
    the next call does not find the error"""
    with pytest.raises(mg.MeshError, match="out of memory"):
        mg.GaugeField(own, 3, 2, mg.Grid([186] * 4))
    assert mg.plaquette(mg.GaugeField(own, 3, 2, mg.Grid([4] * 4)).set_unit()) == 1.0


def test_workspace_grows_beside_a_capture(own):
    """FP64 SU(3) steps that need a (larger) workspace, on the context's stream, while
    the thread captures another stream: the capture stays valid, the momenta are those
    of a step without one"""
    x = torch.zeros(64, device="cuda")
    fields = []
    for dims in ([4, 4, 4, 8], [8, 8, 8, 8]):
        grid = mg.Grid(dims)
        U, P = mg.GaugeField(own, 3, 2, grid).random(1), mg.Momenta(own, 3, 2, grid).random(2)
        fields.append((U, P, mg.Momenta(own, 3, 2, grid).copy_from(P)))
    own.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        x += 1
        for U, P, _ in fields:
            mg.momentum_step(P, U, 5.7, 0.3)
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 1.0
    for U, P, Q in fields:
        mg.momentum_step(Q, U, 5.7, 0.3)
        assert distance(P, Q) < 1e-15
