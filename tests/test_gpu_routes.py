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
