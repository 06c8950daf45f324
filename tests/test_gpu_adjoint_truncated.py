"""The adjoint of the first `count` vertices, cut inside a cell: the edges of
that cell whose vertices lie past the cut take no part, whatever their samples.
One cell of case 1 (three vertices) with one edge so short in value, 2e-25, that
the derivative of its crossing overflows FP32; against the FP64 adjoint of the
counted vertices.  Tolerance as in test_gpu_adjoint.py: 1e-5 of the sum of
|terms| per sample."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("normals", [0, 1])
def test_edges_past_the_cut_take_no_part(hpmc, oracle, axis, normals):
    import torch

    field = np.ones((2, 2, 2), np.float32)
    field[0, 0, 0] = -1e-25
    tiny = [0, 0, 0]
    tiny[2 - axis] = 1
    field[tuple(tiny)] = 1e-25
    L = oracle.layout((2, 2, 2))
    levels, total = oracle.pyramid(oracle.codes(field, L, 0.0), L)
    cell, _, _, edge = oracle.traverse(oracle.codes(field, L, 0.0), levels, L, 0, total)
    assert total == 3
    past = [n for n in (1, 2) if (oracle.edge_table()[edge[:n], 3] != axis).all()]  # cuts before the short edge
    rng = np.random.default_rng(axis)
    w, u = (rng.normal(size=(total, 4)).astype(np.float32) for _ in range(2))
    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(torch.from_numpy(field).cuda())
    hp.set_normal_mode(normals)
    hp.build(0.0)
    th = hpmc.TraversalHandle(hp)
    assert hp.acquire_number_of_vertices() == total
    for n in past:
        g = torch.zeros((2, 2, 2), device="cuda")
        th.adjoint(torch.from_numpy(w).cuda(), torch.from_numpy(u).cuda(), n, g)
        want, S = oracle.adjoint(field.astype(np.float64), L, 0.0, cell[:n], edge[:n], w[:n, :3], u[:n, :3],
                                 normal_mode=normals, with_abs=True)
        g = g.double().cpu().numpy()
        assert (np.abs(g - want) <= 1e-5 * S + 1e-9 * np.abs(want).max()).all(), (n, g, want)
    hp.close()


def test_some_cuts_lie_before_the_short_edge(oracle):
    """(The test above is not empty: the last vertex's edge is the short one for one of the axes.)"""
    field = np.ones((2, 2, 2), np.float32)
    field[0, 0, 0] = -1.0
    L = oracle.layout((2, 2, 2))
    codes = oracle.codes(field, L, 0.0)
    levels, total = oracle.pyramid(codes, L)
    edge = oracle.traverse(codes, levels, L, 0, total)[3]
    assert sorted(oracle.edge_table()[edge, 3]) == [0, 1, 2]
