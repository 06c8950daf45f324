"""A build captured once and replayed over changing fields: every count is the
last replay's, also when a count was read before."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sphere(radius):
    x, y, z = np.meshgrid(*[np.linspace(-1, 1, 40, dtype=np.float32)] * 3, indexing="ij")
    return (x * x + y * y + z * z - np.float32(radius * radius)).astype(np.float32)


def _fresh(hpmc, tensor):
    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(tensor)
    hp.build(0.0)
    return hp, hp.acquire_number_of_vertices()


def _captured(hpmc, field):
    """A handle, and a graph with its build of `field`."""
    import torch

    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(field)
    hp.build(0.0)  # sets the handle up: nothing is allocated under capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        hp.set_stream(torch.cuda.current_stream())
        hp.build(0.0)
    hp.set_stream(torch.cuda.current_stream())
    return hp, graph


def test_count_of_every_replay(hpmc):
    import torch

    fields = [torch.from_numpy(_sphere(r)).cuda() for r in (0.4, 0.8, 0.3)]
    want = [_fresh(hpmc, f)[1] for f in fields]
    assert len(set(want)) == 3
    field = fields[0].clone()
    hp, graph = _captured(hpmc, field)
    th = hpmc.TraversalHandle(hp)
    pos = torch.empty((max(want), 4), device="cuda")
    for f, n in zip(fields, want):
        field.copy_(f)
        graph.replay()
        assert hp.acquire_number_of_vertices() == n
        assert th.extract_to(pos, None) == n
