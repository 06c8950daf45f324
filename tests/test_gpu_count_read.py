"""The vertex count of builds that another stream or a captured graph ran: a
handle whose counts are read otherwise leaves them in host memory, which is
only valid for the handle's own stream."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _sphere(radius):
    x, y, z = np.meshgrid(*[np.linspace(-1, 1, 40, dtype=np.float32)] * 3, indexing="ij")
    return (x * x + y * y + z * z - np.float32(radius * radius)).astype(np.float32)


def _count(hpmc, tensor):
    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(tensor)
    hp.build(0.0)
    n = hp.acquire_number_of_vertices()
    hp.close()
    return n


@pytest.mark.parametrize("read_before", [False, True])
@pytest.mark.parametrize("direct_between", [False, True])
def test_count_after_a_replayed_build(hpmc, read_before, direct_between):
    import torch

    small, large = (torch.from_numpy(_sphere(r)).cuda() for r in (0.4, 0.8))
    want = _count(hpmc, large)
    assert 0 < _count(hpmc, small) < want
    field = small.clone()
    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(field)
    hp.build(0.0)  # sets the handle up: nothing is allocated under capture
    if read_before:
        hp.acquire_number_of_vertices()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        hp.set_stream(torch.cuda.current_stream())
        hp.build(0.0)
    if direct_between:
        hp.build(0.0)
        torch.cuda.synchronize()
    field.copy_(large)
    torch.cuda._sleep(2_000_000)
    graph.replay()  # on the default stream, not the handle's
    assert hp.acquire_number_of_vertices() == want
    hp.close()


def test_count_after_the_stream_was_changed(hpmc):
    import torch

    small, large = (torch.from_numpy(_sphere(r)).cuda() for r in (0.4, 0.8))
    want = _count(hpmc, large)
    field = small.clone()
    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(field)
    hp.build(0.0)
    hp.acquire_number_of_vertices()
    field.copy_(large)
    torch.cuda._sleep(2_000_000)
    hp.build(0.0)  # on the default stream, whose work the copy of the count waits for
    hp.set_stream(torch.cuda.Stream())
    assert hp.acquire_number_of_vertices() == want
    hp.close()
