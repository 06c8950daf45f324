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


def _welded(hpmc, hp, n, th=None):
    """unique, indices and positions of the handle's last build, room for n soup vertices."""
    import torch

    th = th or hpmc.TraversalHandle(hp)
    p, q = (torch.full((n, 4), float("nan"), device="cuda") for _ in range(2))
    idx = torch.full((n,), -2, dtype=torch.int32, device="cuda")
    unique, ni = th.extract_indexed(p, q, idx)
    return unique, ni, idx.cpu().numpy(), p.cpu().numpy()


def test_welded_mesh_of_every_replay(hpmc):
    import torch

    fields = [torch.from_numpy(_sphere(r)).cuda() for r in (0.4, 0.8, 0.3)]
    field = fields[0].clone()
    hp, graph = _captured(hpmc, field)
    th = hpmc.TraversalHandle(hp)
    for f in fields:
        fresh, n = _fresh(hpmc, f)
        want = _welded(hpmc, fresh, n)
        hp.acquire_number_of_vertices()  # of the replay before
        field.copy_(f)
        graph.replay()
        got = _welded(hpmc, hp, n, th)
        assert got[:2] == want[:2] and got[1] == n
        np.testing.assert_array_equal(got[2], want[2])
        np.testing.assert_array_equal(got[3], want[3])


def _set_total(hp, total):
    """The device's vertex count, as a build between the count's reading and the weld leaves it."""
    import ctypes as C

    p, v = C.c_void_p(), C.c_ulonglong(total)
    import hpmc_b200

    assert hpmc_b200.lib().HPMCgetDeviceVertexCount(hp.ptr, C.byref(p)) == 0
    assert C.CDLL("libcudart.so.12").cudaMemcpy(p, C.byref(v), C.c_size_t(8), 1) == 0


@pytest.mark.parametrize("binary", [False, True])
@pytest.mark.parametrize("drop", [1, 2, 5, 40])
def test_weld_stays_inside_the_count_it_was_given(hpmc, drop, binary):
    """The weld's scratch is sized by the count the host read.  Where the
    device's total is larger, the first `count` soup vertices are welded; where
    it is smaller, the indices end with it."""
    import torch

    field = torch.from_numpy(_sphere(0.6)).cuda()
    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(field)
    if binary:
        hp.set_field_as_binary()
    hp.build(0.5 if binary else 0.0)
    hp.build(0.5 if binary else 0.0)  # (the count of the first was not read: the second's is copied)
    n = hp.acquire_number_of_vertices()
    unique, _, idx, pos = _welded(hpmc, hp, n)
    assert n > 100
    head = int(idx[:n - drop].max()) + 1  # vertices of the first n - drop soup vertices
    for total, count in ((n, n - drop), (n - drop, n)):
        hp.build(0.5 if binary else 0.0)
        hp.build(0.5 if binary else 0.0)
        _set_total(hp, count)
        assert hp.acquire_number_of_vertices() == count
        _set_total(hp, total)
        u, ni, i, p = _welded(hpmc, hp, n)
        assert (u, ni) == (head, count)
        np.testing.assert_array_equal(i[:n - drop], idx[:n - drop])
        assert (i[n - drop:] == -2).all()
        np.testing.assert_array_equal(p[:head], pos[:head])
        assert np.isnan(p[head:]).all()
