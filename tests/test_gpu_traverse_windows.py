"""The traversal's windows of 32 cells where they can go wrong: checkerboard-
like fields whose windows have more distinct edges than a group holds, sparse
surfaces whose windows span many blocks, narrow layouts, volumes of one cell,
outputs cut inside a cell, and a stream left out.  The plain extraction (no
inspection outputs, its own instantiation) against the oracle in order, with
the parity tolerances: positions 1e-5 of the spacing + 4 ulp, normals 1e-5 rad."""
from __future__ import annotations

import numpy as np
import pytest

from tests.gpu_helpers import EPS32, angle, oracle_expect

pytestmark = pytest.mark.gpu

# (z, y, x)
CASES = {
    "one_cell": ((2, 2, 2), "noise"),
    "narrow": ((9, 40, 6), "noise"),
    "dense": ((6, 35, 34), "checker"),
    "dense_wide": ((4, 66, 100), "noise"),
    "sparse": ((90, 64, 64), "plane"),
    "sparse_odd": ((41, 130, 37), "plane"),
}


def _field(shape, kind):
    rng = np.random.default_rng(sum(shape))
    z, y, x = np.indices(shape)
    if kind == "checker":  # nearly every edge crossed
        return ((-1.0) ** (x + y + z) * rng.uniform(0.5, 1.5, shape)).astype(np.float32)
    if kind == "plane":
        return (0.11 * x + 0.07 * y + z - 0.37 * shape[0] + rng.normal(0, 0.01, shape)).astype(np.float32)
    return rng.normal(size=shape).astype(np.float32)


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("normals", [0, 1])
def test_plain_extraction(hpmc, oracle, name, normals):
    import torch

    field = _field(*CASES[name])
    e = oracle_expect(oracle, field, 0.0, normals=normals)
    n = e["total"]
    assert n > 0
    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(torch.from_numpy(field).cuda())
    hp.set_normal_mode(normals)
    hp.build(0.0)
    th = hpmc.TraversalHandle(hp)

    def run(cap, which):
        out = [torch.full((n + 1, 4), float("nan"), device="cuda") for _ in range(2)]
        th.extract_to(*(o if w else None for o, w in zip(out, which)), cap)
        return [o.cpu().numpy() for o in out]

    pos, nrm = run(n, (True, True))
    assert np.isnan(pos[n:]).all() and np.isnan(nrm[n:]).all()
    spacing = 1.0 / np.array(e["L"].cells, np.float64)
    dp = np.abs(pos[:n, :3].astype(np.float64) - e["pos"])
    assert (dp <= 1e-5 * spacing + 4 * EPS32 * np.abs(e["pos"])).all()
    assert (pos[:n, 3] == 1.0).all() and (nrm[:n, 3] == 0.0).all()
    ang, _, nb = angle(nrm[:n, :3], e["nrm"])
    assert ang[nb > 1e-6 * max(1.0, nb.max())].max(initial=0.0) <= 1e-5
    for cap in sorted({1, n // 2, n // 2 + 1, n - 1}):  # the outputs end inside a cell
        p, q = run(cap, (True, True))
        np.testing.assert_array_equal(p[:cap], pos[:cap])
        np.testing.assert_array_equal(q[:cap], nrm[:cap])
        assert np.isnan(p[cap:]).all() and np.isnan(q[cap:]).all()
    p, q = run(n, (True, False))
    np.testing.assert_array_equal(p[:n], pos[:n])
    p, q = run(n, (False, True))
    np.testing.assert_array_equal(q[:n], nrm[:n])


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("binary", [False, True])
def test_welded_equals_soup(hpmc, name, binary):
    """The indexed output over the same fields: indices name first occurrences
    in order, and a unique vertex is its first soup vertex, bit for bit."""
    import torch

    field = _field(*CASES[name])
    hp = hpmc.HistoPyramid(hpmc.default_constants())
    hp.set_field_device(torch.from_numpy(field).cuda())
    if binary:
        hp.set_field_as_binary()
    for _ in range(2):  # the scratch is reused
        hp.build(0.0)
        n = hp.acquire_number_of_vertices()
        th = hpmc.TraversalHandle(hp)
        pos, nrm, p, q = (torch.full((n, 4), float("nan"), device="cuda") for _ in range(4))
        idx = torch.full((n,), -1, dtype=torch.int32, device="cuda")
        th.extract_to(pos, nrm, n)
        unique, ni = th.extract_indexed(p, q, idx)
        assert ni == n
        idx = idx.cpu().numpy()
        new = np.maximum.accumulate(np.concatenate(([-1], idx[:-1]))) < idx  # first occurrences, numbered in order
        assert new.sum() == unique and (idx[new] == np.arange(unique)).all()
        np.testing.assert_array_equal(p[:unique].cpu().numpy(), pos.cpu().numpy()[new])
        np.testing.assert_array_equal(q[:unique].cpu().numpy(), nrm.cpu().numpy()[new])
        np.testing.assert_array_equal(p.cpu().numpy()[idx], pos.cpu().numpy())  # a position per edge
