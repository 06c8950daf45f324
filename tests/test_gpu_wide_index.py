"""Fields whose element indices need 64 bits (here: a slice pitch far beyond the
slices) against the same samples stored contiguously: every output bit for bit,
interior and boundary cells, the gradient up to the order of its sums."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPE = (21, 34, 39)  # (z, y, x): odd rows, two tiles each way


@pytest.mark.parametrize("dtype", ["f32", "u8", "unorm8"])
@pytest.mark.parametrize("normals", [0, 1])
def test_wide_index_equals_contiguous(hpmc, dtype, normals):
    import torch

    rng = np.random.default_rng(3)
    if dtype == "f32":
        field, iso = rng.normal(size=SHAPE).astype(np.float32), 0.1
    else:
        field, iso = rng.integers(0, 256, SHAPE).astype(np.uint8), 0.5 if dtype == "unorm8" else 127.5
    small = torch.from_numpy(field).cuda()
    pitch = -(-(1 << 31) // SHAPE[0]) // 4 * 4  # x (slices + 1) >= 2^31 elements
    assert pitch * (SHAPE[0] + 1) >= 1 << 31
    wide = torch.empty(pitch * SHAPE[0], dtype=small.dtype, device="cuda").as_strided(SHAPE, (pitch, 40, 1))
    wide.copy_(small)
    out = []
    for f in (small, wide):
        hp = hpmc.HistoPyramid(hpmc.default_constants())
        hp.set_field_device(f, unorm=dtype == "unorm8")
        hp.set_normal_mode(normals)
        hp.build(iso)
        n = hp.acquire_number_of_vertices()
        assert n > 10000
        th = hpmc.TraversalHandle(hp)
        pos, nrm, p, q = (torch.empty((n, 4), device="cuda") for _ in range(4))
        idx = torch.empty((n,), dtype=torch.int32, device="cuda")
        th.extract_to(pos, nrm, n)
        unique, _ = th.extract_indexed(p, q, idx)
        b = hpmc.Batch([f, small], [iso, iso], normals=normals, unorm=dtype == "unorm8")
        bp, bq = (torch.empty((2 * n, 4), device="cuda") for _ in range(2))
        b.extract(bp, bq)
        assert b.offsets() == [0, n, 2 * n]
        out.append([pos, nrm, p[:unique], q[:unique], idx, bp, bq])
    for a, b in zip(*out):
        assert torch.equal(a, b)
    if dtype == "f32":
        g = []
        cot = torch.randn((2, n, 4), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
        for f in (small, wide):
            hp = hpmc.HistoPyramid(hpmc.default_constants())
            hp.set_field_device(f)
            hp.set_normal_mode(normals)
            hp.build(iso)
            th = hpmc.TraversalHandle(hp)
            d = torch.empty(f.stride(0) * SHAPE[0], device="cuda").as_strided(SHAPE, f.stride())
            d.zero_()
            th.adjoint(cot[0], cot[1], n, d)
            g.append(d.double())
        # at most a few hundred FP32 terms a sample, added in another order
        assert (g[0] - g[1]).abs().max() <= 1e-4 * g[0].abs().max()
