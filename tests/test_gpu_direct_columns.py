"""The direct column classifier (column layouts without a tensor map) at the
edges of its tiles: footprints of 17, 32, 33 and 64 cells with remainders,
columns of one slice, of a whole box of 8 layers and one layer more.  Codes,
levels, order and geometry against the oracle (bit-exact topology, the parity
tolerances of tests/gpu_helpers.py)."""
from __future__ import annotations

import numpy as np
import pytest

from tests.gpu_helpers import compare, oracle_expect, run_gpu

pytestmark = pytest.mark.gpu

# (z, y, x)
SHAPES = [(2, 18, 18), (8, 33, 33), (9, 34, 18), (10, 18, 65), (17, 66, 33), (65, 35, 34)]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("kind", ["f32", "f32_pitched", "u8", "unorm8", "f32x4", "functor"])
def test_direct_columns(hpmc, oracle, shape, kind):
    rng = np.random.default_rng(sum(shape) + len(kind))
    kw, iso, okw = {}, 0.0, {}
    if kind.startswith("f32"):
        field = rng.normal(size=shape + ((4,) if kind == "f32x4" else ())).astype(np.float32)
        kw = {"pitch_pad": 3} if kind == "f32_pitched" else {"texture": True} if kind == "f32x4" else {}
    elif kind == "functor":
        field, iso = oracle.Functor("hpmc:cayley", [], shape), 0.1
    else:
        field = rng.integers(100, 156, size=shape).astype(np.uint8)
        okw = {"unorm": kind == "unorm8"}
        iso = 128.0 / 255.0 if kind == "unorm8" else 128.0
    g = run_gpu(hpmc, field, iso, **kw, **okw)
    row_bytes = {"f32": 4 * shape[2], "f32_pitched": 4 * (shape[2] + 3), "u8": shape[2], "unorm8": shape[2]}.get(kind, 1)
    assert g["path"] == (1 if row_bytes % 16 == 0 else 0)  # a tensor map covers rows of 16-byte multiples
    compare(g, oracle_expect(oracle, field, iso, **okw))


@pytest.mark.parametrize("dtype", ["f32", "u8"])
def test_batch_without_tensor_maps(hpmc, dtype):
    """One launch classifies every volume without a tensor map, columns and
    narrow ones; after an iso-value update the captured sequence uses the new
    values.  Per volume the handle path's vertices, bit for bit."""
    import torch

    rng = np.random.default_rng(7)
    shapes = [(5, 33, 33), (12, 9, 11), (9, 18, 65), (20, 7, 30), (3, 70, 18), (34, 35, 37)]
    if dtype == "f32":
        fields, isos = [rng.normal(size=s).astype(np.float32) for s in shapes], [[0.0] * 6, [0.3] * 6]
    else:
        fields, isos = [rng.integers(100, 156, size=s).astype(np.uint8) for s in shapes], [[128.0] * 6, [120.0] * 6]
    b = hpmc.Batch([torch.from_numpy(f).cuda() for f in fields], isos[0])
    pos = torch.empty((2_000_000, 4), device="cuda")
    nrm = torch.empty_like(pos)
    for values in isos:
        b.set_iso_values(values)
        b.extract(pos, nrm)
        offs = b.offsets()
        for i, f in enumerate(fields):
            g = run_gpu(hpmc, f, values[i], capture_codes=False)
            assert offs[i + 1] - offs[i] == g["n"]
            np.testing.assert_array_equal(pos[offs[i]:offs[i + 1]].cpu().numpy(), g["pos"])
            np.testing.assert_array_equal(nrm[offs[i]:offs[i + 1]].cpu().numpy(), g["nrm"])
    b.close()
