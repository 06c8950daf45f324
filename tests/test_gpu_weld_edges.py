"""The welded output of the window fields by the edges themselves: as many unique
vertices as the soup has distinct lattice edges, numbered by first occurrence,
and every soup vertex indexed to its own edge -- whether a window's cells share
the edge or different windows, blocks or slices list it."""
from __future__ import annotations

import numpy as np
import pytest

from tests.test_gpu_indexed import _expected, _soup_and_indexed
from tests.test_gpu_traverse_windows import CASES, _field

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name", sorted(CASES))
@pytest.mark.parametrize("binary", [False, True])
def test_one_vertex_per_edge(hpmc, oracle, name, binary):
    field = _field(*CASES[name])
    g = _soup_and_indexed(hpmc, field, 0.0, binary=binary)
    assert g["n"] > 0 and g["ni"] == g["n"]
    idx, first = _expected(oracle, field.shape, g)
    assert g["nu"] == len(first)
    np.testing.assert_array_equal(g["idx"], idx)
    np.testing.assert_array_equal(g["upos"], g["pos"][first])
    np.testing.assert_array_equal(g["unrm"], g["nrm"][first])
