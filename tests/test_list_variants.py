"""Variants of the neighbour-list passes at the sizes where their branches part.

* Candidate lists whose fluid candidates fit but whose boundary candidates do not (those are then walked): the
  passes must still give the cell walks' results bit for bit.
"""
import numpy as np
import pytest

from test_pcisph_lists import drop, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("case,precision,lists", [("impact", "f32", 44), ("impact", "f64", 40), ("wcsph", "f32", 34)])
def test_boundary_candidates_beyond_the_list(gpu_lib, case, precision, lists):
    x, v, b, p = drop(case)
    a, w = (run(x, v, b, p, precision, n, 12, True) for n in (lists, 0))
    for f in ("x", "v", "rho"):
        assert np.array_equal(a.get(f), w.get(f)), f
