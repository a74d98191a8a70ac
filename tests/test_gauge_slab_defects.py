"""The FP64 unitarity bound of a time slab. The mean bound of the whole lattice
holds because its loops count every link alike; a slab counts the loops of its
first slices, so that links off the group there would weigh up to Lt / t_starts
times as much: one link above 1e-14 takes the exact product.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("scale,method", [(1 + 1.9e-13, "exact"), (1.0, "gauge")])
def test_links_of_the_counted_slices(nc, scale, method):
    dims = (6, 4, 5, 40)
    links = generate_config(dims, nc, 0.25, 72, 0)
    links[3:4 * 120:4] *= scale  # slice 0: a mean defect of 1e-14 over 40 slices
    with Lattice(dims, nc, "fp64") as lat:
        lat.upload(links)
        w = lat.wilson_loop_tslab(1, 1, 2, 1, 3)
        assert lat.wilson_method_used() == method
        lat.set_wilson_method("exact")
        exact = lat.wilson_loop_tslab(1, 1, 2, 1, 3)
    assert np.array_equal(w, exact) if method == "exact" else np.max(abs(w - exact)) <= 1e-13
