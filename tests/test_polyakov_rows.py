"""Polyakov correlators row by row (a block of rows and dy values in shared
memory) against the oracle: extents that the row, site and dy tiles do not
divide, one and several dx tiles, distances beyond the extents.

Tolerance: averages over the sites of products of O(1) lines, FP64 sums in
another order than the oracle's: 1e-13 absolute (values of order 1e-3 to 1);
mixed lines (FP32 links): 1e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-13, "mixed": 1e-6}


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,dims,d", [
    (3, (8, 8, 8, 4), 4), (3, (9, 5, 7, 3), 5), (3, (17, 4, 3, 2), 3), (3, (12, 13, 12, 2), 12),
    (2, (7, 10, 6, 5), 6), (2, (16, 3, 5, 2), 1), (2, (4, 4, 4, 3), 0), (2, (11, 12, 10, 2), 10),
])
def test_matches_oracle(port, precision, nc, dims, d):
    links = generate_config(dims, nc, 0.25, 61, 0)
    with Lattice(dims, nc, precision) as lat:
        lat.upload(links)
        for singlet in (True, False):
            want = port.polyakov_correlator(nc, dims, links, d, singlet)
            got = lat.polyakov_correlator(d, singlet)
            assert np.array_equal(got == 0, want == 0)
            assert np.max(abs(got - want)) <= TOL[precision]


@pytest.mark.parametrize("singlet", [True, False])
def test_distances_beyond_the_extents(singlet):
    """C is periodic: an entry at D and at D shifted by an extent agree."""
    dims, d = (4, 3, 5, 3), 9
    with Lattice(dims, 3, "fp64") as lat:
        lat.upload(generate_config(dims, 3, 0.25, 62, 0))
        n = 2 * d + 1
        c = lat.polyakov_correlator(d, singlet).reshape(n, n, n)  # [z][y][x]
    for x, y, z in ((1, 1, 1), (2, 0, 1), (3, 0, 2), (0, -2, 3)):
        base = c[z + d, y + d, x + d]
        for i, ext in enumerate(dims[:3]):
            v = [x, y, z]
            v[i] += ext
            assert abs(c[v[2] + d, v[1] + d, v[0] + d] - base) <= 1e-13
