"""Spatial Wilson loops in the gauge of their time axis against the exact
product of links (which the oracle and the reference's fixtures check).

Tolerances as for the other gauge forms: FP64 1e-12 of the largest value
(reassociated products of at most 2 (R + T) links), mixed 1e-6 (FP32 links).
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "mixed": 1e-6}


def _both(lat, *args):
    out = []
    for method in ("auto", "exact"):
        lat.set_wilson_method(method)
        out.append(lat.wilson_spatial_3d(*args))
    assert out[0].keys() == out[1].keys()
    a, b = (np.array([w[k] for k in sorted(w)]) for w in out)
    return a, b


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,dims,args", [
    # r, T ranges, alpha, smearing start / end / step; unequal extents, so that
    # each plane's reordered lattice has its own
    (3, (8, 6, 10, 4), (1, 4, 1, 3, 0.5, 1, 5, 2)),
    (3, (5, 7, 4, 3), (1, 6, 1, 2, 0.5, 1, 2, 1)),
    (2, (12, 9, 10, 5), (1, 3, 1, 4, 0.4, 1, 4, 3)),
    (2, (33, 32, 34, 2), (1, 2, 1, 16, 0.5, 1, 1, 1)),
    (3, (4, 4, 6, 3), (2, 3, 1, 2, 0.5, 1, 2, 1)),  # r_min > 1: exact in both
    (3, (4, 6, 4, 3), (1, 2, 1, 3, 0.5, 1, 2, 1)),  # T > L/2 on two axes: exact
])
def test_matches_the_exact_product(precision, nc, dims, args):
    with Lattice(dims, nc, precision) as lat:
        lat.upload(generate_config(dims, nc, 0.25, 51, 0))
        a, b = _both(lat, *args)
        assert np.max(abs(a - b)) <= TOL[precision] * np.max(abs(b))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("axis", [0, 1, 2])
def test_one_axis_off_the_group(precision, axis):
    """A link of one axis scaled: its planes take the exact product, the
    others' loops do not change; the table is the exact one's."""
    dims = (6, 8, 4, 4)
    links = generate_config(dims, 3, 0.25, 52, 0).reshape(-1, 4, 18)
    links[29, axis] *= 1.001
    with Lattice(dims, 3, precision) as lat:
        lat.upload(links.reshape(-1, 18))
        a, b = _both(lat, 1, 3, 1, 2, 0.5, 1, 3, 1)
        assert np.max(abs(a - b)) <= TOL[precision] * np.max(abs(b))
