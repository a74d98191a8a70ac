"""Off-axis and spatial loops of few lines take the exact product (preparing the
gauge costs more than their walk): the same bits as with the method set to exact.
With more lines the gauge form runs (other roundings) and agrees within the
form's accuracy (FP64 1e-12, mixed 1e-6: products of a few links, values of order
one).
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "mixed": 1e-6}


def _both(nc, precision, dims, call):
    with Lattice(dims, nc, precision) as lat:
        lat.upload(generate_config(dims, nc, 0.25, 9, 0))
        out = []
        for method in ("auto", "exact"):
            lat.set_wilson_method(method)
            w = call(lat)
            out.append(np.array([w[k] for k in sorted(w)] if isinstance(w, dict)
                                else [x[0] for x in w]))
    return out


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,dims,dirs,r_max,t_max,gauge", [
    (3, (12, 12, 12, 8), [[1, 0, 0]], 1.0, 4, False), (2, (10, 12, 9, 8), [[1, 0, 0]], 5.0, 3, False),
    (3, (8, 8, 8, 8), [[1, 0, 0]], 6.0, 3, True), (2, (8, 6, 7, 8), [[1, 1, 0]], 4.0, 3, True),
])
def test_offaxis(nc, precision, dims, dirs, r_max, t_max, gauge):
    auto, exact = _both(nc, precision, dims,
                        lambda lat: lat.wilson_offaxis(dirs, 0.9, r_max, 1, t_max))
    assert np.array_equal(auto, exact) != gauge
    assert np.max(abs(auto - exact)) <= TOL[precision]


@pytest.mark.parametrize("nc,precision,r,t,steps,gauge", [
    (3, "fp64", 1, 4, 2, False), (3, "fp64", 2, 1, 0, True), (2, "mixed", 1, 4, 1, False),
    (2, "mixed", 2, 1, 0, True), (3, "mixed", 2, 2, 0, False), (3, "mixed", 2, 1, 3, False),
    (3, "mixed", 2, 2, 1, True), (3, "mixed", 3, 2, 0, True),
])
def test_spatial(nc, precision, r, t, steps, gauge):
    auto, exact = _both(nc, precision, (8, 10, 8, 6),
                        lambda lat: lat.wilson_spatial_3d(1, r, 1, t, 0.5, 0, steps, 1))
    assert np.array_equal(auto, exact) != gauge
    assert np.max(abs(auto - exact)) <= TOL[precision]
