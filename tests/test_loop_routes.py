"""Off-axis loops of few lines take the exact product (preparing the
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
            out.append(np.array([x[0] for x in w]))
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
