"""GEVP loops take the gauge form where its preparation pays, by extents and
range: on either side of the rule's lines the method that ran is the one stated,
and the tables agree (FP64 1e-12, mixed 1e-6: reassociated products of at most
2 (R + T) links, loops of order one).
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu

CASES = [
    (3, "fp64", (16, 16, 16, 4), 6, 2, "exact"), (3, "fp64", (12, 12, 12, 8), 4, 3, "gauge"),
    (3, "fp64", (10, 10, 10, 10), 4, 3, "exact"), (3, "fp64", (10, 10, 10, 10), 4, 4, "gauge"),
    (3, "mixed", (12, 12, 12, 12), 6, 6, "exact"), (3, "mixed", (8, 8, 8, 14), 5, 5, "exact"),
    (3, "mixed", (8, 8, 8, 14), 5, 6, "gauge"), (2, "fp64", (12, 12, 12, 12), 6, 6, "exact"),
    (2, "mixed", (14, 14, 14, 14), 6, 6, "gauge"), (2, "mixed", (20, 20, 20, 10), 8, 5, "exact"),
]


@pytest.mark.parametrize("nc,precision,dims,r,t,method", CASES)
def test_route(nc, precision, dims, r, t, method):
    with Lattice(dims, nc, precision) as a, Lattice(dims, nc, precision) as b:
        a.upload(generate_config(dims, nc, 0.2, 3, 0))
        b.copy_from(a)
        b.ape(0.5, 2)
        w = a.wilson_gevp(b, 1, r, 1, t)
        assert a.wilson_method_used() == method
        a.set_wilson_method("exact")
        exact = a.wilson_gevp(b, 1, r, 1, t)
        assert np.max(abs(w - exact)) <= (1e-12 if precision == "fp64" else 1e-6)
