"""Adjoint loops of SU(2) in the temporal gauge with two and with four start
slices per thread, on either side of the volume where the number changes, whole
lattices and slabs, against the exact product.

Tolerance: reassociated products of at most 2 (R + T) links, |Tr|^2 of order four:
FP64 1e-12; mixed, FP32 links and traces, 1e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "mixed": 1e-6}


@pytest.mark.parametrize("precision,dims", [
    ("mixed", (16, 16, 16, 16)), ("mixed", (16, 16, 16, 20)), ("mixed", (17, 15, 18, 18)),
    ("fp64", (20, 20, 20, 20)), ("fp64", (20, 20, 21, 20)), ("fp64", (19, 21, 20, 22)),
])
def test_both_numbers_of_starts(precision, dims):
    with Lattice(dims, 2, precision) as lat:
        lat.generate(0.3, 12)
        lat.ape(0.5, 2)
        for t_starts in (None, 7):
            out = []
            for method in ("auto", "exact"):
                lat.set_wilson_method(method)
                out.append(lat.wilson_loop_adjoint(1, 3, 1, 8) if t_starts is None else
                           lat.wilson_loop_tslab(t_starts, 1, 3, 1, 8, adjoint=True))
                assert lat.wilson_method_used() == ("gauge" if method == "auto" else "exact")
            assert np.max(abs(out[0] - out[1])) <= TOL[precision]
