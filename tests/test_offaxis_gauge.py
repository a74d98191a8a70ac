"""Off-axis loops in the temporal gauge (the default where the links pass the
device's check and T <= Lt/2) against the exact product of links, which the
oracle and the reference's fixtures check.

Tolerances: FP64, a loop is a product of at most 30 links and two reassociated
time lines, an average of loops of order one: 1e-12 relative to the largest
value. Mixed: FP32 links and traces, 1e-6 (the form's accuracy bar).
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "mixed": 1e-6}


def _both(lat, dirs, *rng, adjoint=False):
    out = []
    for method in ("auto", "exact"):
        lat.set_wilson_method(method)
        out.append(lat.wilson_offaxis(dirs, *rng, adjoint=adjoint))
    (a, b) = out
    assert [x[1:] for x in a] == [x[1:] for x in b]
    return np.array([x[0] for x in a]), np.array([x[0] for x in b])


DIRS = [[1, 0, 0], [1, 1, 0], [1, 1, 1], [2, 1, 0], [2, 2, 1], [3, 2, 1], [4, 3, 3]]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,dims,rng", [
    (3, (4, 4, 4, 8), (0.9, 3.1, 1, 4)),       # T up to Lt/2: both cuts on every slice
    (3, (5, 3, 7, 9), (0.9, 6.5, 2, 3)),       # odd extents, lines longer than the lattice
    (2, (6, 4, 3, 10), (0.9, 5.0, 1, 5)),
    (2, (3, 5, 4, 13), (1.9, 4.0, 1, 1)),
    (3, (4, 2, 3, 40), (0.9, 2.0, 1, 6)),      # more slots than a block's usual threads
    (2, (2, 3, 2, 200), (0.9, 1.0, 3, 100)),   # the largest block that fits, or the exact form
])
def test_gauge_form_matches_the_exact_product(precision, nc, dims, rng):
    with Lattice(dims, nc, precision) as lat:
        lat.upload(generate_config(dims, nc, 0.25, 31, 0))
        lat.hyp(1.0, 0.75, 0.6, 1)
        lat.ape(0.5, 2)
        for adjoint in (False, True):
            a, b = _both(lat, DIRS, *rng, adjoint=adjoint)
            assert len(a) and np.max(abs(a - b)) <= TOL[precision] * np.max(abs(b))


def test_merged_table_and_repeated_directions():
    dims = (6, 6, 6, 8)
    with Lattice(dims, 3, "fp64") as lat:
        lat.upload(generate_config(dims, 3, 0.25, 32, 0))
        got = lat.wilson_offaxis_result(1.0, 5.0, 1, 3)
        lat.set_wilson_method("exact")
        want = lat.wilson_offaxis_result(1.0, 5.0, 1, 3)
        assert got.keys() == want.keys()
        assert max(abs(got[k] - want[k]) for k in want) <= 1e-12
        lat.set_wilson_method("auto")
        a, _ = _both(lat, [[1, 1, 0], [1, 1, 0]], 0.9, 3.0, 1, 2)
        assert np.array_equal(a[:len(a) // 2], a[len(a) // 2:])


@pytest.mark.parametrize("precision,which", [("fp64", 3), ("mixed", 3), ("mixed", 1)])
def test_links_that_are_not_unitary_take_the_exact_product(precision, which):
    """A time link (and, for 12-real storage, a spatial link) scaled off the
    group: bit for bit the exact form's loops."""
    dims = (4, 3, 4, 6)
    links = generate_config(dims, 3, 0.25, 33, 0).reshape(-1, 4, 18)
    links[17, which] *= 1.001
    with Lattice(dims, 3, precision) as lat:
        lat.upload(links.reshape(-1, 18))
        a, b = _both(lat, DIRS[:4], 0.9, 2.5, 1, 3)
        assert np.array_equal(a, b)
        w = lat.wilson_loop(1, 2, 1, 3)
        lat.set_wilson_method("auto")
        assert np.array_equal(w, lat.wilson_loop(1, 2, 1, 3))
