"""The temporal-gauge form's unitarity check in FP64: single links off by more
than the mean bound stay in the form (the loops' averages agree with the exact
product's), a mean above it or one link far off takes the exact product.

Tolerance: reassociated products of at most 2 (R + T) links and sums of loops
of order one, 1e-12; a link off by 5e-13 enters at most that many of the
loops' factors once each.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu
DIMS = {2: (5, 7, 3, 24), 3: (8, 4, 4, 10)}


def _run(nc, links, want):
    rng = (1, 3, 1, 5)
    with Lattice(DIMS[nc], nc, "fp64") as lat:
        lat.upload(links)
        w = lat.wilson_loop(*rng)
        assert lat.wilson_method_used() == want
        lat.set_wilson_method("exact")
        e = lat.wilson_loop(*rng)
        assert lat.wilson_method_used() == "exact"
    assert np.max(abs(w - e)) <= 1e-12 or want == "exact" and np.array_equal(w, e, equal_nan=True)


def _links(nc):
    return generate_config(DIMS[nc], nc, 0.25, 71, 0)


@pytest.mark.parametrize("nc", [2, 3])
def test_single_links_above_the_mean_bound(nc):
    links = _links(nc)
    temporal = links[3::4]
    temporal[::211] *= 1 + 2.5e-13  # |U U^dag - 1| = 5e-13, less than one link in 200
    _run(nc, links, "gauge")


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("step,scale", [(1, 1 + 2e-14), (97, 1 + 1e-12), (97, float("nan"))])
def test_mean_or_one_link_off(nc, step, scale):
    links = _links(nc)
    links[3::4][::step] *= scale
    _run(nc, links, "exact")
