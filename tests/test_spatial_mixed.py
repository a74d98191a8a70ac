"""Mixed SU(3) spatial loops on a rough field, where planar sums do not project
onto the group in six steps and leave links off it: the loops in the gauge of the
third axis carry all 18 reals of a link, and agree with the exact product to its
1e-6 all the same. One link off the group, stored by an upload, does the same,
and along the third axis sends its plane to the exact product.

(1e-6: FP32 links and lines of at most 2 x 3 + 2 x 3 products, values of order
one; the accuracy bar of the mixed form.)
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu


def _tables(dims, links, alpha, steps):
    with Lattice(dims, 3, "mixed") as lat:
        lat.upload(links)
        out = []
        for method in ("auto", "exact"):
            lat.set_wilson_method(method)
            w = lat.wilson_spatial_3d(1, 3, 1, 3, alpha, 0, steps, 1)
            out.append(np.array([w[k] for k in sorted(w)]))
    return out


@pytest.mark.parametrize("dims", [(8, 8, 8, 6), (6, 9, 7, 5), (24, 24, 24, 3)])
def test_rough_field(dims):
    auto, exact = _tables(dims, generate_config(dims, 3, 0.6, 5, 0), 0.5, 2)
    assert np.max(abs(auto - exact)) <= 1e-6
    assert np.any(auto != exact)  # (the exact product would give the same bits)


@pytest.mark.parametrize("mu", [0, 1, 2])
def test_one_link_off_the_group(mu):
    dims = (8, 6, 10, 4)
    links = generate_config(dims, 3, 0.25, 6, 0).reshape(-1, 4, 18)
    links[333, mu] *= 1.1
    auto, exact = _tables(dims, links.reshape(-1, 18), 0.5, 1)
    assert np.max(abs(auto - exact)) <= 1e-6
    assert np.any(auto != exact)
