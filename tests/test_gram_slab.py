"""Time slabs whose lattice has more slices than the slab's loops touch, by the
FP64 matrix products (gc_wilson_gram.cu), against the exact product of links.

Tolerance: FP64, reassociated products of at most 2 (R + T) links and sums of
loops of order one: 1e-12.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("dims,t_starts,rng", [
    ((5, 3, 2, 50), 14, (1, 2, 2, 30)),
    ((4, 3, 3, 64), 3, (1, 2, 1, 13)),
    ((4, 3, 3, 40), 8, (1, 2, 13, 16)),
])
def test_slab_of_a_long_lattice(nc, dims, t_starts, rng):
    with Lattice(dims, nc, "fp64") as lat:
        lat.upload(generate_config(dims, nc, 0.25, 53, 0))
        lat.hyp(1.0, 0.75, 0.6, 1)
        got = lat.wilson_loop_tslab(t_starts, *rng)
        lat.set_wilson_method("exact")
        want = lat.wilson_loop_tslab(t_starts, *rng)
        assert np.max(abs(got - want)) <= 1e-12 * np.max(abs(want))
