"""HYP of the FP64 SU(3) form on lattices whose sites do not fill the blocks of
levels 2 and 3 (96 sites), and on the smallest extents, against the oracle.

Tolerance: the operations of the reference in its order, the projection exact
to rounding: 1e-12.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2, 2), (2, 3, 4, 4), (3, 5, 2, 7), (5, 4, 6, 8)])
def test_matches_oracle(port, dims):
    links = generate_config(dims, 3, 0.25, 91, 0)
    want = links.copy()
    port.hyp(3, dims, want, 1.0, 0.75, 0.6, 1)
    with Lattice(dims, 3, "fp64") as lat:
        lat.upload(links)
        lat.hyp(1.0, 0.75, 0.6, 1)
        assert np.max(abs(lat.download() - want)) <= 1e-12
