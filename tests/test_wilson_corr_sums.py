"""FP32 sums of the correlation form (gc_wilson_corr.cu) over long time extents.
On links of one constant phase every product of a sum is the same number, so
that all roundings add up: W(1, T) = (c^2 + s^2) for SU(2), (2 (c^2 + s^2) + 1)/3
for SU(3), with c and s the FP32 cosine and sine of the phase.

Tolerance, with u = 2^-24: a chain of n equal terms is off by at most
(n + 1)/2 u; eight products, eight such groups, two sums over lanes: 11 u; the
rebuilt third row of an SU(3) line 2 u more.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice

pytestmark = pytest.mark.gpu


def _links(dims, nc, c, s):
    v = int(np.prod(dims))
    u = np.zeros((v, 4, 4 if nc == 2 else 18))
    if nc == 2:
        u[:, :, 0] = 1.0
        u[:, :3, 0], u[:, :3, 3] = c, s
    else:
        u[:, :, 0] = u[:, :, 8] = u[:, :, 16] = 1.0
        u[:, :3, 0], u[:, :3, 1], u[:, :3, 8], u[:, :3, 9] = c, s, c, -s
    return u.reshape(4 * v, -1)


@pytest.mark.parametrize("nc,lt,tmax", [(2, 240, 20), (2, 67, 24), (3, 240, 12), (3, 65, 16)])
def test_constant_phase(nc, lt, tmax):
    dims = (4, 4, 4, lt)
    with Lattice(dims, nc, "mixed") as lat:
        for angle in np.linspace(0.1, 1.5, 12):
            c, s = np.float32(np.cos(angle)), np.float32(np.sin(angle))
            norm = float(c) ** 2 + float(s) ** 2
            lat.upload(_links(dims, nc, c, s))
            w = lat.wilson_loop(1, 1, 1, tmax)
            assert lat.wilson_method_used() == "gauge"
            want = norm if nc == 2 else (2 * norm + 1) / 3
            assert np.max(abs(w - want)) <= 13 * 2.0 ** -24
