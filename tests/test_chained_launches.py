"""Chains of dependent launches: smearing steps issued back to back give the
links that the same steps give with a synchronisation after each, bit for bit
(each kernel sees all that the one before it wrote), and so does a chain on
another stream.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu


def _links(lat, raw, n, wait):
    lat.copy_from(raw)
    lat.hyp(1.0, 0.75, 0.6, 1)
    for _ in range(n):
        lat.ape(0.5, 1)
        if wait:
            lat.synchronize()
    w = lat.wilson_loop(1, 2, 1, 3)
    return lat.download(), w


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,dims", [(2, (4, 4, 4, 6)), (3, (5, 3, 4, 7)), (3, (16, 16, 16, 12)),
                                     (2, (24, 24, 24, 16))])
def test_back_to_back_steps(precision, nc, dims):
    import torch
    links = generate_config(dims, nc, 0.25, 83, 0)
    with Lattice(dims, nc, precision) as raw, Lattice(dims, nc, precision) as lat:
        raw.upload(links)
        raw.synchronize()
        want, w = _links(lat, raw, 25, True)
        for _ in range(3):
            got, v = _links(lat, raw, 25, False)
            assert np.array_equal(got, want) and np.array_equal(v, w)
        stream = torch.cuda.Stream()
        lat.set_stream(stream.cuda_stream)
        got, v = _links(lat, raw, 25, False)
        assert np.array_equal(got, want) and np.array_equal(v, w)
