"""Fundamental loops as correlations of the space lines' elements along time
(gc_wilson_corr.cu), against the exact product of links: T ranges that start
anywhere in a 16-byte vector, one and several windows of T, time extents that a
vector does not divide, blocks of columns past the lattice, and slabs.

Tolerances: FP64, reassociated products of at most 2 (R + T) links and sums of
loops of order one: 1e-12; mixed, FP32 links: 1e-6 (the form's accuracy bar).
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "mixed": 1e-6}


def _check(precision, nc, dims, rng, t_starts=None):
    with Lattice(dims, nc, precision) as lat:
        lat.upload(generate_config(dims, nc, 0.25, 47, 0))
        lat.hyp(1.0, 0.75, 0.6, 1)
        out = []
        for method in ("auto", "exact"):
            lat.set_wilson_method(method)
            out.append(lat.wilson_loop(*rng) if t_starts is None
                       else lat.wilson_loop_tslab(t_starts, *rng))
            if method == "auto":
                assert lat.wilson_method_used() == "gauge"
        a, b = out
        assert np.max(abs(a - b)) <= TOL[precision] * np.max(abs(b))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("dims,rng", [
    ((8, 3, 2, 40), (1, 2, 1, 12)),
    ((8, 3, 2, 41), (1, 9, 2, 11)),   # R past the extent
    ((5, 3, 3, 42), (2, 3, 3, 8)),
    ((9, 5, 2, 43), (1, 2, 4, 12)),
    ((3, 2, 3, 90), (1, 2, 12, 12)),
    ((16, 2, 3, 48), (1, 2, 1, 24)),
    ((16, 2, 3, 51), (1, 2, 1, 25)),
    ((3, 3, 3, 65), (1, 2, 5, 32)),
])
def test_whole_lattice(precision, nc, dims, rng):
    _check(precision, nc, dims, rng)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc", [2, 3])
@pytest.mark.parametrize("dims,t_starts,rng", [
    ((8, 3, 2, 40), 29, (1, 2, 1, 11)),
    ((5, 3, 2, 50), 14, (1, 2, 2, 30)),
])
def test_start_slices_of_a_slab(precision, nc, dims, t_starts, rng):
    _check(precision, nc, dims, rng, t_starts)
