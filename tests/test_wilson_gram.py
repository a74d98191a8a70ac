"""Fundamental loops by FP64 matrix products of the transformed space lines
(gc_wilson_gram.cu) and the one-column kernels' ragged time extents, against the
exact product of links.

Tolerances: FP64, reassociated products of at most 2 (R + T) links and sums of
loops of order one: 1e-12; mixed, FP32 links: 1e-6 (the form's accuracy bar).
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice, generate_config

pytestmark = pytest.mark.gpu
TOL = {"fp64": 1e-12, "mixed": 1e-6}


def _both(lat, *rng, t_starts=None):
    out = []
    for method in ("auto", "exact"):
        lat.set_wilson_method(method)
        out.append(lat.wilson_loop(*rng) if t_starts is None
                   else lat.wilson_loop_tslab(t_starts, *rng))
    lat.set_wilson_method("auto")
    return out


def _smeared(dims, nc, precision):
    lat = Lattice(dims, nc, precision)
    lat.upload(generate_config(dims, nc, 0.25, 41, 0))
    lat.hyp(1.0, 0.75, 0.6, 1)
    return lat


# time extents around multiples of the 8-slice tiles and of four starts; T up to
# Lt/2, T ranges that start late, one, four and more tiles, several passes over
# the end tiles, column blocks past the lattice
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,dims,rng", [
    (3, (4, 3, 5, 8), (1, 3, 1, 4)),
    (3, (3, 2, 3, 9), (2, 4, 2, 4)),
    (3, (5, 4, 2, 15), (1, 2, 1, 7)),
    (3, (3, 3, 3, 28), (1, 3, 1, 14)),
    (3, (2, 3, 4, 33), (1, 2, 9, 16)),
    (3, (2, 2, 3, 70), (1, 2, 1, 35)),
    (3, (2, 2, 2, 140), (1, 1, 60, 70)),
    (3, (3, 3, 3, 2), (1, 2, 1, 1)),
    (2, (7, 3, 5, 24), (1, 4, 1, 12)),
    (2, (3, 5, 3, 27), (2, 3, 1, 13)),
    (2, (4, 2, 3, 50), (1, 2, 3, 25)),
    (2, (2, 2, 3, 129), (1, 1, 1, 64)),
    (2, (5, 3, 3, 5), (1, 2, 1, 2)),
    (2, (9, 2, 3, 6), (1, 2, 2, 3)),
])
def test_whole_lattice(precision, nc, dims, rng):
    with _smeared(dims, nc, precision) as lat:
        a, b = _both(lat, *rng)
        lat.wilson_loop(*rng)
        assert lat.wilson_method_used() == "gauge"
        assert np.max(abs(a - b)) <= TOL[precision] * np.max(abs(b))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,dims,t_starts,rng", [
    (3, (3, 4, 3, 24), 9, (1, 2, 1, 15)),
    (3, (3, 2, 3, 20), 17, (1, 2, 2, 3)),
    (2, (4, 3, 3, 30), 13, (1, 2, 1, 17)),
    (2, (4, 3, 3, 11), 6, (1, 2, 1, 5)),
])
def test_start_slices_of_a_slab(precision, nc, dims, t_starts, rng):
    with _smeared(dims, nc, precision) as lat:
        a, b = _both(lat, *rng, t_starts=t_starts)
        assert np.max(abs(a - b)) <= TOL[precision] * np.max(abs(b))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nc,dims,rng", [
    (3, (4, 3, 5, 8), (1, 7, 1, 4)),
    (3, (3, 2, 5, 13), (2, 6, 2, 6)),
    (3, (3, 3, 2, 42), (1, 2, 1, 21)),
    (2, (5, 4, 3, 10), (1, 5, 1, 5)),
    (2, (3, 4, 3, 36), (1, 2, 5, 18)),
    (2, (3, 4, 3, 9), (1, 4, 1, 7)),  # T > Lt/2: the exact product in both
    (3, (4, 3, 5, 8), (1, 2, 1, 2)),  # few loops: the exact product in both
])
def test_two_configurations(precision, nc, dims, rng):
    with _smeared(dims, nc, precision) as a, Lattice(dims, nc, precision) as b:
        b.copy_from(a)
        b.ape(0.5, 3)
        got = a.wilson_gevp(b, *rng)
        same = a.wilson_gevp(a, *rng)
        table = a.wilson_loop(*rng)
        a.set_wilson_method("exact")
        want = a.wilson_gevp(b, *rng)
        top = np.max(abs(want))
        assert np.max(abs(got - want)) <= TOL[precision] * top
        assert np.max(abs(same - table)) <= TOL[precision] * top


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_second_configuration_off_the_group(precision):
    """The second configuration's links need be in SU(3) only where they are
    stored as 12 reals; the first one's time links always."""
    dims = (4, 3, 4, 6)
    links = generate_config(dims, 3, 0.25, 43, 0)
    bad = links.reshape(-1, 4, 18).copy()
    bad[11, 2] *= 1.001
    with Lattice(dims, 3, precision) as a, Lattice(dims, 3, precision) as b:
        a.upload(links)
        b.upload(bad.reshape(-1, 18))
        got = a.wilson_gevp(b, 1, 9, 1, 3)
        assert a.wilson_method_used() == ("gauge" if precision == "fp64" else "exact")
        a.set_wilson_method("exact")
        want = a.wilson_gevp(b, 1, 9, 1, 3)
        assert np.max(abs(got - want)) <= TOL["fp64"] * np.max(abs(want))
