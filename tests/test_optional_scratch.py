"""Device memory that only an optional form wants. Handles whose memory comes
from a pool of limited size: where the gauge form's scratch does not fit, the
GEVP, off-axis and spatial loops are the exact product's; where it does fit and
HYP or a download later needs the room, it is given back. (The limit is the
pool's own, set on the host; nothing exhausts the device.)
"""
from __future__ import annotations

import ctypes

import numpy as np
import pytest

from general_code_b200 import Lattice, _lib, generate_config
from general_code_b200._lib import check, dims_arg, lib

pytestmark = pytest.mark.gpu
DIMS = (24, 24, 24, 16)  # a field of FP64 SU(3) links: 31.9 MB
FIELD = 144 * 24 ** 3 * 16


@pytest.fixture
def pool():
    """limit(bytes): handles created from then on take their memory from a pool
    of that size, on a stream of their own."""
    rt = pytest.importorskip("cuda.bindings.runtime")
    made, streams = [], []

    def call(r):
        assert r[0] == rt.cudaError_t.cudaSuccess, r[0]
        return r[1] if len(r) > 1 else None

    call(rt.cudaSetDevice(0))
    call(rt.cudaFree(0))

    def limit(size):
        props = rt.cudaMemPoolProps()
        props.allocType = rt.cudaMemAllocationType.cudaMemAllocationTypePinned
        props.location.type = rt.cudaMemLocationType.cudaMemLocationTypeDevice
        props.location.id = 0
        props.maxSize = size
        made.append(call(rt.cudaMemPoolCreate(props)))
        call(rt.cudaDeviceSetMemPool(0, made[-1]))
        streams.append(call(rt.cudaStreamCreate()))
        return int(streams[-1])

    yield limit
    call(rt.cudaDeviceSetMemPool(0, call(rt.cudaDeviceGetDefaultMemPool(0))))
    for s in streams:
        call(rt.cudaStreamSynchronize(s))
        call(rt.cudaStreamDestroy(s))
    for p in made:
        call(rt.cudaMemPoolDestroy(p))


def _handle(stream):
    lat = Lattice.__new__(Lattice)
    lat.dims, lat.nc, lat.precision, lat._h = DIMS, 3, "fp64", ctypes.c_void_p()
    check(lib().gc_lattice_create_on_stream(dims_arg(DIMS), 3, _lib.GC_PREC_FP64,
                                            ctypes.c_void_p(stream), ctypes.byref(lat._h)))
    return lat


def _calls(lat, other):
    spatial = lat.wilson_spatial_3d(1, 2, 1, 2, 0.5, 0, 1, 1)
    return [np.array([spatial[k] for k in sorted(spatial)]),
            np.array([x[0] for x in lat.wilson_offaxis([[1, 1, 0], [2, 1, 0]], 0.9, 5.0, 1, 3)]),
            np.array(lat.wilson_gevp(other, 1, 4, 1, 4))]


@pytest.fixture(scope="module")
def want():
    links = generate_config(DIMS, 3, 0.25, 4, 0)
    with Lattice(DIMS, 3, "fp64") as lat, Lattice(DIMS, 3, "fp64") as other:
        lat.upload(links)
        other.copy_from(lat)
        other.ape(0.5, 1)
        lat.set_wilson_method("exact")
        exact = _calls(lat, other)
        second = other.download()
        lat.hyp(1.0, 0.75, 0.6, 1)
        return links, second, exact, lat.download()


# Fields that a handle holds: 8 of links, 4 of host staging (upload, download), 6
# of the spatial loops, 15 of HYP; the gauge scratch takes 6.4 (spatial), 4.6
# (off-axis) and 8.6 (GEVP, T <= 4).


def test_no_room_for_the_scratch(pool, want):
    links, second, exact, _ = want
    with Lattice(DIMS, 3, "fp64") as first, Lattice(DIMS, 3, "fp64") as other:
        first.upload(links)
        other.upload(second)
        first.synchronize()
        with _handle(pool(16 * FIELD)) as lat:
            lat.copy_from(first)
            for got, x in zip(_calls(lat, other), exact):
                assert np.array_equal(got, x)


@pytest.mark.parametrize("fields", [19, 25])
def test_scratch_makes_room_for_a_download(pool, want, fields):
    _, second, _, _ = want
    with Lattice(DIMS, 3, "fp64") as other:
        other.upload(second)
        other.synchronize()
        with _handle(pool(fields * FIELD)) as lat:
            lat.copy_from(other)
            lat.wilson_gevp(other, 1, 4, 1, 4)
            assert lat.wilson_method_used() == "gauge"
            assert np.array_equal(lat.download(), second)


def test_scratch_makes_room_for_hyp(pool, want):
    links, second, exact, hyp = want
    with Lattice(DIMS, 3, "fp64") as other:
        other.upload(second)
        other.synchronize()
        with _handle(pool(36 * FIELD)) as lat:
            lat.upload(links)
            for got, x in zip(_calls(lat, other), exact):
                assert np.max(abs(got - x)) <= 1e-12
            lat.hyp(1.0, 0.75, 0.6, 1)
            assert np.array_equal(lat.download(), hyp)
