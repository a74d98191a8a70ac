"""The polynomial SU(3) projection near the edge of its region: matrices with one
singular value up to 1.54 times the rms and the other two equal, where the
inverse square root's starting series is nearly zero. The functions of the
header are compiled for the host in both precisions; the GPU runs the FP64 form
as an APE step with alpha = 0.

Oracle: the unitary factor V W of A = V diag(s) W, which six steps reach to
4e-15 inside the region. Tolerances: FP64 a few roundings over the smallest pair
sum of singular values (1.1) and that 4e-15, 2e-14; FP32 a few dozen roundings
of 6e-8 (dot products of six and nine terms, twice), 4e-6. A matrix that the
form refuses goes to the matrix steps, which the GPU test covers.
"""
from __future__ import annotations

import ctypes
import subprocess
from pathlib import Path

import numpy as np
import pytest

from test_projection import DIMS, _haar, _host, _six_steps, _spatial
from general_code_b200 import Lattice

CSRC = Path(__file__).resolve().parents[1] / "general_code_b200" / "csrc"

SOURCE = """
#include "gc_algebra.cuh"
using namespace gc;
template <class T> static int polar(const double *in, double *out) {
  SU3<T> A, U;
  for (int k = 0; k < 9; k++)
    A.e[k / 3][k % 3] = {T(in[2 * k]), T(in[2 * k + 1])};
  if (!polar_su3(A, U))
    return 0;
  for (int k = 0; k < 9; k++) {
    out[2 * k] = U.e[k / 3][k % 3].re;
    out[2 * k + 1] = U.e[k / 3][k % 3].im;
  }
  return 1;
}
extern "C" int polar64(const double *in, double *out) { return polar<double>(in, out); }
extern "C" int polar32(const double *in, double *out) { return polar<float>(in, out); }
"""


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("algebra")
    (d / "polar.cpp").write_text(SOURCE)
    lib = d / "libpolar.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-I", str(CSRC),
                    str(d / "polar.cpp"), "-o", str(lib)], check=True)
    return ctypes.CDLL(str(lib))


def _edge(n, seed):
    """n matrices V diag(s) W and V W: s = (x, o, o) of rms 1, x = 1.40 ... 1.54."""
    rng = np.random.default_rng(seed)
    x = np.linspace(1.40, 1.54, n)
    o = np.sqrt((3 - x * x) / 2)
    v, w = _haar(rng, n), _haar(rng, n)
    v[: n // 2] = w[: n // 2] = np.eye(3)
    return v @ (np.stack([o, x, o], -1)[:, :, None] * w), v @ w


@pytest.mark.parametrize("bits,tol", [(64, 2e-14), (32, 4e-6)])
def test_accepted_matrices_have_converged(host, bits, tol):
    a, limit = _edge(564, 5)
    polar = getattr(host, f"polar{bits}")
    out = np.empty(18)
    ptr = ctypes.POINTER(ctypes.c_double)
    accepted = 0
    for m, u in zip(a, limit):
        buf = np.ascontiguousarray(np.stack([m.real, m.imag], -1).ravel())
        if polar(buf.ctypes.data_as(ptr), out.ctypes.data_as(ptr)):
            got = (out[0::2] + 1j * out[1::2]).reshape(3, 3)
            assert np.max(abs(got - u)) <= tol
            accepted += 1
    assert accepted > 400  # (the region's interior keeps the form)


@pytest.mark.gpu
def test_projection_near_the_edge():
    n = 3 * int(np.prod(DIMS))
    a, _ = _edge(n, 6)
    with Lattice(DIMS, 3, "fp64") as lat:
        lat.upload(_host(a))
        lat.ape(0.0, 1)
        got = _spatial(lat.download())
    assert np.max(abs(got - _six_steps(a))) <= 2e-14
