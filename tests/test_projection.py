"""SU(3) projection on chosen matrices: an APE step with alpha = 0 projects the
links themselves, so links A = V diag(s) W phase with chosen singular values and
determinant phase exercise the polynomial form, the reference's steps outside
its region, and the region's edge. Oracle: the six steps in extended precision
(numpy longdouble).

Tolerances. FP64: where the singular values are at least 0.3 of their mean a
few roundings and the 4e-15 by which six steps may miss the limit at the
region's edge: 2e-14; elsewhere rounding grows with the inverse of the smallest
(0.05 at least) over the six steps: 1e-12. Mixed (links rounded to FP32, their
third row rebuilt): the FP32 rounding 6e-8 of the input and of a step's sums,
over the smallest pair sum of singular values: 2e-6.
"""
from __future__ import annotations

import numpy as np
import pytest

from general_code_b200 import Lattice

pytestmark = pytest.mark.gpu
DIMS = (4, 4, 2, 3)  # 96 sites, 288 spatial links


def _haar(rng, n):
    z = rng.normal(size=(n, 3, 3)) + 1j * rng.normal(size=(n, 3, 3))
    q, r = np.linalg.qr(z)
    q = q * (np.diagonal(r, axis1=1, axis2=2) / abs(np.diagonal(r, axis1=1, axis2=2)))[:, None]
    return q / np.linalg.det(q)[:, None, None] ** (1 / 3)


def _six_steps(a):
    a = a.astype(np.clongdouble)
    for _ in range(6):
        a = 1.5 * a - 0.5 * (a @ a.conj().swapaxes(1, 2)) @ a
        det = (a[:, 0] * np.cross(a[:, 1], a[:, 2])).sum(-1)
        a = (1 - (det - 1) / 3)[:, None, None] * a
    return a


def _host(a):
    """(288, 3, 3) spatial links -> the host array (the time links are 1)."""
    n = a.shape[0] // 3
    u = np.zeros((n, 4, 3, 3), dtype=complex)
    u[:, :3] = a.reshape(n, 3, 3, 3)
    u[:, 3] = np.eye(3)
    return np.ascontiguousarray(np.stack([u.real, u.imag], -1).reshape(4 * n, 18))


def _spatial(links):
    m = np.asarray(links).reshape(-1, 4, 3, 3, 2)[:, :3]
    return (m[..., 0] + 1j * m[..., 1]).reshape(-1, 3, 3)


# name, (singular values over their rms, rms, phase) samplers, FP64 tolerance
CASES = {
    "smeared": (0.02, (0.95, 1.0), 0.02, 2e-14),
    "ordinary": (0.35, (0.55, 1.0), 0.5, 2e-14),
    "rough": (1.0, (0.4, 1.05), 0.9, 1e-12),
}


def _matrices(name, seed):
    spread, rms, phase, tol = CASES[name]
    rng = np.random.default_rng(seed)
    n = 3 * int(np.prod(DIMS))
    s = np.clip(1 + spread * rng.uniform(-0.95, 0.95, (n, 3)), 0.05, None)
    s *= (rng.uniform(*rms, n) / np.sqrt((s ** 2).mean(1)))[:, None]
    th = rng.uniform(-phase, phase, n)
    a = _haar(rng, n) @ (s[:, :, None] * _haar(rng, n)) * np.exp(1j * th / 3)[:, None, None]
    return a, tol


@pytest.mark.parametrize("name", sorted(CASES))
def test_fp64_projection(name):
    a, tol = _matrices(name, 11)
    with Lattice(DIMS, 3, "fp64") as lat:
        lat.upload(_host(a))
        lat.ape(0.0, 1)
        got = _spatial(lat.download())
    assert np.max(abs(got - _six_steps(a))) <= tol


@pytest.mark.parametrize("name", ["smeared", "ordinary"])
def test_mixed_projection(name):
    """The 12-real links: matrices whose third row is conj(row0 x row1)."""
    a, _ = _matrices(name, 12)
    a = (a.real.astype(np.float32) + 1j * a.imag.astype(np.float32)).astype(complex)
    a[:, 2] = np.cross(a[:, 0], a[:, 1]).conj()
    with Lattice(DIMS, 3, "mixed") as lat:
        lat.upload(_host(a))
        lat.ape(0.0, 1)
        got = _spatial(lat.download())
    assert np.max(abs(got - _six_steps(a))) <= 2e-6


def test_scalar_matrices_and_the_region_edge():
    """Multiples of one SU(3) matrix from rms 0.3 to 1.2 (the edges 0.5 and
    1.0005 of the polynomial form's region between them) and unit links."""
    n = 3 * int(np.prod(DIMS))
    a = _haar(np.random.default_rng(3), 1) * np.linspace(0.3, 1.2, n)[:, None, None]
    a[0] = np.eye(3)
    with Lattice(DIMS, 3, "fp64") as lat:
        lat.upload(_host(a))
        lat.ape(0.0, 1)
        got = _spatial(lat.download())
    assert np.max(abs(got - _six_steps(a))) <= 2e-14
