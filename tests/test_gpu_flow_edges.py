"""The flow kernels at the edges of their tiles, and the exponential on both sides of its series rule.

Lattices whose half-volume is below, at and just past multiples of the 32-site tiles and of the block
shapes, every storage, against the oracle's RK3 steps.
"""
import math

import numpy as np
import pytest

from conftest import rel_err

pytestmark = pytest.mark.gpu

# half-sites: 8, 24, 120, 128, 648 (20.25 tiles), 1050 (32.8 tiles)
LATTICES = [(2, 2, 2, 2), (6, 2, 2, 4), (10, 6, 2, 2), (4, 4, 4, 4), (6, 6, 6, 6), (14, 10, 6, 2)]


@pytest.mark.parametrize("L", LATTICES)
@pytest.mark.parametrize("prec,store", [(64, 0), (64, 1), (32, 0), (32, 1)])
def test_flow_steps_at_tile_edges(gpu, orc, L, prec, store):
    """Two RK3 steps, and the measured flow's links.  FP64: the 1e-12 of the parity tests.  FP32: a
    link's entries (at most 1) pass through 6 stages of about 60 roundings of 2^-24 each in the worst
    direction, 6 * 60 * 6e-8 = 2e-5."""
    U = orc.hot_start(L, 31)
    f = gpu.GaugeField(L, 64, 0)
    f.upload(U)
    ref = orc.flow_rk3(U, L, 0.02, 2)
    fl = gpu.GradientFlow(f, 0.02, prec=prec, store=store)
    fl.rk3_step(2)
    tol = 1e-12 if prec == 64 else 2e-5
    plain = fl.field.download()
    assert rel_err(plain, ref) < tol
    fl.measure(f, 3, 1)
    assert np.array_equal(fl.field.download(), plain)  # stage 1 with the halves writes the same links


@pytest.mark.parametrize("prec,tol", [(64, 1e-14), (32, 1e-6)])
def test_exp_on_both_sides_of_the_series_rule(gpu, orc, prec, tol):
    """The exponential takes fewer terms for t = -Re Tr(X^2)/2 <= 1/32: scales that put t far below, at
    both sides of and far above the line.  FP64: the bound of the parity test.  FP32: about ten roundings
    of 6e-8 on entries of at most 1."""
    rng = np.random.default_rng(5)
    Z = np.stack([orc.proj_lie_su3(rng.normal(size=(3, 3)) + 1j * rng.normal(size=(3, 3))) for _ in range(48)])
    t = -0.5 * np.einsum("nij,nji->n", Z, Z).real
    for want in (0.0, 1e-6, 0.03125 * (1 - 1e-9), 0.03125 * (1 + 1e-9), 0.5, 2.0):
        X = Z * np.sqrt(want / t)[:, None, None]
        ref = np.stack([orc.exp_su3(x, 1.0) for x in X])
        assert np.max(np.abs(gpu.exp_su3(X, 1.0, prec) - ref)) < tol, want


def test_exp_of_a_matrix_off_the_algebra(gpu, orc):
    """The diagnostic exponential takes any matrix.  One with a part of 0.1 outside the algebra gets the
    Cayley-Hamilton form of its own entries: X^2 from the upper triangle of the full product, t from its
    trace, d from the full determinant.  Some forty FP64 operations on entries of order one: 1e-14."""
    rng = np.random.default_rng(6)
    noise = rng.normal(size=(2, 16, 3, 3))
    X = np.stack([orc.proj_lie_su3(z) for z in noise[0] + 1j * noise[1]]) * 0.3
    X = X + 0.1 * (rng.normal(size=X.shape) + 1j * rng.normal(size=X.shape))
    up = np.triu(X @ X, 1)
    X2 = up + np.conj(np.swapaxes(up, 1, 2)) + np.einsum("nii->ni", (X @ X).real)[:, :, None] * np.eye(3)
    t, d = -0.5 * np.einsum("nii->n", X2).real, -np.linalg.det(X).imag
    q0, q1, q2 = (np.zeros(16, complex) for _ in range(3))
    for n in range(18, -1, -1):
        q0, q1, q2 = 1 / math.factorial(n) - 1j * d * q2, q0 - t * q2, q1
    ref = q0[:, None, None] * np.eye(3) + q1[:, None, None] * X + q2[:, None, None] * X2
    assert np.max(np.abs(gpu.exp_su3(X, 1.0) - ref)) < 1e-14
