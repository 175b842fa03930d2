"""The branch-free reciprocal, quotient, square root and quadrant over the
ranges that their callers admit, bit for bit against numpy's f32 operations
(IEEE 754, rounded to nearest): every mantissa at the ends and in the middle
of the exponents, quotients next to midpoints of two numbers, and the
neighbourhood of every multiple of pi/2 below 1e7."""
from __future__ import annotations

import numpy as np
import pytest

F = np.float32
RCP, DIV, SQRT, QUADRANT = 9, 10, 11, 12
MANTISSAS = np.arange(1 << 23, dtype=np.uint32)


def at(exponent: int) -> np.ndarray:
    """Every f32 in [2^exponent, 2^(exponent + 1))."""
    return (MANTISSAS | np.uint32((exponent + 127) << 23)).view(F)


def differ(got: np.ndarray, want: np.ndarray) -> int:
    return int((got.view(np.uint32) != want.view(np.uint32)).sum())


@pytest.mark.gpu
@pytest.mark.parametrize("exponent", [-64, -63, -39, -25, -2, -1, 0, 1, 24, 40, 62])
def test_reciprocals_of_every_mantissa(device, exponent):
    """Half extents down to 2^-25, a direction's component (at least 2^-40)
    over one of them, and twice the roots of up to 1e23."""
    x = at(exponent)
    assert differ(device.math(RCP, x), F(1.0) / x) == 0
    assert differ(device.math(RCP, -x[::16]), F(1.0) / -x[::16]) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("exponent", [-77, -76, -75, -2, -1, 0, 1, 74, 75, 76])
def test_roots_of_every_mantissa(device, exponent):
    x = at(exponent)
    x = x[(x > F(1e-23)) & (x < F(1e23))]
    assert len(x) > 0 and differ(device.math(SQRT, x), np.sqrt(x)) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("seed", range(4))
def test_quotients(device, seed):
    """A distance from a box's bound over its half extent (2^-25 to 2^24): all
    exponents, of the quotient from 2^-40 to 2^24, half of the quotients next
    to a midpoint."""
    rng = np.random.default_rng(seed)
    n = 1 << 22
    d = (rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-25, 25, n)).astype(F)
    q = rng.uniform(1.0, 2.0, n).astype(F).astype(np.float64)
    mid = (q + 2.0 ** -24) * 2.0 ** rng.integers(-40, 25, n)
    near = (d.astype(np.float64) * mid * rng.choice([-1.0, 1.0], n)).astype(F)
    far = (rng.uniform(-2.0, 2.0, n) * 2.0 ** rng.integers(-64, 25, n)).astype(F)
    for x, y in ((near, d), (far, d)):
        assert differ(device.math(DIV, x, y), x / y) == 0
    # of either zero: zero, as a number (its sign may be another)
    assert np.array_equal(device.math(DIV, np.array([0.0, -0.0], F), d[:2]), np.zeros(2, F))


@pytest.mark.gpu
def test_quadrants(device):
    half = F(1.5707963267948966)
    k = np.arange(-6366197, 6366198, dtype=np.float64)
    mult = (k * np.float64(half)).astype(F)
    mult = mult[np.abs(mult) < F(1e7)]
    rng = np.random.default_rng(0)
    some = (rng.uniform(-2.0, 2.0, 1 << 22) * 2.0 ** rng.integers(-149, 23, 1 << 22)).astype(F)
    edge = np.array([0.0, -0.0, 1e-45, -1e-45, 0.5, -0.5, np.nextafter(F(0.5), F(0)), np.nextafter(F(-0.5), F(0)),
                     np.nextafter(F(1e7), F(0)), np.nextafter(F(-1e7), F(0))], F)
    for x in (mult, np.nextafter(mult, F(np.inf)), np.nextafter(mult, F(-np.inf)), some, edge):
        x = x[np.abs(x) < F(1e7)]
        got, want = device.math(QUADRANT, x), np.floor(x / half)
        assert np.array_equal(got, want)
