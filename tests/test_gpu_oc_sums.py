"""Sums in element order of the OC update, taken in parallel (OcOptimizer.cs:28-33, :134-175): whole runs of terms as
one integer step while the running sum stays in a binade, term by term where it leaves it. Each input puts the
volume target on the sequential V(lambda) itself with a tolerance of zero, so the bisection stops at its first trial
only if both the total of s and V(lambda) have the bits of the sequential sums.
"""
import numpy as np
import pytest

from mycel_b200 import api

pytestmark = pytest.mark.gpu


def _s(kind, n, rng):
    if kind == "even":
        return 0.5 + rng.random(n)
    if kind == "wide":
        return 10.0 ** rng.uniform(-12.0, 8.0, n)
    if kind == "zeros":  # runs that add nothing, and -0
        s = np.where(rng.random(n) < 0.9, np.where(rng.random(n) < 0.5, 0.0, -0.0), rng.random(n))
        s[-1] = 0.75
        return s
    if kind == "signs":  # no step holds where a term is negative
        return np.where(rng.random(n) < 0.01, -1.0, 1.0) * rng.random(n)
    if kind == "huge":   # outside the range of the steps
        return 1e290 * (0.5 + rng.random(n))
    s = 0.5 * rng.integers(0, 8, n)  # "ties": halves of the unit of a sum that starts at 2^52
    s[0] = 2.0 ** 52
    return s


def _target(s, c):
    # f with fl(f * sum(s)) == sum(s c), both in element order
    ts, v = float(np.cumsum(s)[-1]), float(np.cumsum(s * c)[-1])
    f = v / ts
    for _ in range(8):
        if f * ts == v:
            return f
        f = float(np.nextafter(f, np.inf if f * ts < v else -np.inf))
    return None


@pytest.mark.parametrize("kind", ["even", "wide", "zeros", "signs", "huge", "ties"])
# a piece (128), a tile (1024), the line between one block and the grid (2048), chunks of 256 and longer ones,
# chunks of more than a tile
@pytest.mark.parametrize("n", [1, 127, 129, 1024, 1025, 2048, 2049, 2304, 75_777, 400_003])
def test_sums_have_the_sequential_bits(oracle, ctx, kind, n):
    for seed in range(20):
        rng = np.random.default_rng(1000 * seed + n % 97)
        s = _s(kind, n, rng)
        pas = (rng.random(n) < 0.5).astype(np.uint8)
        rho = np.full(n, 0.5)
        dc = np.zeros(n)  # every free element goes to rho - move, whatever lambda is
        f = _target(s, np.where(pas == 1, 1.0, 0.25))
        if f is not None and np.isfinite(f):
            break
    assert f is not None
    ol = oracle.oc_update(rho, dc, s, pas, f, 0.25, 1e-3, 1.0, 60, 0.0)
    gl = api.oc_update(rho, dc, s, pas, f, 0.25, 1e-3, 1.0, 60, 0.0, ctx=ctx)
    if f > 0.0 and kind != "signs":
        assert ol[1] == 1.0
    assert gl[1] == ol[1]
    assert np.array_equal(gl[0], ol[0])
