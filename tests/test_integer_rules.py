"""Rules by which the step kernel leaves FP64 instructions out, restated with numpy: a cell certain from its
high words to stay wet never falls below its bathymetry plus the dry tolerance, and the middle f-wave speed's
sign and magnitude follow from the two outer speeds."""
import numpy as np
import pytest


def high(x):
    return (np.abs(x).view(np.int64) >> 32).astype(np.int64)


def sample(rng, n, lo, hi):
    x = np.ldexp(rng.uniform(1.0, 2.0, n), rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)
    x[rng.random(n) < 0.02] = 0.0
    return x


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_cell_that_stays_wet(seed):
    rng = np.random.default_rng(seed)
    n = 2_000_000
    b = sample(rng, n, -30, 60)
    d0 = np.abs(sample(rng, n, -40, 12))
    with np.errstate(all="ignore"):
        h = b + d0
        depth = h - b
        tol = np.abs(sample(rng, n, -60, 4))
        dh = sample(rng, n, -70, 12)
        near = rng.random(n) < 0.7  # changes and tolerances about as large as the rule allows
        dh[near] = (depth * rng.choice([-0.125, -0.126, -0.13], n))[near]
        tol[near] = (depth * rng.choice([0.124, 0.125, 0.126], n))[near]
        dh[rng.random(n) < 0.01] = np.nan
        h[rng.random(n) < 0.005] = np.inf
        deep = depth > tol
        room = high(depth)
        stays = deep & (np.maximum(high(dh), high(tol)) <= room - (3 << 20))
        stays &= (np.maximum(high(h), high(b)) - (45 << 20) <= room) & (room < (1900 << 20))
        assert stays.sum() > n // 20
        assert np.all((h + dh)[stays] >= (b + tol)[stays])


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_middle_speed(seed):
    rng = np.random.default_rng(seed)
    n = 1_000_000
    s1 = sample(rng, n, -500, 500)
    s2 = s1 + sample(rng, n, -20, 20)
    k = rng.random(n)
    s2 = np.where(k < 0.3, sample(rng, n, -500, 500), s2)
    s2 = np.where((k >= 0.3) & (k < 0.6), np.nextafter(-s1, rng.choice([-np.inf, 0.0, np.inf], n)), s2)
    s2 = np.where((k >= 0.6) & (k < 0.65), -s1, s2)
    ok = np.abs(s2 - s1) >= 2.0 ** -500  # the quotients' divisor is in range
    s1, s2 = s1[ok], s2[ok]
    mid = 0.5 * (s1 + s2)
    assert np.array_equal(np.sign(mid), np.where(s1 < -s2, -1.0, np.where(s1 > -s2, 1.0, 0.0)))
    assert np.all(np.abs(mid) <= np.maximum(np.abs(s1), np.abs(s2)))
