"""The fixed-point FP64 collision (csrc/lbgb_fix64.cuh, compiled for the host)
loses nothing against the FP64 evaluation: over the whole range of populations
and omega, nodes that it takes have no larger error in any population (root mean
square) nor at most, against extended precision; nodes with a population whose
last place is finer than its unit, 2^-61, are left to the FP64 evaluation."""

import numpy as np
import pytest

from test_fix64_host import collide, lib, states  # noqa: F401

CX = np.array([0, 1, 0, -1, 0, 1, -1, -1, 1])
CY = np.array([0, 0, 1, 0, -1, 1, 1, -1, -1])
W = np.array([4 / 9] + [1 / 9] * 4 + [1 / 36] * 4)


def evaluate(f, omega, real):
    """The reference's collision of f (n, 9) in the type ``real``, sums channel by channel."""
    f, om, one = f.astype(real), real(omega), real(1)
    r = f[:, 0]
    for c in range(1, 9):
        r = r + f[:, c]
    ux = (f[:, 1] - f[:, 3] + f[:, 5] - f[:, 6] - f[:, 7] + f[:, 8]) / r
    uy = (f[:, 2] - f[:, 4] + f[:, 5] + f[:, 6] - f[:, 7] - f[:, 8]) / r
    w = np.array([4 * one / 9] + [one / 9] * 4 + [one / 36] * 4, dtype=real)
    cu = CX * ux[:, None] + CY * uy[:, None]
    feq = w * r[:, None] * (1 + 3 * cu + real(4.5) * cu * cu - real(1.5) * (ux * ux + uy * uy)[:, None])
    return f + om * (feq - f)


def small_populations(n, least, seed):
    """Populations log-uniform from ``least``, the rest population making up a density of 0.8 to 1.2."""
    rng = np.random.default_rng(seed)
    f = np.exp2(rng.uniform(np.log2(least), -3.2, (n, 9)))
    f[:, 0] = rng.uniform(0.8, 1.2, n) - f[:, 1:].sum(1)
    return f[(f[:, 0] > 2.0 ** -9) & (f[:, 0] < 1)]


STATES = {"rest": lambda: states(100000, 1e-8, 0.0, 11), "slow": lambda: states(100000, 0.01, 1e-3, 11),
          "fast": lambda: states(100000, 0.16, 0.01, 11), "rough": lambda: states(100000, 0.1, 0.6, 3),
          "small": lambda: small_populations(100000, 2.0 ** -21, 5), "least": lambda: small_populations(100000, 2.0 ** -9, 6)}


@pytest.mark.parametrize("omega", [1e-6, 1e-3, 0.01, 0.03, 0.05, 0.1, 0.2, 0.249, 0.25, 0.3, 0.6, 1.0, 1.6, 1.99])
@pytest.mark.parametrize("kind", sorted(STATES))
def test_no_population_loses_precision(lib, kind, omega):  # noqa: F811
    f = STATES[kind]()
    out, _, taken = collide(lib, f, omega)
    ok = (taken & 1) == 1
    if omega < 0.25:
        assert not ok.any()
        return
    assert ok.any()
    if kind in ("rest", "slow", "fast"):
        assert ok.all()
    f, out = f[ok], out[ok]
    exact = evaluate(f, omega, np.longdouble)
    here = np.abs((out - exact).astype(np.float64))
    fp64 = np.abs((evaluate(f, omega, np.float64) - exact).astype(np.float64))
    assert here.max() <= fp64.max()
    if len(f) > 1000:  # of "small" a dozen are taken: too few for a mean
        assert (np.sqrt((here ** 2).mean(0)) <= np.sqrt((fp64 ** 2).mean(0))).all()


def test_small_populations_are_left_alone(lib):  # noqa: F811
    f = small_populations(200000, 2.0 ** -21, 7)
    for omega in (0.0, 0.3, 1.7):
        out, _, taken = collide(lib, f, omega)
        low = (f < 2.0 ** -9).any(1)
        assert low.mean() > 0.5
        assert (taken[low] & 1 == 0).all() and np.isnan(out[low]).all()
        assert (taken[low] & 2 == 2).all()  # their velocities too
        if omega == 0.0:
            ok = taken & 1 == 1
            assert ok.any() and np.array_equal(out[ok], f[ok])
        # nor is a result below 2^-9 taken
        assert not (out[taken & 1 == 1] < 2.0 ** -9).any()
