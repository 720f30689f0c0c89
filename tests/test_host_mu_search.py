"""solve_mu_fixed_n's search alone, on counts given as functions of mu (no GPU)."""
import math

import pytest

from lresdft_gb300.solver import LResGPU


def _search(count, mu0, N, e_lo=-2.0, slope=None):
    s = object.__new__(LResGPU)
    s.mu, s.e_lo, s._slope, s.calls = mu0, e_lo, slope, []

    def pole_pass(x, e, want_density=True):
        s.calls.append(x)
        return None, count(x), 0.0
    s.pole_pass = pole_pass
    return s, s.solve_mu_fixed_n(N=N)


def _levels(lam, width):
    return lambda mu: sum(2 / (1 + math.exp(min(max((x - mu) / width, -700), 700))) for x in lam)


def test_a_search_leaves_nothing_for_the_next():
    count = _levels([-1.0, -0.4, -0.3, 0.5], 0.05)
    first, a = _search(count, -0.2, 6.0 - 1e-3)
    again, b = _search(count, -0.2, 6.0 - 1e-3, slope=first._slope)
    assert first._slope is None and a == b and first.calls == again.calls


@pytest.mark.parametrize("slope", [None, 1e-9, 1e-3, 1.0, 1e9])
def test_any_stored_slope_finds_the_root(slope):
    """A slope left by another crystal or state only costs passes."""
    count = _levels([-1.0, -0.4, -0.3, 0.5], 0.05)
    for mu0 in (-0.9, -0.35, 0.1, 0.8):
        s, (mu, n, _) = _search(count, mu0, 5.0, slope=slope)
        assert abs(n - 5.0) <= 1e-10 and len(s.calls) <= 40


@pytest.mark.parametrize("far", [5.0, 60.0, 4000.0])
def test_root_across_a_wide_gap(far):
    """The next level far above a filled one: the steps keep growing while the count stands still."""
    count = _levels([-1.0, far], 0.05)
    s, (mu, n, _) = _search(count, -0.9, 3.0)
    assert abs(n - 3.0) <= 1e-10 and abs(mu - far) < 1e-9 * far
