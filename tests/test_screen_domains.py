"""CPU: the screened evaluation in domains that trajectories leave on their way.

A point is decided when its trajectory keeps within the limits, so these have to cover where
the domain's trajectories go, not only the domain: around a saddle a small box of initial
points is carried far out and back.  What is decided is checked against the oracle's
arithmetic as elsewhere."""
import numpy as np
import pytest

from test_screen import check, coupled, forced, lorenz, random_boxes


@pytest.mark.parametrize("radius", [0.3, 1.0, 5.0, 10.0, 20.0])
@pytest.mark.parametrize("depth,fma", [(15, 0), (21, 1), (24, 0)])
def test_lorenz_around_the_saddle(radius, depth, fma):
    spec = lorenz(center=(0.0, 0.0, 0.0), radius=(radius,) * 3, fma=fma)
    codes, off = random_boxes(np.random.default_rng([depth, fma]), 3, depth, 1200, on_faces=0.0)
    on, share = check(spec, depth, codes, off)
    assert on and share >= 0.98


@pytest.mark.parametrize("radius", [0.1, 0.3, 0.5, 0.7, 1.0])
@pytest.mark.parametrize("depth", [12, 19, 22])
def test_forced_duffing_around_the_saddle(radius, depth):
    spec = forced(radius=(radius, radius))
    codes, off = random_boxes(np.random.default_rng(depth), 2, depth, 800, on_faces=0.0)
    on, share = check(spec, depth, codes, off)
    assert on and share >= 0.98


@pytest.mark.parametrize("h,steps", [(0.05, 40), (0.1, 20), (-0.05, 30)])
def test_coupled_duffing_over_longer_times(h, steps):
    spec = coupled(h=h, steps=steps, radius=(0.4,) * 4)
    codes, off = random_boxes(np.random.default_rng(steps), 4, 20, 800, on_faces=0.0)
    on, share = check(spec, 20, codes, off)
    assert on and share >= 0.98


def test_trajectories_that_end_far_away():
    """Backward in time most trajectories diverge: nothing is proven of those, and what is holds."""
    spec = lorenz(h=-0.02, steps=12, center=(0.0, 0.0, 27.0), radius=(25.0, 25.0, 25.0))
    codes, off = random_boxes(np.random.default_rng(1), 3, 15, 800)
    check(spec, 15, codes, off)
