"""The constants of a resistive wall's samples (ResistiveWall.function_transverse
.wall) against the wake function itself, for every form of the pipe radius that
the wake function takes: the array of the constructor, a plain number set
later, an array of shape ()."""
import numpy as np
import pytest

from pyheadtail_gb300.impedances import wakes as W


@pytest.mark.parametrize('radius', [0.02, np.float64(0.02), np.array(0.02),
                                    np.array([0.02]), 2])
def test_constants_give_the_wake(radius):
    src = W.CircularResistiveWall(0.05, 6911., 1e6, 1e-12)
    src.pipe_radius = radius
    wake = src.function_transverse(1.)
    dt = np.array([-1e-9, -1e-12, -1e-13, 0., 1e-10])
    coef, (num, dt_min, post) = wake.wall(0.99)
    sign = np.sign(dt + dt_min).astype(int)
    got = np.array(coef)[1 + sign] * np.sqrt(num / dt.clip(max=-dt_min)) * post
    assert np.array_equal(got, np.ravel(wake(dt, beta=0.99)))


def test_several_radii_are_left_to_the_wake_function():
    src = W.CircularResistiveWall(0.05, 6911., 1e6, 1e-12)
    src.pipe_radius = np.array([0.02, 0.03, 0.04])
    assert src.function_transverse(1.).wall(0.99) is None
