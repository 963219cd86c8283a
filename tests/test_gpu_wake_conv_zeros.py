"""phk_wake, integer convolution, units whose moments or samples are all zero:
empty slices and causal wakes, with signed zeros, subnormals (which are no
zeros), infinities and NaN on the other side.

Finite cases against extended precision with the bar of the units' scales
(2^-52 of the stored turns' S max|m| max|table|); zeros times infinity or NaN
reach the targets that a floating-point loop gives them to."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from test_gpu_wake_conv import _run, _want    # noqa: E402


@pytest.mark.parametrize('S,R', [(1000, 1), (1024, 2), (300, 20)])
def test_causal_wake_and_empty_slices(S, R):
    rs = np.random.RandomState(S)
    moments = rs.normal(0, 1., (R, 3, S))
    moments[:, :, :S // 3] = 0.
    moments[:, :, -S // 4:] = -0.
    t = np.arange(2 * S - 1) - (S - 1.)
    table = np.array([np.where(t < 0, np.exp(t / 50.), -0.) * 0.5**a
                      for a in range(R)])
    got = _run(moments, [table], [R], 0)[0]
    want, bound = _want(moments, table, R, 0, 1)
    assert np.all(np.abs(got - want) <= 2.0**-52 * bound)
    assert np.all(got[want == 0] == 0)


def test_subnormals_are_no_zeros():
    S = 1000
    moments = np.zeros((1, 3, S))
    moments[0, 1, 500:540] = 5e-324 * np.arange(1, 41)
    table = np.full((1, 2 * S - 1), 1e10)
    got = _run(moments, [table], [1], 0)[0]
    want = -1.5 * 1e10 * moments[0, 1].sum()
    assert np.all(np.abs(got / want - 1) <= 40 * 2.0**-52)


@pytest.mark.parametrize('bad', [np.inf, -np.inf, np.nan])
def test_zeros_times_infinity(bad):
    S = 1000
    moments = np.zeros((1, 3, S))
    moments[0, 1, 10] = 1.
    table = np.zeros((1, 2 * S - 1))
    table[0, S - 1 + 300] = bad              # 300 slices behind each source
    got = _run(moments, [table], [1], 0)[0]
    want = np.zeros(S)
    for i in range(S):
        with np.errstate(invalid='ignore'):
            want[i] = -1.5 * np.sum(moments[0, 1] *
                                    table[0, i + S - 1 - np.arange(S)])
    assert np.array_equal(np.isnan(got), np.isnan(want))
    keep = ~np.isnan(want)
    assert np.array_equal(got[keep], want[keep])
