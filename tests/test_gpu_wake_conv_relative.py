"""phk_wake, numpy path, integer convolution: targets whose terms are all far
below the largest of their windows, each relative to its own terms.  The head of
a bunch in a causal wake (wide cuts, empty slices ahead and behind), a bunch with
a gap and a wake that dies within the gap, moments that differ by orders of
magnitude between neighbours.

The fixed point's error of a target that it keeps is at most a sixteenth of n
2^-53 of the sum of its n terms' magnitudes (rms; four times that allowed here);
sums of units, warps and CTAs round once each, at most lags * ceil(S / 16) / 64 +
24 in a row (a target summed in FP64: lags S / 2048 + 24)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from test_gpu_wake_conv import _run    # noqa: E402


def _moments(case, R, S, rs):
    at = np.linspace(-6., 6., S)
    if case == 'gap':
        dens = np.where(np.abs(np.abs(at) - 3.) < 1., 1e5, 0.)
        dens[S // 2] = 1.
    elif case == 'scales':
        return rs.normal(0, 1., (R, 3, S)) * 10.**rs.uniform(-12, 0, (R, 3, S))
    else:
        dens = np.floor(1e6 * np.exp(-at**2 / 2))
    m = rs.normal(0, 1e-4, (R, 3, S)) * np.sqrt(dens) + 1e-6 * dens
    m[:, 0] = dens
    return m


def _table(wake, R, S):
    t = (np.arange(2 * S - 1) - (S - 1.)) * 1e-11
    rows = []
    for a in range(R):
        if wake == 'wall':
            u = t - 2.3e-5 * a
            rows.append(np.where(u < 0, -1e15 / np.sqrt(np.clip(-u, 1e-12, None)),
                                 0.))
        else:
            rate = 2e10 if wake == 'dying' else 3e9
            u = np.minimum(t, 0.)
            rows.append(np.exp(rate * u) * np.sin(1e10 * u) * 1e17 * 1e-3**a)
    return np.array(rows)


@pytest.mark.parametrize('S,R', [(800, 1), (1000, 1), (4096, 1), (500, 3),
                                 (500, 50), (1000, 2)])
@pytest.mark.parametrize('case', ['tails', 'gap', 'scales'])
def test_relative_to_the_terms(case, S, R):
    rs = np.random.RandomState(S + R)
    moments = _moments(case, R, S, rs)
    tables = [_table(k, R, S) for k in ('wall', 'resonator', 'dying')]
    got = _run(moments, tables, [R] * 3, 0)
    steps = R * -(-S // 16) / 64. + R * S / 2048. + 48 + R * S / 4.
    for k, table in enumerate(tables):
        want, size = np.zeros(S, dtype=np.longdouble), np.zeros(S)
        for a in range(R):
            m = moments[(0 - a) % R, 1 + k % 2]
            want += np.convolve(m.astype(np.longdouble),
                                table[a].astype(np.longdouble), 'valid')
            size += np.convolve(np.abs(m), np.abs(table[a]), 'valid')
        bar = 1.5 * (steps + 1) * 2.0**-53 * size * (1 + 1e-9)
        err = np.abs(got[k] + 1.5 * want)
        assert np.all(err <= bar), (k, int(np.argmax(err - bar)))
