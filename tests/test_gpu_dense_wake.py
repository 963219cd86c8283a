"""Dot-product wakes (slices that are not a fixed grid).

The resistive-wall samples made on the device against the wake function of
the kick, which is the reference's formula in NumPy: the same bits, no
tolerance; both signs of the Yokoya factors, several stored turns, sizes at
the edges of the 16-target blocks.

The kicks against exact-product sums in 64 bits and more on the host.  Bar:
every product and addition of the n_lags S terms of a target rounds once, in
a chain of at most n_lags ceil(S / 32) + 5 additions and one factor, relative
to the sum of the terms' magnitudes; plus one rounding of the output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


def _field(S, lags, wall):
    import gpu_cases as G
    from pyheadtail_gb300.impedances import wakes as W
    from pyheadtail_gb300.particles.slicing import UniformChargeSlicer
    coords = {}
    n = 40 * S + 3
    rng = np.random.RandomState(S)
    for k, s in zip(('x', 'xp', 'y', 'yp', 'z', 'dp'),
                    (1e-3, 1e-5, 1e-3, 1e-5, 0.23, 1e-3)):
        coords[k] = rng.normal(0, s, n)
    import cases as C
    return G, C, W, UniformChargeSlicer, coords, n


@pytest.mark.parametrize('S,lags', [(1, 1), (2, 3), (15, 2), (16, 1), (17, 2),
                                    (33, 4), (500, 1), (250, 2)])
@pytest.mark.parametrize('wall', ['ParallelPlatesResistiveWall',
                                  'CircularResistiveWall'])
@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
def test_samples_and_kicks(S, lags, wall, precision):
    G, C, W, UniformChargeSlicer, coords, n = _field(S, lags, wall)
    beam = G.make_beam(C.beam_params(n, 3), coords, precision=precision)
    src = getattr(W, wall)(pipe_radius=5e-2, resistive_wall_length=6911.,
                           conductivity=1e6, dt_min=1e-3 / 299792458.,
                           n_turns_wake=lags)
    field = W.WakeField(UniformChargeSlicer(S), src)
    for turn in range(lags):
        field.track(beam)
    sets = list(field.slice_set_deque)
    ages = list(field.slice_set_age_deque)
    st = field._state
    mom = st.moments.cpu().numpy()
    u = 2.0**-53
    out_u = u if precision == 'fp64' else 2.0**-24
    for k, kick in enumerate(field.wake_kicks):
        assert kick._dense
        got = kick._table.cpu().numpy()
        total = np.zeros(S, dtype=np.longdouble)
        size = np.zeros(S)
        for a in range(lags):
            want = np.asarray(kick._samples(
                sets[0]._times, sets[a]._times + ages[a], sets[a].beta))
            assert np.array_equal(got[a], want.ravel())
            slot = (st.head - a) % st.n_ring
            m = mom[slot][{'count': 0, 'x': 1, 'y': 2}[kick.moment]]
            total += (m.astype(np.longdouble)[:, None] * want).sum(0)
            size += np.abs(m[:, None] * want).sum(0)
        f = kick._wake_factor(beam)
        out = st.kick_out[k].double().cpu().numpy()
        steps = lags * -(-S // 32) + 5 + 1
        bar = steps * u * size * abs(f) * (1 + 1e-6)
        bar = bar + out_u * np.abs(total.astype(float) * f) * (1 + 1e-6)
        assert np.all(np.abs(out - total * f) <= bar + 1e-300)
