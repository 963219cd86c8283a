"""Plain form: slice means of bunches whose first particles say nothing about
the rest.  Bunches on the axis with an angle (the position appears in the
pass itself), slices whose values are far smaller than the others', planes
that are tiny as a whole, zeros up to the last particles, ordered bunches, a
lone particle near the axis, a large beta function at the end of the turn.

Every mean is compared with the exact sum of the beam's own coordinates,
relative to its slice's terms: the columns (or one CTA's values outside its
window, at most all of the slice's) are added in FP64, one rounding each."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

COORDS = ('x', 'xp', 'y', 'yp', 'z', 'dp')
SIGMAS = (1e-3, 1e-5, 2e-3, 3e-5, 0.23, 1e-3)


def _coords(case, n):
    rs = np.random.RandomState(n % 1000)
    c = {k: rs.normal(0, s, n) for k, s in zip(COORDS, SIGMAS)}
    if case == 'axis':
        c['x'][:] = 0.
        c['xp'] *= 1e-4
        c['y'][:] = c['yp'][:] = 0.
    elif case == 'tiny slices':
        for k in ('x', 'xp'):
            c[k][c['z'] > 0.2] *= 1e-10
    elif case == 'tiny':
        for k in ('x', 'xp'):
            c[k] *= 1e-200
        for k in ('y', 'yp'):
            c[k] *= 1e-290
    elif case == 'zeros first':
        for k in ('x', 'xp'):
            c[k][:n - n // 8] = 0.
        for k in ('y', 'yp'):
            c[k][:-3] = 0.
    elif case == 'lone':
        for k in ('x', 'xp', 'y', 'yp'):
            c[k][-1] *= 1e-12
    return c


def _track(case, n, S):
    """One fused pass: transverse map and the slicing of a wake field."""
    import cases as C
    import gpu_cases as G
    optics = C.smooth_transverse()
    if case == 'beta':
        optics['beta_x'] = optics['beta_y'] = [50., 5e6]
    elements = [optics, C.wake(C.slicer(S), C.resonator())]
    beam = G.make_beam(C.beam_params(n, 1), _coords(case, n))
    if case == 'ordered':
        beam.sort_for('x')
    spec = dict(beam=C.beam_params(n, 1), n_turns=1, elements=elements)
    els = [el for _, el in G.make_elements(spec, beam)]
    for el in els:
        el.track(beam)
    ss = els[-1].slice_set_deque[0]
    return beam, ss


@pytest.mark.parametrize('n,S', [(257, 5), (70001, 40), (400009, 1000)])
@pytest.mark.parametrize('case', ['axis', 'tiny slices', 'tiny', 'ordered',
                                  'zeros first', 'lone', 'beta'])
def test_means_relative_to_their_slice(case, n, S):
    import cases as C
    beam, ss = _track(case, n, S)
    tail, head = C.Z_CUTS
    u = {k: getattr(beam, k).cpu().numpy() for k in COORDS}
    idx = np.floor((u['z'] - tail) / ((head - tail) / float(S)))
    counts = ss.n_macroparticles_per_slice.cpu().numpy()
    got = {k: getattr(ss, 'mean_' + k).cpu().numpy() for k in 'xy'}
    order = np.argsort(idx, kind='stable')
    cut = np.searchsorted(idx[order], np.arange(S + 1))
    for s in range(S):
        at = order[cut[s]:cut[s + 1]]
        k = len(at)
        assert counts[s] == k
        for q in 'xy':
            v = u[q][at]
            want = math.fsum(v) / k if k else 0.
            bar = (456 + 8 + k) * 2.0**-53 * np.abs(v).sum() / max(k, 1)
            assert abs(got[q][s] - want) <= bar, (s, q)


@pytest.mark.parametrize('case', ['plain', 'axis', 'ordered', 'beta'])
def test_bits_are_the_same_on_every_launch(case):
    a, b = (_track(case, 300007, 100)[1] for _ in range(2))
    assert a.mean_x.cpu().numpy().tobytes() == b.mean_x.cpu().numpy().tobytes()
    assert a.mean_y.cpu().numpy().tobytes() == b.mean_y.cpu().numpy().tobytes()
