"""Per-slice moments of bunches whose first particles say nothing about the
rest: ordered by z with cuts inside the bunch, hardly a particle within the
cuts, slices whose values are far smaller than the others', coordinates that
are tiny as a whole.  Every sum is compared with extended precision relative
to its own slice's terms.

A total adds at most 304 CTAs' exact sums and, one by one, the values that
the CTAs' fixed point does not hold, so at most 304 + n roundings of 2^-53 of
sum |v|; a centred value and its mean round by 2^-53 of |u| each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

COORDS = ('x', 'xp', 'y', 'yp', 'z', 'dp')
SIGMAS = (1e-3, 1e-5, 2e-3, 3e-5, 0.23, 1e-3)
PAIRS = (('x', 'x'), ('y', 'y'), ('z', 'z'), ('dp', 'dp'), ('x', 'xp'),
         ('y', 'yp'), ('z', 'dp'), ('xp', 'xp'), ('yp', 'yp'), ('x', 'dp'),
         ('y', 'dp'), ('xp', 'dp'), ('yp', 'dp'))
PAIRS3 = ((0, 0), (0, 1), (1, 1), (0, 2), (1, 2), (2, 2))


def _sums(u, idx, S):
    L = np.longdouble
    out = np.zeros(S, dtype=L)
    order = np.argsort(idx, kind='stable')
    at = np.searchsorted(idx[order], np.arange(S))
    have = np.bincount(idx, minlength=S) > 0
    out[have] = np.add.reduceat(u[order].astype(L), at[have])
    return out


def _bunch(case, n, precision):
    import cases as C
    import gpu_cases as G
    rs = np.random.RandomState(n % 1000)
    c = {k: rs.normal(0, s, n) for k, s in zip(COORDS, SIGMAS)}
    c['xp'] += 0.01 * c['x']
    cuts = (-0.46, 0.46)
    if case == 'ordered':
        c['yp'] *= 1e-2                     # a vertical emittance of 1 pm
    elif case == 'narrow':
        cuts = (0.1, 0.1002)
    elif case == 'tiny slices':
        c['x'][c['z'] > 0.1] *= 1e-9
        c['xp'][c['z'] > 0.1] *= 1e-9
    elif case == 'tiny':
        c['yp'] *= 1e-13
        c['dp'] *= 1e-20 if precision == 'fp64' else 1e-10
    elif case == 'zeros first':
        c['x'][:n - n // 8] = 0.
    beam = G.make_beam(C.beam_params(n, 3), c, precision=precision)
    if case == 'ordered':
        beam.sort_for('z')
    return beam, cuts


@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('n,S', [(700001, 60), (5000, 7)])
@pytest.mark.parametrize('case', ['ordered', 'narrow', 'tiny slices', 'tiny',
                                  'zeros first'])
def test_moments_relative_to_their_slice(case, n, S, precision):
    from pyheadtail_gb300.particles import slicing
    beam, cuts = _bunch(case, n, precision)
    ss = slicing.UniformBinSlicer(S, z_cuts=cuts).slice(beam)
    u = {k: getattr(beam, k).double().cpu().numpy() for k in COORDS}
    idx = np.floor((u['z'] - cuts[0]) / ((cuts[1] - cuts[0]) / float(S)))
    at = (idx >= 0) & (idx < S)
    idx = idx[at].astype(int)
    u = {k: v[at] for k, v in u.items()}
    count = np.bincount(idx, minlength=S)
    k = np.maximum(count, 1)
    eps = 2.0**-53
    adds = (304 + count) * eps
    mean = {q: _sums(u[q], idx, S) / k for q in COORDS}
    size = {q: _sums(np.abs(u[q]), idx, S) / k for q in COORDS}
    dev = {q: u[q].astype(np.longdouble) - mean[q][idx] for q in COORDS}

    def check(got_mean, got_cov, names, pairs, got_count):
        assert np.array_equal(got_count.cpu().numpy(), count)
        for q, m in zip(names, got_mean.cpu().numpy()):
            assert np.all(np.abs(m - mean[q]) <= (adds + 2 * eps) * size[q]), q
        for (a, b), v in zip(pairs, got_cov.cpu().numpy()):
            d = np.where(count > 1, count - 1, 1)
            want = _sums(dev[a] * dev[b], idx, S) / d
            bar = (adds + 4 * eps) * _sums(np.abs(dev[a] * dev[b]), idx, S) / d
            bar += 4 * eps * (
                _sums(np.abs(u[a] * dev[b]), idx, S) +
                _sums(np.abs(u[b] * dev[a]), idx, S)) / d
            # the means' own errors, twice
            bar += k * (adds + 4 * eps)**2 * size[a] * size[b] / d
            assert np.all(np.abs(v - want) <= bar), (a, b)

    means, cov, counts = slicing._all_slice_moments(ss, beam)
    check(means, cov, COORDS, PAIRS, counts)
    for names in (('y', 'yp', 'dp'), ('x', 'xp')):
        means, cov, counts = slicing._slice_moments(ss, beam, list(names))
        check(means[:len(names)], torch.stack(
            [cov[i] for i, p in enumerate(PAIRS3) if max(p) < len(names)]),
            names, [(names[i], names[j]) for i, j in PAIRS3
                    if max(i, j) < len(names)], counts)
