"""Per-slice moments behind Slicer.add_statistics: fixed-point digits per
CTA in shared memory, FP64 totals.  Both entry points (all statistics at
once, one at a time) against NumPy in extended precision, at ragged sizes,
slice counts that do and do not fit in shared memory, more values per CTA
than a digit counter holds, and values outside the fixed point's range.

A total is the FP64 sum of at most 304 CTA totals, each rounded once:
|error| <= 400 * 2^-53 of the largest |value| (of the largest product for a
second moment); the unit's truncation is far below."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

COORDS = ('x', 'xp', 'y', 'yp', 'z', 'dp')
SIGMAS = (1e-3, 1e-5, 2e-3, 3e-5, 0.23, 1e-3)
CUTS = (-0.5, 0.45)
NAMES = ['mean_' + k for k in COORDS] + ['sigma_' + k for k in
                                         ('x', 'y', 'z', 'dp')]
TOL = 400 * 2.0**-53


def _beam(n, seed, precision, spoil=None):
    import cases as C
    import gpu_cases as G
    rs = np.random.RandomState(seed)
    coords = {k: rs.normal(0, s, n) for k, s in zip(COORDS, SIGMAS)}
    coords['xp'] += 0.01 * coords['x'] + 0.3 * coords['dp']
    if spoil is not None:
        spoil(coords)
    return G.make_beam(C.beam_params(n, seed), coords, precision=precision)


def _reference(beam, S):
    u = {k: getattr(beam, k).double().cpu().numpy() for k in COORDS}
    width = (CUTS[1] - CUTS[0]) / float(S)
    idx = np.floor((u['z'] - CUTS[0]) / width)
    inside = (idx >= 0) & (idx < S)
    idx = idx[inside].astype(int)
    n = np.bincount(idx, minlength=S)
    L = np.longdouble
    order = np.argsort(idx, kind='stable')
    at = np.searchsorted(idx[order], np.arange(S))

    def total(v):
        if not len(v):
            return np.zeros(S, dtype=L)
        t = np.add.reduceat(np.append(v[order], L(0)), at)
        return np.where(n > 0, t, 0)

    mean, dev = {}, {}
    for k in COORDS:
        v = u[k][inside].astype(L)
        mean[k] = total(v) / np.maximum(n, 1)
        dev[k] = v - mean[k][idx]
    cov = lambda a, b: total(dev[a] * dev[b]) / np.maximum(n - 1, 1)
    top = {k: max(float(np.max(np.abs(dev[k]), initial=0)), 1e-300)
           for k in COORDS}
    size = {k: float(np.max(np.abs(u[k][inside]), initial=0)) for k in COORDS}
    return n, mean, cov, top, size


def _check(ss, ref, beam, slicing_means=False):
    n, mean, cov, top, size = ref
    assert np.array_equal(ss.n_macroparticles_per_slice.cpu().numpy(), n)
    for k in COORDS:
        if k in 'xy' and beam.precision == 'fp32' and slicing_means:
            continue        # the slicing pass's own FP32 sums
        got = getattr(ss, 'mean_' + k).cpu().numpy()
        assert np.max(np.abs(got - mean[k])) <= TOL * size[k], k
    for k in ('x', 'y', 'z', 'dp'):
        got = getattr(ss, 'sigma_' + k).cpu().numpy()
        err = np.abs(got**2 - cov(k, k))
        assert np.max(err) <= 2 * TOL * top[k]**2, k
    many = n > 20
    if np.any(many) and hasattr(ss, 'epsn_x'):
        c = {p: cov(*p) for p in (('x', 'x'), ('x', 'xp'), ('xp', 'xp'),
                                  ('x', 'dp'), ('xp', 'dp'), ('dp', 'dp'))}
        dd = np.where(many, c['dp', 'dp'], 1)
        s11 = c['x', 'x'] - c['x', 'dp']**2 / dd
        s12 = c['x', 'xp'] - c['x', 'dp'] * c['xp', 'dp'] / dd
        s22 = c['xp', 'xp'] - c['xp', 'dp']**2 / dd
        want = np.sqrt(np.where(many, s11 * s22 - s12**2, 0)) * beam.betagamma
        got = ss.epsn_x.cpu().numpy()
        # the determinant loses what its terms exceed it by (cond < 1e4)
        assert np.max(np.abs(got - want)[many] / want[many]) <= 1e4 * TOL


@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('n,S', [(1, 1), (513, 7), (100003, 200),
                                 (300001, 1100), (12000000, 3)])
def test_all_statistics(n, S, precision):
    from pyheadtail_gb300.particles.slicing import UniformBinSlicer
    beam = _beam(n, n % 97, precision)
    ss = UniformBinSlicer(S, z_cuts=CUTS).slice(beam, statistics=True)
    _check(ss, _reference(beam, S), beam, slicing_means=True)


@pytest.mark.parametrize('precision', ['fp64', 'fp32'])
@pytest.mark.parametrize('n,S', [(1000, 3), (70001, 130), (50000, 4096)])
def test_one_statistic_at_a_time(n, S, precision):
    from pyheadtail_gb300.particles.slicing import UniformBinSlicer
    beam = _beam(n, 5, precision)
    ss = UniformBinSlicer(S, z_cuts=CUTS).slice(beam)
    for k in NAMES:
        ss_k = UniformBinSlicer(S, z_cuts=CUTS)
        ss_k.add_statistics(ss, beam, [k])
    _check(ss, _reference(beam, S), beam)


def test_values_outside_the_fixed_point():
    """Huge and tiny values keep their FP64 accuracy, NaN and infinities
    reach their own slice alone."""
    from pyheadtail_gb300.particles.slicing import UniformBinSlicer
    n, S = 60000, 19

    def spoil(c):
        c['x'][1000:1010] *= 1e6
        c['y'][2000:2500] *= 1e-30
        c['x'][3000], c['z'][3000] = np.nan, -0.49
        c['yp'][3001], c['z'][3001] = np.inf, 0.44

    beam = _beam(n, 8, 'fp64', spoil)
    ss = UniformBinSlicer(S, z_cuts=CUTS).slice(beam, statistics=True)
    assert np.flatnonzero(np.isnan(ss.mean_x.cpu().numpy())).tolist() == [0]
    assert np.isposinf(ss.mean_yp.cpu().numpy()[S - 1])
    n_ref, mean, _, _, size = _reference(beam, S)
    keep = slice(1, S - 1)
    for k in COORDS:
        got = getattr(ss, 'mean_' + k).cpu().numpy()[keep]
        top = np.nanmax(np.where(np.isfinite(getattr(beam, k).cpu().numpy()),
                                 np.abs(getattr(beam, k).cpu().numpy()), 0))
        assert np.max(np.abs(got - mean[k][keep])) <= TOL * top, k
