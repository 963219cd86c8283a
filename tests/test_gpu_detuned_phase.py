"""Plain form: the detuned transverse map (fixed-point phase, sine and cosine)
against extended precision, for unit and general optics, chromaticity of
order 1 to 4 and amplitude detuning, detunings from zero to beyond the
fixed-point range, NaN.

With A the size of a particle's terms, D the sum of the magnitudes of its
detuning's terms and phi its phase advance, |error| <= A (16 + 16 * 2 pi D +
4 |phi|) 2^-53: a dozen roundings in the detuning and in the map, and the
phase (Q + dQ) 2 pi rounded as the reference rounds it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

L = np.longdouble
TWO_PI = 2 * L('3.14159265358979323846264338327950288')


def _detuning(seg, beam, u):
    """dQ_x, dQ_y and the sums of the magnitudes of their terms."""
    from pyheadtail_gb300.trackers.detuners import ChromaticitySegment
    dq = [np.zeros(len(u['x']), dtype=L) for _ in range(4)]
    for d in seg.segment_detuners:
        if isinstance(d, ChromaticitySegment):
            for k, c in enumerate((d.coeffs_x, d.coeffs_y)):
                for i, v in enumerate(c):
                    term = L(v) * u['dp']**(i + 1)
                    dq[k] = dq[k] + term
                    dq[k + 2] = dq[k + 2] + np.abs(term)
        else:
            j, m = [], []
            for a, b, q, p in ((d.alpha_x, d.beta_x, u['x'], u['xp']),
                               (d.alpha_y, d.beta_y, u['y'], u['yp'])):
                terms = ((1 + L(a)**2) / L(b) * q**2, 2 * L(a) * q * p,
                         L(b) * p**2)
                j.append(sum(terms))
                m.append(sum(np.abs(t) for t in terms))
            p0 = 2 * L(beam.p0)
            for k, (c0, c1) in enumerate(((d.dapp_x, d.dapp_xy),
                                          (d.dapp_yx, d.dapp_y))):
                dq[k] = dq[k] + (L(c0) * j[0] + L(c1) * j[1]) / p0
                dq[k + 2] = dq[k + 2] + (abs(c0) * m[0] + abs(c1) * m[1]) / p0
    return dq


@pytest.mark.parametrize('alpha', [0., 0.7])
@pytest.mark.parametrize('order,amplitude,size', [
    (1, False, 1.), (3, True, 1.), (1, True, 1.), (1, True, 40.),
    (1, True, 3e3), (2, False, 0.)])
def test_against_extended_precision(alpha, order, amplitude, size):
    import cases as C
    import gpu_cases as G
    from pyheadtail_gb300.trackers.detuners import (AmplitudeDetuning,
                                                    Chromaticity)
    from pyheadtail_gb300.trackers.transverse_tracking import TransverseMap
    if np.finfo(L).nmant < 63:
        pytest.skip('no extended precision on this host')
    n = 3001
    rs = np.random.RandomState(11)
    sig = dict(x=1e-3, xp=2e-5, y=1e-3, yp=2e-5, z=0.2, dp=1e-3)
    coords = {k: rs.normal(0, s, n) * (size if k in ('x', 'xp', 'y', 'yp') else 1.)
              for k, s in sig.items()}
    coords['dp'][:3] = [0., -0., 0.3]
    beam = G.make_beam(C.beam_params(n, 0), coords)
    qp = [5., -300., 2e4][:order]
    dets = [Chromaticity(qp, qp[::-1])]
    if amplitude:
        dets.append(AmplitudeDetuning(1e-11, 2e-11, -5e-12))
    s = np.array([0., 4000., C.C_SPS])
    ax = np.array([alpha, -0.3 * alpha, alpha])
    b = np.array([50., 50. + 20. * alpha, 50.])
    z3 = np.zeros(3)
    segs = list(TransverseMap(s, ax, b, z3, -ax, b, z3, 20.13, 20.18, dets))
    u = {k: v.astype(L) for k, v in coords.items()}
    seg = segs[0]
    dq = _detuning(seg, beam, u)
    seg.track(beam)
    got = {k: getattr(beam, k).cpu().numpy().astype(L) for k in coords}
    for plane, d, D, q, o in (('x', dq[0], dq[2], seg.dQ_x, 0),
                              ('y', dq[1], dq[3], seg.dQ_y, 2)):
        p, pp = plane, plane + 'p'
        phi = TWO_PI * (L(q) + d)
        c, sn = np.cos(phi), np.sin(phi)
        for row, name in ((0, p), (1, pp)):
            I, J = seg.I[o + row, o:o + 2], seg.J[o + row, o:o + 2]
            want = ((L(I[0]) * c + L(J[0]) * sn) * u[p] +
                    (L(I[1]) * c + L(J[1]) * sn) * u[pp])
            A = ((abs(I[0]) + abs(J[0])) * np.abs(u[p]) +
                 (abs(I[1]) + abs(J[1])) * np.abs(u[pp]))
            rel = 16 + TWO_PI * D * 16 + 4 * np.abs(phi)
            err = np.abs(got[name] - want)
            assert np.all(err <= A * rel * L(2)**-53), (
                name, float(np.max(err / np.maximum(A * rel * L(2)**-53,
                                                    L(1e-300)))))


def test_nan_and_infinite_detuning():
    import cases as C
    import gpu_cases as G
    n = 600
    rs = np.random.RandomState(1)
    coords = {k: rs.normal(0, 1e-3, n) for k in ('x', 'xp', 'y', 'yp', 'z', 'dp')}
    coords['dp'][5], coords['dp'][6], coords['x'][7] = np.nan, np.inf, np.nan
    beam = G.make_beam(C.beam_params(n, 0), coords)
    spec = dict(elements=[C.smooth_transverse(chroma=[5., 5.],
                                              amplitude=[1e-11, 1e-11, -5e-12])])
    for _, m in G.make_elements(spec, beam):
        m.track(beam)
    for k in ('x', 'xp', 'y', 'yp'):
        bad = np.isnan(getattr(beam, k).cpu().numpy())
        assert np.array_equal(np.flatnonzero(bad), [5, 6, 7]), k
