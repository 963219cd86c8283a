"""Plain form: the RF kick of particles near the zero of the wave.

dp = 0 before the kick, so that dp is A sin(phi) alone.  The sine of a small
phase is as accurate relative to itself as its FP64 phase was: the phase's
constant and product, the amplitude and the result round, together at most
2^-51 of the result; from a phase of 2^-10.4 on the fixed point adds its 2^-61.
With an offset the absolute bar of the fixed point holds (2^-60 and 2^-61 of the
phase), beside an offset below 2^-8 the relative one of the larger term."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

H, C_RING, V = 4620, 6911.5038378975451, 4.5e6


def _kick(z, offset, program):
    """dp / A of one RF kick, in the specialised and the generic program."""
    import cases as C
    import gpu_cases as G
    from scipy.constants import c
    from pyheadtail_gb300.trackers.longitudinal_tracking import RFSystems
    n = len(z)
    coords = {k: np.zeros(n) for k in ('x', 'xp', 'y', 'yp', 'dp')}
    coords['z'] = z
    beam = G.make_beam(C.beam_params(n, 0), coords)
    rf = RFSystems(C_RING, [H], [V], [0.], [beam.gamma**-2 + 1e-3],
                   beam.gamma, charge=beam.charge, mass=beam.mass)
    rf.phi_offsets[0] = offset
    if program == 'specialised':
        for _, m in G.make_elements(dict(elements=[C.smooth_transverse()]),
                                    beam):
            m.track(beam)
    rf.track(beam)
    A = np.abs(beam.charge) * V / (beam.beta * c) / beam.p0
    return beam.dp.cpu().numpy() / A


def _z():
    rs = np.random.RandomState(1)
    per = C_RING / H
    small = rs.choice([-1, 1], 3000) * per * 2.0**rs.uniform(-300, -9, 3000)
    edge = per / (2 * np.pi) * 2.0**np.arange(-14, -4)
    return np.concatenate([small, edge, -edge, np.nextafter(edge, 0), [0.]])


@pytest.mark.parametrize('program', ['specialised', 'generic'])
@pytest.mark.parametrize('offset', [0., 1e-12, -1e-4, 3e-3, np.pi])
def test_relative_accuracy_of_small_phases(offset, program):
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip('no extended precision on this host')
    z = _z()
    got = _kick(z, offset, program)
    L = np.longdouble
    pi = L('3.14159265358979323846264338327950288')
    wave = 2 * pi * (L(H) * z.astype(L) / L(C_RING))
    want = np.sin(wave + L(offset))
    bar = 2.0**-51 * (np.abs(wave) + np.abs(offset))
    bar = bar + np.where(np.abs(wave) >= 2.0**-10.4, 2.0**-61, 0.)
    if abs(offset) > 2.0**-8:
        bar = 2.0**-51 * np.abs(want) + 2.0**-60 + 2.0**-61 * np.abs(
            wave + L(offset))
    err = np.abs(got.astype(L) - want)
    assert np.all(err <= bar), float(np.max(err / np.maximum(bar, 1e-300)))
