"""Plain form: RF kicks with phase offsets that are not finite or far beyond a
turn, in the specialised and the generic program: NaN, and the sine of the FP64
phase, as for any other offset too large for the fixed point."""
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
@pytest.mark.parametrize('offset', [np.nan, np.inf, -np.inf])
def test_offsets_that_are_not_finite(offset, program):
    assert np.all(np.isnan(_kick(_z(), offset, program)))


@pytest.mark.parametrize('program', ['specialised', 'generic'])
@pytest.mark.parametrize('offset', [1e10, -1e18, 1e300])
def test_huge_offsets_take_the_sine_of_the_rounded_phase(offset, program):
    z = _z()
    got = _kick(z, offset, program)
    phase = H * 2 * np.pi / C_RING * z + offset
    assert np.max(np.abs(got - np.sin(phase))) <= 2.0**-50 + \
        (2.0**-52 * 1e10 if abs(offset) <= 1e10 else 0.)
