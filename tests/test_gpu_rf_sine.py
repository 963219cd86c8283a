"""Plain form: the RF kick's fixed-point sine against extended precision.

[TransverseSegmentMap, RFSystems] on particles with dp = 0, so that the kick
is A sin(2 pi h z / C + offset) alone and z reaches the kick unchanged.  The
fixed-point sine is within 2^-61 of the exact one (table rounding and one
truncation per product); the phase keeps 62 bits (h / C and the product, each
truncated), the result adds the rounding of A / p0 and of the product:
|error| <= A (2^-60 + 2^-61 |phase| + 2^-51 |sin|)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

H, C_RING, V = 4620, 6911.5038378975451, 4.5e6


def _z():
    """Quarter-wave points, their neighbours, table points, both signs,
    zeros, subnormals, many turns, particles far beyond the fixed point."""
    rs = np.random.RandomState(4)
    per = C_RING / H
    grid = per * np.concatenate([np.arange(-16, 17) / 4.,
                                 np.arange(0, 4097, 37) / 4096.])
    near = np.concatenate([np.nextafter(grid, -np.inf), grid,
                           np.nextafter(grid, np.inf)])
    tiny = np.array([0., -0., 5e-324, 1e-310, 1e-300, 1e-30, 1e-18, -1e-17,
                     3e-10, -1e-5])
    many = per * rs.uniform(-1000, 1000, 2000)
    far = np.array([1e4, -1e5, 1.7e6])
    return np.concatenate([near, tiny, many, far,
                           rs.normal(0, 0.23, 20001)])


@pytest.mark.parametrize('offset', [0., np.pi, -2.5, 40.])
def test_against_extended_precision(offset):
    import cases as C
    import gpu_cases as G
    from scipy.constants import c, e
    from pyheadtail_gb300.trackers.longitudinal_tracking import RFSystems
    if np.finfo(np.longdouble).nmant < 63:
        pytest.skip('no extended precision on this host')
    z = _z()
    n = len(z)
    coords = {k: np.zeros(n) for k in ('x', 'xp', 'y', 'yp', 'dp')}
    coords['z'] = z
    beam = G.make_beam(C.beam_params(n, 0), coords)
    rf = RFSystems(C_RING, [H], [V], [offset], [beam.gamma**-2 + 1e-3],
                   beam.gamma, charge=beam.charge, mass=beam.mass)
    A = np.abs(beam.charge) * V / (beam.beta * c) / beam.p0
    spec = dict(elements=[C.smooth_transverse()])
    for _, m in G.make_elements(spec, beam):
        m.track(beam)
    rf.track(beam)
    got = beam.dp.cpu().numpy()
    L = np.longdouble
    pi = L('3.14159265358979323846264338327950288')
    phi = 2 * pi * (L(H) * z.astype(L) / L(C_RING)) + L(offset)
    want = np.sin(phi)
    near = np.abs(z) < 2**9 * C_RING / H
    err = np.abs(got.astype(L) / L(A) - want)
    bar = 2.0**-60 + 2.0**-61 * np.abs(phi) + 2.0**-51 * np.abs(want)
    assert np.all(err[near] <= bar[near]), float(np.max((err / bar)[near]))
    # many turns: at least as good as the library's sine of the FP64 phase
    far = ~near
    assert np.all(err[far] <= np.abs(phi[far]) * 2.0**-51)
