"""FP32 batches: slice means of bunches whose first tiles say nothing about the
rest.  A finite particle far beyond the others, zeros up to the last tiles,
planes of zeros, slices whose values are far smaller than the others', tiny
and huge planes: finite values give the finite sum.

Compared with FP64 sums of the beam's own FP32 values, relative to each
slice's terms: a CTA's sums are exact but for values outside its window,
which are added in FP64, as the columns are (at most 500 + the slice's
particles roundings, and the host's own)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

from test_gpu_batch_sums import _coords, _one_turn    # noqa: E402


def _bunch(case, n, seed):
    c = _coords(n, seed)
    if case == 'diverging':
        c['x'][n // 2], c['xp'][n // 2] = 1e3, 0.
        c['y'][-1], c['yp'][-1] = 3e30, 0.
    elif case == 'zeros first':
        for k in ('x', 'xp', 'y', 'yp'):
            c[k][:n - 700] = 0.
        c['x'][-300:] *= 1e4              # metres
        c['y'][-300:] *= 1e-6             # nanometres
    elif case == 'zero plane':
        c['y'][:] = c['yp'][:] = 0.
    elif case == 'tiny slices':
        for k in ('x', 'xp'):
            c[k][c['z'] > 0.2] *= 1e-9
    elif case == 'scales':
        for k in ('x', 'xp'):
            c[k] *= 1e-30
        for k in ('y', 'yp'):
            c[k] *= 1e30
    return c


@pytest.mark.parametrize('config', [
    dict(threads=128, unit_tiles=2, ctas_per_sm=0),
    dict(threads=256, unit_tiles=8, ctas_per_sm=1),
    dict(threads=512, unit_tiles=32, ctas_per_sm=1)])
@pytest.mark.parametrize('case', ['plain', 'diverging', 'zeros first',
                                  'zero plane', 'tiny slices', 'scales'])
def test_means_relative_to_their_slice(case, config):
    import cases as C
    S = 60
    coords = [_bunch(case, n, b) for b, n in enumerate((300, 30001, 400003))]
    turn, beams = _one_turn(S, coords, **config)
    tail, head = C.Z_CUTS
    for b, beam in enumerate(beams):
        z = beam.z.double().cpu().numpy()
        idx = np.floor((z - tail) / ((head - tail) / float(S)))
        at = (idx >= 0) & (idx < S)
        k = idx[at].astype(np.int64)
        counts = np.bincount(k, minlength=S)
        np.testing.assert_array_equal(turn.counts[b].cpu().numpy(), counts)
        for q, got in (('x', turn.mean_x), ('y', turn.mean_y)):
            u = getattr(beam, q).double().cpu().numpy()[at]
            n = np.maximum(counts, 1)
            mean = np.bincount(k, weights=u, minlength=S) / n
            size = np.bincount(k, weights=np.abs(u), minlength=S) / n
            got = got[b].cpu().numpy()
            assert np.all(np.isfinite(got)), (b, q)
            bar = (500 + 2 * counts) * 2.0**-53 * size
            assert np.all(np.abs(got - mean) <= bar), (b, q)
