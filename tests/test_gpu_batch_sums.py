"""FP32 batches: per-slice sums are exact fixed-point sums.

Each CTA adds the particles of a bunch as integers at a power-of-two scale
that its first tile of the bunch sets (the largest |u| of it maps to
[2^26, 2^27)), so every value rounds by at most 2^-27 of the bunch's largest
|u|; counts are exact.  Checked against FP64 sums of the beam's own FP32
values at sizes around the tiles, the counters' carry (more than 2^16
particles in one slice of one CTA), bunches of one particle, first tiles
that are all zero, and values far above the first tile's (64-bit level);
NaN and infinities mark their slice as a floating-point sum would; two
launches give the same bits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

COORDS = ('x', 'xp', 'y', 'yp', 'z', 'dp')
SIGMAS = (1e-3, 1e-5, 1e-3, 1e-5, 0.23, 1e-3)


def _coords(n, seed, **given):
    rng = np.random.RandomState(seed)
    c = {k: rng.normal(0, s, n) for k, s in zip(COORDS, SIGMAS)}
    c.update(given)
    return c


def _one_turn(S, coords, **config):
    """One batched turn of the bunches (RF and a resonator's slicing; x and y
    are only rotated): the tracker and its beams."""
    import gpu_cases as G
    import cases as C
    from pyheadtail_gb300.batch import BatchedTurn, BunchBatch
    beams, maps = [], []
    for b, c in enumerate(coords):
        spec = dict(beam=C.beam_params(len(c['x']), b), n_turns=1, elements=[
            C.smooth_transverse(chroma=[2., -1.]), C.rf(),
            C.wake(C.slicer(S), C.resonator())])
        beams.append(G.make_beam(spec['beam'], c, precision='fp32'))
        maps.append([el for _, el in G.make_elements(spec, beams[-1])])
    turn = BatchedTurn(BunchBatch(beams), maps, config=config)
    turn.track(1)
    return turn, beams


def _check(turn, beams, S):
    import cases as C
    tail, head = C.Z_CUTS
    width = (head - tail) / float(S)
    for b, beam in enumerate(beams):
        z = beam.z.double().cpu().numpy()
        idx = np.floor((z - tail) / width)
        inside = (idx >= 0) & (idx < S)
        k = idx[inside].astype(np.int64)
        counts = np.bincount(k, minlength=S)
        np.testing.assert_array_equal(turn.counts[b].cpu().numpy(), counts)
        for q, got in (('x', turn.mean_x), ('y', turn.mean_y)):
            u = getattr(beam, q).double().cpu().numpy()
            sums = np.bincount(k, weights=u[inside], minlength=S)
            mean = np.where(counts > 0, sums / np.maximum(counts, 1), 0.)
            # the fixed point's rounding, and the FP64 sums of the host
            bar = np.max(np.abs(u)) * (2.0**-27 + len(u) * 2.0**-52)
            err = np.max(np.abs(got[b].cpu().numpy() - mean))
            assert err <= bar, (b, q, err, bar)


@pytest.mark.parametrize('S', [1, 50, 333])
@pytest.mark.parametrize('config', [
    dict(threads=128, unit_tiles=2, ctas_per_sm=0),
    dict(threads=256, unit_tiles=8, ctas_per_sm=0),
    dict(threads=512, unit_tiles=32, ctas_per_sm=1)])
def test_sums_of_uneven_bunches_and_bits(S, config):
    sizes = [1, 2, 511, 513, 1027, 40000, 300001]
    coords = [_coords(n, 10 + b) for b, n in enumerate(sizes)]
    runs = [_one_turn(S, coords, **config) for _ in range(2)]
    _check(*runs[0], S)
    for q in ('counts', 'mean_x', 'mean_y'):
        assert torch.equal(getattr(runs[0][0], q).view(torch.int32),
                           getattr(runs[1][0], q).view(torch.int32))


def test_carry_of_a_full_slice():
    """All of 1.2e7 particles in one slice, about 79000 of them in each CTA's
    counters."""
    n = 12 * 10**6
    _check(*_one_turn(10, [_coords(n, 1, z=np.full(n, 0.01),
                                   dp=np.zeros(n))],
                      threads=512, unit_tiles=32, ctas_per_sm=1), 10)


def test_zero_first_tile_and_large_values():
    """A bunch whose first tiles are zero (scale 2^40), one whose later values
    are 2^10 times those of its first tile (64-bit level)."""
    n = 200000
    x = np.random.RandomState(3).normal(0, 1e-3, n)
    zero, large = x.copy(), x.copy()
    zero[:150000] = 0.
    large[100000:] *= 1024.
    xp = np.zeros(n)
    _check(*_one_turn(20, [_coords(n, 4, x=zero, xp=xp),
                           _coords(n, 5, x=large, xp=xp)],
                      threads=256, unit_tiles=8, ctas_per_sm=1), 20)


def test_nan_and_infinities_mark_their_slice():
    """x of slice 3: NaN; 4: +inf; 5: both infinities; 6: -inf.  The rotation
    mixes x and xp; y, yp and the other slices stay finite."""
    import cases as C
    n, S = 5000, 10
    tail, head = C.Z_CUTS
    centre = tail + (np.arange(S) + 0.5) * (head - tail) / S
    c = _coords(n, 6)
    c['dp'] = np.zeros(n)
    at = np.arange(n - 5, n)
    c['z'][at] = centre[[3, 4, 5, 5, 6]]
    c['x'][at] = [np.nan, np.inf, np.inf, -np.inf, -np.inf]
    turn, (beam,) = _one_turn(S, [c], threads=256, unit_tiles=8,
                              ctas_per_sm=0)
    x = beam.x.double().cpu().numpy()
    idx = np.floor((beam.z.double().cpu().numpy() - tail) / ((head - tail) / S))
    got = turn.mean_x[0].cpu().numpy()
    with np.errstate(invalid='ignore'):
        want = np.array([x[idx == s].sum() if np.any(idx == s) else 0.
                         for s in range(S)])
    bad = ~np.isfinite(want)
    assert bad.sum() == 4
    np.testing.assert_array_equal(np.isnan(got), np.isnan(want))
    np.testing.assert_array_equal(got[np.isinf(want)], want[np.isinf(want)])
    assert np.all(np.isfinite(got[~bad]))
    assert np.all(np.isfinite(turn.mean_y[0].cpu().numpy()))
