"""Batches with thousands of slices, up to the most that a launch takes (kick
tables of 48 KB per bunch): every bunch against the single-bunch pass on the
same coordinates.  A batch whose kick tables are larger still runs the turn
before there are kicks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

COORDS = ('x', 'xp', 'y', 'yp', 'z', 'dp')


def _spec(n, seed, S, kind, n_sources):
    import cases as C
    return dict(beam=C.beam_params(n, seed), n_turns=1, elements=[
        C.smooth_transverse(chroma=[2., 3.]), C.rf(),
        C.wake(C.slicer(S), *[C.resonator(kind=kind, f=(1. + i) * 1e9)
                              for i in range(n_sources)])])


@pytest.mark.parametrize('precision,tol', [('fp64', 1e-12), ('fp32', 1e-5)])
@pytest.mark.parametrize('S,kind,n_sources,turns', [
    (500, 'circular', 1, 3), (3072, 'circular', 1, 3),
    (4096, 'longitudinal', 1, 3), (768, 'parallel_horizontal', 2, 3),
    (4060, 'circular', 1, 1), (2190, 'parallel_horizontal', 2, 1)])
@pytest.mark.parametrize('threads', [128, 512])
def test_against_single_bunches(S, kind, n_sources, turns, precision, tol,
                                threads):
    import gpu_cases as G
    from oracle import cases as OC
    from pyheadtail_gb300.batch import BatchedTurn, BunchBatch
    specs = [_spec(n, 5 + b, S, kind, n_sources)
             for b, n in enumerate((20001, 301))]
    coords = [OC.make_beam(s['beam']).coords() for s in specs]
    beams = [G.make_beam(s['beam'], c, precision=precision)
             for s, c in zip(specs, coords)]
    maps = [[el for _, el in G.make_elements(s, b)]
            for s, b in zip(specs, beams)]
    turn = BatchedTurn(BunchBatch(beams), maps,
                       config=dict(threads=threads, unit_tiles=4, ctas_per_sm=0))
    turn.track(turns)
    assert turn.read_status() == 0
    for s, c, beam in zip(specs, coords, beams):
        one = G.make_beam(s['beam'], c, precision=precision)
        elements = [el for _, el in G.make_elements(s, one)]
        for _ in range(turns):
            for el in elements:
                el.track(one)
        got, want = beam.coords_numpy(), one.coords_numpy()
        for k in COORDS:
            ref = np.sqrt(np.mean(np.asarray(want[k], dtype=float)**2))
            err = np.max(np.abs(np.asarray(got[k], dtype=float) - want[k]))
            assert err <= tol * ref, (k, err / ref)
