"""phk_wake_batch where its work is split otherwise: many bunches with more than
512 terms per target (16 chains per warp) and few bunches (a warp per target),
on both sides of the rules, against sums in extended precision on the host.

Bar: the chains of a target's n terms are at most lags (S / 128 + 3) + 8
additions long (a warp's lanes: lags ceil(S / 128) + 8), each rounding once
relative to the sum of the terms' magnitudes, then one factor."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('nb,S,lags', [
    (40, 100, 5), (40, 100, 6), (40, 33, 20), (80, 129, 4), (20, 1000, 1),
    (20, 515, 1), (2, 128, 1), (2, 129, 1), (2, 200, 50), (1, 1000, 3)])
@pytest.mark.parametrize('dense', [0, 1])
def test_against_extended_precision(nb, S, lags, dense):
    if dense and S > 200:
        pytest.skip('the tables of the host are S x S')
    from pyheadtail_gb300 import _native as N
    N.load()
    rng = np.random.RandomState(S + lags)
    row = S * S if dense else 2 * S - 1
    mom = rng.normal(size=(nb, lags, 3, S)) * 10.**rng.uniform(-3, 3, S)
    tab = rng.normal(size=(nb, lags, row))
    m_dev, t_dev = torch.from_numpy(mom).cuda(), torch.from_numpy(tab).cuda()
    out = torch.full((nb, S), np.nan, dtype=torch.float64, device='cuda')
    sets = (N.WakeSet * nb)()
    for b in range(nb):
        w = sets[b]
        w.n_slices, w.ring_len, w.head, w.n_kicks, w.out_dtype = S, lags, 0, 1, 0
        w.moments = m_dev[b].data_ptr()
        kk = w.kick[0]
        kk.source, kk.n_lags, kk.dense, kk.factor = 1, lags, dense, 0.75
        kk.table, kk.out = t_dev[b].data_ptr(), out[b].data_ptr()
    dev = torch.from_numpy(np.frombuffer(bytes(sets), dtype=np.uint8)
                           .copy()).cuda()
    N.call('phk_wake_batch', dev.data_ptr(), nb, S, 1, None)
    got = out.cpu().numpy()
    at = np.arange(S)[:, None] + S - 1 - np.arange(S)[None, :]
    steps = lags * (S // 128 + 3) + 8 + 2
    for b in range(0, nb, max(1, nb // 4)):
        total, mag = np.zeros(S, dtype=np.longdouble), np.zeros(S)
        for a in range(lags):
            m = mom[b, (0 - a) % lags, 1]
            M = tab[b, a].reshape(S, S).T if dense else tab[b, a][at]
            total += (M.astype(np.longdouble) * m).sum(1)
            mag += np.abs(M * m).sum(1)
        bar = 0.75 * (steps + 1) * 2.0**-53 * mag * (1 + 1e-6)
        assert np.all(np.abs(got[b] - 0.75 * total) <= bar), b
