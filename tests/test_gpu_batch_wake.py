"""Batched wakes (phk_wake_batch) against sums in extended precision on the
host, called through the C ABI: convolutions and dot-product tables, several
stored turns in a ring, sizes at the edges of the 32-target blocks and on both
sides of the 512 terms per target where the lane-split sums take over, bunches
with fewer kicks than the launch, both output types.

Bar: the n terms of a target are added in chains of at most ceil(n / 32) + 8
additions (either path), each rounding once relative to the sum of the terms'
magnitudes, then one factor and one rounding of the output."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('S,lags,ring', [
    (1, 1, 1), (2, 3, 4), (31, 2, 2), (32, 1, 3), (33, 4, 4), (100, 1, 1),
    (100, 5, 6), (100, 6, 6), (512, 1, 1), (513, 1, 2), (700, 2, 2)])
@pytest.mark.parametrize('dense', [0, 1])
@pytest.mark.parametrize('code', [0, 1])
def test_against_extended_precision(S, lags, ring, dense, code):
    from pyheadtail_gb300 import _native as N
    N.load()
    rng = np.random.RandomState(S + 10 * lags + dense)
    nb, nk = 3, 2
    dt = torch.float64 if code == 0 else torch.float32
    keep, want, size, outs = [], [], [], []
    sets = (N.WakeSet * nb)()
    row = S * S if dense else 2 * S - 1
    for b in range(nb):
        mom = rng.normal(size=(ring, 3, S)) * 10.**rng.uniform(-3, 3, S)
        w = sets[b]
        w.n_slices, w.ring_len, w.head = S, ring, int(rng.randint(ring))
        w.n_kicks = nk - (b == 1)
        w.out_dtype = code
        m_dev = torch.from_numpy(mom).cuda()
        w.moments = m_dev.data_ptr()
        keep.append(m_dev)
        for k in range(w.n_kicks):
            tab = rng.normal(size=(lags, row))
            t_dev = torch.from_numpy(tab).cuda()
            out = torch.full((S,), np.nan, dtype=dt, device='cuda')
            kk = w.kick[k]
            kk.source, kk.n_lags, kk.dense = (b + k) % 3, lags, dense
            kk.factor = float(rng.normal())
            kk.table, kk.out = t_dev.data_ptr(), out.data_ptr()
            keep.append(t_dev)
            total = np.zeros(S, dtype=np.longdouble)
            mag = np.zeros(S)
            for a in range(lags):
                m = mom[(w.head - a) % ring, kk.source]
                if dense:
                    M = tab[a].reshape(S, S).T
                else:
                    at = np.arange(S)[:, None] + S - 1 - np.arange(S)[None, :]
                    M = tab[a][at]
                total += (M.astype(np.longdouble) * m).sum(1)
                mag += np.abs(M * m).sum(1)
            want.append(total * kk.factor)
            size.append(mag * abs(kk.factor))
            outs.append(out)
    dev = torch.from_numpy(np.frombuffer(bytes(sets), dtype=np.uint8)
                           .copy()).cuda()
    N.call('phk_wake_batch', dev.data_ptr(), nb, S, nk, None)
    torch.cuda.synchronize()
    u, out_u = 2.0**-53, (2.0**-53 if code == 0 else 2.0**-24)
    steps = -(-S * lags // 32) + 8 + 2
    for out, ref, mag in zip(outs, want, size):
        got = out.double().cpu().numpy()
        bar = (steps * u * mag + out_u * np.abs(ref.astype(float))) * (1 + 1e-6)
        assert np.all(np.abs(got - ref) <= bar)
