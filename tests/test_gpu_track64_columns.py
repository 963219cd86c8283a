"""FP64 slicing with the partial columns a caller chooses: one CTA per column,
or clusters of four where there are fewer columns than SMs and tiles.  Counts
are exact; the sums are compared with exact sums of the host.

Bar: every value rounds by at most 2^-56 of the largest |u|, the columns and
their merge by 2^-53 of the partial sums (at most grid + 8 additions)."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


@pytest.mark.parametrize('n', [1, 257, 40001, 300007])
@pytest.mark.parametrize('grid', ['default', 1, 3, 'sms-1', 'sms', 'sms+1'])
@pytest.mark.parametrize('S', [5, 130])
def test_counts_and_sums(n, grid, S):
    from pyheadtail_gb300 import _native as N
    from pyheadtail_gb300._engine import DeviceSlicer
    L = N.load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    G = {'default': L.phk_track_grid(n, 0, S), 'sms-1': sms - 1, 'sms': sms,
         'sms+1': sms + 1}.get(grid, grid)
    rng = np.random.RandomState(n + S)
    x, y, z = rng.normal(0, 1e-3, n), rng.normal(0, 2., n), rng.normal(0, .3, n)
    dev = [torch.from_numpy(a).cuda() for a in (x, y, z)]
    sl = DeviceSlicer(-0.69, 0.69, S, 0, 'cuda')
    c = N.Coords()
    c.x = c.xp = dev[0].data_ptr()
    c.y = c.yp = dev[1].data_ptr()
    c.z = c.dp = dev[2].data_ptr()
    c.n, c.dtype = n, 0
    part = torch.full((3 * S * G,), np.nan, dtype=torch.float64, device='cuda')
    acc = N.Accum()
    acc.slicer, acc.partials = sl.struct, part.data_ptr()
    acc.partials_len, acc.grid = part.numel(), G
    counts = torch.empty(S, dtype=torch.int32, device='cuda')
    mean = torch.empty(2, S, dtype=torch.float64, device='cuda')
    stream = torch.cuda.current_stream().cuda_stream
    N.call('phk_track', ctypes.byref(N.Program()), ctypes.byref(c), None,
           ctypes.byref(acc), stream)
    N.call('phk_slice_finalize', ctypes.byref(acc), counts.data_ptr(),
           mean[0].data_ptr(), mean[1].data_ptr(), None, stream)
    idx = np.floor((z - sl.tail) / sl.width)
    for s in range(S):
        at = idx == s
        k = int(at.sum())
        assert int(counts[s]) == k
        for q, u in enumerate((x, y)):
            want = math.fsum(u[at]) / k if k else 0.
            bar = (2.0**-56 * np.abs(u).max() +
                   (G + 8) * 2.0**-53 * (np.abs(u[at]).sum() / max(k, 1)))
            assert abs(float(mean[q, s]) - want) <= bar
