"""Plain form: per-slice sums of the fused pass are 64-bit fixed-point sums
per thread-block cluster (unit: at most 2^-56 of a typical value of the
cluster's first tiles), slices with values far above that, infinite or NaN
ones are summed again in FP64.  Checked against exactly rounded sums (math.fsum) where the fixed
point, its carries and the second sum can go wrong: ragged sizes, one slice
holding everything, more values per CTA than a counter holds, values far
above the first tiles', non-finite values, first tiles of zeros, and the
largest slice count with pending kicks."""
import ctypes
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

CUTS = (-0.69, 0.69)


def _pass(x, y, z, S, grid=None, kicks=()):
    """phk_track (empty program, accumulation; kicks on xp pending) and
    phk_slice_finalize on FP64 arrays; grid: partial columns."""
    from pyheadtail_gb300 import _native as N
    from pyheadtail_gb300._engine import DeviceSlicer
    L = N.load()
    n = len(x)
    t = {k: torch.as_tensor(np.asarray(v, dtype=np.float64)).cuda()
         for k, v in (('x', x), ('y', y), ('z', z))}
    mom = [torch.zeros(n, dtype=torch.float64, device='cuda') for _ in range(3)]
    c = N.Coords()
    c.x, c.y, c.z = (t[k].data_ptr() for k in 'xyz')
    c.xp, c.yp, c.dp = (m.data_ptr() for m in mom)
    c.n, c.dtype = n, 0
    sl = DeviceSlicer(CUTS[0], CUTS[1], S, 0, 'cuda')
    acc = N.Accum()
    acc.slicer = sl.struct
    acc.grid = grid or L.phk_track_grid(n, 0, S)
    part = torch.empty(3 * S * acc.grid, dtype=torch.float64, device='cuda')
    acc.partials, acc.partials_len = part.data_ptr(), part.numel()
    ks = None
    if kicks:
        ks = N.KickSet()
        ks.slicer = sl.struct
        ks.n_kicks = len(kicks)
        for i, k in enumerate(kicks):
            ks.target[i], ks.quad[i], ks.kick[i] = 1, -1, k.data_ptr()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    N.call('phk_track', ctypes.byref(N.Program()), ctypes.byref(c),
           ctypes.byref(ks) if ks is not None else None, ctypes.byref(acc),
           stream)
    cnt = torch.empty(S, dtype=torch.int32, device='cuda')
    mx, my = (torch.empty(S, dtype=torch.float64, device='cuda')
              for _ in range(2))
    N.call('phk_slice_finalize', ctypes.byref(acc), cnt.data_ptr(),
           mx.data_ptr(), my.data_ptr(), 0, stream)
    return (cnt.cpu().numpy(), mx.cpu().numpy(), my.cpu().numpy(),
            mom[0].cpu().numpy(), acc.grid)


def _bins(z, S):
    idx = np.floor((z - CUTS[0]) / ((CUTS[1] - CUTS[0]) / float(S)))
    return np.where((idx >= 0) & (idx < S), idx, -1).astype(int)


def _exact_means(u, idx, S):
    order = np.argsort(idx, kind='stable')
    cut = np.searchsorted(idx[order], np.arange(S + 1))
    return np.array([math.fsum(u[order[a:b]]) / (b - a) if b > a else 0.
                     for a, b in zip(cut[:-1], cut[1:])])


def _check(got, x, y, z, S, scale=None):
    """One rounding per column and of the mean; the unit's truncation is far
    below."""
    idx = _bins(z, S)
    cnt, mx, my, _, grid = got
    np.testing.assert_array_equal(cnt, np.bincount(idx[idx >= 0], minlength=S))
    for u, m in ((x, mx), (y, my)):
        top = np.max(np.abs(u)) if scale is None else scale
        tol = 2.0**-58 * top + (grid + 3) * 2.0**-53 * np.max(np.abs(u))
        assert np.max(np.abs(m - _exact_means(u, idx, S))) <= tol


def _bunch(n, seed):
    rs = np.random.RandomState(seed)
    return rs.normal(0, 1e-3, n), rs.normal(0, 1e-5, n), rs.normal(0, 0.3, n)


@pytest.mark.parametrize('n,S', [(1, 1), (511, 3), (513, 50), (2049, 7),
                                 (300007, 200), (1000001, 1000)])
def test_sums_and_reproducibility(n, S):
    x, y, z = _bunch(n, n)
    a = _pass(x, y, z, S)
    _check(a, x, y, z, S)
    b = _pass(x, y, z, S)
    assert a[1].tobytes() == b[1].tobytes()
    assert a[2].tobytes() == b[2].tobytes()


@pytest.mark.parametrize('sign', [1., -1.])
def test_more_values_than_a_counter_holds(sign):
    """One cluster, one slice: 140000 values per CTA, all near the largest,
    so that every digit counter passes 2^16 values and carries."""
    n = 4 * 140000 + 77
    rs = np.random.RandomState(1)
    x = sign * (1e-3 - 1e-6 * rs.rand(n))
    y = -x[::-1].copy()
    z = np.full(n, 0.1)
    _check(_pass(x, y, z, 5, grid=1), x, y, z, 5)


def test_values_above_the_first_tiles():
    """Values 2^3 to 2^80 times their neighbours: the slices that hold one
    beyond 2^5 times a typical value are summed again."""
    n, S = 400000, 20
    x, y, z = _bunch(n, 5)
    x[300000:300040] *= 2.0 ** np.linspace(3, 80, 40)
    y[-1] = 4.0
    idx = _bins(z, S)
    got = _pass(x, y, z, S)
    big = np.zeros(S, dtype=bool)
    big[idx[300000:300040]] = True
    for u, m, hit in ((x, got[1], big),
                      (y, got[2], np.arange(S) == idx[-1])):
        want = _exact_means(u, idx, S)
        cnt = np.bincount(idx[idx >= 0], minlength=S)
        sums = np.bincount(idx[idx >= 0], weights=np.abs(u[idx >= 0]),
                           minlength=S)
        # FP64 sums of cnt values in any order
        tol = np.where(hit, cnt * 2.0**-53 * sums / np.maximum(cnt, 1),
                       100 * 2.0**-53 * np.max(np.abs(y)) + 1e-16 * 1e-3)
        assert np.all(np.abs(m - want) <= tol)


def test_non_finite_values():
    n, S = 50000, 10
    x, y, z = _bunch(n, 6)
    centre = CUTS[0] + (np.arange(S) + 0.5) * (CUTS[1] - CUTS[0]) / S
    z[-6:] = centre[[1, 2, 3, 4, 4, 5]]
    x[-6:] = [np.nan, np.inf, -np.inf, np.inf, -np.inf, 1e300]
    _, mx, my, _, _ = _pass(x, y, z, S)
    assert np.isnan(mx[1]) and mx[2] == np.inf and mx[3] == -np.inf
    assert np.isnan(mx[4]) and np.isfinite(mx[5]) and mx[5] > 1e290
    idx = _bins(z, S)
    rest = [0, 6, 7, 8, 9]
    x[-6:] = 0.
    want = _exact_means(x, idx, S)
    assert np.max(np.abs(mx[rest] - want[rest])) <= 1e-16
    assert np.max(np.abs(my - _exact_means(y, idx, S))) <= 1e-18


@pytest.mark.parametrize('later', [1e-3, 1e-300, 3e5])
def test_first_tiles_of_zeros(later):
    n, S = 700000, 8
    x, y, z = _bunch(n, 7)
    x[:640 * 512] = 0.
    x[640 * 512:] *= later / 1e-3
    idx = _bins(z, S)
    got = _pass(x, y, z, S)
    want = _exact_means(x, idx, S)
    cnt = np.bincount(idx[idx >= 0], minlength=S)
    # the unit is 2^-60 with nothing to scale by; sums beyond 4 are FP64
    tol = 2.0**-58 if later < 1 else cnt.max() * 2.0**-53 * np.max(np.abs(x))
    assert np.max(np.abs(got[1] - want)) <= tol + 100 * 2.0**-53 * \
        np.max(np.abs(want))


@pytest.mark.parametrize('n_kicks', [1, 2])
def test_largest_slice_count_with_kicks(n_kicks):
    """4096 slices: one kick table fits beside the histogram, two stay in
    global memory; both are applied."""
    n, S = 100003, 4096
    x, y, z = _bunch(n, 8)
    rs = np.random.RandomState(9)
    tables = [rs.normal(0, 1e-6, S) for _ in range(n_kicks)]
    dev = [torch.as_tensor(t).cuda() for t in tables]
    got = _pass(x, y, z, S, kicks=dev)
    _check(got, x, y, z, S)
    idx = _bins(z, S)
    want = np.where(idx >= 0, sum(t[idx] for t in tables), 0.)
    assert np.max(np.abs(got[3] - want)) <= 2 * 2.0**-53 * np.max(np.abs(want))
