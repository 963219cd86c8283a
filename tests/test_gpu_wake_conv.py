"""phk_wake, numpy path: the fixed-point convolution against extended
precision at the edges of its blocks (32 targets, up to 96 sources, 4 CTAs of
16 warps) and where a unit has to run in FP64 (infinite, subnormal or extreme
factors); below a million multiply-adds the direct kernel runs.

Every factor is off by at most 2^-54 of the largest of its unit, a unit's sum
is rounded once and at most lags * chunks + 16 sums are added:
|error| <= 2^-52 * sum over stored turns of S * max|m| * max|table|."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')


def _run(moments, tables, lags, head, dtype=0):
    """Every kick's convolution; moments [R][3][S], tables [kick][lags][2S-1],
    kick k from moment 1 + k % 2."""
    from pyheadtail_gb300 import _native as N
    N.load()
    R, _, S = moments.shape
    m = torch.as_tensor(moments).cuda()
    t = [torch.as_tensor(np.ascontiguousarray(x)).cuda() for x in tables]
    out = torch.full((len(t), S), np.nan, device='cuda',
                     dtype=torch.float64 if dtype == 0 else torch.float32)
    w = N.WakeSet()
    w.n_slices, w.ring_len, w.head, w.n_kicks = S, R, head, len(t)
    w.out_dtype, w.moments = dtype, m.data_ptr()
    for k, x in enumerate(t):
        st = w.kick[k]
        st.source, st.n_lags, st.dense, st.factor = 1 + k % 2, lags[k], 0, -1.5
        st.table, st.out = x.data_ptr(), out[k].data_ptr()
    N.call('phk_wake', ctypes.byref(w),
           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    return out.cpu().numpy()


def _want(moments, table, lags, head, source):
    R, _, S = moments.shape
    L = np.longdouble
    out, bound = np.zeros(S, dtype=L), 0.
    for a in range(lags):
        m = moments[(head - a) % R, source]
        with np.errstate(invalid='ignore', over='ignore'):
            out = out + np.convolve(m.astype(L), table[a].astype(L), 'valid')
        bound += S * np.max(np.abs(m)) * np.max(np.abs(table[a]))
    return L(-1.5) * out, 1.5 * bound


@pytest.mark.parametrize('dtype', [0, 1])
@pytest.mark.parametrize('S,R', [(1, 1), (2, 3), (63, 1), (64, 2), (65, 9),
                                 (128, 1), (129, 5), (500, 50), (1000, 3),
                                 (4096, 2), (33, 600), (64, 140), (96, 60),
                                 (97, 61), (192, 15)])
def test_against_extended_precision(S, R, dtype):
    rs = np.random.RandomState(S + R)
    moments = rs.normal(0, 1., (R, 3, S)) * np.exp(rs.uniform(-3, 3, S))
    lags = [1, R, max(1, R - 1)]
    t = np.arange(2 * S - 1) - (S - 1.)
    tables = [np.where(t < 0, np.exp(t / 9.) * np.sin(t), 0.)[None] * 3e17,
              np.array([-1e15 / np.sqrt(abs(t.min()) + 2. + t + 2 * S * a)
                        for a in range(R)]),
              rs.normal(0, 1., (R, 2 * S - 1))]
    head = R // 2
    got = _run(moments, tables, lags, head, dtype)
    for k in range(3):
        want, bound = _want(moments, tables[k], lags[k], head, 1 + k % 2)
        tol = 2.0**-52 * bound
        if dtype == 1:
            tol = tol + 2.0**-24 * np.abs(want).astype(float)
        assert np.all(np.abs(got[k] - want) <= tol), k


def test_zero_moments_and_extreme_scales():
    S, R = 200, 16
    rs = np.random.RandomState(3)
    moments = np.zeros((R, 3, S))
    moments[0, 1, 50:60] = rs.normal(0, 1e-120, 10)     # turn of age 0
    moments[1, 2, 100:] = rs.normal(0, 1e120, S - 100)
    tables = [rs.normal(0, 1e-120, (R, 2 * S - 1)),
              rs.normal(0, 1e90, (R, 2 * S - 1))]
    tables[0][0, ::7] = 0.
    got = _run(moments, tables, [R, R], 0)
    for k in range(2):
        want, bound = _want(moments, tables[k], R, 0, 1 + k)
        assert np.all(np.abs(got[k] - want) <= 2.0**-52 * bound), k
    assert np.any(got[0] != 0) and np.any(got[1] != 0)


def test_non_finite_factors_stay_where_they_belong():
    """NaN and infinite factors reach the targets a floating-point loop
    would give them to, and no other."""
    S = 1100
    rs = np.random.RandomState(4)
    moments = rs.normal(0, 1., (1, 3, S))
    table = rs.normal(0, 1., (1, 2 * S - 1))
    table[0, 2 * S - 3] = np.inf          # target S-1 from source 1, S-2 from 0
    got = _run(moments, [table], [1], 0)[0]
    assert np.flatnonzero(~np.isfinite(got)).tolist() == [S - 2, S - 1]
    want, bound = _want(moments, np.where(np.isfinite(table), table, 0.), 1, 0, 1)
    keep = slice(0, S - 2)
    assert np.all(np.abs(got[keep] - want[keep]) <= 2.0**-52 * bound)
    moments[0, 1, 7] = np.nan
    assert np.all(np.isnan(_run(moments, [np.ones((1, 2 * S - 1))], [1], 0)[0]))
