"""Plain form: the undetuned transverse map bit for bit against NumPy's
separately rounded products and sums, where its integer products could go
wrong: exact ties, results that round up to the next power of two, either
normalisation, factors with few bits, and the particles and matrices that
leave them (zeros, subnormals, huge values, infinities, NaN)."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip('torch')

ONE = 1.0
MATRICES = [
    [0.68, 36.6, -0.0146, 0.68, 0.43, 45.2, -0.018, 0.43],
    [1.5, 0.75, 3.0, -1.25, 1 - 2.0**-53, 1 + 2.0**-52, -2 + 2.0**-52, 0.5],
    [1.0, 2.0**-400, -2.0**400, 1.0, 1 / 3., 2 / 3., -1 / 7., 1e-17],
    [0.0, 50.0, -0.02, 0.0, 1.0, 0.0, 0.0, 1.0],        # exact zeros
    [1e200, 1.0, 1.0, 1e-200, 1.0, 1e-308, 1.0, 1.0],   # outside the window
]


def _coordinates(n, special):
    rs = np.random.RandomState(7)
    out = []
    for k in range(4):
        v = rs.normal(0, 1., n) * 10.0 ** rs.uniform(-6, 0, n)
        bits = v.view(np.uint64).copy()
        # few significant bits, all ones, one bit set at either end
        keep = rs.randint(0, 53, n).astype(np.uint64)
        cut = rs.rand(n) < 0.5
        bits[cut] &= ~((np.uint64(1) << keep[cut]) - np.uint64(1))
        ones = rs.rand(n) < 0.1
        bits[ones] |= np.uint64((1 << 52) - 1)
        v = bits.view(np.float64)
        if special:
            odd = np.array([0., -0., 5e-324, -1e-310, 2.3e-308, 1e-160, 1e160,
                            -1e300, 1.7e308, np.inf, -np.inf, np.nan,
                            2.0**-511, 2.0**512, 2.0**-512, 2.0**511])
            v[rs.randint(0, n, n // 8)] = odd[rs.randint(0, len(odd), n // 8)]
        out.append(v)
    return out


@pytest.mark.parametrize('special', [False, True])
@pytest.mark.parametrize('M', MATRICES)
def test_bits(M, special):
    from pyheadtail_gb300 import _native as N
    N.load()
    n = 100001
    x, xp, y, yp = _coordinates(n, special)
    dev = [torch.as_tensor(v.copy()).cuda() for v in (x, xp, y, yp)]
    rest = [torch.zeros(n, dtype=torch.float64, device='cuda') for _ in range(2)]
    c = N.Coords()
    c.x, c.xp, c.y, c.yp, c.z, c.dp = (t.data_ptr() for t in dev + rest)
    c.n, c.dtype = n, 0
    prog = N.Program()
    prog.n_ops = 1
    prog.op[0].kind = N.OP_TRANSVERSE
    for i, v in enumerate(M):
        prog.op[0].p[i] = v
    N.call('phk_track', ctypes.byref(prog), ctypes.byref(c), None, None,
           ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    with np.errstate(all='ignore'):
        want = [M[0] * x + M[1] * xp, M[2] * x + M[3] * xp,
                M[4] * y + M[5] * yp, M[6] * y + M[7] * yp]
    for k in range(4):
        got = dev[k].cpu().numpy()
        nan = np.isnan(want[k])
        assert np.array_equal(np.isnan(got), nan)
        same = got.view(np.uint64) == want[k].view(np.uint64)
        assert np.all(same | nan), (k, int(np.sum(~(same | nan))))
