"""phk_exact_edges against the definition of the table: every edge is the
smallest float of its type whose reference index, floor((z - tail) / width),
reaches k (mirrored for width < 0), so its predecessor does not; no tolerance.
Sizes from no slice to thousands, tables through zero and far from it, widths
down to a few spacings of the floats, brackets that span zero with large
values; and what is refused."""
import numpy as np
import pytest

from pyheadtail_gb300 import _engine as E
from pyheadtail_gb300 import _native as N


@pytest.mark.parametrize('code', [N.PHK_F64, N.PHK_F32])
@pytest.mark.parametrize('tail,width,S', [
    (-0.69, 0.00276, 500), (0.69, -0.00276, 500), (-1e-9, 1e-12, 2000),
    (0., 1., 1), (0., 0.3, 0), (-5., 10., 3), (1.1e6, -1.7e6, 7),
    (0.25, 1e-3, 5000), (1., 2.**-21, 50), (-1e20, 1e19, 33)])
def test_edges_are_the_smallest_floats_of_their_slice(code, tail, width, S):
    e, neg = E.exact_edges(tail, width, S, code)
    dt = np.float64 if code == N.PHK_F64 else np.float32
    assert e.dtype == dt and e.shape == (S + 1,) and neg == (width < 0)
    k = np.arange(S + 1)

    def index(u):
        z = -u.astype(np.float64) if neg else u.astype(np.float64)
        return E.reference_index(z, tail, width)
    assert np.all(index(e) >= k)
    assert np.all(index(np.nextafter(e, dt(-np.inf))) < k)


@pytest.mark.parametrize('tail,width', [
    (1., 1e-30), (0., 0.), (np.inf, 1.), (0., np.nan), (np.nan, 1.)])
def test_what_has_no_edges_is_refused(tail, width):
    with pytest.raises(N.PhkError):
        E.exact_edges(tail, width, 10, N.PHK_F64)
