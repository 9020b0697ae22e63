"""Band sums of the covariance (k_cov_bands) against the element-by-element kernel, for bands of
uneven width (one multipole to several tiles), different binnings on the two sides and every
number of components.

Bound: double-precision sums of the same terms in another order (1e-13 of the largest entry)."""

import numpy as np
import pytest
import torch

from gmaster_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrows,nk,nblocks", [(4, 1, 1), (9, 3, 4), (16, 8, 16)])
def test_band_sums_match_elements(cuda, nrows, nk, nblocks):
    L = 150
    rng = np.random.default_rng(nrows)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    xi, spec = rng.normal(size=(nk, L, L)), rng.normal(size=(nrows, L))
    nterm = rng.integers(0, 20, size=nblocks)
    bptr = np.concatenate([[0], np.cumsum(nterm)]).astype(np.int32)
    terms = np.stack([rng.integers(0, nk, bptr[-1]), rng.integers(0, nrows, bptr[-1]),
                      rng.integers(0, nrows, bptr[-1])], 1).astype(np.int32)
    signs = rng.choice([-1.0, 1.0], size=bptr[-1])

    def bands(edges):
        ells = rng.permutation(np.arange(edges[0], edges[-1])).astype(np.int32)
        return (np.array(edges) - edges[0]).astype(np.int32), ells, rng.normal(size=L)

    (pa, ea, wa), (pb, eb, wb) = bands([2, 3, 19, 20, 37, 120]), bands([0, 16, 32, 97, 150])
    na, nb = len(pa) - 1, len(pb) - 1
    t = [dev(x) for x in (xi, spec, terms, signs, bptr, pa, ea, wa, pb, eb, wb)]
    want = torch.empty((nblocks, na, nb), dtype=torch.float64, device="cuda")
    got = torch.full_like(want, np.nan)
    st = _lib.stream_handle()
    p = [_lib.ptr(x) for x in t]
    _lib.call("gm_cov_binned", L - 1, nblocks, p[0], p[1], p[2], p[3], p[4], na, p[5], p[6], p[7], nb, p[8], p[9], p[10],
              _lib.ptr(want), st)
    host = [x.ctypes.data for x in (terms, signs, bptr)]
    _lib.call("gm_cov_bands", L - 1, nblocks, nk, _lib.ptr_array(list(t[0])), nrows, p[1], *host, na, p[5], p[6], p[7],
              nb, p[8], p[9], p[10], _lib.ptr(got), st)
    assert float((got - want).abs().max() / want.abs().max()) < 1e-13
    with pytest.raises(_lib.GMError):   # a term past the kernels given
        _lib.call("gm_cov_bands", L - 1, nblocks, 0, _lib.ptr_array(list(t[0])), nrows, p[1], *host, na, p[5], p[6],
                  p[7], nb, p[8], p[9], p[10], _lib.ptr(got), st)
