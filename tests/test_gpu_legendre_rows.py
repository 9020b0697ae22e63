"""FP64-recurrence Legendre passes (legendre.cu) against the oracle at the edges of the 128-row
segments and eight-row blocks, spins 0 to 3, both precisions of the contraction, for lanes that
fill a CTA in part.

Bound: double precision 1e-11 of the largest value (thousands of roundings of 1e-16 of the row
scale), single-precision contraction 2e-6."""

import numpy as np
import pytest
import torch

import oracle
from gmaster_b200 import sht, sht_tc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax", [(2, 5), (8, 23), (32, 127), (64, 128), (64, 135)])
@pytest.mark.parametrize("spin", [0, 1, 2, 3])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 2e-6)])
def test_rows_match_oracle(cuda, monkeypatch, spin, nside, lmax, precision, tol):
    monkeypatch.setattr(sht_tc, "USE_CHECKPOINTS", False)   # the FP64 recurrence in both precisions
    n = 1 if spin == 0 else 2
    rng = np.random.default_rng(nside + lmax + spin)
    maps = rng.normal(size=(n, 12 * nside ** 2))
    got = sht.map2alm_device(torch.from_numpy(maps).cuda(), spin, nside, lmax, 1, precision)
    want = oracle.map2alm(maps, spin, nside, lmax, 1)
    assert float(np.max(np.abs(got.cpu().numpy() - want)) / np.max(np.abs(want))) < tol
    back = sht.alm2map_device(torch.from_numpy(want).cuda(), spin, nside, lmax, precision).cpu().numpy()
    ref = oracle.alm2map(want, spin, nside, lmax)
    assert float(np.max(np.abs(back - ref)) / np.max(np.abs(ref))) < tol
