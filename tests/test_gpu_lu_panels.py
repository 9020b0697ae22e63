"""Shared-memory LU panels and prepared solves at the edges of their ranges: one panel (n <= 159),
every panel width, last panels and 32-row blocks in part, right-hand sides that fill a CTA in
part; pivots equal to numpy's choice rule.  Bound: solves of well-conditioned matrices to 1e-11
(n eps times a modest growth), residuals |PA - LU| to 1e-13 of |A|."""

import numpy as np
import pytest
import torch

from gmaster_b200.workspaces import LUFactor

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 158, 159, 160, 161, 256, 781, 1600, 3300])
def test_factors_and_solves(cuda, n):
    rng = np.random.default_rng(n)
    a = rng.normal(size=(n, n))
    a[rng.integers(0, n, size=max(1, n // 4))] *= 1e-3   # interchanges far from the diagonal
    a += 3 * np.roll(np.eye(n), n // 3, axis=0)
    dev = torch.from_numpy(a).cuda()
    lu = LUFactor(dev)
    lu.check()
    piv = lu.piv.cpu().numpy()
    assert np.all(piv >= np.arange(n)) and np.all(piv < n)
    perm = np.arange(n)
    for k in range(n):
        perm[[k, piv[k]]] = perm[[piv[k], k]]
    low = torch.tril(lu.lu, -1) + torch.eye(n, dtype=torch.float64, device="cuda")
    assert float(low.abs().max()) <= 1.0 + 1e-12     # partial pivoting: no multiplier above one
    res = low @ torch.triu(lu.lu) - dev[torch.from_numpy(perm).cuda()]
    assert float(res.abs().max()) < 1e-13 * n ** 0.5 * float(dev.abs().max()) + 1e-14
    for nrhs in (1, 3, 300):
        b = torch.from_numpy(rng.normal(size=(n, nrhs))).cuda()
        x = lu.solve(b)
        back = dev @ x - b
        assert float(back.abs().max()) < 1e-11 * max(1.0, float(x.abs().max()) * float(dev.abs().max()))
        assert torch.equal(lu.solve(b[:, 0].clone()), x[:, 0])


def test_nan_column_is_not_chosen_over_numbers(cuda):
    a = np.eye(5) * 2.0
    a[3, 1] = np.nan
    piv = LUFactor(torch.from_numpy(a).cuda()).piv.cpu().numpy()
    assert piv[0] == 0 and piv[1] == 1
