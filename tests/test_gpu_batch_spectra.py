"""Batched pseudo-spectra against one pair at a time and the definition, and the fused binning
and decoupling against its two steps, at the edges of the degree and row blocks and of a launch."""

import numpy as np
import pytest
import torch

import gmaster_b200 as nmt
from gmaster_b200.workspaces import LUFactor, pseudo_cl, pseudo_cl_pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax", [0, 31, 32, 200])
@pytest.mark.parametrize("n1,n2", [(1, 1), (1, 2), (2, 1), (2, 2), (3, 2)])
def test_pseudo_cl_pairs(cuda, n1, n2, lmax):
    """Any number of pairs equals one pair at a time bit for bit, and the definition to rounding."""
    nelem = (lmax + 1) * (lmax + 2) // 2
    npairs = 67
    a = torch.randn((npairs, n1, nelem), dtype=torch.complex128, device="cuda")
    b = torch.randn((npairs, n2, nelem), dtype=torch.complex128, device="cuda")
    got = pseudo_cl_pairs(list(a), list(b), lmax)
    ell, m = nmt.NmtAlmInfo(lmax).ell_m()
    w = torch.from_numpy(np.where(m == 0, 1.0, 2.0) / (2 * ell + 1.0)).cuda()
    for i in (0, 63, 66):
        assert torch.equal(got[i], pseudo_cl(a[i], b[i], lmax))
        for q in range(n1 * n2):
            c = torch.zeros(lmax + 1, dtype=torch.float64, device="cuda")
            c.index_add_(0, torch.from_numpy(ell).cuda(), w * (a[i, q // n2] * b[i, q % n2].conj()).real)
            assert float((got[i][q] - c).abs().max()) < 1e-13 * float(w.sum())


@pytest.mark.parametrize("ncells", [1, 5, 300])
@pytest.mark.parametrize("lmax,nlb,ncls", [(40, 5, 1), (191, 8, 4), (500, 3, 2)])
def test_decouple_is_bin_and_solve(cuda, lmax, nlb, ncls, ncells):
    """The fused binning and solve gives the solve of the binned spectra bit for bit, for spectra
    longer than lmax + 1 too."""
    bins = nmt.NmtBin.from_lmax_linear(lmax, nlb)
    n = bins.n_bands * ncls
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    mat = torch.randn((n, n), generator=gen, dtype=torch.float64, device="cuda") + 4 * torch.eye(
        n, dtype=torch.float64, device="cuda") * n ** 0.5
    lu = LUFactor(mat)
    cells = [torch.randn((ncls, lmax + 1 + 3), generator=gen, dtype=torch.float64, device="cuda") for _ in range(ncells)]
    got = lu.decouple(cells, bins)
    binned = torch.stack([bins.bin_cell(c[:, :lmax + 1].contiguous()) for c in cells])       # (cells, ncls, nb)
    want = lu.solve(binned.permute(2, 1, 0).reshape(n, ncells).contiguous())
    assert torch.equal(got, want)
