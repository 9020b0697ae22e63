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


@pytest.mark.parametrize("lmax", [0, 1, 30, 511, 512, 1023, 1024, 1500])
@pytest.mark.parametrize("n1,n2", [(1, 1), (1, 2), (2, 2)])
def test_spectra_where_the_blocks_of_degrees_change(cuda, lmax, n1, n2):
    """Against torch sums in another order: 2^-53 times the square root of the terms, 1e-13."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(lmax)
    L = lmax + 1
    m = torch.repeat_interleave(torch.arange(L, device="cuda"), torch.arange(L, 0, -1, device="cuda"))
    ell = torch.arange(m.shape[0], device="cuda") - m * (2 * lmax + 1 - m) // 2
    a, b = (torch.randn((n, m.shape[0]), generator=gen, dtype=torch.complex128, device="cuda") for n in (n1, n2))
    for y in (b, a):
        got = pseudo_cl(a, y, lmax)
        prod = (a[:, None] * y[None].conj()).real.flatten(0, 1) * torch.where(m == 0, 1.0, 2.0)
        want = torch.zeros((prod.shape[0], L), dtype=torch.float64, device="cuda").index_add_(1, ell, prod)
        want /= 2.0 * torch.arange(L, device="cuda") + 1.0
        assert float((got - want).abs().max()) < 1e-13 * float(want.abs().max())


def test_one_pair_of_long_spectra_reads_at_the_memorys_rate(cuda):
    """Two (E, B) fields at lmax 3071 in less than 2.2 times a copy of the same bytes (three times
    where blocks of 32 degrees left a third of the chip idle)."""
    lmax = 3071
    a = torch.randn((4, (lmax + 1) * (lmax + 2) // 2), dtype=torch.complex128, device="cuda")
    dst = torch.empty_like(a[:2])

    def best(f):
        f()
        times = []
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(20):
                f()
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    assert best(lambda: pseudo_cl(a[:2], a[2:], lmax)) < 2.2 * best(lambda: dst.copy_(a[:2]))
