"""Binning of the coupling blocks by one warp and by eight warps per pair of bands: few, wide, many and
uneven bands, against dense products."""

import numpy as np
import pytest
import torch

import gmaster_b200 as nmt
from gmaster_b200 import _lib

pytestmark = pytest.mark.gpu


def _bin(bins, blocks, beam, ncls):
    """(ncls nb, ncls nb) binned matrix of blocks (4, L, L)."""
    nb, dev = bins.get_n_bands(), blocks.device
    ops = bins.device_operators(dev)
    out = torch.empty((ncls * nb,) * 2, dtype=torch.float64, device=dev)
    scratch = torch.empty(2 * nb * nb, dtype=torch.float64, device=dev)
    _lib.call("gm_bin_coupling_csr", bins.lmax, nb, ncls, _lib.ptr(blocks), _lib.ptr(ops["ptr"]), _lib.ptr(ops["ells"]),
              _lib.ptr(ops["wfl"]), _lib.ptr(ops["inv_fl"]), _lib.ptr(beam), _lib.ptr(scratch), _lib.ptr(out),
              _lib.stream_handle(dev))
    return out


# bands (first degree, end): one, few and wide, 48 and 49 of eight rows, 50 of 64, uneven with gaps
BANDS = [([2], [300]), ([2, 40, 41], [40, 41, 200]), (range(0, 384, 8), range(8, 392, 8)),
         (range(0, 392, 8), range(8, 400, 8)), (range(0, 3200, 64), range(64, 3264, 64)), ([3, 50, 90], [7, 90, 95])]


@pytest.mark.parametrize("first,end", BANDS)
@pytest.mark.parametrize("ncls", [1, 2, 4])
def test_binned_blocks(cuda, first, end, ncls):
    """Sums of at most L^2 products in another order: 1e-12 of the largest."""
    bins = nmt.NmtBin.from_edges(np.array(first), np.array(end), is_Dell=False)
    L, nb = bins.lmax + 1, bins.get_n_bands()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(L)
    blocks = torch.randn((4, L, L), generator=gen, dtype=torch.float64, device="cuda")
    beam = torch.rand(L, generator=gen, dtype=torch.float64, device="cuda") + 0.5
    ops = bins.device_operators(blocks.device)
    B, T = (torch.zeros((nb, L), dtype=torch.float64, device="cuda") for _ in range(2))
    for k, (a, b) in enumerate(zip(first, end)):
        B[k, a:b], T[k, a:b] = ops["wfl"][a:b], ops["inv_fl"][a:b]
    full = [B @ blocks[q] @ (T * beam).T for q in range(4)]
    got = _bin(bins, blocks, beam, ncls).reshape(nb, ncls, nb, ncls)
    diag = {1: full[0], 2: full[1], 4: full[2]}[ncls]
    for c in range(ncls):
        assert float((got[:, c, :, c] - diag).abs().max()) < 1e-12 * float(diag.abs().max())
    if ncls == 4:
        for a, b, sign in ((0, 3, 1), (1, 2, -1), (2, 1, -1), (3, 0, 1)):
            assert float((got[:, a, :, b] - sign * full[3]).abs().max()) < 1e-12 * float(full[3].abs().max())


def test_one_wide_band_is_spread_over_a_cta(cuda):
    """One band of 768 degrees, a single CTA, in less than 80 times twelve bands of 64 (40 times by eight
    warps, 200 by one)."""
    blocks = torch.randn((4, 768, 768), dtype=torch.float64, device="cuda")
    beam = torch.ones(768, dtype=torch.float64, device="cuda")

    def best(width):
        bins = nmt.NmtBin.from_edges(np.arange(0, 768, width), np.arange(width, 768 + width, width), is_Dell=False)
        _bin(bins, blocks, beam, 4)
        times = []
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(10):
                _bin(bins, blocks, beam, 4)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    assert best(768) < 80 * best(64)
