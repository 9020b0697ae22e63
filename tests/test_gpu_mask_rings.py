"""Mask apodisation where the search passes over rings: masked pixels at the poles and on both sides
of the longitude origin, single pixels, rings of four pixels and rings longer than a warp, radii
from one pixel to the whole sphere, against the minimum over all pairs of pixels.

Bound: the chord of a pair to a few roundings of 1e-16, the taper's slope 2 / radius: 1e-11."""

import numpy as np
import pytest
import torch

import gmaster_b200 as nmt
from gmaster_b200 import _lib
from gmaster_b200.utils import pix2vec_ring

pytestmark = pytest.mark.gpu


def _want(mask, radius, apotype):
    v = torch.from_numpy(pix2vec_ring(int(round((mask.size / 12) ** 0.5)))).cuda()
    m = torch.from_numpy(mask).cuda()
    bad, good = v[m <= 0], torch.nonzero(m > 0)[:, 0]
    out = m.clone()
    if len(bad) == 0:
        return out
    d2 = torch.cat([((v[g][:, None] - bad[None]) ** 2).sum(2).min(1).values for g in good.split(512)])
    thr = 1 - np.cos(radius)
    x = torch.sqrt(0.5 * d2 / thr)
    f = x - torch.sin(2 * np.pi * x) / (2 * np.pi) if apotype == "C1" else 0.5 * (1 - torch.cos(np.pi * x))
    out[good] *= torch.where(d2 < 2 * thr, f, torch.ones_like(x))
    return out


@pytest.mark.parametrize("nside,degrees", [(2, 80.0), (4, 60.0), (16, 5.0), (16, 179.0), (32, 12.0), (64, 2.0)])
@pytest.mark.parametrize("pattern", ["poles", "seam", "single", "sparse", "none"])
@pytest.mark.parametrize("apotype", ["C1", "C2"])
def test_nearest_masked_pixel(cuda, nside, degrees, pattern, apotype):
    npix = 12 * nside ** 2
    rng = np.random.default_rng(nside)
    mask = rng.uniform(0.5, 1.5, size=npix)
    offset = np.concatenate([[0], np.cumsum([4 * min(i, nside, 4 * nside - i) for i in range(1, 4 * nside)])])[:-1]
    if pattern == "poles":
        mask[[0, 2, npix - 1]] = 0.0
    elif pattern == "seam":   # the last pixel of some rings, the first of others
        mask[offset[nside] - 1] = mask[offset[2 * nside]] = mask[offset[2 * nside + 1] - 1] = -1.0
    elif pattern == "single":
        mask[npix // 3] = 0.0
    elif pattern == "sparse":
        mask[rng.integers(0, npix, size=max(2, npix // 300))] = 0.0
    got = nmt.mask_apodization(torch.from_numpy(mask).cuda(), degrees, apotype=apotype)
    want = _want(mask, np.radians(degrees), apotype)
    assert float((got - want).abs().max()) < 1e-11


@pytest.mark.parametrize("nside,degrees", [(4, 90.0), (16, 179.0), (32, 10.0), (64, 3.0)])
@pytest.mark.parametrize("pattern", ["half", "one ring", "rows", "last pixel", "all"])
def test_dense_masks_and_whole_empty_rings(cuda, nside, degrees, pattern):
    """Masks whose search ends at the neighbours, and rings far from the nearest masked pixel."""
    npix = 12 * nside ** 2
    rng = np.random.default_rng(nside)
    mask = rng.uniform(0.5, 1.5, size=npix)
    offset = np.concatenate([[0], np.cumsum([4 * min(i, nside, 4 * nside - i) for i in range(1, 4 * nside)])])
    if pattern == "half":
        mask[rng.integers(0, 2, size=npix) == 0] = 0.0
    elif pattern == "one ring":
        mask[offset[nside]:offset[nside + 1]] = 0.0
    elif pattern == "rows":
        for r in range(1, 4 * nside - 1, 3):
            mask[offset[r]:offset[r + 1]:2] = 0.0
    elif pattern == "last pixel":
        mask[-1] = 0.0
    else:
        mask[:] = 0.0
    for apotype in ("C1", "C2"):
        got = nmt.mask_apodization(torch.from_numpy(mask).cuda(), degrees, apotype=apotype)
        assert float((got - _want(mask, np.radians(degrees), apotype)).abs().max()) < 1e-11


@pytest.mark.parametrize("nside", [1, 2, 8, 9, 64, 300])
def test_ring_gaps(cuda, nside):
    """Distances to the nearest ring with a masked pixel."""
    rng = np.random.default_rng(nside)
    nring, npix = 4 * nside - 1, 12 * nside ** 2
    offset = np.concatenate([[0], np.cumsum([4 * min(i, nside, 4 * nside - i) for i in range(1, 4 * nside)])])[:-1]
    for full in ([], [0], [nring - 1], sorted(rng.choice(nring, size=max(1, nring // 20), replace=False))):
        prev = torch.full((npix,), -1, dtype=torch.int32, device="cuda")
        prev[torch.from_numpy(offset[np.array(full, dtype=int)]).cuda()] = 0
        gaps = torch.empty(nring, dtype=torch.int32, device="cuda")
        _lib.call("gm_mask_ring_gaps", nside, _lib.ptr(prev), _lib.ptr(gaps), _lib.stream_handle(prev.device))
        want = (np.abs(np.arange(nring)[:, None] - np.array(full)[None]).min(1) if full
                else np.full(nring, 2 ** 31 - 1))
        np.testing.assert_array_equal(gaps.cpu().numpy(), want)


def test_the_search_ends_where_nothing_nearer_can_be_found(cuda):
    """The time of masks whose distances are known at once does not grow with the radius: no masked
    pixel, and every second one (10 and 5 times as long at 20 degrees when all rings are tested)."""
    def best(mask, degrees):
        nmt.mask_apodization(mask, degrees)
        times = []
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(5):
                nmt.mask_apodization(mask, degrees)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    npix = 12 * 512 ** 2
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1)
    ones = torch.ones(npix, dtype=torch.float64, device="cuda")
    for mask in (ones, (torch.rand(npix, generator=gen, device="cuda") < 0.5).double()):
        assert best(mask, 20.0) < 2.0 * best(mask, 1.0)
