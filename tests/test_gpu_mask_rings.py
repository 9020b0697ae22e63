"""Mask apodisation where the search passes over rings: masked pixels at the poles and on both sides
of the longitude origin, single pixels, rings of four pixels and rings longer than a warp, radii
from one pixel to the whole sphere, against the minimum over all pairs of pixels.

Bound: the chord of a pair to a few roundings of 1e-16, the taper's slope 2 / radius: 1e-11."""

import numpy as np
import pytest
import torch

import gmaster_b200 as nmt
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
