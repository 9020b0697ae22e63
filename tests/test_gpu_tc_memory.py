"""Batched transforms whose full-size buffers cannot be allocated: they run over windows of
orders instead, with the results of the windowed transforms."""

import numpy as np
import pytest
import torch

from gmaster_b200 import sht_tc

pytestmark = pytest.mark.gpu


def _no_memory(*args, **kwargs):
    raise torch.cuda.OutOfMemoryError("no memory for the full-size buffers")


@pytest.mark.parametrize("spin,ncomp", [(0, 1), (0, 3), (2, 4)])
def test_transforms_fall_back_to_windows(cuda, monkeypatch, spin, ncomp):
    nside, lmax = 16, 47
    rng = np.random.default_rng(5 + spin)
    maps = torch.from_numpy(rng.normal(size=(ncomp, 12 * nside ** 2))).cuda()
    mask = torch.from_numpy(rng.uniform(size=12 * nside ** 2)).cuda()
    want = sht_tc.map2alm_tc(maps, spin, nside, lmax, 2, mask=mask, window=lmax + 1)
    synth = sht_tc.alm2map_tc(want, spin, nside, lmax, window=lmax + 1)
    monkeypatch.setattr(sht_tc, "_map2alm_full", _no_memory)
    monkeypatch.setattr(sht_tc, "_synthesis_full", _no_memory)
    got = sht_tc.map2alm_tc(maps, spin, nside, lmax, 2, mask=mask)
    # the same kernels over the same window: only the order of the two hemisphere additions of
    # an alm (FP64) can differ, and what the single-precision iterations make of it (two of
    # them, each within 2^-22 of the largest value)
    assert float((got - want).abs().max() / want.abs().max()) < 2 * 2.0 ** -22
    assert torch.equal(sht_tc.alm2map_tc(want, spin, nside, lmax), synth)
