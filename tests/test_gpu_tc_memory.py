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


def test_ring_spectra_are_released_once_packed(cuda, monkeypatch):
    """Ring spectra handed over in a list are gone when the first analysis runs; a tensor handed
    over is counted as held in the memory estimate."""
    import weakref

    import gmaster_b200 as nmt
    from gmaster_b200 import _lib, sht

    nside, lmax, nsims = 16, 47, 3
    maps = torch.randn((nsims, 12 * nside ** 2), dtype=torch.float64, device="cuda")
    mask = torch.rand(12 * nside ** 2, dtype=torch.float64, device="cuda")
    want = [f.get_alms() for f in nmt.fields_from_maps(mask, maps, n_iter=1, precision="mixed")]
    box = [sht.ring_analysis(sht.get_plan(nside, lmax), maps, _lib.MIXED, mask=mask)]
    ref, seen = weakref.ref(box[0]), []
    analysis = sht_tc._Batch.analysis

    def probe(self, scale):
        seen.append(ref() is None)
        return analysis(self, scale)

    monkeypatch.setattr(sht_tc._Batch, "analysis", probe)
    got = [f.get_alms() for f in nmt.fields_from_maps(mask, maps, n_iter=1, precision="mixed", ring_spectra=box)]
    assert box == [] and seen == [True, True]
    for g, w in zip(got, want):
        assert float((g - w).abs().max()) < 1e-12 * float(w.abs().max())
    tp = sht_tc.get_tc_plan(nside, lmax)
    spec = nsims * tp.plan.nring * tp.plan.L * 8
    assert sht_tc._full_path_bytes(tp, 0, nsims, 3, True) == sht_tc._full_path_bytes(tp, 0, nsims, 3) + spec


@pytest.mark.parametrize("spin,ncomp", [(0, 3), (2, 4)])
def test_transforms_that_run_out_of_memory_half_way(cuda, monkeypatch, spin, ncomp):
    """An allocation that fails between the iterations of the full-size transform, its buffers
    held: they are released before the transform starts again over windows."""
    nside, lmax = 64, 191
    gen = torch.Generator(device="cuda")
    gen.manual_seed(spin)
    maps = torch.randn((ncomp, 12 * nside ** 2), generator=gen, dtype=torch.float64, device="cuda")
    want = sht_tc.map2alm_tc(maps, spin, nside, lmax, 2, window=lmax + 1)
    synth = sht_tc.alm2map_tc(want, spin, nside, lmax, window=lmax + 1)
    sht_tc.map2alm_tc(maps, spin, nside, lmax, 2)   # the tables that are kept with the plan
    sht_tc.alm2map_tc(want, spin, nside, lmax)
    synthesis, windowed, held = sht_tc._Batch.synthesis, sht_tc.map2alm_tc_windowed, []

    def late(self, synd=None):
        out = synthesis(self, synd)
        torch.cuda.synchronize()
        _no_memory()
        return out

    def start(*args, **kwargs):
        held.append(torch.cuda.memory_allocated())
        return windowed(*args, **kwargs)

    monkeypatch.setattr(sht_tc._Batch, "synthesis", late)
    monkeypatch.setattr(sht_tc, "map2alm_tc_windowed", start)
    before = torch.cuda.memory_allocated()
    got = sht_tc.map2alm_tc(maps, spin, nside, lmax, 2)
    assert held == [before]
    assert float((got - want).abs().max() / want.abs().max()) < 2 * 2.0 ** -22
    assert torch.equal(sht_tc.alm2map_tc(want, spin, nside, lmax), synth)
