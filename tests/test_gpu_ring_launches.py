"""The launches of the ring stages: all rings in one up to Nside 128, the longest caps with the belt,
components shared by a CTA or not; a map's result does not depend on the maps beside it."""

import pytest
import torch

from gmaster_b200 import _lib, sht

pytestmark = pytest.mark.gpu


def _stages(nside, lmax, ncomp, prec, seed=0):
    plan = sht.get_plan(nside, lmax)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    real = torch.float64 if prec == _lib.FP64 else torch.float32
    maps = torch.randn((ncomp, plan.npix), generator=gen, dtype=torch.float64, device="cuda")
    syn = torch.randn((plan.L, plan.nlanes, ncomp, 4), generator=gen, dtype=real, device="cuda")
    return plan, maps, syn


@pytest.mark.parametrize("nside", [1, 2, 8, 64, 66, 127, 128, 129, 134, 256, 257])
@pytest.mark.parametrize("prec", [_lib.MIXED, _lib.FP64])
def test_components_do_not_depend_on_one_another(cuda, nside, prec):
    """One map alone and first and last of 50.  Single precision: the same analysis bit for bit, and
    a synthesis whose alias sums (at most L / 4 terms) are in another order, 1e-6; double precision:
    2^-53 a step also where rings of prime factors above 64 go directly instead of by Bluestein's
    method, 1e-13."""
    plan, maps, syn = _stages(nside, 2 * nside, 50, prec)
    spec, out = sht.ring_analysis(plan, maps, prec), sht.ring_synthesis(plan, syn, prec)
    for c in (0, 49):
        one = sht.ring_analysis(plan, maps[c:c + 1], prec)[0]
        back = sht.ring_synthesis(plan, syn[:, :, c:c + 1].contiguous(), prec)[0]
        tol = 1e-6 if prec == _lib.MIXED else 1e-13
        assert torch.equal(spec[c], one) or (prec == _lib.FP64 and
                                             float((spec[c] - one).abs().max()) <= tol * float(one.abs().max()))
        assert float((out[c] - back).abs().max()) <= tol * float(back.abs().max())


@pytest.mark.parametrize("nside", [128, 256])
def test_single_precision_rings_match_double(cuda, nside):
    plan, maps, syn = _stages(nside, 3 * nside - 1, 3, _lib.FP64)
    for stage, x, y in ((sht.ring_analysis, maps, maps), (sht.ring_synthesis, syn, syn.float())):
        want, got = stage(plan, x, _lib.FP64), stage(plan, y, _lib.MIXED)
        assert float((got - want).norm() / want.norm()) < 1e-6   # 3 transforms of at most 2^10 points


@pytest.mark.parametrize("prec", [_lib.MIXED, _lib.FP64])
def test_sixteen_small_maps_run_side_by_side(cuda, prec):
    """16 maps at Nside 64 in less than 3.2 times the time of one (eight components in turn per CTA: 4
    to 4.4 times; side by side 2)."""
    def best(ncomp):
        plan, maps, _ = _stages(64, 191, ncomp, prec)
        out = sht.ring_analysis(plan, maps, prec)
        times = []
        for _ in range(8):
            e0, e1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            e0.record()
            for _ in range(50):
                sht.ring_analysis(plan, maps, prec, out=out)
            e1.record()
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    assert best(16) < 3.2 * best(1)


@pytest.mark.parametrize("prec", [_lib.MIXED, _lib.FP64])
def test_synthesis_without_room_for_the_folded_spectra(cuda, monkeypatch, prec):
    """The transform that took no workspace before still runs where none can be had (single
    precision: sums in another order, 1e-6; double 1e-12)."""
    plan, _, syn = _stages(128, 300, 2, prec)
    want = sht.ring_synthesis(plan, syn, prec)
    empty = torch.empty

    def full(*args, **kwargs):
        if kwargs.get("dtype") is torch.uint8:
            raise torch.cuda.OutOfMemoryError("no memory for the workspace")
        return empty(*args, **kwargs)

    monkeypatch.setattr(torch, "empty", full)
    got = sht.ring_synthesis(plan, syn, prec)
    assert float((got - want).norm() / want.norm()) < (1e-6 if prec == _lib.MIXED else 1e-12)
