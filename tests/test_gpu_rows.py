"""One-field mixed-precision Legendre passes (legendre_rows.cu) against the FP64 passes on the
same operands, for every tile shape, at the edges of the 128-row segments and 8-row blocks,
with lanes that fill a CTA in part and with more maps than a tile holds.

Bound: a row carries the checkpoint's and 128 steps' single-precision roundings (below 2e-6 of
the row scale) and the sums are single precision over at most 3072 rows or 512 lanes of
random sign: 3e-6 of the result in the 2-norm."""

import pytest
import torch

from gmaster_b200 import _lib, autotune, sht

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax", [(4, 11), (16, 47), (32, 127), (32, 128), (64, 130), (96, 255), (256, 701)])
@pytest.mark.parametrize("spin,ncomp", [(0, 1), (0, 2), (0, 5), (2, 2), (2, 4)])
def test_rows_match_fp64(cuda, spin, ncomp, nside, lmax):
    plan = sht.get_plan(nside, lmax)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(nside + lmax + ncomp)
    rhs = torch.randn((plan.L, plan.nlanes, ncomp, 4), generator=gen, dtype=torch.float32, device="cuda")
    rhs[:, -1, :, 2:] = rhs[:, -1, :, :2]   # the equator has no southern ring: Diff = Sum
    alm = torch.randn((ncomp, plan.nelem), generator=gen, dtype=torch.complex128, device="cuda")
    ck = sht.ck_args(plan, spin, _lib.MIXED)
    assert ck is not None

    def both(prec, tile, ck):
        real = torch.float64 if prec == _lib.FP64 else torch.float32
        a = torch.zeros((ncomp, plan.nelem), dtype=torch.complex128, device="cuda")
        s = torch.empty((plan.L, plan.nlanes, ncomp, 4), dtype=real, device="cuda")
        sht.run_legendre(plan, spin, ncomp, prec, "ana", tile, rhs.to(real), a, -1.0, ck)
        sht.run_legendre(plan, spin, ncomp, prec, "syn", tile, alm, s, ck=ck)
        s[:, -1, :, 2:] = 0   # no southern ring: unspecified
        return a, s.to(torch.float64)

    want = both(_lib.FP64, -1, None)
    for tile in range(-1, len(autotune.tiles(spin))):
        for g, w in zip(both(_lib.MIXED, tile, ck), want):
            err = float(torch.linalg.vector_norm(g - w) / torch.linalg.vector_norm(w))
            assert err < 3e-6, (tile, err)


def test_a_pass_follows_the_settings_of_the_tables(cuda, monkeypatch):
    """Each setting that decides whether a pass takes the tables is looked at again when it changes."""
    from gmaster_b200 import sht_tc

    plan = sht.get_plan(16, 47)
    rhs = torch.randn((plan.L, plan.nlanes, 1, 4), device="cuda")
    alm = torch.zeros((1, plan.nelem), dtype=torch.complex128, device="cuda")

    def entry():
        before = dict(_lib.CALLS)
        sht.legendre_analysis(plan, 0, rhs, alm, 1.0, _lib.MIXED)
        return {k for k, v in _lib.CALLS.items() if v != before.get(k, 0) and k.startswith("gm_legendre_analysis")}

    entry()
    assert entry() == {"gm_legendre_analysis_ck"}
    for name, value in (("CK_MAX_LANES", 0), ("CK_MEMORY_SHARE", 0.0), ("USE_CHECKPOINTS", False)):
        with monkeypatch.context() as m:
            m.setattr(sht_tc, name, value)
            entry()
            assert entry() == {"gm_legendre_analysis_tile"}, name
        assert entry() == {"gm_legendre_analysis_ck"}
