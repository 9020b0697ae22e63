"""E and B of the one-field passes under E >> B: neither carries the rounding of the other."""

import pytest
import torch

from gmaster_b200 import _lib, sht

pytestmark = pytest.mark.gpu

CASES = [(16, 47, 2, "mixed"), (64, 150, 2, "mixed"), (64, 191, 1, "mixed"), (32, 95, 3, "mixed"),
         (32, 77, 8, "mixed"), (32, 95, 2, "fp64"), (32, 90, 5, "fp64")]


def _setup(nside, lmax, precision):
    prec = _lib.FP64 if precision == "fp64" else _lib.MIXED
    real = torch.float64 if precision == "fp64" else torch.float32
    gen = torch.Generator(device="cuda")
    gen.manual_seed(nside + lmax)
    return sht.get_plan(nside, lmax), prec, real, gen


@pytest.mark.parametrize("nside,lmax,spin,precision", CASES)
def test_analysis_of_order_zero_keeps_q_and_u_apart(cuda, nside, lmax, spin, precision):
    """At m = 0 both row variants are equal: Q alone gives E alone, U alone gives B alone, exactly;
    and a U of 1e-4 Q gives B to the accuracy of the rows: 2e-6 of the row scale in single
    precision, and 2^-24 for each of at most 16 levels of the sums."""
    plan, prec, real, gen = _setup(nside, lmax, precision)
    rhs = torch.randn((plan.L, plan.nlanes, 2, 4), generator=gen, device="cuda", dtype=real)
    for zero in (0, 1):
        one = rhs.clone()
        one[:, :, zero] = 0
        alm = torch.zeros((2, plan.nelem), dtype=torch.complex128, device="cuda")
        sht.legendre_analysis(plan, spin, one, alm, 1.0, prec)
        assert bool((alm[zero, : plan.L] == 0).all())
        assert bool((alm[1 - zero, spin: plan.L] != 0).any())
    rhs[:, :, 1] *= 1e-4
    got = torch.zeros((2, plan.nelem), dtype=torch.complex128, device="cuda")
    want = torch.zeros_like(got)
    sht.legendre_analysis(plan, spin, rhs, got, 1.0, prec)
    sht.legendre_analysis(plan, spin, rhs.double(), want, 1.0, _lib.FP64)
    err = (got - want)[1, : plan.L].norm() / want[1, : plan.L].norm()
    assert float(err) < 3e-6


@pytest.mark.parametrize("nside,lmax,spin,precision", CASES)
def test_synthesis_of_order_zero_keeps_e_and_b_apart(cuda, nside, lmax, spin, precision):
    """At m = 0 Q comes from E alone and U from B alone, a B of 1e-4 E included (bound: 2e-6 for
    the rows, 2^-24 times the square root of the lmax + 1 terms of a sum, twice)."""
    plan, prec, real, gen = _setup(nside, lmax, precision)
    alm = torch.randn((2, plan.nelem), generator=gen, device="cuda", dtype=torch.complex128)
    for zero in (0, 1):
        one = alm.clone()
        one[zero] = 0
        syn = sht.legendre_synthesis(plan, spin, one, 2, prec)
        assert bool((syn[0, :, zero] == 0).all())
        assert bool((syn[0, :, 1 - zero] != 0).any())
    alm[1] *= 1e-4
    got = sht.legendre_synthesis(plan, spin, alm, 2, prec).double()
    want = sht.legendre_synthesis(plan, spin, alm, 2, _lib.FP64)
    err = (got - want)[0, :, 1].norm() / want[0, :, 1].norm()
    assert float(err) < 4e-6


@pytest.mark.parametrize("nside,lmax,spin,tiles", [(256, 767, 1, {0: 0, 1: 1, 2: 2, 3: 9}),
                                                   (256, 767, 4, {0: 0, 2: 2}), (64, 191, 1, {0: 0})])
def test_single_precision_sums_of_spin_s_err_no_more_than_those_of_spin_zero(cuda, nside, lmax, spin, tiles):
    """Mixed passes from double-precision rows: the error is that of the single-precision sums,
    R lanes a thread and 32 threads a tree (analysis) or the rows of an order (synthesis), for E and B
    as for one spin-0 map with the same R (tiles: spin s -> spin 0); 3 % for the draw."""
    plan, prec, real, gen = _setup(nside, lmax, "mixed")
    rhs = torch.randn((plan.L, plan.nlanes, 2, 4), generator=gen, device="cuda", dtype=real)
    alm = torch.randn((2, plan.nelem), generator=gen, device="cuda", dtype=torch.complex128)

    def errors(s, tile):
        nc = 1 if s == 0 else 2
        out = []
        for kind, src in (("ana", rhs[:, :, :nc].contiguous()), ("syn", alm[:nc].contiguous())):
            shape, kinds = ((nc, plan.nelem), (torch.complex128,) * 2) if kind == "ana" else (
                (plan.L, plan.nlanes, nc, 4), (torch.float32, torch.float64))
            got, want = (torch.zeros(shape, dtype=k, device="cuda") for k in kinds)
            sht.run_legendre(plan, s, nc, prec, kind, tile, src, got)
            sht.run_legendre(plan, s, nc, _lib.FP64, kind, -1, src.double() if kind == "ana" else src, want)
            out.append(float((got - want).norm() / want.norm()))
        return out

    for tile, same in tiles.items():
        for got, ref in zip(errors(spin, tile), errors(0, same)):
            assert got < 1.03 * ref
